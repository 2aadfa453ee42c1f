// The scan on box grids: FFT sizes chosen per axis (Nx, Ny, Nz), as the
// reference sizes its grid (findBestSize<N_dim> per axis over the padded
// receptor box, include/PRODDL/docking_fft.hpp:541-553 and
// include/PRODDL/Math/fft.hpp:141-168), and cubic edges without a compiled
// plan.  Same pipeline and conventions as the cubic kernels -- ligand prep
// (rotate, toLogical per axis, stable sort by (term, x)), pencil stage
// (y/z stages as direct sums over the ligand's entries, x transform,
// spectrum product summed over terms, inverse x transform), plane stage
// (inverse y transform, real inverse z transform, exact per-plane top 16),
// finalize (merge, FP64 direct-space rescoring, sort, maxValCorr, unwrap per
// axis) -- with every transform length a runtime value: one warp per line
// runs a mixed-radix Stockham FFT (radices 4, 6, 2, 9, 3, 5, 7, 11, 13 in
// that order of preference) out of shared memory with a twiddle table per
// axis (even-length plane rows: two lines per warp, 16 lanes each).  The receptor's transforms
// run the same line FFT in FP64.
//
// Layout (Hz = Nz/2 + 1, pencil p = ky Hz + kz, PP = Ny Hz rounded up to 32):
//   spec  [K][Nx][PP]  float2  R^_t(kx, p) / V
//   rgrid [K][V]       double  real-space receptor terms (FP64 rescoring)
//   ent   [B][n_ent]   uint32  t << 24 | x << 16 | y << 8 | z, sorted by (t, x)
//   offs  [B][K Nx+1]  int32   start of bin (t, x)
//   g2    [B][Nx][PP]  float2  per-x complex (ky, kz) planes
//   cand  [B][Nx][16]          per-plane FP32 candidate pools
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "fft_core.cuh"
#include "internal.h"
#include "pencil_tc.cuh"
#include "scan_kernels.cuh"

namespace fftdock {

namespace {

constexpr int kBoxWarps = 8;  // lines (pencils, columns, rows) per CTA

// radices in Stockham stage order; false if n has another prime factor
bool factor_plan(int n, BoxPlan& pl) {
    static const int radices[] = {4, 6, 2, 9, 3, 5, 7, 11, 13};
    pl.n = n;
    pl.nf = 0;
    int m = n;
    for (int r : radices)
        while (m % r == 0 && pl.nf < kBoxMaxFactors) {
            pl.f[pl.nf++] = r;
            m /= r;
        }
    return m == 1 && n >= 2;
}

template <typename T2> __device__ __forceinline__ T2 c_mul(T2 a, T2 b) {
    T2 r;
    r.x = a.x * b.x - a.y * b.y;
    r.y = a.x * b.y + a.y * b.x;
    return r;
}
// table entry W_n^m = e^{-2 pi i m / n}, conjugated for the inverse transform
template <typename T2, int SIGN> __device__ __forceinline__ T2 tw_at(const T2* tw, int m) {
    T2 w = tw[m];
    if (SIGN > 0) w.y = -w.y;
    return w;
}

// one Stockham stage of radix R over a line of n points held in src:
// butterfly j reads src[j + r n/R], applies the twiddles W^(j mod Ns) r n/(Ns R),
// and writes its R-point DFT to dst[(j / Ns) Ns R + j mod Ns + k Ns].  The
// twiddle index (j mod Ns) r n/(Ns R) stays below n; the R-th roots of unity
// are held in registers for the whole stage, radices 2 and 4 need none, 6
// is two 3-point DFTs joined by W6 twiddles.
template <typename T2, int SIGN, int R>
__device__ __forceinline__ void stockham_stage(const T2* src, T2* dst, const T2* tw, int n, int ns, int lane) {
    using S = decltype(T2::x);
    const int nb = n / R;
    const int tstep = n / (ns * R);
    // j / ns as a multiply-high by ceil(2^32 / ns) (ns > 1): exact for
    // j < 2^32 / ns^2 (here j < 256 and ns <= 256)
    const unsigned magic = ns > 1 ? 0xffffffffu / (unsigned)ns + 1u : 0u;
    T2 root[R];
    root[0].x = 1;  // W^0 (a composite odd radix pairs some q k = 0 mod R)
    root[0].y = 0;
#pragma unroll
    for (int m = 1; m < R; ++m) root[m] = tw_at<T2, SIGN>(tw, m * nb);
    for (int j = lane; j < nb; j += 32) {
        T2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = src[j + r * nb];
        const int jq = ns > 1 ? (int)__umulhi((unsigned)j, magic) : j;
        const int jm = j - jq * ns;
        const int step = jm * tstep;
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = c_mul(v[r], tw_at<T2, SIGN>(tw, step * r));
        T2* out = dst + jq * ns * R + jm;
        if constexpr (R == 2) {
            T2 o0 = v[0], o1 = v[0];
            o0.x += v[1].x; o0.y += v[1].y;
            o1.x -= v[1].x; o1.y -= v[1].y;
            out[0] = o0;
            out[ns] = o1;
        } else if constexpr (R == 6) {
            // two 3-point DFTs of the even and odd inputs, the odd ones
            // turned by W6^k (W6 = e^(SIGN i pi / 3)): out_k = e_k + W6^k o_k,
            // out_(k+3) = e_k - W6^k o_k
            constexpr S c3 = (S)0.86602540378443864676;  // sin(pi / 3)
            constexpr S sg = SIGN < 0 ? (S)-1 : (S)1;
            T2 e3[3], o3[3];
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const T2 x0 = v[t], x1 = v[t + 2], x2 = v[t + 4];
                T2 sm, df, u;
                sm.x = x1.x + x2.x; sm.y = x1.y + x2.y;
                df.x = sg * c3 * (x1.x - x2.x); df.y = sg * c3 * (x1.y - x2.y);
                u.x = x0.x - (S)0.5 * sm.x; u.y = x0.y - (S)0.5 * sm.y;
                T2* y = t == 0 ? e3 : o3;
                y[0].x = x0.x + sm.x; y[0].y = x0.y + sm.y;
                // y1 = u + i df, y2 = u - i df
                y[1].x = u.x - df.y; y[1].y = u.y + df.x;
                y[2].x = u.x + df.y; y[2].y = u.y - df.x;
            }
            // W6 = (1/2, sg c3), W6^2 = (-1/2, sg c3)
            T2 t1, t2;
            t1.x = (S)0.5 * o3[1].x - sg * c3 * o3[1].y; t1.y = (S)0.5 * o3[1].y + sg * c3 * o3[1].x;
            t2.x = (S)-0.5 * o3[2].x - sg * c3 * o3[2].y; t2.y = (S)-0.5 * o3[2].y + sg * c3 * o3[2].x;
            T2 o;
            o.x = e3[0].x + o3[0].x; o.y = e3[0].y + o3[0].y; out[0] = o;
            o.x = e3[1].x + t1.x; o.y = e3[1].y + t1.y; out[ns] = o;
            o.x = e3[2].x + t2.x; o.y = e3[2].y + t2.y; out[2 * ns] = o;
            o.x = e3[0].x - o3[0].x; o.y = e3[0].y - o3[0].y; out[3 * ns] = o;
            o.x = e3[1].x - t1.x; o.y = e3[1].y - t1.y; out[4 * ns] = o;
            o.x = e3[2].x - t2.x; o.y = e3[2].y - t2.y; out[5 * ns] = o;
        } else if constexpr (R == 4) {
            // W4 = e^(SIGN i pi / 2): out1 = (v0 - v2) + W4 (v1 - v3), out3 = (v0 - v2) - W4 (v1 - v3)
            T2 a, b, c, d, e;
            a.x = v[0].x + v[2].x; a.y = v[0].y + v[2].y;
            b.x = v[0].x - v[2].x; b.y = v[0].y - v[2].y;
            c.x = v[1].x + v[3].x; c.y = v[1].y + v[3].y;
            e.x = v[1].x - v[3].x; e.y = v[1].y - v[3].y;
            if (SIGN < 0) { d.x = e.y; d.y = -e.x; } else { d.x = -e.y; d.y = e.x; }
            T2 o;
            o.x = a.x + c.x; o.y = a.y + c.y; out[0] = o;
            o.x = b.x + d.x; o.y = b.y + d.y; out[ns] = o;
            o.x = a.x - c.x; o.y = a.y - c.y; out[2 * ns] = o;
            o.x = b.x - d.x; o.y = b.y - d.y; out[3 * ns] = o;
        } else {
            // odd R: pairs a_q = v_q + v_(R-q), b_q = v_q - v_(R-q); with
            // root[m] = (cos, s sin) of the stage's direction,
            // out_k = v0 + sum_q cos(qk) a_q + i sum_q s sin(qk) b_q and
            // out_(R-k) the same with - i
            constexpr int P = (R - 1) / 2;
            T2 o0 = v[0];
#pragma unroll
            for (int q = 1; q <= P; ++q) {
                o0.x += v[q].x + v[R - q].x;
                o0.y += v[q].y + v[R - q].y;
            }
            out[0] = o0;
#pragma unroll
            for (int k = 1; k <= P; ++k) {
                T2 re = v[0];
                S ix = 0, iy = 0;
#pragma unroll
                for (int q = 1; q <= P; ++q) {
                    const T2 w = root[(q * k) % R];
                    re.x += w.x * (v[q].x + v[R - q].x);
                    re.y += w.x * (v[q].y + v[R - q].y);
                    ix += w.y * (v[q].x - v[R - q].x);
                    iy += w.y * (v[q].y - v[R - q].y);
                }
                // i (ix + i iy) = (-iy, ix)
                T2 o;
                o.x = re.x - iy; o.y = re.y + ix; out[k * ns] = o;
                o.x = re.x + iy; o.y = re.y - ix; out[(R - k) * ns] = o;
            }
        }
    }
}

// Unnormalised DFT of the warp's line in a (n points), b a second buffer of
// n points; returns the buffer that holds the result.  SIGN -1: forward
// e^{-2 pi i jk/n}; +1: inverse.  Ends with __syncwarp..
template <typename T2, int SIGN>
__device__ T2* warp_fft(T2* a, T2* b, const T2* tw, const BoxPlan& pl, int lane) {
    T2* src = a;
    T2* dst = b;
    int ns = 1;
    __syncwarp();
    for (int s = 0; s < pl.nf; ++s) {
        const int R = pl.f[s];
        switch (R) {
            case 4: stockham_stage<T2, SIGN, 4>(src, dst, tw, pl.n, ns, lane); break;
            case 6: stockham_stage<T2, SIGN, 6>(src, dst, tw, pl.n, ns, lane); break;
            case 2: stockham_stage<T2, SIGN, 2>(src, dst, tw, pl.n, ns, lane); break;
            case 3: stockham_stage<T2, SIGN, 3>(src, dst, tw, pl.n, ns, lane); break;
            case 5: stockham_stage<T2, SIGN, 5>(src, dst, tw, pl.n, ns, lane); break;
            case 7: stockham_stage<T2, SIGN, 7>(src, dst, tw, pl.n, ns, lane); break;
            case 9: stockham_stage<T2, SIGN, 9>(src, dst, tw, pl.n, ns, lane); break;
            case 11: stockham_stage<T2, SIGN, 11>(src, dst, tw, pl.n, ns, lane); break;
            default: stockham_stage<T2, SIGN, 13>(src, dst, tw, pl.n, ns, lane); break;
        }
        __syncwarp();
        T2* t = src;
        src = dst;
        dst = t;
        ns *= R;
    }
    return src;
}

// ---------------------------------------------------------------------------
// receptor transforms (FP64), one warp per line: line L starts at
// (L / inner_count) outer_stride + (L % inner_count) inner_stride, element e
// at + e elem_stride; in place
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(32 * kBoxWarps) box_line_fft64_kernel(double2* __restrict__ data,
                                                                       const double2* __restrict__ tw, BoxPlan pl,
                                                                       long n_lines, long elem_stride,
                                                                       long inner_count, long inner_stride,
                                                                       long outer_stride) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = pl.n;
    double2* tws = reinterpret_cast<double2*>(smem_raw);  // [n]
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double2* a = tws + n + (size_t)w * 2 * n;
    double2* b = a + n;
    for (int i = threadIdx.x; i < n; i += blockDim.x) tws[i] = tw[i];
    __syncthreads();
    const long L = (long)blockIdx.x * kBoxWarps + w;
    if (L >= n_lines) return;
    double2* line = data + (L / inner_count) * outer_stride + (L % inner_count) * inner_stride;
    for (int e = lane; e < n; e += 32) a[e] = line[(long)e * elem_stride];
    const double2* r = warp_fft<double2, -1>(a, b, tws, pl, lane);
    for (int e = lane; e < n; e += 32) line[(long)e * elem_stride] = r[e];
}

// [Nx][Ny][Nz] complex -> [Nx][Ny][Hz]
__global__ void box_half_extract_kernel(const double2* __restrict__ full, double2* __restrict__ half, int nx, int ny,
                                        int nz, int hz) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t tot = (size_t)nx * ny * hz;
    if (i >= tot) return;
    const size_t row = i / hz;
    const int kz = (int)(i - row * hz);
    half[i] = full[row * nz + kz];
}

// ---------------------------------------------------------------------------
// ligand prep: rotate (the reference's operation order, no FMA), toLogical
// per axis, bins (t, x), stable sort (one CTA per rotation)
// ---------------------------------------------------------------------------
// ent_t (tensor form): the transposed entries of ligand_prep_kernel
__global__ void __launch_bounds__(256) box_prep_kernel(const double* __restrict__ rot,
                                                       const double* __restrict__ lig_xyz,
                                                       const int32_t* __restrict__ lig_term, int n_ent, int K, Geo geo,
                                                       uint32_t* __restrict__ ent_out, int32_t* __restrict__ offs_out,
                                                       int32_t* __restrict__ status, const float* __restrict__ w_in,
                                                       uint4* __restrict__ ent4, int32_t* __restrict__ idx_out,
                                                       uint32_t* __restrict__ ent_t, const int32_t* __restrict__ tpad,
                                                       int n_pad, int x0, int W, int qc) {
    extern __shared__ unsigned char smem_raw[];
    const int nx = geo.n[0], ny = geo.n[1], nz = geo.n[2];
    // bins (t, x, y mod qc), qc = 1 or 2
    const int nbins = K * nx * qc, qm = qc - 1;
    int32_t* cnt = reinterpret_cast<int32_t*>(smem_raw);           // [nbins + 1]
    uint32_t* keys = reinterpret_cast<uint32_t*>(cnt + nbins + 1);  // [n_ent]
    __shared__ int bad;
    __shared__ int wsum[8];
    const int q = blockIdx.x;
    const int tid = threadIdx.x;
    for (int i = tid; i <= nbins; i += blockDim.x) cnt[i] = 0;
    if (tid == 0) bad = 0;
    __syncthreads();
    const double* m = rot + 9 * (size_t)q;
    for (int i = tid; i < n_ent; i += blockDim.x) {
        const double x0 = lig_xyz[3 * i], x1 = lig_xyz[3 * i + 1], x2 = lig_xyz[3 * i + 2];
        const double p0 = __dadd_rn(__dadd_rn(__dmul_rn(m[0], x0), __dmul_rn(m[1], x1)), __dmul_rn(m[2], x2));
        const double p1 = __dadd_rn(__dadd_rn(__dmul_rn(m[3], x0), __dmul_rn(m[4], x1)), __dmul_rn(m[5], x2));
        const double p2 = __dadd_rn(__dadd_rn(__dmul_rn(m[6], x0), __dmul_rn(m[7], x1)), __dmul_rn(m[8], x2));
        int c0 = logical_q(p0, geo, 0), c1 = logical_q(p1, geo, 1), c2 = logical_q(p2, geo, 2);
        const bool ok = c0 >= 1 && c0 <= nx && c1 >= 1 && c1 <= ny && c2 >= 1 && c2 <= nz;
        if (!ok) atomicOr(&bad, 1);
        // out-of-grid atoms are clamped for memory safety; the rotation is
        // reported and gives no peaks
        c0 = min(max(c0 - 1, 0), nx - 1);
        c1 = min(max(c1 - 1, 0), ny - 1);
        c2 = min(max(c2 - 1, 0), nz - 1);
        const int t = lig_term[i];
        keys[i] = ((uint32_t)t << 24) | ((uint32_t)c0 << 16) | ((uint32_t)c1 << 8) | (uint32_t)c2;
        atomicAdd(&cnt[(t * nx + c0) * qc + (c1 & qm)], 1);
    }
    __syncthreads();
    {
        const int per = (nbins + blockDim.x - 1) / blockDim.x;
        const int b0 = min(tid * per, nbins), b1 = min(b0 + per, nbins);
        int local = 0;
        for (int i = b0; i < b1; ++i) local += cnt[i];
        const int lane = tid & 31, wid = tid >> 5;
        int incl = local;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) wsum[wid] = incl;
        __syncthreads();
        int wbase = 0;
        for (int k = 0; k < wid; ++k) wbase += wsum[k];
        int run = wbase + incl - local;
        for (int i = b0; i < b1; ++i) {
            const int c = cnt[i];
            cnt[i] = run;
            run += c;
        }
        __syncthreads();
        if (tid == 0) cnt[nbins] = n_ent;
        __syncthreads();
    }
    int32_t* offs = offs_out + (size_t)q * (nbins + 1);
    for (int i = tid; i <= nbins; i += blockDim.x) offs[i] = cnt[i];
    __syncthreads();
    if (tid < 32) {
        uint32_t* ent = ent_out + (size_t)q * n_ent;
        for (int base = 0; base < n_ent; base += 32) {
            const int i = base + tid;
            const bool act = i < n_ent;
            const uint32_t key = act ? keys[i] : 0xffffffffu;
            const int bin = act ? (int)((key >> 24) * nx + ((key >> 16) & 255u)) * qc + (int)((key >> 8) & qm) : -1;
            const unsigned peers = __match_any_sync(0xffffffffu, bin);
            const int rank = __popc(peers & ((1u << tid) - 1u));
            const int leader = __ffs(peers) - 1;
            int dst = 0;
            if (act) dst = cnt[bin] + rank;
            __syncwarp();
            if (act) ent[dst] = key;
            // [q / 128][row / 4][q % 128][row % 4], x relative to x0 (cells
            // outside the window at the dummy row W), as in ligand_prep_kernel
            if (act && ent_t) {
                const size_t row = (size_t)(dst + __ldg(tpad + (key >> 24)));
                ent_t[(((size_t)(q >> 7) * (n_pad >> 2) + (row >> 2)) * 128 + (q & 127)) * 4 + (row & 3)] =
                    (min(((key >> 16) - (uint32_t)x0) & 255u, (uint32_t)W) << 24) | (((key >> 8) & 255u) << 16) |
                    (key & 255u);
            }
            if (act && ent4) {
                // ljComp: entry i < n_ent / 2 weighs atom i into term 0, entry
                // i + n_ent / 2 the same atom into term 1
                const int half = n_ent >> 1;
                if (i < half)
                    ent4[(size_t)q * half + dst] =
                        make_uint4(key, __float_as_uint(w_in[i]), __float_as_uint(w_in[i + half]), 0u);
                idx_out[(size_t)q * n_ent + dst] = i;
            }
            if (act && tid == leader) cnt[bin] += __popc(peers);
            __syncwarp();
        }
    }
    if (tid == 0) status[q] = bad;
}

// ---------------------------------------------------------------------------
// finalize: merge the Nx x KC pools, FP64 direct-space rescoring of the KC
// best cells (mod each axis' size), sort by (energy, offset), maxValCorr,
// translation = h unwrap(cell) per axis.  One CTA per rotation.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) box_finalize_kernel(
    const float* __restrict__ cand_v, const int32_t* __restrict__ cand_i, const uint32_t* __restrict__ ent,
    const int32_t* __restrict__ status, const double* __restrict__ rgrid, int n_ent, int nx, int ny, int nz,
    int peak_stride, int k_out, double max_val, double h, int first_rot_id, fftdock_peak* __restrict__ peaks,
    int32_t* __restrict__ n_peaks, float* __restrict__ pool_v, int32_t* __restrict__ pool_i,
    const double* __restrict__ w64, const int32_t* __restrict__ ent_idx) {
    __shared__ float lv_s[8 * KC];
    __shared__ int li_s[8 * KC];
    __shared__ double score_s[KC];
    const int q = blockIdx.x;
    const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
    const long V = (long)nx * ny * nz;
    const int ncand = nx * KC;
    WarpTopK tk;
    tk.init();
    const float* cv = cand_v + (size_t)q * ncand;
    const int32_t* ci = cand_i + (size_t)q * ncand;
    for (int base = w * 32; base < ncand; base += 256) {
        const int e = base + l;
        tk.offer(e < ncand ? cv[e] : INFINITY, e < ncand ? ci[e] : 0x7fffffff, l);
    }
    if (l < KC) {
        lv_s[w * KC + l] = tk.lv;
        li_s[w * KC + l] = tk.li;
    }
    __syncthreads();
    if (w == 0) {
        merge_lists(lv_s, li_s, 8 * KC, tk, l);
        __syncwarp();
        if (l < KC) {
            lv_s[l] = tk.lv;
            li_s[l] = tk.li;
        }
    }
    __syncthreads();
    if (pool_v != nullptr && tid < KC) {
        pool_v[(size_t)q * KC + tid] = lv_s[tid];
        pool_i[(size_t)q * KC + tid] = li_s[tid];
    }
    const uint32_t* e_q = ent + (size_t)q * n_ent;
    for (int c = w; c < KC; c += 8) {
        const int off = li_s[c];
        double sum = 0.0;
        const bool ok = off >= 0 && off < V;
        if (ok) {
            const int sx = off / (ny * nz), sy = (off / nz) % ny, sz = off % nz;
            for (int j = l; j < n_ent; j += 32) {
                const uint32_t u = e_q[j];
                const int t = (int)(u >> 24);
                const int ax = (int)((u >> 16) & 255u), ay = (int)((u >> 8) & 255u), az = (int)(u & 255u);
                const int gx = ax - sx < 0 ? ax - sx + nx : ax - sx;
                const int gy = ay - sy < 0 ? ay - sy + ny : ay - sy;
                const int gz = az - sz < 0 ? az - sz + nz : az - sz;
                const double rv = rgrid[(size_t)t * V + ((size_t)gx * ny + gy) * nz + gz];
                sum = __dadd_rn(sum, w64 ? __dmul_rn(w64[ent_idx[(size_t)q * n_ent + j]], rv) : rv);
            }
            for (int o = 16; o > 0; o >>= 1) sum = __dadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, o));
        }
        if (l == 0) score_s[c] = ok ? sum : INFINITY;
    }
    __syncthreads();
    if (tid == 0) {
        double sc[KC];
        int of[KC];
        for (int c = 0; c < KC; ++c) {
            sc[c] = score_s[c];
            of[c] = li_s[c];
        }
        for (int a2 = 1; a2 < KC; ++a2) {
            const double s = sc[a2];
            const int o = of[a2];
            int b2 = a2 - 1;
            while (b2 >= 0 && (sc[b2] > s || (sc[b2] == s && of[b2] > o))) {
                sc[b2 + 1] = sc[b2];
                of[b2 + 1] = of[b2];
                --b2;
            }
            sc[b2 + 1] = s;
            of[b2 + 1] = o;
        }
        int n = 0;
        if (status[q] == 0) {
            const int dims[3] = {nx, ny, nz};
            for (int c = 0; c < KC && n < k_out; ++c) {
                if (!(sc[c] < max_val) || of[c] < 0 || of[c] >= V) continue;
                fftdock_peak pk;
                pk.rot_id = first_rot_id + q;
                pk.cell[0] = of[c] / (ny * nz);
                pk.cell[1] = (of[c] / nz) % ny;
                pk.cell[2] = of[c] % nz;
                for (int d = 0; d < 3; ++d) {
                    int yv = -pk.cell[d];
                    if (yv < -(dims[d] / 2)) yv += dims[d];
                    pk.t[d] = h * (double)yv;
                }
                pk.score = sc[c];
                peaks[(size_t)q * peak_stride + n] = pk;
                ++n;
            }
        }
        n_peaks[q] = n;
    }
}

// the pencil stage's share of the size limit a ligand is accepted under
// (tables, line buffers and staged entries of 8 pencils per CTA;
// pencil_lines_kernel needs less and nothing per entry)
size_t pencil_limit_bytes(int nx, int ny, int nz, int K, int n_ent, bool weighted) {
    return (size_t)(nx + ny + nz) * sizeof(float2) + (size_t)kBoxWarps * (ny + nz + 3 * nx) * sizeof(float2) +
           (size_t)kBoxWarps * nx * sizeof(float2) + (size_t)n_ent * sizeof(uint32_t) * (weighted ? 2 : 1) +
           ((size_t)K + 1) * sizeof(int32_t);
}
// the plane's share of the size limit a ligand is accepted under (plane,
// twiddles and 16 line buffers; plane_lines_kernel needs less)
size_t plane_limit_bytes(int ny, int nz) {
    const int hz = nz / 2 + 1, lmax = std::max(ny, nz);
    return ((size_t)ny * (hz | 1) + ny + nz + nz / 2 + (size_t)16 * 2 * lmax) * sizeof(float2);
}
size_t prep_smem_bytes(int nx, int K, int n_ent, int qc) {
    return ((size_t)K * nx * qc + 1) * sizeof(int32_t) + (size_t)n_ent * sizeof(uint32_t);
}

cudaError_t set_smem(const void* fn, size_t bytes) {
    if (bytes <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

cudaError_t box_prep(const BatchArgs& a, cudaStream_t s) {
    const int nb = a.n_rot;
    if (nb <= 0) return cudaSuccess;
    const size_t sm = prep_smem_bytes(a.box.n[0], a.K, a.n_ent, a.classes());
    cudaError_t e = set_smem((const void*)box_prep_kernel, sm);
    if (e != cudaSuccess) return e;
    box_prep_kernel<<<nb, 256, sm, s>>>(a.rot, a.lig_xyz, a.lig_term, a.n_ent, a.K, a.box, a.ent, a.offs, a.status,
                                        a.lig_w32, a.lig_w32 ? a.ent4 : nullptr, a.ent_idx,
                                        a.use_tc ? a.ent_t : nullptr, a.tpad, a.n_pad, a.x0, a.W, a.classes());
    return cudaGetLastError();
}

cudaError_t box_middle(const BatchArgs& a, cudaStream_t s) {
    const int nb = a.n_rot;
    if (nb <= 0) return cudaSuccess;
    const int nx = a.box.n[0], ny = a.box.n[1], nz = a.box.n[2];
    const float2* twx = a.box_tw32;
    const float2* twy = twx + nx;
    const float2* twz = twy + ny;
    cudaError_t e;
    if (a.ev && (e = cudaEventRecord(a.ev[0], s)) != cudaSuccess) return e;
    const int np = ny * (nz / 2 + 1);
    if (a.use_tc) {
        // tensor form: the x stage as split-FP16 tcgen05 GEMMs over 128
        // rotations per CTA, then the plane stage from its x-quads
        const int nxp = (nx + 3) / 4 * 4;
        const size_t smt = tc_smem_bytes_box(nx, ny, nz, a.W / 8, a.n_tc_terms);
        dim3 gridt(np, (nb + TC_ROT - 1) / TC_ROT);
        const int tg = a.tc_group > 0 ? a.tc_group : FFTDOCK_TC_TERMS_PER_SUM_DEFAULT;
        const TcBox bx{nx, ny, nz, nz / 2 + 1, np, nxp, twy, twz};
        if (tc_tiles(nx) == 1) {
            if ((e = set_smem((const void*)pencil_tc_kernel<0, 1>, smt)) != cudaSuccess) return e;
            pencil_tc_kernel<0, 1><<<gridt, TC_THREADS, smt, s>>>(a.circ, a.cscale, a.ent_t, a.tinfo, a.n_tc_terms,
                                                                 nullptr, a.g2t, a.n_pad, nb, a.x0, a.W, tg,
                                                                 a.tc_slots, a.tc_n_slots, bx, a.err);
        } else {
            if ((e = set_smem((const void*)pencil_tc_kernel<0, 2>, smt)) != cudaSuccess) return e;
            pencil_tc_kernel<0, 2><<<gridt, TC_THREADS, smt, s>>>(a.circ, a.cscale, a.ent_t, a.tinfo, a.n_tc_terms,
                                                                 nullptr, a.g2t, a.n_pad, nb, a.x0, a.W, tg,
                                                                 a.tc_slots, a.tc_n_slots, bx, a.err);
        }
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        if (a.ev && (e = cudaEventRecord(a.ev[1], s)) != cudaSuccess) return e;
        e = box_plane(a, twy, twz, true, s);
        if (e != cudaSuccess) return e;
        if (a.ev && (e = cudaEventRecord(a.ev[2], s)) != cudaSuccess) return e;
        return cudaSuccess;
    }
    if ((e = box_pencil(a, twx, twy, twz, s)) != cudaSuccess) return e;
    if (a.ev && (e = cudaEventRecord(a.ev[1], s)) != cudaSuccess) return e;
    e = box_plane(a, twy, twz, false, s);
    if (e != cudaSuccess) return e;
    if (a.ev && (e = cudaEventRecord(a.ev[2], s)) != cudaSuccess) return e;
    return cudaSuccess;
}

cudaError_t box_finish(const BatchArgs& a, cudaStream_t s) {
    const int nb = a.n_rot;
    if (nb <= 0) return cudaSuccess;
    box_finalize_kernel<<<nb, 256, 0, s>>>(a.cand_v, a.cand_i, a.ent, a.status, a.rgrid, a.n_ent, a.box.n[0],
                                           a.box.n[1], a.box.n[2], a.peak_stride, a.k_out, a.max_val, a.h,
                                           a.first_rot_id, a.peaks, a.n_peaks, a.pool_v, a.pool_i, a.lig_w64,
                                           a.lig_w64 ? a.ent_idx : nullptr);
    return cudaGetLastError();
}

cudaError_t box_scan_batch(const BatchArgs& a, cudaStream_t s) {
    cudaError_t e = box_prep(a, s);
    if (e != cudaSuccess) return e;
    BatchArgs m = a;
    m.ev = nullptr;
    if ((e = box_middle(m, s)) != cudaSuccess) return e;
    return box_finish(a, s);
}

size_t box_pencil_smem_unknown(int, int) { return 0; }

cudaError_t box_load_kernels(int) {
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, (const void*)box_prep_kernel);
    if (e == cudaSuccess) e = box_pencil_load();
    if (e == cudaSuccess) e = box_plane_load();
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, (const void*)box_finalize_kernel);
    return e;
}

}  // namespace

bool box_plan(int n, BoxPlan* pl) { return factor_plan(n, *pl); }

size_t box_pencil_smem(int nx, int ny, int nz, int K, int n_ent, bool weighted) {
    return std::max(pencil_limit_bytes(nx, ny, nz, K, n_ent, weighted),
                    std::max(plane_limit_bytes(ny, nz), prep_smem_bytes(nx, K, n_ent, 1)));
}

// Forward transform of one real FP64 term grid [Nx][Ny][Nz] into spec_t
// ([Nx][PP] float2, scaled 1 / V): complex z transforms, the half spectrum
// kz < Hz, then y and x transforms, each a batch of line FFTs.
cudaError_t box_receptor_fft(const double* rgrid_t, double2* cbuf, double2* hbuf, const double2* tw64,
                             const int dims[3], void* spec_t, int PP, float2* circ_t, cudaStream_t s) {
    const int nx = dims[0], ny = dims[1], nz = dims[2], hz = nz / 2 + 1;
    BoxPlan px, py, pz;
    if (!factor_plan(nx, px) || !factor_plan(ny, py) || !factor_plan(nz, pz)) return cudaErrorInvalidValue;
    const double2* twx = tw64;
    const double2* twy = twx + nx;
    const double2* twz = twy + ny;
    const size_t V = (size_t)nx * ny * nz;
    complexify_kernel<<<(unsigned)((V + 255) / 256), 256, 0, s>>>(rgrid_t, cbuf, V);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    auto lines = [&](double2* data, const double2* tw, const BoxPlan& pl, long n_lines, long es, long ic, long is,
                     long os) -> cudaError_t {
        const size_t sm = ((size_t)pl.n + (size_t)kBoxWarps * 2 * pl.n) * sizeof(double2);
        cudaError_t e2 = set_smem((const void*)box_line_fft64_kernel, sm);
        if (e2 != cudaSuccess) return e2;
        const long blocks = (n_lines + kBoxWarps - 1) / kBoxWarps;
        box_line_fft64_kernel<<<(unsigned)blocks, 32 * kBoxWarps, sm, s>>>(data, tw, pl, n_lines, es, ic, is, os);
        return cudaGetLastError();
    };
    // z: lines (x, y), contiguous
    if ((e = lines(cbuf, twz, pz, (long)nx * ny, 1, 1, 0, nz)) != cudaSuccess) return e;
    const size_t nh = (size_t)nx * ny * hz;
    box_half_extract_kernel<<<(unsigned)((nh + 255) / 256), 256, 0, s>>>(cbuf, hbuf, nx, ny, nz, hz);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    // y: lines (x, kz) of [Nx][Ny][Hz]
    if ((e = lines(hbuf, twy, py, (long)nx * hz, hz, hz, 1, (long)ny * hz)) != cudaSuccess) return e;
    if (circ_t) {
        // transformed along z and y only: the tensor stage's circulant samples
        const size_t tot = (size_t)nx * ny * hz;
        pack_circ_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(hbuf, circ_t, nx, ny * hz,
                                                                     1.0 / ((double)ny * nz));
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    // x: lines p = (ky, kz)
    if ((e = lines(hbuf, twx, px, (long)ny * hz, (long)ny * hz, (long)ny * hz, 1, 0)) != cudaSuccess) return e;
    const size_t tot = (size_t)nx * PP;
    pack_spectrum_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(hbuf, static_cast<float2*>(spec_t), nx, ny * hz, PP,
                                                                       1.0 / (double)V);
    return cudaGetLastError();
}

cudaError_t box_circ_scales(const float2* circ, int K, int nh, int nx, int8_t* cscale, cudaStream_t s) {
    circ_scale_box_kernel<<<(nh + 127) / 128, 128, 0, s>>>(circ, K, nh, nx, cscale);
    return cudaGetLastError();
}

size_t box_tc_smem(const int dims[3], int n_chunks, int n_terms) {
    return tc_smem_bytes_box(dims[0], dims[1], dims[2], n_chunks, n_terms);
}

size_t cubic_tc_smem(int n, int n_chunks, int n_terms) { return tc_smem_bytes(n, n_chunks, n_terms); }

const SizeOps* box_ops() {
    static const SizeOps o{0, nullptr, nullptr, false, &box_scan_batch, &box_pencil_smem_unknown, &box_prep,
                           &box_middle, &box_finish, &box_load_kernels};
    return &o;
}

}  // namespace fftdock
