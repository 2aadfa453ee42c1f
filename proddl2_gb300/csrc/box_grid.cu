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
// axis) -- with every transform length a runtime value.  This file holds prep,
// finalize and the launches; the stages are pencil_tcp.cuh / pencil_tc.cuh (tensor
// form), pencil_lines.cuh through pencil_box*.cu (FFT form), plane_lines.cuh
// through plane_box.cu, and receptor_fft.cu for the receptor's transforms.
//
// Layout (Hz = Nz/2 + 1, pencil p = ky Hz + kz, PP = Ny Hz rounded up to 32):
//   spec  [K][Nx][PP]  float2  R^_t(kx, p) / V
//   rgrid [K][V]       double  real-space receptor terms (FP64 rescoring)
//   ent   [B][n_ent]   uint32  t << 24 | x << 16 | y << 8 | z, sorted by (t, x, y mod qc);
//                             tensor form: by (t, x), read by the rescoring only
//   offs  [B][K Nx qc+1]  int32  start of bin (t, x, y mod qc)
//   g2    [B][Nx][PP]  float2  per-x complex (ky, kz) planes
//   cand  [B][Nx][16]          per-plane FP32 candidate pools
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "fft_core.cuh"
#include "internal.h"
#include "pencil_tc.cuh"
#include "pencil_tcp.cuh"
#include "scan_kernels.cuh"

namespace fftdock {

namespace {

constexpr int kBoxWarps = 8;  // lines (pencils, columns, rows) per CTA

// ---------------------------------------------------------------------------
// ligand prep: rotate (the reference's operation order, no FMA), toLogical
// per axis, bins (t, x, y mod qc), stable sort (one CTA per rotation)
// ---------------------------------------------------------------------------
// ent_t (tensor form): the transposed entries of ligand_prep_kernel
__global__ void __launch_bounds__(256) box_prep_kernel(const double* __restrict__ rot,
                                                       const double* __restrict__ lig_xyz,
                                                       const int32_t* __restrict__ lig_term, int n_ent, int K, Geo geo,
                                                       uint32_t* __restrict__ ent_out, int32_t* __restrict__ offs_out,
                                                       int32_t* __restrict__ status, const float* __restrict__ w_in,
                                                       uint4* __restrict__ ent4, int32_t* __restrict__ idx_out,
                                                       uint32_t* __restrict__ ent_t, const int32_t* __restrict__ tpad,
                                                       int n_pad, int x0, int W, int qc, const int32_t* __restrict__ tinfo,
                                                       int ka) {
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
    if (!ent_t)  // (the tensor form does not read them)
        for (int i = tid; i <= nbins; i += blockDim.x) offs[i] = cnt[i];
    // pencil pairs: which staging rows of each term hold an entry, one bit per
    // row, after the term rows (a quad of rows per term)
    for (int i = tid; i < 3 * ka; i += blockDim.x) {
        const int kk = i / 3, word = i - 3 * kk, t = tinfo[ka + 1 + kk];
        uint32_t m = 0;
        for (int j = 0; j < 16; ++j) {
            const int xr = 16 * word + j, c = xr + x0;
            if (xr < W && c >= 0 && c < nx) {
                const int b = (t * nx + c) * qc;
                m |= (uint32_t)(cnt[b + 1] > cnt[b]) << (2 * j) | (uint32_t)(cnt[b + 2] > cnt[b + 1]) << (2 * j + 1);
            }
        }
        ent_t[(((size_t)(q >> 7) * (n_pad >> 2) + (tinfo[ka] >> 2) + kk) * 128 + (q & 127)) * 4 + word] = m;
    }
    __syncthreads();
    if (ka) pair_counts(cnt, nbins);
    auto scatter = [&](auto pairs) {
        uint32_t* ent = ent_out + (size_t)q * n_ent;
        for (int base = 0; base < n_ent; base += 32) {
            const int i = base + tid;
            const bool act = i < n_ent;
            const uint32_t key = act ? keys[i] : 0xffffffffu;
            const int bin = act ? (int)((key >> 24) * nx + ((key >> 16) & 255u)) * qc + (int)((key >> 8) & qm) : -1;
            const EntrySlot at = entry_slot<decltype(pairs)::value>(cnt, bin, tid);
            const int leader = __ffs(at.peers) - 1;
            __syncwarp();
            if (act) ent[at.tx] = key;
            // [q / 128][row / 4][q % 128][row % 4], x relative to x0 (cells
            // outside the window at the dummy row W), as in ligand_prep_kernel
            if (act && ent_t) {
                const size_t row = (size_t)(at.bin + __ldg(tpad + (key >> 24)));
                uint32_t xr = min(((key >> 16) - (uint32_t)x0) & 255u, (uint32_t)W);
                if (decltype(pairs)::value) xr = 2 * xr + (xr < (uint32_t)W ? (key >> 8) & 1u : 0u);
                ent_t[(((size_t)(q >> 7) * (n_pad >> 2) + (row >> 2)) * 128 + (q & 127)) * 4 + (row & 3)] =
                    (xr << 24) | (((key >> 8) & 255u) << 16) | (key & 255u);
            }
            if (act && ent4) {
                // ljComp: entry i < n_ent / 2 weighs atom i into term 0, entry
                // i + n_ent / 2 the same atom into term 1
                const int half = n_ent >> 1;
                if (i < half)
                    ent4[(size_t)q * half + at.bin] =
                        make_uint4(key, __float_as_uint(w_in[i]), __float_as_uint(w_in[i + half]), 0u);
                idx_out[(size_t)q * n_ent + at.bin] = i;
            }
            if (act && tid == leader) cnt[bin] += __popc(at.peers);
            __syncwarp();
        }
    };
    if (tid < 32) {
        if (ka) scatter(std::true_type{});
        else scatter(std::false_type{});
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

cudaError_t box_prep(const BatchArgs& a, cudaStream_t s) {
    const int nb = a.n_rot;
    if (nb <= 0) return cudaSuccess;
    const size_t sm = prep_smem_bytes(a.box.n[0], a.K, a.n_ent, a.classes());
    cudaError_t e = allow_smem((const void*)box_prep_kernel, sm);
    if (e != cudaSuccess) return e;
    box_prep_kernel<<<nb, 256, sm, s>>>(a.rot, a.lig_xyz, a.lig_term, a.n_ent, a.K, a.box, a.ent, a.offs, a.status,
                                        a.lig_w32, a.lig_w32 ? a.ent4 : nullptr, a.ent_idx,
                                        a.use_tc ? a.ent_t : nullptr, a.tpad, a.n_pad, a.x0, a.W, a.classes(), a.tinfo,
                                        a.mask_terms());
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
        if (a.tc_pair) {
            if ((e = launch_pencil_tcp<0>(a, nx, ny, nz, nullptr, bx, s)) != cudaSuccess) return e;
        } else if (tc_tiles(nx) == 1) {
            if ((e = allow_smem((const void*)pencil_tc_kernel<0, 1>, smt)) != cudaSuccess) return e;
            pencil_tc_kernel<0, 1><<<gridt, TC_THREADS, smt, s>>>(a.circ, a.cscale, a.ent_t, a.tinfo, a.n_tc_terms,
                                                                 nullptr, a.g2t, a.n_pad, nb, a.x0, a.W, tg,
                                                                 a.tc_slots, a.tc_n_slots, bx, a.err);
        } else {
            if ((e = allow_smem((const void*)pencil_tc_kernel<0, 2>, smt)) != cudaSuccess) return e;
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

bool box_size(int n) {
    for (int p : {2, 3, 5, 7, 11, 13})
        while (n % p == 0 && n > 1) n /= p;
    return n == 1;
}

size_t box_pencil_smem(int nx, int ny, int nz, int K, int n_ent, bool weighted) {
    return std::max(pencil_limit_bytes(nx, ny, nz, K, n_ent, weighted),
                    std::max(plane_limit_bytes(ny, nz), prep_smem_bytes(nx, K, n_ent, 1)));
}

size_t box_tc_smem(const int dims[3], int n_chunks, int n_terms) {
    return tc_smem_bytes_box(dims[0], dims[1], dims[2], n_chunks, n_terms);
}

size_t cubic_tc_smem(int n, int n_chunks, int n_terms) { return tc_smem_bytes(n, n_chunks, n_terms); }

// Pencil pairs measured faster than one pencil at a time at every cubic edge from
// 24 to 128 (figures in pencil_tcp.cuh), so wherever they fit
bool tc_pairs_fit(const int dims[3], bool box, int K, int n_ent, int n_chunks, int n_terms) {
    if (dims[0] > TC_ROT || dims[1] % 2 != 0 || n_chunks > TP_MAX_CHUNKS) return false;
    if (prep_smem_bytes(dims[0], K, n_ent, 2) > kTpMaxSmem) return false;
    return (box ? tp_smem_box(dims[0], dims[1], dims[2], n_chunks, n_terms, 8)
                : tp_smem_cubic(dims[0], n_chunks, n_terms)) <= kTpMaxSmem;
}

const SizeOps* box_ops() {
    static const SizeOps o{0, false, &box_scan_batch, &box_pencil_smem_unknown, &box_prep,
                           &box_middle, &box_finish, &box_load_kernels};
    return &o;
}

}  // namespace fftdock
