// Pencil stage for term sets of few terms (shape, ljAvg, ljComp; every set on
// box grids): forward transform of the ligand, spectrum product summed over
// the terms, inverse transform along x.
//
// CTA = one rotation x 32 base pencils (ky0, kz), lane = base pencil, for the
// Q pencils ky0 + j Ny / Q (j < Q) of each (Q = 2, or 1 for odd Ny).  The y and z stages of the forward
// transform are direct sums over the ligand's entries (the ligand grid is 99 %
// empty).  The phase of an entry at ky0 + j Ny / Q is its phase at ky0 times
// e^{-2 pi i j y / Q}, which depends on y mod Q only, so the entries of an x
// bin are summed once per class y mod Q (ligand prep sorts them by (term, x,
// class)) and a Q-point DFT over the class sums gives all Q pencils: 1 / Q of
// the lookups and additions.  PAIRED (ljComp: both terms weigh the same
// atoms): one walk feeds both terms' sums.  Entries are the same for all lanes
// of a warp (uniform loads), so no lane diverges; the only shared-memory
// traffic per entry is the phase lookup.
//
// The transforms along x run in place in shared memory ([line][x][32 lanes]),
// as in plane_lines.cuh: the first forward pass takes its inputs straight from
// the walk's registers, the last forward pass, the product with conj(R^_t) and
// the first inverse pass work on the same block of positions without leaving
// registers, and the last inverse pass writes global memory.
//
// Bound: latency of the phase lookups and transforms with 16 warps per SM.  At
// 128^3 ljComp they issue in 53 % of the slots (38 K warp instructions per 64 pencils,
// about half of them the walk), the L1 data path is 59 % busy, the FMA pipe 31 %.
// Against one pencil per lane with register-resident x
// transforms (cubic: pencil_kernel) and one warp per pencil with segmented
// scans (box grids), pencil stage: ljComp 128^3, 1500 atoms 26.9 -> 16.0 ms per
// 2000 rotations; ljComp 90 x 96 x 100, 800 atoms 47.6 -> 5.4 ms per 1000; shape
// 64^3, 450 atoms 1.60 -> 1.22 ms per 2000.
//
// Layouts: spec [K][Nx][PP], g2 [B][Nx][PP] (pencil p = ky Hz + kz), offs
// [B][K Nx Q + 1] bin starts, ent [B][n_ent] = t << 24 | x << 16 | y << 8 | z,
// ent4 [B][n_ent / 2] = (entry, weight in term 0, weight in term 1, -).
#pragma once

#include <algorithm>

#include "plane_lines.cuh"

namespace fftdock {

// Threads per CTA: 256; the paired form takes 512 where its line buffers (two
// terms, Q pencils) leave room for one CTA per SM.  ljComp, ms per 1000
// rotations, 512 | 2 x 256 threads: 64^3 1.16 | 0.80, 80^3 2.02 | 1.90 (Q = 2 both);
// above, two CTAs need Q = 1: 96^3 3.44 | 3.79, 128^3 8.30 | 9.87.
constexpr int kPencilThreads = 256, kPencilWideThreads = 512;

// x plan: the first radix holds Q T lines per thread, so it stays at 10 or
// less where two passes allow it
constexpr bool pencil_radices(int nx, LineRadices& r) {
    int best = 1 << 30;
    for (int a = 2; a <= 10; ++a) {
        if (nx % a != 0 || nx / a > 16) continue;
        // the first pass deals nx / a butterflies to 16 warps
        const int b = nx / a, cost = 13 * a + 10 * b + 60 * (16 - b) / 16;
        if (cost < best) {
            best = cost;
            r.n = nx;
            r.np = 2;
            r.r[0] = a;
            r.r[1] = b;
        }
    }
    return best < (1 << 30) || line_radices(nx, 2, 13, r);
}
template <int N> constexpr LineRadices fixed_pencil_radices() {
    LineRadices r{};
    // 8-point first passes where they divide the edge
    r.n = N;
    r.np = 2;
    r.r[0] = N % 8 == 0 && N / 8 <= 16 ? 8 : N <= 16 ? 4 : N == 144 ? 9 : 6;
    r.r[1] = N / r.r[0];
    return r;
}

// One unweighted term on a cubic edge: from 24 on.  16^3 has three tiles of 32 pencils,
// which leave most of the warps idle: pencil stage of 4000 rotations 0.51 ms, with
// pencil_kernel 0.45; 24^3 0.58 and 0.63.
constexpr bool pencil_lines_one_term(int n) { return n > 16; }

// cubic edges: classes y mod Q (four classes leave too few CTAs per SM: shape
// at 64^3 0.62 against 0.52 ms per 1000 rotations) and resident CTAs
constexpr int kPencilQ = 2;
constexpr int pencil_ctas(int n, bool paired) { return paired ? (n <= 80 ? 2 : 1) : n <= 64 ? 4 : n <= 96 ? 3 : 2; }
constexpr int pencil_threads(int n, bool paired) { return paired && n > 80 ? kPencilWideThreads : kPencilThreads; }

// shared memory: line buffers, x twiddles, phase tables ([N][16] on a cubic
// grid; [nz][32] of the lanes' z phases and [ny][ky0s of the tile] on a box)
constexpr int pencil_tile_kys(int hz) { return 31 / hz + 2; }
constexpr size_t pencil_lines_smem_cubic(int n, int q, bool paired) {
    return ((size_t)(paired ? 2 : 1) * q * n * 32 + n + (size_t)n * 16) * sizeof(float2);
}
constexpr size_t pencil_lines_smem_box(int nx, int ny, int nz, int k, int q, bool paired) {
    return ((size_t)(paired || k > 1 ? 2 : 1) * q * nx * 32 + nx + (size_t)nz * 32 +
            (size_t)ny * pencil_tile_kys(nz / 2 + 1)) * sizeof(float2);
}

// The rotation's entries and bin starts are staged in shared memory when they
// fit there (`staged`; every entry is read by one warp only, but from global
// memory each pair of entries would cost an L2 round trip in the walk's
// serial chain: ljComp at 128^3 31.0 against 19.0 ms per 2000 rotations).
constexpr size_t pencil_stage_bytes(int nx, int k, int q, int n_ent, bool paired) {
    return 16 + (paired ? (size_t)(n_ent / 2) * sizeof(uint4) : (size_t)n_ent * sizeof(uint32_t)) +
           ((size_t)(paired ? 1 : k) * nx * q + 1) * sizeof(int32_t);
}

// tiles of one rotation are dealt to gridDim.y CTAs: several per CTA (the
// set-up is then shared) while at least about eight CTAs per SM remain
inline int pencil_grid_y(int n_rot, int n_tiles) {
    const int want = (1216 + n_rot - 1) / n_rot;
    const int per = std::max(1, std::min(8, n_tiles / std::max(1, want)));
    return (n_tiles + per - 1) / per;
}

// N > 0: cubic edge (K = 1, or PAIRED); N = 0: a box grid of any K.
template <int N, typename SpecT, bool PAIRED, int Q, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) pencil_lines_kernel(
    const SpecT* __restrict__ spec, const uint32_t* __restrict__ ent, const uint4* __restrict__ ent4,
    const int32_t* __restrict__ offs, const float2* __restrict__ twx_g, const float2* __restrict__ twy_g,
    const float2* __restrict__ twz_g, const __grid_constant__ LineRadices rx, int nx_rt, int ny_rt, int nz_rt, int pp,
    int K, int n_ent, int staged, float2* __restrict__ g2) {
    constexpr bool BOX = N == 0;
    constexpr LineRadices FR = fixed_pencil_radices<(N > 0 ? N : 16)>();
    constexpr int RA = BOX ? 0 : FR.r[0], RB = BOX ? 0 : FR.r[1];
    static_assert(BOX || (RA * RB == N && RA <= 13 && RB <= 16 && N % Q == 0), "no two-pass x plan for this edge");
    constexpr int T = PAIRED ? 2 : 1;
    constexpr int NW = NT / 32;
    const int nx = BOX ? nx_rt : N, ny = BOX ? ny_rt : N, nz = BOX ? nz_rt : N;
    const int hz = nz / 2 + 1;
    const int lines = Q * nx * 32;  // complex values of one buffer
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    float2* buf = reinterpret_cast<float2*>(smem_raw);        // [T][Q][nx][32]; K > 1 unpaired: the second holds the sum
    const bool two_bufs = PAIRED || (BOX && K > 1);
    float2* acc_buf = buf + (BOX && !PAIRED && K > 1 ? lines : 0);
    float2* twx = buf + (two_bufs ? 2 : 1) * lines;           // [nx]
    float2* btab = twx + nx;                                  // cubic: [N][16]; box: [nz][32]
    float2* atab = btab + (BOX ? nz * 32 : 0);                // box: [ny][kys]

    const int q = blockIdx.x;
    const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
    const int nb = (ny / Q) * hz;                             // base pencils
    const int n_walk = PAIRED ? n_ent >> 1 : n_ent;
    const int n_offs = (PAIRED ? 1 : K) * nx * Q + 1;         // (PAIRED: the second term's bins repeat the first's)
    const uint32_t* eq = ent + (PAIRED ? 0 : (size_t)q * n_walk);
    const uint4* eq4 = PAIRED ? ent4 + (size_t)q * n_walk : nullptr;
    const int32_t* oq = offs + (size_t)q * ((size_t)K * nx * Q + 1);
    uint4* es4 = reinterpret_cast<uint4*>(
        smem_raw + (((char*)(btab + (BOX ? nz * 32 + ny * pencil_tile_kys(hz) : N * 16)) - (char*)smem_raw + 15) & ~(ptrdiff_t)15));
    uint32_t* es = reinterpret_cast<uint32_t*>(es4);
    int32_t* os = reinterpret_cast<int32_t*>(es4) + (PAIRED ? 4 : 1) * n_walk;
    if (staged) {
        if constexpr (PAIRED) {
            for (int i = tid; i < n_walk; i += NT) es4[i] = eq4[i];
        } else {
            for (int i = tid; i < n_walk; i += NT) es[i] = eq[i];
        }
        for (int i = tid; i < n_offs; i += NT) os[i] = oq[i];
    }
    for (int i = tid; i < nx; i += NT) twx[i] = twx_g[i];
    if constexpr (!BOX)
        for (int i = tid; i < N * 16; i += NT) btab[i] = twx_g[i >> 4];
    const int kys = pencil_tile_kys(hz);
    const int ra = BOX ? rx.r[0] : RA, rb = BOX ? rx.r[rx.np - 1] : RB;
    const int n_tiles = (nb + 31) / 32;

    // the CTA's tiles: entries, bin starts and tables are set up once
    for (int tile = blockIdx.y; tile < n_tiles; tile += gridDim.y) {
    __syncthreads();
    const int b0 = tile * 32;
    const bool valid = b0 + l < nb;
    const int bp = valid ? b0 + l : nb - 1;
    const int ky0 = bp / hz, kz = bp - ky0 * hz;
    const int kyf = b0 / hz;                                  // the tile's first ky0
    if constexpr (BOX) {
        for (int z = w; z < nz; z += NW) btab[z * 32 + l] = twz_g[(int)((unsigned)(kz * z) % (unsigned)nz)];
        for (int i = tid; i < ny * kys; i += NT) {
            const int y = i / kys, ky = kyf + (i - y * kys);
            atab[i] = twy_g[(int)((unsigned)(ky * y) % (unsigned)ny)];
        }
        __syncthreads();
    }

    // this lane's phase of entry u
    const float2* bl = btab + (BOX ? l : (l & 15));
    const float2* al = atab + (ky0 - kyf);
    // cubic: table row of ky y + kz z (bytes 1 and 0 of the entry) as one
    // two-way dot product: power-of-two edges scale it by the 128-byte row
    constexpr bool POW2 = !BOX && (N & (N - 1)) == 0;
    constexpr unsigned ROW = POW2 ? 128u : 1u;
    const unsigned kk = (unsigned)kz * ROW | ((unsigned)ky0 * ROW) << 16;
    const uint32_t bl_s = static_cast<uint32_t>(__cvta_generic_to_shared(bl));
    auto phase = [&](uint32_t u) -> float2 {
        if constexpr (BOX) {
            return cmul(al[((u >> 8) & 255u) * kys], bl[(u & 255u) * 32]);
        } else {
            const unsigned s = __dp2a_lo(kk, u, 0u);
            const uint32_t at = bl_s + (POW2 ? s & ((unsigned)(N - 1) * 128u) : s % (unsigned)N * 128u);
            float2 z;
            asm("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(z.x), "=f"(z.y) : "r"(at));
            return z;
        }
    };

    // in-place pass over every line of n_bufs buffers from `b`: forward =
    // DFT then twiddle, inverse = twiddle then DFT (mirrored)
    auto mid_pass = [&](float2* b, int n_bufs, int R_, int len, bool inverse) {
        with_radix<0, 13>(R_, [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            const int m = len / R, per = nx / R, tstep = nx / len;
            for (int it = w; it < n_bufs * Q * per; it += NW) {
                const int ln = it / per, qb = it - ln * per;
                const int blk = qb / m, j = qb - blk * m;
                float2* p = b + ((size_t)ln * nx + blk * len + j) * 32 + l;
                float2 v[R];
#pragma unroll
                for (int r = 0; r < R; ++r) v[r] = p[r * m * 32];
                if (inverse) {
#pragma unroll
                    for (int r = 1; r < R; ++r) v[r] = ctwiddle<+1>(v[r], twx[tstep * j * r]);
                    dft<R, +1>(v);
                } else {
                    dft<R, -1>(v);
#pragma unroll
                    for (int r = 1; r < R; ++r) v[r] = ctwiddle<-1>(v[r], twx[tstep * j * r]);
                }
#pragma unroll
                for (int r = 0; r < R; ++r) p[r * m * 32] = v[r];
            }
        });
        __syncthreads();
    };

    const int n_loop = PAIRED || !BOX ? 1 : K;
    for (int t = 0; t < n_loop; ++t) {
        // ---- the walk and the first forward pass: butterfly j's bins x = j + m r ----
        auto walk = [&](const uint32_t* en, const uint4* en4, const int32_t* of, auto unroll) {
        constexpr int U = decltype(unroll)::value;
        with_radix<RA, 13>(ra, [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            const int m = nx / R;
#pragma unroll 1
            for (int j = w; j < m; j += NW) {
                float2 v[T * Q][R];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int32_t* o = of + (t * nx + j + m * r) * Q;
                    int e0 = o[0];
                    float2 s0[Q], s1[Q];
#pragma unroll
                    for (int c = 0; c < Q; ++c) {
                        const int e1 = o[c + 1];
                        float2 a0 = make_float2(0.f, 0.f), a1 = make_float2(0.f, 0.f);
#pragma unroll U
                        for (int i = e0; i < e1; ++i) {
                            if constexpr (PAIRED) {
                                const uint4 e = en4[i];
                                const float2 z = phase(e.x);
                                const float w0 = __uint_as_float(e.y), w1 = __uint_as_float(e.z);
                                a0.x = fmaf(w0, z.x, a0.x);
                                a0.y = fmaf(w0, z.y, a0.y);
                                a1.x = fmaf(w1, z.x, a1.x);
                                a1.y = fmaf(w1, z.y, a1.y);
                            } else {
                                a0 = a0 + phase(en[i]);
                            }
                        }
                        s0[c] = a0;
                        s1[c] = a1;
                        e0 = e1;
                    }
                    dft<Q, -1>(s0);
                    if constexpr (PAIRED) dft<Q, -1>(s1);
#pragma unroll
                    for (int c = 0; c < Q; ++c) {
                        v[c][r] = s0[c];
                        if constexpr (PAIRED) v[Q + c][r] = s1[c];
                    }
                }
                float2 tw[R];
#pragma unroll
                for (int r = 1; r < R; ++r) tw[r] = twx[j * r];
#pragma unroll
                for (int c = 0; c < T * Q; ++c) {
                    dft<R, -1>(v[c]);
                    float2* p = buf + ((size_t)c * nx + j) * 32 + l;
                    p[0] = v[c][0];
#pragma unroll
                    for (int r = 1; r < R; ++r) p[r * m * 32] = ctwiddle<-1>(v[c][r], tw[r]);
                }
            }
        });
        };
        if (staged) walk(es, es4, os, std::integral_constant<int, 4>{});
        else walk(eq, eq4, oq, std::integral_constant<int, 1>{});
        __syncthreads();
        if constexpr (BOX) {
            int len = nx / rx.r[0];
            for (int s = 1; s + 1 < rx.np; ++s) {
                mid_pass(buf, T, rx.r[s], len, false);
                len /= rx.r[s];
            }
        }
        // ---- last forward pass, spectrum product, (last term) first inverse pass ----
        with_radix<RB, 16>(rb, [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            const int nblk = nx / R;
#pragma unroll 1
            for (int it = w; it < Q * nblk; it += NW) {
                const int c = it / nblk, b = it - c * nblk;
                // the lane's pencil is bp + c nb; frequency of output r: kx = digits(b) + r nblk
                const int kx0 = BOX ? line_digits(rx, b) : b;
                float2 s[R];
#pragma unroll
                for (int u = 0; u < T; ++u) {
                    const SpecT* sp = spec + ((size_t)(t + u) * nx + kx0) * pp + bp + c * nb;
                    const float2* p = buf + (((size_t)u * Q + c) * nx + b * R) * 32 + l;
                    // the spectrum's loads are in flight during the transform
                    float2 f[R], g[R];
#pragma unroll
                    for (int r = 0; r < R; ++r) g[r] = spec_load(sp + (size_t)(r * nblk) * pp);
#pragma unroll
                    for (int r = 0; r < R; ++r) f[r] = p[r * 32];
                    dft<R, -1>(f);
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float2 pr = cmul_conj(f[r], g[r]);
                        s[r] = u == 0 ? pr : s[r] + pr;
                    }
                }
                float2* d = acc_buf + ((size_t)c * nx + b * R) * 32 + l;
                if (BOX && t > 0) {
#pragma unroll
                    for (int r = 0; r < R; ++r) s[r] = s[r] + d[r * 32];
                }
                if (t + 1 == n_loop) dft<R, +1>(s);
#pragma unroll
                for (int r = 0; r < R; ++r) d[r * 32] = s[r];
            }
        });
        __syncthreads();
    }
    if constexpr (BOX) {
        // mirrored middle passes
        int len = rx.r[rx.np - 1];
        for (int s = rx.np - 2; s >= 1; --s) {
            len *= rx.r[s];
            mid_pass(acc_buf, 1, rx.r[s], len, true);
        }
    }
    // ---- last inverse pass: x = j + m r ----
    with_radix<RA, 13>(ra, [&](auto radix) {
        constexpr int R = decltype(radix)::value;
        const int m = nx / R;
#pragma unroll 1
        for (int it = w; it < Q * m; it += NW) {
            const int c = it / m, j = it - c * m;
            const float2* p = acc_buf + ((size_t)c * nx + j) * 32 + l;
            float2 v[R];
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = p[r * m * 32];
#pragma unroll
            for (int r = 1; r < R; ++r) v[r] = ctwiddle<+1>(v[r], twx[j * r]);
            dft<R, +1>(v);
            if (valid) {
                float2* dst = g2 + ((size_t)q * nx + j) * pp + bp + c * nb;
#pragma unroll
                for (int r = 0; r < R; ++r) dst[(size_t)(r * m) * pp] = v[r];
            }
        }
    });
    }
}

// FFT-form launches on box grids, one translation unit each
cudaError_t box_pencil_plain(const BatchArgs& a, const float2* twx, const float2* twy, const float2* twz, cudaStream_t s);
cudaError_t box_pencil_paired(const BatchArgs& a, const float2* twx, const float2* twy, const float2* twz, cudaStream_t s);
cudaError_t box_pencil_paired_wide(const BatchArgs& a, const float2* twx, const float2* twy, const float2* twz,
                                   cudaStream_t s);
constexpr size_t kPencilMaxSmem = 227 * 1024;

template <bool PAIRED, int Q, int NT>
cudaError_t launch_box_pencil(const BatchArgs& a, const float2* twx, const float2* twy, const float2* twz,
                              cudaStream_t s) {
    const auto fn = &pencil_lines_kernel<0, float2, PAIRED, Q, NT, 512 / NT>;
    const int nx = a.box.n[0], ny = a.box.n[1], nz = a.box.n[2];
    LineRadices rx{};
    if (!pencil_radices(nx, rx)) return cudaErrorInvalidValue;
    size_t sm = pencil_lines_smem_box(nx, ny, nz, a.K, Q, PAIRED);
    const size_t st = pencil_stage_bytes(nx, a.K, Q, a.n_ent, PAIRED);
    const int staged = sm + st <= kPencilMaxSmem ? 1 : 0;
    if (staged) sm += st;
    const cudaError_t e = allow_smem((const void*)fn, sm);
    if (e != cudaSuccess) return e;
    const dim3 grid(a.n_rot, pencil_grid_y(a.n_rot, ((ny / Q) * (nz / 2 + 1) + 31) / 32));
    fn<<<grid, NT, sm, s>>>(static_cast<const float2*>(a.spec), a.ent, a.ent4, a.offs, twx, twy, twz, rx, nx, ny, nz,
                            a.PP, a.K, a.n_ent, staged, a.g2);
    return cudaGetLastError();
}

}  // namespace fftdock
