// Tensor-core pencil stage over pencil pairs (tcgen05, sm_103a): the stage of
// pencil_tc.cuh -- a circular correlation along x as split-FP16 GEMMs -- for
// the pencils A = (ky, kz) and B = (ky + Ny/2, kz) of 128 rotations in one CTA.
//
// * One walk for two pencils.  An entry's phases in A and B differ by (-1)^y,
//   so the ligand sums are taken once per y parity: staging rows 2 x' + (y mod
//   2) hold E and O, and F_A = E + O, F_B = E - O (ligand prep sorts by (term, x,
//   y parity) and writes the row into the entry's top byte).  Half the entry
//   loads, phase lookups and staging stores per pencil.
// * Operands swapped: the ligand tile is the M = 128 operand, the circulant the
//   N operand with the real and imaginary output rows of an x interleaved, so
//   one MMA of N = 2 Nx gives both: D[rotation][2 x + {re, im}].  Against M = x,
//   N = rotation with separate real and imaginary MMAs: a quarter fewer operand
//   bytes per flop, no MMA work for x >= Nx, and a thread of the epilogue holds
//   whole x-quads of its rotation (one 32-byte store each).
// * One CTA per SM (all 512 tensor-memory columns) and staging apart from the
//   operand tiles, so that production and MMAs overlap inside the CTA.  Warps
//   0-7 walk the next term's entries while the tensor core works; warp 8 issues
//   the MMAs; warps 9-15 build the circulant tiles of the pencil whose MMAs are
//   done; warps 8-15 drain the accumulators between term groups; all but warp 8
//   convert the staging rows to hi/lo tiles (rows without an entry, known from
//   ligand prep's bit masks, count as zero and are never cleared).  Per term:
//     walk k | E_A(k) after MMA A(k-1)        -> barrier
//     convert: A tiles stored, B tiles held in registers
//                                             -> barrier, MMA A(k) issued
//     after MMA B(k-1): B tiles stored, E_B(k) -> MMA B(k) issued; walk k+1 ...
//   so pencil A's MMAs run while B's tiles are stored and B's while the next
//   term is walked.
// Accumulator groups, scales, splits and the order of the products are those of
// pencil_tc.cuh; the running sums use the SM's two slots as [x][rotation].
//
// Shared memory bounds the window (40 cells at Nx = 128); larger ligands, odd Ny
// and Nx > 128 run pencil_tc_kernel.  All waits are bounded.
//
// Measured (GB300, 18 terms, ms per 1000 rotations, one pencil at a time -> pairs,
// with the ligand's atoms and window): 32^3 0.88 -> 0.59 (60, 16), 48^3 2.19 -> 1.59
// (150, 24), 64^3 3.79 -> 2.73 (300, 24), 80^3 6.59 -> 5.51 (400, 24), 96^3 11.6 -> 9.5
// (700, 32), 112^3 16.9 -> 14.0 (1000, 32), 128^3 24.9 -> 20.6 (1500, 40), box 112 x
// 120 x 126 25.9 -> 20.8 (1500, 40).  Bound at 128^3 by shared-memory bandwidth: per term
// the MMAs read 2,880 wavefronts of operands, walk, conversion and circulant tiles
// take about 3,900 and global accesses (entries, slots, output) share the same
// path: 92 % of its cycles busy, tensor pipe 37 %.
#pragma once

#include <type_traits>

#include "pencil_tc.cuh"

namespace fftdock {

constexpr int TP_THREADS = 512, TP_CONV = 480;
constexpr int TP_MAX_CHUNKS = 5;  // a converting thread holds at most three of the 256 n_chunks tasks
static_assert(256 * TP_MAX_CHUNKS <= 3 * TP_CONV && 4 * ((128 + 8 * TP_MAX_CHUNKS - 8) / 4) <= TP_CONV - 256,
              "conversion tasks and circulant rows per thread");

__host__ __device__ constexpr int tp_groups(int nx8, int n_chunks) { return (nx8 + 8 * n_chunks - 8) / 4; }
constexpr size_t tp_smem_core(int nx, int n_chunks, int n_terms) {
    const int nx8 = (nx + 7) / 8 * 8;
    return (size_t)2 * n_chunks * TC_FCHUNK + (size_t)(16 * n_chunks + 1) * 1024 +
           (size_t)4 * tp_groups(nx8, n_chunks) * 256 + (size_t)2 * nx * sizeof(TcPair) + (size_t)TC_ROT * 8 +
           (size_t)((2 * n_terms + 1) * 4 + 15) / 16 * 16;
}
constexpr size_t tp_smem_cubic(int n, int n_chunks, int n_terms) { return tp_smem_core(n, n_chunks, n_terms) + (size_t)n * 128; }
// z_copies: copies of the z phase table (lanes of a half-warp; 16: no bank is
// shared, 8: two lanes share one)
constexpr size_t tp_smem_box(int nx, int ny, int nz, int n_chunks, int n_terms, int z_copies) {
    return tp_smem_core(nx, n_chunks, n_terms) + (size_t)ny * 128 + (size_t)nz * 8 * z_copies;
}
constexpr size_t kTpMaxSmem = 226 * 1024;  // + the static barriers and flags

__device__ __forceinline__ void st_global_v8(float2* p, const float2 (&v)[4]) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0].x), "f"(v[0].y),
                 "f"(v[1].x), "f"(v[1].y), "f"(v[2].x), "f"(v[2].y), "f"(v[3].x), "f"(v[3].y)
                 : "memory");
}

// zero unless on
__device__ __forceinline__ float2 ld_shared_f2_if(uint32_t addr, uint32_t on) {
    float2 v;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\tmov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\t"
        "@p ld.shared.v2.f32 {%0, %1}, [%2];\n\t}"
        : "=&f"(v.x), "=&f"(v.y)
        : "r"(addr), "r"(on));
    return v;
}

// tc_entries8 with rows in the entries' top bytes and 128-byte table rows
template <bool SIDE, int N>
__device__ __forceinline__ void tp_entries8(const uint32_t (&e)[8], uint32_t kyz, uint32_t twl, uint32_t tzl,
                                            uint32_t zrow, uint32_t stg, uint32_t sd, unsigned first, unsigned& cur,
                                            float2& acc) {
    float2 z[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        if constexpr (N == 0) {
            const float2 a = ld_shared_f2_const(twl + ((e[q] >> 16) & 255u) * 128u);
            const float2 b = ld_shared_f2_const(tzl + (e[q] & 255u) * zrow);
            z[q] = make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
        } else if constexpr ((N & (N - 1)) == 0) {
            z[q] = ld_shared_f2_const(twl + (((e[q] * kyz) >> 9) & ((unsigned)(N - 1) << 7)));
        } else {
            z[q] = ld_shared_f2_const(twl + tc_phase<N>(e[q], kyz) * 128u);
        }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const unsigned xr = e[q] >> 24;
        const float keep = xr != cur ? 0.f : 1.f;
        acc.x = fmaf(acc.x, keep, z[q].x);
        acc.y = fmaf(acc.y, keep, z[q].y);
        cur = xr;
        uint32_t dst = stg + xr * 1024u;
        if (SIDE) dst = xr == first ? sd : dst;
        st_shared_f2(dst, acc.x, acc.y);
    }
}

// tinfo, ent_t: as pencil_tc_kernel, entries padded with row 2 W.  nb = (Ny / 2)
// Hz base pencils (grid x); N = 0: a box grid.
template <int N>
__global__ void __launch_bounds__(TP_THREADS, 1) pencil_tcp_kernel(
    const float2* __restrict__ circ, const int8_t* __restrict__ cscale, const uint32_t* __restrict__ ent_t,
    const int32_t* __restrict__ tinfo, int Ka, const float2* __restrict__ tw, float2* __restrict__ g2t, int n_pad,
    int n_rot, int x0, int W, int tg, float2* __restrict__ slots, int n_slots, TcBox bx, int z_copies,
    int* __restrict__ err) {
    constexpr bool BOX = N == 0;
    const int nx = BOX ? bx.nx : N;
    const int H = BOX ? bx.hz : N / 2 + 1;
    const int NH = BOX ? bx.nh : N * (N / 2 + 1);
    const int NXP = BOX ? bx.nxp : N;
    const int nx8 = (nx + 7) / 8 * 8;
    const int NC = W >> 3;
    const int RG = tp_groups(nx8, NC);  // 8-row groups of a circulant tile part
    const int nb = NH >> 1;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* fbuf = smem_raw;                                         // [2][NC][hi | lo]
    unsigned char* sbuf = fbuf + 2 * NC * TC_FCHUNK;                        // [2 W + 1][128] float2
    unsigned char* abuf = sbuf + (2 * W + 1) * 1024;                        // [2][hi | lo][RG][256]
    float2* twr = reinterpret_cast<float2*>(abuf + 4 * RG * 256);           // [N][16]; box: [ny][16], [nz][z_copies]
    const int tw_len = BOX ? bx.ny * 16 + bx.nz * z_copies : N * 16;
    TcPair* pr = reinterpret_cast<TcPair*>(twr + tw_len);                   // [2][nx]
    float2* side = reinterpret_cast<float2*>(pr + 2 * nx);                  // [128]
    int32_t* tinf = reinterpret_cast<int32_t*>(side + TC_ROT);              // [2 Ka + 1]
    __shared__ __align__(8) uint64_t bar[2];                                // MMAs of pencil A, B of a term
    __shared__ __align__(8) uint64_t done_bar;                              // every MMA issued
    __shared__ uint32_t tmem_base;
    __shared__ int abort_flag;

    const int pA = blockIdx.x;
    const int g = blockIdx.y;
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const unsigned ky = (unsigned)(pA / H), kz = (unsigned)(pA - (pA / H) * H);
    const uint32_t kyz = (kz << 16) | ky;

    if (tid == 0) abort_flag = *(volatile int*)err;
    __syncthreads();
    // a timeout elsewhere in this launch already failed the scan: do nothing
    if (abort_flag) return;

    if constexpr (BOX) {
        for (int i = tid; i < bx.ny * 16; i += TP_THREADS) {
            const float2 v = bx.twy[(int)(((unsigned)(i >> 4) * ky) % (unsigned)bx.ny)];
            twr[i] = make_float2(v.x * TC_F_SCALE, v.y * TC_F_SCALE);
        }
        for (int i = tid; i < bx.nz * z_copies; i += TP_THREADS)
            twr[bx.ny * 16 + i] = bx.twz[(int)(((unsigned)(i / z_copies) * kz) % (unsigned)bx.nz)];
    } else {
        for (int i = tid; i < N * 16; i += TP_THREADS) {
            const float2 v = tw[i >> 4];
            twr[i] = make_float2(v.x * TC_F_SCALE, v.y * TC_F_SCALE);
        }
    }
    for (int i = tid; i <= 2 * Ka; i += TP_THREADS) tinf[i] = tinfo[i];
    const uint32_t fb = tc::smem_u32(fbuf), sb = tc::smem_u32(sbuf), ab = tc::smem_u32(abuf), prb = tc::smem_u32(pr);
    if (warp == 0) {
        tc::tmem_alloc(&tmem_base, 512);
        tc::tmem_relinquish();
    }
    if (tid == 0) {
        tc::mbar_init(&bar[0], 1);
        tc::mbar_init(&bar[1], 1);
        tc::mbar_init(&done_bar, 1);
        tc::fence_barrier_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_base;
    const int ng = (Ka + tg - 1) / tg;
    auto group_of = [&](int k) { return (k * ng) / Ka; };
    auto starts_group = [&](int k) { return k == 0 || group_of(k) != group_of(k - 1); };

    // this thread observes the completion of pencil u's MMAs of term k
    auto wait_mma = [&](int u, int k) {
        if (!*(volatile int*)&abort_flag && !tc::mbar_wait(&bar[u], (uint32_t)(k & 1), TC_WAIT_NS)) {
            atomicOr(err, 2 << u);
            abort_flag = 1;
        }
    };
    // the same for a warp that only writes shared memory: one lane polls
    auto wait_mma_warp = [&](int u, int k) {
        if (lane == 0) wait_mma(u, k);
        __syncwarp();
    };

    // running sums of the completed groups: the SM's two slots, [x][rotation]
    uint32_t smid;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
    const int slot = (int)smid * 2;
    const bool slot_ok = slot + 1 < n_slots;
    if (ng > 1 && !slot_ok && tid == 0) {
        atomicOr(err, 32);
        abort_flag = 1;
    }
    const bool with_sum = ng > 1 && slot_ok;
    float2* const sums = slots + (size_t)(slot_ok ? slot : 0) * (TC_ROT * 128) + 32 * (warp & 3) + lane;
    const uint32_t trow = (uint32_t)(32 * (warp & 3)) << 16;  // this warp's tensor-memory lanes
    // four warps, one per lane quarter: pencil u's group sum into its slot
    // (stored first, then added with FP32 atomics: one thread per element, in
    // program order; read after a CTA barrier)
    auto drain = [&](int u, bool first) {
        if (!slot_ok) return;
        float2* const st = sums + (size_t)u * (TC_ROT * 128);
#pragma unroll 1
        for (int c0 = 0; c0 < 2 * nx; c0 += 16) {
            uint32_t d[16];
            tc::tmem_ld_32x32b_x16(tmem + 256u * u + trow + c0, d);
            tc::tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float2 v = make_float2(__uint_as_float(d[2 * j]), __uint_as_float(d[2 * j + 1]));
                float2* p = st + (size_t)(c0 / 2 + j) * TC_ROT;
                if (first) st_relaxed_f2(p, v);
                else atomicAdd(p, v);
            }
        }
    };

    // before a group of terms restarts the accumulator: its sum goes to the slot
    // (every thread orders its tensor-memory loads after its own wait)
    auto drain_before = [&](int u, int k) {
        if (k >= 1 && starts_group(k) && __all_sync(0xffffffffu, !*(volatile int*)&abort_flag)) {
            wait_mma(u, k - 1);
            __syncwarp();
            tc::fence_after_sync();
            drain(u, group_of(k - 1) == 0);
            tc::fence_before_sync();
        }
    };

    // converting thread ct: the occupied rows of its tasks ct + 480 i (task t: half
    // chunk t / 128 of rotation t % 128) of term kk
    uint32_t mk[3] = {0u, 0u, 0u};
    auto load_mask = [&](int ct, int kk) {
        const uint32_t* occ = ent_t + ((size_t)g * (n_pad / 4) + (tinf[Ka] >> 2) + kk) * (4 * TC_ROT);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int t = ct + TP_CONV * i;
            if (t < 256 * NC) mk[i] = __ldg(occ + 4 * (t & 127) + (t >> 9));
        }
    };

    if (warp < 8) {
        // ---------------- walkers: thread (r, half) ----------------
        const int r = tid & 127, half = tid >> 7;
        const uint4* ent_g = reinterpret_cast<const uint4*>(ent_t) + (size_t)g * (n_pad / 4) * TC_ROT + r;
        const uint32_t twl = tc::smem_u32(twr) + (uint32_t)(lane & 15) * 8u;
        const uint32_t zrow = BOX ? 8u * z_copies : 0u;
        const uint32_t tzl = BOX ? tc::smem_u32(twr) + (uint32_t)bx.ny * 128u + (uint32_t)(lane & (z_copies - 1)) * 8u : 0u;
        const uint32_t stg = sb + (uint32_t)r * 8u;
        const uint32_t sd = tc::smem_u32(side) + (uint32_t)r * 8u;
        uint4 pa0, pa1, pb0, pb1;
        uint32_t plast = 0;  // the last entry of the first half
        auto preload = [&](int kk) {
            const int jt = tinf[kk], m8 = (tinf[kk + 1] - jt) >> 3;
            const int bb = half ? (m8 + 1) >> 1 : 0;
            const uint4* q = ent_g + (size_t)((jt >> 2) + 2 * bb) * TC_ROT;
            if (half) plast = __ldg(&q[-TC_ROT].w);
            pa0 = __ldg(q);
            pa1 = __ldg(q + TC_ROT);
            pb0 = __ldg(q + 2 * TC_ROT);
            pb1 = __ldg(q + 3 * TC_ROT);
        };
        auto walk = [&](auto side_tag, const uint4* eq, int nblk, unsigned first) {
            constexpr bool SIDE = decltype(side_tag)::value;
            unsigned cur = 0xffffffffu;
            float2 acc = make_float2(0.f, 0.f);
            if (nblk <= 0) return;
            uint4 a0 = pa0, a1 = pa1, b0 = pb0, b1 = pb1, c0, c1;
            auto ld = [&](int blk, uint4& y0, uint4& y1) {
                y0 = __ldg(eq + (size_t)(2 * blk) * TC_ROT);
                y1 = __ldg(eq + (size_t)(2 * blk + 1) * TC_ROT);
            };
            auto sum = [&](const uint4& y0, const uint4& y1) {
                const uint32_t e[8] = {y0.x, y0.y, y0.z, y0.w, y1.x, y1.y, y1.z, y1.w};
                tp_entries8<SIDE, N>(e, kyz, twl, tzl, zrow, stg, sd, first, cur, acc);
            };
            for (int blk = 0; blk < nblk; blk += 3) {
                ld(blk + 2, c0, c1);
                sum(a0, a1);
                if (blk + 1 >= nblk) break;
                ld(blk + 3, a0, a1);
                sum(b0, b1);
                if (blk + 2 >= nblk) break;
                ld(blk + 4, b0, b1);
                sum(c0, c1);
            }
        };
        preload(0);
        for (int k = 0; k < Ka; ++k) {
            const int jt0 = tinf[k], n8 = (tinf[k + 1] - jt0) >> 3, na = (n8 + 1) >> 1;
            const int b0 = half ? na : 0, nb8 = half ? n8 - na : na;
            const uint4* eq = ent_g + (size_t)((jt0 >> 2) + 2 * b0) * TC_ROT;
            // the second half's first row may continue the first half's last
            // one: it goes to the side slot
            const unsigned first = half && nb8 > 0 ? (pa0.x >> 24) : 0xfffffffeu;
            const bool cont = (plast >> 24) == first;
            load_mask(tid, k);
            if (half) walk(std::true_type{}, eq, nb8, first);
            else walk(std::false_type{}, eq, nb8, first);
            asm volatile("bar.sync 2, 256;" ::: "memory");
            if (half && first < (unsigned)(2 * W)) {
                const float2 b = ld_shared_f2(sd);
                float2 a = make_float2(0.f, 0.f);
                if (cont) a = ld_shared_f2(stg + first * 1024u);
                st_shared_f2(stg + first * 1024u, a.x + b.x, a.y + b.y);
            }
            if (k + 1 < Ka) preload(k + 1);
#define TP_CONVERT(ct)                                                                                             \
            asm volatile("bar.sync 1, 512;" ::: "memory");                                                            \
            uint32_t bh[3][4], bl[3][4];                                                                              \
            _Pragma("unroll") for (int i = 0; i < 3; ++i) {                                                           \
                const int t = (ct) + TP_CONV * i;                                                                     \
                if (t < 256 * NC) {                                                                                   \
                    const uint32_t m = mk[i] >> (((t >> 7) & 3) * 8);                                                 \
                    const uint32_t row = sb + (uint32_t)((t >> 7) * 8) * 1024u + (uint32_t)(t & 127) * 8u;            \
                    float2 ev[4], od[4];                                                                              \
                    _Pragma("unroll") for (int j = 0; j < 4; ++j) {                                                   \
                        ev[j] = ld_shared_f2_if(row + (uint32_t)(2 * j) * 1024u, m & (1u << (2 * j)));                \
                        od[j] = ld_shared_f2_if(row + (uint32_t)(2 * j + 1) * 1024u, m & (2u << (2 * j)));            \
                    }                                                                                                 \
                    uint32_t ah[4], al[4];                                                                            \
                    _Pragma("unroll") for (int j = 0; j < 4; ++j) {                                                   \
                        const float2 fa = ev[j] + od[j], fo = ev[j] - od[j];                                          \
                        __half2 h, l2;                                                                                \
                        split_h2(fa.x, fa.y, h, l2);                                                                  \
                        ah[j] = h2u(h);                                                                               \
                        al[j] = h2u(l2);                                                                              \
                        split_h2(fo.x, fo.y, h, l2);                                                                  \
                        bh[i][j] = h2u(h);                                                                            \
                        bl[i][j] = h2u(l2);                                                                           \
                    }                                                                                                 \
                    const uint32_t d = tp_tile(fb, t);                                                                \
                    st_shared_v4(d, ah[0], ah[1], ah[2], ah[3]);                                                      \
                    st_shared_v4(d + TC_FTILE, al[0], al[1], al[2], al[3]);                                           \
                }                                                                                                     \
            }                                                                                                         \
            tc::fence_proxy_async_smem();                                                                             \
            asm volatile("bar.sync 1, 512;" ::: "memory");                                                            \
            if (k >= 1) wait_mma_warp(1, k - 1);                                                                      \
            _Pragma("unroll") for (int i = 0; i < 3; ++i) {                                                           \
                const int t = (ct) + TP_CONV * i;                                                                     \
                if (t < 256 * NC) {                                                                                   \
                    const uint32_t d = tp_tile(fb + (uint32_t)NC * TC_FCHUNK, t);                                     \
                    st_shared_v4(d, bh[i][0], bh[i][1], bh[i][2], bh[i][3]);                                          \
                    st_shared_v4(d + TC_FTILE, bl[i][0], bl[i][1], bl[i][2], bl[i][3]);                               \
                }                                                                                                     \
            }
            // task t: half chunk t / 128 (4 cells, one 16-byte operand row) of
            // rotation t % 128
            auto tp_tile = [](uint32_t base, int t) {
                const uint32_t rr = (uint32_t)t & 127u, hc = (uint32_t)t >> 7;
                return base + (hc >> 1) * TC_FCHUNK + (rr >> 3) * TC_SBO + (hc & 1u) * TC_LBO + (rr & 7u) * 16u;
            };
            TP_CONVERT(tid)
            tc::fence_proxy_async_smem();
            asm volatile("bar.arrive 4, 512;" ::: "memory");
        }
    } else if (warp == 8) {
        // ---------------- MMA issue ----------------
        const uint32_t idesc = tc::idesc_f16_f32(128, 2 * nx8);
        auto issue = [&](int u, int k) {
            const uint32_t f0 = fb + (uint32_t)u * NC * TC_FCHUNK, e0 = ab + (uint32_t)u * 2 * RG * 256;
            const uint32_t d = tmem + 256u * u;
            for (int c = 0; c < NC; ++c) {
                const uint64_t f_h = tc::smem_desc(f0 + c * TC_FCHUNK, TC_LBO, TC_SBO);
                const uint64_t f_l = tc::smem_desc(f0 + c * TC_FCHUNK + TC_FTILE, TC_LBO, TC_SBO);
                // chunk c's rows start 2 (NC - 1 - c) groups into the tile
                const uint32_t eo = e0 + (uint32_t)(NC - 1 - c) * 2u * TC_SBO;
                const uint64_t e_h = tc::smem_desc(eo, TC_LBO, TC_SBO);
                const uint64_t e_l = tc::smem_desc(eo + (uint32_t)RG * 256u, TC_LBO, TC_SBO);
                tc::mma_f16(d, f_h, e_h, idesc, starts_group(k) && c == 0 ? 0u : 1u);
                tc::mma_f16(d, f_l, e_h, idesc, 1u);
                tc::mma_f16(d, f_h, e_l, idesc, 1u);
            }
            tc::mma_commit(&bar[u]);
        };
        for (int k = 0; k < Ka; ++k) {
            asm volatile("bar.sync 1, 512;" ::: "memory");  // staging complete
            asm volatile("bar.sync 1, 512;" ::: "memory");  // A's tiles complete
            if (lane == 0 && !*(volatile int*)&abort_flag) {
                tc::fence_after_sync();
                issue(0, k);
            }
            __syncwarp();
            drain_before(1, k);
            asm volatile("bar.sync 4, 512;" ::: "memory");  // B's tiles complete
            if (lane == 0 && !*(volatile int*)&abort_flag) {
                tc::fence_after_sync();
                issue(1, k);
            }
            __syncwarp();
        }
        // covers every MMA before the tensor memory is released
        if (lane == 0) {
            tc::mma_commit(&done_bar);
            if (!tc::mbar_wait(&done_bar, 0, TC_WAIT_NS)) atomicOr(err, 16);
        }
        __syncwarp();
    } else {
        // ---------------- helpers: circulant tiles, drains ----------------
        const int ht = tid - 288;  // 0 .. 223
        const int n_e = 4 * RG;    // x rows of a tile
        float2 cA = make_float2(0.f, 0.f), cB = cA;
        auto load_c = [&](int kk) {
            if (ht < nx) {
                const float2* c = circ + ((size_t)tinf[Ka + 1 + kk] * NH + pA) * nx + ht;
                cA = __ldg(c);
                cB = __ldg(c + (size_t)nb * nx);
            }
        };
        const float sA = ldexpf(1.0f, (int)cscale[pA]), sB = ldexpf(1.0f, (int)cscale[pA + nb]);
        auto put_sample = [&](int u, float2 c, float sc) {
            if (ht < nx) {
                const float cr = c.x * sc, ci = c.y * sc;
                __half2 rh, rl, ih, il;
                split_h2(cr, -ci, rh, rl);
                split_h2(ci, cr, ih, il);
                st_shared_v4(prb + (uint32_t)(u * nx + ht) * 16u, h2u(rh), h2u(ih), h2u(rl), h2u(il));
            }
        };
        // row pair e (re, im) of pencil u's tile: k = 2 i + {re, im} -> c((x0 + W - 8 + i - e) mod nx)
        auto build = [&](int u, int e0, int step) {
#pragma unroll 1
            for (int e = e0; e < n_e; e += step) {
                int d0 = (x0 + W - 8 - e) % nx;
                if (d0 < 0) d0 += nx;
                TcPair v[8];
#pragma unroll
                for (int i2 = 0; i2 < 8; ++i2) {
                    int d = d0 + i2;
                    while (d >= nx) d -= nx;
                    v[i2] = ld_pair(prb + (uint32_t)(u * nx + d) * 16u);
                }
                const uint32_t hi = ab + (uint32_t)u * 2 * RG * 256, lo = hi + (uint32_t)RG * 256;
                // odd quads of rows store the imaginary row first: eight lanes
                // of a store cover all banks
                const bool odd = (e >> 2) & 1;
                const uint32_t o_a = (uint32_t)(e >> 2) * TC_SBO + (uint32_t)(e & 3) * 32u + (odd ? 16u : 0u);
                const uint32_t o_b = o_a ^ 16u;
#pragma unroll
                for (int kh = 0; kh < 2; ++kh) {
                    uint32_t h1[4], h2[4], l1[4], l2[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const TcPair& a = v[4 * kh + j];
                        h1[j] = odd ? h2u(a.im_h) : h2u(a.re_h);
                        h2[j] = odd ? h2u(a.re_h) : h2u(a.im_h);
                        l1[j] = odd ? h2u(a.im_l) : h2u(a.re_l);
                        l2[j] = odd ? h2u(a.re_l) : h2u(a.im_l);
                    }
                    const uint32_t ko = kh * TC_LBO;
                    st_shared_v4(hi + o_a + ko, h1[0], h1[1], h1[2], h1[3]);
                    st_shared_v4(hi + o_b + ko, h2[0], h2[1], h2[2], h2[3]);
                    st_shared_v4(lo + o_a + ko, l1[0], l1[1], l1[2], l1[3]);
                    st_shared_v4(lo + o_b + ko, l2[0], l2[1], l2[2], l2[3]);
                }
            }
        };
        load_c(0);
        for (int k = 0; k < Ka; ++k) {
            load_mask(tid - 32, k);
            put_sample(0, cA, sA);
            asm volatile("bar.sync 3, 224;" ::: "memory");
            // (every helper has left the previous term's build of B)
            put_sample(1, cB, sB);
            if (k + 1 < Ka) load_c(k + 1);
            if (k >= 1) wait_mma_warp(0, k - 1);
            // A's last group and A's tile: warps 12-15 and 9-11
            if (warp >= 12) drain_before(0, k);
            else build(0, tid - 288, 96);
            auto tp_tile = [](uint32_t base, int t) {
                const uint32_t rr = (uint32_t)t & 127u, hc = (uint32_t)t >> 7;
                return base + (hc >> 1) * TC_FCHUNK + (rr >> 3) * TC_SBO + (hc & 1u) * TC_LBO + (rr & 7u) * 16u;
            };
            TP_CONVERT(tid - 32)
            // B's: warps 8-11 and 12-15
            if (warp < 12) drain_before(1, k);
            else build(1, tid - 384, 128);
            tc::fence_proxy_async_smem();
            asm volatile("bar.arrive 4, 512;" ::: "memory");
        }
    }
#undef TP_CONVERT
    // ---- epilogue: TMEM (+ running sum) -> x-quads g2t[rot][x/4][p][x%4].  Warp:
    // lane quarter warp % 4, pencil and every second quad by warp / 4 ----
    __syncthreads();  // the slots' last additions come before these threads' loads
    {
        const int u = warp >> 3, q0 = (warp >> 2) & 1, n_quads = (nx + 3) >> 2;
        const int rot = g * TC_ROT + 32 * (warp & 3) + lane;
        const float inv = 1.0f / (ldexpf(1.0f, (int)cscale[pA + u * nb]) * TC_F_SCALE);
        const float2* const st = sums + (size_t)u * (TC_ROT * 128);
        float2* const ob = g2t + (size_t)rot * NH * NXP + (size_t)(pA + u * nb) * 4;
        float2 run[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) run[i][j] = make_float2(0.f, 0.f);
        // four quads at a time: their 16 slot loads are in flight together
        auto load_run = [&](int xq) {
            if (with_sum)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (xq + 2 * i < n_quads)
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            run[i][j] = ld_relaxed_f2(st + (size_t)(4 * (xq + 2 * i) + j) * TC_ROT);
        };
        load_run(q0);
        wait_mma(0, Ka - 1);
        wait_mma(1, Ka - 1);
        __syncwarp();
        tc::fence_after_sync();
#pragma unroll 1
        for (int xq = q0; xq < n_quads; xq += 8) {
            if (xq != q0) load_run(xq);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (xq + 2 * i >= n_quads) break;
                uint32_t d[8];
                tc::tmem_ld_32x32b_x8(tmem + 256u * u + trow + 8u * (xq + 2 * i), d);
                tc::tmem_wait_ld();
                float2 v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 t = make_float2(run[i][j].x + __uint_as_float(d[2 * j]),
                                                 run[i][j].y + __uint_as_float(d[2 * j + 1]));
                    v[j] = make_float2(t.x * inv, t.y * inv);
                }
                if (rot < n_rot) st_global_v8(ob + (size_t)(xq + 2 * i) * NH * 4, v);
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 512);
}

// launch over the pencil pairs of nx x ny x nz
template <int N>
cudaError_t launch_pencil_tcp(const BatchArgs& a, int nx, int ny, int nz, const float2* tw, const TcBox& bx,
                              cudaStream_t s) {
    const int nc = a.W / 8, zc = N > 0 || tp_smem_box(nx, ny, nz, nc, a.n_tc_terms, 16) <= kTpMaxSmem ? 16 : 8;
    const size_t sm = N > 0 ? tp_smem_cubic(nx, nc, a.n_tc_terms) : tp_smem_box(nx, ny, nz, nc, a.n_tc_terms, zc);
    const cudaError_t e = allow_smem((const void*)pencil_tcp_kernel<N>, sm);
    if (e != cudaSuccess) return e;
    const int tg = a.tc_group > 0 ? a.tc_group : FFTDOCK_TC_TERMS_PER_SUM_DEFAULT;
    const dim3 grid(ny / 2 * (nz / 2 + 1), (a.n_rot + TC_ROT - 1) / TC_ROT);
    pencil_tcp_kernel<N><<<grid, TP_THREADS, sm, s>>>(a.circ, a.cscale, a.ent_t, a.tinfo, a.n_tc_terms, tw, a.g2t,
                                                      a.n_pad, a.n_rot, a.x0, a.W, tg, a.tc_slots, a.tc_n_slots, bx, zc,
                                                      a.err);
    return cudaGetLastError();
}

}  // namespace fftdock
