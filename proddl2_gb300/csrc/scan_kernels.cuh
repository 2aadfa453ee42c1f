// Device kernels of the correlation scan.  Templated on the grid edge N;
// instantiated per N by kernels_nXX.cu through dispatch_impl.cuh.
//
// Data layout in HBM (N = grid edge, H = N/2+1, PP = N*H rounded up to 32,
// pencil index p = ky*H + kz):
//   spec  [K][N][PP]   float2  receptor spectra R^_t(kx, p) / N^3
//   rgrid [K][N^3]     double  real-space receptor terms (FP64 rescoring)
//   ent   [B][n_ent]   uint32  per-rotation ligand entries t<<24|x<<16|y<<8|z,
//                              sorted by (t, x, y mod qc), atom order inside a bin
//                              (tensor form: by (t, x), read by the rescoring only)
//   offs  [B][K*N*qc+1]  int32  start of bin (t, x, y mod qc)
//   g2    [B][N][PP]   float2  sum_t conj(R^_t) L^_t inverse-transformed
//                              along x: one complex (ky, kz) plane per x
//   cand  [B][N][KC]           per-plane FP32 candidate pools
#pragma once

#include <cuda_bf16.h>
#include <math.h>
#include <stdint.h>

#include "fft_core.cuh"
#include "fftdock.h"
#include "internal.h"

namespace fftdock {

constexpr int KC = 16;  // FP32 candidates kept per plane / per rotation

// Warps per line transform of pencil_kernel: G*G | N.
template <int N> struct SizeTraits;
template <> struct SizeTraits<16> { static constexpr int G = 4; };
template <> struct SizeTraits<24> { static constexpr int G = 2; };
template <> struct SizeTraits<32> { static constexpr int G = 4; };
template <> struct SizeTraits<48> { static constexpr int G = 4; };
template <> struct SizeTraits<64> { static constexpr int G = 8; };
template <> struct SizeTraits<80> { static constexpr int G = 4; };
template <> struct SizeTraits<96> { static constexpr int G = 4; };
template <> struct SizeTraits<112> { static constexpr int G = 4; };
template <> struct SizeTraits<128> { static constexpr int G = 8; };
template <> struct SizeTraits<144> { static constexpr int G = 12; };

// Pencil kernel occupancy: exchange buffers (2: one barrier per term; 1: two
// barriers per term but N*32 complex less shared memory) and the CTAs per SM
// its launch bounds ask for (which caps the registers).  Chosen per edge from
// timed scans on GB300 (shape + 18 terms; pencil-kernel time against the
// two-buffer, unbounded form): 64 -22 %, 80 -11 %, 96 -12 %, 128 -6 %,
// 144 -25 %; 112 gained nothing.
template <int N> struct PencilTraits { static constexpr int BUFS = 2, MINB = 1; };
template <> struct PencilTraits<64> { static constexpr int BUFS = 1, MINB = 4; };
template <> struct PencilTraits<80> { static constexpr int BUFS = 1, MINB = 4; };
template <> struct PencilTraits<96> { static constexpr int BUFS = 1, MINB = 4; };
template <> struct PencilTraits<128> { static constexpr int BUFS = 1, MINB = 3; };
template <> struct PencilTraits<144> { static constexpr int BUFS = 2, MINB = 2; };


// toLogical: int((x - zero_h) / h) - 1, truncation toward zero, no FMA.
// Returns the truncated quotient; the cell is q - 1.
__device__ __forceinline__ int logical_q(double x, const Geo& g, int d) {
    return __double2int_rz(__ddiv_rn(__dsub_rn(x, g.zero_h[d]), g.h));
}
__device__ __forceinline__ double cell_centre(int i, const Geo& g, int d) {
    return __dadd_rn(g.center0[d], __dmul_rn(g.h, (double)i));
}

// ---------------------------------------------------------------------------
// warp top-k (KC smallest by (value, index); lanes < KC hold the sorted list)
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool better(float a, int ia, float b, int ib) {
    return a < b || (a == b && ia < ib);
}

// Compare-exchange with lane ^ j under better(): this lane keeps the better
// of the two pairs when keep_min, else the other one.
__device__ __forceinline__ void warp_cmp_swap(float& v, int& i, int j, bool keep_min) {
    const float pv = __shfl_xor_sync(0xffffffffu, v, j);
    const int pi = __shfl_xor_sync(0xffffffffu, i, j);
    if (better(pv, pi, v, i) == keep_min) {
        v = pv;
        i = pi;
    }
}

// Bitonic sort of one (value, index) pair per lane, ascending by better()
// across the warp (15 compare-exchange steps).
__device__ __forceinline__ void warp_sort32(float& v, int& i, int lane) {
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) warp_cmp_swap(v, i, j, ((lane & k) == 0) == ((lane & j) == 0));
}

// Lanes 0..15 ascending and lanes 16..31 descending (a bitonic sequence) ->
// all 32 ascending: lanes < 16 then hold the 16 best of both halves.
__device__ __forceinline__ void warp_merge32(float& v, int& i, int lane) {
#pragma unroll
    for (int j = 16; j > 0; j >>= 1) warp_cmp_swap(v, i, j, (lane & j) == 0);
}

struct WarpTopK {
    float lv;
    int li;
    float tv;  // current KC-th value (threshold)
    int ti;
    __device__ __forceinline__ void init() { lv = INFINITY; li = 0x7fffffff; tv = INFINITY; ti = 0x7fffffff; }
    // offer one candidate per lane (all lanes of the warp must call)
    __device__ __forceinline__ void offer(float v, int idx, int lane) {
        // v <= tv is necessary for (v, idx) < (tv, ti); the exact test runs
        // only on the rare candidates
        if (__ballot_sync(0xffffffffu, v <= tv) == 0u) return;
        unsigned mask = __ballot_sync(0xffffffffu, better(v, idx, tv, ti));
        if (__popc(mask) > 6) {
            // many at once: sort the qualifying offers and merge them with
            // the list (lanes < KC ascending, the best KC offers descending
            // above them: one bitonic sequence) -- the same KC best by
            // (value, index) as one insertion each
            static_assert(KC == 16, "the batch merge takes lists of 16");
            float sv = (mask >> lane) & 1u ? v : INFINITY;
            int si = (mask >> lane) & 1u ? idx : 0x7fffffff;
            warp_sort32(sv, si, lane);
            const float rv = __shfl_sync(0xffffffffu, sv, 31 - lane);
            const int ri = __shfl_sync(0xffffffffu, si, 31 - lane);
            float mv = lane < KC ? lv : rv;
            int mi = lane < KC ? li : ri;
            warp_merge32(mv, mi, lane);
            lv = mv;
            li = mi;
            tv = __shfl_sync(0xffffffffu, lv, KC - 1);
            ti = __shfl_sync(0xffffffffu, li, KC - 1);
            return;
        }
        while (mask) {
            const int src = __ffs(mask) - 1;
            const float cv = __shfl_sync(0xffffffffu, v, src);
            const int ci = __shfl_sync(0xffffffffu, idx, src);
            const unsigned below = __ballot_sync(0xffffffffu, lane < KC && better(lv, li, cv, ci));
            const int pos = __popc(below);
            const float upv = __shfl_up_sync(0xffffffffu, lv, 1);
            const int upi = __shfl_up_sync(0xffffffffu, li, 1);
            if (pos < KC) {
                if (lane == pos) { lv = cv; li = ci; }
                else if (lane > pos && lane < KC) { lv = upv; li = upi; }
            }
            tv = __shfl_sync(0xffffffffu, lv, KC - 1);
            ti = __shfl_sync(0xffffffffu, li, KC - 1);
            mask &= ~(1u << src);
            mask &= __ballot_sync(0xffffffffu, better(v, idx, tv, ti));
        }
    }
};

// Merge per-warp lists staged in shared memory (nw lists of KC) into warp 0's
// list; the caller syncs before and reads lanes < KC of warp 0 after.
__device__ __forceinline__ void merge_lists(const float* sv, const int* si, int n, WarpTopK& tk, int lane) {
    tk.init();
    for (int base = 0; base < n; base += 32) {
        const int e = base + lane;
        const float v = e < n ? sv[e] : INFINITY;
        const int i = e < n ? si[e] : 0x7fffffff;
        tk.offer(v, i, lane);
    }
}

// Where ligand prep's scatter puts the entry of lane `l` (bin -1: none): its
// place `bin` among the sorted rows of the pencil stage, and `tx` in the order
// (term, x), atom order inside, that the FP64 rescoring sums in whatever the
// pencil form (a rotation's scores do not depend on the form that found its
// cells).  They differ for pencil pairs only (PAIRS: bins (t, x, y mod 2)), whose
// odd bins hold start << 16 | entries so far (pair_counts; at most 32768 entries).
// peers: the lanes of the same bin.
struct EntrySlot {
    int bin, tx;
    unsigned peers;
};
template <bool PAIRS> __device__ __forceinline__ EntrySlot entry_slot(const int32_t* cnt, int bin, int l) {
    const unsigned below = (1u << l) - 1u;
    const unsigned peers_tx = __match_any_sync(0xffffffffu, PAIRS ? bin >> 1 : bin);
    EntrySlot s{0, 0, peers_tx};
    if constexpr (PAIRS) {
        const unsigned odd_lanes = __ballot_sync(0xffffffffu, bin & 1);
        s.peers &= (bin & 1) ? odd_lanes : ~odd_lanes;
    }
    const int rank = __popc(s.peers & below);
    if (bin >= 0) {
        if constexpr (PAIRS) {
            const int even = cnt[bin & ~1];
            const uint32_t odd = (uint32_t)cnt[bin | 1];
            const int n_odd = (int)(odd & 0xffffu);
            s.bin = ((bin & 1) ? (int)(odd >> 16) + n_odd : even) + rank;
            s.tx = even + n_odd + __popc(peers_tx & below);
        } else {
            s.bin = s.tx = cnt[bin] + rank;
        }
    }
    return s;
}
__device__ __forceinline__ void pair_counts(int32_t* cnt, int nbins) {
    for (int i = 2 * threadIdx.x + 1; i < nbins; i += 2 * blockDim.x) cnt[i] = (int32_t)((uint32_t)cnt[i] << 16);
    __syncthreads();
}

// ---------------------------------------------------------------------------
// K1: rotate + bin + stable sort of the ligand entries of one rotation
// (MolForceRadial::projectLigand, docking_molforce.hpp:351-368, with
// Rotation::operator(), transformation.hpp:206-222).  One CTA per rotation.
// ---------------------------------------------------------------------------
template <int N>
__global__ void __launch_bounds__(256) ligand_prep_kernel(
    const double* __restrict__ rot, const double* __restrict__ lig_xyz, const int32_t* __restrict__ lig_term,
    int n_ent, int K, Geo geo, uint32_t* __restrict__ ent_out, int32_t* __restrict__ offs_out,
    int32_t* __restrict__ status, const float* __restrict__ w_in, uint4* __restrict__ ent4,
    int32_t* __restrict__ idx_out, uint32_t* __restrict__ ent_t, const int32_t* __restrict__ tpad, int n_pad,
    int x0, int W, int qc, const int32_t* __restrict__ tinfo,
    int ka) {
    extern __shared__ unsigned char smem_raw[];
    int32_t* cnt = reinterpret_cast<int32_t*>(smem_raw);               // [K*N*qc + 1]
    uint32_t* keys = reinterpret_cast<uint32_t*>(cnt + K * N * qc + 1);  // [n_ent]
    __shared__ int bad;
    __shared__ int wsum[8];
    const int q = blockIdx.x;
    const int tid = threadIdx.x;
    // bins (t, x, y mod qc), qc = 1 or 2
    const int nbins = K * N * qc, qm = qc - 1;
    for (int i = tid; i <= nbins; i += blockDim.x) cnt[i] = 0;
    if (tid == 0) bad = 0;
    __syncthreads();
    const double* m = rot + 9 * (size_t)q;
    const double m00 = m[0], m01 = m[1], m02 = m[2], m10 = m[3], m11 = m[4], m12 = m[5], m20 = m[6], m21 = m[7],
                 m22 = m[8];
    for (int i = tid; i < n_ent; i += blockDim.x) {
        const double x0 = lig_xyz[3 * i], x1 = lig_xyz[3 * i + 1], x2 = lig_xyz[3 * i + 2];
        // y_i = ((m_i0 x0) + m_i1 x1) + m_i2 x2, each product rounded (no FMA)
        const double p0 = __dadd_rn(__dadd_rn(__dmul_rn(m00, x0), __dmul_rn(m01, x1)), __dmul_rn(m02, x2));
        const double p1 = __dadd_rn(__dadd_rn(__dmul_rn(m10, x0), __dmul_rn(m11, x1)), __dmul_rn(m12, x2));
        const double p2 = __dadd_rn(__dadd_rn(__dmul_rn(m20, x0), __dmul_rn(m21, x1)), __dmul_rn(m22, x2));
        int c0 = logical_q(p0, geo, 0), c1 = logical_q(p1, geo, 1), c2 = logical_q(p2, geo, 2);
        const bool ok = c0 >= 1 && c0 <= N && c1 >= 1 && c1 <= N && c2 >= 1 && c2 <= N;
        if (!ok) atomicOr(&bad, 1);
        c0 = min(max(c0 - 1, 0), N - 1);
        c1 = min(max(c1 - 1, 0), N - 1);
        c2 = min(max(c2 - 1, 0), N - 1);
        const int t = lig_term[i];
        keys[i] = ((uint32_t)t << 24) | ((uint32_t)c0 << 16) | ((uint32_t)c1 << 8) | (uint32_t)c2;
        atomicAdd(&cnt[(t * N + c0) * qc + (c1 & qm)], 1);
    }
    __syncthreads();
    // exclusive scan of cnt[0..nbins) -> starts; cnt[nbins] = n_ent
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
            if (xr < W && c >= 0 && c < N) {
                const int b = (t * N + c) * qc;
                m |= (uint32_t)(cnt[b + 1] > cnt[b]) << (2 * j) | (uint32_t)(cnt[b + 2] > cnt[b + 1]) << (2 * j + 1);
            }
        }
        ent_t[(((size_t)(q >> 7) * (n_pad >> 2) + (tinfo[ka] >> 2) + kk) * 128 + (q & 127)) * 4 + word] = m;
    }
    __syncthreads();
    if (ka) pair_counts(cnt, nbins);
    // stable scatter by one warp: ranks within equal keys follow atom order
    auto scatter = [&](auto pairs) {
        uint32_t* ent = ent_out + (size_t)q * n_ent;
        for (int base = 0; base < n_ent; base += 32) {
            const int i = base + tid;
            const bool act = i < n_ent;
            const uint32_t key = act ? keys[i] : 0xffffffffu;
            const int bin = act ? (int)((key >> 24) * N + ((key >> 16) & 255u)) * qc + (int)((key >> 8) & qm) : -1;
            const EntrySlot at = entry_slot<decltype(pairs)::value>(cnt, bin, tid);
            const int leader = __ffs(at.peers) - 1;
            __syncwarp();
            if (act) ent[at.tx] = key;
            // transposed copy for the tensor pencil stage,
            // [q / 128][row / 4][q % 128][row % 4], with each term's rows
            // padded to a multiple of 8; the term is implied by the row and
            // x is stored relative to the window start x0 (mod 256: cells
            // outside the window stay outside it); entry = row << 24 | y << 16
            // | z, so that one multiply by kz << 16 | ky gives the phase; row =
            // x', or 2 x' + y mod 2 for pencil pairs
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
// K2: pencil kernel of the term sets of several unweighted terms (one term
// and ljComp: pencil_lines.cuh).  CTA = one rotation x 32 consecutive pencils (ky, kz),
// G warps.  For every term t:
//   F(x) = sum over entries of bin (t, x) of w^(ky*y + kz*z)   (the y and z
//          stages of the forward transform, as direct sums over atoms)
//   L^_t(kx) = FFT_x(F); S(kx) += conj(R^_t(kx)) L^_t(kx)
// then S is inverse-transformed along x and written as one column of g2.
// (FFTCorrelator::correlate, docking_fft.hpp:622-633, summed over terms as
// MolForceComp::collectTotal does in real space, docking_molforce.hpp:172-184.)
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 spec_load(const float2* p) { return __ldg(p); }
__device__ __forceinline__ float2 spec_load(const __nv_bfloat162* p) { return __bfloat1622float2(*p); }

// Complex type of its arithmetic: packed adds (float2) but for 128 with FP32
// spectra, whose generated code is slower with them (80 registers either way):
// pencil stage of 200 rotations of 18 terms, packed | scalar: 128^3 FP32 9.05 | 8.78 ms,
// 128^3 BF16 8.55 | 8.76, 64^3 0.77 | 0.82, 96^3 4.30 | 4.60.
template <int N, typename SpecT>
using PencilC = std::conditional_t<N == 128 && std::is_same<SpecT, float2>::value, scalar2, float2>;

template <int N, typename SpecT>
__global__ void __launch_bounds__(32 * SizeTraits<N>::G, PencilTraits<N>::MINB) pencil_kernel(
    const SpecT* __restrict__ spec, const uint32_t* __restrict__ ent, const int32_t* __restrict__ offs,
    const float2* __restrict__ tw, float2* __restrict__ g2, int K, int n_ent) {
    using P = LinePlan<N, SizeTraits<N>::G>;
    constexpr int G = P::G, R1 = P::R1, H = N / 2 + 1;
    constexpr int PP = pencil_pitch(N);
    constexpr int BUFS = PencilTraits<N>::BUFS;
    using C = PencilC<N, SpecT>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* xbuf = reinterpret_cast<C*>(smem_raw);  // [BUFS][N][32]
    C* tws = xbuf + BUFS * N * 32;             // [N]
    // the phase table once per half-warp lane ([phase][16]): a warp's lanes
    // are consecutive pencils, whose phases for one entry step by its z, so
    // a single table would put lanes on the same banks whenever z is even
    float2* twr = reinterpret_cast<float2*>(tws + N);             // [N][16]
    uint32_t* ent_s = reinterpret_cast<uint32_t*>(twr + N * 16);  // [n_ent]
    int32_t* offs_s = reinterpret_cast<int32_t*>(ent_s + n_ent);  // [K*N+1]

    const int q = blockIdx.x;
    const int tile = blockIdx.y;
    const int tid = threadIdx.x;
    const int w = tid >> 5, l = tid & 31;
    const int p = tile * 32 + l;
    const unsigned ky = (unsigned)(p / H), kz = (unsigned)(p - (p / H) * H);
    // entries staged as y << 16 | z (x and the term are the bin's): bits 16 and
    // up of u * (kz << 16 | ky) (mod 2^32) hold ky y + kz z (< 2^16 for N <=
    // 144; the z ky term stays below bit 16), one multiply per phase
    const uint32_t kyz = (kz << 16) | ky;

    for (int i = tid; i < N; i += blockDim.x) tws[i] = C{tw[i].x, tw[i].y};
    for (int i = tid; i < N * 16; i += blockDim.x) twr[i] = tw[i >> 4];
    const int32_t* offs_g = offs + (size_t)q * (K * N + 1);
    for (int i = tid; i <= K * N; i += blockDim.x) offs_s[i] = offs_g[i];
    const uint32_t* ent_g = ent + (size_t)q * n_ent;
    for (int i = tid; i < n_ent; i += blockDim.x) {
        const uint32_t u = ent_g[i];
        ent_s[i] = (((u >> 8) & 255u) << 16) | (u & 255u);
    }
    __syncthreads();

    C S[R1];
#pragma unroll
    for (int i = 0; i < R1; ++i) S[i] = C{0.f, 0.f};

    for (int t = 0; t < K; ++t) {
        C v[R1];
#pragma unroll
        for (int r = 0; r < R1; ++r) {
            const int x = w + G * r;
            const int b = offs_s[t * N + x], e = offs_s[t * N + x + 1];
            C acc{0.f, 0.f};
            for (int j = b; j < e; ++j) {
                const uint32_t yz = (ent_s[j] * kyz) >> 16;
                const unsigned ph = (N & (N - 1)) == 0 ? (yz & (unsigned)(N - 1)) : yz % (unsigned)N;
                const float2 z = twr[ph * 16 + (l & 15)];
                acc.x += z.x;
                acc.y += z.y;
            }
            v[r] = acc;
        }
        dft<R1, -1>(v);
        C* buf = xbuf + (BUFS == 2 ? (t & 1) * N * 32 : 0);
#pragma unroll
        for (int r = 0; r < R1; ++r) buf[(w * R1 + r) * 32 + l] = v[r];
        __syncthreads();
        C F[R1];
        line_pass2<P, -1, 1, 32>(buf, w, l, tws, F);
        if constexpr (BUFS == 1) __syncthreads();  // buf is rewritten by the next term
        const SpecT* sp = spec + (size_t)t * N * PP + p;
#pragma unroll
        for (int i = 0; i < P::NB; ++i)
#pragma unroll
            for (int r = 0; r < G; ++r) {
                const int kx = w + G * i + R1 * r;
                const float2 rv = spec_load(sp + (size_t)kx * PP);
                const C f = F[i * G + r];
                S[i * G + r].x += f.x * rv.x + f.y * rv.y;
                S[i * G + r].y += f.y * rv.x - f.x * rv.y;
            }
    }
    C v[R1];
    pass2_to_pass1_order<P>(S, v);
    dft<R1, +1>(v);
    C* buf = xbuf + (BUFS == 2 ? (K & 1) * N * 32 : 0);
#pragma unroll
    for (int r = 0; r < R1; ++r) buf[(w * R1 + r) * 32 + l] = v[r];
    __syncthreads();
    C out[R1];
    line_pass2<P, +1, 1, 32>(buf, w, l, tws, out);
    float2* dst = g2 + (size_t)q * N * PP + p;
#pragma unroll
    for (int i = 0; i < P::NB; ++i)
#pragma unroll
        for (int r = 0; r < G; ++r) {
            const int x = w + G * i + R1 * r;
            dst[(size_t)x * PP] = make_float2(out[i * G + r].x, out[i * G + r].y);
        }
}

// K3, the plane stage: plane_lines.cuh

// ---------------------------------------------------------------------------
// K4: per-rotation merge of the plane pools, FP64 direct-space rescoring of
// the KC survivors, ascending order and the maxValCorr limit, translation by
// WrappedIndex::unwrap (docking_fft.hpp:316-389, Math/fft.hpp:199-206,
// Common/queue.hpp:221-251).
// ---------------------------------------------------------------------------
template <int N>
__global__ void __launch_bounds__(256) finalize_kernel(
    const float* __restrict__ cand_v, const int32_t* __restrict__ cand_i, const uint32_t* __restrict__ ent,
    const int32_t* __restrict__ status, const double* __restrict__ rgrid, int n_ent, int peak_stride, int k_out,
    double max_val, double h, int first_rot_id, fftdock_peak* __restrict__ peaks, int32_t* __restrict__ n_peaks,
    float* __restrict__ pool_v, int32_t* __restrict__ pool_i, const double* __restrict__ w64,
    const int32_t* __restrict__ ent_idx) {
    __shared__ float lv_s[8 * KC];
    __shared__ int li_s[8 * KC];
    __shared__ double score_s[KC];
    const int q = blockIdx.x;
    const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
    const long V = (long)N * N * N;
    WarpTopK tk;
    tk.init();
    const float* cv = cand_v + (size_t)q * N * KC;
    const int32_t* ci = cand_i + (size_t)q * N * KC;
    for (int base = w * 32; base < N * KC; base += 256) {
        const int e = base + l;
        const float v = e < N * KC ? cv[e] : INFINITY;
        const int i = e < N * KC ? ci[e] : 0x7fffffff;
        tk.offer(v, i, l);
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
            const int sx = off / (N * N), sy = (off / N) % N, sz = off % N;
            for (int j = l; j < n_ent; j += 32) {
                const uint32_t u = e_q[j];
                const int t = (int)(u >> 24);
                const int ax = (int)((u >> 16) & 255u), ay = (int)((u >> 8) & 255u), az = (int)(u & 255u);
                const int gx = ax - sx < 0 ? ax - sx + N : ax - sx;
                const int gy = ay - sy < 0 ? ay - sy + N : ay - sy;
                const int gz = az - sz < 0 ? az - sz + N : az - sz;
                const double rv = rgrid[(size_t)t * V + ((size_t)gx * N + gy) * N + gz];
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
        for (int c = 0; c < KC; ++c) { sc[c] = score_s[c]; of[c] = li_s[c]; }
        for (int a = 1; a < KC; ++a) {
            const double s = sc[a];
            const int o = of[a];
            int b = a - 1;
            while (b >= 0 && (sc[b] > s || (sc[b] == s && of[b] > o))) {
                sc[b + 1] = sc[b]; of[b + 1] = of[b]; --b;
            }
            sc[b + 1] = s; of[b + 1] = o;
        }
        int n = 0;
        if (status[q] == 0) {
            for (int c = 0; c < KC && n < k_out; ++c) {
                if (!(sc[c] < max_val) || of[c] < 0 || of[c] >= V) continue;
                const int sx = of[c] / (N * N), sy = (of[c] / N) % N, sz = of[c] % N;
                fftdock_peak pk;
                pk.rot_id = first_rot_id + q;
                pk.cell[0] = sx; pk.cell[1] = sy; pk.cell[2] = sz;
                const int s3[3] = {sx, sy, sz};
                for (int d = 0; d < 3; ++d) {
                    int yv = -s3[d];
                    if (yv < -(N / 2)) yv += N;
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

__device__ __forceinline__ void spec_store(float2* p, float x, float y) { *p = make_float2(x, y); }
__device__ __forceinline__ void spec_store(__nv_bfloat162* p, float x, float y) { *p = __floats2bfloat162_rn(x, y); }

}  // namespace fftdock
