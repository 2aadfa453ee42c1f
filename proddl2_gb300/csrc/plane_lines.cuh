// Plane stage with in-place line passes: CTA = one (rotation, x) plane.
//
// The half-spectrum plane [ny][hz] of one x is transformed inverse along y
// and then to reals along z inside one shared-memory copy of the plane, and
// its KC smallest (value, offset) cells are selected exactly (FFTW c2r of
// FFTCorrelator::correlate + CorrelationProcessor::selectIntoQueue,
// docking_fft.hpp:452-468).
//
// Every transform is a decimation-in-frequency mixed-radix DFT in place: a
// pass of radix R over sub-blocks of length L reads and writes the elements
// b L + j + r L / R (r < R) of a line, so no second buffer is needed and one
// CTA barrier separates passes.  The last pass leaves frequency
// k1 + R1 (k2 + R2 k3 ..) at position (k1 R2 + k2) R3 + k3 ..; nothing puts
// the lines back in order: a row's y and a value's z are looked up when the
// cell's offset is needed.  A warp's lanes are neighbouring lines (columns kz
// in the y passes, rows in the z passes, rows at an odd pitch), so every
// access of a half-warp hits distinct banks, the twiddle is the same for all
// lanes, and no lane idles whatever the radices: work items are (line,
// butterfly) pairs spread over the whole CTA.
//
// Folded passes (even nz, ns = nz / 2):
// * the real columns kz = 0 and ns travel as one complex column
//   X0 + i Xns through the y passes (ns columns instead of ns + 1);
// * the first z pass takes the butterflies j and m - j of a row together:
//   their inputs hold every k with its mirror ns - k, so they are first folded
//   to Y[k] = A + i w^k B, A = X[k] + conj(X[ns - k]), B = X[k] -
//   conj(X[ns - k]), w = e^{2 pi i / nz}; the row is then one ns-point complex
//   transform whose output m holds the real values of z = 2 m and 2 m + 1;
// * the first y pass reads global memory.  From the tensor pencil stage's
//   x-quads (four planes interleaved) every CTA reads its 8 of each 32 bytes,
//   or, on larger planes, a cluster of 4 CTAs shares the pass: each CTA does a
//   quarter of the butterflies for all four planes, two planes per thread from
//   one 16-byte load, and stores the results into the planes' CTAs through
//   distributed shared memory (kPlaneQuad, kPlaneQuadCluster).
// Odd nz: two rows a, b travel as one complex line a + i b of nz points.
//
// Bound: latency between the barriers of the passes.  At 128^3 24 warps per SM
// issue in 49 % of the slots from planes and 34 % from x-quads (16 K warp
// instructions per plane; stalls at barriers, the clusters' among them, and on the
// first pass's loads), the L1 data path is 66 % and 53 % busy, and the plane's bytes
// move at 2.4 and 2.2 TB/s.  Against the kernels it replaced -- on
// cubic edges a two-pass transform with its lines spread over warps (exchange
// barriers in every pass, (value, offset) minima, one re-read of all cells),
// on box grids one warp per line through two buffers -- in ms per 1000
// rotations, planes | x-quads (shape + 18 terms): 48^3 0.46 -> 0.31 | 0.82 ->
// 0.31, 64^3 0.76 -> 0.51 | 0.99 -> 0.56, 80^3 3.21 -> 1.12 | 3.65 -> 1.01, 96^3
// 3.47 -> 1.60 | 4.11 -> 1.58, 112^3 7.91 -> 2.35 | 8.57 -> 2.69, 128^3 4.98 ->
// 3.53 | 5.70 -> 3.93, 144^3 11.6 -> 5.8 | 15.4 -> 6.4; 90 x 96 x 100 14.9 -> 2.9 |,
// 112 x 120 x 126 | 20.0 -> 4.5.
#pragma once

#include <type_traits>

#include "fft_core.cuh"
#include "internal.h"
#include "scan_kernels.cuh"

namespace fftdock {

// Radices of one axis, first pass first.  Two passes cover most sizes; the
// rest take three or four.
struct LineRadices {
    int n;
    int np;      // passes (>= 2; a radix of 1 pads a prime length)
    int r[4];
};

// two passes: first radix up to amax, last up to 16, least wa a + wb b (the
// first pass holds two planes or two butterflies per thread, so it weighs more)
constexpr bool line_radices(int n, int amin, int amax, LineRadices& out) {
    out.n = n;
    out.np = 0;
    int best = 1 << 30;
    for (int a = amin; a <= amax; ++a) {
        if (n % a != 0 || n / a > 16) continue;
        const int b = n / a, cost = 13 * a + 10 * b;
        if (cost < best) {
            best = cost;
            out.np = 2;
            out.r[0] = a;
            out.r[1] = b;
        }
    }
    if (out.np) return true;
    // three passes, then four: the least sum of radices, largest last
    for (int np = 3; np <= 4; ++np) {
        best = 1 << 30;
        for (int a = 2; a <= 13; ++a) {
            if (n % a != 0) continue;
            for (int b = 2; b <= a; ++b) {
                if ((n / a) % b != 0) continue;
                const int c = n / a / b;
                if (np == 3) {
                    if (c < 2 || c > b) continue;
                    if (a + b + c < best) {
                        best = a + b + c;
                        out.np = 3;
                        out.r[0] = c;
                        out.r[1] = b;
                        out.r[2] = a;
                    }
                } else {
                    for (int d = 2; d <= b; ++d) {
                        if (c % d != 0 || c / d < 2 || c / d > d) continue;
                        if (a + b + d + c / d < best) {
                            best = a + b + d + c / d;
                            out.np = 4;
                            out.r[0] = c / d;
                            out.r[1] = d;
                            out.r[2] = b;
                            out.r[3] = a;
                        }
                    }
                }
            }
        }
        if (out.np) return true;
    }
    return false;
}

struct PlanePlan {
    LineRadices y;    // ny
    LineRadices z;    // ns = nz / 2 (even nz) or nz (odd)
    int ny, nz, hz;
    int ncol;         // columns of the y passes: ns (even nz) or hz
    int pitch;        // row pitch in complex values, odd
    // ceil(2^32 / d) for the index divisions: exact while index * d < 2^32
    unsigned m_col, m_row;
    int nrow;         // lines of the z passes: ny (even nz) or ceil(ny / 2)
};

constexpr unsigned div_magic(int d) { return d > 1 ? 0xffffffffu / (unsigned)d + 1u : 0u; }

constexpr bool plane_plan(int ny, int nz, PlanePlan& p) {
    p.ny = ny;
    p.nz = nz;
    p.hz = nz / 2 + 1;
    p.pitch = p.hz | 1;
    const bool even = nz % 2 == 0;
    p.ncol = even ? nz / 2 : p.hz;
    p.nrow = even ? ny : (ny + 1) / 2;
    p.m_col = div_magic(p.ncol);
    p.m_row = div_magic(p.nrow);
    return line_radices(ny, 2, 13, p.y) && (even ? line_radices(nz / 2, 1, 11, p.z) : line_radices(nz, 2, 13, p.z));
}
template <int N> constexpr PlanePlan fixed_plane_plan() {
    PlanePlan p{};
    plane_plan(N, N, p);
    return p;
}

constexpr int kPlaneCand = 256;  // candidate list of the selection
// input of plane_lines_kernel: [B][nx][pp] planes, or the tensor pencil
// stage's x-quads [B][nxp / 4][ny hz][4], read by each CTA alone (8 of every
// 32 bytes) or shared by clusters of 4 CTAs.  Measured per 1000 rotations
// (shape + 18 terms), alone | cluster: 48^3 0.37 | 0.66 ms, 64^3 0.56 | 0.93,
// 80^3 1.01 | 1.39, 96^3 1.58 | 1.95, 112^3 3.00 | 2.68, 128^3 4.50 | 3.86, 112 x
// 120 x 126 4.71 | 4.48: alone while the four-fold reads stay cheap beside
// the cluster's barriers, the line between the 96 and 112 edges.
constexpr int kPlanePlanes = 0, kPlaneQuad = 1, kPlaneQuadCluster = 2;
constexpr int plane_quad_mode(int ny, int nz) { return ny * (nz / 2 + 1) <= 5400 ? kPlaneQuad : kPlaneQuadCluster; }

// dynamic shared memory: plane, twiddles of both axes, y of a row position,
// the warps' top-KC lists
constexpr size_t plane_lines_smem(int ny, int nz) {
    const size_t hz = nz / 2 + 1, rows = (size_t)ny + (ny & 1);  // a lone last row's line (odd nz) spans two
    return (rows * (hz | 1) + ny + nz) * sizeof(float2) + ((size_t)ny + 2) * sizeof(int) + (size_t)8 * KC * 8;
}

__device__ __forceinline__ int div_by(int i, int d, unsigned magic) {
    return d > 1 ? (int)__umulhi((unsigned)i, magic) : i;
}

// runs f<R>() for the plan's radix: a direct call for compile-time plans
template <int FIXED, int RMAX, class F> __device__ __forceinline__ void with_radix(int r, F&& f) {
    if constexpr (FIXED > 0) {
        f(std::integral_constant<int, FIXED>{});
    } else {
        switch (r) {
            case 1: f(std::integral_constant<int, 1>{}); break;
            case 2: f(std::integral_constant<int, 2>{}); break;
            case 3: f(std::integral_constant<int, 3>{}); break;
            case 4: f(std::integral_constant<int, 4>{}); break;
            case 5: f(std::integral_constant<int, 5>{}); break;
            case 6: f(std::integral_constant<int, 6>{}); break;
            case 7: f(std::integral_constant<int, 7>{}); break;
            case 8: f(std::integral_constant<int, 8>{}); break;
            case 9: f(std::integral_constant<int, 9>{}); break;
            case 10: f(std::integral_constant<int, 10>{}); break;
            case 11: f(std::integral_constant<int, 11>{}); break;
            case 12: f(std::integral_constant<int, 12>{}); break;
            case 13: f(std::integral_constant<int, 13>{}); break;
            case 14: if constexpr (RMAX >= 14) f(std::integral_constant<int, 14>{}); break;
            case 15: if constexpr (RMAX >= 15) f(std::integral_constant<int, 15>{}); break;
            case 16: if constexpr (RMAX >= 16) f(std::integral_constant<int, 16>{}); break;
            default: break;
        }
    }
}

// frequency held at block b's output k of the last pass is digits(b) + k step
__device__ __forceinline__ int line_digits(const LineRadices& l, int b) {
    if (l.np == 2) return b;
    // b = (k1 R2 + k2) R3 + ..: digits in reverse weight
    int f = 0, w = l.n / l.r[l.np - 1];
    for (int s = l.np - 2; s >= 0; --s) {
        const int k = b % l.r[s];
        b /= l.r[s];
        w /= l.r[s];
        f += k * w;
    }
    return f;
}

// N > 0: the cubic edge N at compile time; 0: the plan in `rp`.  NT threads.
// dbg (optional, [B][nx][ny][nz]): also write the plane's values.
template <int N, int MODE, int NT>
__global__ void __launch_bounds__(NT, 768 / NT) plane_lines_kernel(
    const float2* __restrict__ g2, const float2* __restrict__ twy_g, const float2* __restrict__ twz_g,
    const __grid_constant__ PlanePlan rp,
    int nx_rt, int nxp_rt, int pp, float* __restrict__ cand_v, int32_t* __restrict__ cand_i, float* __restrict__ dbg) {
    constexpr bool QUAD = MODE != kPlanePlanes, CLUSTER = MODE == kPlaneQuadCluster;
    constexpr PlanePlan FP = fixed_plane_plan<(N > 0 ? N : 16)>();
    PlanePlan P;  // compile-time plans: every field is a constant
    if constexpr (N > 0) P = FP;
    else P = rp;
    auto ydigits = [&](int b) { return N > 0 ? b : line_digits(rp.y, b); };
    auto zdigits = [&](int b) { return N > 0 ? b : line_digits(rp.z, b); };
    constexpr int RY0 = N > 0 ? FP.y.r[0] : 0, RYL = N > 0 ? FP.y.r[FP.y.np - 1] : 0;
    constexpr int RZ0 = N > 0 ? FP.z.r[0] : 0, RZL = N > 0 ? FP.z.r[FP.z.np - 1] : 0;
    static_assert(N == 0 || (FP.y.np == 2 && FP.z.np == 2), "the cubic edges take two passes per axis");
    const int nx = N > 0 ? N : nx_rt, nxp = N > 0 ? N : nxp_rt;
    const int ny = P.ny, nz = P.nz, hz = P.hz, pitch = P.pitch;
    const bool even = N > 0 ? N % 2 == 0 : (nz & 1) == 0;
    const int ns = nz / 2;

    extern __shared__ __align__(1024) unsigned char smem_raw[];
    float2* plane = reinterpret_cast<float2*>(smem_raw);  // [ny rounded up to even][pitch]
    float2* twy = plane + (size_t)(ny + (ny & 1)) * pitch;  // [ny]
    float2* twz = twy + ny;                               // [nz]
    int* ytab = reinterpret_cast<int*>(twz + nz);         // [ny] y of row position p
    float* lv_s = reinterpret_cast<float*>(ytab + ((ny + 1) & ~1));  // [8][KC]
    int* li_s = reinterpret_cast<int*>(lv_s + 8 * KC);
    __shared__ float cand_sv[kPlaneCand];
    __shared__ int cand_si[kPlaneCand];
    __shared__ int n_cand;
    __shared__ int nonzero;  // some input value of this plane is not zero

    const int x = blockIdx.x, q = blockIdx.y;
    const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
    if (tid == 0) nonzero = 0;
    if constexpr (CLUSTER) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    for (int i = tid; i < ny; i += NT) twy[i] = twy_g[i];
    for (int i = tid; i < nz; i += NT) twz[i] = twz_g[i];
    {
        const int rl = N > 0 ? RYL : rp.y.r[rp.y.np - 1];
        for (int p = tid; p < ny; p += NT) {
            const int b = p / rl;
            ytab[p] = ydigits(b) + (p - b * rl) * (ny / rl);
        }
    }
    const size_t nh = (size_t)ny * hz;
    // A plane whose input is all zeros (the ligand reaches no receptor cell at
    // this x: exact zeros from the tensor stage) transforms to all zeros; its
    // KC best cells are its first KC.  A third of the planes at 128^3 with
    // 4000 / 1500 atoms.
    auto zero_plane = [&]() {
        const int cells = ny * nz;
        if (tid < KC) {
            const size_t o = ((size_t)q * nx + x) * KC + tid;
            cand_v[o] = tid < cells ? 0.f : INFINITY;
            cand_i[o] = tid < cells ? x * cells + tid : 0x7fffffff;
        }
        if (dbg)
            for (int i = tid; i < cells; i += NT) dbg[((size_t)q * nx + x) * cells + i] = 0.f;
    };
    __syncthreads();

    // element (line, pos) of an in-place pass over sub-blocks of length len
    auto mid_pass = [&](int R_, int n, int len, int n_lines, unsigned magic, int ls, int es, const float2* tw, int tws) {
        with_radix<0, 13>(R_, [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            const int m = len / R, items = n_lines * (n / R), tstep = tws * (n / len);
            for (int it = tid; it < items; it += NT) {
                const int qb = div_by(it, n_lines, magic);
                float2* p = plane + (it - qb * n_lines) * ls;
                const int b = qb / m, j = qb - b * m;
                p += (b * len + j) * es;
                float2 v[R];
#pragma unroll
                for (int r = 0; r < R; ++r) v[r] = p[r * m * es];
                dft<R, +1>(v);
#pragma unroll
                for (int r = 1; r < R; ++r) v[r] = ctwiddle<+1>(v[r], tw[tstep * j * r]);
#pragma unroll
                for (int r = 0; r < R; ++r) p[r * m * es] = v[r];
            }
        });
    };

    // ---- y, first pass: butterfly j of column kz reads ky = j + r ny / R ----
    if constexpr (CLUSTER) {
        uint32_t rank;
        asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
        const float4* src = reinterpret_cast<const float4*>(g2 + (size_t)q * nh * nxp + (size_t)((x - (int)rank) >> 2) * nh * 4);
        // this thread's planes: 2 h and 2 h + 1 of the quad
        const int h = tid & 1;
        uint32_t d0, d1;
        const uint32_t loc = static_cast<uint32_t>(__cvta_generic_to_shared(plane));
        const uint32_t flag = static_cast<uint32_t>(__cvta_generic_to_shared(&nonzero));
        {
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d0) : "r"(loc), "r"(2 * h));
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d1) : "r"(loc), "r"(2 * h + 1));
        }
        with_radix<RY0, 13>(N > 0 ? RY0 : rp.y.r[0], [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            const int m = ny / R, total = P.ncol * m, share = (total + 3) / 4;
            const int i0 = (int)rank * share, i1 = min(i0 + share, total);
            bool arrived = false;
            unsigned any_a = 0, any_b = 0;
#pragma unroll 1
            for (int it = i0 + (tid >> 1); it < i1; it += NT / 2) {
                const int j = div_by(it, P.ncol, P.m_col);
                const int kz = it - j * P.ncol;
                float2 va[R], vb[R];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float4 t = __ldg(src + (size_t)((j + r * m) * hz + kz) * 2 + h);
                    va[r] = make_float2(t.x, t.y);
                    vb[r] = make_float2(t.z, t.w);
                    any_a |= __float_as_uint(t.x) | __float_as_uint(t.y);
                    any_b |= __float_as_uint(t.z) | __float_as_uint(t.w);
                }
                if (even && kz == 0) {
                    // the real columns 0 and ns as one complex column
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float4 t = __ldg(src + (size_t)((j + r * m) * hz + ns) * 2 + h);
                        va[r] = make_float2(va[r].x - t.y, va[r].y + t.x);
                        vb[r] = make_float2(vb[r].x - t.w, vb[r].y + t.z);
                        any_a |= __float_as_uint(t.x) | __float_as_uint(t.y);
                        any_b |= __float_as_uint(t.z) | __float_as_uint(t.w);
                    }
                }
                dft<R, +1>(va);
                dft<R, +1>(vb);
#pragma unroll
                for (int r = 1; r < R; ++r) {
                    const float2 t = twy[j * r];
                    va[r] = ctwiddle<+1>(va[r], t);
                    vb[r] = ctwiddle<+1>(vb[r], t);
                }
                if (!arrived) {
                    asm volatile("barrier.cluster.wait;" ::: "memory");  // every CTA of the cluster runs
                    arrived = true;
                }
                const uint32_t off = (uint32_t)(j * pitch + kz) * 8u, st = (uint32_t)(m * pitch) * 8u;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(d0 + off + r * st), "f"(va[r].x),
                                 "f"(va[r].y)
                                 : "memory");
                    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(d1 + off + r * st), "f"(vb[r].x),
                                 "f"(vb[r].y)
                                 : "memory");
                }
            }
            if (!arrived) asm volatile("barrier.cluster.wait;" ::: "memory");
            // (x & 0x7fffffff: -0 counts as zero)
            if (any_a & 0x7fffffffu) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(d0 - loc + flag), "r"(1) : "memory");
            if (any_b & 0x7fffffffu) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(d1 - loc + flag), "r"(1) : "memory");
        });
        asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
        if (x >= nx) return;  // a padding plane of the last quad
        if (nonzero == 0) {
            zero_plane();
            return;
        }
    } else {
        const float2* src = QUAD ? g2 + (size_t)q * nh * nxp + (size_t)(x >> 2) * nh * 4 + (x & 3)
                                 : g2 + ((size_t)q * nx + x) * pp;
        constexpr int SS = QUAD ? 4 : 1;
        unsigned any = 0;
        with_radix<RY0, 13>(N > 0 ? RY0 : rp.y.r[0], [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            const int m = ny / R, items = P.ncol * m;
#pragma unroll 1
            for (int it = tid; it < items; it += NT) {
                const int j = div_by(it, P.ncol, P.m_col);
                const int kz = it - j * P.ncol;
                float2 v[R];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    v[r] = __ldg(src + SS * ((j + r * m) * hz + kz));
                    if (QUAD) any |= __float_as_uint(v[r].x) | __float_as_uint(v[r].y);
                }
                if (even && kz == 0) {
                    // the real columns 0 and ns as one complex column
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float2 o = __ldg(src + SS * ((j + r * m) * hz + ns));
                        v[r] = make_float2(v[r].x - o.y, v[r].y + o.x);
                        if (QUAD) any |= __float_as_uint(o.x) | __float_as_uint(o.y);
                    }
                }
                dft<R, +1>(v);
#pragma unroll
                for (int r = 1; r < R; ++r) v[r] = ctwiddle<+1>(v[r], twy[j * r]);
#pragma unroll
                for (int r = 0; r < R; ++r) plane[(j + r * m) * pitch + kz] = v[r];
            }
        });
        if (QUAD) {
            // (-0 counts as zero)
            if (!__syncthreads_or((any & 0x7fffffffu) != 0u)) {
                zero_plane();
                return;
            }
        } else {
            __syncthreads();
        }
    }
    if constexpr (N == 0) {
        int len = ny / P.y.r[0];
        for (int s = 1; s + 1 < P.y.np; ++s) {
            mid_pass(rp.y.r[s], ny, len, P.ncol, P.m_col, 1, pitch, twy, 1);
            len /= rp.y.r[s];
            __syncthreads();
        }
    }
    // ---- y, last pass ----
    with_radix<RYL, 16>(N > 0 ? RYL : rp.y.r[rp.y.np - 1], [&](auto radix) {
        constexpr int R = decltype(radix)::value;
        const int items = P.ncol * (ny / R);
#pragma unroll 1
        for (int it = tid; it < items; it += NT) {
            const int b = div_by(it, P.ncol, P.m_col);
            float2* p = plane + b * R * pitch + (it - b * P.ncol);
            float2 v[R];
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = p[r * pitch];
            dft<R, +1>(v);
#pragma unroll
            for (int r = 0; r < R; ++r) p[r * pitch] = v[r];
        }
    });
    __syncthreads();
    if (!even) {
        // rows at positions 2 t, 2 t + 1 -> one complex line a + i b of nz points
        for (int t = w; t < P.nrow; t += NT / 32) {
            float2* la = plane + 2 * t * pitch;
            const bool has_b = 2 * t + 1 < ny;
            float2 a[4], b[4];  // hz <= 128
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int k = l + 32 * u;
                a[u] = k < hz ? la[k] : make_float2(0.f, 0.f);
                b[u] = k < hz && has_b ? la[pitch + k] : make_float2(0.f, 0.f);
            }
            __syncwarp();
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int k = l + 32 * u;
                if (k < hz) {
                    la[k] = make_float2(a[u].x - b[u].y, a[u].y + b[u].x);
                    if (k > 0) la[nz - k] = make_float2(a[u].x + b[u].y, b[u].x - a[u].y);
                }
            }
        }
        __syncthreads();
    }

    // ---- z passes over the rows ----
    const int nl = even ? ns : nz;                    // points per line
    const int lstride = even ? pitch : 2 * pitch;     // line stride
    const int nrow = P.nrow, tws = even ? 2 : 1;      // w_nl = w_nz^tws
    if (even) {
        with_radix<RZ0, 11>(N > 0 ? RZ0 : rp.z.r[0], [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            const int m = nl / R, items = nrow * ((m + 1) >> 1);
#pragma unroll 1
            for (int it = tid; it < items; it += NT) {
                // butterflies i and m - i of a row; i = 0: butterfly 0 and,
                // for even m, m / 2 (each its own mirror)
                const int i = div_by(it, nrow, P.m_row);
                const bool two = i > 0 || (m & 1) == 0;
                const int i2 = i > 0 ? m - i : (two ? m >> 1 : 0);
                float2* row = plane + (it - i * nrow) * lstride;
                float2 va[R], vb[R];
#pragma unroll
                for (int r = 0; r < R; ++r) va[r] = row[i + r * m];
#pragma unroll
                for (int r = 0; r < R; ++r) vb[r] = row[i2 + r * m];
                // X = X[k], Xm = X[ns - k] -> Y[k], Y[ns - k]
                auto fold = [&](float2& X, float2& Xm, int k) {
                    const float2 A = make_float2(X.x + Xm.x, X.y - Xm.y);
                    const float2 B = make_float2(X.x - Xm.x, X.y + Xm.y);
                    const float2 C = cmul_conj(B, twz[k]);
                    X = make_float2(A.x - C.y, A.y + C.x);
                    Xm = make_float2(A.x + C.y, C.x - A.y);
                };
                auto fold_self = [&](float2& X) { X = make_float2(2.f * X.x, -2.f * X.y); };  // k = ns / 2
                if (i > 0) {
#pragma unroll
                    for (int r = 0; r < R; ++r) fold(va[r], vb[R - 1 - r], i + r * m);
                } else {
                    va[0] = make_float2(va[0].x + va[0].y, va[0].x - va[0].y);  // the packed X0 + i Xns
#pragma unroll
                    for (int r = 1; 2 * r < R; ++r) fold(va[r], va[R - r], r * m);
                    if (R % 2 == 0) fold_self(va[R / 2]);
#pragma unroll
                    for (int r = 0; 2 * r + 1 < R; ++r) fold(vb[r], vb[R - 1 - r], i2 + r * m);
                    if (R % 2 == 1) fold_self(vb[R / 2]);
                }
                dft<R, +1>(va);
                dft<R, +1>(vb);
#pragma unroll
                for (int r = 1; r < R; ++r) va[r] = ctwiddle<+1>(va[r], twz[2 * i * r]);
#pragma unroll
                for (int r = 0; r < R; ++r) row[i + r * m] = va[r];
                if (two) {
#pragma unroll
                    for (int r = 1; r < R; ++r) vb[r] = ctwiddle<+1>(vb[r], twz[2 * i2 * r]);
#pragma unroll
                    for (int r = 0; r < R; ++r) row[i2 + r * m] = vb[r];
                }
            }
        });
    } else {
        with_radix<RZ0, 13>(N > 0 ? RZ0 : rp.z.r[0], [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            const int m = nl / R, items = nrow * m;
#pragma unroll 1
            for (int it = tid; it < items; it += NT) {
                const int j = div_by(it, nrow, P.m_row);
                float2* p = plane + (it - j * nrow) * lstride + j;
                float2 v[R];
#pragma unroll
                for (int r = 0; r < R; ++r) v[r] = p[r * m];
                dft<R, +1>(v);
#pragma unroll
                for (int r = 1; r < R; ++r) v[r] = ctwiddle<+1>(v[r], twz[j * r]);
#pragma unroll
                for (int r = 0; r < R; ++r) p[r * m] = v[r];
            }
        });
    }
    __syncthreads();
    if constexpr (N == 0) {
        int len = nl / P.z.r[0];
        for (int s = 1; s + 1 < P.z.np; ++s) {
            mid_pass(rp.z.r[s], nl, len, nrow, P.m_row, lstride, 1, twz, tws);
            len /= rp.z.r[s];
            __syncthreads();
        }
    }
    // last pass: real values back into the rows; every thread keeps the
    // smallest value it produced
    const int zl = N > 0 ? RZL : rp.z.r[rp.z.np - 1];
    const int zstep = nl / zl, zitems = nrow * zstep;
    float bmin = INFINITY;
    with_radix<RZL, 16>(zl, [&](auto radix) {
        constexpr int R = decltype(radix)::value;
#pragma unroll 1
        for (int it = tid; it < zitems; it += NT) {
            const int b = div_by(it, nrow, P.m_row);
            const int line = it - b * nrow;
            float2* p = plane + line * lstride + b * R;
            float2 v[R];
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = p[r];
            dft<R, +1>(v);
            // odd nz and ny: the lone last line carries no second row
            const bool both = even || 2 * line + 1 < ny;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                p[r] = v[r];
                bmin = fminf(bmin, v[r].x);
                if (both) bmin = fminf(bmin, v[r].y);
            }
        }
    });

    // ---- selection: the KC-th smallest of the threads' minima bounds the
    // plane's KC-th value from above (at least KC cells lie at or below it),
    // so the plane's KC best by (value, offset) are among the cells at or
    // below it (usually 16 to 30).  Bitonic warp sorts, lists merged as a
    // tree over the warps. ----
    static_assert(KC == 16, "the bitonic selection keeps 16 of 32 lanes");
    constexpr int NW = NT / 32;
    {
        float v = bmin;
#pragma unroll
        for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
            for (int j = k >> 1; j > 0; j >>= 1) {
                const float o = __shfl_xor_sync(0xffffffffu, v, j);
                v = ((l & k) == 0) == ((l & j) == 0) ? fminf(v, o) : fmaxf(v, o);
            }
        if (l < KC) lv_s[w * KC + l] = v;
    }
    if (tid == 0) n_cand = 0;
    for (int step = 1; step < NW; step <<= 1) {
        __syncthreads();
        if ((w & (2 * step - 1)) == 0 && w + step < NW) {
            float v = l < KC ? lv_s[w * KC + l] : lv_s[(w + step) * KC + 31 - l];
#pragma unroll
            for (int j = 16; j > 0; j >>= 1) {
                const float o = __shfl_xor_sync(0xffffffffu, v, j);
                v = (l & j) == 0 ? fminf(v, o) : fmaxf(v, o);
            }
            if (l < KC) lv_s[w * KC + l] = v;
        }
    }
    __syncthreads();
    const float bound = lv_s[KC - 1];
    // offset of (line, frequency f): even nz: z = 2 f (+ 1: the imaginary
    // part) of row `line`; odd nz: z = f of rows 2 line and 2 line + 1
    const int xrow = x * ny, fmul = even ? 2 : 1;
    auto offs = [&](int line, int& o0, int& o1) {
        if (even) {
            o0 = (xrow + ytab[line]) * nz;
            o1 = o0 + 1;
        } else {
            o0 = (xrow + ytab[2 * line]) * nz;
            o1 = 2 * line + 1 < ny ? (xrow + ytab[2 * line + 1]) * nz : -1;
        }
    };
    if (dbg) {
        // the plane's values, whole rows (the pass barriers above cover the writes)
        float* out = dbg + ((size_t)q * nx + x) * (size_t)ny * nz;
        for (int t = w; t < nrow; t += NW) {
            const float2* row = plane + t * lstride;
            for (int p = l; p < nl; p += 32) {
                const int b = p / zl;
                const int f = zdigits(b) + (p - b * zl) * zstep;
                const float2 o = row[p];
                if (even) {
                    reinterpret_cast<float2*>(out + (size_t)ytab[t] * nz)[f] = o;
                } else {
                    out[(size_t)ytab[2 * t] * nz + f] = o.x;
                    if (2 * t + 1 < ny) out[(size_t)ytab[2 * t + 1] * nz + f] = o.y;
                }
            }
        }
    }
    // only a thread whose own minimum is at or below the bound holds cells at
    // or below it (a few per plane): its warp re-reads that thread's values
    // together, one per lane
    auto offer = [&](float v, int off) {
        if (v <= bound) {
            const int at = atomicAdd(&n_cand, 1);
            if (at < kPlaneCand) { cand_sv[at] = v; cand_si[at] = off; }
        }
    };
    // (single-warp CTAs, 16^3: half of the threads qualify, so each offers its own
    // cells; 4000 rotations 0.77 -> 0.54 ms)
    if constexpr (NT == 32) {
        for (int it = tid; bmin <= bound && it < zitems; it += NT) {
            const int b = div_by(it, nrow, P.m_row);
            const int line = it - b * nrow;
            int o0, o1;
            offs(line, o0, o1);
            for (int r = 0; r < zl; ++r) {
                const float2 o = plane[line * lstride + b * zl + r];
                const int f = (zdigits(b) + r * zstep) * fmul;
                offer(o.x, o0 + f);
                if (even || o1 >= 0) offer(o.y, o1 + f);
            }
        }
    }
    unsigned qual = NT == 32 ? 0u : __ballot_sync(0xffffffffu, bmin <= bound);
    while (qual) {
        const int it0 = w * 32 + __ffs(qual) - 1;
        qual &= qual - 1u;
        const int cells = it0 < zitems ? ((zitems - 1 - it0) / NT + 1) * zl : 0;
        for (int c = l; c < cells; c += 32) {
            const int k = c / zl, r = c - k * zl;
            const int it = it0 + k * NT;
            const int b = div_by(it, nrow, P.m_row);
            const int line = it - b * nrow;
            const float2 o = plane[line * lstride + b * zl + r];
            int o0, o1;
            offs(line, o0, o1);
            const int f = (zdigits(b) + r * zstep) * fmul;
            offer(o.x, o0 + f);
            if (even || o1 >= 0) offer(o.y, o1 + f);
        }
    }
    __syncthreads();
    const int nc = n_cand;
    // lists 0 .. n - 1 (lv_s, li_s, ascending) merged pairwise into list 0
    auto tree_merge = [&](int n_lists) {
        for (int step = 1; step < n_lists; step <<= 1) {
            __syncthreads();
            if ((w & (2 * step - 1)) == 0 && w + step < n_lists) {
                float sv = l < KC ? lv_s[w * KC + l] : lv_s[(w + step) * KC + 31 - l];
                int si = l < KC ? li_s[w * KC + l] : li_s[(w + step) * KC + 31 - l];
                warp_merge32(sv, si, l);
                if (l < KC) {
                    lv_s[w * KC + l] = sv;
                    li_s[w * KC + l] = si;
                }
            }
        }
        __syncthreads();
    };
    float* ov = cand_v + ((size_t)q * nx + x) * KC;
    int32_t* oi = cand_i + ((size_t)q * nx + x) * KC;
    if (nc <= kPlaneCand) {
        // warp w sorts chunks w, w + 8, .. of 32 candidates and keeps their
        // best KC in list w; the lists are then tree-merged
        const int nchunk = (nc + 31) >> 5;
        float sv = INFINITY;
        int si = 0x7fffffff;
        for (int c = w; c < nchunk; c += NW) {
            const int e = 32 * c + l;
            float cv = e < nc ? cand_sv[e] : INFINITY;
            int ci = e < nc ? cand_si[e] : 0x7fffffff;
            warp_sort32(cv, ci, l);
            if (c == w) {
                sv = cv;
                si = ci;
            } else {
                const float rv = __shfl_sync(0xffffffffu, cv, 31 - l);
                const int ri = __shfl_sync(0xffffffffu, ci, 31 - l);
                if (l >= KC) {
                    sv = rv;
                    si = ri;
                }
                warp_merge32(sv, si, l);
            }
        }
        if (l < KC) {
            lv_s[w * KC + l] = sv;
            li_s[w * KC + l] = si;
        }
        tree_merge(nchunk < NW ? nchunk : NW);
        if (w == 0 && l < KC) {
            ov[l] = lv_s[l];
            oi[l] = li_s[l];
        }
        return;
    }
    // many cells tie at the bound (a flat plane): every warp offers its rows'
    // values, then warp 0 merges the warps' lists
    WarpTopK tk;
    tk.init();
    for (int t = w; t < nrow; t += NW) {
        const float2* row = plane + t * lstride;
        int o0, o1;
        offs(t, o0, o1);
        for (int p0 = 0; p0 < nl; p0 += 32) {
            const int p = p0 + l;
            const bool ok = p < nl;
            const float2 o = ok ? row[p] : make_float2(INFINITY, INFINITY);
            const int b = p / zl;
            const int f = (zdigits(b) + (p - b * zl) * zstep) * fmul;
            tk.offer(ok ? o.x : INFINITY, ok ? o0 + f : 0x7fffffff, l);
            const bool ok1 = ok && (even || o1 >= 0);
            tk.offer(ok1 ? o.y : INFINITY, ok1 ? o1 + f : 0x7fffffff, l);
        }
    }
    __syncthreads();
    if (l < KC) {
        lv_s[w * KC + l] = tk.lv;
        li_s[w * KC + l] = tk.li;
    }
    __syncthreads();
    if (w == 0) {
        merge_lists(lv_s, li_s, NW * KC, tk, l);
        if (l < KC) {
            ov[l] = tk.lv;
            oi[l] = tk.li;
        }
    }
}

// launch with the cluster shape of MODE (4 CTAs along x: the planes of a quad)
template <int MODE, class... P, class... Args>
cudaError_t launch_planes(void (*fn)(P...), dim3 grid, int threads, size_t sm, cudaStream_t s, Args... args) {
    const cudaError_t e = allow_smem((const void*)fn, sm);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = sm;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    if (MODE == kPlaneQuadCluster) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = 4;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&cfg, fn, static_cast<P>(args)...);
}

}  // namespace fftdock
