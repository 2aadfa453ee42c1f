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
// * the last y pass takes the columns kz and ns - kz together and writes the
//   Hermitian-folded half spectrum Y[kz] = A + i w^kz B, A = X[kz] +
//   conj(X[ns - kz]), B = X[kz] - conj(X[ns - kz]), w = e^{2 pi i / nz}: each
//   row is then one ns-point complex transform whose output m holds the real
//   values of z = 2 m and 2 m + 1;
// * the first y pass reads the plane straight from global memory when it is
//   stored plane by plane.
// Odd nz: two rows a, b travel as one complex line a + i b of nz points.
//
// Bound: the shared-memory passes (seven reads and writes of the plane) and
// their barriers.  Measured on box grids against one warp per line through
// two shared buffers (runtime Stockham stages, lanes idle in short rows,
// per-lane twiddles, an insertion list per warp), per 1024 rotations: 112 x
// 120 x 126 x-quads 20.5 -> 6.0 ms; per 1000 rotations: 90 x 96 x 100 planes
// 14.9 -> 3.1 ms (1.1 TB/s of plane bytes).
#pragma once

#include <type_traits>

#include "fft_core.cuh"
#include "internal.h"
#include "scan_kernels.cuh"

namespace fftdock {

// Radices of one axis, first pass first.  Two passes cover every size that is
// a product of a radix up to 16 and one up to 13; the rest take three or
// four (the last radix stays small: its pass holds two columns).
struct LineRadices {
    int n;
    int np;      // passes (>= 2; a radix of 1 pads a prime length)
    int r[4];
};

constexpr bool line_radices(int n, LineRadices& out) {
    out.n = n;
    out.np = 0;
    int best = 1 << 30;
    for (int a = 2; a <= 16; ++a) {
        if (n % a != 0 || n / a > 13) continue;
        const int b = n / a, cost = 10 * a + 14 * b;
        if (cost < best) {
            best = cost;
            out.np = 2;
            out.r[0] = a;
            out.r[1] = b;
        }
    }
    if (out.np) return true;
    // three passes, then four: the least sum of radices
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
                        out.r[0] = a;
                        out.r[1] = b;
                        out.r[2] = c;
                    }
                } else {
                    for (int d = 2; d <= b; ++d) {
                        if (c % d != 0 || c / d < 2 || c / d > d) continue;
                        if (a + b + d + c / d < best) {
                            best = a + b + d + c / d;
                            out.np = 4;
                            out.r[0] = a;
                            out.r[1] = b;
                            out.r[2] = d;
                            out.r[3] = c / d;
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
    unsigned m_hz, m_col, m_pair, m_row;
    int npair;        // column pairs of the folded last y pass (even nz)
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
    p.npair = even ? (nz / 2 + 1) / 2 : 0;
    p.nrow = even ? ny : (ny + 1) / 2;
    p.m_hz = div_magic(p.hz);
    p.m_col = div_magic(p.ncol);
    p.m_pair = div_magic(p.npair);
    p.m_row = div_magic(p.nrow);
    return line_radices(ny, p.y) && line_radices(even ? nz / 2 : nz, p.z);
}
template <int N> constexpr PlanePlan fixed_plane_plan() {
    PlanePlan p{};
    plane_plan(N, N, p);
    return p;
}

constexpr int kPlaneThreads = 256;
constexpr int kPlaneCand = 256;  // candidate list of the selection

// dynamic shared memory: plane, twiddles of both axes, y of a row position,
// the warps' top-KC lists
constexpr size_t plane_lines_smem(int ny, int nz) {
    const size_t hz = nz / 2 + 1, rows = (size_t)ny + (ny & 1);  // a lone last row's line (odd nz) spans two
    return (rows * (hz | 1) + ny + nz) * sizeof(float2) + ((size_t)ny + 2) * sizeof(int) +
           (size_t)(kPlaneThreads / 32) * KC * 8;
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

// FIXED: N > 0 = the cubic edge N at compile time, 0 = the plan in `rp`.
// QUAD: input = the tensor pencil stage's x-quads [B][nxp / 4][ny hz][4],
// staged by clusters of 4 CTAs (see plane_kernel); else [B][nx][pp].
// dbg (optional, [B][nx][ny][nz]): also write the plane's values.
template <int N, bool QUAD>
__global__ void __launch_bounds__(kPlaneThreads, 3) plane_lines_kernel(
    const float2* __restrict__ g2, const float2* __restrict__ twy_g, const float2* __restrict__ twz_g,
    const __grid_constant__ PlanePlan rp,
    int nx_rt, int nxp_rt, int pp, float* __restrict__ cand_v, int32_t* __restrict__ cand_i, float* __restrict__ dbg) {
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
    int* li_s = reinterpret_cast<int*>(lv_s + (kPlaneThreads / 32) * KC);
    __shared__ float cand_sv[kPlaneCand];
    __shared__ int cand_si[kPlaneCand];
    __shared__ int n_cand;

    const int x = blockIdx.x, q = blockIdx.y;
    const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
    if constexpr (QUAD) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    for (int i = tid; i < ny; i += kPlaneThreads) twy[i] = twy_g[i];
    for (int i = tid; i < nz; i += kPlaneThreads) twz[i] = twz_g[i];
    {
        const int rl = N > 0 ? RYL : rp.y.r[rp.y.np - 1];
        for (int p = tid; p < ny; p += kPlaneThreads) {
            const int b = p / rl;
            ytab[p] = ydigits(b) + (p - b * rl) * (ny / rl);
        }
    }
    const int nh = ny * hz;
    if constexpr (QUAD) {
        uint32_t rank;
        asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
        const int xb = x - (int)rank;  // the cluster's first plane
        // this CTA's quarter of the pencils as 16-byte halves of their quads
        // (planes xb, xb + 1 | xb + 2, xb + 3), coalesced, loads in batches
        // ahead of their stores
        const int q4 = (nh + 3) / 4, p0 = (int)rank * q4, n2 = 2 * max(0, min(q4, nh - p0));
        const float4* gs = reinterpret_cast<const float4*>(g2 + (size_t)q * nh * nxp + (size_t)(xb >> 2) * nh * 4) +
                           (size_t)2 * p0;
        const uint32_t loc = static_cast<uint32_t>(__cvta_generic_to_shared(plane));
        uint32_t rb[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rb[j]) : "r"(loc), "r"(j));
        const uint32_t d0 = (tid & 1) ? rb[2] : rb[0], d1 = (tid & 1) ? rb[3] : rb[1];
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");  // every CTA of the cluster runs
        constexpr int BATCH = 8;
        for (int e0 = tid; e0 < n2; e0 += BATCH * kPlaneThreads) {
            float4 a[BATCH];
#pragma unroll
            for (int k = 0; k < BATCH; ++k) {
                const int e = e0 + k * kPlaneThreads;
                if (e < n2) a[k] = __ldg(gs + e);
            }
#pragma unroll
            for (int k = 0; k < BATCH; ++k) {
                const int e = e0 + k * kPlaneThreads;
                if (e < n2) {
                    const int p = p0 + (e >> 1);
                    const int ky = div_by(p, hz, P.m_hz);
                    const uint32_t off = (uint32_t)(p + ky * (pitch - hz)) * 8u;
                    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(d0 + off), "f"(a[k].x), "f"(a[k].y)
                                 : "memory");
                    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(d1 + off), "f"(a[k].z), "f"(a[k].w)
                                 : "memory");
                }
            }
        }
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (x >= nx) return;  // a padding plane of the last quad
    }
    __syncthreads();

    // element (line, pos) of an in-place pass over sub-blocks of length len
    auto mid_pass = [&](int R_, int n, int len, int n_lines, unsigned magic, int ls, int es, const float2* tw, int tws) {
        with_radix<0, 13>(R_, [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            const int m = len / R, items = n_lines * (n / R), tstep = tws * (n / len);
            for (int it = tid; it < items; it += kPlaneThreads) {
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
    {
        const float2* src = g2 + ((size_t)q * nx + x) * pp;
        with_radix<RY0, 16>(P.y.r[0], [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            const int m = ny / R, items = P.ncol * m;
#pragma unroll 1
            for (int it = tid; it < items; it += kPlaneThreads) {
                const int j = div_by(it, P.ncol, P.m_col);
                const int kz = it - j * P.ncol;
                float2 v[R];
#pragma unroll
                for (int r = 0; r < R; ++r)
                    v[r] = QUAD ? plane[(j + r * m) * pitch + kz] : __ldg(src + (j + r * m) * hz + kz);
                if (even && kz == 0) {
                    // the real columns 0 and ns as one complex column
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float2 o = QUAD ? plane[(j + r * m) * pitch + ns] : __ldg(src + (j + r * m) * hz + ns);
                        v[r] = make_float2(v[r].x - o.y, v[r].y + o.x);
                    }
                }
                dft<R, +1>(v);
#pragma unroll
                for (int r = 1; r < R; ++r) v[r] = ctwiddle<+1>(v[r], twy[j * r]);
#pragma unroll
                for (int r = 0; r < R; ++r) plane[(j + r * m) * pitch + kz] = v[r];
            }
        });
    }
    __syncthreads();
    if constexpr (N == 0) {
        int len = ny / P.y.r[0];
        for (int s = 1; s + 1 < P.y.np; ++s) {
            mid_pass(rp.y.r[s], ny, len, P.ncol, P.m_col, 1, pitch, twy, 1);
            len /= rp.y.r[s];
            __syncthreads();
        }
    }
    // ---- y, last pass ----
    if (even) {
        with_radix<RYL, 13>(N > 0 ? RYL : rp.y.r[rp.y.np - 1], [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            const int items = P.npair * (ny / R);
#pragma unroll 1
            for (int it = tid; it < items; it += kPlaneThreads) {
                const int b = div_by(it, P.npair, P.m_pair);
                const int i = it - b * P.npair;
                // column pair (i, ns - i); pair 0 = the packed columns 0 | ns
                // and the self-paired column ns / 2 (even ns)
                const bool two = i > 0 || (ns & 1) == 0;
                const int c2 = i > 0 ? ns - i : (two ? ns >> 1 : 0);
                float2* pa = plane + b * R * pitch + i;
                float2* pc = plane + b * R * pitch + c2;
                float2 va[R], vc[R];
#pragma unroll
                for (int r = 0; r < R; ++r) va[r] = pa[r * pitch];
#pragma unroll
                for (int r = 0; r < R; ++r) vc[r] = pc[r * pitch];
                dft<R, +1>(va);
                dft<R, +1>(vc);
                if (i > 0) {
                    const float2 wk = twz[i];  // conj(w^i)
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float2 X = va[r], Xm = vc[r];
                        const float2 A = make_float2(X.x + Xm.x, X.y - Xm.y);
                        const float2 B = make_float2(X.x - Xm.x, X.y + Xm.y);
                        const float2 C = cmul_conj(B, wk);
                        pa[r * pitch] = make_float2(A.x - C.y, A.y + C.x);
                        pc[r * pitch] = make_float2(A.x + C.y, C.x - A.y);
                    }
                } else {
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        pa[r * pitch] = make_float2(va[r].x + va[r].y, va[r].x - va[r].y);
                        if (two) pc[r * pitch] = make_float2(2.f * vc[r].x, -2.f * vc[r].y);
                    }
                }
            }
        });
        __syncthreads();
    } else {
        with_radix<RYL, 13>(N > 0 ? RYL : rp.y.r[rp.y.np - 1], [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            const int items = P.ncol * (ny / R);
#pragma unroll 1
            for (int it = tid; it < items; it += kPlaneThreads) {
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
        // rows at positions 2 t, 2 t + 1 -> one complex line a + i b of nz points
        for (int t = w; t < P.nrow; t += kPlaneThreads / 32) {
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
    with_radix<RZ0, 16>(P.z.r[0], [&](auto radix) {
            constexpr int R = decltype(radix)::value;
        const int m = nl / R, items = nrow * m;
#pragma unroll 1
        for (int it = tid; it < items; it += kPlaneThreads) {
            const int j = div_by(it, nrow, P.m_row);
            float2* p = plane + (it - j * nrow) * lstride + j;
            float2 v[R];
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = p[r * m];
            dft<R, +1>(v);
#pragma unroll
            for (int r = 1; r < R; ++r) v[r] = ctwiddle<+1>(v[r], twz[tws * j * r]);
#pragma unroll
            for (int r = 0; r < R; ++r) p[r * m] = v[r];
        }
    });
    __syncthreads();
    if constexpr (N == 0) {
        int len = nl / P.z.r[0];
        for (int s = 1; s + 1 < P.z.np; ++s) {
            mid_pass(rp.z.r[s], nl, len, nrow, P.m_row, lstride, 1, twz, tws);
            len /= rp.z.r[s];
            __syncthreads();
        }
    }
    // last pass: real values back into the rows, every thread keeps the
    // smallest (value, offset) it produced.  each_own(f) calls
    // f(value, offset) for this thread's values again.
    const int zl = N > 0 ? RZL : rp.z.r[rp.z.np - 1];
    const int zstep = nl / zl, zitems = nrow * zstep;
    float bmin_v = INFINITY;
    int bmin_i = 0x7fffffff;
    const int xrow = x * ny;
    // offsets of the two reals of line position (line, block frequency f):
    // even nz: z = 2 f, 2 f + 1 of row `line`; odd: z = f of rows 2 line, 2 line + 1
    auto offs = [&](int line, int& o0, int& o1) {
        if (even) {
            o0 = (xrow + ytab[line]) * nz;
            o1 = o0 + 1;
        } else {
            o0 = (xrow + ytab[2 * line]) * nz;
            o1 = 2 * line + 1 < ny ? (xrow + ytab[2 * line + 1]) * nz : -1;
        }
    };
    const int fmul = even ? 2 : 1;
    with_radix<RZL, 13>(zl, [&](auto radix) {
            constexpr int R = decltype(radix)::value;
#pragma unroll 1
        for (int it = tid; it < zitems; it += kPlaneThreads) {
            const int b = div_by(it, nrow, P.m_row);
            const int line = it - b * nrow;
            float2* p = plane + line * lstride + b * R;
            float2 v[R];
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = p[r];
            dft<R, +1>(v);
            int o0, o1;
            offs(line, o0, o1);
            const int f0 = zdigits(b) * fmul, fs = zstep * fmul;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                p[r] = v[r];
                const int f = f0 + r * fs;
                if (better(v[r].x, o0 + f, bmin_v, bmin_i)) { bmin_v = v[r].x; bmin_i = o0 + f; }
                if ((even || o1 >= 0) && better(v[r].y, o1 + f, bmin_v, bmin_i)) { bmin_v = v[r].y; bmin_i = o1 + f; }
            }
        }
    });

    // ---- selection (as in plane_kernel): the KC-th best of the threads'
    // minima bounds the plane's KC-th best from above ----
    static_assert(KC == 16, "the bitonic selection keeps 16 of 32 lanes");
    constexpr int NW = kPlaneThreads / 32;
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
    {
        float sv = bmin_v;
        int si = bmin_i;
        warp_sort32(sv, si, l);
        if (l < KC) {
            lv_s[w * KC + l] = sv;
            li_s[w * KC + l] = si;
        }
    }
    if (tid == 0) n_cand = 0;
    tree_merge(NW);
    const float tv = lv_s[KC - 1];
    const int ti = li_s[KC - 1];
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
    // or below it (a few per plane): it re-reads its own values
    if (!better(tv, ti, bmin_v, bmin_i)) {
        for (int it = tid; it < zitems; it += kPlaneThreads) {
            const int b = div_by(it, nrow, P.m_row);
            const int line = it - b * nrow;
            const float2* p = plane + line * lstride + b * zl;
            int o0, o1;
            offs(line, o0, o1);
            const int f0 = zdigits(b) * fmul, fs = zstep * fmul;
            for (int r = 0; r < zl; ++r) {
                const float2 o = p[r];
                const int f = f0 + r * fs;
                if (!better(tv, ti, o.x, o0 + f)) {
                    const int at = atomicAdd(&n_cand, 1);
                    if (at < kPlaneCand) { cand_sv[at] = o.x; cand_si[at] = o0 + f; }
                }
                if ((even || o1 >= 0) && !better(tv, ti, o.y, o1 + f)) {
                    const int at = atomicAdd(&n_cand, 1);
                    if (at < kPlaneCand) { cand_sv[at] = o.y; cand_si[at] = o1 + f; }
                }
            }
        }
    }
    __syncthreads();
    const int nc = n_cand;
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

}  // namespace fftdock
