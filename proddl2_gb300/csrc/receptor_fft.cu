// Receptor transforms, once per pair: every FP64 term grid [Nx][Ny][Nz] of a
// pair forward along z, y and x (real input, half spectrum kz < Hz), the
// results rounded once to the pencil stages' operands: the spectra [Nx][PP]
// (FP32 or BF16 pairs, / V) and, for the tensor form, the circulant samples
// [Ny Hz][Nx] (transformed along z and y only, conjugated, / (Ny Nz)) with a
// power-of-two scale exponent per pencil.
//
// One launch per axis covers all terms (or a chunk of them, see kRfWork).  A CTA transforms 32 lines in shared
// memory ([position][32 lanes], in place, decimation in frequency as in
// plane_lines.cuh); two real rows travel along z as one complex line; the x
// launch writes the circulant samples, their maxima and the spectra from the
// lines it holds.
//
// Bound: FP64 arithmetic (this chip issues two FP64 operations per SM and
// clock); rows and columns the receptor does not reach are skipped.  Against
// one launch per term, axis and conversion (complex copy, complex z transform,
// half extraction, packing, a scale pass over all samples; 127 launches),
// 96^3, shape + 18 terms: 2.1 -> 1.0 ms.
#include <algorithm>

#include "fft_core.cuh"
#include "internal.h"
#include "plane_lines.cuh"

namespace fftdock {
namespace {

constexpr int kRfThreads = 256, kRfPitch = 33;

// passes of radix up to 10 (FP64 registers), larger only for the primes 11, 13
constexpr bool rf_radices(int n, LineRadices& r) {
    int best = 1 << 30;
    for (int a = 1; a <= 13; ++a) {
        if (n % a != 0 || n / a > 13) continue;
        const int b = n / a;
        const int cost = a + b + (a > 10 && a % 11 && a % 13 ? 8 : 0) + (b > 10 && b % 11 && b % 13 ? 8 : 0);
        if (cost < best) {
            best = cost;
            r.n = n;
            r.np = 2;
            r.r[0] = a;
            r.r[1] = b;
        }
    }
    if (best < 20) return true;
    LineRadices t{};
    // the least sum over three passes (line_radices' fallback, reached by
    // asking for a first radix that does not exist)
    if (line_radices(n, 14, 13, t)) {
        r = t;
        return true;
    }
    return best < (1 << 30);
}

// forward transform of the CTA's 32 lines; natural order in, frequency
// line_freq(p) at position p out
__device__ __forceinline__ void lines64(double2* buf, const LineRadices& rx, const double2* tw) {
    const int n = rx.n, w = threadIdx.x >> 5, l = threadIdx.x & 31;
    int len = n;
    for (int s = 0; s < rx.np; ++s) {
        with_radix<0, 13>(rx.r[s], [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            const int m = len / R, tstep = n / len;
            for (int it = w; it < n / R; it += kRfThreads / 32) {
                const int blk = it / m, j = it - blk * m;
                double2* p = buf + (size_t)(blk * len + j) * kRfPitch + l;
                double2 v[R];
#pragma unroll
                for (int r = 0; r < R; ++r) v[r] = p[r * m * kRfPitch];
                dft<R, -1>(v);
                if (m > 1) {
#pragma unroll
                    for (int r = 1; r < R; ++r) v[r] = cmul(v[r], tw[tstep * j * r]);
                }
#pragma unroll
                for (int r = 0; r < R; ++r) p[r * m * kRfPitch] = v[r];
            }
        });
        len /= rx.r[s];
        __syncthreads();
    }
}
__device__ __forceinline__ int line_freq(const LineRadices& rx, int p) {
    const int rl = rx.r[rx.np - 1], b = p / rl;
    return line_digits(rx, b) + (p - b * rl) * (rx.n / rl);
}

size_t rf_smem(int n) { return (size_t)n * (kRfPitch + 1) * sizeof(double2) + (size_t)n * sizeof(int) + 32 * sizeof(int); }

__device__ __forceinline__ void rf_tables(const LineRadices& rx, const double2* tw_g, double2* tw, int* pos) {
    for (int i = threadIdx.x; i < rx.n; i += kRfThreads) {
        tw[i] = tw_g[i];
        pos[line_freq(rx, i)] = i;
    }
}

// z: rows 64 b .. of term blockIdx.y as 32 complex lines; half spectra (times
// two: the separation of the two rows is not halved) to half[t][row][Hz]
__global__ void __launch_bounds__(kRfThreads) rf_z_kernel(const double* __restrict__ rgrid, double2* __restrict__ half,
                                                          const double2* __restrict__ tw_g,
                                                          const __grid_constant__ LineRadices rx, long rows) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const int n = rx.n, hz = n / 2 + 1;
    double2* buf = reinterpret_cast<double2*>(smem_raw);
    double2* tw = buf + (size_t)n * kRfPitch;
    int* pos = reinterpret_cast<int*>(tw + n);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    rf_tables(rx, tw_g, tw, pos);
    const long row0 = (long)blockIdx.x * 64;
    const double* src = rgrid + (size_t)blockIdx.y * rows * n;
    bool any = false;
    for (int r = w; r < 64; r += kRfThreads / 32) {
        const long row = row0 + r;
        double* d = reinterpret_cast<double*>(buf) + (r & 1);
        for (int z = l; z < n; z += 32) {
            const double v = row < rows ? src[(size_t)row * n + z] : 0.0;
            d[2 * (z * kRfPitch + (r >> 1))] = v;
            any |= v != 0.0;
        }
    }
    // rows the receptor does not reach are zero and stay zero
    if (__syncthreads_or(any)) lines64(buf, rx, tw);
    double2* out = half + (size_t)blockIdx.y * rows * hz;
    for (int i = w; i < 32; i += kRfThreads / 32) {
        const long row = row0 + 2 * i;
        if (row >= rows) break;
        for (int k = l; k < hz; k += 32) {
            const double2 z = buf[(size_t)pos[k] * kRfPitch + i], m = buf[(size_t)pos[k ? n - k : 0] * kRfPitch + i];
            // 2 A = Z[k] + conj(Z[n - k]), 2 B = -i (Z[k] - conj(Z[n - k]))
            out[(size_t)row * hz + k] = make_double2(z.x + m.x, z.y - m.y);
            if (row + 1 < rows) out[(size_t)(row + 1) * hz + k] = make_double2(z.y + m.y, m.x - z.x);
        }
    }
}

// y: lines (x, kz) of half[t][Nx][Ny][Hz], in place
__global__ void __launch_bounds__(kRfThreads) rf_y_kernel(double2* __restrict__ half, const double2* __restrict__ tw_g,
                                                          const __grid_constant__ LineRadices rx, int nx, int hz) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const int n = rx.n;
    double2* buf = reinterpret_cast<double2*>(smem_raw);
    double2* tw = buf + (size_t)n * kRfPitch;
    int* pos = reinterpret_cast<int*>(tw + n);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    rf_tables(rx, tw_g, tw, pos);
    const int L = blockIdx.x * 32 + l;
    const bool ok = L < nx * hz;
    const int x = L / hz;
    double2* line = half + (size_t)blockIdx.y * nx * n * hz + (size_t)x * n * hz + (L - x * hz);
    bool any = false;
    for (int y = w; y < n; y += kRfThreads / 32) {
        const double2 v = ok ? line[(size_t)y * hz] : make_double2(0.0, 0.0);
        buf[(size_t)y * kRfPitch + l] = v;
        any |= v.x != 0.0 || v.y != 0.0;
    }
    if (!__syncthreads_or(any)) return;  // all zero: the lines are their own transforms
    lines64(buf, rx, tw);
    if (ok)
        for (int k = w; k < n; k += kRfThreads / 32) line[(size_t)k * hz] = buf[(size_t)pos[k] * kRfPitch + l];
}

// x: lines p = (ky, kz) of half[t][Nx][Ny Hz]: circulant samples and their
// per-pencil maxima (float bits), then the spectra
template <typename SpecT>
__global__ void __launch_bounds__(kRfThreads) rf_x_kernel(const double2* __restrict__ half,
                                                          const double2* __restrict__ tw_g,
                                                          const __grid_constant__ LineRadices rx, int nh, int pp,
                                                          double spec_scale, double circ_scale,
                                                          SpecT* __restrict__ spec, float2* __restrict__ circ,
                                                          int* __restrict__ cmax) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const int n = rx.n, t = blockIdx.y;
    double2* buf = reinterpret_cast<double2*>(smem_raw);
    double2* tw = buf + (size_t)n * kRfPitch;
    int* pos = reinterpret_cast<int*>(tw + n);
    int* mx = pos + n;  // [32]
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    rf_tables(rx, tw_g, tw, pos);
    if (threadIdx.x < 32) mx[threadIdx.x] = 0;
    const int p0 = blockIdx.x * 32, p = p0 + l;
    const double2* src = half + (size_t)t * n * nh + p;
    for (int x = w; x < n; x += kRfThreads / 32)
        buf[(size_t)x * kRfPitch + l] = p < nh ? src[(size_t)x * nh] : make_double2(0.0, 0.0);
    __syncthreads();
    if (circ) {
        for (int i = w; i < 32 && p0 + i < nh; i += kRfThreads / 32) {
            float m = 0.f;
            float2* dst = circ + ((size_t)t * nh + p0 + i) * n;
            for (int x = l; x < n; x += 32) {
                const double2 v = buf[(size_t)x * kRfPitch + i];
                const float2 c = make_float2((float)(v.x * circ_scale), (float)(-v.y * circ_scale));
                dst[x] = c;
                m = fmaxf(m, fmaxf(fabsf(c.x), fabsf(c.y)));
            }
            for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (l == 0) mx[i] = __float_as_int(m);
        }
        __syncthreads();
        // non-negative floats order as their bits
        if (threadIdx.x < 32 && p0 + (int)threadIdx.x < nh) atomicMax(cmax + p0 + threadIdx.x, mx[threadIdx.x]);
    }
    lines64(buf, rx, tw);
    if (p < pp)
        for (int k = w; k < n; k += kRfThreads / 32) {
            const double2 v = buf[(size_t)pos[k] * kRfPitch + l];
            spec_store(spec + ((size_t)t * n + k) * pp + p, (float)(v.x * spec_scale), (float)(v.y * spec_scale));
        }
}

// per-pencil power-of-two exponent so that the largest circulant component of
// the pencil (over all terms) scales to about 2^13
__global__ void circ_exponent_kernel(const int* __restrict__ cmax, int nh, int8_t* __restrict__ cscale) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nh) return;
    const float m = __int_as_float(cmax[p]);
    int e = 0;
    if (m > 0.f) {
        int ex;
        frexpf(m, &ex);  // m in [2^(ex-1), 2^ex)
        e = 13 - ex;
    }
    cscale[p] = (int8_t)(e < -100 ? -100 : (e > 100 ? 100 : e));
}

}  // namespace

// The half spectra of the terms in flight are work memory that a context keeps
// for the next receptor: at most kRfWork.  Larger term sets are transformed in
// equal chunks of terms, which costs the tails of the launches: 144^3, 18 terms
// (436 MB) 5.29 ms in one chunk, 5.40 in two.
constexpr size_t kRfWork = size_t(512) << 20;
static size_t rf_term_bytes(const int dims[3]) {
    return (size_t)dims[0] * dims[1] * (dims[2] / 2 + 1) * sizeof(double2);
}
static int rf_chunk_terms(const int dims[3], int K) {
    const int most = (int)std::max<size_t>(1, kRfWork / rf_term_bytes(dims)), chunks = (K + most - 1) / most;
    return (K + chunks - 1) / chunks;
}

size_t receptor_fft_work(const int dims[3], int K) { return rf_chunk_terms(dims, K) * rf_term_bytes(dims); }

cudaError_t receptor_fft(const ReceptorFftArgs& a, cudaStream_t s) {
    const int nx = a.dims[0], ny = a.dims[1], nz = a.dims[2], hz = nz / 2 + 1, nh = ny * hz;
    LineRadices px{}, py{}, pz{};
    if (!rf_radices(nx, px) || !rf_radices(ny, py) || !rf_radices(nz, pz)) return cudaErrorInvalidValue;
    const double2* twx = a.tw64;
    const double2* twy = a.shared_tw ? a.tw64 : twx + nx;
    const double2* twz = a.shared_tw ? a.tw64 : twy + ny;
    const long rows = (long)nx * ny;
    // (the z launch leaves every value doubled)
    const double ss = 0.5 / ((double)nx * ny * nz), cs = 0.5 / ((double)ny * nz);
    const auto xb = &rf_x_kernel<__nv_bfloat162>;
    const auto xf = &rf_x_kernel<float2>;
    cudaError_t e;
    if ((e = allow_smem((const void*)rf_z_kernel, rf_smem(nz))) != cudaSuccess) return e;
    if ((e = allow_smem((const void*)rf_y_kernel, rf_smem(ny))) != cudaSuccess) return e;
    if ((e = allow_smem(a.spec_bf16 ? (const void*)xb : (const void*)xf, rf_smem(nx))) != cudaSuccess) return e;
    if (a.circ && (e = cudaMemsetAsync(a.cmax, 0, (size_t)nh * sizeof(int), s)) != cudaSuccess) return e;
    const int chunk = rf_chunk_terms(a.dims, a.K);
    for (int t0 = 0; t0 < a.K; t0 += chunk) {
        const int k = std::min(chunk, a.K - t0);
        rf_z_kernel<<<dim3((unsigned)((rows + 63) / 64), k), kRfThreads, rf_smem(nz), s>>>(
            a.rgrid + (size_t)t0 * rows * nz, a.half, twz, pz, rows);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        rf_y_kernel<<<dim3((nx * hz + 31) / 32, k), kRfThreads, rf_smem(ny), s>>>(a.half, twy, py, nx, hz);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        const dim3 gx((a.pp + 31) / 32, k);
        const size_t spec0 = (size_t)t0 * nx * a.pp;
        float2* circ = a.circ ? a.circ + (size_t)t0 * nh * nx : nullptr;
        if (a.spec_bf16)
            xb<<<gx, kRfThreads, rf_smem(nx), s>>>(a.half, twx, px, nh, a.pp, ss, cs,
                                                   static_cast<__nv_bfloat162*>(a.spec) + spec0, circ, a.cmax);
        else
            xf<<<gx, kRfThreads, rf_smem(nx), s>>>(a.half, twx, px, nh, a.pp, ss, cs,
                                                   static_cast<float2*>(a.spec) + spec0, circ, a.cmax);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    if (a.circ) {
        circ_exponent_kernel<<<(nh + 127) / 128, 128, 0, s>>>(a.cmax, nh, a.cscale);
        e = cudaGetLastError();
    }
    return e;
}

}  // namespace fftdock
