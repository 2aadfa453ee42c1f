// Receptor term grids in real space (once per pair, FP64): shape flags,
// per-type desolvation densities mixed into the K folded terms, LJ fields.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "internal.h"
#include "scan_kernels.cuh"

namespace fftdock {
namespace {

// ---------------------------------------------------------------------------
// Receptor builders (once per pair; FP64)
// ---------------------------------------------------------------------------
// Cells of the cropped toLogical(c +- cut) box (project.hpp:87-98).
struct Box {
    int lo[3], hi[3];
};
__device__ __forceinline__ bool projection_box(const double* c, double cut, const Geo& g, Box& b) {
    for (int d = 0; d < 3; ++d) {
        int lo = logical_q(__dsub_rn(c[d], cut), g, d) - 1;
        int hi = logical_q(__dadd_rn(c[d], cut), g, d) - 1;
        b.lo[d] = max(lo, 0);
        b.hi[d] = min(hi, g.n[d] - 1);
        if (b.lo[d] > b.hi[d]) return false;
    }
    return true;
}

__device__ __forceinline__ double dist2(const double* c, int ix, int iy, int iz, const Geo& g) {
    const double dx = __dsub_rn(cell_centre(ix, g, 0), c[0]);
    const double dy = __dsub_rn(cell_centre(iy, g, 1), c[1]);
    const double dz = __dsub_rn(cell_centre(iz, g, 2), c[2]);
    return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

// shape term flags: 2 = core (r^2 <= rc2), 1 = surface (r^2 <= rs2)
__global__ void shape_flags_kernel(const double* __restrict__ xyz, int n, Geo g, double cut, double rc2, double rs2,
                                   int* __restrict__ flags) {
    const int a = blockIdx.x;
    if (a >= n) return;
    const double c[3] = {xyz[3 * a], xyz[3 * a + 1], xyz[3 * a + 2]};
    Box b;
    if (!projection_box(c, cut, g, b)) return;
    const int nx = b.hi[0] - b.lo[0] + 1, ny = b.hi[1] - b.lo[1] + 1, nz = b.hi[2] - b.lo[2] + 1;
    const int tot = nx * ny * nz;
    for (int i = threadIdx.x; i < tot; i += blockDim.x) {
        const int ix = b.lo[0] + i / (ny * nz), iy = b.lo[1] + (i / nz) % ny, iz = b.lo[2] + i % nz;
        const double r2 = dist2(c, ix, iy, iz, g);
        const int f = r2 <= rc2 ? 2 : (r2 <= rs2 ? 1 : 0);
        if (f) atomicMax(&flags[((size_t)ix * g.n[1] + iy) * g.n[2] + iz], f);
    }
}

// each atom's cropped projection box (project.hpp:87-98; empty boxes get
// lo > hi), its rounded coordinates and type
__global__ void atom_cell_kernel(const double* __restrict__ xyz, const int32_t* __restrict__ type, int n, Geo g,
                                 double cut, AtomCell* __restrict__ cells) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= n) return;
    const double c[3] = {xyz[3 * a], xyz[3 * a + 1], xyz[3 * a + 2]};
    Box b;
    const bool ok = projection_box(c, cut, g, b);
    AtomCell o;
    o.x = (float)c[0];
    o.y = (float)c[1];
    o.z = (float)c[2];
    o.type = type ? type[a] : 0;
    for (int d = 0; d < 3; ++d) {
        o.lo[d] = ok ? b.lo[d] : 1;
        o.hi[d] = ok ? b.hi[d] : 0;
    }
    o.pad[0] = o.pad[1] = 0;
    cells[a] = o;
}

// The radial fields are gathered per cell in a fixed bin and atom order (bins
// (bx, by, bz) around the cell ascending, atoms in index order inside a bin),
// so the FP64 sums do not depend on scheduling.  A warp takes a run of up to
// 32 cells of one grid row.  FP64 arithmetic is scarce (two operations per SM
// and clock) and the field of one (atom, cell) pair costs tens of them, so the
// pairs, not the cells, are dealt to the lanes:
//   1. the atoms of the 3 x 3 bin columns around the row are tested 32 at a
//      time (cropped box, FP32 distance with a safe margin) and the passing
//      ones listed in order, each with its chord of cells in the run;
//   2. for every 32 listed atoms the pairs are numbered through a prefix sum
//      and evaluated 32 at a time into shared memory (a pair beyond the cutoff
//      gives zero);
//   3. each lane adds its cell's values in list order.
constexpr int kFieldWarps = 4;

// conservative FP32 margins: rounded coordinates are off by at most 2^-24 of
// the largest one
struct FieldReach {
    float cut2;    // squared distance above which an atom is certainly beyond the cutoff
    float h;
    int max_len;   // cells of the longest chord
};
inline FieldReach field_reach(const Geo& g, double cut) {
    double c = cut;
    for (int d = 0; d < 3; ++d) c = fmax(c, fabs(g.zero_h[d]) + g.h * (g.n[d] + 2) + cut);
    FieldReach r;
    r.cut2 = (float)(cut * cut * (1.0 + 1e-5) + 4e-6 * c * cut);
    r.h = (float)g.h;
    const double len = 2.0 * sqrt((double)r.cut2) / g.h + 4.0;
    r.max_len = len < 32.0 ? (int)len : 32;
    return r;
}

// shared memory of one warp: pair values [NV][32 max_len], pair -> list slot
// [32 max_len], and of 64 listed atoms: atom, first cell | length << 8, offset
template <int NV> __host__ __device__ inline size_t field_warp_bytes(int max_len) {
    return ((size_t)32 * max_len * (8 * NV + 1) + 64 * 4 * 2 + 33 * 4 + 15) / 16 * 16;
}

// value(atom, cell z, r2 clamped to minDist^2, out[NV]) of a pair within the
// cutoff; add(lane's own cell, atom, value[NV]) in list order
template <int NV, class Value, class Add>
__device__ __forceinline__ void gather_fields(unsigned char* smem, const double* __restrict__ xyz,
                                              const AtomCell* __restrict__ cells, const AtomBins& bins, const Geo& g,
                                              const FieldReach& fr, double cut2, double mind2, int ix, int iy, int z0,
                                              int nzr, const Value& value, const Add& add) {
    const int l = threadIdx.x & 31;
    const int cap = 32 * fr.max_len;
    double* val = reinterpret_cast<double*>(smem);           // [NV][cap]
    int* la = reinterpret_cast<int*>(val + NV * cap);        // [64] atom
    int* lc = la + 64;                                       // [64] first | length << 8
    int* lo = lc + 64;                                       // [33] offset of the atom's pairs
    unsigned char* slot = reinterpret_cast<unsigned char*>(lo + 33);  // [cap]
    const float fx = (float)cell_centre(ix, g, 0), fy = (float)cell_centre(iy, g, 1);
    const float fz = (float)cell_centre(z0, g, 2);

    auto process = [&](int cnt) {
        // number the pairs of the first cnt listed atoms
        const int c = l < cnt ? lc[l] : 0;
        const int len = c >> 8;
        int incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (l >= o) incl += t;
        }
        const int off = incl - len, total = __shfl_sync(0xffffffffu, incl, 31);
        lo[l] = off;
        for (int i = 0; i < len; ++i) slot[off + i] = (unsigned char)l;
        __syncwarp();
        for (int p = l; p < total; p += 32) {
            const int sl = slot[p], a = la[sl];
            const int z = z0 + (lc[sl] & 255) + (p - lo[sl]);
            const double ctr[3] = {xyz[3 * a], xyz[3 * a + 1], xyz[3 * a + 2]};
            double r2 = dist2(ctr, ix, iy, z, g);
            double v[NV];
#pragma unroll
            for (int k = 0; k < NV; ++k) v[k] = 0.0;
            if (r2 <= cut2) {
                if (r2 < mind2) r2 = mind2;
                value(a, r2, v);
            }
#pragma unroll
            for (int k = 0; k < NV; ++k) val[k * cap + p] = v[k];
        }
        __syncwarp();
        for (int i = 0; i < cnt; ++i) {
            const int ci = lc[i], d = l - (ci & 255);
            if (d >= 0 && d < (ci >> 8)) {
                double v[NV];
#pragma unroll
                for (int k = 0; k < NV; ++k) v[k] = val[k * cap + lo[i] + d];
                add(la[i], v);
            }
        }
        __syncwarp();
    };

    int b0[3];
    const int ic[3] = {ix, iy, z0};
    for (int d = 0; d < 3; ++d) {
        const double t = floor((cell_centre(ic[d], g, d) - bins.lo[d]) / bins.size);
        b0[d] = t < -2.0 ? -2 : (t > (double)bins.nb[d] + 1.0 ? bins.nb[d] + 1 : (int)t);
    }
    int bz1;  // bin of the run's last cell
    {
        const double t = floor((cell_centre(z0 + nzr - 1, g, 2) - bins.lo[2]) / bins.size);
        bz1 = t < -2.0 ? -2 : (t > (double)bins.nb[2] + 1.0 ? bins.nb[2] + 1 : (int)t);
    }
    const int zb0 = max(b0[2] - 1, 0), zb1 = min(bz1 + 1, bins.nb[2] - 1);
    int listed = 0;
    if (zb0 <= zb1)
        for (int bx = max(b0[0] - 1, 0); bx <= min(b0[0] + 1, bins.nb[0] - 1); ++bx)
            for (int by = max(b0[1] - 1, 0); by <= min(b0[1] + 1, bins.nb[1] - 1); ++by) {
                const int row = (bx * bins.nb[1] + by) * bins.nb[2];
                const int k1 = bins.start[row + zb1 + 1];
                for (int k = bins.start[row + zb0]; k < k1; k += 32) {
                    int first = 0, len = 0, a = 0;
                    if (k + l < k1) {
                        a = bins.atoms[k + l];
                        const float4 f = __ldg(reinterpret_cast<const float4*>(cells + a));
                        const float dx = fx - f.x, dy = fy - f.y;
                        const float left = fr.cut2 - (dx * dx + dy * dy);
                        const AtomCell& c = cells[a];
                        // (a NaN or infinite coordinate has an empty box)
                        if (!(left < 0.f) && ix >= c.lo[0] && ix <= c.hi[0] && iy >= c.lo[1] && iy <= c.hi[1]) {
                            const float half = sqrtf(left) * 1.0001f + 1e-3f * fr.h, dz = f.z - fz;
                            first = max(max((int)ceilf((dz - half) / fr.h - 1e-3f), c.lo[2] - z0), 0);
                            const int last = min(min((int)floorf((dz + half) / fr.h + 1e-3f), c.hi[2] - z0), nzr - 1);
                            len = min(max(last - first + 1, 0), fr.max_len);
                        }
                    }
                    const unsigned m = __ballot_sync(0xffffffffu, len > 0);
                    if (len > 0) {
                        const int at = listed + __popc(m & ((1u << l) - 1u));
                        la[at] = a;
                        lc[at] = first | (len << 8);
                    }
                    listed += __popc(m);
                    __syncwarp();
                    if (listed >= 32) {
                        process(32);
                        listed -= 32;
                        // the rest moves to the front
                        const int ra = l < listed ? la[32 + l] : 0, rc = l < listed ? lc[32 + l] : 0;
                        __syncwarp();
                        if (l < listed) {
                            la[l] = ra;
                            lc[l] = rc;
                        }
                        __syncwarp();
                    }
                }
            }
    if (listed > 0) process(listed);
}

// the run of this warp: row (ix, iy), cells z0 .. z0 + nzr - 1; false past the grid
__device__ __forceinline__ bool field_run(const Geo& g, int& ix, int& iy, int& z0, int& nzr) {
    const int segs = (g.n[2] + 31) / 32;
    const long run = (long)blockIdx.x * kFieldWarps + (threadIdx.x >> 5);
    const long row = run / segs;
    z0 = (int)(run - row * segs) * 32;
    nzr = min(32, g.n[2] - z0);
    ix = (int)(row / g.n[1]);
    iy = (int)(row % g.n[1]);
    return ix < g.n[0];
}

// Shape + desolvation terms R_t = sum_u E[u][t] G_u - S: per-type densities
// G_tau(x) = sum_i g(r) (PotAce::f2, potentials_inc.hpp:394-397; projection as
// project.hpp:143-159: atom i reaches cell x if x lies in i's cropped box and
// r^2 <= cut^2, r^2 clamped to minDist^2) in shared memory, mixed by the warps
// that reached an atom.  96^3, 2500 atoms, 18 types: one thread per cell with
// the densities in global memory and a mix pass over all cells took 3.26 ms.
__global__ void __launch_bounds__(32 * kFieldWarps) ace_terms_kernel(
    const double* __restrict__ xyz, const AtomCell* __restrict__ cells, AtomBins bins, Geo g, FieldReach fr, double cut2,
    double mind2, double ab, double ak, double aa, const int* __restrict__ flags, const double* __restrict__ emat,
    int n_types, double* __restrict__ rgrid) {
    extern __shared__ __align__(16) unsigned char field_smem[];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    double* em = reinterpret_cast<double*>(field_smem);              // [n_types][n_types]
    double* dens = em + n_types * n_types + threadIdx.x;             // [n_types][threads]
    unsigned char* work = reinterpret_cast<unsigned char*>(em + n_types * n_types + n_types * 32 * kFieldWarps) +
                          w * field_warp_bytes<1>(fr.max_len);
    for (int i = threadIdx.x; i < n_types * n_types; i += 32 * kFieldWarps) em[i] = emat[i];
    for (int u = 0; u < n_types; ++u) dens[u * 32 * kFieldWarps] = 0.0;
    __syncthreads();
    int ix, iy, z0, nzr;
    if (!field_run(g, ix, iy, z0, nzr)) return;
    bool hit = false;
    gather_fields<1>(
        work, xyz, cells, bins, g, fr, cut2, mind2, ix, iy, z0, nzr,
        [&](int, double r2, double (&v)[1]) {
            const double r = sqrt(r2);
            v[0] = __ddiv_rn(1.0, __dadd_rn(1.0, exp(__dmul_rn(ab, __dsub_rn(__dmul_rn(ak, r), aa)))));
        },
        [&](int a, const double (&v)[1]) {
            double* dt = dens + cells[a].type * 32 * kFieldWarps;
            *dt = __dadd_rn(*dt, v[0]);
            hit = true;
        });
    const bool any = __ballot_sync(0xffffffffu, hit) != 0u;
    if (l >= nzr) return;
    const size_t V = (size_t)g.n[0] * g.n[1] * g.n[2];
    const size_t cell = ((size_t)ix * g.n[1] + iy) * g.n[2] + z0 + l;
    const int f = flags[cell];
    const double s = f == 2 ? -15.0 : (f == 1 ? 1.0 : 0.0);
    for (int t = 0; t < n_types; ++t) {
        double d = 0.0;
        if (any)
            for (int u = 0; u < n_types; ++u)
                d = __dadd_rn(d, __dmul_rn(em[u * n_types + t], dens[u * 32 * kFieldWarps]));
        rgrid[(size_t)t * V + cell] = __dsub_rn(d, s);
    }
}

// The reference's LJ fields (SoftCoreLJRep / SoftCoreLJAttr for ljComp,
// SoftCoreLJ with the force-shifted cutoff for ljAvg; potentials_inc.hpp:
// 142-354), projected like ProjectorRadialField::projectFields
// (project.hpp:143-176): f2(max(r^2, minDist^2)) of every atom whose cropped
// box holds the cell and with r^2 <= cut^2.  K = 2 (ljComp: repulsion,
// attraction) or 1 (ljAvg).
template <int K>
__global__ void __launch_bounds__(32 * kFieldWarps) lj_field_kernel(
    const double* __restrict__ xyz, const double* __restrict__ lc, const AtomCell* __restrict__ cells, AtomBins bins,
    Geo g, FieldReach fr, double cut2, double mind2, double* __restrict__ rgrid) {
    extern __shared__ __align__(16) unsigned char field_smem[];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    int ix, iy, z0, nzr;
    if (!field_run(g, ix, iy, z0, nzr)) return;
    double acc[K];
#pragma unroll
    for (int k = 0; k < K; ++k) acc[k] = 0.0;
    gather_fields<K>(
        field_smem + w * field_warp_bytes<K>(fr.max_len), xyz, cells, bins, g, fr, cut2, mind2, ix, iy, z0, nzr,
        [&](int a, double r2, double (&v)[K]) {
            const double* p = lc + 5 * a;  // as6, 4es6, 4es12, fshift, gshift
            const double A = __dadd_rn(__dmul_rn(__dmul_rn(r2, r2), r2), p[0]);
            if constexpr (K == 2) {
                v[0] = __ddiv_rn(__ddiv_rn(p[2], A), A);
                v[1] = __ddiv_rn(-p[1], A);
            } else {
                v[0] = __dadd_rn(__dadd_rn(__ddiv_rn(__dsub_rn(__ddiv_rn(p[2], A), p[1]), A), p[3]),
                                 __dmul_rn(p[4], sqrt(r2)));
            }
        },
        [&](int, const double (&v)[K]) {
#pragma unroll
            for (int k = 0; k < K; ++k) acc[k] = __dadd_rn(acc[k], v[k]);
        });
    if (l >= nzr) return;
    const size_t V = (size_t)g.n[0] * g.n[1] * g.n[2];
    const size_t cell = ((size_t)ix * g.n[1] + iy) * g.n[2] + z0 + l;
#pragma unroll
    for (int k = 0; k < K; ++k) rgrid[k * V + cell] = acc[k];
}

// shape alone: R_0 = -S
__global__ void shape_term_kernel(const int* __restrict__ flags, size_t V, double* __restrict__ rgrid) {
    const size_t cell = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (cell >= V) return;
    const int f = flags[cell];
    const double s = f == 2 ? -15.0 : (f == 1 ? 1.0 : 0.0);
    rgrid[cell] = -s;
}

}  // namespace

cudaError_t build_receptor_grids(const ReceptorGridArgs& a, cudaStream_t s) {
    const size_t V = (size_t)a.geo.n[0] * a.geo.n[1] * a.geo.n[2];
    const double md = a.geo.h / 4.0;
    const bool lj = a.term_set == FFTDOCK_TERMS_LJ_COMP || a.term_set == FFTDOCK_TERMS_LJ_AVG;
    const unsigned blocks = (unsigned)((V + 255) / 256);
    cudaError_t e = cudaSuccess;
    if (lj || a.term_set == FFTDOCK_TERMS_SHAPE_ACE) {
        if (a.n > 0) {
            atom_cell_kernel<<<(a.n + 127) / 128, 128, 0, s>>>(a.xyz, a.type, a.n, a.geo, lj ? a.lj_cut : a.ace_cut,
                                                               a.cells);
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
        }
    }
    const long runs = (long)a.geo.n[0] * a.geo.n[1] * ((a.geo.n[2] + 31) / 32);
    const unsigned run_blocks = (unsigned)((runs + kFieldWarps - 1) / kFieldWarps);
    if (lj) {
        const FieldReach fr = field_reach(a.geo, a.lj_cut);
        auto run = [&](auto fn, size_t sm) -> cudaError_t {
            cudaError_t e2 = allow_smem((const void*)fn, sm);
            if (e2 != cudaSuccess) return e2;
            fn<<<run_blocks, 32 * kFieldWarps, sm, s>>>(a.xyz, a.lj_c, a.cells, a.bins, a.geo, fr, a.lj_cut * a.lj_cut,
                                                        md * md, a.rgrid);
            return cudaGetLastError();
        };
        return a.term_set == FFTDOCK_TERMS_LJ_COMP
                   ? run(&lj_field_kernel<2>, kFieldWarps * field_warp_bytes<2>(fr.max_len))
                   : run(&lj_field_kernel<1>, kFieldWarps * field_warp_bytes<1>(fr.max_len));
    }
    if ((e = cudaMemsetAsync(a.flags, 0, V * sizeof(int), s)) != cudaSuccess) return e;
    if (a.n > 0) {
        const double cut = a.shape_core + a.shape_width;
        shape_flags_kernel<<<a.n, 128, 0, s>>>(a.xyz, a.n, a.geo, cut, a.shape_core * a.shape_core, cut * cut,
                                               a.flags);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    if (a.term_set == FFTDOCK_TERMS_SHAPE) {
        shape_term_kernel<<<blocks, 256, 0, s>>>(a.flags, V, a.rgrid);
    } else {
        const FieldReach fr = field_reach(a.geo, a.ace_cut);
        const size_t sm = ((size_t)a.n_types * a.n_types + (size_t)a.n_types * 32 * kFieldWarps) * sizeof(double) +
                          kFieldWarps * field_warp_bytes<1>(fr.max_len);
        if ((e = allow_smem((const void*)ace_terms_kernel, sm)) != cudaSuccess) return e;
        ace_terms_kernel<<<run_blocks, 32 * kFieldWarps, sm, s>>>(a.xyz, a.cells, a.bins, a.geo, fr,
                                                                  a.ace_cut * a.ace_cut, md * md, a.ace_b, a.ace_k,
                                                                  a.ace_a, a.flags, a.emat, a.n_types, a.rgrid);
    }
    return cudaGetLastError();
}

// counting sort of the atoms into bins of edge cut * (1 + 1e-6) (at least
// 1e-3 A), atoms in index order inside each bin
void bin_atoms(const double* xyz, int n, double cut, HostAtomBins& out) {
    out.size = std::max(cut * (1.0 + 1e-6), 1e-3);
    double hi[3] = {0, 0, 0};
    for (int d = 0; d < 3; ++d) out.lo[d] = n > 0 ? xyz[d] : 0.0;
    for (int d = 0; d < 3; ++d) hi[d] = out.lo[d];
    for (int i = 0; i < n; ++i)
        for (int d = 0; d < 3; ++d) {
            out.lo[d] = std::min(out.lo[d], xyz[3 * i + d]);
            hi[d] = std::max(hi[d], xyz[3 * i + d]);
        }
    for (int d = 0; d < 3; ++d) out.nb[d] = (int)std::floor((hi[d] - out.lo[d]) / out.size) + 1;
    const int nbins = out.nb[0] * out.nb[1] * out.nb[2];
    std::vector<int> bin(n);
    out.start.assign(nbins + 1, 0);
    for (int i = 0; i < n; ++i) {
        int b[3];
        for (int d = 0; d < 3; ++d) {
            b[d] = (int)std::floor((xyz[3 * i + d] - out.lo[d]) / out.size);
            b[d] = std::min(std::max(b[d], 0), out.nb[d] - 1);
        }
        bin[i] = (b[0] * out.nb[1] + b[1]) * out.nb[2] + b[2];
        ++out.start[bin[i] + 1];
    }
    for (int k = 0; k < nbins; ++k) out.start[k + 1] += out.start[k];
    out.atoms.assign(n, 0);
    std::vector<int> fill(out.start.begin(), out.start.end() - 1);
    for (int i = 0; i < n; ++i) out.atoms[fill[bin[i]]++] = i;
}

}  // namespace fftdock
