// Per-size launchers.  Included by the kernels_nXX.cu translation units, each
// of which instantiates SizeOpsImpl<N> for its grid sizes.
#pragma once

#include "internal.h"
#include "scan_kernels.cuh"
#include "pencil_tc.cuh"
#include "pencil_tcp.cuh"
#include "pencil_lines.cuh"
#include "plane_lines.cuh"

namespace fftdock {

// threads of a cubic edge's plane CTA: about one first-pass butterfly each at
// the small edges.  Measured against 256 threads, ms per 1000 rotations:
// 24^3 0.21 -> 0.14, 32^3 0.26 -> 0.16, 48^3 0.40 -> 0.31, 64^3 planes 0.61 -> 0.51
// (its x-quads: 0.56 -> 0.69, so 256 there).
constexpr int plane_threads(int n, bool quad) { return n <= 16 ? 32 : n <= 32 ? 64 : n <= (quad ? 48 : 64) ? 128 : 256; }

template <int N> struct SizeOpsImpl {
    static constexpr int G = SizeTraits<N>::G;
    static constexpr int H = N / 2 + 1;

    // shared memory of pencil_kernel, and the size limit a ligand is accepted under
    static size_t pencil_smem(int K, int n_ent) {
        return (size_t)PencilTraits<N>::BUFS * N * 32 * sizeof(float2) + (size_t)N * 17 * sizeof(float2) +
               ((size_t)K * N + 1) * sizeof(int32_t) +
               (size_t)n_ent * sizeof(uint32_t);
    }

    static constexpr bool kLinesOneTerm = pencil_lines_one_term(N);

    // the tensor pencil stage: one 128-row x tile up to 128, two up to 256
    static constexpr bool kHasTc = N <= 256;


    template <typename SpecT> static cudaError_t launch_pencil(const BatchArgs& a, int nb, cudaStream_t s) {
        const size_t sm2 = pencil_smem(a.K, a.n_ent);
        cudaError_t e = allow_smem((const void*)pencil_kernel<N, SpecT>, sm2);
        if (e != cudaSuccess) return e;
        dim3 grid2(nb, a.PP / 32);
        pencil_kernel<N, SpecT><<<grid2, 32 * G, sm2, s>>>(static_cast<const SpecT*>(a.spec), a.ent, a.offs, a.tw32,
                                                           a.g2, a.K, a.n_ent);
        return cudaGetLastError();
    }
    // one term, or ljComp's two terms over the same atoms
    template <typename SpecT, bool PAIRED>
    static cudaError_t launch_pencil_lines(const BatchArgs& a, int nb, cudaStream_t s) {
        constexpr int Q = kPencilQ, NT = pencil_threads(N, PAIRED);
        const auto fn = &pencil_lines_kernel<N, SpecT, PAIRED, Q, NT, pencil_ctas(N, PAIRED)>;
        size_t sm = pencil_lines_smem_cubic(N, Q, PAIRED);
        const size_t st = pencil_stage_bytes(N, a.K, Q, a.n_ent, PAIRED);
        const int staged = sm + st <= kPencilMaxSmem ? 1 : 0;
        if (staged) sm += st;
        cudaError_t e = allow_smem((const void*)fn, sm);
        if (e != cudaSuccess) return e;
        const dim3 grid(nb, pencil_grid_y(nb, (N / Q * H + 31) / 32));
        fn<<<grid, NT, sm, s>>>(static_cast<const SpecT*>(a.spec), a.ent, a.ent4, a.offs, a.tw32, a.tw32, a.tw32,
                                LineRadices{}, N, N, N, a.PP, a.K, a.n_ent, staged, a.g2);
        return cudaGetLastError();
    }

    template <bool QUAD>
    static cudaError_t plane(int nb, const float2* src, const BatchArgs& a, float* corr, cudaStream_t s) {
        constexpr int MODE = QUAD ? plane_quad_mode(N, N) : kPlanePlanes;
        constexpr int NT = plane_threads(N, QUAD);
        return launch_planes<MODE>(&plane_lines_kernel<N, MODE, NT>, dim3(N, nb), NT, plane_lines_smem(N, N), s, src,
                                   a.tw32, a.tw32, PlanePlan{}, N, N, a.PP, a.cand_v, a.cand_i, corr);
    }

    // K1 over a.n_rot rotations
    static cudaError_t prep(const BatchArgs& a, cudaStream_t s) {
        const int nb = a.n_rot;
        if (nb <= 0) return cudaSuccess;
        const Geo geo = make_geo(a.h, N, N, N);
        const size_t sm1 = a.offs_stride(N) * sizeof(int32_t) + (size_t)a.n_ent * sizeof(uint32_t);
        cudaError_t e = allow_smem((const void*)ligand_prep_kernel<N>, sm1);
        if (e != cudaSuccess) return e;
        ligand_prep_kernel<N><<<nb, 256, sm1, s>>>(a.rot, a.lig_xyz, a.lig_term, a.n_ent, a.K, geo, a.ent, a.offs,
                                                    a.status, a.lig_w32, a.lig_w32 ? a.ent4 : nullptr, a.ent_idx,
                                                    a.use_tc ? a.ent_t : nullptr, a.tpad, a.n_pad, a.x0,
                                                    a.W, a.classes(), a.tinfo, a.mask_terms());
        return cudaGetLastError();
    }

    // K2 + K3 over a.n_rot rotations (and, on the queue + clustering path,
    // the selection that writes the peaks).  a.ev (optional): events recorded
    // before K2, between K2 and K3, after K3 and after the clustering stage.
    static cudaError_t middle(const BatchArgs& a, cudaStream_t s) {
        const int nb = a.n_rot;
        if (nb <= 0) return cudaSuccess;
        cudaError_t e = cudaSuccess;
        if (a.ev && (e = cudaEventRecord(a.ev[0], s)) != cudaSuccess) return e;
        bool tc = false;
        if constexpr (kHasTc) {
            if (a.use_tc) {
                tc = true;
                constexpr int MT = tc_tiles(N);
                if (MT == 1 && a.tc_pair) {
                    if constexpr (MT == 1) e = launch_pencil_tcp<N>(a, N, N, N, a.tw32, TcBox{}, s);
                    if (e != cudaSuccess) return e;
                } else {
                    const size_t smt = tc_smem_bytes(N, a.W / 8, a.n_tc_terms);
                    if ((e = allow_smem((const void*)pencil_tc_kernel<N, MT>, smt)) != cudaSuccess) return e;
                    dim3 gridt(N * H, (nb + TC_ROT - 1) / TC_ROT);
                    const int tg = a.tc_group > 0 ? a.tc_group : FFTDOCK_TC_TERMS_PER_SUM_DEFAULT;
                    pencil_tc_kernel<N, MT><<<gridt, TC_THREADS, smt, s>>>(a.circ, a.cscale, a.ent_t, a.tinfo,
                                                                          a.n_tc_terms, a.tw32, a.g2t, a.n_pad, nb, a.x0,
                                                                          a.W, tg, a.tc_slots, a.tc_n_slots, TcBox{},
                                                                          a.err);
                    if ((e = cudaGetLastError()) != cudaSuccess) return e;
                }
            }
        }
        if (!tc) {
            if (a.lig_w32) {
                if (a.spec_bf16) return cudaErrorNotSupported;  // weighted sets run with FP32 spectra
                e = launch_pencil_lines<float2, true>(a, nb, s);
            } else if (a.K == 1 && kLinesOneTerm) {
                if constexpr (kLinesOneTerm)
                    e = a.spec_bf16 ? launch_pencil_lines<__nv_bfloat162, false>(a, nb, s)
                                    : launch_pencil_lines<float2, false>(a, nb, s);
            } else {
                e = a.spec_bf16 ? launch_pencil<__nv_bfloat162>(a, nb, s) : launch_pencil<float2>(a, nb, s);
            }
            if (e != cudaSuccess) return e;
        }
        if (a.ev && (e = cudaEventRecord(a.ev[1], s)) != cudaSuccess) return e;
        // K3 (the queue + clustering path also writes every correlation grid)
        float* corr = a.dbg_corr ? a.dbg_corr : a.wide.corr;
        if constexpr (kHasTc) {
            if (tc) e = plane<true>(nb, a.g2t, a, corr, s);  // the tensor stage's x-quads
        }
        if (!tc) e = plane<false>(nb, a.g2, a, corr, s);
        if (e != cudaSuccess) return e;
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        if (a.ev && (e = cudaEventRecord(a.ev[2], s)) != cudaSuccess) return e;
        if (a.wide.corr) {
            BatchArgs w = a;
            w.wide.corr = corr;
            if ((e = wide_select_batch(w, N, s)) != cudaSuccess) return e;
            if (a.ev && (e = cudaEventRecord(a.ev[3], s)) != cudaSuccess) return e;
        }
        return cudaSuccess;
    }

    // K4 over a.n_rot rotations (not on the queue + clustering path)
    static cudaError_t finish(const BatchArgs& a, cudaStream_t s) {
        const int nb = a.n_rot;
        if (nb <= 0 || a.wide.corr) return cudaSuccess;
        finalize_kernel<N><<<nb, 256, 0, s>>>(a.cand_v, a.cand_i, a.ent, a.status, a.rgrid, a.n_ent, a.peak_stride,
                                              a.k_out, a.max_val, a.h, a.first_rot_id, a.peaks, a.n_peaks,
                                              a.pool_v, a.pool_i, a.lig_w64, a.lig_w64 ? a.ent_idx : nullptr);
        return cudaGetLastError();
    }

    // the whole pipeline for one batch (work buffers sized for a.n_rot)
    static cudaError_t scan_batch(const BatchArgs& a, cudaStream_t s) {
        cudaError_t e = prep(a, s);
        if (e != cudaSuccess) return e;
        BatchArgs m = a;
        m.ev = nullptr;
        if ((e = middle(m, s)) != cudaSuccess) return e;
        return finish(a, s);
    }

    // cudaFuncGetAttributes loads a kernel's code under lazy module loading
    static cudaError_t load_fft_form(int spec_bf16) {
        cudaFuncAttributes fa;
        cudaError_t e = cudaFuncGetAttributes(&fa, (const void*)ligand_prep_kernel<N>);
        [[maybe_unused]] constexpr int C = pencil_ctas(N, false);
        if (e == cudaSuccess)
            e = spec_bf16 ? cudaFuncGetAttributes(&fa, (const void*)pencil_kernel<N, __nv_bfloat162>)
                          : cudaFuncGetAttributes(&fa, (const void*)pencil_kernel<N, float2>);
        if constexpr (kLinesOneTerm) {
            if (e == cudaSuccess)
                e = spec_bf16 ? cudaFuncGetAttributes(
                                    &fa, (const void*)pencil_lines_kernel<N, __nv_bfloat162, false, kPencilQ, kPencilThreads, C>)
                              : cudaFuncGetAttributes(&fa,
                                                      (const void*)pencil_lines_kernel<N, float2, false, kPencilQ, kPencilThreads, C>);
        }
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, (const void*)plane_lines_kernel<N, kPlanePlanes, plane_threads(N, false)>);
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, (const void*)finalize_kernel<N>);
        return e;
    }

    static const SizeOps* ops() {
        static const SizeOps o{N, kHasTc, &scan_batch, &pencil_smem, &prep, &middle,
                               &finish, &load_fft_form};
        return &o;
    }
};

}  // namespace fftdock
