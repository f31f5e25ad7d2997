// bw_transform.cuh -- launches of the transform kernels (K1..K3) of one
// arithmetic, instantiated by one translation unit each (bw_tr_*.cu) so that
// they compile side by side.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "../../include/birdwing.h"
#include "bw_host.h"
#include "bw_internal.h"
#include "bw_ntt.cuh"

namespace bw {

constexpr int kMaxDynSmem = 200 * 1024;

template <class Ar, bool SPLIT16>
int bw_set_transform_attrs() {
    static std::once_flag once;
    static cudaError_t st = cudaSuccess;
    std::call_once(once, [] {
        auto set = [](const void* f) {
            cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 kMaxDynSmem);
            if (e != cudaSuccess) st = e;
        };
        if constexpr (sizeof(typename Ar::T) == 8) {
            if constexpr (!Ar::kF64) {
                set((const void*)k_fwd_col<Ar, SPLIT16, 4, true, false, true>);
                set((const void*)k_fwd_col<Ar, SPLIT16, 4, false, false, true>);
            }
            set((const void*)k_fwd_col<Ar, SPLIT16, 4, true, true, true>);
            set((const void*)k_fwd_col<Ar, SPLIT16, 4, false, true, true>);
        } else {
            set((const void*)k_fwd_col<Ar, SPLIT16, 4, true, !SPLIT16>);
            set((const void*)k_fwd_col<Ar, SPLIT16, 4, false, !SPLIT16>);
        }
        set((const void*)k_inv_col<Ar, 4, true>);
        set((const void*)k_inv_col<Ar, 4, false>);
        set((const void*)k_row<Ar, 64, 4>);
        set((const void*)k_row<Ar, 256, 4>);
        set((const void*)k_row<Ar, 512, 4>);
        set((const void*)k_mid_col<Ar, false>);
        set((const void*)k_mid_col<Ar, true>);
    });
    if (st != cudaSuccess) return bw_fail(BW_ECUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(st));
    return BW_OK;
}


// Raise a kernel's dynamic shared-memory limit once.
template <auto KERN>
cudaError_t allow_smem() {
    static const cudaError_t st = cudaFuncSetAttribute(
        (const void*)KERN, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
    return st;
}

// Calls f(integral_constant<L>) for the runtime length l in [LO, HI].
template <int LO, int HI, class F>
cudaError_t with_length(int l, F f) {
    if constexpr (LO > HI) {
        return cudaErrorInvalidValue;
    } else {
        if (l == LO) return f(std::integral_constant<int, LO>{});
        return with_length<LO + 1, HI>(l, f);
    }
}

// Whether a pass of `ctas` CTAs starts early (launch_after): only with at least
// four waves of them.  A grid that fits the SMs at once is placed on the SMs
// the previous pass leaves first, many CTAs on some and few on others: rows and
// inverse columns started early took a 2^20-point product from 48 to 53 us and
// a 2^17-point one from 23 to 31; with five waves or more it gained 1.5%.
inline bool start_early(size_t ctas, int per_sm) { return ctas >= (size_t)4 * 148 * per_sm; }

template <class Ar>
cudaError_t launch_row2(const bw_plan* pl, const PlanDev<Ar>& pd, typename Ar::T* ra,
                        const typename Ar::T* rb, int sq, bool early, cudaStream_t s) {
    return with_length<kRow2MinLog, kRow2MaxLog>(pl->log_c, [&](auto lc) {
        constexpr int LC = decltype(lc)::value;
        using Cfg = RowCfg<Ar, LC>;
        const cudaError_t e = allow_smem<&k_row2<Ar, LC>>();
        if (e != cudaSuccess) return e;
        const dim3 g(1u << (pl->log_r + pl->log_r2), pl->K);
        early = early && start_early((size_t)g.x * g.y, Cfg::kMinCtas);
        return launch_after(early, k_row2<Ar, LC>, g, Cfg::NT, Cfg::smem(sq != 0), s, pd, ra, rb,
                            sq);
    });
}

// f(integral_constant<log_r>) for a plan's columns.
template <class Ar, class F>
cudaError_t with_columns(int log_r, F f) {
    return with_length<kCol2MinLog, sizeof(typename Ar::T) == 8 ? kCol2MaxLog64 : kCol2MaxLog32>(
        log_r, f);
}

template <class Ar, int CW>
cudaError_t launch_fwd_col2(const bw_plan* pl, const PlanDev<Ar>& pd, const uint32_t* a,
                            size_t na, const uint32_t* b, size_t nb, typename Ar::T* ra,
                            typename Ar::T* rb, unsigned zt, int tile0, int ntiles, bool square,
                            Sum* sums, cudaStream_t s) {
    return with_columns<Ar>(pl->log_r, [&](auto lr) {
        constexpr int LR = decltype(lr)::value;
        using Cfg = ColCfg<Ar, LR>;
        const cudaError_t e = allow_smem<&k_fwd_col2<Ar, LR, CW>>();
        if (e != cudaSuccess) return e;
        const dim3 g((unsigned)ntiles * pl->K, 1, square ? 1 : 2);
        k_fwd_col2<Ar, LR, CW><<<g, Cfg::NT, Cfg::smem, s>>>(pd, a, na, b, nb, ra, rb, zt, tile0,
                                                               sums);
        return cudaSuccess;
    });
}

template <class Ar>
cudaError_t launch_inv_col2(const bw_plan* pl, const PlanDev<Ar>& pd, typename Ar::T* ra,
                            CarryState* cst, int tiles, bool early, cudaStream_t s) {
    return with_columns<Ar>(pl->log_r, [&](auto lr) {
        constexpr int LR = decltype(lr)::value;
        using Cfg = ColCfg<Ar, LR>;
        const cudaError_t e = allow_smem<&k_inv_col2<Ar, LR>>();
        if (e != cudaSuccess) return e;
        early = early && start_early((size_t)tiles * pl->K, Cfg::kMinCtas);
        return launch_after(early, k_inv_col2<Ar, LR>, dim3(tiles, pl->K), Cfg::NT, Cfg::smem, s,
                            pd, ra, cst);
    });
}

// Middle pass of `ops` operands (forward: one or two; inverse: one).
template <class Ar, bool INV>
cudaError_t launch_mid2(const bw_plan* pl, const PlanDev<Ar>& pd, typename Ar::T* ra,
                        typename Ar::T* rb, int ops, cudaStream_t s) {
    return with_length<kMid2MinLog, kMid2MaxLog>(pl->log_r2, [&](auto lr) {
        constexpr int LR = decltype(lr)::value;
        using Cfg = MidCfg<Ar, LR>;
        const cudaError_t e = allow_smem<&k_mid_col2<Ar, LR, INV>>();
        if (e != cudaSuccess) return e;
        const dim3 g(1u << (pl->log_c - pl->log_cb2), 1u << pl->log_r, pl->K * ops);
        k_mid_col2<Ar, LR, INV><<<g, Cfg::NT, Cfg::smem, s>>>(pd, ra, rb);
        return cudaSuccess;
    });
}

// The any-length row pass: rows shorter than 2^5 or longer than 2^13 points, or
// past the 58-bit primes' room.
template <class Ar>
void launch_row(const bw_plan* pl, const PlanDev<Ar>& pd, typename Ar::T* ra,
                const typename Ar::T* rb, int sq, size_t smem, cudaStream_t s) {
    const dim3 g(1u << (pl->log_r + pl->log_r2), pl->K);
    // one thread per sub-problem of a round, 64 to 512 threads (at most 256 on
    // the 32-bit path, so that more than one CTA fits an SM)
    const int want = 1 << (pl->log_c > 4 ? pl->log_c - 4 : 0);
    if (want <= 64) {
        k_row<Ar, 64, 4><<<g, 64, smem, s>>>(pd, ra, rb, sq);
    } else if (want <= 256 || sizeof(typename Ar::T) == 4) {
        k_row<Ar, 256, 4><<<g, 256, smem, s>>>(pd, ra, rb, sq);
    } else {
        k_row<Ar, 512, 4><<<g, 512, smem, s>>>(pd, ra, rb, sq);
    }
}

// Copy words [w0, w1) of every row (row length wc words) of an operand of lx
// words: one 2D copy over the full rows, one plain copy of the partial last
// row's part.  Nothing at or beyond lx is read or written.
inline cudaError_t copy_cols(cudaStream_t s, uint32_t* dst, const uint32_t* src, size_t lx, size_t wc,
                      size_t w0, size_t w1) {
    const size_t full = lx / wc;
    cudaError_t e = cudaSuccess;
    if (full)
        e = cudaMemcpy2DAsync(dst + w0, wc * 4, src + w0, wc * 4, (w1 - w0) * 4, full,
                              cudaMemcpyHostToDevice, s);
    const size_t lo = full * wc + w0, hi = std::min(lx, full * wc + w1);
    if (e == cudaSuccess && hi > lo)
        e = cudaMemcpyAsync(dst + lo, src + lo, (hi - lo) * 4, cudaMemcpyHostToDevice, s);
    return e;
}

// Enqueue K1..K3 (the transform part) for one product.  With io (chunks > 1)
// the operands' copy-in runs on the context's copy stream in column blocks
// and K1 runs block by block behind it.
template <class Ar, bool SPLIT16, bool W64>
int bw_enqueue_transform(bw_ctx* c, const uint32_t* a, const uint32_t* b, bool square,
                      bool timing, const HostIO* io) {
    using T = typename Ar::T;
    const bw_plan* pl = c->plan;
    const PlanDev<Ar>& pd = plan_dev<Ar>(pl);
    if (!pl->v2_cols || !pl->v2_rows || (pl->log_r2 && !pl->v2_mid)) {
        const int rc = bw_set_transform_attrs<Ar, SPLIT16>();
        if (rc) return rc;
    }
    const int R = 1 << pl->log_r, C = 1 << pl->log_c, CB = 1 << pl->log_cb;
    T* ra = reinterpret_cast<T*>(c->d_res_a);
    T* rb = reinterpret_cast<T*>(c->d_res_b);
    const bool ts = pl->tw_smem_r != 0;
    const size_t tw_bytes = ts ? (size_t)R * sizeof(Tw<T>) : 0;

    const int CB1 = 1 << pl->log_cb1;
    // the any-length pass: the 64-bit path stages the coefficients inside the
    // residue tile and runs one prime per CTA (grid.x = tile * K + prime); the
    // 32-bit path keeps a u16 (16-bit) or u64 (64-bit coefficients) copy
    constexpr bool PP = sizeof(T) == 8;
    // (64-bit coefficients on the 32-bit path: the u64 copy holds the loaded
    // rows only, half the tile when both operands fill at most half of it)
    const size_t coef_rows = (W64 && sizeof(T) == 4 && pl->coef_half) ? (size_t)R / 2 : R;
    const size_t smem1 = tw_bytes + tile_elems((size_t)R * CB1) * sizeof(T) +
                         coef_rows * CB1 * (PP ? 0 : SPLIT16 ? 2 : W64 ? 8 : 4) +
                         (W64 && sizeof(T) == 4 ? 16 : 0);
    // K1 takes coefficient counts, or word counts for 64-bit coefficients
    const size_t in_a = W64 ? pl->la : pl->nca, in_b = W64 ? pl->lb : pl->ncb;
    const int cols_outer = 1 << (pl->log_c + pl->log_r2);
    const int tiles1 = cols_outer / CB1;
    const unsigned zt = (pl->zt_a ? 1u : 0u) | (pl->zt_b ? 2u : 0u);
    cudaError_t ke = cudaSuccess;  // a fixed-length launch's status
    auto k1 = [&](int tile0, int ntiles) {
        // (bw_plan_setup: no fixed columns for 64-bit coefficients in 58-bit primes)
        if constexpr (!W64 || !std::is_same<Ar, Ar64>::value) {
            if (pl->v2_cols) {
                ke = launch_fwd_col2<Ar, W64 ? 64 : SPLIT16 ? 16 : 32>(
                    pl, pd, a, in_a, b, in_b, ra, rb, zt, tile0, ntiles, square, c->sums,
                    c->stream);
                return;
            }
        }
        dim3 g1(ntiles * (PP ? pl->K : 1), 1, square ? 1 : 2);
        if (ts) {
            k_fwd_col<Ar, SPLIT16, 4, true, W64, PP><<<g1, kColThreads, smem1, c->stream>>>(
                pd, a, in_a, b, in_b, ra, rb, zt, tile0, c->sums);
        } else {
            k_fwd_col<Ar, SPLIT16, 4, false, W64, PP><<<g1, kColThreads, smem1, c->stream>>>(
                pd, a, in_a, b, in_b, ra, rb, zt, tile0, c->sums);
        }
    };
    if (!io || io->chunks <= 1) {
        k1(0, tiles1);
    } else {
        // the copy stream starts where the context stream is (the previous
        // product has read the staging buffer); block k: copy, event, K1
        // words per row of coefficients: cols / 2 (16-bit), cols (32-bit),
        // 2 cols (64-bit coefficients)
        const int S = io->chunks, per = tiles1 / S, cpw = SPLIT16 ? 2 : 1;
        const size_t wpc = W64 ? 2 : 1;
        const size_t wc = (size_t)cols_outer * wpc / cpw;
        uint32_t* da = const_cast<uint32_t*>(a);
        uint32_t* db = const_cast<uint32_t*>(b);
        BW_CUDA(cudaEventRecord(c->ready_ev, c->stream));
        BW_CUDA(cudaStreamWaitEvent(c->in_stream, c->ready_ev, 0));
        BW_CUDA(io->order->begin(0, c->in_stream));
        BW_CUDA(io->order->begin(1, c->stream));
        for (int k = 0; k < S; ++k) {
            const size_t w0 = ((size_t)k * per << pl->log_cb1) * wpc / cpw;
            const size_t w1 = ((size_t)(k + 1) * per << pl->log_cb1) * wpc / cpw;
            BW_CUDA(copy_cols(c->in_stream, da, io->ha, pl->la, wc, w0, w1));
            if (!square) BW_CUDA(copy_cols(c->in_stream, db, io->hb, pl->lb, wc, w0, w1));
            BW_CUDA(cudaEventRecord(c->in_ev[k], c->in_stream));
            if (k == S - 1) BW_CUDA(io->order->end(0, c->in_stream));
            BW_CUDA(cudaStreamWaitEvent(c->stream, c->in_ev[k], 0));
            k1(k * per, per);
        }
    }
    // three passes: middle column pass with the outer twiddle
    const int CB2 = 1 << pl->log_cb2;
    const size_t smem_mid = (((size_t)1 << pl->log_r2) + CB2) * sizeof(Tw<T>) +
                            tile_elems((size_t)CB2 << pl->log_r2) * sizeof(T);
    if (pl->v2_mid) {
        BW_CUDA(ke);
        BW_CUDA((launch_mid2<Ar, false>(pl, pd, ra, rb, square ? 1 : 2, c->stream)));
    } else if (pl->log_r2) {
        dim3 gm(C / CB2, R, pl->K * (square ? 1 : 2));
        k_mid_col<Ar, false><<<gm, kColThreads, smem_mid, c->stream>>>(pd, ra, rb);
    }
    if (timing) cudaEventRecord(c->ev[2], c->stream);

    const int la = pl->log_c / 2;
    const size_t ntab = 2 * (((size_t)1 << la) + ((size_t)C >> la));
    const size_t smem2 = ntab * sizeof(Tw<T>) + tile_elems(C) * sizeof(T) * (square ? 1 : 2);
    const T* rbs = square ? ra : rb;
    const int sq = square ? 1 : 0;
    BW_CUDA(ke);
    if (pl->v2_rows) {
        BW_CUDA(launch_row2<Ar>(pl, pd, ra, rbs, sq, !timing, c->stream));
    } else {
        launch_row<Ar>(pl, pd, ra, rbs, sq, smem2, c->stream);
    }
    if (timing) cudaEventRecord(c->ev[3], c->stream);

    if (pl->v2_mid) {
        BW_CUDA((launch_mid2<Ar, true>(pl, pd, ra, ra, 1, c->stream)));
    } else if (pl->log_r2) {
        dim3 gm(C / CB2, R, pl->K);
        k_mid_col<Ar, true><<<gm, kColThreads, smem_mid, c->stream>>>(pd, ra, ra);
    }
    const size_t smem3 = tw_bytes + tile_elems((size_t)R * CB) * sizeof(T);
    dim3 g3(cols_outer / CB, pl->K);
    if (pl->v2_cols) {
        BW_CUDA(launch_inv_col2<Ar>(pl, pd, ra, c->cst, cols_outer / CB, !timing, c->stream));
    } else if (ts) {
        k_inv_col<Ar, 4, true><<<g3, kColThreads, smem3, c->stream>>>(pd, ra, c->cst);
    } else {
        k_inv_col<Ar, 4, false><<<g3, kColThreads, smem3, c->stream>>>(pd, ra, c->cst);
    }
    if (timing) cudaEventRecord(c->ev[4], c->stream);
    BW_CUDA(cudaGetLastError());
    return BW_OK;
}

}  // namespace bw
