// bw_group.cuh -- launches of one group of products (batch buckets and serving
// groups) in one arithmetic, instantiated by one translation unit each.
#pragma once
#include "bw_transform.cuh"

using namespace bw;

// Dynamic shared-memory limits of the any-length kernels (once).
template <class Ar, bool SPLIT16>
cudaError_t group_attrs() {
    static const cudaError_t st = [] {
        cudaError_t r = cudaSuccess;
        for (auto f : {(const void*)ks_product<Ar, SPLIT16, 64>,
                       (const void*)ks_product<Ar, SPLIT16, 128>,
                       (const void*)ks_product<Ar, SPLIT16, 256>,
                       (const void*)kb_fwd_col<Ar, SPLIT16, 4>, (const void*)kb_inv_col<Ar, 4>,
                       (const void*)kb_row<Ar, 64, 4>, (const void*)kb_row<Ar, 512, 4>}) {
            const cudaError_t e =
                cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
            if (e != cudaSuccess) r = e;
        }
        return r;
    }();
    return st;
}

// A kernel is loaded at its first use, or here (once) by a query that needs it
// on the device.
template <auto KERN>
cudaError_t load_kernel() {
    static const cudaError_t st = [] {
        cudaFuncAttributes at;
        return cudaFuncGetAttributes(&at, (const void*)KERN);
    }();
    return st;
}
template <auto KERN>
cudaError_t group_kernel(bool load) {
    const cudaError_t e = allow_smem<KERN>();
    return e == cudaSuccess && load ? load_kernel<KERN>() : e;
}

// np = 0: the kernels of the plan's groups are loaded and nothing is launched.
template <class Ar, bool SPLIT16>
cudaError_t bw_enqueue_group_of(const bw_group_launch& g, cudaStream_t s) {
    using T = typename Ar::T;
    const bw_plan& pl = *g.plan;
    const PlanDev<Ar>& P = plan_dev<Ar>(&pl);
    const unsigned np = g.np;
    const bool load = np == 0;
    T* ra = static_cast<T*>(g.res_a);
    T* rb = static_cast<T*>(g.res_b);
    constexpr int CW = SPLIT16 ? 16 : 32;
    if (pl.small && pl.v2_one) {
        return with_length<kOneMinLog, kOneMaxLog>(pl.log_n, [&](auto ln) {
            constexpr int LN = decltype(ln)::value;
            using Cfg = OneCfg<Ar, LN>;
            // one round of both operands of one prime at a time, at most 256
            // threads
            constexpr int TH = 2 * Cfg::G < 32 ? 32 : 2 * Cfg::G > 256 ? 256 : 2 * Cfg::G;
            const cudaError_t e = group_kernel<&kb_one<Ar, LN, CW, TH>>(load);
            if (e != cudaSuccess || load) return e;
            kb_one<Ar, LN, CW, TH><<<np, TH, Cfg::smem(pl.K, 1), s>>>(P, g.d_desc, g.d_err);
            return cudaGetLastError();
        });
    }
    if (pl.small) {
        const cudaError_t ea = group_attrs<Ar, SPLIT16>();
        if (ea != cudaSuccess || load) return ea;
        const int n = 1 << pl.log_n;
        const size_t smem = 2 * tile_elems(n) * sizeof(T);
        const int want = std::min(256, std::max(64, n >> 4));
        if (want >= 256) {
            ks_product<Ar, SPLIT16, 256><<<np, 256, smem, s>>>(P, g.d_desc, ra, g.d_err);
        } else if (want >= 128) {
            ks_product<Ar, SPLIT16, 128><<<np, 128, smem, s>>>(P, g.d_desc, ra, g.d_err);
        } else {
            ks_product<Ar, SPLIT16, 64><<<np, 64, smem, s>>>(P, g.d_desc, ra, g.d_err);
        }
        return cudaGetLastError();
    }
    if (!pl.v2_rows || !pl.v2_cols) {
        const cudaError_t ea = group_attrs<Ar, SPLIT16>();
        if (ea != cudaSuccess) return ea;
    }
    const int R = 1 << pl.log_r, C = 1 << pl.log_c, CB = 1 << pl.log_cb;
    const int CB1 = 1 << pl.log_cb1;
    const size_t smem1 = tile_elems((size_t)R * CB1) * sizeof(T) + (size_t)R * CB1 * (SPLIT16 ? 2 : 4);
    if (pl.v2_cols) {
        const cudaError_t e = with_columns<Ar>(pl.log_r, [&](auto lr) {
            constexpr int LR = decltype(lr)::value;
            using Cfg = ColCfg<Ar, LR>;
            const cudaError_t e1 = group_kernel<&kb_fwd_col2<Ar, LR, CW>>(load);
            if (e1 != cudaSuccess || load) return e1;
            kb_fwd_col2<Ar, LR, CW><<<dim3(C / CB1 * pl.K, 1, 2 * np), Cfg::NT, Cfg::smem, s>>>(
                P, g.d_desc, ra, rb);
            return cudaSuccess;
        });
        if (e != cudaSuccess) return e;
    } else if (!load) {
        kb_fwd_col<Ar, SPLIT16, 4><<<dim3(C / CB1, 1, 2 * np), kColThreads, smem1, s>>>(
            P, g.d_desc, ra, rb);
    }
    const int la = pl.log_c / 2;
    const size_t ntab = 2 * (((size_t)1 << la) + ((size_t)C >> la));
    const size_t smem2 = ntab * sizeof(Tw<T>) + tile_elems(C) * sizeof(T) * 2;
    const dim3 g2(R, pl.K, np);
    if (pl.v2_rows) {
        const cudaError_t e = with_length<kRow2MinLog, kRow2MaxLog>(pl.log_c, [&](auto lc) {
            constexpr int LC = decltype(lc)::value;
            using Cfg = RowCfg<Ar, LC>;
            const cudaError_t e1 = group_kernel<&kb_row2<Ar, LC>>(load);
            if (e1 != cudaSuccess || load) return e1;
            kb_row2<Ar, LC><<<g2, Cfg::NT, Cfg::smem(false), s>>>(P, g.d_desc, ra, rb);
            return cudaSuccess;
        });
        if (e != cudaSuccess) return e;
    } else if (!load && C <= 1024) {
        kb_row<Ar, 64, 4><<<g2, 64, smem2, s>>>(P, g.d_desc, ra, rb);
    } else if (!load) {
        kb_row<Ar, 512, 4><<<g2, 512, smem2, s>>>(P, g.d_desc, ra, rb);
    }
    const size_t smem3 = tile_elems((size_t)R * CB) * sizeof(T);
    if (pl.v2_cols) {
        const cudaError_t e = with_columns<Ar>(pl.log_r, [&](auto lr) {
            constexpr int LR = decltype(lr)::value;
            using Cfg = ColCfg<Ar, LR>;
            const cudaError_t e1 = group_kernel<&kb_inv_col2<Ar, LR>>(load);
            if (e1 != cudaSuccess || load) return e1;
            kb_inv_col2<Ar, LR><<<dim3(C / CB, pl.K, np), Cfg::NT, Cfg::smem, s>>>(P, g.d_desc, ra);
            return cudaSuccess;
        });
        if (e != cudaSuccess) return e;
    } else if (!load) {
        kb_inv_col<Ar, 4><<<dim3(C / CB, pl.K, np), kColThreads, smem3, s>>>(P, g.d_desc, ra);
    }
    if (load) {
        cudaError_t e = load_kernel<&kb_garner_carry<Ar, SPLIT16>>();
        if (e == cudaSuccess) e = load_kernel<&kb_carry_words<Ar, SPLIT16>>();
        return e == cudaSuccess ? load_kernel<&kb_carry_fix>() : e;
    }
    if (g.inject_residue_fault) {
        const cudaError_t e = cudaMemcpyAsync(ra, ra + 1, sizeof(T), cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) return e;
    }
    if (bw_group_lookback(g)) {
        kb_garner_carry<Ar, SPLIT16><<<dim3((unsigned)g.ntiles, np), kCarryThreads, 0, s>>>(
            P, g.d_desc, ra, 1u, g.inject_wait_fault ? 1u + (1u << 27) : 1u, g.d_err,
            g.spin_limit);
    } else {
        kb_carry_words<Ar, SPLIT16><<<dim3((unsigned)g.ntiles, np), kWordsThreads, 0, s>>>(
            P, g.d_desc, ra, g.d_err);
        if (g.ntiles > 1)
            kb_carry_fix<<<dim3(fix_ctas(g.ntiles), np), kFixThreads, 0, s>>>(
                g.d_desc, ((size_t)1 << pl.log_n) / (SPLIT16 ? 2 : 1));
    }
    return cudaGetLastError();
}
