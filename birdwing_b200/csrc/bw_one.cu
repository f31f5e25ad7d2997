// bw_one.cu -- single products in one CTA (k_one).
#include "bw_transform.cuh"

using namespace bw;

cudaError_t bw_launch_one(const bw_plan* pl, const uint32_t* a, const uint32_t* b, uint32_t* out,
                          bool square, uint32_t* err, cudaStream_t s) {
    return with_length<kOneMinLog, kOneMaxLogSingle>(pl->log_n, [&](auto ln) {
        constexpr int LN = decltype(ln)::value;
        using Cfg = OneCfg<Ar32, LN>;
        // both operands of two primes side by side
        constexpr int TH = 4 * Cfg::G < 32 ? 32 : 4 * Cfg::G;
        const cudaError_t e = allow_smem<&k_one<Ar32, LN, 16, TH>>();
        if (e != cudaSuccess) return e;
        k_one<Ar32, LN, 16, TH><<<1, TH, Cfg::smem(pl->K, pl->K), s>>>(
            pl->pd_one, a, (uint32_t)pl->la, b, (uint32_t)pl->lb, out, square ? 1 : 0, err);
        return cudaGetLastError();
    });
}
