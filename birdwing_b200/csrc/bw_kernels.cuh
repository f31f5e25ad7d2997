// bw_kernels.cuh -- device side of the product pipeline (both prime paths):
// helpers, the passes for any length, Garner and carry.  The common lengths run
// the passes of bw_ntt.cuh, which follow the same scheme.
//
// A product of two operands is computed as a cyclic convolution of length
// n = 2^log_n = R * C per prime with a 4-step NTT (R rows, C columns,
// element (r, c) = coefficient r*C + c):
//
//   K1 fwd_col   per operand, per tile of CB columns: limb split + virtual
//                zero pad, R-point forward NTT down each column, write.
//   K2 row       per prime, per row p (k1 = bitrev(p)): inter-pass twiddle
//                w_n^(c k1) on load, C-point forward NTT of the A row and the
//                B row, pointwise Montgomery product, C-point inverse NTT,
//                inverse twiddle w_n^(-c k1) n^-1 2^bits, write in place.
//   K3 inv_col   per prime, per column tile: R-point inverse NTT down each
//                column, full reduction, write residues in natural order.
//   K4 garner_carry  per tile of 2048 output words: Garner reconstruction of
//                every coefficient from its K residues, carry generation, and
//                carry propagation across tiles by decoupled look-back.
//
// Forward transforms are Cooley-Tukey with natural-order input and
// bit-reversed output; inverse transforms are Gentleman-Sande with
// bit-reversed input and natural output.  Stage s (m = 2^s groups) uses the
// twiddle table entries W[m .. 2m), W[m + i] = w_{2m}^{bitrev_s(i)}.  Each
// round processes up to 2^RLOG elements per thread in registers (radix 8 or
// 16); rounds exchange data through swizzled shared memory.  Stage twiddles
// are read through L1 (the column pass stages them in shared memory when the
// plan asks for it, BW_PLAN_TW_SMEM).  The inter-pass twiddle
// of a row is split as w_n^(c k1) = F[c mod 2^a] G[c >> a] with per-row
// tables F, G (about 2 sqrt(C) entries) built in shared memory at the start
// of K2, their Shoup companions computed on the device.
//
// The reference runs these stages as separate kernels with separate HBM
// passes: zero_pad (src/zero_pad.cu:3-57), GPU-NTT forward/inverse
// (src/gpu_ntt.cu:577-581,742-747), pointwise_mul_kernel
// (src/gpu_ntt.cu:216-238), crt_combine_kernel (src/crt_gpu.cu:157-276) and the
// three carry kernels (src/carry_prop.cu:8-211).
#pragma once
#include <cstdint>
#include <type_traits>
#include "bw_arith.cuh"

namespace bw {

// Primes of a plan: 2 or 3, or 6 on the 32-bit path with 64-bit coefficients.
constexpr int kMaxPrimes = 6;
// Primes the digit-sum Garner (16- and 32-bit coefficients) reads.
constexpr int kDigitPrimes = 3;
constexpr int kCarryThreads = 256;
constexpr int kCarryWordsPerThread = 8;
constexpr int kCarryTileWords = kCarryThreads * kCarryWordsPerThread;  // 2048
constexpr int kColThreads = 256;

// Per-prime device view of a plan.
template <class Ar>
struct PrimeDev {
    using T = typename Ar::T;
    const Tw<T>* WRf;  // column (R-point) forward stage twiddles, R entries
    const Tw<T>* WRi;  // column inverse
    const Tw<T>* WCf;  // row (C-point) forward, C entries
    const Tw<T>* WCi;  // row inverse
    const Tw<T>* TLf;  // row-level twiddle w_m^e for e < 2^lo (m = R_row * C,
    const Tw<T>* THf;  //   R_row the last column length): w_m^(e 2^lo)
    const Tw<T>* TLi;  // w_m^-e
    const Tw<T>* THi;  // w_m^-(e 2^lo) * n^-1 * 2^bits
    const Tw<T>* WMf;  // three-pass schedule: middle (R2-point) stage twiddles
    const Tw<T>* WMi;
    const Tw<T>* OLf;  // three-pass schedule: outer twiddle w_n^e, e < 2^lo_out
    const Tw<T>* OHf;  //   w_n^(e 2^lo_out)
    Ar ar;
    T one_q;           // floor(2^bits / p): Shoup companion of 1 (x mod p)
    Tw<T> scale;       // n^-1 * 2^bits (single-pass transforms of small products)
};

// Garner constants (reference: CRTGarnerParams, include/crt_gpu.h:11-17,
// computed by compute_garner_params, src/crt_gpu.cu:70-105).
template <class Ar>
struct GarnerDev {
    using T = typename Ar::T;
    T inv1, inv1q;      // p0^-1 mod p1
    T p0m2, p0m2q;      // p0 mod p2 (double precision: p0^-1 mod p2)
    T inv2, inv2q;      // (p0 p1)^-1 mod p2 (double precision: p1^-1 mod p2)
    uint64_t p0;        // p0 as an integer
    // 64-bit coefficients (garner_words_w64_at), 32-bit limbs:
    uint32_t m[kMaxPrimes][5];  // M_k = P / p_k, P the product of the primes
    uint32_t np[5];             // 2^160 - P mod 2^160
    uint32_t v[kMaxPrimes];     // six primes: floor(2^61 / p_k)
    double vi[kDigitPrimes];    // three primes: 1 / p_k
    // a product's coefficients stay below this times 2^128 (min(na, nb)); one
    // that reaches it flags an error
    uint64_t top_bound;
};

template <class Ar>
struct PlanDev {
    PrimeDev<Ar> pr[kMaxPrimes];
    GarnerDev<Ar> gar;
    int K;
    int log_n, log_r, log_c, lo;  // lo: split of the row-level twiddle exponent
    int log_cb;                   // outer column tile width CB = 2^log_cb (inverse pass)
    int log_cb1;                  // forward column pass tile width
    int tw_smem_r;                // stage the R-point twiddles in shared memory
    int log_fa;                   // per-row twiddle split a (F has 2^a entries)
    // three-pass schedule (n = R * R2 * C): log_r2 > 0, otherwise 0
    int log_r2, log_cb2, lo_out;
};

// Carry look-back state of one context.
struct CarryState {
    uint32_t counter;   // dynamic tile ticket (reset by K3 before every K4)
    uint32_t any;       // some tile's kind is not kill (k_carry_words; reset by K3)
    uint32_t pad[2];
};

// One product of a batch (device memory).  Residues of product i live at
// element offset res_off of the bucket's residue arenas (K * n elements in
// each of the A and B arenas).
struct BatchProd {
    const uint32_t* a;
    const uint32_t* b;
    uint32_t* out;
    uint32_t la, lb;       // operand words (out receives la + lb words)
    uint32_t square;       // b is a
    uint32_t pad;
    uint64_t res_off;
    CarryState* cst;       // carry look-back state (4-step buckets)
    uint4* rec_x;
    uint32_t* rec_s;
};

// ------------------------------------------------------------------ helpers

// Shared-memory layouts of a tile: element e lives at e + MUL (e >> SH), one
// or two pad slots after every 2^SH elements (1/16 extra either way).  A
// round's sub-problem reads elements E0 + k 2^D (k < 2^RL, the bits of k clear
// of E0's), whose physical indices are p(E0) + p(k 2^D): for D >= SH (and
// D == 0) that is p(E0) + k S with one stride S = 2^D + MUL 2^(D - SH) per
// round, so an access costs one add instead of a swizzle computation; the
// other rounds compute their offsets.  Each kernel's tile is private, so each
// takes the layout whose strides suit its rounds (a model of the warp's
// accesses, bank by bank):
//   LayRow = e + e/16: conflict-free for 8-byte residues at every stride; for
//     4-byte residues one 2-way conflict per warp access at strides >= 32.
//   e + 2 (e/32), 4-byte column tiles (1-8 columns): conflict-free there.
// (An XOR swizzle, conflict-free, measured more ALU work per access in these
// issue-bound kernels.)
template <int SH, int MUL>
struct Lay {
    static __device__ __forceinline__ int p(int e) { return e + MUL * (e >> SH); }
    static __device__ __forceinline__ bool lin(int D) { return D >= SH || D == 0; }
    static __device__ __forceinline__ int stride(int D) {
        return D >= SH ? (1 << D) + MUL * (1 << (D - SH)) : 1;
    }
    // offset of element k of a sub-problem at round stride D: p(k 2^D)
    template <bool LIN>
    static __device__ __forceinline__ int off(int k, int D, int S) {
        return LIN ? k * S : (k << D) + MUL * ((k << D) >> SH);
    }
};
using LayRow = Lay<4, 1>;
template <typename T>
using LayCol = typename std::conditional<sizeof(T) == 4, Lay<5, 2>, Lay<4, 1>>::type;
// Elements of a padded tile of n logical elements (either layout).
__host__ __device__ constexpr size_t tile_elems(size_t n) { return n + (n >> 4); }

__device__ __forceinline__ uint32_t bitrev(uint32_t x, int bits) {
    return bits == 0 ? 0u : (__brev(x) >> (32 - bits));
}

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(uint32_t* p, uint32_t v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Programmatic dependent launch: grid_wait returns once the previous kernel of
// the stream has finished and its writes are visible (at once when this kernel
// was launched without the attribute); grid_release lets the next one start
// when every CTA of this one has called it or exited.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Sums of 32-bit words modulo 2^32 - 1, where a number is congruent to the sum
// of its words: the check of products with 64-bit coefficients, whose primes
// leave no room to see a wrong residue.  K1 sums the operands' words as it loads
// them, K4 the product's digits before the carry is resolved, and the last kernel
// compares: a product that went wrong in between passes with probability 2^-32.
// (By its size alone 98% of wrong coefficients of 2^22-coefficient operands
// pass: three 51-bit primes hold 2^150.03, the coefficients reach 2^150.)  Three
// sums (a, b, c) of kSumSlots partial ones each, which the comparison clears.
// Cost: 2^23 words 754 -> 756 us, 2^21 words (six primes) 184.5 -> 185.5, others
// within the noise.
// A word enters seven times (prime to 2^32 - 1): one wide multiply-add each, on
// a pipe that these kernels leave idle, where a 64-bit addition takes two of the
// instructions that they are short of.
constexpr int kSumSlots = 16;
constexpr uint32_t kSumWeight = 7;
using Sum = unsigned long long;
__device__ __forceinline__ void add_word(uint64_t& acc, uint32_t w) {
    asm("mad.wide.u32 %0, %1, %2, %0;" : "+l"(acc) : "r"(w), "n"(kSumWeight));
}

// A CTA's partial sum, of up to 8 warps: each warp leaves its own (acc: of
// add_word), and after a barrier one warp adds them to a slot.  (One atomic a
// warp on the slots' line took K4 from 0.24 to 0.42 ms at 2^25 words.)
struct SumParts {
    uint2 w[8];
};
__device__ __forceinline__ void sum_part(SumParts& s, uint64_t acc) {
    const uint64_t v = (acc & 0xffffffffu) + (acc >> 32);
    const uint32_t x = (uint32_t)v + (uint32_t)(v >> 32);
    const uint32_t lo = __reduce_add_sync(0xffffffffu, x & 0xffffu);
    const uint32_t hi = __reduce_add_sync(0xffffffffu, x >> 16);
    if ((threadIdx.x & 31) == 0) s.w[threadIdx.x >> 5] = make_uint2(lo, hi);
}
__device__ __forceinline__ void sum_parts(Sum* slots, uint32_t slot, const SumParts& s,
                                          int warps) {
    const int lane = threadIdx.x & 31;
    const uint2 p = lane < warps ? s.w[lane] : make_uint2(0, 0);
    const uint32_t lo = __reduce_add_sync(0xffffffffu, p.x);
    const uint32_t hi = __reduce_add_sync(0xffffffffu, p.y);
    if (lane == 0) atomicAdd(slots + (slot & (kSumSlots - 1)), (Sum)lo + ((Sum)hi << 16));
}

// Compares and clears the sums of one product, by one warp; load: what each lane
// reads of them.
struct SumLanes {
    Sum v[3] = {0, 0, 0};
};
__device__ __forceinline__ SumLanes load_sums(const Sum* sums) {
    SumLanes r;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < 3; ++k)
        if (lane < kSumSlots) r.v[k] = __ldcg(sums + k * kSumSlots + lane);
    return r;
}
__device__ __forceinline__ void check_sums(Sum* sums, SumLanes s, bool square, uint32_t* err) {
    constexpr Sum m = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    // (partial sums stay below 2^59, sixteen of them below 2^63)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (lane < kSumSlots) sums[k * kSumSlots + lane] = 0;
#pragma unroll
        for (int d = kSumSlots / 2; d > 0; d >>= 1) s.v[k] += __shfl_xor_sync(0xffffffffu, s.v[k], d);
        s.v[k] %= m;
    }
    // (7 a) (7 b) = 7 (7 c)
    if (lane == 0 && s.v[0] * (square ? s.v[0] : s.v[1]) % m != kSumWeight * s.v[2] % m)
        atomicOr(err, 2u);
}

// Asynchronous global -> shared copy of one element (cp.async): a tile's
// loads are all issued at once and land while the CTA builds its twiddle
// tables; the issuing thread waits for its own copies with cp_async_wait.
template <typename T>
__device__ __forceinline__ void cp_async_elem(T* smem_dst, const T* gsrc) {
    static_assert(sizeof(T) == 4 || sizeof(T) == 8, "4- or 8-byte elements");
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
    if constexpr (sizeof(T) == 8) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gsrc) : "memory");
    } else {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gsrc) : "memory");
    }
}
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// Round schedule of a 2^log_len-point transform with rounds of up to RLOG
// stages: the remainder round comes first, where the sub-problem stride is
// largest and shared-memory accesses are conflict-free.  Computed
// arithmetically (no arrays, so nothing goes to local memory).
template <int RLOG>
__host__ __device__ __forceinline__ int sched_rounds(int log_len) {
    return (log_len + RLOG - 1) / RLOG;
}
template <int RLOG>
__host__ __device__ __forceinline__ int sched_rl(int log_len, int r) {
    const int rem = log_len % RLOG;
    return (rem && r == 0) ? rem : RLOG;
}
template <int RLOG>
__host__ __device__ __forceinline__ int sched_s0(int log_len, int r) {
    const int rem = log_len % RLOG;
    return rem ? (r == 0 ? 0 : rem + RLOG * (r - 1)) : RLOG * r;
}

// Twiddle load from shared (TS) or global memory.
template <bool TS, typename T>
__device__ __forceinline__ Tw<T> ld_w(const Tw<T>* p) {
    if constexpr (TS) {
        return *p;
    } else {
        return ld_tw(p);
    }
}

// Two consecutive twiddles of 8 bytes each in one 16-byte load (the pair's
// first entry has an even index in a 16-byte-aligned table).
template <bool TS, typename T>
__device__ __forceinline__ void ld_w2(const Tw<T>* p, Tw<T>& a, Tw<T>& b) {
    static_assert(sizeof(Tw<T>) == 8, "8-byte entries");
    if constexpr (sizeof(T) == 8) {
        const double2 v = TS ? *reinterpret_cast<const double2*>(p)
                             : __ldg(reinterpret_cast<const double2*>(p));
        a.w = v.x;
        b.w = v.y;
    } else {
        const uint4 v = TS ? *reinterpret_cast<const uint4*>(p)
                           : __ldg(reinterpret_cast<const uint4*>(p));
        a = Tw<T>{v.x, v.y};
        b = Tw<T>{v.z, v.w};
    }
}

// Forward CT stages s0 .. s0+RL-1 on one sub-problem of 2^RL elements that
// belongs to group g of stage s0.  In the first round of a transform (s0 = 0)
// stage 0 has twiddle 1 and inputs in [0, 2p), so its butterflies need no
// multiply; with zt (first round of a zero-padded column) the second half is
// zero and stage 0 just duplicates the first half.
template <class Ar, int RL, bool TS>
__device__ __forceinline__ void ct_stages(typename Ar::T* x, int s0, int g,
                                          const Tw<typename Ar::T>* __restrict__ W,
                                          const Ar& ar, bool zt) {
    using T = typename Ar::T;
#pragma unroll
    for (int l = 0; l < RL; ++l) {
        const int h = 1 << (RL - l - 1);
        if constexpr (Ar::kF64) {
#pragma unroll
            for (int u = 0; u < (1 << RL); ++u) x[u] = ar.ct_enter(x[u], u, 1 << (RL - 1), l, s0 > 0);
        }
        if (l == 0 && s0 == 0) {
            if (zt) {
#pragma unroll
                for (int u = 0; u < h; ++u) x[u + h] = x[u];
            } else {
#pragma unroll
                for (int u = 0; u < h; ++u) ar.ct1(x[u], x[u + h]);
            }
            continue;
        }
        const Tw<T>* Ws = W + (1 << (s0 + l)) + (g << l);
        if constexpr (sizeof(Tw<T>) == 8) {
            if (l > 0) {
                // the level's 2^l twiddles in pairs
#pragma unroll
                for (int q = 0; q < (1 << l); q += 2) {
                    Tw<T> w[2];
                    ld_w2<TS>(Ws + q, w[0], w[1]);
#pragma unroll
                    for (int e = 0; e < 2; ++e)
#pragma unroll
                        for (int u = 0; u < h; ++u) {
                            const int k = ((q + e) << (RL - l)) + u;
                            ar.ct(x[k], x[k + h], w[e]);
                        }
                }
                continue;
            }
        }
#pragma unroll
        for (int q = 0; q < (1 << l); ++q) {
            const Tw<T> w = ld_w<TS>(Ws + q);
#pragma unroll
            for (int u = 0; u < h; ++u) {
                const int k = (q << (RL - l)) + u;
                ar.ct(x[k], x[k + h], w);
            }
        }
    }
}

// Inverse GS stages s0+RL-1 down to s0 (the mirror of ct_stages); stage 0
// has twiddle 1.
template <class Ar, int RL, bool TS>
__device__ __forceinline__ void gs_stages(typename Ar::T* x, int s0, int g,
                                          const Tw<typename Ar::T>* __restrict__ W,
                                          const Ar& ar) {
    using T = typename Ar::T;
#pragma unroll
    for (int l = RL - 1; l >= 0; --l) {
        const int h = 1 << (RL - l - 1);
        if (l == 0 && s0 == 0) {
#pragma unroll
            for (int u = 0; u < h; ++u) ar.gs1(x[u], x[u + h]);
            continue;
        }
        const Tw<T>* Ws = W + (1 << (s0 + l)) + (g << l);
        if constexpr (sizeof(Tw<T>) == 8) {
            if (l > 0) {
#pragma unroll
                for (int q = 0; q < (1 << l); q += 2) {
                    Tw<T> w[2];
                    ld_w2<TS>(Ws + q, w[0], w[1]);
#pragma unroll
                    for (int e = 0; e < 2; ++e)
#pragma unroll
                        for (int u = 0; u < h; ++u) {
                            const int k = ((q + e) << (RL - l)) + u;
                            if constexpr (Ar::kF64) {
                                if (l == 0 || ((RL - 1 - l) & 1)) {
                                    ar.template gs<true>(x[k], x[k + h], w[e]);
                                } else {
                                    ar.template gs<false>(x[k], x[k + h], w[e]);
                                }
                            } else {
                                ar.gs(x[k], x[k + h], w[e]);
                            }
                        }
                }
                continue;
            }
        }
#pragma unroll
        for (int q = 0; q < (1 << l); ++q) {
            const Tw<T> w = ld_w<TS>(Ws + q);
#pragma unroll
            for (int u = 0; u < h; ++u) {
                const int k = (q << (RL - l)) + u;
                if constexpr (Ar::kF64) {
                    if (l == 0 || ((RL - 1 - l) & 1)) {
                        ar.template gs<true>(x[k], x[k + h], w);
                    } else {
                        ar.template gs<false>(x[k], x[k + h], w);
                    }
                } else {
                    ar.gs(x[k], x[k + h], w);
                }
            }
        }
    }
}

// One round over all sub-problems of a batch of 2^log_cb vectors of length
// 2^log_len.  ld(v, idx, p) / st(v, idx, p, val) move element idx of vector v,
// whose shared-memory tile slot is p (tile element (idx << log_cb) + v in
// layout L).  LIN: the round's stride D = d + log_cb lets the slots advance
// by a fixed stride (L::stride); otherwise each offset is computed (L::off).
// FCB >= 0: the round has stride 1 in the vector (d_log = 0) and the batch
// width is 2^FCB, both known at compile time, so that every slot offset is an
// immediate (a tile's stride-1 round; log_cb is then ignored).
template <class Ar, class L, int RL, bool INV, bool TS, bool LIN, int FCB = -1, class LD,
          class ST>
__device__ __forceinline__ void run_round(int log_len, int log_cb_rt, int s0,
                                          const Tw<typename Ar::T>* __restrict__ W,
                                          const Ar& ar, bool zt, LD ld, ST st) {
    using T = typename Ar::T;
    const int log_cb = FCB >= 0 ? FCB : log_cb_rt;
    const int d_log = FCB >= 0 ? 0 : log_len - s0 - RL;
    const int D = d_log + log_cb;
    const int S = L::stride(D);
    const int nsub = 1 << (log_cb + log_len - RL);
    for (int sp = threadIdx.x; sp < nsub; sp += blockDim.x) {
        const int v = sp & ((1 << log_cb) - 1);
        const int rest = sp >> log_cb;
        const int j = rest & ((1 << d_log) - 1);
        const int g = rest >> d_log;
        const int base = (g << (d_log + RL)) + j;
        const int p0 = L::p((base << log_cb) + v);
        T x[1 << RL];
#pragma unroll
        for (int k = 0; k < (1 << RL); ++k)
            x[k] = ld(v, base + (k << d_log), p0 + L::template off<LIN>(k, D, S));
        if constexpr (!INV) {
            ct_stages<Ar, RL, TS>(x, s0, g, W, ar, zt);
        } else {
            gs_stages<Ar, RL, TS>(x, s0, g, W, ar);
        }
#pragma unroll
        for (int k = 0; k < (1 << RL); ++k)
            st(v, base + (k << d_log), p0 + L::template off<LIN>(k, D, S), x[k]);
    }
}

// Dispatch on the round's radix and addressing: only the remainder round (the
// first round of a transform) is narrower than 2^RLOG, so the full radix has
// one instantiation per call site and the narrow ones stay small.  A round
// whose stride the layout steps through linearly adds one stride per slot; a
// stride-1 round of a tile up to 16 vectors wide gets compile-time offsets;
// the others compute their offsets.
template <class Ar, class L, int RLOG, bool INV, bool TS, class LD, class ST>
__device__ __forceinline__ void run_round_rl(int rl, int log_len, int log_cb, int s0,
                                             const Tw<typename Ar::T>* __restrict__ W,
                                             const Ar& ar, bool zt, LD ld, ST st) {
    const int d_log = log_len - s0 - rl;
    const int D = d_log + log_cb;
    if (rl == RLOG) {
        // (4-byte residues only: on the 64-bit path the extra instantiations
        // measured slower, the inverse column pass 0.231 -> 0.247 ms)
        if constexpr (sizeof(typename Ar::T) == 4) {
            if (d_log == 0 && log_cb <= 4) {
                switch (log_cb) {
                    case 0:
                        run_round<Ar, L, RLOG, INV, TS, false, 0>(log_len, 0, s0, W, ar,
                                                                  zt, ld, st);
                        return;
                    case 1:
                        run_round<Ar, L, RLOG, INV, TS, false, 1>(log_len, 1, s0, W, ar,
                                                                  zt, ld, st);
                        return;
                    case 2:
                        run_round<Ar, L, RLOG, INV, TS, false, 2>(log_len, 2, s0, W, ar,
                                                                  zt, ld, st);
                        return;
                    case 3:
                        run_round<Ar, L, RLOG, INV, TS, false, 3>(log_len, 3, s0, W, ar,
                                                                  zt, ld, st);
                        return;
                    default:
                        run_round<Ar, L, RLOG, INV, TS, false, 4>(log_len, 4, s0, W, ar,
                                                                  zt, ld, st);
                        return;
                }
            }
        }
        if (L::lin(D)) {
            run_round<Ar, L, RLOG, INV, TS, true>(log_len, log_cb, s0, W, ar, zt, ld, st);
        } else {
            run_round<Ar, L, RLOG, INV, TS, false>(log_len, log_cb, s0, W, ar, zt, ld, st);
        }
    } else if (rl == 3) {
        if (L::lin(D)) {
            run_round<Ar, L, 3, INV, TS, true>(log_len, log_cb, s0, W, ar, zt, ld, st);
        } else {
            run_round<Ar, L, 3, INV, TS, false>(log_len, log_cb, s0, W, ar, zt, ld, st);
        }
    } else if (rl == 2) {
        run_round<Ar, L, 2, INV, TS, false>(log_len, log_cb, s0, W, ar, zt, ld, st);
    } else {
        run_round<Ar, L, 1, INV, TS, false>(log_len, log_cb, s0, W, ar, zt, ld, st);
    }
}

// Copy a stage twiddle table (2^log_len entries) into shared memory.
template <typename T>
__device__ __forceinline__ void stage_table(Tw<T>* dst, const Tw<T>* src, int log_len) {
    for (int i = threadIdx.x; i < (1 << log_len); i += blockDim.x) dst[i] = ld_tw(src + i);
}

// ------------------------------------------------------------------ K1
// Forward column pass for one operand (blockIdx.z) and one tile of CB
// columns (tile0 + blockIdx.x: a launch may cover a range of tiles, so that
// the pass runs behind a copy-in split by columns); loops over the K primes
// reusing the loaded
// coefficients.  ncoef = number of coefficients of the operand; the column
// tail beyond it is the virtual zero pad.  zt_mask bit z says operand z has
// all coefficients in the top half of the rows (rows >= R/2 are zero).
// W64 (64-bit path): 64-bit coefficients, two words each; ncoef is then the
// operand's word count (an odd count leaves the last coefficient's high word
// zero), and each coefficient enters the transform reduced to [0, 3p).
// PP (64-bit path): the CTA transforms for one prime, kp0, and stages the
// coefficients straight into its residue tile, where the first round runs in
// place like the others; without PP it loops over the K primes and keeps a
// separate copy of the coefficients, which halves the tile width its shared
// memory allows.
template <class Ar, bool SPLIT16, int RLOG, bool TS, bool W64 = false, bool PP = false>
__device__ __forceinline__ void fwd_col_body(const PlanDev<Ar>& P,
                                             const uint32_t* __restrict__ limbs, size_t ncoef,
                                             typename Ar::T* res, bool zt_in, int tile,
                                             unsigned char* smem_raw, int kp0 = 0,
                                             Sum* sum = nullptr) {
    static_assert(!PP || (!SPLIT16 && sizeof(typename Ar::T) == 8), "PP: 64-bit path");
    using T = typename Ar::T;
    const bool zt = zt_in && P.log_r > 0;
    const int log_r = P.log_r, log_c = P.log_c + P.log_r2, log_cb = P.log_cb1;
    const int R = 1 << log_r, CB = 1 << log_cb;
    const size_t C = (size_t)1 << log_c;  // stride between rows (R2 * C columns)
    const size_t n = (size_t)R * C;
    const int c0 = tile << log_cb;
    const int rows_loaded = zt ? R / 2 : R;
    // staged coefficients: 16-bit halves (32-bit path), 32-bit limbs or
    // 64-bit limb pairs (64-bit path)
    using CT = typename std::conditional<
        SPLIT16, uint16_t, typename std::conditional<W64, uint64_t, uint32_t>::type>::type;

    Tw<T>* tws = reinterpret_cast<Tw<T>*>(smem_raw);         // R entries if TS
    T* buf = reinterpret_cast<T*>(smem_raw + (TS ? (size_t)R * sizeof(Tw<T>) : 0));
    // 64-bit coefficients after a 4-byte residue tile start at the next 16-byte
    // boundary (the tile's 17 (R CB / 16) elements may leave it 4 bytes off)
    size_t coef_off = tile_elems((size_t)R << log_cb) * sizeof(T);
    if constexpr (W64 && sizeof(T) == 4) coef_off = (coef_off + 15) & ~(size_t)15;
    CT* coef = reinterpret_cast<CT*>(reinterpret_cast<unsigned char*>(buf) + coef_off);

    if constexpr (SPLIT16) {
        if (CB >= 2) {
            // whole limbs (two 16-bit coefficients each) by cp.async into the
            // u16 tile: limb e of the tile holds its coefficients 2e and
            // 2e + 1, exactly the little-endian u16 layout the first round
            // reads (CB is even and C is even, so every row segment is whole
            // limbs)
            const int hcb = CB >> 1;
            uint32_t* coef32 = reinterpret_cast<uint32_t*>(coef);
            const size_t nlimbs = (ncoef + 1) >> 1;
            for (int e = threadIdx.x; e < rows_loaded * hcb; e += blockDim.x) {
                const size_t li = ((size_t)(e / hcb) * C + c0) / 2 + (e % hcb);
                if (li < nlimbs) {
                    cp_async_elem(coef32 + e, limbs + li);
                } else {
                    coef32[e] = 0;
                }
            }
        } else {
            for (int e = threadIdx.x; e < (rows_loaded << log_cb); e += blockDim.x) {
                const size_t ci = (size_t)(e >> log_cb) * C + c0 + (e & (CB - 1));
                coef[e] = (CT)(ci < ncoef ? (__ldg(limbs + (ci >> 1)) >> ((ci & 1) * 16)) & 0xFFFFu
                                          : 0u);
            }
        }
    } else if (W64 && PP && (reinterpret_cast<uintptr_t>(limbs) & 7u) == 0) {
        // 64-bit coefficients of an 8-byte-aligned operand: one 8-byte copy
        // each into the residue tile (a lone last word: 4 bytes, high word 0)
        for (int e = threadIdx.x; e < (rows_loaded << log_cb); e += blockDim.x) {
            const size_t wi = 2 * ((size_t)(e >> log_cb) * C + c0 + (e & (CB - 1)));
            T* dst = buf + LayCol<T>::p(e);
            if (wi + 1 < ncoef) {
                cp_async_elem(dst, reinterpret_cast<const T*>(limbs + wi));
            } else if (wi < ncoef) {
                uint32_t* d32 = reinterpret_cast<uint32_t*>(dst);
                cp_async_elem(d32, limbs + wi);
                d32[1] = 0;
            } else {
                *dst = 0;
            }
        }
    } else {
        const bool al8 = (reinterpret_cast<uintptr_t>(limbs) & 7u) == 0;
        for (int e = threadIdx.x; e < (rows_loaded << log_cb); e += blockDim.x) {
            const size_t ci = (size_t)(e >> log_cb) * C + c0 + (e & (CB - 1));
            if constexpr (PP) {
                // into the residue tile at the first round's (swizzled) slot
                uint32_t* dst = reinterpret_cast<uint32_t*>(buf + LayCol<T>::p(e));
                const size_t wi = W64 ? 2 * ci : ci;
                if (wi < ncoef) {
                    cp_async_elem(dst, limbs + wi);
                } else {
                    dst[0] = 0;
                }
                if (W64 && wi + 1 < ncoef) {
                    cp_async_elem(dst + 1, limbs + wi + 1);
                } else {
                    dst[1] = 0;
                }
            } else if constexpr (W64) {
                // one 8-byte copy from an 8-byte-aligned operand, else two
                // 4-byte copies (the operand may start at an odd word)
                uint32_t* dst = reinterpret_cast<uint32_t*>(coef + e);
                const size_t wi = 2 * ci;
                if (al8 && wi + 1 < ncoef) {
                    cp_async_elem(reinterpret_cast<uint64_t*>(dst),
                                  reinterpret_cast<const uint64_t*>(limbs + wi));
                } else {
                    if (wi < ncoef) {
                        cp_async_elem(dst, limbs + wi);
                    } else {
                        dst[0] = 0;
                    }
                    if (wi + 1 < ncoef) {
                        cp_async_elem(dst + 1, limbs + wi + 1);
                    } else {
                        dst[1] = 0;
                    }
                }
            } else {
                // 32-bit limbs land in shared memory without passing registers
                if (ci < ncoef) {
                    cp_async_elem(coef + e, limbs + ci);
                } else {
                    coef[e] = 0;
                }
            }
        }
    }
    cp_async_wait();
    if constexpr (W64) {
        // the words this thread staged, once per operand
        if (!PP || kp0 == 0) {
            uint64_t acc = 0;
            for (int e = threadIdx.x; e < (rows_loaded << log_cb); e += blockDim.x) {
                const uint32_t* w = PP ? reinterpret_cast<const uint32_t*>(buf + LayCol<T>::p(e))
                                       : reinterpret_cast<const uint32_t*>(coef + e);
                add_word(acc, w[0]);
                add_word(acc, w[1]);
            }
            __shared__ SumParts sp;
            sum_part(sp, acc);
            __syncthreads();
            if (threadIdx.x < 32) sum_parts(sum, (uint32_t)tile, sp, kColThreads / 32);
        }
    }

    const int nr = sched_rounds<RLOG>(log_r);
    for (int kp = PP ? kp0 : 0; kp < (PP ? kp0 + 1 : P.K); ++kp) {
        const PrimeDev<Ar>& pr = P.pr[kp];
        const Ar ar = pr.ar;
        T* gout = res + (size_t)kp * n;
        const Tw<T>* W = pr.WRf;
        if constexpr (TS) {
            if (kp > 0) __syncthreads();
            stage_table(tws, pr.WRf, log_r);
            W = tws;
        }
        __syncthreads();
        for (int r = 0; r < nr; ++r) {
            const bool first = (r == 0), last = (r == nr - 1);
            // first round reads the coefficient tile (zero pad virtual), last
            // round writes to global memory
            auto ld = [&](int v, int idx, int p) -> T {
                if (first) {
                    if (zt && idx >= R / 2) return T(0);
                    if constexpr (W64 && sizeof(T) == 4) {
                        // 32-bit path: the staged 64-bit coefficient reduced
                        // to [0, 2p) for this prime
                        return ar.from_u64(coef[(idx << log_cb) + v]);
                    } else {
                        if constexpr (Ar::kF64) {
                            // the staged coefficient's bits as a residue
                            if constexpr (PP && W64) {
                                return ar.from_u64((uint64_t)__double_as_longlong(buf[p]));
                            } else {
                                return ar.from_u32((uint32_t)coef[(idx << log_cb) + v]);
                            }
                        }
                        T x = PP ? buf[p] : (T)coef[(idx << log_cb) + v];
                        if constexpr (W64 && !Ar::kF64) {
                            // a 64-bit coefficient (up to 64p) enters reduced
                            // to [0, 2p), leaving the transform its headroom
                            x = ar.from_u64(x);
                        }
                        return x;
                    }
                }
                return buf[p];
            };
            auto st = [&](int v, int idx, int p, T val) {
                if (last) {
                    gout[(size_t)idx * C + c0 + v] = val;
                } else {
                    buf[p] = val;
                }
            };
            run_round_rl<Ar, LayCol<T>, RLOG, false, TS>(sched_rl<RLOG>(log_r, r), log_r, log_cb,
                                              sched_s0<RLOG>(log_r, r), W, ar, first && zt, ld,
                                              st);
            __syncthreads();
        }
    }
}

// PP (64-bit path): blockIdx.x = tile * K + prime, so the K CTAs of one tile
// are launched next to each other and run together: the first brings the
// tile's operand words into L2 and the others read them from there (with the
// prime as grid.y, the residue writes of the tiles in between evicted them and
// every prime re-read its operands from DRAM).  Three CTAs per SM (at most 85
// registers; the 64-bit kernels then spill 32-80 bytes to the stack): the
// shared-memory tile allows three, and the 2^28-bit product measured K1 4%
// faster than at two (the inverse pass measured slower with the same bound).
template <class Ar, bool SPLIT16, int RLOG, bool TS, bool W64 = false, bool PP = false>
__global__ void __launch_bounds__(kColThreads, 3)
k_fwd_col(const PlanDev<Ar> P, const uint32_t* __restrict__ limbs_a, size_t ncoef_a,
          const uint32_t* __restrict__ limbs_b, size_t ncoef_b, typename Ar::T* res_a,
          typename Ar::T* res_b, unsigned zt_mask, int tile0, Sum* __restrict__ sums) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int op = blockIdx.z;
    fwd_col_body<Ar, SPLIT16, RLOG, TS, W64, PP>(P, op ? limbs_b : limbs_a,
                                                 op ? ncoef_b : ncoef_a, op ? res_b : res_a,
                                                 (zt_mask >> op) & 1u,
                                                 tile0 + (int)(PP ? blockIdx.x / P.K : blockIdx.x),
                                                 smem_raw, PP ? (int)(blockIdx.x % P.K) : 0,
                                                 sums + op * kSumSlots);
}

// batched: blockIdx.z = 2 * product + operand
template <class Ar, bool SPLIT16, int RLOG>
__global__ void __launch_bounds__(kColThreads)
kb_fwd_col(const PlanDev<Ar> P, const BatchProd* __restrict__ D, typename Ar::T* res_a,
           typename Ar::T* res_b) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const BatchProd d = D[blockIdx.z >> 1];
    const int op = blockIdx.z & 1;
    if (op && d.square) return;
    const size_t ncoef = (size_t)(op ? d.lb : d.la) * (SPLIT16 ? 2 : 1);
    const size_t n = (size_t)1 << P.log_n;
    fwd_col_body<Ar, SPLIT16, RLOG, false>(P, op ? d.b : d.a, ncoef,
                                           (op ? res_b : res_a) + d.res_off, ncoef <= n / 2,
                                           blockIdx.x, smem_raw);
}

// ------------------------------------------------------------------ K2
// Per-row twiddle tables: F[i] = w^(i k1), G[j] = w^(j 2^a k1) (forward) and
// the inverse pair with n^-1 2^bits folded into Gi.  w^e comes from the
// plan's two-level tables; each entry's Shoup companion is computed here.
template <class Ar>
__device__ __forceinline__ Tw<typename Ar::T> pow_entry(const Ar& ar, uint64_t e, int lo,
                                                        const Tw<typename Ar::T>* TL,
                                                        const Tw<typename Ar::T>* TH) {
    using T = typename Ar::T;
    const auto a = ld_tw(TL + (e & ((1ull << lo) - 1)));
    const auto b = ld_tw(TH + (e >> lo));
    return ar.mul_tw(a, b);
}

// Fused row pass for row blockIdx.x and prime blockIdx.y: inter-pass twiddle
// on load, forward C-point NTT of both rows, pointwise product, inverse
// C-point NTT, inverse twiddle.  The result overwrites the A row.
// square: B is A.
template <class Ar, int NT, int RLOG>
__device__ __forceinline__ void row_body(const PlanDev<Ar>& P, typename Ar::T* res_a,
                                         const typename Ar::T* res_b, int square, int prow,
                                         int kp, unsigned char* smem_raw) {
    using T = typename Ar::T;
    const int log_c = P.log_c;
    const int C = 1 << log_c;
    const size_t n = (size_t)1 << P.log_n;  // residues per prime
    // rows come in groups of R_row = 2^log_rr: the last column pass's length
    const int log_rr = P.log_r2 ? P.log_r2 : P.log_r;
    const size_t n_row = (size_t)C << log_rr;  // length of the row-level twiddle
    const PrimeDev<Ar>& pr = P.pr[kp];
    const Ar ar = pr.ar;
    T* ga = res_a + (size_t)kp * n + (size_t)prow * C;
    const T* gb = res_b + (size_t)kp * n + (size_t)prow * C;
    const int la = P.log_fa, nf = 1 << la, ng = C >> la;
    Tw<T>* F = reinterpret_cast<Tw<T>*>(smem_raw);
    Tw<T>* G = F + nf;
    Tw<T>* Fi = G + ng;
    Tw<T>* Gi = Fi + nf;
    T* bufA = reinterpret_cast<T*>(Gi + ng);
    T* bufB = bufA + tile_elems(C);

    const uint64_t k1 = bitrev((uint32_t)prow & ((1u << log_rr) - 1), log_rr);
    const uint64_t nmask = n_row - 1;
    // F[i] = w^(i k1), G[j] = w^(j 2^a k1), Fi[i] = w^(-i k1) (forward tables
    // at exponent n - e), Gi[j] = w^(-j 2^a k1) n^-1 2^bits (inverse tables,
    // whose high table carries the scale)
    for (int i = threadIdx.x; i < nf + ng; i += NT) {
        if (i < nf) {
            const uint64_t e = ((uint64_t)i * k1) & nmask;
            F[i] = pow_entry(ar, e, P.lo, pr.TLf, pr.THf);
            Fi[i] = pow_entry(ar, (n_row - e) & nmask, P.lo, pr.TLf, pr.THf);
        } else {
            const uint64_t e = (((uint64_t)(i - nf) << la) * k1) & nmask;
            G[i - nf] = pow_entry(ar, e, P.lo, pr.TLf, pr.THf);
            Gi[i - nf] = pow_entry(ar, e, P.lo, pr.TLi, pr.THi);
        }
    }
    __syncthreads();

    // (loading the rows by cp.async during the table build measured slower:
    // the in-place twiddle then costs one more shared-memory pass)
    for (int i = threadIdx.x; i < C; i += NT) {
        const Tw<T> f = F[i & (nf - 1)], g = G[i >> la];
        bufA[LayRow::p(i)] = ar.mulc(ar.mulc(ga[i], f), g);
        if (!square) bufB[LayRow::p(i)] = ar.mulc(ar.mulc(gb[i], f), g);
    }
    __syncthreads();

    const int nr = sched_rounds<RLOG>(log_c);
    auto ldA = [&](int, int, int p) -> T { return bufA[p]; };
    auto st_glob = [&](int idx, T v) {
        const Tw<T> f = Fi[idx & (nf - 1)], g = Gi[idx >> la];
        ga[idx] = ar.mulc(ar.mulc(v, f), g);
    };

    // forward rounds: A fully (all but the last when squaring), B all but the
    // last (its last round is fused with the product below)
    for (int op = 0; op < (square ? 1 : 2); ++op) {
        T* buf = op ? bufB : bufA;
        const int rounds = (op == 0 && !square) ? nr : nr - 1;
        auto ld = [&](int, int, int p) -> T { return buf[p]; };
        auto st = [&](int, int, int p, T v) { buf[p] = v; };
        for (int r = 0; r < rounds; ++r) {
            run_round_rl<Ar, LayRow, RLOG, false, false>(sched_rl<RLOG>(log_c, r), log_c, 0,
                                                 sched_s0<RLOG>(log_c, r), pr.WCf, ar, false,
                                                 ld, st);
            __syncthreads();
        }
    }

    // fused round: last forward round of B (or A), pointwise product, first
    // inverse round -- one sub-problem stays in registers throughout.  The
    // last round of the schedule has stride 1 (d_log = 0), so the slots of a
    // sub-problem are swz(base) + k.
    {
        const int r = nr - 1;
        const int rl = sched_rl<RLOG>(log_c, r), s0 = sched_s0<RLOG>(log_c, r);
        const int d_log = log_c - s0 - rl;
        const int nsub = 1 << (log_c - rl);
        const bool final_round = (nr == 1);
        T* src = square ? bufA : bufB;
        for (int sp = threadIdx.x; sp < nsub; sp += NT) {
            const int j = sp & ((1 << d_log) - 1);
            const int g = sp >> d_log;
            const int base = (g << (d_log + rl)) + j;
            const int p0 = LayRow::p(base);
            T x[1 << RLOG];
#define BW_FUSED_BODY(RL)                                                              \
    {                                                                                  \
        _Pragma("unroll") for (int k = 0; k < (1 << RL); ++k) x[k] = src[p0 + k];     \
        ct_stages<Ar, RL, false>(x, s0, g, pr.WCf, ar, false);                         \
        _Pragma("unroll") for (int k = 0; k < (1 << RL); ++k) {                        \
            const T xa = ar.fwd_to_2p(x[k]);                                           \
            const T ya = square ? xa : bufA[p0 + k];                                   \
            x[k] = ar.pointwise(ya, xa);                                               \
        }                                                                              \
        gs_stages<Ar, RL, false>(x, s0, g, pr.WCi, ar);                                \
        _Pragma("unroll") for (int k = 0; k < (1 << RL); ++k) {                        \
            if (final_round) st_glob(base + k, x[k]); else bufA[p0 + k] = x[k];        \
        }                                                                              \
    }
            if (rl == RLOG) {
                BW_FUSED_BODY(RLOG)
            } else if (rl == 3) {
                BW_FUSED_BODY(3)
            } else if (rl == 2) {
                BW_FUSED_BODY(2)
            } else {
                BW_FUSED_BODY(1)
            }
#undef BW_FUSED_BODY
        }
        __syncthreads();
    }

    // remaining inverse rounds, the last one writes to global with the twiddle
    for (int r = nr - 2; r >= 0; --r) {
        const bool last = (r == 0);
        auto st = [&](int, int idx, int p, T v) {
            if (last) {
                st_glob(idx, v);
            } else {
                bufA[p] = v;
            }
        };
        run_round_rl<Ar, LayRow, RLOG, true, false>(sched_rl<RLOG>(log_c, r), log_c, 0,
                                            sched_s0<RLOG>(log_c, r), pr.WCi, ar, false, ldA, st);
        __syncthreads();
    }
}

template <class Ar, int NT, int RLOG>
__global__ void __launch_bounds__(NT)
k_row(const PlanDev<Ar> P, typename Ar::T* res_a, const typename Ar::T* res_b, int square) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    row_body<Ar, NT, RLOG>(P, res_a, res_b, square, blockIdx.x, blockIdx.y, smem_raw);
}

// batched: blockIdx.z = product
template <class Ar, int NT, int RLOG>
__global__ void __launch_bounds__(NT)
kb_row(const PlanDev<Ar> P, const BatchProd* __restrict__ D, typename Ar::T* res_a,
       const typename Ar::T* res_b) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const BatchProd d = D[blockIdx.z];
    row_body<Ar, NT, RLOG>(P, res_a + d.res_off, (d.square ? res_a : res_b) + d.res_off,
                           d.square, blockIdx.x, blockIdx.y, smem_raw);
}

// ------------------------------------------------------------------ K1b / K3b
// Middle column pass of the three-pass schedule (n = R * R2 * C).  Sub-matrix
// s (blockIdx.y, k1 = bitrev(s) over R) is the contiguous span
// [s R2 C, (s+1) R2 C) viewed as R2 rows of C; a CTA takes CB2 columns of it
// for one prime and operand (blockIdx.z = operand * K + prime).  Forward: the
// outer twiddle w_n^((i2 C + c) k1) on load, then an R2-point forward NTT.
// Inverse: an R2-point inverse NTT, then w_n^-((i2 C + c) k1) on store.  The
// twiddle is split as w_n^(i2 C k1) * w_n^(c k1), both factors in per-CTA
// tables.
template <class Ar, bool INV>
__global__ void __launch_bounds__(kColThreads)
k_mid_col(const PlanDev<Ar> P, typename Ar::T* res_a, typename Ar::T* res_b) {
    using T = typename Ar::T;
    constexpr int RLOG = 4;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int log_r2 = P.log_r2, log_c = P.log_c, log_cb = P.log_cb2;
    const int R2 = 1 << log_r2, CB = 1 << log_cb;
    const size_t n = (size_t)1 << P.log_n;
    const int s = blockIdx.y;
    const int kp = blockIdx.z % P.K;
    const int op = blockIdx.z / P.K;
    const PrimeDev<Ar>& pr = P.pr[kp];
    const Ar ar = pr.ar;
    T* g = (op ? res_b : res_a) + (size_t)kp * n + ((size_t)s << (log_r2 + log_c));
    const int c0 = blockIdx.x << log_cb;
    Tw<T>* Trow = reinterpret_cast<Tw<T>*>(smem_raw);  // R2 entries
    Tw<T>* Tcol = Trow + R2;                             // CB entries
    T* buf = reinterpret_cast<T*>(Tcol + CB);

    // the tile's loads first: they land while the twiddle tables are built
    for (int e = threadIdx.x; e < (R2 << log_cb); e += blockDim.x)
        cp_async_elem(buf + LayCol<T>::p(e), g + ((size_t)(e >> log_cb) << log_c) + c0 + (e & (CB - 1)));
    const uint64_t k1 = bitrev((uint32_t)s, P.log_r);
    const uint64_t nmask = n - 1;
    for (int i = threadIdx.x; i < R2 + CB; i += blockDim.x) {
        uint64_t e = i < R2 ? (((uint64_t)i << log_c) * k1) & nmask
                            : ((uint64_t)(c0 + i - R2) * k1) & nmask;
        if (INV) e = (n - e) & nmask;
        const Tw<T> t = pow_entry(ar, e, P.lo_out, pr.OLf, pr.OHf);
        if (i < R2) {
            Trow[i] = t;
        } else {
            Tcol[i - R2] = t;
        }
    }
    cp_async_wait();  // this thread's elements
    __syncthreads();

    const int nr = sched_rounds<RLOG>(log_r2);
    if constexpr (!INV) {
        for (int e = threadIdx.x; e < (R2 << log_cb); e += blockDim.x) {
            const int i2 = e >> log_cb, v = e & (CB - 1);
            const Tw<T> a = Tcol[v], b = Trow[i2];
            buf[LayCol<T>::p(e)] = ar.mulc(ar.mulc(buf[LayCol<T>::p(e)], a), b);
        }
        __syncthreads();
        for (int r = 0; r < nr; ++r) {
            const bool last = (r == nr - 1);
            auto ld = [&](int, int, int p) -> T { return buf[p]; };
            auto st = [&](int v, int idx, int p, T val) {
                if (last) {
                    g[((size_t)idx << log_c) + c0 + v] = val;
                } else {
                    buf[p] = val;
                }
            };
            run_round_rl<Ar, LayCol<T>, RLOG, false, false>(sched_rl<RLOG>(log_r2, r), log_r2, log_cb,
                                                 sched_s0<RLOG>(log_r2, r), pr.WMf, ar, false,
                                                 ld, st);
            __syncthreads();
        }
    } else {
        for (int r = nr - 1; r >= 0; --r) {
            const bool last = (r == 0);
            auto ld = [&](int, int, int p) -> T { return buf[p]; };
            auto st = [&](int v, int idx, int p, T val) {
                if (last) {
                    const Tw<T> a = Tcol[v], b = Trow[idx];
                    g[((size_t)idx << log_c) + c0 + v] =
                        ar.mulc(ar.mulc(val, a), b);
                } else {
                    buf[p] = val;
                }
            };
            run_round_rl<Ar, LayCol<T>, RLOG, true, false>(sched_rl<RLOG>(log_r2, r), log_r2, log_cb,
                                                sched_s0<RLOG>(log_r2, r), pr.WMi, ar, false, ld,
                                                st);
            __syncthreads();
        }
    }
}

// ------------------------------------------------------------------ K3
// Inverse column pass for prime blockIdx.y, column tile blockIdx.x.  Writes
// fully reduced residues of the cyclic convolution in natural order, in place.
// Block (0,0) also resets the carry ticket for the K4 launch that follows.
template <class Ar, int RLOG, bool TS>
__device__ __forceinline__ void inv_col_body(const PlanDev<Ar>& P, typename Ar::T* res,
                                             CarryState* cst, int tile, int kp,
                                             unsigned char* smem_raw) {
    using T = typename Ar::T;
    if (tile == 0 && kp == 0 && threadIdx.x == 0) cst->counter = cst->any = 0;
    const int log_r = P.log_r, log_c = P.log_c + P.log_r2, log_cb = P.log_cb;
    const int R = 1 << log_r;
    const size_t C = (size_t)1 << log_c;
    const size_t n = (size_t)R * C;
    const int c0 = tile << log_cb;
    const PrimeDev<Ar>& pr = P.pr[kp];
    const Ar ar = pr.ar;
    T* g = res + (size_t)kp * n;
    Tw<T>* tws = reinterpret_cast<Tw<T>*>(smem_raw);
    T* buf = reinterpret_cast<T*>(smem_raw + (TS ? (size_t)R * sizeof(Tw<T>) : 0));
    const Tw<T>* W = pr.WRi;
    if constexpr (TS) {
        stage_table(tws, pr.WRi, log_r);
        W = tws;
        __syncthreads();
    }

    // the whole tile in flight at once (cp.async), then every round from
    // shared memory; the last round reduces and writes global memory
    for (int e = threadIdx.x; e < (R << log_cb); e += blockDim.x)
        cp_async_elem(buf + LayCol<T>::p(e), g + (size_t)(e >> log_cb) * C + c0 + (e & ((1 << log_cb) - 1)));
    cp_async_wait();
    __syncthreads();

    const int nr = sched_rounds<RLOG>(log_r);
    for (int r = nr - 1; r >= 0; --r) {
        const bool last = (r == 0);
        auto ld = [&](int, int, int p) -> T { return buf[p]; };
        auto st = [&](int v, int idx, int p, T val) {
            if (last) {
                g[(size_t)idx * C + c0 + v] = ar.inv_out(val);
            } else {
                buf[p] = val;
            }
        };
        run_round_rl<Ar, LayCol<T>, RLOG, true, TS>(sched_rl<RLOG>(log_r, r), log_r, log_cb,
                                         sched_s0<RLOG>(log_r, r), W, ar, false, ld, st);
        __syncthreads();
    }
}

template <class Ar, int RLOG, bool TS>
__global__ void __launch_bounds__(kColThreads)
k_inv_col(const PlanDev<Ar> P, typename Ar::T* res, CarryState* cst) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    inv_col_body<Ar, RLOG, TS>(P, res, cst, blockIdx.x, blockIdx.y, smem_raw);
}

// batched: blockIdx.z = product
template <class Ar, int RLOG>
__global__ void __launch_bounds__(kColThreads)
kb_inv_col(const PlanDev<Ar> P, const BatchProd* __restrict__ D, typename Ar::T* res_a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const BatchProd d = D[blockIdx.z];
    inv_col_body<Ar, RLOG, false>(P, res_a + d.res_off, d.cst, blockIdx.x, blockIdx.y,
                                  smem_raw);
}

// ------------------------------------------------------------------ K4
// Garner + carry.  Output word j of the product collects the "digit sum"
// D_j (< 2^96): the coefficient j (32-bit coefficients), or coefficients
// 2j + 2^16 * (2j+1) (16-bit coefficients).  The product is sum D_j 2^(32 j).
//
// Every thread turns its 8 digit sums into 8 words plus a carry-out X
// (< 2^66), computed with carry-in zero.  The true carry into a span of
// words is "X of the span just before it" plus a single bit eps (the sum of
// the words with that carry overflows at most once), and eps obeys
// generate / propagate / kill rules.  So thread- and tile-level carries
// reduce to 1-bit scans: ballots inside a warp, a short loop across warps,
// and a decoupled look-back across tiles.  A tile publishes its carry words
// (the last thread's X) before it waits on anything, then its status, then
// its inclusive eps.  Tiles are claimed in order through an atomic ticket,
// so every tile a CTA waits on is already running.  Every wait is bounded;
// on timeout bit 0 of *err is set and the kernel finishes.  Records are
// written with tag `epoch` and awaited with tag `wait_epoch` (equal except
// under the fault-injection test hook, which makes every wait run out).
//
// Reference: crt_combine_kernel (src/crt_gpu.cu:157-203, 231-276) and the
// three-pass carry (src/carry_prop.cu:8-80) with its host-polled fixup loop
// (src/gpu_ntt.cu:908-924).

// One coefficient below p0 p1 (16- or 32-bit coefficients) from its residues.
// Sets *bad when the redundant third prime disagrees.
template <class Ar>
__device__ __forceinline__ unsigned __int128 garner_one(const PlanDev<Ar>& P, typename Ar::T r0,
                                                        typename Ar::T r1, typename Ar::T r2,
                                                        uint32_t& bad) {
    using T = typename Ar::T;
    const Ar a1 = P.pr[1].ar;
    const GarnerDev<Ar>& G = P.gar;
    if constexpr (Ar::kF64) {
        // k1 = (r1 - r0) p0^-1 mod p1; the residues are integers in doubles
        auto whole = [](double d) {
            return (uint64_t)__double_as_longlong(__dadd_rn(d, 4503599627370496.0)) &
                   0x000fffffffffffffull;
        };
        const double k1 = a1.inv_out(a1.mul(__dsub_rn(r1, r0), G.inv1));
        if (P.K == 3) {
            // the third prime is redundant for every supported size: the
            // mixed-radix digit ((r2 - r0) p0^-1 - k1) p1^-1 mod p2 must be 0,
            // otherwise flag an error
            const Ar a2 = P.pr[2].ar;
            const double t = __dsub_rn(a2.mul(__dsub_rn(r2, r0), G.p0m2), k1);
            bad |= (uint32_t)(a2.mul(t, G.inv2) != 0.0);
        }
        return (unsigned __int128)G.p0 * whole(k1) + whole(r0);
    } else {
        // k1 = (r1 - r0) * p0^-1 mod p1
        const T r0m1 = a1.red1(a1.shoup(r0, 1, P.pr[1].one_q));
        const T t1 = r1 >= r0m1 ? r1 - r0m1 : r1 + a1.p - r0m1;
        const T k1 = a1.red1(a1.shoup(t1, G.inv1, G.inv1q));
        if (P.K == 3) {
            // (as above)
            const Ar a2 = P.pr[2].ar;
            const T r0m2 = a2.red1(a2.shoup(r0, 1, P.pr[2].one_q));
            const T y = a2.red1(r0m2 + a2.red1(a2.shoup(k1, G.p0m2, G.p0m2q)));
            const T t2 = r2 >= y ? r2 - y : r2 + a2.p - y;
            const T k2 = a2.red1(a2.shoup(t2, G.inv2, G.inv2q));
            bad |= (uint32_t)(k2 != 0);
        }
        // (two 30-bit primes: the coefficient fits 64 bits)
        if constexpr (sizeof(T) == 4) return (uint64_t)(uint32_t)G.p0 * k1 + r0;
        return (unsigned __int128)G.p0 * k1 + r0;
    }
}

// Digit sums D[e] < 2^96 of E output words from their coefficients' residues
// r[k] (one coefficient per word, or two 16-bit ones).  Sets *bad when the
// redundant third prime disagrees or a value reaches its bound.
template <class Ar, bool SPLIT16, int E>
__device__ __forceinline__ void garner_combine(
    const PlanDev<Ar>& P, const typename Ar::T (&r)[kDigitPrimes][E * (SPLIT16 ? 2 : 1)],
    unsigned __int128 (&D)[E], uint32_t* bad_out) {
    uint32_t bad = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        if constexpr (SPLIT16) {
            const unsigned __int128 lo = garner_one(P, r[0][2 * e], r[1][2 * e], r[2][2 * e], bad);
            D[e] = lo + (garner_one(P, r[0][2 * e + 1], r[1][2 * e + 1], r[2][2 * e + 1], bad)
                         << 16);
        } else {
            D[e] = garner_one(P, r[0][e], r[1][e], r[2][e], bad);
        }
        // (double precision: the coefficient's own bound, n/2 2^64 -- two 50-bit
        // primes hold 2^100, so the 2^96 that two 58-bit ones leave far behind
        // would let one wrong coefficient in 16 pass)
        if constexpr (Ar::kF64) {
            bad |= (uint32_t)(((uint64_t)(D[e] >> 64) >> (P.log_n - 1)) != 0);
        } else {
            bad |= (uint32_t)((D[e] >> 96) != 0);
        }
    }
    *bad_out |= bad;
}

// Garner reconstruction of the E output words starting at word j0.  Words at
// or beyond NL read nothing and are zero.
// base: this thread's first residue of prime 0; prime k's residues start
// pstride elements later.  valid: the words exist (false: they read as zero).
template <class Ar, bool SPLIT16, int E, bool NC = true>
__device__ __forceinline__ void garner_digits_at(const PlanDev<Ar>& P,
                                                 const typename Ar::T* __restrict__ base,
                                                 size_t pstride, bool valid,
                                                 unsigned __int128 (&D)[E], uint32_t* bad_out) {
    using T = typename Ar::T;
    constexpr int CPW = SPLIT16 ? 2 : 1;
    T r[kDigitPrimes][E * CPW];
#pragma unroll
    for (int kp = 0; kp < kDigitPrimes; ++kp)
#pragma unroll
        for (int q = 0; q < E * CPW; ++q) r[kp][q] = 0;
    if (valid) {
        // 128-bit vector loads of E*CPW consecutive residues per prime
#pragma unroll
        for (int kp = 0; kp < kDigitPrimes; ++kp) {
            if (kp >= P.K) break;
            const uint4* src = reinterpret_cast<const uint4*>(base + (size_t)kp * pstride);
#pragma unroll
            for (int q = 0; q < (E * CPW * (int)sizeof(T)) / 16; ++q) {
                // NC: read-only path (residues from an earlier kernel);
                // L2 loads when this kernel wrote them or started before
                // that one had finished
                const uint4 v = NC ? __ldg(src + q) : __ldcg(src + q);
                if constexpr (Ar::kF64) {
                    r[kp][2 * q] = __hiloint2double((int)v.y, (int)v.x);
                    r[kp][2 * q + 1] = __hiloint2double((int)v.w, (int)v.z);
                } else if constexpr (sizeof(T) == 8) {
                    r[kp][2 * q] = ((uint64_t)v.y << 32) | v.x;
                    r[kp][2 * q + 1] = ((uint64_t)v.w << 32) | v.z;
                } else {
                    r[kp][4 * q] = v.x;
                    r[kp][4 * q + 1] = v.y;
                    r[kp][4 * q + 2] = v.z;
                    r[kp][4 * q + 3] = v.w;
                }
            }
        }
    }
    garner_combine<Ar, SPLIT16, E>(P, r, D, bad_out);
}

template <class Ar, bool SPLIT16, int E, bool NC = true>
__device__ __forceinline__ void garner_digits(const PlanDev<Ar>& P,
                                              const typename Ar::T* __restrict__ res, size_t n,
                                              size_t j0, size_t NL, unsigned __int128 (&D)[E],
                                              uint32_t* bad_out) {
    garner_digits_at<Ar, SPLIT16, E, NC>(P, res + j0 * (SPLIT16 ? 2 : 1), n, j0 < NL, D,
                                         bad_out);
}

// Multi-word additions by carry chains.
// w[0..N] = sum_i col[i] 2^(32 i), col[i] 64 bits
template <int N>
__device__ __forceinline__ void columns_to_words(const uint64_t (&col)[N], uint32_t (&w)[N + 1]) {
    uint32_t h = (uint32_t)(col[0] >> 32);
    w[0] = (uint32_t)col[0];
#pragma unroll
    for (int i = 1; i < N; ++i) {
        const uint32_t lo = (uint32_t)col[i], hi = (uint32_t)(col[i] >> 32);
        asm("add.cc.u32 %0, %2, %3;\n\taddc.u32 %1, %4, 0;"
            : "=&r"(w[i]), "=r"(h)
            : "r"(lo), "r"(h), "r"(hi));
    }
    w[N] = h;
}
// a += b (5 words; the carry out of the last is dropped)
__device__ __forceinline__ void add5(uint32_t (&a)[5], const uint32_t (&b)[5]) {
    asm("add.cc.u32 %0, %0, %5;\n\taddc.cc.u32 %1, %1, %6;\n\taddc.cc.u32 %2, %2, %7;\n\t"
        "addc.cc.u32 %3, %3, %8;\n\taddc.u32 %4, %4, %9;"
        : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4])
        : "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]));
}

// 64-bit coefficients: the E output words from word j0 (j0 even, E/2
// coefficients from coefficient j0/2) and the carry-out X.  The inverse
// transform's scale carries the factor (P / p_k)^-1 mod p_k besides n^-1, so
// the residues are y_k with
//
//   c = sum_k y_k M_k - q P,   M_k = P / p_k,   q = floor(sum_k y_k / p_k)
//
// -- no modular arithmetic is left here (mixed-radix digits took 6 to 15
// modular products in a chain per coefficient: 177 (six primes) to 235 (three)
// instructions, bound by the multiply pipe at 70-83%).  All of it runs modulo
// 2^160, above every coefficient: y_k M_k as columns of 32 x 32-bit products,
// y_k whole (six primes, two sets of columns so that none overflows) or in two
// parts of B bits (two sets, the second shifted by B), and -q P as q (2^160 - P).
// q: c / P stays below 1 - 2^-13 (three primes; 2^-27 for six), so the estimate
// of the sum plus 2^-20 (2^-28) has the right floor.  Coefficients of a product
// stay below min(na, nb) 2^128: a c at or above it flags an error.
// The words are the low 32 E bits of V = sum_q c_q 2^(64 q), X = V >> 32 E
// (< 2^96).  Coefficients at or beyond NL / 2 read nothing and are zero.
template <class Ar, int E, bool NC = true>
__device__ __forceinline__ void garner_words_w64_at(const PlanDev<Ar>& P,
                                                    const typename Ar::T* __restrict__ base,
                                                    size_t pstride, bool valid,
                                                    uint32_t (&l)[E], uint32_t (&X)[3],
                                                    uint32_t* bad_out) {
    using T = typename Ar::T;
    constexpr bool SIX = sizeof(T) == 4;
    constexpr int Q = E / 2, K = SIX ? 6 : 3, ML = SIX ? 5 : 4;
    constexpr int B = Ar::kF64 ? 26 : 29;  // the lower part of a residue
    constexpr int PER = 16 / (int)sizeof(T);
    static_assert(Q % PER == 0, "whole 16-byte loads");
    uint4 raw[K][Q / PER];
#pragma unroll
    for (int kp = 0; kp < K; ++kp) {
        const uint4* src = reinterpret_cast<const uint4*>(base + (size_t)kp * pstride);
#pragma unroll
        for (int h = 0; h < Q / PER; ++h)
            raw[kp][h] = valid ? (NC ? __ldg(src + h) : __ldcg(src + h)) : make_uint4(0, 0, 0, 0);
    }
    const GarnerDev<Ar>& G = P.gar;
    uint32_t bad = 0;
    uint32_t acc[5] = {0, 0, 0, 0, 0};  // running carry (< 2^96)
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        // c0, c1: the two sets' columns
        uint64_t c0[ML] = {}, c1[ML] = {};
        uint32_t quo;
        if constexpr (SIX) {
            uint64_t s61 = 1ull << 33;
#pragma unroll
            for (int kp = 0; kp < K; ++kp) {
                const uint4 v = raw[kp][q / 4];
                const uint32_t y = q % 4 == 0 ? v.x : q % 4 == 1 ? v.y : q % 4 == 2 ? v.z : v.w;
                s61 += (uint64_t)y * G.v[kp];
#pragma unroll
                for (int i = 0; i < ML; ++i) (kp < 4 ? c0 : c1)[i] += (uint64_t)y * G.m[kp][i];
            }
            quo = (uint32_t)(s61 >> 61);
#pragma unroll
            for (int i = 0; i < ML; ++i) c1[i] += (uint64_t)quo * G.np[i];
        } else {
            double sd = 1.0 / (1 << 20) - 0.5;
#pragma unroll
            for (int kp = 0; kp < K; ++kp) {
                const uint4 v = raw[kp][q / 2];
                uint32_t lo = q % 2 == 0 ? v.x : v.z, hi = q % 2 == 0 ? v.y : v.w;
                if constexpr (Ar::kF64) {
                    const double d = __hiloint2double((int)hi, (int)lo);
                    sd = __fma_rn(d, G.vi[kp], sd);
                    // the integer is the low 52 bits of d + 2^52
                    const double z = __dadd_rn(d, 4503599627370496.0);
                    lo = (uint32_t)__double2loint(z);
                    hi = (uint32_t)__double2hiint(z) & 0xfffffu;
                } else {
                    sd = __fma_rn((double)(((uint64_t)hi << 32) | lo), G.vi[kp], sd);
                }
                const uint32_t y0 = lo & ((1u << B) - 1), y1 = __funnelshift_r(lo, hi, B);
#pragma unroll
                for (int i = 0; i < ML; ++i) {
                    c0[i] += (uint64_t)y0 * G.m[kp][i];
                    c1[i] += (uint64_t)y1 * G.m[kp][i];
                }
            }
            // the floor: (sum + 2^-20) - 1/2 rounded to an integer
            quo = (uint32_t)__double2loint(__dadd_rn(sd, 6755399441055744.0));
        }
        uint32_t c[5], d[5];
        if constexpr (SIX) {
            uint32_t w0[6], w1[6];
            columns_to_words<5>(c0, w0);
            columns_to_words<5>(c1, w1);
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                c[i] = w0[i];
                d[i] = w1[i];
            }
        } else {
            uint64_t c0p[5] = {c0[0], c0[1], c0[2], c0[3], 0};
#pragma unroll
            for (int i = 0; i < 5; ++i) c0p[i] += (uint64_t)quo * G.np[i];
            uint32_t w0[6], w1[5];
            columns_to_words<5>(c0p, w0);
            columns_to_words<4>(c1, w1);
            d[0] = w1[0] << B;
#pragma unroll
            for (int i = 1; i < 5; ++i) d[i] = __funnelshift_l(w1[i - 1], w1[i], B);
#pragma unroll
            for (int i = 0; i < 5; ++i) c[i] = w0[i];
        }
        add5(c, d);
        bad |= (uint32_t)(c[4] >= (uint32_t)G.top_bound);
        // add c to the running carry; emit 64 bits; shift
        add5(c, acc);
        l[2 * q] = c[0];
        l[2 * q + 1] = c[1];
        acc[0] = c[2];
        acc[1] = c[3];
        acc[2] = c[4];
    }
    X[0] = acc[0];
    X[1] = acc[1];
    X[2] = acc[2];
    *bad_out |= bad;
}

template <class Ar, int E, bool NC = true>
__device__ __forceinline__ void garner_words_w64(const PlanDev<Ar>& P,
                                                 const typename Ar::T* __restrict__ res,
                                                 size_t n, size_t j0, size_t NL,
                                                 uint32_t (&l)[E], uint32_t (&X)[3],
                                                 uint32_t* bad_out) {
    garner_words_w64_at<Ar, E, NC>(P, res + j0 / 2, n, j0 < NL, l, X, bad_out);
}

// CTA-wide resolution of a 1-bit carry chain.  Each thread has a status
// st: 0 kill, 1 propagate, 2 generate.  chain_prepare publishes per-warp
// aggregates (carry out for carry-in 0 / 1) in s_w and must be followed by a
// __syncthreads(); chain_out gives the CTA carry-out for a carry-in, and
// chain_mine the carry into the calling thread.
struct ChainMasks {
    uint64_t A, B;
};
__device__ __forceinline__ ChainMasks chain_prepare(int st, uint32_t* s_w) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t G = __ballot_sync(0xffffffffu, st == 2);
    const uint32_t Pm = __ballot_sync(0xffffffffu, st == 1);
    ChainMasks m;
    m.A = (uint64_t)(G | Pm);
    m.B = (uint64_t)G;
    if (lane == 0) {
        const uint32_t c0 = (uint32_t)((m.A + m.B) >> 32) & 1u;
        const uint32_t c1 = (uint32_t)((m.A + m.B + 1) >> 32) & 1u;
        s_w[warp] = c0 | (c1 << 1);
    }
    return m;
}
__device__ __forceinline__ uint32_t chain_out(const uint32_t* s_w, uint32_t cin, int nw) {
    uint32_t c = cin;
    for (int w = 0; w < nw; ++w) c = (s_w[w] >> c) & 1u;
    return c;
}
__device__ __forceinline__ uint32_t chain_mine(const ChainMasks& m, const uint32_t* s_w,
                                               uint32_t cin) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t ci = cin;
    for (int w = 0; w < warp; ++w) ci = (s_w[w] >> ci) & 1u;
    const uint64_t S = m.A + m.B + ci;
    const uint32_t carries = (uint32_t)(S ^ m.A ^ m.B);
    return (carries >> lane) & 1u;
}

// Shared memory of one tile's carry resolution.
struct CarryShared {
    uint32_t w[kCarryThreads / 32];
    uint32_t lastx[kCarryThreads / 32][3];
    uint32_t cin[3];
    uint32_t eps;
    SumParts sum;
};

// A thread's share of the product's word sum: its digits S and the carry c out of
// them.  Before the 1-bit carries are resolved, which move a 1 from a word to a
// carry and so leave the sum as it is.
__device__ __forceinline__ uint64_t digit_sum(const uint32_t (&S)[kCarryWordsPerThread],
                                              uint32_t c) {
    uint64_t acc = 0;
#pragma unroll
    for (int e = 0; e < kCarryWordsPerThread; ++e) add_word(acc, S[e]);
    add_word(acc, c);
    return acc;
}

// Tile t's carry, given every thread's 8 words l (digit sums added with
// carry-in zero) and carry-out X: publish the tile's carry words, take the
// predecessor's, resolve the 1-bit carry chain inside the tile, publish the
// tile status and look back across tiles, then write the final words.  Every
// thread of the CTA calls it; it returns after its last barrier.
// sum: where the product's words are summed (SUM).
template <bool SUM>
__device__ __forceinline__ void carry_finish_tile(
    uint32_t t, size_t j0, const uint32_t (&l)[kCarryWordsPerThread], const uint32_t (&X)[3],
    uint32_t* __restrict__ out, size_t M, uint4* __restrict__ rec_x,
    uint32_t* __restrict__ rec_s, uint32_t epoch, uint32_t wait_epoch,
    uint32_t* __restrict__ err, int spin_limit, CarryShared& sh, Sum* sum) {
    constexpr int E = kCarryWordsPerThread;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    // ---- the tile's carry words: the last thread's X, published at once
    // (it depends on nothing outside the tile)
    if (tid == kCarryThreads - 1) {
        uint32_t* rx = reinterpret_cast<uint32_t*>(rec_x + t);
        st_relaxed(rx + 0, X[0]);
        st_relaxed(rx + 1, X[1]);
        st_relaxed(rx + 2, X[2]);
        st_release(rx + 3, epoch);
    }

    // ---- predecessor's carry words: shuffle, shared memory, or (thread 0)
    // the previous tile's record
    uint32_t PX[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) PX[q] = __shfl_up_sync(0xffffffffu, X[q], 1);
    if (lane == 31) {
        sh.lastx[warp][0] = X[0];
        sh.lastx[warp][1] = X[1];
        sh.lastx[warp][2] = X[2];
    }
    if (tid == 0) {
        sh.cin[0] = sh.cin[1] = sh.cin[2] = 0;
        if (t > 0) {
            const uint32_t* rx = reinterpret_cast<const uint32_t*>(rec_x + (t - 1));
            int it = 0;
            bool ok = true;
            while (ld_acquire(rx + 3) != wait_epoch) {
                if (++it > spin_limit) {
                    ok = false;
                    break;
                }
                __nanosleep(32);
            }
            if (ok) {
                sh.cin[0] = ld_relaxed(rx + 0);
                sh.cin[1] = ld_relaxed(rx + 1);
                sh.cin[2] = ld_relaxed(rx + 2);
            } else {
                atomicOr(err, 1u);
            }
        }
    }
    __syncthreads();
    if (lane == 0) {
#pragma unroll
        for (int q = 0; q < 3; ++q) PX[q] = warp > 0 ? sh.lastx[warp - 1][q] : sh.cin[q];
    }

    // ---- S = l + PX and this thread's status
    uint32_t S[E];
    int st;
    {
        uint64_t c = 0;
        uint32_t all = 0xffffffffu;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const uint64_t sum = (uint64_t)l[e] + (e < 3 ? PX[e] : 0u) + c;
            S[e] = (uint32_t)sum;
            c = sum >> 32;
            all &= S[e];
        }
        st = c ? 2 : (all == 0xffffffffu ? 1 : 0);
        if constexpr (SUM) sum_part(sh.sum, digit_sum(S, (uint32_t)c));
    }

    const ChainMasks cm = chain_prepare(st, sh.w);
    __syncthreads();
    if constexpr (SUM) {
        if (warp == kCarryThreads / 32 - 1) sum_parts(sum, t, sh.sum, kCarryThreads / 32);
    }

    // ---- tile status, publish, look back (thread 0)
    if (tid == 0) {
        const uint32_t c0 = chain_out(sh.w, 0u, kCarryThreads / 32),
                       c1 = chain_out(sh.w, 1u, kCarryThreads / 32);
        const uint32_t kind = c0 ? 2u : (c1 ? 1u : 0u);
        const uint32_t tag = epoch << 4;
        uint32_t eps_in = 0;
        if (t > 0) {
            st_release(rec_s + t, tag | kind);
            int j = (int)t - 1;
            int it = 0;
            for (;;) {
                const uint32_t v = ld_acquire(rec_s + j);
                if ((v >> 4) != (wait_epoch & 0x0fffffffu)) {
                    if (++it > spin_limit) {
                        atomicOr(err, 1u);
                        eps_in = 0;
                        break;
                    }
                    __nanosleep(32);
                    continue;
                }
                if (v & 8u) {
                    eps_in = (v >> 2) & 1u;
                    break;
                }
                const uint32_t k = v & 3u;
                if (k != 1u || j == 0) {
                    eps_in = (k == 2u) ? 1u : 0u;
                    break;
                }
                --j;
            }
        }
        const uint32_t eps_out = kind == 2u ? 1u : (kind == 1u ? eps_in : 0u);
        st_release(rec_s + t, tag | 8u | (eps_out << 2) | kind);
        sh.eps = eps_in;
    }
    __syncthreads();

    // ---- final words
    const uint32_t mc = chain_mine(cm, sh.w, sh.eps);
    uint32_t w[E];
    {
        uint64_t c = mc;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const uint64_t sum = (uint64_t)S[e] + c;
            w[e] = (uint32_t)sum;
            c = sum >> 32;
        }
    }
    if (j0 + E <= M && ((reinterpret_cast<uintptr_t>(out + j0) & 15u) == 0)) {
        uint4* o = reinterpret_cast<uint4*>(out + j0);
        o[0] = make_uint4(w[0], w[1], w[2], w[3]);
        o[1] = make_uint4(w[4], w[5], w[6], w[7]);
    } else {
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (j0 + e < M) out[j0 + e] = w[e];
    }
}

// Words l and carry-out X of E = 8 output words from digit sums (16- and
// 32-bit coefficients) or full coefficients (64-bit), read from `base` (this
// thread's first residue of prime 0, primes pstride apart; global memory or a
// shared-memory tile).
template <class Ar, bool SPLIT16, bool W64, bool NC>
__device__ __forceinline__ void garner_local(const PlanDev<Ar>& P,
                                             const typename Ar::T* __restrict__ base,
                                             size_t pstride, bool valid,
                                             uint32_t (&l)[kCarryWordsPerThread],
                                             uint32_t (&X)[3], uint32_t* bad) {
    constexpr int E = kCarryWordsPerThread;
    if constexpr (W64) {
        garner_words_w64_at<Ar, E, NC>(P, base, pstride, valid, l, X, bad);
    } else {
        unsigned __int128 D[E];
        garner_digits_at<Ar, SPLIT16, E, NC>(P, base, pstride, valid, D, bad);
        unsigned __int128 acc = 0;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            acc += D[e];
            l[e] = (uint32_t)acc;
            acc >>= 32;
        }
        X[0] = (uint32_t)acc;
        X[1] = (uint32_t)(acc >> 32);
        X[2] = (uint32_t)(acc >> 64);
    }
}

// Residue elements of one word of output: two 16-bit coefficients, one 32-bit
// coefficient, or half a 64-bit coefficient.
template <bool SPLIT16, bool W64>
__host__ __device__ constexpr size_t elems_per_word2() {
    return SPLIT16 ? 4 : W64 ? 1 : 2;  // in halves: x2 of the element count
}

template <class Ar, bool SPLIT16, bool W64 = false>
__device__ __forceinline__ void garner_carry_body(
    const PlanDev<Ar>& P, const typename Ar::T* __restrict__ res, uint32_t* __restrict__ out,
    size_t M, size_t NL, CarryState* cst, uint4* __restrict__ rec_x,
    uint32_t* __restrict__ rec_s, uint32_t epoch, uint32_t wait_epoch,
    uint32_t* __restrict__ err, int spin_limit, Sum* sum) {
    constexpr int E = kCarryWordsPerThread;
    constexpr int TL = kCarryTileWords;
    __shared__ uint32_t s_tile;
    __shared__ CarryShared sh;

    const int tid = threadIdx.x;
    if (tid == 0) s_tile = atomicAdd(&cst->counter, 1u);
    __syncthreads();
    const uint32_t t = s_tile;
    const size_t j0 = (size_t)t * TL + (size_t)tid * E;
    const size_t n = (size_t)1 << P.log_n;

    uint32_t l[E];
    uint32_t X[3];
    uint32_t bad = 0;
    garner_local<Ar, SPLIT16, W64, true>(P, res + j0 * elems_per_word2<SPLIT16, W64>() / 2, n,
                                         j0 < NL, l, X, &bad);
    if (bad) atomicOr(err, 2u);
    carry_finish_tile<W64>(t, j0, l, X, out, M, rec_x, rec_s, epoch, wait_epoch, err, spin_limit,
                           sh, sum);
}

// K4 without waits (single products).  The look-back form above keeps every
// CTA of a tile waiting on its predecessor's records: two or three dependent
// L2 round trips per tile with the whole CTA at a barrier.  Here a ninth warp
// computes the carry words X into the tile itself, from the eight words before
// it (a pre-pass kernel for them took 4 us); the 1-bit tile carry is left out
// of the words pass: tile t writes its words as if the carry bit eps into it
// were 0 and records its kind -- the carry bit it passes on for eps = 0 and for
// eps = 1 (kill: 0/0, propagate: 0/1, generate: 1/1).  Where any tile is not
// kill, k_carry_fix scans the kinds (eps into tile 0 is 0) and adds 1 at the
// first word of each tile whose eps is 1, rippling inside the tile (a tile that
// propagates passes the carry on through the next tile's own eps).  For
// operands of random words every tile but an all-ones span kills, and it
// returns at once.  (Letting the tile that finishes last do the fix saves the
// launch, but every tile's arrival then waits for its words to be visible:
// 72 -> 92 us at 2^24 words, and no gain in a graph at 2^16.)
constexpr int kWordsThreads = kCarryThreads + 32;

// The fix runs on up to one CTA per SM, each with a contiguous share of the
// tiles.  The carry into a share comes from the latest tile before it that does
// not propagate; inside it, 256 tiles at a time get their carry-ins by ballots,
// and the tiles whose carry-in is 1 are then taken by warps, 32 words a step.
// All-ones operands, whose product's low half is one long chain, are the worst
// case: 2^23 words 0.78 ms against 0.76 for random ones (8.2 with one thread per
// run of tiles, word by word).  A CTA per 64 tiles, eight to a warp; without
// chains every CTA returns at once.
constexpr int kFixThreads = 256;
inline unsigned fix_ctas(size_t ntiles) {
    return ntiles < 128 ? 1u : ntiles < 64 * 148 ? (unsigned)(ntiles / 64) : 148u;
}

// +1 at the first word of tile t, by one warp; ones: the tile propagates (its
// words are all ones and become zero).
__device__ __forceinline__ void carry_fix_tile(uint32_t t, bool ones, uint32_t* __restrict__ out,
                                               size_t M) {
    const int lane = threadIdx.x & 31;
    const size_t beg = (size_t)t * kCarryTileWords;
    const size_t end = min(M, beg + kCarryTileWords);
    if (ones) {
        for (size_t i = beg + lane; i < end; i += 32) out[i] = 0u;
        return;
    }
    for (size_t i = beg; i < end; i += 32) {
        const size_t j = i + lane;
        const uint32_t v = j < end ? __ldcg(out + j) : 0xffffffffu;
        const uint32_t stop = __ballot_sync(0xffffffffu, v != 0xffffffffu);
        const int f = stop ? __ffs((int)stop) - 1 : 32;
        if (j < end && lane <= f) out[j] = lane == f ? v + 1u : 0u;
        if (stop) break;
    }
}

__device__ __forceinline__ void carry_fix_body(const uint32_t* __restrict__ kinds,
                                               uint32_t ntiles, uint32_t* __restrict__ out,
                                               size_t M, const uint32_t* __restrict__ any,
                                               uint32_t part, uint32_t parts) {
    if (__ldcg(any) == 0u) return;  // every tile kills
    constexpr uint32_t NT = kFixThreads, NW = NT / 32;
    __shared__ uint32_t s_pos, s_n, s_last[NW], s_list[NT];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t share = (ntiles + parts - 1) / parts;
    const uint32_t r0 = min(ntiles, part * share), r1 = min(ntiles, r0 + share);
    // the carry into the share (0 into the first tile)
    uint32_t cin = 0;
    for (uint32_t e = r0; e > 0; e -= min(e, NT)) {
        __syncthreads();
        if (tid == 0) s_pos = NT;
        __syncthreads();
        if (tid < e && __ldcg(kinds + (e - 1 - tid)) != 2u) atomicMin(&s_pos, tid);
        __syncthreads();
        if (s_pos < NT) {
            cin = __ldcg(kinds + (e - 1 - s_pos)) & 1u;
            break;
        }
    }
    for (uint32_t c0 = r0; c0 < r1; c0 += NT) {
        const uint32_t t = c0 + tid;
        const uint32_t k = t < r1 ? __ldcg(kinds + t) : 2u;
        // kill and generate pass on a constant, 0 and 1
        const uint32_t con = __ballot_sync(0xffffffffu, k != 2u);
        const uint32_t val = __ballot_sync(0xffffffffu, k == 3u);
        if (lane == 0) s_last[warp] = con ? (val >> (31 - __clz(con))) & 1u : 2u;
        if (tid == 0) s_n = 0;
        __syncthreads();
        uint32_t eps = cin, cout = cin;
        for (uint32_t w = 0; w < NW; ++w)
            if (s_last[w] != 2u) {
                cout = s_last[w];
                if (w < warp) eps = cout;
            }
        const uint32_t below = con & ((1u << lane) - 1u);
        if (below) eps = (val >> (31 - __clz(below))) & 1u;
        if (eps && t < r1) s_list[atomicAdd(&s_n, 1u)] = 2u * t + (k == 2u ? 1u : 0u);
        __syncthreads();
        for (uint32_t i = warp; i < s_n; i += NW)
            carry_fix_tile(s_list[i] >> 1, (s_list[i] & 1u) != 0, out, M);
        cin = cout;
        __syncthreads();
    }
}

// SUM: the first CTA also compares the product's word sums.
template <bool SUM>
static __global__ void __launch_bounds__(kFixThreads)
k_carry_fix(const uint32_t* __restrict__ kinds, uint32_t ntiles, uint32_t* __restrict__ out,
            size_t M, const uint32_t* __restrict__ any, Sum* __restrict__ sums, int square,
            uint32_t* __restrict__ err) {
    grid_release();
    grid_wait();
    if constexpr (SUM) {
        if (blockIdx.x == 0 && threadIdx.x < 32)
            check_sums(sums, load_sums(sums), square != 0, err);
    }
    carry_fix_body(kinds, ntiles, out, M, any, blockIdx.x, gridDim.x);
}

// The check alone, behind the look-back form's pieces.
static __global__ void __launch_bounds__(32)
k_check_sums(Sum* sums, int square, uint32_t* err) {
    check_sums(sums, load_sums(sums), square != 0, err);
}

// any: set when a tile's kind is not kill (zero before).
// Four CTAs per SM with 64-bit coefficients (56 registers; 2^23 coefficients
// 78 -> 71 us, double precision, 83 -> 77 six primes), three otherwise (at four
// the digit sums spill: 2^20 points 47 -> 50 us for the product).
template <class Ar, bool SPLIT16, bool W64>
__device__ __forceinline__ void carry_words_body(const PlanDev<Ar>& P,
                                                 const typename Ar::T* __restrict__ res,
                                                 uint32_t* __restrict__ out, size_t M, size_t NL,
                                                 uint32_t* __restrict__ kinds,
                                                 uint32_t* __restrict__ any,
                                                 uint32_t* __restrict__ err, Sum* sums,
                                                 bool square) {
    constexpr int E = kCarryWordsPerThread;
    constexpr int TL = kCarryTileWords;
    __shared__ CarryShared sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool own = tid < kCarryThreads;
    const uint32_t t = blockIdx.x;
    // this thread's words; the first thread of the ninth warp takes the eight
    // words before the tile
    const size_t j0 = own ? (size_t)t * TL + (size_t)tid * E : (size_t)t * TL - E;
    const bool valid = (own || (tid == kCarryThreads && t > 0)) && j0 < NL;
    const size_t n = (size_t)1 << P.log_n;
    uint32_t l[E];
    uint32_t X[3];
    uint32_t bad = 0;
    garner_local<Ar, SPLIT16, W64, false>(
        P, res + (valid ? j0 : 0) * elems_per_word2<SPLIT16, W64>() / 2, n, valid, l, X, &bad);
    if (bad && own) atomicOr(err, 2u);
    uint32_t PX[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) PX[q] = __shfl_up_sync(0xffffffffu, X[q], 1);
    if (own ? lane == 31 : lane == 0) {
        uint32_t* d = own ? sh.lastx[warp] : sh.cin;
        d[0] = X[0];
        d[1] = X[1];
        d[2] = X[2];
    }
    __syncthreads();
    if (lane == 0) {
#pragma unroll
        for (int q = 0; q < 3; ++q) PX[q] = warp > 0 ? sh.lastx[own ? warp - 1 : 0][q] : sh.cin[q];
    }
    uint32_t S[E];
    int st;
    {
        uint64_t c = 0;
        uint32_t all = 0xffffffffu;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const uint64_t sum = (uint64_t)l[e] + (e < 3 ? PX[e] : 0u) + c;
            S[e] = (uint32_t)sum;
            c = sum >> 32;
            all &= S[e];
        }
        st = c ? 2 : (all == 0xffffffffu ? 1 : 0);
        if constexpr (W64) {
            if (own) sum_part(sh.sum, digit_sum(S, (uint32_t)c));
        }
    }
    ChainMasks cm{0, 0};
    if (own) cm = chain_prepare(st, sh.w);
    __syncthreads();
    if constexpr (W64) {
        if (!own) {
            sum_parts(sums + 2 * kSumSlots, t, sh.sum, kCarryThreads / 32);
            // a product of one tile has no fix to compare the sums
            if (gridDim.x == 1) {
                __threadfence();
                __syncwarp();
                check_sums(sums, load_sums(sums), square, err);
            }
        }
    }
    if (own) {
        const uint32_t mc = chain_mine(cm, sh.w, 0u);
        uint32_t w[E];
        uint64_t c = mc;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const uint64_t sum = (uint64_t)S[e] + c;
            w[e] = (uint32_t)sum;
            c = sum >> 32;
        }
        if (j0 + E <= M && ((reinterpret_cast<uintptr_t>(out + j0) & 15u) == 0)) {
            uint4* o = reinterpret_cast<uint4*>(out + j0);
            o[0] = make_uint4(w[0], w[1], w[2], w[3]);
            o[1] = make_uint4(w[4], w[5], w[6], w[7]);
        } else {
#pragma unroll
            for (int e = 0; e < E; ++e)
                if (j0 + e < M) out[j0 + e] = w[e];
        }
    }
    if (tid == 0 && gridDim.x > 1) {
        const uint32_t kind = chain_out(sh.w, 0u, kCarryThreads / 32) |
                              (chain_out(sh.w, 1u, kCarryThreads / 32) << 1);
        kinds[t] = kind;
        if (kind) atomicOr(any, 1u);
    }
}

template <class Ar, bool SPLIT16, bool W64 = false>
__global__ void __launch_bounds__(kWordsThreads, W64 ? 4 : 3)
k_carry_words(const PlanDev<Ar> P, const typename Ar::T* __restrict__ res,
              uint32_t* __restrict__ out, size_t M, size_t NL, uint32_t* __restrict__ kinds,
              uint32_t* __restrict__ any, uint32_t* __restrict__ err, Sum* __restrict__ sums,
              int square) {
    grid_release();
    grid_wait();
    carry_words_body<Ar, SPLIT16, W64>(P, res, out, M, NL, kinds, any, err, sums, square != 0);
}

// batched: blockIdx.y = product; the look-back kernel's 22-34% of issue slots
// were waits between a product's tiles (126 products of 2^17 points, 32-bit
// path: 86 us of 470)
template <class Ar, bool SPLIT16>
__global__ void __launch_bounds__(kWordsThreads, 3)
kb_carry_words(const PlanDev<Ar> P, const BatchProd* __restrict__ D,
               const typename Ar::T* __restrict__ res_a, uint32_t* __restrict__ err) {
    const BatchProd d = D[blockIdx.y];
    const size_t NL = ((size_t)1 << P.log_n) / (SPLIT16 ? 2 : 1);
    const size_t M = (size_t)d.la + d.lb;
    if ((size_t)blockIdx.x * kCarryTileWords >= (NL > M ? NL : M)) return;
    carry_words_body<Ar, SPLIT16, false>(P, res_a + d.res_off, d.out, M, NL, d.rec_s, &d.cst->any,
                                         err, nullptr, false);
}
// blockIdx.y = product
static __global__ void __launch_bounds__(kFixThreads)
kb_carry_fix(const BatchProd* __restrict__ D, size_t NL) {
    const BatchProd d = D[blockIdx.y];
    const size_t M = (size_t)d.la + d.lb, words = NL > M ? NL : M;
    carry_fix_body(d.rec_s, (uint32_t)((words + kCarryTileWords - 1) / kCarryTileWords), d.out, M,
                   &d.cst->any, blockIdx.x, gridDim.x);
}

// Carry words of the last thread of every tile but the last (its 8 words'
// carry-out with carry-in zero), published under `epoch` before K4 runs.
// K4 tile t then finds tile t-1's record ready and waits only on the 1-bit
// look-back, not on its predecessor's Garner phase.  One thread per tile.
template <class Ar, bool SPLIT16, bool W64 = false>
__global__ void __launch_bounds__(256)
k_carry_bounds(const PlanDev<Ar> P, const typename Ar::T* __restrict__ res, size_t NL,
               uint4* __restrict__ rec_x, uint32_t ntiles, uint32_t epoch) {
    constexpr int E = kCarryWordsPerThread;
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t + 1 >= ntiles) return;
    const size_t n = (size_t)1 << P.log_n;
    const size_t j0 = (size_t)(t + 1) * kCarryTileWords - E;
    uint32_t X[3];
    uint32_t bad = 0;  // the tile's own pass reports reconstruction errors
    if constexpr (W64) {
        uint32_t l[E];
        garner_words_w64<Ar, E>(P, res, n, j0, NL, l, X, &bad);
    } else {
        unsigned __int128 D[E];
        garner_digits<Ar, SPLIT16, E>(P, res, n, j0, NL, D, &bad);
        unsigned __int128 acc = 0;
#pragma unroll
        for (int e = 0; e < E; ++e) acc = (acc + D[e]) >> 32;
        X[0] = (uint32_t)acc;
        X[1] = (uint32_t)(acc >> 32);
        X[2] = (uint32_t)(acc >> 64);
    }
    uint32_t* rx = reinterpret_cast<uint32_t*>(rec_x + t);
    st_relaxed(rx + 0, X[0]);
    st_relaxed(rx + 1, X[1]);
    st_relaxed(rx + 2, X[2]);
    st_release(rx + 3, epoch);
}

// Four CTAs per SM (at most 64 registers): the tile's barriers and its
// one-bit look-back leave warps idle, which more resident CTAs cover
// (measured 12% faster than three).
template <class Ar, bool SPLIT16, bool W64 = false>
__global__ void __launch_bounds__(kCarryThreads, 4)
k_garner_carry(const PlanDev<Ar> P, const typename Ar::T* __restrict__ res,
               uint32_t* __restrict__ out, size_t M, size_t NL, CarryState* cst,
               uint4* __restrict__ rec_x, uint32_t* __restrict__ rec_s, uint32_t epoch,
               uint32_t wait_epoch, uint32_t* __restrict__ err, int spin_limit,
               Sum* __restrict__ sum) {
    garner_carry_body<Ar, SPLIT16, W64>(P, res, out, M, NL, cst, rec_x, rec_s, epoch,
                                        wait_epoch, err, spin_limit, sum);
}

// batched: blockIdx.y = product
template <class Ar, bool SPLIT16>
__global__ void __launch_bounds__(kCarryThreads, 4)
kb_garner_carry(const PlanDev<Ar> P, const BatchProd* __restrict__ D,
                const typename Ar::T* __restrict__ res_a, uint32_t epoch, uint32_t wait_epoch,
                uint32_t* __restrict__ err, int spin_limit) {
    const BatchProd d = D[blockIdx.y];
    const size_t NL = ((size_t)1 << P.log_n) / (SPLIT16 ? 2 : 1);
    garner_carry_body<Ar, SPLIT16>(P, res_a + d.res_off, d.out, (size_t)d.la + d.lb, NL, d.cst,
                                   d.rec_x, d.rec_s, epoch, wait_epoch, err, spin_limit, nullptr);
}

// ------------------------------------------------------------------ small products
// One CTA computes a whole product whose n-point transform fits in shared
// memory (a batch bucket of equal n, blockIdx.x = product): for each prime
// the forward transforms of both operands, the pointwise product and the
// inverse transform run in shared memory (stage twiddles pr.WCf / pr.WCi of
// length n, scale pr.scale = n^-1 2^bits), the residues go to a per-product
// global scratch (L2-resident at these sizes); then Garner + carry over the
// product's words in tiles of NT*8 words, the carry handed from tile to tile
// inside the CTA, so no look-back is needed.
// Register bounds: 64-bit residues run radix-8 rounds in 64 registers (four
// 256-thread CTAs per SM; radix 16 took 128, two per SM, 12.5% warps
// active); 32-bit residues get at most 128 (unbounded they took 185, one
// 256-thread CTA per SM).
template <class Ar>
constexpr int ks_min_blocks(int nt) {
    return sizeof(typename Ar::T) == 8 ? 1024 / nt : 512 / nt;
}
template <class Ar, bool SPLIT16, int NT>
__device__ __forceinline__ void ks_product_body(const PlanDev<Ar>& P, const BatchProd& d,
                                                typename Ar::T* scratch,
                                                uint32_t* __restrict__ err,
                                                unsigned char* smem_raw) {
    using T = typename Ar::T;
    constexpr int RLOG = sizeof(T) == 8 ? 3 : 4;
    constexpr int E = kCarryWordsPerThread;
    constexpr int CPW = SPLIT16 ? 2 : 1;
    __shared__ uint32_t s_w[NT / 32];
    __shared__ uint32_t s_lastx[NT / 32][3];
    __shared__ uint32_t s_cin[3];
    __shared__ uint32_t s_eps;
    const int log_n = P.log_n;
    const int n = 1 << log_n;
    T* bufA = reinterpret_cast<T*>(smem_raw);
    T* bufB = bufA + tile_elems(n);
    T* res = scratch + d.res_off;
    const size_t nca = (size_t)d.la * CPW, ncb = (size_t)d.lb * CPW;
    const int sq = d.square;
    const int nr = sched_rounds<RLOG>(log_n);
    auto coef = [&](const uint32_t* src, size_t nc, int i) -> T {
        if ((size_t)i >= nc) return T(0);
        if constexpr (SPLIT16) {
            return (T)((__ldg(src + (i >> 1)) >> ((i & 1) * 16)) & 0xFFFFu);
        } else {
            return Ar::from_u32(__ldg(src + i));
        }
    };
    auto ldA = [&](int, int, int p) -> T { return bufA[p]; };

    for (int kp = 0; kp < P.K; ++kp) {
        const PrimeDev<Ar>& pr = P.pr[kp];
        const Ar ar = pr.ar;
        const Tw<T> sc = pr.scale;
        auto st_res = [&](int idx, T v) {
            res[(size_t)kp * n + idx] = ar.scale_out(v, sc);
        };
        for (int i = threadIdx.x; i < n; i += NT) {
            bufA[LayRow::p(i)] = coef(d.a, nca, i);
            if (!sq) bufB[LayRow::p(i)] = coef(d.b, ncb, i);
        }
        __syncthreads();
        for (int op = 0; op < (sq ? 1 : 2); ++op) {
            T* buf = op ? bufB : bufA;
            const int rounds = (op == 0 && !sq) ? nr : nr - 1;
            auto ld = [&](int, int, int p) -> T { return buf[p]; };
            auto st = [&](int, int, int p, T v) { buf[p] = v; };
            for (int r = 0; r < rounds; ++r) {
                run_round_rl<Ar, LayRow, RLOG, false, false>(sched_rl<RLOG>(log_n, r), log_n, 0,
                                                     sched_s0<RLOG>(log_n, r), pr.WCf, ar, false,
                                                     ld, st);
                __syncthreads();
            }
        }
        {
            // last forward round of B (or A), product, first inverse round
            const int r = nr - 1;
            const int rl = sched_rl<RLOG>(log_n, r), s0 = sched_s0<RLOG>(log_n, r);
            const int d_log = log_n - s0 - rl;
            const int nsub = 1 << (log_n - rl);
            const bool final_round = (nr == 1);
            T* src = sq ? bufA : bufB;
            for (int sp = threadIdx.x; sp < nsub; sp += NT) {
                const int j = sp & ((1 << d_log) - 1);
                const int g = sp >> d_log;
                const int base = (g << (d_log + rl)) + j;
                const int p0 = LayRow::p(base);   // last round: stride 1 (d_log = 0)
                T x[1 << RLOG];
#define BW_SMALL_FUSED(RL)                                                             \
    {                                                                                  \
        _Pragma("unroll") for (int k = 0; k < (1 << RL); ++k) x[k] = src[p0 + k];     \
        ct_stages<Ar, RL, false>(x, s0, g, pr.WCf, ar, false);                         \
        _Pragma("unroll") for (int k = 0; k < (1 << RL); ++k) {                        \
            const T xa = ar.fwd_to_2p(x[k]);                                           \
            const T ya = sq ? xa : bufA[p0 + k];                                       \
            x[k] = ar.pointwise(ya, xa);                                               \
        }                                                                              \
        gs_stages<Ar, RL, false>(x, s0, g, pr.WCi, ar);                                \
        _Pragma("unroll") for (int k = 0; k < (1 << RL); ++k) {                        \
            if (final_round) st_res(base + k, x[k]); else bufA[p0 + k] = x[k];         \
        }                                                                              \
    }
                if (rl == RLOG) {
                    BW_SMALL_FUSED(RLOG)
                } else if (rl == 3) {
                    BW_SMALL_FUSED(3)
                } else if (rl == 2) {
                    BW_SMALL_FUSED(2)
                } else {
                    BW_SMALL_FUSED(1)
                }
#undef BW_SMALL_FUSED
            }
            __syncthreads();
        }
        for (int r = nr - 2; r >= 0; --r) {
            const bool last = (r == 0);
            auto st = [&](int, int idx, int p, T v) {
                if (last) {
                    st_res(idx, v);
                } else {
                    bufA[p] = v;
                }
            };
            run_round_rl<Ar, LayRow, RLOG, true, false>(sched_rl<RLOG>(log_n, r), log_n, 0,
                                                sched_s0<RLOG>(log_n, r), pr.WCi, ar, false, ldA,
                                                st);
            __syncthreads();
        }
    }

    // ---- Garner + carry, tile by tile; the carry into a tile is the previous
    // tile's last carry words (s_cin) plus its chain carry-out bit (s_eps)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const size_t NL = (size_t)n / CPW, M = (size_t)d.la + d.lb;
    const size_t words = NL > M ? NL : M;
    if (tid == 0) {
        s_cin[0] = s_cin[1] = s_cin[2] = 0;
        s_eps = 0;
    }
    __syncthreads();
    uint32_t bad = 0;
    for (size_t t0 = 0; t0 < words; t0 += (size_t)NT * E) {
        const size_t j0 = t0 + (size_t)tid * E;
        unsigned __int128 Dg[E];
        garner_digits<Ar, SPLIT16, E, false>(P, res, n, j0, NL, Dg, &bad);
        uint32_t l[E], X[3];
        {
            unsigned __int128 acc = 0;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                acc += Dg[e];
                l[e] = (uint32_t)acc;
                acc >>= 32;
            }
            X[0] = (uint32_t)acc;
            X[1] = (uint32_t)(acc >> 32);
            X[2] = (uint32_t)(acc >> 64);
        }
        uint32_t PX[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) PX[q] = __shfl_up_sync(0xffffffffu, X[q], 1);
        if (lane == 31) {
            s_lastx[warp][0] = X[0];
            s_lastx[warp][1] = X[1];
            s_lastx[warp][2] = X[2];
        }
        __syncthreads();
        if (lane == 0) {
#pragma unroll
            for (int q = 0; q < 3; ++q) PX[q] = warp > 0 ? s_lastx[warp - 1][q] : s_cin[q];
        }
        uint32_t S[E];
        int st;
        {
            uint64_t c = 0;
            uint32_t all = 0xffffffffu;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const uint64_t s = (uint64_t)l[e] + (e < 3 ? PX[e] : 0u) + c;
                S[e] = (uint32_t)s;
                c = s >> 32;
                all &= S[e];
            }
            st = c ? 2 : (all == 0xffffffffu ? 1 : 0);
        }
        const ChainMasks cm = chain_prepare(st, s_w);
        __syncthreads();
        const uint32_t eps_in = s_eps;
        const uint32_t mc = chain_mine(cm, s_w, eps_in);
        const uint32_t cout = chain_out(s_w, eps_in, NT / 32);
        {
            uint64_t c = mc;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const uint64_t s = (uint64_t)S[e] + c;
                if (j0 + e < M) d.out[j0 + e] = (uint32_t)s;
                c = s >> 32;
            }
        }
        __syncthreads();  // every thread has read s_cin, s_eps, s_lastx, s_w
        if (tid == NT - 1) {
            s_cin[0] = X[0];
            s_cin[1] = X[1];
            s_cin[2] = X[2];
        }
        if (tid == 0) s_eps = cout;
        __syncthreads();
    }
    if (bad) atomicOr(err, 2u);
}

template <class Ar, bool SPLIT16, int NT>
__global__ void __launch_bounds__(NT, ks_min_blocks<Ar>(NT))
ks_product(const PlanDev<Ar> P, const BatchProd* __restrict__ D, typename Ar::T* scratch,
           uint32_t* __restrict__ err) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ks_product_body<Ar, SPLIT16, NT>(P, D[blockIdx.x], scratch, err, smem_raw);
}

// Persistent form of the small buckets of one prime path
// (BW_BATCH_PERSISTENT): a grid of a few CTAs per SM pulls work items --
// (bucket, product) pairs, largest transforms first -- from a device queue
// (an atomic head) and runs each as ks_product does, reading the bucket's
// plan and descriptor from device arrays.  The queue head is cleared before
// every run; a CTA stops at the first item past the end.  No waits.
struct SmallItem {
    uint32_t bucket;
    uint32_t prod;
};
template <class Ar>
struct SmallBucketDev {
    PlanDev<Ar> plan;
    const BatchProd* desc;
    typename Ar::T* scratch;
};
template <class Ar, bool SPLIT16, int NT>
__global__ void __launch_bounds__(NT, ks_min_blocks<Ar>(NT))
kq_small(const SmallBucketDev<Ar>* __restrict__ buckets, const SmallItem* __restrict__ items,
         uint32_t count, uint32_t* __restrict__ head, uint32_t* __restrict__ err) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint32_t s_item;
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(head, 1u);
        __syncthreads();
        const uint32_t it = s_item;
        if (it >= count) break;
        const SmallItem w = items[it];
        const SmallBucketDev<Ar>& b = buckets[w.bucket];
        ks_product_body<Ar, SPLIT16, NT>(b.plan, b.desc[w.prod], b.scratch, err, smem_raw);
        __syncthreads();  // every thread has read s_item and left the body
    }
}

}  // namespace bw
