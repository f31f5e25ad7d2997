// bw_ntt.cuh -- the transform passes with lengths known at compile time.
//
// The passes of bw_kernels.cuh take any length at run time.  The common
// lengths run these instead: every stride, slot offset and trip count is an
// immediate, the first round of a pass loads global memory straight into
// registers and the last one stores from them (nothing is staged through
// shared memory only to be moved), and the twiddles of a round come in an
// order in which a warp's loads are consecutive.
//
// Twiddle order.  A transform of length 2^L runs rounds of 4 stages, a
// remainder round of L mod 4 stages first.  The round that starts at stage
// S0 uses the table range [2^S0, 2^(S0+RL)); inside it the entries are stored
// by (position in the sub-problem, group) rather than by (stage, group,
// position), the positions in pairs:
//   stage S0:      entry of group g at 2^S0 + g
//   stage S0 + l:  positions q, q + 1 (q even) of group g at
//                  2^(S0+1) + 2 (P 2^S0 + g), P = 2^(l-1) - 1 + q / 2
// In a row's last round every thread has a group of its own: its 15 twiddles,
// contiguous in the (stage, group, position) order, put the lanes of a warp 8
// to 64 bytes apart, 86 wavefronts per sub-problem against the 32 (4-byte
// residues) of its data; in this order they are 30.  tw_place maps an entry to
// its place.
#pragma once
#include "bw_kernels.cuh"

namespace bw {

// Lengths the passes are instantiated for (log2): rows, and columns of 4- and
// 8-byte residues.
constexpr int kRow2MinLog = 5, kRow2MaxLog = 13;
constexpr int kCol2MinLog = 3, kCol2MaxLog32 = 12, kCol2MaxLog64 = 13;
constexpr int kMid2MinLog = 5, kMid2MaxLog = 11;

// Rounds of a 2^L-point transform: the remainder round first.
__host__ __device__ constexpr int first_rl(int L) { return L % 4 == 0 ? (L < 4 ? L : 4) : L % 4; }

// Place of the stage table's entry 2^s + i in the round order.
__host__ __device__ inline uint32_t tw_place(int s, uint32_t i, int L) {
    const int rl0 = first_rl(L);
    const int s0 = s < rl0 ? 0 : rl0 + (s - rl0) / 4 * 4;
    const int l = s - s0;
    const uint32_t g = i >> l, q = i & ((1u << l) - 1), G = 1u << s0;
    if (l == 0) return G + g;
    return 2 * G + 2 * (((1u << (l - 1)) - 1 + (q >> 1)) * G + g) + (q & 1);
}

// The stage of place i (i >= 1) when the first round has rl0 stages.
__device__ __forceinline__ int stage_of_place(int i, int rl0) {
    int s0 = rl0;
    while (i >= (16 << s0)) s0 += 4;
    if (i < (1 << rl0)) s0 = 0;
    const int u = (i - (1 << s0)) >> s0;  // 0: first stage; else 2 P + 1, 2 P + 2
    return s0 + (u == 0 ? 0 : 32 - __clz((u + 1) >> 1));
}

// One round's twiddles of a thread's sub-problem in group g (G = 2^S0 groups).
template <typename T, int G, bool SM>
struct RoundTw {
    const Tw<T>* p1;
    const Tw<T>* p2;
    __device__ __forceinline__ RoundTw(const Tw<T>* W, int g) : p1(W + G + g), p2(W + 2 * G + 2 * g) {}
    __device__ __forceinline__ Tw<T> one() const { return ld_w<SM>(p1); }
    // positions 2 j, 2 j + 1 of stage l: P = 2^(l-1) - 1 + j
    __device__ __forceinline__ void pair(int P, Tw<T>& a, Tw<T>& b) const {
        const Tw<T>* p = p2 + (size_t)P * 2 * G;
        if constexpr (sizeof(Tw<T>) == 8) {
            ld_w2<SM>(p, a, b);
        } else {
            a = ld_w<SM>(p);
            b = ld_w<SM>(p + 1);
        }
    }
};

// Forward (CT) round on a sub-problem in registers.  ONE: the first stage's
// twiddle is 1 (stage 0 of a column); ZT: the upper half is zero and the first
// stage (twiddle 1) copies the lower one; ENT: the inputs may be any forward
// output (ArD reduces some of them; the integer arithmetics ignore it).
template <class Ar, int RL, bool ONE, bool ZT, bool ENT, class TW>
__device__ __forceinline__ void ct_round(typename Ar::T* x, const Ar& ar, const TW& tw) {
    using T = typename Ar::T;
#pragma unroll
    for (int l = 0; l < RL; ++l) {
        const int h = 1 << (RL - l - 1);
        if constexpr (Ar::kF64) {
#pragma unroll
            for (int u = 0; u < (1 << RL); ++u) x[u] = ar.ct_enter(x[u], u, 1 << (RL - 1), l, ENT);
        }
        if (l == 0) {
            if constexpr (ZT) {
#pragma unroll
                for (int u = 0; u < h; ++u) x[u + h] = x[u];
            } else if constexpr (ONE) {
#pragma unroll
                for (int u = 0; u < h; ++u) ar.ct1(x[u], x[u + h]);
            } else {
                const Tw<T> w = tw.one();
#pragma unroll
                for (int u = 0; u < h; ++u) ar.ct(x[u], x[u + h], w);
            }
            continue;
        }
#pragma unroll
        for (int q = 0; q < (1 << l); q += 2) {
            Tw<T> w[2];
            tw.pair((1 << (l - 1)) - 1 + q / 2, w[0], w[1]);
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int u = 0; u < h; ++u) {
                    const int k = ((q + e) << (RL - l)) + u;
                    ar.ct(x[k], x[k + h], w[e]);
                }
        }
    }
}

// Inverse (GS) round, the mirror of ct_round.  LAST: ArD reduces the sums of
// the round's last stage (not needed before a multiplication).
template <class Ar, int RL, bool ONE, bool LAST, class TW>
__device__ __forceinline__ void gs_round(typename Ar::T* x, const Ar& ar, const TW& tw) {
    using T = typename Ar::T;
    auto gs = [&](T& a, T& b, const Tw<T>& w, bool red) {
        if constexpr (Ar::kF64) {
            if (red) {
                ar.template gs<true>(a, b, w);
            } else {
                ar.template gs<false>(a, b, w);
            }
        } else {
            ar.gs(a, b, w);
        }
    };
#pragma unroll
    for (int l = RL - 1; l >= 0; --l) {
        const int h = 1 << (RL - l - 1);
        const bool red = l == 0 ? LAST : ((RL - 1 - l) & 1) != 0;
        if (l == 0) {
            if constexpr (ONE) {
#pragma unroll
                for (int u = 0; u < h; ++u) ar.gs1(x[u], x[u + h]);
            } else {
                const Tw<T> w = tw.one();
#pragma unroll
                for (int u = 0; u < h; ++u) gs(x[u], x[u + h], w, red);
            }
            continue;
        }
#pragma unroll
        for (int q = 0; q < (1 << l); q += 2) {
            Tw<T> w[2];
            tw.pair((1 << (l - 1)) - 1 + q / 2, w[0], w[1]);
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int u = 0; u < h; ++u) {
                    const int k = ((q + e) << (RL - l)) + u;
                    gs(x[k], x[k + h], w[e], red);
                }
        }
    }
}

// Resident threads per SM the register bounds aim at: 1024 of 64 registers
// (32-bit path), 768 of 80 (double precision), 512 of 128 (64-bit integers).
template <class Ar>
__host__ __device__ constexpr int resident_threads() {
    return sizeof(typename Ar::T) == 4 ? 1024 : Ar::kF64 ? 768 : 512;
}

// Row layout: 8-byte residues e + e/16, conflict-free for every round (a
// 64-bit access is served 16 lanes at a time).  4-byte residues e + e/32:
// conflict-free for unit-stride lanes and for the stride-16 lanes of a last
// round; the 16 x 16 middle round takes groups two apart in one warp
// (row_group), which puts its two runs of 16 lanes on different banks.
template <typename T>
using LayRow2 = typename std::conditional<sizeof(T) == 4, Lay<5, 1>, Lay<4, 1>>::type;

// Sub-problem sp of a round with 2^D sub-problems per group -> (group, j).
template <typename T, int D, int NSUB>
__device__ __forceinline__ void row_group(int sp, int& g, int& j) {
    j = sp & ((1 << D) - 1);
    g = sp >> D;
    if constexpr (sizeof(T) == 4 && D == 4 && NSUB >= 64) {
        // swap the group's two low bits: lanes 0-15 and 16-31 of a warp take
        // groups two apart
        g = (g & ~3) | ((g & 1) << 1) | ((g >> 1) & 1);
    }
}

// ------------------------------------------------------------------ rows
// Fused row pass for one row and prime: forward transforms of both operands'
// rows, pointwise product, inverse transform, with the twiddles between the
// passes, w^(c k1) on element c, mostly folded into the stage twiddles.  The
// row's transform evaluates sum_c x_c y^c at y = zeta w_C^j with zeta = w^k1:
// CT stages on y^C - zeta^C split it by (y^(C/2m) - r)(y^(C/2m) + r) with
// r = zeta^(C/2m) W[m + i], so a table R[m + i] = zeta^(C/2m) W[m + i] of
// C / 16 entries per row, built in shared memory, takes the first stages
// through the whole twist; before the last round, whose sub-problems are 16
// consecutive elements, substituting y = zeta z leaves zeta^j on element j and
// the plain twiddles after it.  One multiplication per element and transform
// instead of two, and the inverse mirrors it (zeta^-j n^-1 2^bits after its
// first round).
template <class Ar, int LOGC>
struct RowCfg {
    static constexpr int C = 1 << LOGC;
    static constexpr int RLAST = LOGC < 4 ? LOGC : 4;
    static constexpr int S1 = LOGC - RLAST;  // stages with row twiddles
    static constexpr int NSUB = C >> RLAST;
    static constexpr int NT = NSUB < 32 ? 32 : NSUB > 256 ? 256 : NSUB;
    // shared memory: row twiddles, their inverses, zeta powers, two row buffers
    static constexpr size_t smem(bool sq) {
        return ((size_t)2 * (1 << S1) + 32 + 32) * sizeof(Tw<typename Ar::T>) +
               tile_elems(C) * sizeof(typename Ar::T) * (sq ? 1 : 2);
    }
    static constexpr int kMinCtas = resident_threads<Ar>() / NT;
};

// A thread's elements of a row's first round, all loaded at once (rows of one
// sub-problem of 16 per thread): they arrive while the twiddles are built, or
// while the other operand's round runs.  L2 loads: the previous kernel wrote
// them, and each is read once.
template <class Ar, int LOGC>
struct RowPre {
    static constexpr int RL = first_rl(LOGC), D = LOGC - RL;
    static constexpr int NT = RowCfg<Ar, LOGC>::NT, IT = (1 << D) < NT ? 1 : (1 << D) / NT;
    typename Ar::T x[IT << RL];
    __device__ __forceinline__ void load(const typename Ar::T* g) {
#pragma unroll
        for (int i = 0; i < IT; ++i)
#pragma unroll
            for (int k = 0; k < (1 << RL); ++k)
                x[(i << RL) + k] = __ldcg(g + threadIdx.x + i * NT + (k << D));
    }
    // the round itself, into shared memory
    __device__ __forceinline__ void round(typename Ar::T* buf, const Ar& ar,
                                          const Tw<typename Ar::T>* W) {
        using T = typename Ar::T;
        using L = LayRow2<T>;
#pragma unroll
        for (int i = 0; i < IT; ++i) {
            const int p0 = L::p(threadIdx.x + i * NT);
            ct_round<Ar, RL, false, false, true>(x + (i << RL), ar, RoundTw<T, 1, true>(W, 0));
#pragma unroll
            for (int k = 0; k < (1 << RL); ++k)
                buf[p0 + L::template off<false>(k, D, 0)] = x[(i << RL) + k];
        }
    }
};

// One CT round (starting at stage S0) of a row in shared memory, from global
// memory when FROM_G.
template <class Ar, int LOGC, int S0, int RL, bool FROM_G, class TWB>
__device__ __forceinline__ void row_ct(const typename Ar::T* gsrc, typename Ar::T* buf,
                                       const Ar& ar, const TWB* W) {
    using T = typename Ar::T;
    using L = LayRow2<T>;
    constexpr int D = LOGC - S0 - RL, NSUB = 1 << (LOGC - RL), NT = RowCfg<Ar, LOGC>::NT;
#pragma unroll 1
    for (int sp = threadIdx.x; sp < NSUB; sp += NT) {
        int g, j;
        row_group<T, D, NSUB>(sp, g, j);
        const int base = (g << (D + RL)) + j;
        const int p0 = L::p(base);
        T x[1 << RL];
#pragma unroll
        for (int k = 0; k < (1 << RL); ++k) {
            if constexpr (FROM_G) {
                x[k] = __ldcg(gsrc + base + (k << D));
            } else {
                x[k] = buf[p0 + L::template off<false>(k, D, 0)];
            }
        }
        ct_round<Ar, RL, false, false, true>(x, ar, RoundTw<T, (1 << S0), true>(W, g));
#pragma unroll
        for (int k = 0; k < (1 << RL); ++k) buf[p0 + L::template off<false>(k, D, 0)] = x[k];
    }
}

// One GS round of a row in shared memory, to global memory when TO_G.
template <class Ar, int LOGC, int S0, int RL, bool TO_G, class TWB>
__device__ __forceinline__ void row_gs(typename Ar::T* gdst, typename Ar::T* buf,
                                       const Ar& ar, const TWB* W) {
    using T = typename Ar::T;
    using L = LayRow2<T>;
    constexpr int D = LOGC - S0 - RL, NSUB = 1 << (LOGC - RL), NT = RowCfg<Ar, LOGC>::NT;
#pragma unroll 1
    for (int sp = threadIdx.x; sp < NSUB; sp += NT) {
        int g, j;
        row_group<T, D, NSUB>(sp, g, j);
        const int base = (g << (D + RL)) + j;
        const int p0 = L::p(base);
        T x[1 << RL];
#pragma unroll
        for (int k = 0; k < (1 << RL); ++k) x[k] = buf[p0 + L::template off<false>(k, D, 0)];
        gs_round<Ar, RL, false, true>(x, ar, RoundTw<T, (1 << S0), true>(W, g));
#pragma unroll
        for (int k = 0; k < (1 << RL); ++k) {
            if constexpr (TO_G) {
                gdst[base + (k << D)] = x[k];
            } else {
                buf[p0 + L::template off<false>(k, D, 0)] = x[k];
            }
        }
    }
}

// WAIT: the rows come from a kernel that may still be running (grid_wait before
// they are read; the twiddles do not depend on it).
template <class Ar, int LOGC, bool WAIT>
__device__ __forceinline__ void row2_body(const PlanDev<Ar>& P, typename Ar::T* res_a,
                                          const typename Ar::T* res_b, bool square, int prow,
                                          int kp, unsigned char* smem_raw) {
    using T = typename Ar::T;
    using Cfg = RowCfg<Ar, LOGC>;
    using L = LayRow2<T>;
    constexpr int C = Cfg::C, S1 = Cfg::S1, RLAST = Cfg::RLAST, NT = Cfg::NT, NSUB = Cfg::NSUB;
    constexpr int RL0 = first_rl(LOGC), NE = 1 << RLAST;
    static_assert(LOGC > 4 && LOGC <= 13, "two to four rounds");
    const size_t n = (size_t)1 << P.log_n;
    const int log_rr = P.log_r2 ? P.log_r2 : P.log_r;
    const PrimeDev<Ar>& pr = P.pr[kp];
    const Ar ar = pr.ar;
    T* ga = res_a + (size_t)kp * n + (size_t)prow * C;
    const T* gb = res_b + (size_t)kp * n + (size_t)prow * C;
    Tw<T>* R = reinterpret_cast<Tw<T>*>(smem_raw);   // row twiddles
    Tw<T>* Ri = R + (1 << S1);                       // inverse
    Tw<T>* Z = Ri + (1 << S1);                       // zeta^j, then zeta^-j n^-1 2^bits
    Tw<T>* ZL = Z + 32;                              // zeta^(C/2m) and inverse, by stage
    T* bufA = reinterpret_cast<T*>(ZL + 32);
    T* bufB = bufA + tile_elems(C);

    // ---- the rows' elements, where every thread takes 16: A's (4-byte
    // residues: B's too) before the tables, which need neither
    constexpr bool PRE = NSUB == NT && sizeof(T) == 4;
    RowPre<Ar, PRE ? LOGC : 8> xa, xb;

    // ---- the row's powers of zeta, then its twiddles
    {
        const size_t n_row = (size_t)C << log_rr;
        const uint64_t nmask = n_row - 1;
        const uint64_t k1 = bitrev((uint32_t)prow & ((1u << log_rr) - 1), log_rr);
        for (int i = threadIdx.x; i < 2 * NE + 2 * S1; i += NT) {
            if (i < NE) {
                Z[i] = pow_entry(ar, ((uint64_t)i * k1) & nmask, P.lo, pr.TLf, pr.THf);
            } else if (i < 2 * NE) {
                Z[i] = pow_entry(ar, ((uint64_t)(i - NE) * k1) & nmask, P.lo, pr.TLi, pr.THi);
            } else {
                const int s = (i - 2 * NE) >> 1;
                uint64_t e = (((uint64_t)C >> (s + 1)) * k1) & nmask;
                if (i & 1) e = (n_row - e) & nmask;
                ZL[i - 2 * NE] = pow_entry(ar, e, P.lo, pr.TLf, pr.THf);
            }
        }
        __syncthreads();
        if (WAIT) grid_wait();
        if constexpr (PRE) {
            xa.load(ga);
            if (!square) xb.load(gb);
        }
        for (int i = 1 + threadIdx.x; i < (1 << S1); i += NT) {
            const int s = stage_of_place(i, RL0);
            R[i] = ar.mul_tw(ZL[2 * s], ld_tw(pr.WCf + i));
            Ri[i] = ar.mul_tw(ZL[2 * s + 1], ld_tw(pr.WCi + i));
        }
        __syncthreads();
    }

    // ---- forward rounds with row twiddles, global memory -> shared memory
    if constexpr (PRE) {
        xa.round(bufA, ar, R);
        if (!square) xb.round(bufB, ar, R);
    } else {
        row_ct<Ar, LOGC, 0, RL0, true>(ga, bufA, ar, R);
        if (!square) row_ct<Ar, LOGC, 0, RL0, true>(gb, bufB, ar, R);
    }
    __syncthreads();
    if constexpr (S1 > RL0) {
        row_ct<Ar, LOGC, RL0, 4, false>(nullptr, bufA, ar, R);
        if (!square) row_ct<Ar, LOGC, RL0, 4, false>(nullptr, bufB, ar, R);
        __syncthreads();
    }
    if constexpr (S1 > RL0 + 4) {
        row_ct<Ar, LOGC, RL0 + 4, 4, false>(nullptr, bufA, ar, R);
        if (!square) row_ct<Ar, LOGC, RL0 + 4, 4, false>(nullptr, bufB, ar, R);
        __syncthreads();
    }

    // ---- last forward round of both, product, first inverse round: 16
    // consecutive elements per thread, no exchange in between
#pragma unroll 1
    for (int g = threadIdx.x; g < NSUB; g += NT) {
        const int p0 = L::p(g << RLAST);
        const RoundTw<T, (1 << S1), false> tf(pr.WCf, g), ti(pr.WCi, g);
        T x[NE];
        auto fwd = [&](const T* buf) {
#pragma unroll
            for (int k = 0; k < NE; ++k) x[k] = ar.mulc(buf[p0 + k], ld_w<true>(Z + k));
            ct_round<Ar, RLAST, false, false, false>(x, ar, tf);
        };
        fwd(bufA);
        if (square) {
#pragma unroll
            for (int k = 0; k < NE; ++k) {
                const T v = ar.fwd_to_2p(x[k]);
                x[k] = ar.pointwise(v, v);
            }
        } else {
#pragma unroll
            for (int k = 0; k < NE; ++k) bufA[p0 + k] = ar.fwd_to_2p(x[k]);
            fwd(bufB);
#pragma unroll
            for (int k = 0; k < NE; ++k) x[k] = ar.pointwise(x[k], bufA[p0 + k]);
        }
        gs_round<Ar, RLAST, false, false>(x, ar, ti);
#pragma unroll
        for (int k = 0; k < NE; ++k) bufA[p0 + k] = ar.mulc(x[k], ld_w<true>(Z + NE + k));
    }
    __syncthreads();

    // ---- remaining inverse rounds, the last one to global memory
    if constexpr (S1 > RL0 + 4) {
        row_gs<Ar, LOGC, RL0 + 4, 4, false>(nullptr, bufA, ar, Ri);
        __syncthreads();
    }
    if constexpr (S1 > RL0) {
        row_gs<Ar, LOGC, RL0, 4, false>(nullptr, bufA, ar, Ri);
        __syncthreads();
    }
    row_gs<Ar, LOGC, 0, RL0, true>(ga, bufA, ar, Ri);
}

template <class Ar, int LOGC>
__global__ void __launch_bounds__(RowCfg<Ar, LOGC>::NT, RowCfg<Ar, LOGC>::kMinCtas)
k_row2(const PlanDev<Ar> P, typename Ar::T* res_a, const typename Ar::T* res_b, int square) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    grid_release();
    row2_body<Ar, LOGC, true>(P, res_a, res_b, square != 0, blockIdx.x, blockIdx.y, smem_raw);
}

// ------------------------------------------------------------------ columns
// Columns of a tile (log2): 32 bytes (4-byte residues) to 64 wide, whole
// sectors, half of that for the longest columns, and more for short ones, so
// that a tile holds 1024 elements.  Narrower tiles to have more CTAs lose at
// every size: 4-byte residues in 16, 32 or 64 bytes measured, K1 + K3, 33 / 27
// / 31 us (2^21 points of 16-bit coefficients), 0.146 / 0.121 / 0.131 ms (six
// primes, 2^21); 8-byte residues in 16, 32 or 64 bytes 0.134 / 0.106 / 0.104 ms
// (2^21 points).
template <int BYTES>
__host__ __device__ constexpr int col_log_cb(int log_r) {
    const int top = (BYTES == 8 ? 13 : 14) - log_r, lo = BYTES == 8 ? 1 : 2;
    const int cb = log_r <= 7 ? 10 - log_r : 3;
    return cb < top ? cb : top < lo ? lo : top;
}

// A tile is 2^LCB columns (col_log_cb) of a 2^LOGR-point transform, element (idx, v) at
// layout slot p((idx << LCB) + v).  Threads take sub-problems with v fastest,
// so a warp's global accesses cover 2^LCB consecutive elements of several rows.
template <class Ar, int LOGR>
struct ColCfg {
    static constexpr int LCB = col_log_cb<sizeof(typename Ar::T)>(LOGR);
    static constexpr int RLAST = LOGR < 4 ? LOGR : 4;
    static constexpr int NSUB = 1 << (LOGR + LCB - RLAST);
    static constexpr int NT = NSUB < 32 ? 32 : NSUB > 256 ? 256 : NSUB;
    static constexpr size_t smem = tile_elems((size_t)1 << (LOGR + LCB)) * sizeof(typename Ar::T);
    static constexpr int kMinCtas = resident_threads<Ar>() / NT;
};

// The tile's coefficients, as the first forward round reads them.
// CW: coefficient width in bits (16, 32 or 64); ncoef: 16- or 32-bit
// coefficients, or words (64-bit, an odd count's last high word is zero).
template <class Ar, int CW>
struct CoefLoad {
    using T = typename Ar::T;
    const char* __restrict__ limbs;
    uint32_t end;   // bytes of whole coefficients
    uint32_t lone;  // 64-bit: 1 if a single low word follows them
    bool al8;
    static constexpr int kBytes = CW / 8;
    __device__ __forceinline__ CoefLoad(const uint32_t* l, size_t nc)
        : limbs(reinterpret_cast<const char*>(l)) {
        end = (uint32_t)(CW == 64 ? nc >> 1 : nc) * kBytes;
        lone = CW == 64 ? (uint32_t)(nc & 1) : 0u;
        al8 = (reinterpret_cast<uintptr_t>(l) & 7u) == 0;
    }
    using Raw = typename std::conditional<
        CW == 64, uint64_t, typename std::conditional<CW == 32, uint32_t, uint16_t>::type>::type;
    // the coefficient at byte offset o, zero beyond the operand
    __device__ __forceinline__ Raw load(uint32_t o) const {
        if constexpr (CW != 64) {
            return o < end ? __ldg(reinterpret_cast<const Raw*>(limbs + o)) : (Raw)0;
        } else {
            uint64_t v = 0;
            const uint32_t* w = reinterpret_cast<const uint32_t*>(limbs + o);
            if (o < end) {
                if (al8) {
                    v = __ldg(reinterpret_cast<const unsigned long long*>(w));
                } else {
                    v = ((uint64_t)__ldg(w + 1) << 32) | __ldg(w);
                }
            } else if (o == end && lone) {
                v = __ldg(w);
            }
            return v;
        }
    }
    static __device__ __forceinline__ T residue(const Ar& ar, Raw v) {
        if constexpr (CW != 64) {
            return Ar::from_u32(v);
        } else {
            return ar.from_u64(v);
        }
    }
};

// Element at a byte offset of up to 2^32 from a CTA-uniform address: one add
// per access instead of a 64-bit address each.
template <typename T>
__device__ __forceinline__ T ld_off(const T* base, uint32_t o) {
    return __ldcg(reinterpret_cast<const T*>(reinterpret_cast<const char*>(base) + o));
}
template <typename T>
__device__ __forceinline__ void st_off(T* base, uint32_t o, T v) {
    *reinterpret_cast<T*>(reinterpret_cast<char*>(base) + o) = v;
}

// Forward column pass of one tile, operand and prime.  zt: the upper half of
// the rows is zero pad.  sum: where prime 0's CTAs sum the operand's words
// (64-bit coefficients).
template <class Ar, int LOGR, int CW>
__device__ __forceinline__ void fwd_col2_body(const PlanDev<Ar>& P,
                                              const uint32_t* __restrict__ limbs, size_t ncoef,
                                              typename Ar::T* res, bool zt, int tile, int kp,
                                              unsigned char* smem_raw, Sum* sum) {
    using T = typename Ar::T;
    using L = LayCol<T>;
    using Cfg = ColCfg<Ar, LOGR>;
    constexpr int LCB = Cfg::LCB;
    constexpr int RL0 = first_rl(LOGR), NT = Cfg::NT, CB = 1 << LCB;
    const int log_c = P.log_c + P.log_r2;
    const PrimeDev<Ar>& pr = P.pr[kp];
    const Ar ar = pr.ar;
    const uint32_t c0 = (uint32_t)tile << LCB;
    T* gout = res + ((size_t)kp << P.log_n) + c0;
    T* buf = reinterpret_cast<T*>(smem_raw);
    const CoefLoad<Ar, CW> coef(limbs, ncoef);
    uint64_t acc = 0;  // the words' sum (prime 0's CTAs)
    __shared__ SumParts parts;

    auto round = [&](auto s0_, auto rl_, auto zt_) {
        constexpr int S0 = decltype(s0_)::value, RL = decltype(rl_)::value;
        constexpr bool ZT = decltype(zt_)::value;
        constexpr bool FIRST = S0 == 0, LAST = S0 + RL == LOGR;
        constexpr int D = LOGR - S0 - RL, DS = D + LCB, N = 1 << (LOGR + LCB - RL);
        // the first round's loads run one sub-problem ahead of the arithmetic:
        // every thread takes several sub-problems, each a DRAM or L2 latency
        // (six primes at 2^23 words 0.408 -> 0.285 ms; long scoreboard stalls
        // 7.3 per issue before).  Not in double precision, whose 80 registers
        // have no room for it (0.225 -> 0.232 ms).
        constexpr int NL = 1 << (ZT ? RL - 1 : RL);  // coefficients loaded
        using Raw = typename CoefLoad<Ar, CW>::Raw;
        constexpr bool AHEAD =
            FIRST && N > NT && sizeof(T) == 4 && NL * sizeof(Raw) <= 64;
        Raw raw[FIRST ? NL : 1];
        auto load = [&](int sp) {
            const uint32_t v = sp & (CB - 1), j = sp >> LCB;  // g = 0
            const uint32_t o = ((j << log_c) + c0 + v) * coef.kBytes;
            const uint32_t step = ((uint32_t)coef.kBytes << D) << log_c;
#pragma unroll
            for (int k = 0; k < NL; ++k) raw[k] = coef.load(o + k * step);
        };
        if constexpr (AHEAD) load(threadIdx.x);
#pragma unroll 1
        for (int sp = threadIdx.x; sp < N; sp += NT) {
            const int v = sp & (CB - 1), rest = sp >> LCB;
            const int j = rest & ((1 << D) - 1), g = rest >> D;
            const int base = (g << (D + RL)) + j;
            const int p0 = L::p((base << LCB) + v);
            T x[1 << RL];
            if constexpr (FIRST) {
                if constexpr (!AHEAD) load(sp);
                if constexpr (CW == 64) {
                    if (kp == 0) {
#pragma unroll
                        for (int k = 0; k < NL; ++k) {
                            add_word(acc, (uint32_t)raw[k]);
                            add_word(acc, (uint32_t)(raw[k] >> 32));
                        }
                    }
                }
#pragma unroll
                for (int k = 0; k < NL; ++k) x[k] = CoefLoad<Ar, CW>::residue(ar, raw[k]);
                if constexpr (AHEAD) {
                    if (sp + NT < N) load(sp + NT);
                }
            } else {
#pragma unroll
                for (int k = 0; k < (1 << RL); ++k)
                    x[k] = buf[p0 + L::template off<false>(k, DS, 0)];
            }
            ct_round<Ar, RL, FIRST, ZT, !FIRST>(x, ar, RoundTw<T, (1 << S0), false>(pr.WRf, g));
            const uint32_t o = (((uint32_t)base << log_c) + v) * (uint32_t)sizeof(T);
            const uint32_t step = ((uint32_t)sizeof(T) << D) << log_c;
#pragma unroll
            for (int k = 0; k < (1 << RL); ++k) {
                if constexpr (LAST) {
                    st_off(gout, o + k * step, x[k]);
                } else {
                    buf[p0 + L::template off<false>(k, DS, 0)] = x[k];
                }
            }
        }
    };
    using std::false_type;
    using std::true_type;
    if (zt) {
        round(std::integral_constant<int, 0>{}, std::integral_constant<int, RL0>{}, true_type{});
    } else {
        round(std::integral_constant<int, 0>{}, std::integral_constant<int, RL0>{}, false_type{});
    }
    if constexpr (CW == 64) {
        if (kp == 0) sum_part(parts, acc);
    }
    if constexpr (LOGR > RL0 || CW == 64) __syncthreads();
    if constexpr (CW == 64) {
        if (kp == 0 && threadIdx.x < 32) sum_parts(sum, (uint32_t)tile, parts, NT / 32);
    }
    if constexpr (LOGR > RL0) {
        round(std::integral_constant<int, RL0>{}, std::integral_constant<int, 4>{}, false_type{});
    }
    if constexpr (LOGR > RL0 + 4) {
        __syncthreads();
        round(std::integral_constant<int, RL0 + 4>{}, std::integral_constant<int, 4>{},
              false_type{});
    }
    if constexpr (LOGR > RL0 + 8) {
        __syncthreads();
        round(std::integral_constant<int, RL0 + 8>{}, std::integral_constant<int, 4>{},
              false_type{});
    }
}

// blockIdx.x = tile * K + prime: the K CTAs of a tile run side by side, so the
// operand words come from L2 after the first of them.
template <class Ar, int LOGR, int CW>
__global__ void __launch_bounds__(ColCfg<Ar, LOGR>::NT, ColCfg<Ar, LOGR>::kMinCtas)
k_fwd_col2(const PlanDev<Ar> P, const uint32_t* __restrict__ limbs_a, size_t ncoef_a,
           const uint32_t* __restrict__ limbs_b, size_t ncoef_b, typename Ar::T* res_a,
           typename Ar::T* res_b, unsigned zt_mask, int tile0, Sum* __restrict__ sums) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    grid_release();
    const int op = blockIdx.z;
    fwd_col2_body<Ar, LOGR, CW>(P, op ? limbs_b : limbs_a, op ? ncoef_b : ncoef_a,
                                     op ? res_b : res_a, (zt_mask >> op) & 1u,
                                     tile0 + (int)(blockIdx.x / P.K), blockIdx.x % P.K, smem_raw,
                                     sums + op * kSumSlots);
}

// Inverse column pass of one tile and prime, in place, residues fully reduced.
template <class Ar, int LOGR>
__device__ __forceinline__ void inv_col2_body(const PlanDev<Ar>& P, typename Ar::T* res,
                                              CarryState* cst, int tile, int kp,
                                              unsigned char* smem_raw) {
    using T = typename Ar::T;
    using L = LayCol<T>;
    using Cfg = ColCfg<Ar, LOGR>;
    constexpr int LCB = Cfg::LCB;
    constexpr int RL0 = first_rl(LOGR), NT = Cfg::NT, CB = 1 << LCB;
    if (tile == 0 && kp == 0 && threadIdx.x == 0) cst->counter = cst->any = 0;
    const int log_c = P.log_c + P.log_r2;
    const PrimeDev<Ar>& pr = P.pr[kp];
    const Ar ar = pr.ar;
    T* g0 = res + ((size_t)kp << P.log_n) + ((size_t)tile << LCB);
    T* buf = reinterpret_cast<T*>(smem_raw);

    auto round = [&](auto s0_, auto rl_) {
        constexpr int S0 = decltype(s0_)::value, RL = decltype(rl_)::value;
        constexpr bool FIRST = S0 + RL == LOGR, LAST = S0 == 0;
        constexpr int D = LOGR - S0 - RL, DS = D + LCB, N = 1 << (LOGR + LCB - RL);
#pragma unroll 1
        for (int sp = threadIdx.x; sp < N; sp += NT) {
            const int v = sp & (CB - 1), rest = sp >> LCB;
            const int j = rest & ((1 << D) - 1), g = rest >> D;
            const int base = (g << (D + RL)) + j;
            const int p0 = L::p((base << LCB) + v);
            const uint32_t o = (((uint32_t)base << log_c) + v) * (uint32_t)sizeof(T);
            const uint32_t step = ((uint32_t)sizeof(T) << D) << log_c;
            T x[1 << RL];
#pragma unroll
            for (int k = 0; k < (1 << RL); ++k) {
                if constexpr (FIRST) {
                    x[k] = ld_off(g0, o + k * step);
                } else {
                    x[k] = buf[p0 + L::template off<false>(k, DS, 0)];
                }
            }
            gs_round<Ar, RL, LAST, true>(x, ar, RoundTw<T, (1 << S0), false>(pr.WRi, g));
#pragma unroll
            for (int k = 0; k < (1 << RL); ++k) {
                if constexpr (LAST) {
                    st_off(g0, o + k * step, ar.inv_out(x[k]));
                } else {
                    buf[p0 + L::template off<false>(k, DS, 0)] = x[k];
                }
            }
        }
    };
    if constexpr (LOGR > RL0 + 8) {
        round(std::integral_constant<int, RL0 + 8>{}, std::integral_constant<int, 4>{});
        __syncthreads();
    }
    if constexpr (LOGR > RL0 + 4) {
        round(std::integral_constant<int, RL0 + 4>{}, std::integral_constant<int, 4>{});
        __syncthreads();
    }
    if constexpr (LOGR > RL0) {
        round(std::integral_constant<int, RL0>{}, std::integral_constant<int, 4>{});
        __syncthreads();
    }
    round(std::integral_constant<int, 0>{}, std::integral_constant<int, RL0>{});
}

template <class Ar, int LOGR>
__global__ void __launch_bounds__(ColCfg<Ar, LOGR>::NT, ColCfg<Ar, LOGR>::kMinCtas)
k_inv_col2(const PlanDev<Ar> P, typename Ar::T* res, CarryState* cst) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    grid_release();
    grid_wait();
    inv_col2_body<Ar, LOGR>(P, res, cst, blockIdx.x, blockIdx.y, smem_raw);
}

// ------------------------------------------------------------------ middle
// Middle column pass of the three-pass schedule (n = R * R2 * C), fixed length
// R2 = 2^LOGR: sub-matrix s (blockIdx.y, k1 = bitrev(s) over R) is R2 rows of C
// columns; a CTA takes a tile of columns for one prime and operand.  The outer
// twiddle w_n^((i2 C + c) k1) is folded like a row's: zeta = w_n^(C k1) goes
// into the stage twiddles of the first rounds, and one table of 16 x 2^LCB
// factors zeta^j w_n^(c k1), applied before the last round, takes the rest --
// one multiplication per element instead of two, and the tile goes from global
// memory to registers and back without a staging pass.  The inverse mirrors it.
template <class Ar, int LOGR>
struct MidCfg : ColCfg<Ar, LOGR> {
    using Base = ColCfg<Ar, LOGR>;
    static constexpr int S1 = LOGR - 4, CB = 1 << Base::LCB;
    static constexpr size_t tables = ((1 << S1) + 16 * CB + 16) * sizeof(Tw<typename Ar::T>);
    static constexpr size_t smem = tables + Base::smem;
};

template <class Ar, int LOGR, bool INV>
__global__ void __launch_bounds__(ColCfg<Ar, LOGR>::NT, ColCfg<Ar, LOGR>::kMinCtas)
k_mid_col2(const PlanDev<Ar> P, typename Ar::T* res_a, typename Ar::T* res_b) {
    using T = typename Ar::T;
    using L = LayCol<T>;
    using Cfg = MidCfg<Ar, LOGR>;
    constexpr int LCB = ColCfg<Ar, LOGR>::LCB, CB = Cfg::CB, S1 = Cfg::S1;
    constexpr int RL0 = first_rl(LOGR), NT = ColCfg<Ar, LOGR>::NT;
    static_assert(LOGR > 4, "at least two rounds");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int log_c = P.log_c, s = blockIdx.y;
    const int kp = blockIdx.z % P.K, op = blockIdx.z / P.K;
    const PrimeDev<Ar>& pr = P.pr[kp];
    const Ar ar = pr.ar;
    const uint64_t c0 = (uint64_t)blockIdx.x << LCB;
    T* g0 = (op ? res_b : res_a) + ((size_t)kp << P.log_n) + ((size_t)s << (LOGR + log_c)) + c0;
    Tw<T>* R = reinterpret_cast<Tw<T>*>(smem_raw);  // stage twiddles of the first rounds
    Tw<T>* Z = R + (1 << S1);                       // [j][v]: zeta^j w_n^(c k1)
    Tw<T>* ZL = Z + 16 * CB;                        // zeta^(R2 / 2m) by stage
    T* buf = reinterpret_cast<T*>(smem_raw + Cfg::tables);
    const Tw<T>* W = INV ? pr.WMi : pr.WMf;
    {
        const uint64_t nmask = ((uint64_t)1 << P.log_n) - 1;
        const uint64_t k1 = bitrev((uint32_t)s, P.log_r);
        for (int i = threadIdx.x; i < 16 * CB + S1; i += NT) {
            uint64_t e = i < 16 * CB
                             ? (((uint64_t)(i >> LCB) << log_c) + c0 + (i & (CB - 1))) * k1
                             : ((uint64_t)1 << (LOGR - 1 - (i - 16 * CB) + log_c)) * k1;
            e &= nmask;
            if (INV) e = (nmask + 1 - e) & nmask;
            Z[i] = pow_entry(ar, e, P.lo_out, pr.OLf, pr.OHf);  // ZL follows Z
        }
        __syncthreads();
        for (int i = 1 + threadIdx.x; i < (1 << S1); i += NT) {
            const int st = stage_of_place(i, RL0);
            R[i] = ar.mul_tw(ZL[st], ld_tw(W + i));
        }
        __syncthreads();
    }
    auto round = [&](auto s0_, auto rl_) {
        constexpr int S0 = decltype(s0_)::value, RL = decltype(rl_)::value;
        constexpr bool LOW = S0 == 0, HIGH = S0 + RL == LOGR;  // first / last stages
        constexpr bool FROM_G = INV ? HIGH : LOW, TO_G = INV ? LOW : HIGH;
        constexpr int D = LOGR - S0 - RL, DS = D + LCB, N = 1 << (LOGR + LCB - RL);
#pragma unroll 1
        for (int sp = threadIdx.x; sp < N; sp += NT) {
            const int v = sp & (CB - 1), rest = sp >> LCB;
            const int j = rest & ((1 << D) - 1), g = rest >> D;
            const int base = (g << (D + RL)) + j;
            const int p0 = L::p((base << LCB) + v);
            const uint32_t o = (((uint32_t)base << log_c) + v) * (uint32_t)sizeof(T);
            const uint32_t step = ((uint32_t)sizeof(T) << D) << log_c;
            T x[1 << RL];
#pragma unroll
            for (int k = 0; k < (1 << RL); ++k) {
                if constexpr (FROM_G) {
                    x[k] = ld_off(g0, o + k * step);
                } else {
                    x[k] = buf[p0 + L::template off<false>(k, DS, 0)];
                }
                if constexpr (HIGH && !INV) x[k] = ar.mulc(x[k], ld_w<true>(Z + (k << LCB) + v));
            }
            if constexpr (HIGH) {
                const RoundTw<T, (1 << S0), false> tw(W, g);
                if constexpr (INV) {
                    gs_round<Ar, RL, false, false>(x, ar, tw);
                } else {
                    ct_round<Ar, RL, false, false, false>(x, ar, tw);
                }
            } else {
                const RoundTw<T, (1 << S0), true> tw(R, g);
                if constexpr (INV) {
                    gs_round<Ar, RL, false, true>(x, ar, tw);
                } else {
                    ct_round<Ar, RL, false, false, true>(x, ar, tw);
                }
            }
#pragma unroll
            for (int k = 0; k < (1 << RL); ++k) {
                if constexpr (HIGH && INV) x[k] = ar.mulc(x[k], ld_w<true>(Z + (k << LCB) + v));
                if constexpr (TO_G) {
                    st_off(g0, o + k * step, x[k]);
                } else {
                    buf[p0 + L::template off<false>(k, DS, 0)] = x[k];
                }
            }
        }
    };
    using std::integral_constant;
    constexpr bool MID1 = RL0 + 4 < LOGR, MID2 = RL0 + 8 < LOGR;  // rounds between
    if constexpr (!INV) {
        round(integral_constant<int, 0>{}, integral_constant<int, RL0>{});
        __syncthreads();
        if constexpr (MID1) {
            round(integral_constant<int, RL0>{}, integral_constant<int, 4>{});
            __syncthreads();
        }
        if constexpr (MID2) {
            round(integral_constant<int, RL0 + 4>{}, integral_constant<int, 4>{});
            __syncthreads();
        }
        round(integral_constant<int, S1>{}, integral_constant<int, 4>{});
    } else {
        round(integral_constant<int, S1>{}, integral_constant<int, 4>{});
        __syncthreads();
        if constexpr (MID2) {
            round(integral_constant<int, RL0 + 4>{}, integral_constant<int, 4>{});
            __syncthreads();
        }
        if constexpr (MID1) {
            round(integral_constant<int, RL0>{}, integral_constant<int, 4>{});
            __syncthreads();
        }
        round(integral_constant<int, 0>{}, integral_constant<int, RL0>{});
    }
}

// ------------------------------------------------------------------ batched
// The same passes with a product grid dimension.
// blockIdx.x = tile * K + prime, blockIdx.z = 2 * product + operand
template <class Ar, int LOGR, int CW>
__global__ void __launch_bounds__(ColCfg<Ar, LOGR>::NT, ColCfg<Ar, LOGR>::kMinCtas)
kb_fwd_col2(const PlanDev<Ar> P, const BatchProd* __restrict__ D, typename Ar::T* res_a,
            typename Ar::T* res_b) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const BatchProd d = D[blockIdx.z >> 1];
    const int op = blockIdx.z & 1;
    if (op && d.square) return;
    const size_t ncoef = (size_t)(op ? d.lb : d.la) * (CW == 16 ? 2 : 1);
    const size_t n = (size_t)1 << P.log_n;
    fwd_col2_body<Ar, LOGR, CW>(P, op ? d.b : d.a, ncoef, (op ? res_b : res_a) + d.res_off,
                                ncoef <= n / 2, blockIdx.x / P.K, blockIdx.x % P.K, smem_raw,
                                nullptr);
}

// blockIdx.x = row, .y = prime, .z = product
template <class Ar, int LOGC>
__global__ void __launch_bounds__(RowCfg<Ar, LOGC>::NT, RowCfg<Ar, LOGC>::kMinCtas)
kb_row2(const PlanDev<Ar> P, const BatchProd* __restrict__ D, typename Ar::T* res_a,
        const typename Ar::T* res_b) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const BatchProd d = D[blockIdx.z];
    row2_body<Ar, LOGC, false>(P, res_a + d.res_off, (d.square ? res_a : res_b) + d.res_off,
                               d.square != 0, blockIdx.x, blockIdx.y, smem_raw);
}

template <class Ar, int LOGR>
__global__ void __launch_bounds__(ColCfg<Ar, LOGR>::NT, ColCfg<Ar, LOGR>::kMinCtas)
kb_inv_col2(const PlanDev<Ar> P, const BatchProd* __restrict__ D, typename Ar::T* res_a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const BatchProd d = D[blockIdx.z];
    inv_col2_body<Ar, LOGR>(P, res_a + d.res_off, d.cst, blockIdx.x, blockIdx.y, smem_raw);
}

// ------------------------------------------------------------------ one CTA
// A whole product of up to 2^12 points in one CTA and one launch: transforms,
// pointwise product and inverse in shared memory, PG primes side by side (all
// of them for a single product, whose latency counts; one at a time in a
// batch, where the other CTAs fill the SM and shared memory is what limits
// them), then Garner and carry from the residues where they lie.  Against the
// 4-step kernels, five or six dependent launches of 2 to 10 us each with most
// of the chip idle.
// TH: threads; an item is one sub-problem of 16 elements of one operand and
// prime, and threads take items in turn.
// A single product takes it up to 2^11 points (measured alone, one CTA against
// 4-step: 9.1 / 14.8 us at 2^8, 10.6 / 14.7 at 2^11, 16.9 / 14.7 at 2^12), a
// batch up to 2^12 (267 products of 2^12 points on the 32-bit path 31 / 71 us,
// 265 on the 64-bit path 47 / 101).
constexpr int kOneMinLog = 4, kOneMaxLog = 12, kOneMaxLogSingle = 11;

template <class Ar, int LOGN>
struct OneCfg {
    static constexpr int G = 1 << (LOGN - 4);  // sub-problems per transform
    // shared memory with K primes, PG at a time: residues of every prime, and
    // the other operand of PG of them
    static size_t smem(int K, int PG) {
        return (size_t)(K + PG) * tile_elems(1 << LOGN) * sizeof(typename Ar::T);
    }
};

template <class Ar, int LOGN, int CW, int TH>
__device__ __forceinline__ void one_body(const PlanDev<Ar>& P, const uint32_t* a, uint32_t la,
                                         const uint32_t* b, uint32_t lb, uint32_t* out, bool sq,
                                         int pg, uint32_t* err, unsigned char* smem_raw) {
    using T = typename Ar::T;
    using L = LayRow2<T>;
    constexpr int N = 1 << LOGN, RL0 = first_rl(LOGN), G = OneCfg<Ar, LOGN>::G;
    constexpr int CPW = CW == 16 ? 2 : 1;
    constexpr int E = CW == 16 ? 4 : 8;  // words per thread in the carry pass
    const int tid = threadIdx.x, K = P.K;
    T* buf = reinterpret_cast<T*>(smem_raw);
    constexpr size_t TE = N + (N >> 4);
    auto bufA = [&](int k) { return buf + (size_t)k * TE; };
    auto bufB = [&](int s) { return buf + (size_t)(K + s) * TE; };  // s: slot of the group

    for (int k0 = 0; k0 < K; k0 += pg) {
        const int kn = min(pg, K - k0), ops = sq ? 1 : 2;
        // one round of every transform of the group: f(item's operand buffer,
        // prime, sub-problem)
        auto each = [&](int transforms, int nsub, auto f) {
#pragma unroll 1
            for (int it = tid; it < transforms * nsub; it += TH) {
                const int t = it / nsub, sp = it - t * nsub;
                f(t, sp);
            }
        };
        // ... with four items in flight: a short first round's operand loads
        auto each4 = [&](int transforms, int nsub, auto f) {
#pragma unroll 4
            for (int it = tid; it < transforms * nsub; it += TH) {
                const int t = it / nsub, sp = it - t * nsub;
                f(t, sp);
            }
        };
        // forward rounds but the last; the first reads the operands
        auto fwd = [&](auto s0_, auto rl_) {
            constexpr int S0 = decltype(s0_)::value, RL = decltype(rl_)::value;
            constexpr int D = LOGN - S0 - RL, NSUB = 1 << (LOGN - RL);
            auto body = [&](int t, int sp) {
                const int op = t >= kn ? 1 : 0, k = k0 + t - op * kn;
                T* dst = op ? bufB(k - k0) : bufA(k);
                const PrimeDev<Ar>& pr = P.pr[k];
                const Ar ar = pr.ar;
                int g, j;
                row_group<T, D, NSUB>(sp, g, j);
                const int base = (g << (D + RL)) + j;
                const int p0 = L::p(base);
                T x[1 << RL];
                if constexpr (S0 == 0) {
                    const CoefLoad<Ar, CW> coef(op ? b : a, (size_t)(op ? lb : la) * CPW);
#pragma unroll
                    for (int i = 0; i < (1 << RL); ++i)
                        x[i] = CoefLoad<Ar, CW>::residue(ar, coef.load((uint32_t)(base + (i << D)) * coef.kBytes));
                } else {
#pragma unroll
                    for (int i = 0; i < (1 << RL); ++i)
                        x[i] = dst[p0 + L::template off<false>(i, D, 0)];
                }
                ct_round<Ar, RL, S0 == 0, false, S0 != 0>(
                    x, ar, RoundTw<T, (1 << S0), false>(pr.WCf, g));
#pragma unroll
                for (int i = 0; i < (1 << RL); ++i)
                    dst[p0 + L::template off<false>(i, D, 0)] = x[i];
            };
            if constexpr (S0 == 0 && RL <= 2) {
                each4(kn * ops, NSUB, body);
            } else {
                each(kn * ops, NSUB, body);
            }
            __syncthreads();
        };
        using std::integral_constant;
        if constexpr (LOGN > 4) fwd(integral_constant<int, 0>{}, integral_constant<int, RL0>{});
        if constexpr (LOGN > 4 && RL0 + 4 < LOGN)
            fwd(integral_constant<int, RL0>{}, integral_constant<int, 4>{});
        // last forward round of both operands, product, first inverse round
        constexpr int SL = LOGN - 4;
        each(kn, G, [&](int t, int g) {
            const int k = k0 + t;
            const PrimeDev<Ar>& pr = P.pr[k];
            const Ar ar = pr.ar;
            T* A = bufA(k);
            T* B = bufB(t);
            const int p0 = L::p(g << 4);
            const RoundTw<T, (1 << SL), false> tf(pr.WCf, g), ti(pr.WCi, g);
            T x[16];
            auto last = [&](const T* src, const uint32_t* limbs, uint32_t len) {
                if constexpr (SL == 0) {
                    const CoefLoad<Ar, CW> coef(limbs, (size_t)len * CPW);
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        x[i] = CoefLoad<Ar, CW>::residue(ar, coef.load((uint32_t)i * coef.kBytes));
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i) x[i] = src[p0 + L::template off<false>(i, 0, 0)];
                }
                ct_round<Ar, 4, SL == 0, false, SL != 0>(x, ar, tf);
            };
            last(A, a, la);
            if (sq) {
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const T v = ar.fwd_to_2p(x[i]);
                    x[i] = ar.pointwise(v, v);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) A[p0 + i] = ar.fwd_to_2p(x[i]);
                last(B, b, lb);
#pragma unroll
                for (int i = 0; i < 16; ++i) x[i] = ar.pointwise(x[i], A[p0 + i]);
            }
            gs_round<Ar, 4, SL == 0, true>(x, ar, ti);
#pragma unroll
            for (int i = 0; i < 16; ++i) A[p0 + i] = SL == 0 ? ar.scale_out(x[i], pr.scale) : x[i];
        });
        __syncthreads();
        // remaining inverse rounds; the last one scales and reduces
        auto inv = [&](auto s0_, auto rl_) {
            constexpr int S0 = decltype(s0_)::value, RL = decltype(rl_)::value;
            constexpr int D = LOGN - S0 - RL, NSUB = 1 << (LOGN - RL);
            each(kn, NSUB, [&](int t, int sp) {
                const PrimeDev<Ar>& pr = P.pr[k0 + t];
                const Ar ar = pr.ar;
                T* A = bufA(k0 + t);
                int g, j;
                row_group<T, D, NSUB>(sp, g, j);
                const int p0 = L::p((g << (D + RL)) + j);
                T x[1 << RL];
#pragma unroll
                for (int i = 0; i < (1 << RL); ++i) x[i] = A[p0 + L::template off<false>(i, D, 0)];
                gs_round<Ar, RL, S0 == 0, true>(x, ar, RoundTw<T, (1 << S0), false>(pr.WCi, g));
#pragma unroll
                for (int i = 0; i < (1 << RL); ++i)
                    A[p0 + L::template off<false>(i, D, 0)] =
                        S0 == 0 ? ar.scale_out(x[i], pr.scale) : x[i];
            });
            __syncthreads();
        };
        if constexpr (LOGN > 4 && RL0 + 4 < LOGN)
            inv(integral_constant<int, RL0>{}, integral_constant<int, 4>{});
        if constexpr (LOGN > 4) inv(integral_constant<int, 0>{}, integral_constant<int, RL0>{});
    }

    // ---- Garner + carry, tile by tile; the carry into a tile is the previous
    // tile's last carry words (s_cin) plus its chain carry-out bit (s_eps)
    __shared__ uint32_t s_w[TH / 32];
    __shared__ uint32_t s_lastx[TH / 32][3];
    __shared__ uint32_t s_cin[3];
    __shared__ uint32_t s_eps;
    const int lane = tid & 31, warp = tid >> 5;
    const uint32_t NLW = N / CPW, M = la + lb;
    const uint32_t words = NLW > M ? NLW : M;
    if (tid == 0) {
        s_cin[0] = s_cin[1] = s_cin[2] = 0;
        s_eps = 0;
    }
    __syncthreads();
    uint32_t bad = 0;
    for (uint32_t t0 = 0; t0 < words; t0 += TH * E) {
        const uint32_t j0 = t0 + tid * E;
        T r[kDigitPrimes][E * CPW];
#pragma unroll
        for (int k = 0; k < kDigitPrimes; ++k)
#pragma unroll
            for (int q = 0; q < E * CPW; ++q)
                r[k][q] = k < K && j0 < NLW ? bufA(k)[L::p(j0 * CPW) + L::p(q)] : T(0);
        unsigned __int128 Dg[E];
        garner_combine<Ar, CW == 16, E>(P, r, Dg, &bad);
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
                const uint64_t v = (uint64_t)l[e] + (e < 3 ? PX[e] : 0u) + c;
                S[e] = (uint32_t)v;
                c = v >> 32;
                all &= S[e];
            }
            st = c ? 2 : (all == 0xffffffffu ? 1 : 0);
        }
        const ChainMasks cm = chain_prepare(st, s_w);
        __syncthreads();
        const uint32_t eps_in = s_eps;
        const uint32_t mc = chain_mine(cm, s_w, eps_in);
        const uint32_t cout = chain_out(s_w, eps_in, TH / 32);
        {
            uint64_t c = mc;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const uint64_t v = (uint64_t)S[e] + c;
                if (j0 + e < M) out[j0 + e] = (uint32_t)v;
                c = v >> 32;
            }
        }
        if (t0 + TH * E >= words) break;
        __syncthreads();  // every thread has read s_cin, s_eps, s_lastx, s_w
        if (tid == TH - 1) {
            s_cin[0] = X[0];
            s_cin[1] = X[1];
            s_cin[2] = X[2];
        }
        if (tid == 0) s_eps = cout;
        __syncthreads();
    }
    if (bad) atomicOr(err, 2u);
}

// A single product (all primes side by side).
template <class Ar, int LOGN, int CW, int TH>
__global__ void __launch_bounds__(TH)
k_one(const PlanDev<Ar> P, const uint32_t* __restrict__ a, uint32_t la,
      const uint32_t* __restrict__ b, uint32_t lb, uint32_t* __restrict__ out, int square,
      uint32_t* __restrict__ err) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    one_body<Ar, LOGN, CW, TH>(P, a, la, b, lb, out, square != 0, P.K, err, smem_raw);
}

// Batched: blockIdx.x = product.
template <class Ar, int LOGN, int CW, int TH>
__global__ void __launch_bounds__(TH, (sizeof(typename Ar::T) == 8 ? 768 : 1024) / TH)
kb_one(const PlanDev<Ar> P, const BatchProd* __restrict__ D, uint32_t* __restrict__ err) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const BatchProd d = D[blockIdx.x];
    one_body<Ar, LOGN, CW, TH>(P, d.a, d.la, d.square ? d.a : d.b, d.lb, d.out, d.square != 0, 1,
                               err, smem_raw);
}

}  // namespace bw
