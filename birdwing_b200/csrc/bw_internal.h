// bw_internal.h -- plan layout shared by the library's translation units.
#pragma once
#include <cstddef>
#include <cstdint>
#include <mutex>

#include "bw_host.h"

#include "bw_kernels.cuh"

// Stage order of the host-pointer products of one plan.  Contexts of one
// plan used in turn form a three-stage pipeline (copy-in, kernels,
// copy-out): each stage of a product waits for the same stage of the plan's
// previous product, so every stage runs alone at full speed while the three
// overlap.  Unordered, the products in flight share the PCIe link and the SMs
// evenly and finish together, and the copies hide little of the kernels.
// Only plans with more than one live context order their products.
struct bw_stage_order {
    std::mutex mu;
    int contexts = 0;              // live contexts of the plan
    cudaEvent_t last[3] = {};      // end of the previous product's stage i
    const void* owner[3] = {};     // context that recorded last[i]
};

struct bw_plan {
    int path = 0, K = 0;
    size_t la = 0, lb = 0, nca = 0, ncb = 0;
    int log_n = 0, log_r = 0, log_c = 0, log_cb = 0, lo = 0;
    int log_cb1 = 0;     // forward column pass tile width (its own shared-memory budget)
    int tw_smem_r = 0;   // column stage twiddles staged in shared memory
    int log_r2 = 0;      // three-pass schedule: middle column length (0: two passes)
    int log_cb2 = 0, lo_out = 0;
    int small = 0;       // single-pass plan: the whole n-point transform in one CTA
    int w64 = 0;         // 64-bit coefficients (two words each): K = 3 on the 64-bit
                         // path, K = 6 on the 32-bit path
    int coef_half = 0;   // ... prime loop: both operands in the low half, half the u64 copy
    int device = 0;
    bool zt_a = false, zt_b = false;
    void* d_tables = nullptr;
    size_t table_bytes = 0;
    bw::PlanDev<bw::Ar32> pd32{};
    bw::PlanDev<bw::Ar64> pd64{};
    // double-precision transforms (64-bit path, 64-bit coefficients): 0 off,
    // 1 primes just above 2^50, 2 primes just above 2^51.66 (pd64 then holds
    // the Garner constants of the same primes)
    int f64 = 0;
    // passes with compile-time lengths (bw_ntt.cuh); their tables are stored in
    // round order
    int v2_rows = 0, v2_cols = 0, v2_mid = 0, v2_one = 0;
    bool no_v2_one = false;  // set before bw_plan_setup: tables in stage order (kq_small)
    // a single product of at most 2^12 points with 16-bit coefficients and no
    // tuning flags: one CTA (k_one), with its own n-point tables
    bool one = false;
    bw::PlanDev<bw::Ar32> pd_one{};
    bw::PlanDev<bw::ArD<0>> pdd0{};
    bw::PlanDev<bw::ArD<1>> pdd1{};
    uint64_t primes[bw::kMaxPrimes] = {};
    bw_stage_order* order = nullptr;  // plans of bw_plan_create only
};

// Split, tables and constants of a plan for transform length 2^log_n.
// mode 0: the 4-step pipeline (two or three passes) for batch groups;
// mode 1: single-pass products of one CTA each (n-point stage tables and the
// n^-1 scale); mode 2: the 4-step pipeline for one product at a time, with
// column tiles narrowed for small n so that the column passes fill the SMs.
int bw_plan_setup(bw_plan* pl, int path, int K, int log_n, unsigned flags, int mode);

// bw_plan_create with the arithmetic of 64-bit coefficients on the 64-bit path
// named (0: 58-bit integer primes, 2: the second double-precision set, -1: by
// the operands), for tests: left to itself a plan takes the integers above 2^27
// coefficients of the shorter operand and the second set above 2^22.
extern "C" int bw_plan_create_arith(bw_plan** out, int path, size_t la, size_t lb, int num_primes,
                                    unsigned flags, int arith);

// Largest transform of a launch group: the two-pass schedule.
constexpr int kMaxGroupLogN = 26;

// One launch group: np products of one plan (equal path, K and transform
// length), product q described by d_desc[q].  A single-pass plan (small)
// runs kb_one, one CTA per product (beyond 2^12 points ks_product, with residue
// scratch res_a, np * K * n elements); a 4-step plan runs kb_fwd_col2, kb_row2,
// kb_inv_col2 (or their any-length forms) and a carry over residue arenas res_a
// and res_b of the same size, with per-product carry state (zeroed before the
// launch, epoch 1).
struct bw_group_launch {
    const bw_plan* plan;
    const bw::BatchProd* d_desc;
    unsigned np;
    void* res_a;
    void* res_b;
    size_t ntiles;      // carry tiles per product (bw_group_ntiles)
    uint32_t* d_err;    // bit 0: look-back wait timed out; bit 1: check failed
    int spin_limit;
    bool inject_wait_fault = false;  // test hook: every look-back wait runs out
    bool inject_residue_fault = false;  // test hook (4-step): residue 0 of product 0 is residue 1
};
// np 0: nothing is launched, the kernels that the plan's groups run are loaded.
int bw_enqueue_group(const bw_group_launch& g, cudaStream_t s);
// Carry form of a 4-step group.  Few tiles (at most the chip holds at once): the
// look-back form, one launch, whose waits are short there -- a serving group's
// cost is its launches on the host.  Also for the test hook that makes the
// waits run out.
inline bool bw_group_lookback(const bw_group_launch& g) {
    return g.inject_wait_fault || g.np * g.ntiles <= 3 * 148;
}
// Kernels bw_enqueue_group launches for a group.
inline int bw_group_kernels(const bw_group_launch& g) {
    if (g.plan->small) return 1;
    return bw_group_lookback(g) || g.ntiles <= 1 ? 4 : 5;
}
// ... of one arithmetic (bw_group_*.cu).
template <class Ar, bool SPLIT16>
cudaError_t bw_enqueue_group_of(const bw_group_launch& g, cudaStream_t s);
// One product in one CTA (plans with `one`).
cudaError_t bw_launch_one(const bw_plan* pl, const uint32_t* a, const uint32_t* b, uint32_t* out,
                          bool square, uint32_t* err, cudaStream_t s);
// Carry tiles of a group whose longest product has max_words output words.
size_t bw_group_ntiles(int path, int log_n, size_t max_words);
// Bytes of one product's look-back state (16-byte multiple).
size_t bw_group_state_stride(size_t ntiles);
// Kernel form (single-pass or 4-step) and 4-step split for a transform
// length, from the tune table (bw_batch_autotune / bw_tune_table_set).
void bw_tune_lookup(int path, int K, int log_n, int* small, int* log_cols);
// Point a descriptor's look-back fields into its state block.
void bw_group_fill_state(bw::BatchProd& d, unsigned char* state, size_t ntiles);

// Most chunks a host copy is split into (see bw_ctx::copy_chunks).
constexpr int kMaxCopyChunks = 16;

struct bw_ctx {
    const bw_plan* plan = nullptr;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    void* d_res_a = nullptr;
    void* d_res_b = nullptr;
    uint32_t* d_in = nullptr;   // staging: a then b
    uint32_t* d_out = nullptr;  // staging: product
    unsigned char* d_state = nullptr;
    size_t state_bytes = 0;
    bw::CarryState* cst = nullptr;
    uint32_t* err = nullptr;
    uint4* rec_x = nullptr;
    uint32_t* rec_s = nullptr;
    bw::Sum* sums = nullptr;    // word sums (64-bit coefficients)
    size_t ntiles = 0;
    // look-back record tag of the last product that used the look-back carry
    uint32_t epoch = 1;
    cudaGraphExec_t gexec = nullptr;  // device-pointer product, replayed while
    const void* g_a = nullptr;        // the pointers stay the same
    const void* g_b = nullptr;
    const void* g_out = nullptr;
    bool g_sq = false;
    uint32_t* h_err = nullptr;  // pinned
    cudaEvent_t ev[8] = {};
    cudaEvent_t stage_ev[3] = {};  // ends of copy-in, kernels, copy-out (stage order)
    bool counted = false;          // included in the plan's live contexts
    // host copies split into chunks that overlap the first and last kernels
    // (created on first use): copy-in on in_stream, copy-out on out_stream
    int copy_chunks = 0;           // 0: automatic, 1: whole copies on the stream
    cudaStream_t in_stream = nullptr, out_stream = nullptr;
    cudaEvent_t in_ev[kMaxCopyChunks] = {}, out_ev[kMaxCopyChunks] = {};
    cudaEvent_t ready_ev = nullptr, out_done_ev = nullptr;
    int out_pieces = 0;            // K4 launches of the last chunked product
    size_t out_tiles_per = 0;      // carry tiles per K4 launch
    int spin_limit = 1 << 22;
    bool inject_wait_fault = false;
    bool inject_residue_fault = false;  // residue fault_at of prime 0 is its neighbour's
    size_t fault_at = 0;
};

// Stage order of one host-pointer product (bw_stage_order): begin(i, s)
// makes stream s wait for stage i of the plan's previous product; end(i, s)
// records this product's stage i on s.  Off with one live context.  A
// previous product of the same context needs no wait: every stream of a
// product starts behind the context stream, which ends behind all of the
// previous product's work.
struct StageOrder {
    bw_stage_order* so = nullptr;
    const bw_ctx* c = nullptr;
    bool on = false;
    cudaError_t begin(int i, cudaStream_t s) const {
        if (!on || !so->last[i] || so->owner[i] == c) return cudaSuccess;
        return cudaStreamWaitEvent(s, so->last[i], 0);
    }
    cudaError_t end(int i, cudaStream_t s) const {
        if (!on) return cudaSuccess;
        const cudaError_t e = cudaEventRecord(c->stage_ev[i], s);
        so->last[i] = c->stage_ev[i];
        so->owner[i] = c;
        return e;
    }
};

// Host operands of a product whose copy-in is split into `chunks` column
// blocks: block k holds the words of forward-column tiles
// [k T/chunks, (k+1) T/chunks) of every row, and K1 runs over those tiles
// as soon as the block has landed.
struct HostIO {
    const uint32_t* ha = nullptr;
    const uint32_t* hb = nullptr;  // nullptr when squaring
    int chunks = 1;
    const StageOrder* order = nullptr;
};

// Return a failed CUDA call's status from a function that returns one.
#define BW_CUDA(call)                                                                   \
    do {                                                                                \
        cudaError_t e_ = (call);                                                        \
        if (e_ != cudaSuccess) {                                                        \
            return bw_fail(e_ == cudaErrorMemoryAllocation ? BW_ENOMEM : BW_ECUDA,      \
                           "%s failed: %s", #call, cudaGetErrorString(e_));             \
        }                                                                               \
    } while (0)

namespace bw {

// A plan's device view in one arithmetic.
template <class Ar>
const PlanDev<Ar>& plan_dev(const bw_plan* pl);
template <>
inline const PlanDev<Ar32>& plan_dev<Ar32>(const bw_plan* pl) {
    return pl->pd32;
}
template <>
inline const PlanDev<Ar64>& plan_dev<Ar64>(const bw_plan* pl) {
    return pl->pd64;
}
template <>
inline const PlanDev<ArD<0>>& plan_dev<ArD<0>>(const bw_plan* pl) {
    return pl->pdd0;
}
template <>
inline const PlanDev<ArD<1>>& plan_dev<ArD<1>>(const bw_plan* pl) {
    return pl->pdd1;
}

// Launch a kernel behind the previous one in the stream.  early: it may start
// while that one's last CTAs run (programmatic dependent launch); the kernel
// must then run grid_wait() before it reads what that one writes.  Not for a
// product's first kernel, which reads operands of the caller's.
template <class... P, class... A>
cudaError_t launch_after(bool early, void (*kern)(P...), dim3 grid, unsigned block, size_t smem,
                         cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

// Enqueue K1..K3 (the transform part) for one product.  With io (chunks > 1)
// the operands' copy-in runs on the context's copy stream in column blocks
// and K1 runs block by block behind it.
template <class Ar, bool SPLIT16, bool W64 = false>
int bw_enqueue_transform(bw_ctx* c, const uint32_t* a, const uint32_t* b, bool square,
                         bool timing, const HostIO* io = nullptr);
// Set the dynamic shared-memory limit of one arithmetic's kernels (once).
template <class Ar, bool SPLIT16>
int bw_set_transform_attrs();

}  // namespace bw
