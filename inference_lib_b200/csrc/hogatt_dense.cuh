// Dense attention on the 5th-generation tensor cores (tcgen05): calls with many query rows per kv head -- prompts,
// causal chunks -- where the op is bound by the tensor pipe and the exponentials instead of HBM (16-token chunks of 8
// workers with GQA 8 are 1,024 rows per kv head: about 1,000 flop per K/V byte).  One kernel for fragment tensors
// and (PAGED) for packed queries over a paged cache.
//
// Decomposition.  Query rows are cut into tiles of 128 (the MMA's M).  A block is two tiles that read the same keys, a
// unit is (block, kv head).  dense_plan_kernel finds, per tile and fragment, how many keys any of its rows sees; a
// block walks only those, 128 keys per step -- of a causal prompt just over half (4,000 tokens: 543 us per call when
// every block walked every key, 152 now) -- and the steps of all units are one list that a persistent grid of one
// CTA per SM cuts into balanced contiguous ranges.  A unit that lies inside one range is normalised and stored by
// its CTA; where units are cut into a few parts, the CTA that finishes last folds the partials of the others, else they are
// left to dense_merge_kernel.
//
// A step.  Both tiles of the block use the K and V tile (64 KiB of copies per 16.8 MFLOP; each tile alone would be at
// the SM's L2 bandwidth).  Where a block has only one tile, the second softmax group takes every other key tile
// of the same queries instead, and the two halves are two partials.
//   warp 16  query and K copies (TMA, rings of 2 and 3 tiles)      warp 19  the walk over the steps, V copies (ring of 2)
//   warp 17  S = Q K^T: one S buffer in tensor memory, used by the two groups in turn
//   warp 18  O_g += P_g V, P as the tensor-memory A operand
//   warps 0-7 / 8-15  softmax of group 0 / 1: two threads per query row, 64 columns each (with one, which has 128
//            exponentials in a row, a 1,024-row chunk call took 128 us instead of 122).  The scores go to registers at once, which frees the S buffer for the other
//            group's product; the halves of a row need each other's maximum only when the row's scale has to change, and
//            each other's sum at the end.  The groups run half a step apart: one's tensor-memory round trips and waits lie
//            under the other's exponentials.
// Tensor memory, all 512 columns: O_0, O_1 (128 each), S (128), P_0, P_1 (64 each: two 16-bit probabilities a column).
// Issuing one tcgen05.mma costs the issuing thread 60-70 cycles, hence two issuing threads.  O is rescaled in tensor
// memory only when a row's maximum has grown by more than 2^8 since the scale it is stored at (then exp2 arguments
// stay below 8); the stored scale travels with the partial, so the merge is exact.
//
// Every wait is bounded.  The reference has no counterpart: its kernel gives every (kv head, worker, token) its own
// CTAs and re-reads the KV once per (worker, token) on CUDA cores (src/kernels/kernel_v21.cuh:62-66,957-964).
#pragma once
#include <cuda.h>
#include <limits.h>

#include "hogatt_device.cuh"
#include "hogatt_merge.cuh"

namespace hogatt {

constexpr int kDenseMaxFragments = 16;      // tensor maps travel in the kernel arguments
constexpr int kDenseRows = 128;             // query rows per tile (MMA M)
constexpr int kDenseTile = 128;             // keys per tile (MMA N of S, K of PV)
constexpr int kDenseBlock = 2 * kDenseRows;
constexpr int kDenseSoftmaxWarps = 16;      // two groups of eight: one group per query tile, two threads per row
constexpr int kDenseThreads = (kDenseSoftmaxWarps + 4) * 32;
constexpr int kDensePlanThreads = 1024;
constexpr int kDenseMaxCtas = 256;
constexpr int kDenseMergeWarps = 8;         // warps per CTA of the merge step; with many partials per row they share a row's
constexpr int kDenseMergeBatch = 4;         // partials of a row that a thread of it has in flight (one in the lean instantiation)
// Where no unit has more CTAs than this, the last CTA of a unit to finish folds the others' partials into its own rows, 128 KiB of
// each, and nothing of it is left to the merge step (which then ends 1.5 us after the attention kernel instead of 12).  us per
// call, folded up to 3 / merged: three parts at most (3 x 256 tokens, 5,700 keys, G = 5) 111.5 / 117.5, a 4,000-token prompt 134 /
// 145 (a line at 2: 134).  Two more conditions, both for all units of a call:
//   * one unit of more CTAs makes the call wait for the merge step anyway, which then gets every shared unit (512 tokens, 4,000
//     packed keys, 64 units of which two have four CTAs: 49.4; folding the others as well 53.2; with a line at 4 50.2);
//   * where the steps do not fill the SMs, the merge step's CTAs are resident on the idle ones before the attention kernel ends
//     (128 tokens, 512 packed keys 22.7, folded 26.4).
// The two halves that one CTA leaves of a block of one tile are always folded there (six single tokens beside two chunks of 512
// tokens: 112, in the merge step 120).
constexpr int kDenseFoldParts = 3;
constexpr int kDenseFoldInts = 20;          // per unit: first CTA, CTAs (0: not folded there), two unused, arrivals left of 16 warps

struct alignas(64) DenseMaps {
    CUtensorMap q;                          // rotated queries as [F, W, Hq, S, E] or [F, W, Hkv, G*S, E]; paged: [F, total_q, Hkv, G, E]
    CUtensorMap k[kDenseMaxFragments];      // fragments: [Hkv, rows, E] each; paged: k[0] = [blocks, Hkv, block_size, E]
    CUtensorMap v[kDenseMaxFragments];
};

struct DenseArgs {
    int F, W, Hq, Hkv, G, S;
    int tiles;             // query tiles per kv head (paged: upper bound)
    int blocks;            // blocks per kv head: pairs of tiles (paged: upper bound)
    int tile_span;         // fragments: workers per tile (G*S <= 128) or tiles per worker; paged: query tokens per tile
    int tile_tokens;       // fragments, G*S > 128: tokens per tile, all G heads of each (0: 128 consecutive rows, token fastest)
    int total_q;           // paged: packed query tokens
    int block_size, max_blocks;
    float l2scale;         // scale * log2(e)
    int cap[kDenseMaxFragments];     // rows of the fragment tensors (or the host's bound); unused when paged
    const int* loc;        // [F, W, S] or [F, total_q]
    const int* flen;       // [F] (may be null) or [F, W]
    const int* cu;         // paged: [W + 1]
    const int* block_table;
    // the plan, written by dense_plan_kernel
    long long* pre;        // [blocks + 1] steps of the blocks before block b, per kv head
    long long* cost;       // [blocks + 1] the same with the units' fixed costs (used by the plan kernel alone)
    int* vis;              // [2 * blocks][F] visible keys per (tile, fragment)
    int4* start;           // [ctas] block, kv head, step inside the unit, steps of this CTA
    int4* merge;           // [blocks * Hkv] units left to the merge step: unit, first CTA, partials, one query tile
    int* fold;             // [blocks * Hkv][kDenseFoldInts], written for units that more than one CTA, or two halves of one, work on
    int* nmerge;           // [0] units on that list; [1] a CTA of the attention kernel gave up a wait: the call's result is void
    int4* rec;             // paged: [blocks] worker, first token, tokens
    // Partials.  The one CTA c leaves of unit u is slot c + u (both only ever grow along the list).  Four columns of a row are one
    // element and the rows are contiguous: a warp, one row per lane, stores and loads 512 consecutive bytes.
    float4* ws_o;          // [slots][128 / 4][256]
    float* ws_m;           // [slots][256]
    float* ws_l;
    int ctas;              // the grid; CTAs that get work: as many of them as there are steps
    int* status;
    void* out;             // [W, Hq, S, 128] or [total_q, Hq, 128]
    int world, rank;       // > 0: every finished row goes to the full-size output of every rank
    void* peer_out[HOGATT_MAX_PEERS];
};

struct DenseCfg {
    static constexpr int HD = 128;
    static constexpr int ATOM_BYTES = 128 * 128;            // [128 rows][64 16-bit columns], rows of 128 bytes, swizzled
    static constexpr int TILE_BYTES = 2 * ATOM_BYTES;       // a 128 x 128 operand tile: two column halves
    static constexpr int NQ = 2, NK = 3, NV = 2;            // rings of query, K and V tiles
    static constexpr int OFF_Q = 0;
    static constexpr int OFF_K = OFF_Q + NQ * TILE_BYTES;
    static constexpr int OFF_V = OFF_K + NK * TILE_BYTES;
    static constexpr int OFF_BAR = OFF_V + NV * TILE_BYTES;                 // 224 KiB of tiles
    static constexpr int OFF_STAT = OFF_BAR;                                // [2 groups][2 halves][128 rows]: maxima or sums handed over
    // barriers: q_full[NQ], q_empty[NQ], k_full[NK], k_empty[NK], v_full[NV], v_empty[NV], s_full[2], s_free, p_full[2], o_done[2],
    // segment full / empty
    static constexpr int NBAR = 2 * NQ + 2 * NK + 2 * NV + 2 + 1 + 2 + 2 + 2 * 4;
    static constexpr int OFF_MBAR = OFF_STAT + 2 * 2 * kDenseRows * 4;
    static constexpr int OFF_SEG = (OFF_MBAR + NBAR * 8 + 15) / 16 * 16;
    static constexpr int OFF_MISC = OFF_SEG + 4 * 32;                       // tmem base
    static constexpr int OFF_END = OFF_MISC + 16;
    static constexpr int TMEM_COLS = 512;
    static constexpr int COL_O = 0, COL_S = 256, COL_P = 384;               // O_g at 128 g, P_g at 384 + 64 g
};

constexpr size_t kDenseSmemBytes = DenseCfg::OFF_END;       // (227 KiB is all there is: dynamic shared memory starts on a 1 KiB boundary)

// ---- tcgen05 / TMA wrappers -------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// arrive on `bar` once every MMA this thread has issued so far has completed
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// D[tmem] (+)= A[smem] * B[smem], 128 x N x 16, fp32 accumulate
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// D[tmem] (+)= A[tmem] * B[smem]: A is 128 rows (lanes) x 16 k (8 columns, two 16-bit elements each, lower k in the low half)
__device__ __forceinline__ void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Shared-memory matrix descriptor, 128-byte swizzle: start address, leading / stride byte offsets in 16-byte units,
// descriptor version 1 (bits 46-47), layout type 2 = SWIZZLE_128B (bits 61-63).
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo_bytes >> 4) << 16) | ((uint64_t)(sbo_bytes >> 4) << 32) |
           (1ull << 46) | (2ull << 61);
}
// Instruction descriptor, kind::f16: fp32 accumulator (bits 4-5 = 1), A/B format (bits 7-9, 10-12: 0 f16, 1 bf16),
// A K-major, B K-major or MN-major (bit 16), N >> 3 (bits 17-22), M >> 4 (bits 24-28).
template <class T>
__host__ __device__ constexpr uint32_t umma_idesc(bool b_mn_major, int m, int n) {
    const uint32_t fmt = sizeof(T) == 2 && std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
    return (1u << 4) | (fmt << 7) | (fmt << 10) | ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, int c4,
                                            uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(bar)
        : "memory");
}

// 32 consecutive fp32 columns of this thread's tensor-memory lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t* r = reinterpret_cast<uint32_t*>(v);
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
// 2^x, the hardware approximation (about two units in the last place); -inf gives 0
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// 16 consecutive 32-bit columns of this thread's tensor-memory lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
                 "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
// 32 bytes (a whole sector) in one store, 32-byte aligned
__device__ __forceinline__ void store_sector(void* dst, const uint32_t (&v)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]),
                 "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Kernels that move registers between warps (setmaxnreg) cannot have calls, and the roles' loops together have to stay in
// the instruction cache: with the timer of mbar_wait_bounded inlined at every wait the kernel was 70 KB and twice as slow.
__device__ __forceinline__ bool mbar_wait_polls(uint32_t bar, uint32_t parity, int* status, int bit) {
    const bool ok = wait_polls(bar, parity);
    if (!ok && status) atomicOr(status, bit);
    return ok;
}
// bar.red over the two warps on hardware barrier `id`: is `x` true in any of their threads
__device__ __forceinline__ bool pair_any(int id, bool x) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %2, 0;\n\tbarrier.cta.red.or.pred q, %1, 64, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(r) : "r"(id), "r"((uint32_t)x) : "memory");
    return r != 0;
}
// one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

// ---- geometry ----------------------------------------------------------------------------------------------------
// Fragments: a tile holds whole workers (tile_span of them), or tile_tokens tokens of one worker with all their heads, so
// that its rows end at nearly the same key of a causal prompt; where G does not divide 128, 128 consecutive rows of a
// worker, tokens fastest.  Paged: a tile is tile_span tokens of one worker's packed run, G rows each.
struct DenseRow {
    bool valid;
    int w, g, s;           // s: token of the worker (fragments), packed token index (paged)
};
template <bool PAGED>
__device__ __forceinline__ DenseRow dense_row(const DenseArgs& a, int tile, int i, const int4& rec) {
    DenseRow r;
    if constexpr (PAGED) {
        const int tok = (tile & 1) * a.tile_span + i / a.G;
        r.valid = i < a.tile_span * a.G && tok < rec.z;
        r.w = rec.x;
        r.g = i % a.G;
        r.s = rec.y + tok;
    } else if (a.tile_tokens > 0) {
        r.w = tile / a.tile_span;
        r.g = i / a.tile_tokens;
        r.s = (tile - r.w * a.tile_span) * a.tile_tokens + i - r.g * a.tile_tokens;
        r.valid = r.w < a.W && r.s < a.S;
    } else {
        const int gs = a.G * a.S;
        int x = i;
        if (gs > kDenseRows) {
            r.w = tile / a.tile_span;
            x += (tile - r.w * a.tile_span) * kDenseRows;
        } else {
            r.w = tile * a.tile_span + i / gs;
            x = i % gs;
        }
        r.valid = r.w < a.W && x < gs && (gs > kDenseRows || i < a.tile_span * gs);
        r.g = x / a.S;
        r.s = x - r.g * a.S;
    }
    return r;
}
// rows of fragment f that hold keys and values (worker w's, when paged)
template <bool PAGED>
__device__ __forceinline__ int dense_length(const DenseArgs& a, int f, int w) {
    if constexpr (PAGED) return a.flen[f * a.W + w];
    return a.flen ? min(a.cap[f], a.flen[f]) : a.cap[f];
}
template <bool PAGED>
__device__ __forceinline__ int dense_location(const DenseArgs& a, int f, const DenseRow& r) {
    if constexpr (PAGED) return a.loc[(size_t)f * a.total_q + r.s];
    return a.loc[((size_t)f * a.W + r.w) * a.S + r.s];
}
// does block b hold one query tile only (its groups then take every other key tile each)
template <bool PAGED>
__device__ __forceinline__ bool dense_single(const DenseArgs& a, int b) {
    if constexpr (PAGED) return a.rec[b].z <= a.tile_span;
    return 2 * b + 1 >= a.tiles;
}
__device__ __forceinline__ int dense_steps(int vis0, int vis1, bool single) {
    return single ? (vis0 + 2 * kDenseTile - 1) / (2 * kDenseTile) : (max(vis0, vis1) + kDenseTile - 1) / kDenseTile;
}

// ---- the plan: one CTA, beside the rotation kernel where there is one ----------------------------------------------
// Writes what the other two kernels would otherwise each have to search for: visible keys per (tile, fragment), the prefix
// of steps over blocks, where every CTA starts, and which units are left to the merge step.  The arrays stay in shared
// memory while they are worked on, if they fit.
constexpr int kDensePlanVis = 4096, kDensePlanBlocks = 1024, kDensePlanRecs = 512;
template <bool PAGED>
__global__ void __launch_bounds__(kDensePlanThreads) dense_plan_kernel(const __grid_constant__ DenseArgs a) {
    __shared__ int s_vis[kDensePlanVis];
    __shared__ long long s_pre[kDensePlanBlocks + 1], s_cost[kDensePlanBlocks + 1], sums[kDensePlanThreads / 32], pos[kDenseMaxCtas + 1];
    __shared__ int4 s_rec[PAGED ? kDensePlanRecs : 1];
    __shared__ int s_list, s_most;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = kDensePlanThreads / 32;
    if (tid == 0) s_list = s_most = 0;
    pdl_wait();
    // The rotation kernel writes nothing that is read here.  It starts at once and makes the loads below slower, but its own
    // time is what the attention kernel waits for (let go behind them it began 4 us later: 4,000 tokens 25 -> 15 us to the end
    // of both, together with end_after_predecessor).  A packed call has no rotation: the attention kernel is let in behind the
    // loads (0.2 us of every such call: 512 tokens of 2,000 keys 39.3 us with its CTAs there before, 39.1 now).
    if constexpr (!PAGED) pdl_trigger();
    // exclusive prefix of one value per thread over the CTA; *total gets the sum
    auto scan = [&](long long v, long long* total) {
        long long x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        __syncthreads();
        if (lane == 31) sums[warp] = x;
        __syncthreads();
        long long w = sums[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        *total = __shfl_sync(0xffffffffu, w, 31);
        const long long before = __shfl_sync(0xffffffffu, w, warp > 0 ? warp - 1 : 0);
        return (warp > 0 ? before : 0) + x - v;
    };
    int nb = a.blocks;
    if constexpr (PAGED) {
        const int per = (a.W + kDensePlanThreads - 1) / kDensePlanThreads, w0 = min(tid * per, a.W), w1 = min(w0 + per, a.W);
        const int span = 2 * a.tile_span;
        long long mine = 0, total;
        for (int w = w0; w < w1; ++w) mine += (max(0, a.cu[w + 1] - a.cu[w]) + span - 1) / span;
        long long at = scan(mine, &total);
        nb = (int)min(total, (long long)a.blocks);
        for (int w = w0; w < w1; ++w) {
            const int first = a.cu[w], tokens = a.cu[w + 1] - first;
            for (int s = 0; s < tokens; s += span, ++at)
                if (at < a.blocks) {
                    const int4 r = make_int4(w, first + s, min(span, tokens - s), 0);
                    a.rec[at] = r;
                    if (at < kDensePlanRecs) s_rec[at] = r;
                }
        }
        __syncthreads();
    }
    auto record = [&](int b) { return b < kDensePlanRecs ? s_rec[b] : a.rec[b]; };
    auto single_block = [&](int b) {
        if constexpr (PAGED) return record(b).z <= a.tile_span;
        return dense_single<PAGED>(a, b);
    };
    const bool small = nb <= kDensePlanBlocks && 2 * nb * (long long)a.F <= kDensePlanVis;
    int* const vis = small ? s_vis : a.vis;
    long long* const pre = small ? s_pre : a.pre;
    long long* const cost = small ? s_cost : a.cost;
#pragma unroll 4
    for (int i = warp; i < 2 * nb * a.F; i += nwarps) {
        // Which tokens a tile's rows are: a run of locations (of one worker's tokens, round its end, if it has more
        // than 128 rows).  Heads repeat the tokens, so no more than 128 locations are read.
        const int tile = i / a.F, f = i - tile * a.F;
        int from, tokens, wrap = INT_MAX, w = 0;      // locations [from, from + tokens); those at or past `wrap` are a.S further down
        if constexpr (PAGED) {
            const int4 rec = record(tile >> 1);
            const int skip = (tile & 1) * a.tile_span;
            from = rec.y + skip;
            tokens = min(a.tile_span, rec.z - skip);
            w = rec.x;
        } else {
            const int gs = a.G * a.S;
            if (a.tile_tokens > 0) {
                w = tile / a.tile_span;
                const int s0 = (tile - w * a.tile_span) * a.tile_tokens;
                tokens = w < a.W ? min(a.tile_tokens, a.S - s0) : 0;
                from = w * a.S + s0;
            } else if (gs > kDenseRows) {
                w = tile / a.tile_span;
                const int x = (tile - w * a.tile_span) * kDenseRows;
                tokens = w < a.W ? min(min(kDenseRows, gs - x), a.S) : 0;
                from = w * a.S + x % a.S;
                wrap = (w + 1) * a.S;
            } else {
                w = tile * a.tile_span;
                from = w * a.S;
                tokens = (min(w + a.tile_span, a.W) - w) * a.S;
            }
        }
        int top = -1;
        const int* loc = a.loc + (size_t)f * (PAGED ? a.total_q : a.W * a.S);
#pragma unroll
        for (int k = 0; k < kDenseRows; k += 32) {
            int at = from + k + lane;
            if (at >= wrap) at -= a.S;
            if (k + lane < tokens) top = max(top, loc[at]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
        top = tokens > 0 ? max(0, min(top, dense_length<PAGED>(a, f, w) - 1) + 1) : 0;
        if (lane == 0) a.vis[i] = vis[i] = top;
    }
    __syncthreads();
    if constexpr (PAGED) pdl_trigger();
    const int per = (nb + kDensePlanThreads - 1) / kDensePlanThreads, b0 = min(tid * per, nb), b1 = min(b0 + per, nb);
    auto block_steps = [&](int b) {
        const bool single = single_block(b);
        long long n = 0;
        for (int f = 0; f < a.F; ++f) n += dense_steps(vis[2 * b * a.F + f], vis[(2 * b + 1) * a.F + f], single);
        return n;
    };
    long long mine = 0, mine_cost = 0, total, total_cost;
    bool singles = false;
    for (int b = b0; b < b1; ++b) {
        const long long n = block_steps(b);
        mine += n;
        mine_cost += dense_cost(n, single_block(b));
        singles |= single_block(b);
    }
    long long at = scan(mine, &total), at_cost = scan(mine_cost, &total_cost);
    for (int b = b0; b < b1; ++b) {
        const long long n = per == 1 ? mine : block_steps(b);
        a.pre[b] = pre[b] = at;
        cost[b] = at_cost;
        at += n;
        at_cost += dense_cost(n, single_block(b));
    }
    if (tid == 0) {
        a.pre[nb] = pre[nb] = total;
        cost[nb] = total_cost;
    }
    singles = __syncthreads_or(singles);

    // Where every CTA starts: equal shares of the steps and of the units' fixed costs.  pos[c]: its first step in the list of all.
    const long long N = total * a.Hkv, C = total_cost * a.Hkv;
    const int ctas = dense_ctas(N, C, singles, a.ctas);
    int4 st = make_int4(0, 0, 0, 0);
    if (tid < ctas) {
        DenseStart d;
        pos[tid] = dense_share_start(pre, cost, nb, a.Hkv, single_block, cta_first_tile(tid, C, ctas), &d);
        st = make_int4(d.block, d.head, d.step, 0);
    }
    if (tid == ctas) pos[ctas] = N;
    __syncthreads();
    int parts = 0;                               // CTAs of the unit this one starts inside of, if no earlier CTA does
    if (tid < ctas) {
        st.w = (int)(pos[tid + 1] - pos[tid]);
        const long long s = pos[tid] - st.z;
        if (st.z > 0 && pos[tid - 1] <= s) {
            parts = dense_parts(pos, ctas, tid - 1, s + pre[st.x + 1] - pre[st.x]);
            atomicMax(&s_most, parts);
        }
    }
    __syncthreads();
    // Who folds unit u, which `count` CTAs from `first` on work on (in a block of one tile, two halves each).
    const bool few = s_most <= kDenseFoldParts && ctas == a.ctas;
    auto leave = [&](int u, int first, int count, bool single) {
        int4* const fold = reinterpret_cast<int4*>(a.fold + (size_t)u * kDenseFoldInts);
        const int here = count == 1 || few ? count : 0, left = single ? 2 * here : here;
        fold[0] = make_int4(first, here, 0, 0);
        if (here > 0) {
#pragma unroll
            for (int i = 1; i < kDenseFoldInts / 4; ++i) fold[i] = make_int4(left, left, left, left);
        } else {
            a.merge[atomicAdd(&s_list, 1)] = make_int4(u, first, single ? 2 * count : count, single ? 1 : 0);
        }
    };
    if (tid < a.ctas) {
        if (parts > 0 && !single_block(st.x)) leave(st.x * a.Hkv + st.y, tid - 1, parts, false);
        a.start[tid] = st;
    }
    // blocks of one tile (two halves per CTA that worked on them), blocks that see nothing.  (A thread per unit: with one per
    // block, 8 kv heads were 8,000-9,000 cycles of searches in a row; two 512-token chunks beside six single tokens: the plan
    // takes 8.2 us instead of 12.3.)
    for (long long u = tid; u < (long long)nb * a.Hkv; u += kDensePlanThreads) {
        const int b = (int)floor_div(u, a.Hkv), h = (int)(u - (long long)b * a.Hkv);
        const bool single = single_block(b);
        const long long steps = pre[b + 1] - pre[b];
        if (!single && steps > 0) continue;
        if (steps > 0) {
            const long long s = pre[b] * a.Hkv + h * steps;
            const int c0 = dense_first_cta(pos, ctas, s);
            leave((int)u, c0, dense_parts(pos, ctas, c0, s + steps), true);
        } else {
            a.merge[atomicAdd(&s_list, 1)] = make_int4((int)u, 0, 0, single ? 1 : 0);
        }
    }
    __syncthreads();
    if (tid == 0) {
        a.nmerge[0] = s_list;
        a.nmerge[1] = 0;
    }
}

// element offset of an output row
template <bool PAGED>
__device__ __forceinline__ size_t dense_out_offset(const DenseArgs& a, const DenseRow& r, int h) {
    const int hq = h * a.G + r.g;
    if constexpr (PAGED) return ((size_t)r.s * a.Hq + hq) * 128;
    const int all = max(a.world, 1) * a.Hq, off = a.world > 0 ? a.rank * a.Hq : 0;
    return (((size_t)r.w * all + off + hq) * a.S + r.s) * 128;
}

// ---- the walk over this CTA's share, segment by segment ----------------------------------------------------------------
// A segment is a run of steps of one unit inside one fragment.  Its key tiles are [t0, t1); in a block with one query
// tile, group g takes the tiles of parity g.  One warp walks (a step of it is two or three dependent loads) and hands
// the segments to the others through a small ring in shared memory, one segment ahead.
struct DenseSegment {
    int b, h, f, flags;
    int vis0, vis1;        // keys that the rows of query tile 0 / 1 see
    int t0, t1;            // key tiles
    static constexpr int SINGLE = 1, FIRST = 2, LAST = 4, WHOLE = 8, END = 16;
    __device__ __forceinline__ bool single() const { return flags & SINGLE; }         // one query tile
    __device__ __forceinline__ bool first() const { return flags & FIRST; }           // first segment of this CTA's share of the unit
    __device__ __forceinline__ bool last() const { return flags & LAST; }             // last one
    __device__ __forceinline__ bool whole() const { return flags & WHOLE; }           // the share is the whole unit
    // does group g work on key tile t
    __device__ __forceinline__ bool active(int g, int t) const { return single() ? (t & 1) == g : t * kDenseTile < (g ? vis1 : vis0); }
};
struct DenseSegments {     // a consumer's end of the ring (every lane of the warp takes part)
    static constexpr int DEPTH = 4;
    uint32_t slots, full, empty, n;
    __device__ __forceinline__ bool next(DenseSegment& d, int lane, int* status, bool& ok) {
        const uint32_t i = n % DEPTH;
        const bool come = mbar_wait_polls(full + 8 * i, (n / DEPTH) & 1u, status, STATUS_WAIT_SYNC_TIMEOUT);
        if (!__all_sync(0xffffffffu, come)) {
            ok = false;
            return false;
        }
        const uint32_t at = slots + i * (uint32_t)sizeof(DenseSegment);
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(d.b), "=r"(d.h), "=r"(d.f), "=r"(d.flags) : "r"(at) : "memory");
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(d.vis0), "=r"(d.vis1), "=r"(d.t0), "=r"(d.t1) : "r"(at + 16) : "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(empty + 8 * i);
        ++n;
        return !(d.flags & DenseSegment::END);
    }
};
template <bool PAGED>
struct DenseWalk {
    const DenseArgs& a;
    int b, h, f, vis0, vis1, t0, t1;
    bool single, first, last, whole;
    int j, n, left, skip;
    __device__ __forceinline__ DenseWalk(const DenseArgs& a_, const int4& start)
        : a(a_), b(start.x), h(start.y - 1), last(true), j(start.z), n(start.w) {}
    __device__ __forceinline__ bool next() {
        if (last) {
            if (n <= 0) return false;
            if (++h == a.Hkv) {
                h = 0;
                ++b;
                while (a.pre[b + 1] == a.pre[b]) ++b;                // (blocks that see nothing have no steps)
            }
            const int rest = (int)min(a.pre[b + 1] - a.pre[b] - j, (long long)INT_MAX);
            single = dense_single<PAGED>(a, b);
            whole = j == 0 && n >= rest;
            left = min(n, rest);
            n -= left;
            skip = j;
            j = 0;
            f = -1;
        }
        first = last;
        int steps, j0;
        do {
            ++f;
            vis0 = a.vis[2 * b * a.F + f];
            vis1 = a.vis[(2 * b + 1) * a.F + f];
            steps = dense_steps(vis0, vis1, single);
            j0 = min(skip, steps);
            skip -= j0;
        } while (j0 == steps);
        steps = min(steps - j0, left);
        left -= steps;
        last = left == 0;
        t0 = single ? 2 * j0 : j0;
        t1 = single ? min(2 * (j0 + steps), (vis0 + kDenseTile - 1) / kDenseTile) : j0 + steps;
        return true;
    }
};

// One K or V tile (keys tok0 .. tok0 + 127 of fragment f) of kv head h into shared memory.  Whole warp.
template <bool PAGED>
__device__ __forceinline__ void dense_fetch(const DenseArgs& a, const CUtensorMap* maps, int f, int w, int h, int tok0, uint32_t dst,
                                            uint32_t bar, int lane) {
    using C = DenseCfg;
    if constexpr (PAGED) {
        // a lane per (cache block, column half); blocks past the sequence's end are not fetched
        const int step = min(a.block_size, kDenseTile);
        const int rows = min(kDenseTile, a.flen[f * a.W + w] - tok0), n = (rows + step - 1) / step;
        const int i = lane >> 1, half = lane & 1;
        const int tok = tok0 + i * step, blk = tok / a.block_size;
        int place = 0;
        if (i < n) place = a.block_table[(size_t)w * a.max_blocks + min(blk, a.max_blocks - 1)];
        if (lane == 0) mbar_arrive_expect_tx(bar, (uint32_t)n * step * 256u);
        __syncwarp();
        if (i < n) tma_load_4d(dst + half * C::ATOM_BYTES + i * step * 128, maps, half * 64, tok - blk * a.block_size, h, place, bar);
    } else {
        if (lane == 0) {
            mbar_arrive_expect_tx(bar, C::TILE_BYTES);
            tma_load_3d(dst, maps + f, 0, tok0, h, bar);
            tma_load_3d(dst + C::ATOM_BYTES, maps + f, 64, tok0, h, bar);
        }
    }
}

template <class T, bool PAGED>
__global__ void __launch_bounds__(kDenseThreads, 1)
dense_attention_kernel(const __grid_constant__ DenseArgs a, const __grid_constant__ DenseMaps maps) {
    using C = DenseCfg;
    extern __shared__ __align__(1024) unsigned char dense_smem[];       // swizzled tiles start on 1 KiB boundaries
    unsigned char* const base = dense_smem;
    const uint32_t sbase = smem_u32(base);
    const uint32_t q_full = sbase + C::OFF_MBAR, q_empty = q_full + 8 * C::NQ, k_full = q_empty + 8 * C::NQ, k_empty = k_full + 8 * C::NK, v_full = k_empty + 8 * C::NK,
                   v_empty = v_full + 8 * C::NV, s_full = v_empty + 8 * C::NV, s_free = s_full + 16, p_full = s_free + 8,
                   o_done = p_full + 16, seg_full = o_done + 16, seg_empty = seg_full + 8 * DenseSegments::DEPTH;
    constexpr int W_K = kDenseSoftmaxWarps, W_S = W_K + 1, W_V = W_K + 3;        // (W_K + 2: the PV products)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(base + C::OFF_MISC);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int s = 0; s < C::NQ; ++s) {
            mbar_init(q_full + 8 * s, 1);
            mbar_init(q_empty + 8 * s, 1);
        }
        for (int s = 0; s < C::NK; ++s) {
            mbar_init(k_full + 8 * s, 1);
            mbar_init(k_empty + 8 * s, 1);
        }
        for (int s = 0; s < C::NV; ++s) {
            mbar_init(v_full + 8 * s, 1);
            mbar_init(v_empty + 8 * s, 1);
        }
        for (int g = 0; g < 2; ++g) {
            mbar_init(s_full + 8 * g, 1);
            mbar_init(p_full + 8 * g, kDenseSoftmaxWarps / 2);            // one arrival per softmax warp of the group
            mbar_init(o_done + 8 * g, 1);
        }
        mbar_init(s_free, kDenseSoftmaxWarps / 2);
        for (int i = 0; i < DenseSegments::DEPTH; ++i) {
            mbar_init(seg_full + 8 * i, 1);
            mbar_init(seg_empty + 8 * i, kDenseSoftmaxWarps + 3);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async_smem();
    }
    if (warp == W_S) tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_wait();             // rotated queries, plan
    pdl_trigger();
    DenseSegments segs{sbase + C::OFF_SEG, seg_full, seg_empty, 0};
    DenseSegment d;
    bool ok = true;

    if (warp >= W_K) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
        if (warp == W_K) {
            // ============================== query and K copies ==============================
            int stage = 0, q_slot = 0;
            uint32_t phase = 1, q_phase = 1;         // of k_empty and q_empty: the first round finds every stage free
            const int gs = a.G * a.S;
            const uint32_t q_bytes = (uint32_t)(PAGED ? a.tile_span * a.G : (gs > kDenseRows ? kDenseRows : a.tile_span * gs)) * 256u;
            while (ok && segs.next(d, lane, a.status, ok)) {
                const int w = PAGED ? a.rec[d.b].x : 0;
#pragma unroll 1
                for (int t = d.t0; t < d.t1; ++t) {
                    ok = mbar_wait_polls(k_empty + 8 * stage, phase, a.status, STATUS_WAIT_EMPTY_TIMEOUT);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    dense_fetch<PAGED>(a, maps.k, d.f, w, d.h, t * kDenseTile, sbase + C::OFF_K + stage * C::TILE_BYTES, k_full + 8 * stage, lane);
                    if (++stage == C::NK) {
                        stage = 0;
                        phase ^= 1u;
                    }
                    // The segment's query tiles, behind its first K tile: each as soon as the last product with the one before it
                    // in its place has finished.
#pragma unroll 1
                    for (int part = 0; t == d.t0 && part < (d.single() ? 1 : 2); ++part) {
                        ok = mbar_wait_polls(q_empty + 8 * q_slot, q_phase, a.status, STATUS_WAIT_EMPTY_TIMEOUT);
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) break;
                        if (elect_one()) {
                            const uint32_t bar = q_full + 8 * q_slot;
                            mbar_arrive_expect_tx(bar, q_bytes);
#pragma unroll 1
                            for (int i = 0; i < 2; ++i) {               // column halves
                                const uint32_t dst = sbase + C::OFF_Q + q_slot * C::TILE_BYTES + i * C::ATOM_BYTES;
                                const int tile = 2 * d.b + part;
                                if constexpr (PAGED) {
                                    tma_load_5d(dst, &maps.q, i * 64, 0, d.h, a.rec[d.b].y + part * a.tile_span, d.f, bar);
                                } else if (a.tile_tokens > 0) {
                                    const int qw = tile / a.tile_span;
                                    tma_load_5d(dst, &maps.q, i * 64, (tile - qw * a.tile_span) * a.tile_tokens, d.h * a.G, qw, d.f, bar);
                                } else {
                                    const int qw = gs > kDenseRows ? tile / a.tile_span : tile * a.tile_span;
                                    tma_load_5d(dst, &maps.q, i * 64, gs > kDenseRows ? (tile - qw * a.tile_span) * kDenseRows : 0, d.h, qw, d.f, bar);
                                }
                            }
                        }
                        __syncwarp();
                        if (++q_slot == C::NQ) {
                            q_slot = 0;
                            q_phase ^= 1u;
                        }
                    }
                    if (!ok) break;
                }
            }
        } else if (warp == W_V) {
            // ============================== the walk, and the V copies ==============================
            DenseWalk<PAGED> walk(a, a.start[blockIdx.x]);
            uint32_t n = 0;
            auto publish = [&]() {                   // the walk's next segment into the ring; false when there is none left
                const uint32_t i = n % DenseSegments::DEPTH;
                ok = mbar_wait_polls(seg_empty + 8 * i, ((n / DenseSegments::DEPTH) & 1u) ^ 1u, a.status, STATUS_WAIT_EMPTY_TIMEOUT) && ok;
                ok = __all_sync(0xffffffffu, ok);
                const bool more = walk.next();
                if (lane == 0) {
                    DenseSegment* slot = reinterpret_cast<DenseSegment*>(base + C::OFF_SEG) + i;
                    slot->b = walk.b;
                    slot->h = walk.h;
                    slot->f = walk.f;
                    slot->flags = more ? (walk.single ? DenseSegment::SINGLE : 0) | (walk.first ? DenseSegment::FIRST : 0) |
                                             (walk.last ? DenseSegment::LAST : 0) | (walk.whole ? DenseSegment::WHOLE : 0)
                                       : DenseSegment::END;
                    slot->vis0 = walk.vis0;
                    slot->vis1 = walk.vis1;
                    slot->t0 = walk.t0;
                    slot->t1 = walk.t1;
                    mbar_arrive(seg_full + 8 * i);
                }
                __syncwarp();
                ++n;
                return more;
            };
            int stage = 0;
            uint32_t phase = 1;
            bool more = publish();
#pragma unroll 1
            while (ok && more) {
                const int f = walk.f, h = walk.h, t0 = walk.t0, t1 = walk.t1, w = PAGED ? a.rec[walk.b].x : 0;
                more = publish();
#pragma unroll 1
                for (int t = t0; t < t1 && ok; ++t) {
                    ok = mbar_wait_polls(v_empty + 8 * stage, phase, a.status, STATUS_WAIT_EMPTY_TIMEOUT);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    dense_fetch<PAGED>(a, maps.v, f, w, h, t * kDenseTile, sbase + C::OFF_V + stage * C::TILE_BYTES, v_full + 8 * stage, lane);
                    if (++stage == C::NV) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
        } else if (warp == W_S) {
            // ============================== the S MMAs ==============================
            constexpr uint32_t IDESC_S = umma_idesc<T>(false, kDenseRows, kDenseTile);
            // (a k-step only moves the descriptor's start-address field: +32 bytes inside a 64-column swizzle atom,
            // +16 KiB to the second atom)
            const uint64_t q_desc = umma_desc(sbase + C::OFF_Q, 16, 1024), k_desc = umma_desc(sbase + C::OFF_K, 16, 1024);
            int stage = 0, q_slot = 0;
            uint32_t k_phase = 0, q_phase = 0, s_phase = 1;
            while (ok && segs.next(d, lane, a.status, ok)) {
                // this segment's places in the ring of query tiles
                const int slot0 = q_slot, slot1 = slot0 + 1 == C::NQ ? 0 : slot0 + 1;
                const uint32_t phase0 = q_phase, phase1 = slot1 == 0 ? q_phase ^ 1u : q_phase;
#pragma unroll 1
                for (int t = d.t0; t < d.t1 && ok; ++t) {
                    ok = mbar_wait_polls(k_full + 8 * stage, k_phase, a.status, STATUS_WAIT_FULL_TIMEOUT);
                    const uint64_t kd = k_desc + (uint64_t)(uint32_t)(stage * (C::TILE_BYTES >> 4));
#pragma unroll 1
                    for (int g = 0; g < 2; ++g) {
                        const int slot = g && !d.single() ? slot1 : slot0;
                        if (t == d.t0) ok = mbar_wait_polls(q_full + 8 * slot, g && !d.single() ? phase1 : phase0, a.status, STATUS_WAIT_FULL_TIMEOUT) && ok;
                        if (d.active(g, t)) {
                            // S = Q K^T into the S buffer once the scores before it have been read
                            ok = mbar_wait_polls(s_free, s_phase, a.status, STATUS_WAIT_SYNC_TIMEOUT) && ok;
                            ok = __all_sync(0xffffffffu, ok);
                            if (!ok) break;
                            s_phase ^= 1u;
                            tc_fence_after();
                            const uint64_t qd = q_desc + (uint64_t)(uint32_t)(slot * (C::TILE_BYTES >> 4));
                            if (elect_one()) {
#pragma unroll
                                for (int kk = 0; kk < C::HD / 16; ++kk) {
                                    const uint64_t off = (uint64_t)(((kk >> 2) * C::ATOM_BYTES + (kk & 3) * 32) >> 4);
                                    tc_mma(tmem + C::COL_S, qd + off, kd + off, IDESC_S, kk > 0);
                                }
                                tc_commit(s_full + 8 * g);
                            }
                            __syncwarp();
                        }
                        // a query tile is done with when the products so far are (in a block of one tile, the second group's)
                        if (t == d.t1 - 1 && g >= (int)d.single()) {
                            if (elect_one()) tc_commit(q_empty + 8 * slot);
                            __syncwarp();
                        }
                    }
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    if (elect_one()) tc_commit(k_empty + 8 * stage);
                    __syncwarp();
                    if (++stage == C::NK) {
                        stage = 0;
                        k_phase ^= 1u;
                    }
                }
                q_slot += d.single() ? 1 : 2;
                if (q_slot >= C::NQ) {
                    q_slot -= C::NQ;
                    q_phase ^= 1u;
                }
            }
        } else {
            // ============================== the O += P V MMAs ==============================
            constexpr uint32_t IDESC_O = umma_idesc<T>(true, kDenseRows, C::HD);
            const uint64_t v_desc = umma_desc(sbase + C::OFF_V, C::ATOM_BYTES, 1024);
            int stage = 0;
            uint32_t v_phase = 0, g_phase = 0, started = 0;      // bit g: parity of P_g; O_g holds something
            while (ok && segs.next(d, lane, a.status, ok)) {
                if (d.first()) started = 0;
                const int vlen = max(d.vis0, d.vis1);
#pragma unroll 1
                for (int t = d.t0; t < d.t1 && ok; ++t) {
                    ok = __all_sync(0xffffffffu, mbar_wait_polls(v_full + 8 * stage, v_phase, a.status, STATUS_WAIT_FULL_TIMEOUT));
                    if ((t + 1) * kDenseTile > vlen && ok) {
                        // The tile runs past the keys that any row of the block sees: what follows may hold anything (spare
                        // rows of a slab or cache block).  Those probabilities are exactly zero, but 0 * NaN would poison O.
                        unsigned char* vt = base + C::OFF_V + stage * C::TILE_BYTES;
#pragma unroll 1
                        for (int i = (vlen - t * kDenseTile) * 8 + lane; i < kDenseTile * 8; i += 32) {
                            *reinterpret_cast<int4*>(vt + i * 16) = make_int4(0, 0, 0, 0);
                            *reinterpret_cast<int4*>(vt + C::ATOM_BYTES + i * 16) = make_int4(0, 0, 0, 0);
                        }
                        fence_proxy_async_smem();      // generic-proxy writes before the MMA's async-proxy reads
                        __syncwarp();
                    }
                    const uint64_t vd = v_desc + (uint64_t)(uint32_t)(stage * (C::TILE_BYTES >> 4));
#pragma unroll 1
                    for (int g = 0; g < 2; ++g) {
                        if (!d.active(g, t)) continue;
                        ok = mbar_wait_polls(p_full + 8 * g, (g_phase >> g) & 1u, a.status, STATUS_WAIT_SYNC_TIMEOUT) && ok;
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) break;
                        g_phase ^= 1u << g;
                        tc_fence_after();
                        const uint32_t acc = (started >> g) & 1u;
                        if (elect_one()) {
#pragma unroll
                            for (int kk = 0; kk < kDenseTile / 16; ++kk) {
                                // A = P from tensor memory: 16 keys are 8 columns.  V is [key][Ev]: Ev (the MMA's N) is
                                // contiguous -> MN-major; 16 keys per step = two 8-key swizzle atoms (2 KiB)
                                tc_mma_ts(tmem + C::COL_O + g * 128, tmem + C::COL_P + g * 64 + kk * 8, vd + (uint64_t)(kk * 2048 >> 4), IDESC_O,
                                          kk > 0 ? 1u : acc);
                            }
                            tc_commit(o_done + 8 * g);
                        }
                        __syncwarp();
                        started |= 1u << g;
                    }
                    if (!ok) break;
                    if (elect_one()) tc_commit(v_empty + 8 * stage);
                    __syncwarp();
                    if (++stage == C::NV) {
                        stage = 0;
                        v_phase ^= 1u;
                    }
                }
            }
        }
    } else {
        // ============================== softmax: warps 0-7 group 0, 8-15 group 1; warps w and w + 4 share 32 rows ==============================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
        constexpr int COLS = kDenseTile / 2;                              // this thread's columns of S, P and O
        const int g = warp >> 3, half = (warp >> 2) & 1, row = (warp & 3) * 32 + lane;            // row of the tile == tensor-memory lane
        const uint32_t lane_base = tmem + (((uint32_t)((warp & 3) * 32)) << 16);
        const uint32_t s_addr = lane_base + C::COL_S + half * COLS, o_addr = lane_base + C::COL_O + g * 128 + half * COLS,
                       p_addr = lane_base + C::COL_P + g * 64 + half * (COLS / 2);
        float* const stat = reinterpret_cast<float*>(base + C::OFF_STAT) + (g * 2 + half) * kDenseRows + row;
        const float* const other = reinterpret_cast<const float*>(base + C::OFF_STAT) + (g * 2 + (half ^ 1)) * kDenseRows + row;
        const int pair_bar = 1 + g * 4 + (warp & 3);                      // hardware barrier of the two warps that share rows
        const float scale2 = a.l2scale;                        // scores are raw dot products; exp2((s - m) * scale2)
        const float grow_by = 8.f / scale2;                    // raw-score distance that equals a factor 2^8
        float m_run = -INFINITY, l_run = 0.f;                  // running max (raw, the row's) and sum (of this half's columns)
        uint32_t phase = 0;                                    // parity of this group's next S; its last PV has the other one
        bool any = false, ever = false;                        // has worked on a tile of this unit; at all
        DenseRow id = {false, 0, 0, 0};
        // The two warps of a pair leave together, also when a wait has run out: a barrier the other one never reaches
        // could not be given up.
        while (true) {
            const bool more = segs.next(d, lane, a.status, ok);
            if (pair_any(pair_bar, !more)) break;
            if (d.first()) {
                int4 rec = make_int4(0, 0, 0, 0);
                if constexpr (PAGED) rec = a.rec[d.b];
                id = dense_row<PAGED>(a, 2 * d.b + (d.single() ? 0 : g), row, rec);
                m_run = -INFINITY;
                l_run = 0.f;
                any = false;
            }
            int lim = 0;                                       // keys of the fragment that the row sees: [0, lim)
            if (id.valid) lim = min(dense_location<PAGED>(a, d.f, id), dense_length<PAGED>(a, d.f, id.w) - 1) + 1;
            const int stride = d.single() ? 2 : 1, t1 = d.single() ? d.t1 : min(d.t1, ((g ? d.vis1 : d.vis0) + kDenseTile - 1) / kDenseTile);
#pragma unroll 1
            for (int t = d.t0 + (d.single() ? g : 0); t < t1; t += stride) {
                ok = mbar_wait_polls(s_full + 8 * g, phase, a.status, STATUS_WAIT_FULL_TIMEOUT);
                tc_fence_after();
                __syncwarp();
                float s[COLS];
                tmem_ld32(s_addr, *reinterpret_cast<float(*)[32]>(&s[0]));
                tmem_ld32(s_addr + 32, *reinterpret_cast<float(*)[32]>(&s[32]));
                tmem_wait_ld();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(s_free);            // the next S MMA may overwrite the buffer
                const int nvis = lim - t * kDenseTile - half * COLS;      // of this thread's keys the row sees [0, nvis)
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                if (__any_sync(0xffffffffu, nvis < COLS)) {
#pragma unroll
                    for (int k = 0; k < COLS; ++k) s[k] = k < nvis ? s[k] : -INFINITY;
                }
#pragma unroll
                for (int k = 0; k < COLS; k += 8)
#pragma unroll
                    for (int i = 0; i < 4; ++i) mx[i] = max3(mx[i], s[k + 2 * i], s[k + 2 * i + 1]);
                float mt = max3(fmaxf(mx[0], mx[1]), mx[2], mx[3]);
                // ---- P and O become writable once this group's previous second MMA has finished ----
                if (ever) {
                    ok = mbar_wait_polls(o_done + 8 * g, phase ^ 1u, a.status, STATUS_WAIT_SYNC_TIMEOUT) && ok;
                    tc_fence_after();
                }
                // O is stored at scale 2^(-m_run * scale2).  It is only brought to a new scale when a row's max has grown by
                // more than a factor 2^8 (so every exponent below stays <= 8) or nothing has been accumulated yet.  Only
                // then do the two halves of the rows need each other's maxima.
                if (pair_any(pair_bar, mt > m_run + grow_by || !ok)) {
                    ok = !pair_any(pair_bar, !ok);
                    if (!ok) break;
                    *stat = mt;
                    named_barrier_sync(pair_bar, 64);
                    mt = fmaxf(mt, *other);
                    named_barrier_sync(pair_bar, 64);          // (read before it is written again)
                    const bool grow = mt > m_run + grow_by;                     // (m_run = -inf: any finite max grows it)
                    const float m_new = grow ? mt : m_run;
                    const float alpha = grow ? fast_exp2((m_run - m_new) * scale2) : 1.f;      // (m_run = -inf -> 0)
                    m_run = m_new;
                    l_run *= alpha;
                    if (any) {
#pragma unroll 1
                        for (int c = 0; c < COLS; c += 16) {
                            uint32_t o[16];
                            tmem_ld16(o_addr + c, o);
                            tmem_wait_ld();
#pragma unroll
                            for (int k = 0; k < 16; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * alpha);
                            tmem_st16(o_addr + c, o);
                        }
                    }
                }
                const float bias = (m_run == -INFINITY) ? 0.f : -m_run * scale2;
                const uint64_t scale_pair = pair_f32(scale2, scale2), bias_pair = pair_f32(bias, bias);
                uint64_t sum[2] = {0ull, 0ull};                             // (two fp32 zeros each)
#pragma unroll
                for (int c = 0; c < COLS / 32; ++c) {
                    uint32_t packed[16];
#pragma unroll
                    for (int k = 0; k < 16; ++k) {
                        float x0, x1;
                        unpair_f32(fma2(pair_f32(s[c * 32 + 2 * k], s[c * 32 + 2 * k + 1]), scale_pair, bias_pair), x0, x1);
                        x0 = fast_exp2(x0);
                        x1 = fast_exp2(x1);
                        sum[k & 1] = add2(sum[k & 1], pair_f32(x0, x1));
                        packed[k] = pack2<T>(x0, x1);
                    }
                    tmem_st16(p_addr + c * 16, packed);        // P (storage type, two per column): this row's lane
                }
                float l0, l1;
                unpair_f32(add2(sum[0], sum[1]), l0, l1);
                l_run += l0 + l1;
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_full + 8 * g);
                phase ^= 1u;
                any = ever = true;
            }
            if (!ok) break;

            // ---- end of this CTA's share of the unit: the rows themselves, or a partial result ----
            if (d.last()) {
                const bool direct = d.whole() && !d.single(), one_tile = d.single();
                const int unit = d.b * a.Hkv + d.h;
                int* const fold = a.fold + (size_t)unit * kDenseFoldInts;
                int* const left = fold + 4 + (one_tile ? warp & 7 : warp);
                int2 who = make_int2(0, 0);
                int n_left = 0;                                // (asked for in front of the last wait; an old answer costs a partial)
                if (!direct) {
                    who = *reinterpret_cast<const int2*>(fold);
                    if (lane == 0) asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(n_left) : "l"(left) : "memory");
                }
                if (any) {
                    ok = mbar_wait_polls(o_done + 8 * g, phase ^ 1u, a.status, STATUS_WAIT_SYNC_TIMEOUT);
                    tc_fence_after();
                }
                *stat = l_run;
                ok = !pair_any(pair_bar, !ok);
                if (!ok) break;
                const float total = half ? *other + l_run : l_run + *other;
                named_barrier_sync(pair_bar, 64);              // (read before it is written again)
                const int slot_row = g * kDenseRows + row;
                const size_t slot = (size_t)blockIdx.x + unit;
                const float m_own = m_run == -INFINITY ? -INFINITY : m_run * scale2;
                int first = blockIdx.x, parts = 1;             // partials that make up the rows: CTAs from `first` on, or their halves
                bool finish = direct;
                if (!direct) {
                    // Warps of different CTAs that hold the same rows and columns count themselves off; the last one has all
                    // that the others left.  Not known yet to be the last: leave a partial first.  (The count releases the
                    // warp's partial and acquires the others', once: with a full fence on either side of it, the question asked
                    // only here, and the other parts' maxima fetched one after the other, the fold was 1-2 us more: 640 tokens of
                    // 1,024 packed keys 34.2 us, 32.0 now; a 1,500-token prompt of two kv heads 40.4 / 38.1.)
                    if (who.y > 0) {
                        first = who.x;
                        parts = one_tile ? 2 * who.y : who.y;
                        finish = __shfl_sync(0xffffffffu, n_left, 0) == 1;
                        __syncwarp();
                    }
                    if (!finish) {
                        float4* const wo = a.ws_o + (slot * (C::HD / 4) + half * (COLS / 4)) * kDenseBlock + slot_row;
#pragma unroll 1
                        for (int c = 0; c < COLS; c += 32) {
                            float o[32];
                            tmem_ld32(o_addr + c, o);
                            tmem_wait_ld();
#pragma unroll
                            for (int k = 0; k < 32; ++k) o[k] = any ? o[k] : 0.f;          // (a group that saw nothing never touched its O)
#pragma unroll
                            for (int k = 0; k < 8; ++k) wo[(c / 4 + k) * kDenseBlock] = make_float4(o[4 * k], o[4 * k + 1], o[4 * k + 2], o[4 * k + 3]);
                        }
                        a.ws_m[slot * kDenseBlock + slot_row] = m_own;                     // (both halves store the same)
                        a.ws_l[slot * kDenseBlock + slot_row] = total;
                        if (who.y > 0) {
                            __syncwarp();
                            int n = 0;
                            if (lane == 0) asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], -1;" : "=r"(n) : "l"(left) : "memory");
                            finish = __shfl_sync(0xffffffffu, n, 0) == 1;
                            __syncwarp();
                        }
                    }
                }
                if (finish) {
                    // out = sum_p O_p * 2^(m_p - M) / sum_p l_p * 2^(m_p - M), in the order of the parts whoever is last
                    const bool sectors = a.world == 0 && ((uintptr_t)a.out & 31u) == 0;
                    const int own = one_tile ? 2 * ((int)blockIdx.x - first) + g : (int)blockIdx.x - first;
                    auto at = [&](int p) {
                        const size_t sl = (size_t)first + unit + (one_tile ? p >> 1 : p);
                        return sl * kDenseBlock + (one_tile ? (p & 1) * kDenseRows + row : slot_row);
                    };
                    float M = m_own, den = 0.f;
                    if (parts > 1) {                           // (asked for together: each is a round trip to L2)
                        float m[2 * kDenseFoldParts];
#pragma unroll
                        for (int p = 0; p < 2 * kDenseFoldParts; ++p) m[p] = p < parts && p != own ? __ldcg(a.ws_m + at(p)) : -INFINITY;
#pragma unroll
                        for (int p = 0; p < 2 * kDenseFoldParts; ++p) M = fmaxf(M, m[p]);
                    }
                    const size_t offset = dense_out_offset<PAGED>(a, id, d.h) + half * COLS;
#pragma unroll 1
                    for (int c = 0; c < COLS; c += 32) {
                        float acc[32];
#pragma unroll
                        for (int k = 0; k < 32; ++k) acc[k] = 0.f;
                        den = 0.f;
#pragma unroll 1
                        for (int p = 0; p < parts; ++p) {
                            float x[32], m = m_own, l = total;
                            if (p == own) {
                                tmem_ld32(o_addr + c, x);
                                tmem_wait_ld();
                            } else {
                                const size_t i = at(p);
                                m = __ldcg(a.ws_m + i);
                                l = __ldcg(a.ws_l + i);
                                const size_t sl = i / kDenseBlock, r = i % kDenseBlock;
                                const float4* const src = a.ws_o + (sl * (C::HD / 4) + (half * COLS + c) / 4) * kDenseBlock + r;
#pragma unroll
                                for (int k = 0; k < 8; ++k) *reinterpret_cast<float4*>(x + 4 * k) = __ldcg(src + k * kDenseBlock);
                            }
                            const float w = m == -INFINITY ? 0.f : parts == 1 ? 1.f : exp2f(m - M);
                            den = fmaf(l, w, den);
                            if (p != own || any) {             // (what was never touched may hold anything)
#pragma unroll
                                for (int k = 0; k < 32; ++k) acc[k] = fmaf(x[k], w, acc[k]);
                            }
                        }
                        const float inv = den > 0.f ? 1.f / den : 0.f;
                        uint32_t v[2][8];
#pragma unroll
                        for (int k = 0; k < 16; ++k) v[k >> 3][k & 7] = pack2<T>(acc[2 * k] * inv, acc[2 * k + 1] * inv);
#pragma unroll 1
                        for (int q = 0; q < (id.valid ? max(a.world, 1) : 0); ++q) {
                            T* const dst = static_cast<T*>(a.world > 0 ? a.peer_out[q] : a.out) + offset + c;
                            if (sectors) {
                                store_sector(dst, v[0]);
                                store_sector(dst + 16, v[1]);
                            } else {
#pragma unroll
                                for (int k = 0; k < 4; ++k)
                                    reinterpret_cast<uint4*>(dst)[k] = make_uint4(v[k >> 1][(k & 1) * 4], v[k >> 1][(k & 1) * 4 + 1],
                                                                                  v[k >> 1][(k & 1) * 4 + 2], v[k >> 1][(k & 1) * 4 + 3]);
                            }
                        }
                        __syncwarp();
                    }
                }
                tc_fence_before();
            }
        }
    }

    // ---- common exit: nobody leaves before the copies and products in flight have ended and tensor memory can be handed
    // back.  In an ordinary call the last segment's readers have waited for all of them. ----
    tc_fence_before();
    if (__syncthreads_or(!ok)) {
        if (tid == 0) a.nmerge[1] = 1;                         // the merge step leaves NaN
        settle();
        __syncthreads();
    }
    if (warp == W_S) {
        tc_fence_after();
        tmem_dealloc(tmem, C::TMEM_COLS);
    }
}

// The units on the plan's list -- those that several CTAs worked on and none of them folds, or where nothing is visible --: fold
// the partials, normalise, store.  A warp takes 32 rows, one per lane, and 16 columns: every load of a partial is 512 consecutive
// bytes, a lane stores one 32-byte sector.  A CTA is the eight column groups of 32 rows, or with SPLIT eight warps that share the
// partials of the same rows and columns (a unit cut into a hundred parts would be a chain of as many loads); the grid walks the list.
// Bound by its chain of dependent loads -- list, partials, store, about a microsecond each -- and by the wait in front of
// them, so a row's statistics and values are fetched together, BATCH partials at a time, and rescaled when a later batch has
// the larger maximum (1,024 rows of 8 heads, 24,576 keys, 5.6 partials each: 7 us from the attention kernel's end to this
// one's, 10 when the list's length, its entry, the maxima and the values were fetched one after the other).
//   out = sum_p O_p * 2^(m_p - M) / sum_p l_p * 2^(m_p - M),   M = max_p m_p
template <class T, bool PAGED, bool SPLIT, int BATCH>
__global__ void __launch_bounds__(kDenseMergeWarps * 32, BATCH == 1 ? 4 : 2) dense_merge_kernel(const __grid_constant__ DenseArgs a) {
    __shared__ float part[SPLIT ? kDenseMergeWarps : 1][18][32];         // 16 columns, maximum, sum; by row
    constexpr int PER = SPLIT ? 64 : 8;                                  // CTAs' worth of work per unit
    constexpr int STRIDE = SPLIT ? kDenseMergeWarps : 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_wait();
    pdl_trigger();
    int4 e = a.merge[min((int)(blockIdx.x / PER), a.blocks * a.Hkv - 1)];       // (in flight with the list's length; not used past it)
    const int2 head = *reinterpret_cast<const int2*>(a.nmerge);
    if (head.y != 0) {
        // given up: nothing that looks like a result (0x7FFF is a NaN of both types)
        const size_t per = (size_t)(PAGED ? a.total_q : a.S) * a.Hq * (128 / 8), all = (PAGED ? 1 : a.W) * per;
        for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < all; i += (size_t)gridDim.x * blockDim.x) {
            const size_t w = i / per, at = a.world > 0 ? (w * a.world + a.rank) * per + i % per : i;
            for (int p = 0; p < max(a.world, 1); ++p)
                static_cast<uint4*>(a.world > 0 ? a.peer_out[p] : a.out)[at] = make_uint4(0x7FFF7FFFu, 0x7FFF7FFFu, 0x7FFF7FFFu, 0x7FFF7FFFu);
        }
        return;
    }
    for (int64_t i = blockIdx.x; i < (int64_t)head.x * PER; i += gridDim.x) {
        const int task = (int)(i % PER);
        if (i != blockIdx.x) e = a.merge[i / PER];
        const int r = (SPLIT ? task >> 3 : task) * 32 + lane, c4 = (SPLIT ? task & 7 : warp) * 4;
        const int b = e.x / a.Hkv, h = e.x - b * a.Hkv, count = e.z;
        const bool single = e.w != 0;
        // a block of one tile: both 128-row halves of a slot are partials of the same rows
        if (single && (r & ~31) >= kDenseRows) continue;
        int4 rec = make_int4(0, 0, 0, 0);
        if constexpr (PAGED) rec = a.rec[b];
        const int sub = single ? 1 : 0;
        const size_t slot0 = (size_t)e.y + e.x;
        float M = -INFINITY, den = 0.f;
        float4 acc[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
        for (int p0 = SPLIT ? warp : 0; p0 < count; p0 += BATCH * STRIDE) {
            float m[BATCH], l[BATCH];
            float4 x[BATCH][4];
#pragma unroll
            for (int j = 0; j < BATCH; ++j) {
                const int p = p0 + j * STRIDE;
                m[j] = -INFINITY;
                l[j] = 0.f;
#pragma unroll
                for (int k = 0; k < 4; ++k) x[j][k] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (p < count) {
                    const size_t slot = slot0 + (p >> sub), row = (single ? (p & 1) * kDenseRows : 0) + r;
                    m[j] = __ldcg(a.ws_m + slot * kDenseBlock + row);
                    l[j] = __ldcg(a.ws_l + slot * kDenseBlock + row);
                    const float4* src = a.ws_o + (slot * 32 + c4) * kDenseBlock + row;
#pragma unroll
                    for (int k = 0; k < 4; ++k) x[j][k] = __ldcg(src + k * kDenseBlock);
                }
            }
            float top = M;
#pragma unroll
            for (int j = 0; j < BATCH; ++j) top = fmaxf(top, m[j]);
            const float old = M == -INFINITY ? 0.f : exp2f(M - top);
            M = top;
            den *= old;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                acc[k].x *= old;
                acc[k].y *= old;
                acc[k].z *= old;
                acc[k].w *= old;
            }
#pragma unroll
            for (int j = 0; j < BATCH; ++j) {
                const float wgt = m[j] == -INFINITY ? 0.f : exp2f(m[j] - M);       // (a partial that saw nothing holds zeros)
                den = fmaf(l[j], wgt, den);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    acc[k].x = fmaf(x[j][k].x, wgt, acc[k].x);
                    acc[k].y = fmaf(x[j][k].y, wgt, acc[k].y);
                    acc[k].z = fmaf(x[j][k].z, wgt, acc[k].z);
                    acc[k].w = fmaf(x[j][k].w, wgt, acc[k].w);
                }
            }
        }
        float* o = reinterpret_cast<float*>(acc);
        if constexpr (SPLIT) {
            __syncthreads();                             // (the task before has been read)
#pragma unroll
            for (int k = 0; k < 16; ++k) part[warp][k][lane] = o[k];
            part[warp][16][lane] = M;
            part[warp][17][lane] = den;
            __syncthreads();
            if (warp != 0) continue;
            float top = M;
#pragma unroll
            for (int w = 1; w < kDenseMergeWarps; ++w) top = fmaxf(top, part[w][16][lane]);
            const float mine = M == -INFINITY ? 0.f : exp2f(M - top);
            den *= mine;
#pragma unroll
            for (int k = 0; k < 16; ++k) o[k] *= mine;
#pragma unroll
            for (int w = 1; w < kDenseMergeWarps; ++w) {
                const float mw = part[w][16][lane], wgt = mw == -INFINITY ? 0.f : exp2f(mw - top);
                den = fmaf(part[w][17][lane], wgt, den);
#pragma unroll
                for (int k = 0; k < 16; ++k) o[k] = fmaf(part[w][k][lane], wgt, o[k]);
            }
        }
        const DenseRow id = dense_row<PAGED>(a, 2 * b + r / kDenseRows, r % kDenseRows, rec);
        if (!id.valid) continue;
        const float inv = den > 0.f ? 1.f / den : 0.f;
        const size_t offset = dense_out_offset<PAGED>(a, id, h) + c4 * 4;
        uint4 v[2];
        uint32_t* out = reinterpret_cast<uint32_t*>(v);
#pragma unroll
        for (int k = 0; k < 8; ++k) out[k] = pack2<T>(o[2 * k] * inv, o[2 * k + 1] * inv);
        for (int p = 0; p < max(a.world, 1); ++p) {
            uint4* dst = reinterpret_cast<uint4*>(static_cast<T*>(a.world > 0 ? a.peer_out[p] : a.out) + offset);
            dst[0] = v[0];
            dst[1] = v[1];
        }
    }
}

}  // namespace hogatt
