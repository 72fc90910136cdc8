// Forward on the Blackwell tensor path for what the other two tcgen05 kernels are not built for -
// head dims that are any multiple of 8 up to 128, and masks with a row per query, unless the rows are
// so few that warp-MMA is the faster (forward_pair_pays) - and for calls of few keys, or whose rounds of
// SMs it fills better, in which it is the faster (forward_pair_preferred). TMA tile loads, tcgen05.mma with accumulators in tensor memory,
// online softmax with one thread per query row.
//
// A persistent CTA per SM works on two 128-row query tiles at a time, A and B:
//
//   warps 0-3, 4-7     softmax of tile A and of tile B: thread r owns query row r and all 128
//                      keys of a block, with its own running maximum and sum; it writes P (bf16)
//                      to tensor memory and rescales O only when the maximum moved by more than
//                      2^8 (the lazy rescale of ktt_flash/compute.cpp, flash.md "row reference").
//                      No two threads ever exchange anything inside the loop.
//                      (kTurns: its exponentials in turn with the same warp of the other tile)
//   warps 8, 9         issue S = Q K^T and O += P V (P read from tensor memory) of A and of B: while
//                      one tile is in its exponentials the tensor core serves the other
//   warp 10            draws the work and hands the items round, TMA loads of Q and of a ring of K
//                      and V tiles
//
// An item of few blocks runs every role's code once or twice, and a third of the instruction fetches
// missed the cache. Hence one copy of the item
// arithmetic (the producer's), short waits, and loops where a block is not the common one: 94 to
// 150 KB of instructions became 79 to 105, and 16 x 16 heads x 257 rows, D 80, took 42 us where it had
// taken 49 (a fifth of the fetches still miss there, a tenth on the masked call below).
//
// Measured on B200, warp-MMA (mma.sync, 64-row CTAs) and this kernel: 16 x 16 heads x 257 rows, D 80,
// 220 and 36 us; 2 x 16 heads x 2048, D 64, a causal mask with padding as a bf16 tensor, 577 and 57 us.
//
// Tensor memory (512 columns): S_A, S_B (128 each); head dims up to 64: P_A, P_B (64 each) and
// O_A, O_B (64 each), so that the next scores can be computed while P V still reads P; up to 128:
// P overwrites the scores it came from, O_A, O_B (128 each). Head dims between two sizes are
// zero-filled by TMA; the products run over ceil(D / 16) steps and ceil(Dv / 16) columns only.
//
// Two ways to use the two tiles:
//   pair   A and B are neighbours in the list of (query tile, head) of one K / V head: one
//          K / V stream serves both, which halves the traffic from L2
//   dual   (no more tiles than SMs, and the tiles of a last round that leaves half of the SMs idle) A and B are the same query tile, A working on the first half of
//          its key blocks and B on the rest; A's threads then read B's unnormalised O straight
//          out of tensor memory. The longest tile's serial chain is halved. Always A then B:
//          the bits do not depend on timing.
//
// Masks. One row per (batch, head): the 128 terms of a block are fetched by 128 threads and
// shared through shared memory. A row per query: a small kernel in front (mask_plan_kernel)
// sorts the mask into 32-row x 128-key pieces - hidden, without effect, yes / no, values -
// and lays the pieces that matter out so that a warp reads them with coalesced 16-byte loads;
// blocks hidden from a whole tile are not visited at all.
//
// Arithmetic contract as in the reference's flash forward (ktt_flash/compute.cpp:193-491):
// base-2 softmax with fp32 statistics, P rounded to bf16 before P V, fp32 accumulation, O / l
// and lse = ln2 (m + log2 l) at the end.
//
// Every wait on an mbarrier is bounded: when one runs out the CTA records a code in a
// host-visible status word, stops waiting everywhere, frees its tensor memory and exits.
// Launched with programmatic stream serialization: everything before `griddepcontrol.wait`
// may overlap the tail of the previous kernel in the stream.
#include "rounds.h"
#include "tc5.cuh"

namespace ktt {
using namespace tc5;
namespace {

constexpr float kRescaleGap = 8.f;   // log2 units
// Three warpgroups; warp 11 has no role. Registers can only be moved between whole warpgroups: the
// softmax threads, which hold 128 scores each, take 216, the last group keeps 72.
// (208 / 88 and 224 / 56 spill more: 56.9, 53.9 and 55.2 us for 208, 216 and 224 on 2 x 16 heads x
// 2048, D 64, causal mask.)
constexpr int kPairThreads = 384;
constexpr int kSoftmaxRegs = 216, kRoleRegs = 3 * 168 - 2 * kSoftmaxRegs;
static_assert(2 * kSoftmaxRegs + kRoleRegs <= 3 * 168, "an increase beyond what the block started with waits for ever");
constexpr int kMmaWarp = 8, kProducerWarp = 10;   // kMmaWarp + t: tile t

template <int DP>
struct PairPlan {
    static constexpr int kSub = DP / 64;              // 64-column sub-tiles of an operand
    static constexpr int kTile = 128 * 128;           // one [128][64] bf16 sub-tile, 128-byte swizzled rows
    static constexpr int kOperand = kSub * kTile;
    static constexpr int kSlots = DP == 64 ? 12 : 5;  // ring of K and V tiles (K, V, K, V, ...)
    static constexpr int kQ = 0;                      // Q_A, Q_B
    static constexpr int kRing = 2 * kOperand;
    static constexpr int kMaskRow = kRing + kSlots * kOperand;   // float [tile][parity][128]: a block's mask terms
    static constexpr int kBars = kMaskRow + 2 * 2 * 128 * 4;
    static constexpr int kBarBytes = 512;
    static constexpr int kQueue = 4;
    static constexpr int kItems = kBars + kBarBytes;  // Item [kQueue]: what the producer hands to the other roles
    static constexpr int kBytes = kItems + kQueue * 96;
    static_assert(kBytes <= 232448, "shared memory per CTA");
    // dual: float2 [128] of B's (m, l); Q_B is idle then
    static constexpr int kPartial = kQ + kOperand;
    // tensor memory columns
    static constexpr bool kPOverS = DP == 128;        // P overwrites the scores it came from
    static constexpr int kP = kPOverS ? 0 : 256;      // S_A 0, S_B 128
    static constexpr int kPStep = kPOverS ? 128 : 64; // from P_A to P_B
    static constexpr int kO = kPOverS ? 256 : 384;    // + DP per tile
    static_assert(kO + 2 * DP <= 512, "tensor memory columns");
    // Exponentials per 8 pairs that take the FMA-pipe polynomial instead of MUFU. Measured, 0, 1, 2, 3
    // of 8: 36.4, 36.6, 36.1, 37.5 us on 16 x 16 heads x 257, D 80; 57.2, 56.8, 56.9, 58.4 us on 2 x 16
    // heads x 2048, D 64, a causal mask.
    static constexpr int kPolyPairs = 2;
    // barriers (8 bytes each); "+ t": tile
    static constexpr int bQFull = 0;                   // + t
    static constexpr int bQFree = 2;                   // + t
    static constexpr int bSFull = 4;                   // + t
    static constexpr int bSFree = 6;                   // + t: the scores are in registers
    static constexpr int bPFull = 8;                   // + 2 t + half of the keys (64 each; one phase for all where P has columns of its own)
    static constexpr int bPVDone = 12;                 // + t
    static constexpr int bOFree = 14;                  // + t
    static constexpr int bWorkFull = 16;               // + queue slot
    static constexpr int bWorkFree = bWorkFull + kQueue;   // + queue slot
    static constexpr int bMask = bWorkFree + kQueue;   // + t: the block's mask terms are written
    static constexpr int bPartial = bMask + 2;         // dual: B's half is final
    static constexpr int bTurn = bPartial + 1;         // + 4 t + warp: the other tile's warp of this scheduler has had its turn
    static constexpr int bKVFull = bTurn + 8;          // + ring slot
    static constexpr int bKVEmpty = bKVFull + kSlots;  // + ring slot
    static constexpr int bCount = bKVEmpty + kSlots;
    static_assert(bCount * 8 + 32 <= kBarBytes, "barrier area");
};

// What mask_plan_kernel leaves behind, per plane (a (batch, head) of the mask's own sizes),
// 32-row group and 128-key block. `active`: bit per block, set unless the block is hidden from
// the group. `kind`: see PieceKind. `bits`: uint4 per row (bit = visible). `values`: 128 terms
// per row as they were given (16-bit: bf16; else fp32), [16-byte chunk][row].
struct MaskPlan {
    uint32_t* active;
    uint8_t* kind;
    uint4* bits;
    uint4* values;
    int groups, blocks, words;   // 32-row groups, key blocks, active words per group
    int heads;                   // planes per batch entry
    int batched;                 // 0: every batch entry shares the planes
    int wide;                    // values are fp32
};
enum PieceKind : uint8_t { kHidden = 0, kNoEffect = 1, kYesNo = 2, kValues = 3, kAllFloor = 4 };
constexpr int kMaxPlanBlocks = 1024;

struct PairParams {
    AttnParams a;
    int* status;
    int dim_of[3][3];     // per operand (q, k, v): tensor-map slot (1..3) of the row, head and batch dims
    int work;             // items
    int duals;            // items from this one on are halves: a tile each, both tiles of the CTA on it (0: all of them)
    int cut;              // ... of the pairs from this item on, two items each; 0 where every item is a tile
    int* work_counter;    // null: a fixed deal
    int* done_counter;    // with it: the last producer to finish puts both back to zero
    int grouped;          // item order (decode_item)
    Divisor by_batch, by_kv_heads, by_group, by_levels;
    MaskPlan plan;
};

struct alignas(16) Item {
    int b, hk;                  // b < 0: no more items
    int dual;                   // A and B are halves of the keys of one tile
    int h[2], q0[2], kend[2];   // per tile; kend: keys any of its rows sees
    int n[2];                   // key blocks per tile (dual: its share); n[0] >= n[1]
    int valid[2];
    SeqInfo si;
};
static_assert(sizeof(Item) <= 96, "the queue's slots");

// Items of one (batch, K / V head) are neighbours in its list of (query tile, head), last rows first
// (the longest of a causal call), heads fastest; of an odd number of tiles it is the first rows' that
// has no partner. Two orders of the items: with the level slowest every deal in rounds hands out
// similar lengths; `grouped` (needs the counter) keeps all items of one
// (batch, K / V head) together, so that the items in flight share the K / V of a few heads in L2
// (measured on a packed 65,536-token batch with 537 MB of K / V: 4.85 -> 0.81 GB of DRAM reads).
__device__ __forceinline__ Item decode_item(const PairParams& tp, int w) {
    const AttnParams& p = tp.a;
    Item k;
    int level, only = 0;   // only: which of a pair's tiles a half is of
    k.dual = w >= tp.duals;
    if (k.dual && tp.cut) {
        only = (w - tp.duals) & 1;
        w = tp.cut + ((w - tp.duals) >> 1);
    }
    if (tp.grouped) {
        const int plane = div_by(w, tp.by_levels);
        level = w - plane * static_cast<int>(tp.by_levels.d);
        k.b = div_by(plane, tp.by_kv_heads);
        k.hk = plane - k.b * p.kv_heads;
    } else {
        const int t = div_by(w, tp.by_kv_heads);
        k.hk = w - t * p.kv_heads;
        level = div_by(t, tp.by_batch);
        k.b = t - level * p.batch;
    }
    k.si = seq_info(p, k.b);
    const int group = static_cast<int>(tp.by_group.d);
    const int tiles = (k.si.lq + kBM - 1) >> 7;
    const int units = tiles * group;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int u = !k.dual ? 2 * level + t : tp.cut ? 2 * level + only : level;
        k.valid[t] = u < units;
        const int back = div_by(u, tp.by_group);
        k.h[t] = k.hk * group + (u - back * group);
        k.q0[t] = (tiles - 1 - back) * kBM;
        int kend = k.si.klen;
        if (p.causal) kend = min(kend, min(k.q0[t] + kBM, k.si.lq) + k.si.shift);
        k.kend[t] = max(kend, 0);
        k.n[t] = k.valid[t] ? (k.kend[t] + kBN - 1) >> 7 : 0;
    }
    if (k.dual) {
        k.n[1] = k.n[0] >> 1;
        k.n[0] -= k.n[1];
    }
    return k;
}

// Walks the key blocks of an item. Without a plan that is 0, 1, 2, ...; with one it is the
// blocks that are not hidden from both tiles (a dual item: from the tile).
template <bool kPlan>
struct BlockIter {
    int at;
    __device__ __forceinline__ void start(const PairParams&, const Item&, int first) { at = first; }
    __device__ __forceinline__ int next() { return at++; }
};
// The active word `w` of an item (converged warp): lanes 0-7 fetch the words of the two tiles'
// eight 32-row groups.
__device__ __forceinline__ uint32_t active_word(const PairParams& tp, const Item& k, int w) {
    const MaskPlan& m = tp.plan;
    const int lane = threadIdx.x & 31, t = (lane >> 2) & 1;
    uint32_t word = 0;
    if (lane < 8 && k.valid[t]) {
        const int g = (k.q0[t] >> 5) + (lane & 3);
        const int plane = (m.batched ? k.b * m.heads : 0) + (m.heads > 1 ? k.h[t] : 0);
        if (g < m.groups) word = m.active[(static_cast<int64_t>(plane) * m.groups + g) * m.words + w];
    }
    return __reduce_or_sync(0xffffffffu, word);
}
template <>
struct BlockIter<true> {
    const PairParams* tp;
    const Item* k;
    uint32_t word;
    int w;
    __device__ __forceinline__ void start(const PairParams& tp_, const Item& k_, int first) {
        tp = &tp_;
        k = &k_;
        w = 0;
        word = active_word(tp_, k_, 0);
        for (int i = 0; i < first; ++i) next();
    }
    __device__ __forceinline__ int next() {
        while (!word) {
            ++w;
            if (w >= tp->plan.words) return 0;   // not reached: callers take as many as there are
            word = active_word(*tp, *k, w);
        }
        const int bit = __ffs(word) - 1;
        word &= word - 1;
        return w * 32 + bit;
    }
};
// With a plan both tiles of an item walk the blocks that either of them needs.
__device__ __forceinline__ void apply_plan(const PairParams& tp, Item& k) {
    int n = 0;
    for (int w = 0; w < tp.plan.words; ++w) n += __popc(active_word(tp, k, w));
    if (k.dual) {
        k.n[1] = n >> 1;
        k.n[0] = n - k.n[1];
    } else {
        k.n[0] = k.valid[0] ? n : 0;
        k.n[1] = k.valid[1] ? n : 0;
    }
}

__device__ __forceinline__ int snake(int round, int cta, int ctas) {
    return round * ctas + ((round & 1) ? ctas - 1 - cta : cta);
}

__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));   // one three-input instruction
    return d;
}

// Bounded waits of a converged warp, for one barrier or two at once (their polls overlap). Kept
// short: there are two dozen of them in this kernel, and what does not fit the instruction cache
// is fetched again for every item.
__device__ __forceinline__ bool wait_both(uint32_t b0, uint32_t par0, uint32_t b1, uint32_t par1, volatile int* abort_flag, int code) {
    if (__all_sync(0xffffffffu, mbar_try_wait(b0, par0) & mbar_try_wait(b1, par1))) return true;
    const long long t0 = clock64();
#pragma unroll 1
    while (!__all_sync(0xffffffffu, mbar_try_wait(b0, par0) & mbar_try_wait(b1, par1))) {
        const bool late = clock64() - t0 > kWaitCycles;
        if (late) *abort_flag = code;   // reported when the CTA ends
        if (__any_sync(0xffffffffu, late || *abort_flag)) return false;
    }
    return true;
}
__device__ __forceinline__ bool wait_one(uint32_t b, uint32_t par, volatile int* abort_flag, int code) {
    if (__all_sync(0xffffffffu, mbar_try_wait(b, par))) return true;
    const long long t0 = clock64();
#pragma unroll 1
    while (!__all_sync(0xffffffffu, mbar_try_wait(b, par))) {
        const bool late = clock64() - t0 > kWaitCycles;
        if (late) *abort_flag = code;   // reported when the CTA ends
        if (__any_sync(0xffffffffu, late || *abort_flag)) return false;
    }
    return true;
}

// ---- the kernel ------------------------------------------------------------------------

// kMask: 0 none, 1 a row per (batch, head), 2 a plan (a row per query).
// kMixed: of the items some are pairs of tiles and some halves of one (last_round_in_halves).
// kTurns: where P overwrites the scores a tile's products and its softmax are one chain, and two tiles that
// run in step wait for the tensor cores at the same time and then for the exponentials. Taking turns at the
// exponentials, the products of one run under those of the other.
template <int DP, int kMask, bool kTurns, bool kMixed>
__global__ void __launch_bounds__(kPairThreads, 1) fwd_pair_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
    const __grid_constant__ CUtensorMap map_v, const PairParams tp) {
    using P = PairPlan<DP>;
    using Iter = BlockIter<kMask == 2>;
    extern __shared__ __align__(1024) unsigned char smem[];
    const uint32_t sbase = smem_u32(smem);
    if (sbase & 1023u) {   // swizzled tiles need a 1024-byte aligned base
        if (threadIdx.x == 0) atomicCAS_system(tp.status, 0, 900);
        return;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t bars = sbase + P::kBars;
    auto bar = [&](int i) { return bars + 8u * i; };
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + P::kBars + P::bCount * 8);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + P::kBars + P::bCount * 8 + 8);
    Item* queue = reinterpret_cast<Item*>(smem + P::kItems);   // [kQueue]
    const AttnParams& p = tp.a;
    const bool all_dual = tp.duals == 0;

    if (warp == kProducerWarp) {
        for (int i = lane; i < P::bCount; i += 32) {
            uint32_t count = 1;
            // Softmax threads arrive once per warp (mbar_arrive_warp).
            if ((i >= P::bSFree && i < P::bSFree + 2) || (i >= P::bPFull && i < P::bPFull + 4) ||
                (i >= P::bOFree && i < P::bOFree + 2) || (i >= P::bMask && i < P::bMask + 2) || i == P::bPartial) count = 4;
            if (i >= P::bWorkFree && i < P::bWorkFree + P::kQueue) count = 10;   // the softmax and the MMA warps
            // Pair: both tiles release every ring tile. Dual: each has one user, but they share Q. (Mixed: one
            // user, or tile A alone, releases twice.)
            if (i >= P::bKVEmpty && (kMixed || !all_dual)) count = 2;
            if (i == P::bQFree && (kMixed || all_dual)) count = 2;
            mbar_init(bar(i), count);
        }
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
            *abort_flag = 0;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
        __syncwarp();
    } else if (warp == kMmaWarp) {
        tmem_alloc(smem_u32(tmem_slot), 512);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // Nothing of this launch has touched global memory yet, and nothing will before the previous
    // kernel in the stream has completed; the next one may start its own set-up.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    // The producer warp draws the items (from a counter, or the fixed deal of a snake order), works
    // out what they are and hands them to the other roles through a queue in shared memory: one
    // role's divisions and one copy of that code. Positions past the end of a short sequence are
    // left out. A role gives an item back when it no longer reads the queue's copy.
    auto take_item = [&](int n, Item& k, bool& ok) {   // the other roles
        const int slot = n % P::kQueue;
        ok = ok && wait_one(bar(P::bWorkFull + slot), (n / P::kQueue) & 1, abort_flag, 130 + slot);
        k.b = -1;
        if (ok) k = queue[slot];
        return k.b >= 0;
    };
    auto give_item = [&](int n) { mbar_arrive_warp(bar(P::bWorkFree + n % P::kQueue)); };
    // Tensor-map coordinate of slot `slot` (1..3): row, head and batch sit where the host sorted
    // them by stride.
    auto coord = [&](int operand, int slot, int row, int head, int batch) {
        return tp.dim_of[operand][0] == slot ? row : tp.dim_of[operand][1] == slot ? head : batch;
    };

    // The register counts are set inside the roles' branches: in code that both reach, the compiler
    // would have to keep to the smaller one.
    if (warp >= kMmaWarp) {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRoleRegs));
      if (warp == kProducerWarp) {
        // ---------------- producer (whole warp, converged) ----------------
        int items_of[2] = {0, 0};   // Q tiles loaded so far
        int slot = 0, lap = 0;      // next ring slot, times round the ring
        bool ok = true;
        auto wait_for = [&](int b, int parity, int code) {
            ok = ok && wait_one(bar(b), parity, abort_flag, code);
        };
        const bool dynamic = tp.work_counter != nullptr;
        int round = 0;
        auto draw = [&]() -> int {   // the next position in the list of items; -1 = no more
            if (!dynamic) {
                const int64_t first = static_cast<int64_t>(round) * gridDim.x;
                const int w = first < tp.work ? snake(round, blockIdx.x, gridDim.x) : -1;
                ++round;
                return w;
            }
            int w = 0;
            if (lane == 0) w = atomicAdd(tp.work_counter, 1);
            w = __shfl_sync(0xffffffffu, w, 0);
            return w < tp.work ? w : -1;
        };
        auto load_q = [&](const Item& k, int t) {
            if (items_of[t] > 0) wait_for(P::bQFree + t, (items_of[t] - 1) & 1, 110 + t);
            if (!ok) return;
            const int r = k.si.q_off + k.q0[t], b = p.cu_q ? 0 : k.b;
            const int c1 = coord(0, 1, r, k.h[t], b), c2 = coord(0, 2, r, k.h[t], b), c3 = coord(0, 3, r, k.h[t], b);
            mbar_expect_tx(bar(P::bQFull + t), P::kOperand);
            for (int s = 0; s < P::kSub; ++s) {
                tma_load_4d(sbase + P::kQ + t * P::kOperand + s * P::kTile, &map_q, bar(P::bQFull + t), s * 64, c1, c2, c3);
            }
            ++items_of[t];
        };
        auto load_kv = [&](const Item& k, const CUtensorMap* map, int operand, int block) {
            if (lap > 0) wait_for(P::bKVEmpty + slot, (lap - 1) & 1, 100);
            if (!ok) return;
            const int r = k.si.k_off + block * kBN, b = p.cu_q ? 0 : k.b;
            const int c1 = coord(operand, 1, r, k.hk, b), c2 = coord(operand, 2, r, k.hk, b), c3 = coord(operand, 3, r, k.hk, b);
            mbar_expect_tx(bar(P::bKVFull + slot), P::kOperand);
            for (int s = 0; s < P::kSub; ++s) {
                tma_load_4d(sbase + P::kRing + slot * P::kOperand + s * P::kTile, map, bar(P::bKVFull + slot), s * 64, c1, c2, c3);
            }
            if (++slot == P::kSlots) {
                slot = 0;
                ++lap;
            }
        };
        // In the grouped order positions are fetched one ahead: the trip to the counter hides behind
        // an item's loads. Otherwise an item is drawn when its loads start: committing earlier evens
        // the CTAs out less well at the end.
        const bool ahead = tp.grouped != 0;
        int w_next = ahead ? draw() : 0;
        for (int n = 0; ok;) {
            const int w = ahead ? w_next : draw();
            Item k;
            k.b = -1;
            if (w >= 0) {
                if (ahead) w_next = draw();
                if (w >= tp.work) continue;   // the fixed deal's last round
                k = decode_item(tp, w);
                if (!k.valid[0]) continue;
                if constexpr (kMask == 2) apply_plan(tp, k);
            }
            const int q_slot = n % P::kQueue;
            if (n >= P::kQueue) wait_for(P::bWorkFree + q_slot, (n / P::kQueue - 1) & 1, 120 + q_slot);
            if (!ok) break;
            if (lane == 0) {
                queue[q_slot] = k;
                mbar_arrive(bar(P::bWorkFull + q_slot));   // release: the item before the arrival
            }
            __syncwarp();
            ++n;
            if (w < 0) break;
            if (k.n[0] == 0) continue;
            Iter it[2];
            it[0].start(tp, k, 0);
            const bool dual = kMixed ? k.dual != 0 : all_dual;
            if (dual) it[1].start(tp, k, k.n[0]);
            load_q(k, 0);
            const int entries = dual ? k.n[0] + k.n[1] : k.n[0];
            for (int e = 0; ok && e < entries; ++e) {
                const int block = (dual && (e & 1)) ? it[1].next() : it[0].next();
                load_kv(k, &map_k, 1, block);
                if (e == 0 && !dual && k.n[1] > 0) load_q(k, 1);
                load_kv(k, &map_v, 2, block);
            }
        }
        if (*abort_flag) {
            const long long t0 = clock64();
            while (clock64() - t0 < 4000000) {   // let copies in flight land
            }
        } else if (dynamic && tp.done_counter && lane == 0) {
            // This producer draws no more. The last one to say so puts the counters back to zero.
            __threadfence();
            const int done = atomicAdd(tp.done_counter, 1);
            if (done == static_cast<int>(gridDim.x) - 1) {
                *tp.work_counter = 0;
                *tp.done_counter = 0;
                __threadfence();
            }
        }
      } else if (warp < kMmaWarp + 2) {
        // ---------------- MMA issuer of tile t (whole warp, converged) ----------------
        // What stands between two products is this warp's scalar work, at the pace of one warp
        // beside two in their softmax: no divisions, no state in memory, one vote per pair of waits.
        const int t = warp - kMmaWarp;
        const uint64_t q_descs = smem_desc(sbase + P::kQ + (kMixed || all_dual ? 0 : t) * P::kOperand, 16, 1024);
        const uint64_t k_desc = smem_desc(sbase + P::kRing, 16, 1024);
        const uint64_t v_desc = smem_desc(sbase + P::kRing, P::kTile, 1024);
        const int d_steps = (p.d + 15) >> 4;
        const uint32_t d_s = tmem + t * 128, a_p = tmem + P::kP + t * P::kPStep, d_o = tmem + P::kO + t * DP;
        int blk = 0, items = 0;             // this tile's blocks and items so far: parities
        int q_a = 0, q_b = 0;               // Q tiles so far (mixed: Q_A, Q_B)
        int base = 0, base_lap = 0;         // ring position of the item's first tile
        bool ok = true;
        auto wait_two = [&](uint32_t b0, uint32_t par0, uint32_t b1, uint32_t par1, int code) {
            ok = ok && wait_both(b0, par0, b1, par1, abort_flag, code);
        };
        auto wait_bar = [&](uint32_t b, uint32_t par, int code) { ok = ok && wait_one(b, par, abort_flag, code); };
        auto advance = [](int& slot, int& lap, int by) {
            slot += by;
            if (slot >= P::kSlots) {
                slot -= P::kSlots;
                lap ^= 1;
            }
        };
        for (int n = 0; ok; ++n) {
            Item k;
            if (!take_item(n, k, ok)) break;
            give_item(n);
            if (k.n[0] == 0) continue;
            const bool dual = kMixed ? k.dual != 0 : all_dual;
            const int nb = t ? k.n[1] : k.n[0], kend = t ? k.kend[1] : k.kend[0], klen = k.si.klen;
            const int entries = dual ? k.n[0] + k.n[1] : k.n[0];
            const int q_bar = dual ? 0 : t, q_items = kMixed && q_bar ? q_b : q_a;
            const int stride = dual ? 4 : 2;    // ring tiles from one of this tile's blocks to its next
            const uint64_t q_desc = kMixed ? q_descs + static_cast<uint32_t>((q_bar * P::kOperand) >> 4) : q_descs;
            Iter it;
            it.start(tp, k, dual && t ? k.n[0] : 0);
            int s_slot = base, s_lap = base_lap;    // K of the next score product; V is one further
            if (dual && t) advance(s_slot, s_lap, 2);
            int v_slot = s_slot, v_lap = s_lap;
            advance(v_slot, v_lap, 1);
            int block = 0, s_block = 0;             // of the P V and of the score product at hand
            // Scores of block j + 1 go out ahead of P V of block j where P has columns of its own
            // (they only need the scores' columns free), behind it where P overwrites them.
#pragma unroll 1
            for (int j = -1; ok && j < nb; ++j) {
                const bool more = j + 1 < nb;
                if (more) s_block = it.next();
                auto scores = [&]() {
                    const int gb = blk + j + 1;     // this tile's score products so far
                    if (j < 0) {
                        wait_two(bar(P::bQFull + q_bar), q_items & 1, bar(P::bKVFull + s_slot), s_lap, 200 + 2 * t);
                        if (!P::kPOverS && gb > 0) wait_bar(bar(P::bSFree + t), (gb - 1) & 1, 210 + t);
                    } else if (P::kPOverS) {
                        wait_bar(bar(P::bKVFull + s_slot), s_lap, 220 + t);
                    } else {
                        wait_two(bar(P::bKVFull + s_slot), s_lap, bar(P::bSFree + t), (gb - 1) & 1, 222 + 2 * t);
                    }
                    if (!ok) return;
                    tc_fence_after();
                    // In the MMA's steps of 16, or in whole chunks where a mask's terms are added to all
                    // 32 columns of one (`fast` below): what no product has written may be a NaN, which
                    // a term of -inf does not hide.
                    constexpr int kRound = kMask == 1 ? 31 : 15;
                    const int keys = min(kBN, (kend - s_block * kBN + kRound) & ~kRound);
                    const uint64_t kd = k_desc + static_cast<uint32_t>(s_slot * (P::kOperand >> 4));
                    const uint32_t idesc = instr_desc(keys, false);
                    if (d_steps == DP / 16 && keys == kBN) {
#pragma unroll
                        for (int ks = 0; ks < DP / 16; ++ks) {
                            const uint32_t off = ((ks / 4) * P::kTile + (ks % 4) * 32) >> 4;
                            tc_mma(d_s, q_desc + off, kd + off, instr_desc(kBN, false), ks > 0);
                        }
                    } else {
#pragma unroll 1
                        for (int ks = 0; ks < d_steps; ++ks) {
                            const uint32_t off = ((ks / 4) * P::kTile + (ks % 4) * 32) >> 4;
                            tc_mma(d_s, q_desc + off, kd + off, idesc, ks > 0);
                        }
                    }
                    tc_commit(bar(P::bSFull + t));
                    tc_commit(bar(P::bKVEmpty + s_slot));
                    if (kMixed && dual) tc_commit(bar(P::bKVEmpty + s_slot));
                    if (j + 2 == nb) {
                        tc_commit(bar(P::bQFree + q_bar));
                        if (kMixed && !dual && t == 0) tc_commit(bar(P::bQFree));
                    }
                    advance(s_slot, s_lap, stride);
                };
                auto values = [&]() {
                    const int gb = blk + j, keys = min(kBN, (kend - block * kBN + 15) & ~15), seen = klen - block * kBN;
                    wait_two(bar(P::bKVFull + v_slot), v_lap, bar(P::bPFull + 2 * t), gb & 1, 230 + 2 * t);
                    if (j == 0 && items > 0) wait_bar(bar(P::bOFree + t), (items - 1) & 1, 250 + t);
                    if (!ok) return;
                    if (seen < keys) {
                        // Rows past the sequence's keys may hold anything (a cache past its length, a
                        // packed neighbour), and P = 0 times an infinity would still poison the
                        // output. (Pair: both tiles' warps write the same zeros.)
                        unsigned char* vt = smem + P::kRing + v_slot * P::kOperand;
                        const int rows = keys - seen;
#pragma unroll 1
                        for (int i = lane; i < P::kSub * rows * 8; i += 32) {
                            const int sub = i >= rows * 8 ? 1 : 0, rem = i - sub * (rows * 8);
                            *reinterpret_cast<uint4*>(vt + sub * P::kTile + (seen + (rem >> 3)) * 128 + (rem & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
                        }
                        fence_async_smem();
                        __syncwarp();
                    }
                    tc_fence_after();
                    const uint64_t vd = v_desc + static_cast<uint32_t>(v_slot * (P::kOperand >> 4));
                    // A: P, 8 TMEM columns per 16 keys. B: V MN-major, 16 keys = 16 rows of 128 bytes;
                    // the second 64 columns of Dv are one sub-tile further (LBO).
                    const bool whole = keys == kBN && p.dv == DP;
                    if (whole) {
#pragma unroll
                        for (int ks = 0; ks < 4; ++ks) tc_mma_ts(d_o, a_p + ks * 8, vd + ((ks * 2048) >> 4), instr_desc(DP, true), (j > 0 || ks > 0) ? 1u : 0u);
                    }
                    if constexpr (P::kPOverS) {
                        wait_bar(bar(P::bPFull + 2 * t + 1), gb & 1, 240 + t);
                        if (!ok) return;
                        tc_fence_after();
                    }
                    if (whole) {
#pragma unroll
                        for (int ks = 4; ks < 8; ++ks) tc_mma_ts(d_o, a_p + ks * 8, vd + ((ks * 2048) >> 4), instr_desc(DP, true), 1u);
                    } else {
                        const uint32_t idesc = instr_desc((p.dv + 15) & ~15, true);
#pragma unroll 1
                        for (int ks = 0; ks < keys >> 4; ++ks) tc_mma_ts(d_o, a_p + ks * 8, vd + ((ks * 2048) >> 4), idesc, (j > 0 || ks > 0) ? 1u : 0u);
                    }
                    tc_commit(bar(P::bPVDone + t));
                    tc_commit(bar(P::bKVEmpty + v_slot));
                    if (kMixed && dual) tc_commit(bar(P::bKVEmpty + v_slot));
                    advance(v_slot, v_lap, stride);
                };
                if constexpr (P::kPOverS) {
                    if (j >= 0) values();
                    if (more) scores();
                } else {
                    if (more) scores();
                    if (j >= 0) values();
                }
                block = s_block;
            }
            if (!dual && t && nb < entries) {
                // Blocks that only tile A sees: this warp's release of their ring tiles. (Not before
                // they have been loaded: the arrival must not fall into the slot's previous use.)
                for (int e = 0; ok && e < 2 * (entries - nb); ++e) {
                    wait_bar(bar(P::bKVFull + s_slot), s_lap, 260 + t);
                    if (lane == 0) mbar_arrive(bar(P::bKVEmpty + s_slot));
                    __syncwarp();
                    advance(s_slot, s_lap, 1);
                }
            }
            if (dual && nb == 0) {   // Q is released by both
                wait_bar(bar(P::bQFull), q_items & 1, 204);
                if (lane == 0) mbar_arrive(bar(P::bQFree));
                __syncwarp();
            }
            if (nb > 0) ++items;
            if (kMixed) {
                ++q_a;
                if (!dual && nb > 0 && t) ++q_b;
            } else if (nb > 0 || dual) {
                ++q_a;
            }
            blk += nb;
            // 2 * entries can be several times round the ring.
            for (int left = 2 * entries; left > 0; left -= P::kSlots) advance(base, base_lap, min(left, P::kSlots));
        }
      }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSoftmaxRegs));
        // ---------------- softmax: thread = query row of tile t ----------------
        const int t = warp >> 2;
        const int row = (warp & 3) * 32 + lane;         // row inside the tile = TMEM lane
        const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const uint32_t s_addr = tmem + lane_addr + (t ? 128 : 0);
        const uint32_t p_addr = tmem + lane_addr + P::kP + t * P::kPStep;
        const uint32_t o_addr = tmem + lane_addr + P::kO + t * DP;
        int blk = 0;        // key blocks of this tile so far: parity of its barriers
        int shared = 0;     // dual: items in which B had a part
        bool ok = true;
        auto wait_for = [&](int b, int parity, int code) { ok = ok && wait_one(bar(b), parity, abort_flag, code); };
        const float sc = p.scale_log2;
        int turns = 0;      // turns taken so far, the same number by either tile
        const uint32_t my_turn = bar(P::bTurn + t * 4 + (warp & 3)), their_turn = bar(P::bTurn + (1 - t) * 4 + (warp & 3));

        for (int n = 0; ok; ++n) {
            Item k;
            if (!take_item(n, k, ok)) break;
            if (!(t ? k.valid[1] : k.valid[0])) {
                give_item(n);
                continue;
            }
            const bool dual = kMixed ? k.dual != 0 : all_dual;
            // (Selected once: an index that is not a constant would put the item into memory.)
            const int taking = kTurns ? k.n[1] : 0;   // the blocks both tiles have: B has no more than A
            const int nb = t ? k.n[1] : k.n[0], h = t ? k.h[1] : k.h[0], q0 = t ? k.q0[1] : k.q0[0], kend = t ? k.kend[1] : k.kend[0];
            const int qi = q0 + row;                    // row inside the sequence
            const bool real = qi < k.si.lq;
            if (nb == 0) {
                // No key is visible to this tile: zeros, lse = -inf, and no barrier is involved.
                // (Dual: tile A answers for both; B has no part of a tile with one key block.)
                if (real && !(dual && t == 1)) {
                    __nv_bfloat16* og = p.out + k.b * p.os[0] + h * p.os[1] + static_cast<int64_t>(k.si.q_off + qi) * p.os[2];
                    for (int c = 0; c < p.dv; c += 8) *reinterpret_cast<uint4*>(og + c) = make_uint4(0u, 0u, 0u, 0u);
                    if (p.lse) p.lse[k.b * p.ls[0] + h * p.ls[1] + (k.si.q_off + qi) * p.ls[2]] = -INFINITY;
                }
                give_item(n);
                continue;
            }
            // Keys this row may see: [0, row_limit). The smallest limit of the warp is its first
            // row's, the largest its last row's. A warp without a row of the sequence does no
            // arithmetic; what its rows of P hold reaches only rows of O that nobody reads.
            const bool idle = q0 + (warp & 3) * 32 >= k.si.lq;
            auto limit_of = [&](int i) { return p.causal ? min(kend, i + k.si.shift + 1) : kend; };
            const int row_limit = limit_of(qi), limit_lo = limit_of(q0 + (warp & 3) * 32), limit_hi = limit_of(q0 + (warp & 3) * 32 + 31);
            float m_ref = -INFINITY;   // reference maximum (base-2 logits), moved lazily
            float2 l2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
            Iter it;
            it.start(tp, k, (dual && t == 1) ? k.n[0] : 0);
            const uint8_t* kinds = nullptr;
            int64_t piece0 = 0;        // plan: index of this warp's first piece
            if constexpr (kMask == 2) {
                const MaskPlan& m = tp.plan;
                const int g = min((q0 >> 5) + (warp & 3), m.groups - 1);
                const int plane = (m.batched ? k.b * m.heads : 0) + (m.heads > 1 ? h : 0);
                piece0 = (static_cast<int64_t>(plane) * m.groups + g) * m.blocks;
                kinds = m.kind + piece0;
            }

            // A block's mask term is fetched one block ahead. (The kind of a plan's piece as well cost
            // more in registers than it gave: 57.1 -> 58.7 us on 2 x 16 heads x 2048, causal mask.)
            auto term_of = [&](int blk_) {   // (-inf past the last key of the tile: such a block needs no other test)
                const int key = blk_ * kBN + row;
                return key < kend ? mask_value(p, k.b, h, 0, static_cast<int64_t>(k.si.k_off) + key) * kLog2e : -INFINITY;
            };
            float term_ahead = 0.f;
            if constexpr (kMask == 1) term_ahead = term_of(it.at);
            for (int j = 0; ok && j < nb; ++j) {
                const int gb = blk + j;
                const int block = it.next();
                const int limit = row_limit - block * kBN;        // my columns [0, limit) are visible
                const int lo = limit_lo - block * kBN;
                int chunks = min(max(limit_hi - block * kBN + 31, 0) >> 5, 4);   // 32-column chunks with a visible key
                int stored = min((kend - block * kBN + 31) >> 5, 4);             // chunks that P V reads
                int kind = kNoEffect;
                const float* mrow = nullptr;
                if constexpr (kMask == 1) {
                    // One thread per column fetches the block's mask term, the tile's threads share
                    // the row through shared memory. (A bounded mbarrier, not bar.sync: a warp that
                    // gave up elsewhere must not strand the others. Two rows alternate: a row is
                    // written again only after everybody has arrived for the block between.)
                    float* rows = reinterpret_cast<float*>(smem + P::kMaskRow) + (t * 2 + (gb & 1)) * 128;
                    rows[row] = term_ahead;
                    if (j + 1 < nb) term_ahead = term_of(block + 1);
                    mbar_arrive_warp(bar(P::bMask + t));
                    wait_for(P::bMask + t, gb & 1, 340 + t);
                    if (!ok) break;
                    mrow = rows;
                }
                if constexpr (kMask == 2) {
                    kind = kinds[block];
                    if (kind == kHidden) chunks = 0;
                }
                if (idle) chunks = stored = 0;
                // A block every key of which every row of this warp sees, without a mask term or with one
                // that is the same for all rows: the scores go into registers once, in straight-line code.
                // Any other block (the diagonal, the last keys, a mask with a row per query) takes two
                // loops over 32-column chunks: the first puts the finished logits back in their place.
                // (Keys past the end of K are zeros from TMA, and their scores too: the score product covers
                // every chunk that is read. Past a length they are anything.)
                const bool fast = kMask == 1 ? !p.causal && (lo >= kBN || (!p.cu_k && kend == p.sk)) && !idle : lo >= kBN && (kMask == 0 || kind == kNoEffect) && !idle;
                uint4 held = make_uint4(0u, 0u, 0u, 0u);   // plan: this row's visibility bits
                if (kMask == 2 && kind == kYesNo) held = tp.plan.bits[(piece0 + block) * 32 + lane];
                wait_for(P::bSFull + t, gb & 1, 300 + t);
                if (!ok) break;
                tc_fence_after();

                float s[128];
                float mx[2] = {-INFINITY, -INFINITY};
                auto chunk_max = [&](const float* x) {
#pragma unroll
                    for (int e = 0; e < 32; e += 4) {
                        mx[0] = max3(mx[0], x[e], x[e + 1]);
                        mx[1] = max3(mx[1], x[e + 2], x[e + 3]);
                    }
                };
                float fs = kMask == 1 ? 1.f : sc;   // what is left to scale the registers' values by
                if (fast) {
                    tmem_ld32(s_addr, s);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        if (kMask == 1 && c >= stored) continue;
                        float* x = s + c * 32;
                        tmem_wait_ld();
                        if (c < 3 && !(kMask == 1 && c + 1 >= stored)) tmem_ld32(s_addr + (c + 1) * 32, s + (c < 3 ? c + 1 : 3) * 32);
                        else if (!P::kPOverS) {
                            // The scores are in registers: the next Q K^T may have their columns.
                            tc_fence_before();
                            mbar_arrive_warp(bar(P::bSFree + t));
                        }
                        if constexpr (kMask == 1) {
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                const float4 m4 = reinterpret_cast<const float4*>(mrow + c * 32)[e];
                                x[e * 4] = fmaf(x[e * 4], sc, m4.x);
                                x[e * 4 + 1] = fmaf(x[e * 4 + 1], sc, m4.y);
                                x[e * 4 + 2] = fmaf(x[e * 4 + 2], sc, m4.z);
                                x[e * 4 + 3] = fmaf(x[e * 4 + 3], sc, m4.w);
                            }
                        }
                        chunk_max(x);
                    }
                } else {
                    fs = 1.f;
#pragma unroll 1
                    for (int c = 0; c < chunks; ++c) {
                        float x[32];
                        tmem_ld32(s_addr + c * 32, x);
                        if constexpr (kMask == 2) {
                            if (kind == kValues && !tp.plan.wide) {
                                const uint4* v = tp.plan.values + ((piece0 + block) * 16 + c * 4) * 32 + lane;
                                uint4 q[4];
#pragma unroll
                                for (int e = 0; e < 4; ++e) q[e] = v[e * 32];
                                tmem_wait_ld();
#pragma unroll
                                for (int e = 0; e < 4; ++e) {
                                    const uint32_t u[4] = {q[e].x, q[e].y, q[e].z, q[e].w};
#pragma unroll
                                    for (int i = 0; i < 4; ++i) {
                                        const float m0 = fmaxf(__uint_as_float(u[i] << 16), kMaskedLogit), m1 = fmaxf(__uint_as_float(u[i] & 0xffff0000u), kMaskedLogit);
                                        x[e * 8 + i * 2] = fmaf(x[e * 8 + i * 2], sc, m0 * kLog2e);
                                        x[e * 8 + i * 2 + 1] = fmaf(x[e * 8 + i * 2 + 1], sc, m1 * kLog2e);
                                    }
                                }
                            } else if (kind == kValues) {
                                const float4* v = reinterpret_cast<const float4*>(tp.plan.values) + ((piece0 + block) * 32 + c * 8) * 32 + lane;
                                float4 q[8];
#pragma unroll
                                for (int e = 0; e < 8; ++e) q[e] = v[e * 32];
                                tmem_wait_ld();
#pragma unroll
                                for (int e = 0; e < 8; ++e) {
                                    x[e * 4] = fmaf(x[e * 4], sc, fmaxf(q[e].x, kMaskedLogit) * kLog2e);
                                    x[e * 4 + 1] = fmaf(x[e * 4 + 1], sc, fmaxf(q[e].y, kMaskedLogit) * kLog2e);
                                    x[e * 4 + 2] = fmaf(x[e * 4 + 2], sc, fmaxf(q[e].z, kMaskedLogit) * kLog2e);
                                    x[e * 4 + 3] = fmaf(x[e * 4 + 3], sc, fmaxf(q[e].w, kMaskedLogit) * kLog2e);
                                }
                            } else if (kind != kNoEffect) {
                                const uint32_t word = c == 0 ? held.x : c == 1 ? held.y : c == 2 ? held.z : held.w;
                                tmem_wait_ld();
#pragma unroll
                                for (int e = 0; e < 32; ++e) x[e] = fmaf(x[e], sc, (word >> e) & 1u ? 0.f : kMaskedLogit * kLog2e);
                            } else {
                                tmem_wait_ld();
#pragma unroll
                                for (int e = 0; e < 32; ++e) x[e] *= sc;
                            }
                        } else {
                            tmem_wait_ld();
#pragma unroll
                            for (int e = 0; e < 32; ++e) x[e] = kMask == 1 ? fmaf(x[e], sc, mrow[c * 32 + e]) : x[e] * sc;
                        }
                        if (lo < c * 32 + 32) {
#pragma unroll
                            for (int e = 0; e < 32; ++e) x[e] = c * 32 + e < limit ? x[e] : -INFINITY;
                        }
                        tmem_st32(s_addr + c * 32, x);
                        chunk_max(x);
                    }
                    tmem_wait_st();
                }
                const float top = fmaxf(mx[0], mx[1]) * fs;

                // Lazy rescale: move the reference only when this block exceeds it by 2^8.
                const bool move = top > m_ref + kRescaleGap;
                if (__any_sync(0xffffffffu, move)) {
                    float f = 1.f;
                    if (move) {
                        f = fast_exp2(m_ref - top);   // 0 on the first block
                        m_ref = top;
                        l2[0] = __fmul2_rn(l2[0], make_float2(f, f));
                        l2[1] = __fmul2_rn(l2[1], make_float2(f, f));
                    }
                    if (j > 0) {
                        // O holds blocks [0, j): wait for block j - 1's P V.
                        wait_for(P::bPVDone + t, (gb - 1) & 1, 310 + t);
                        if (!ok) break;
                        tc_fence_after();
#pragma unroll 1
                        for (int c = 0; c < DP / 16; ++c) {   // small chunks: this rare path claims no registers
                            float o[16];
                            tmem_ld16(o_addr + c * 16, o);
                            tmem_wait_ld();
#pragma unroll
                            for (int e = 0; e < 16; ++e) o[e] *= f;
                            tmem_st16(o_addr + c * 16, reinterpret_cast<const uint32_t*>(o));
                        }
                        tmem_wait_st();
                    }
                }
                const float m_use = (m_ref == -INFINITY) ? 0.f : m_ref;

                // Tile A goes first: its turn follows B's block before, B's follows A's same block.
                if (kTurns && (t ? taking > 0 : taking > 0 && j <= taking && turns + j > 0)) {
                    ok = ok && wait_one(my_turn, (turns + j - 1 + t) & 1, abort_flag, 390 + t);
                    if (!ok) break;
                }
                auto end_turn = [&]() {
                    if (kTurns && j < taking && lane == 0) mbar_arrive(their_turn);
                };

                // ---- P = 2^(logit - m) as packed bf16 pairs ----
                const float2 sc2 = make_float2(fs, fs), nm2 = make_float2(-m_use, -m_use);
                // P's columns are free once the previous block's P V has read them.
                auto wait_p_free = [&]() {
                    if (!P::kPOverS && j > 0) {
                        wait_for(P::bPVDone + t, (gb - 1) & 1, 320 + t);
                        tc_fence_after();
                    }
                };
                if (fast) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        if (kMask == 1 && c >= stored) continue;
                        uint32_t wv[16];
                        const float* x = s + c * 32;
#pragma unroll
                        for (int e = 0; e < 16; ++e) {
                            const float2 y = __ffma2_rn(make_float2(x[2 * e], x[2 * e + 1]), sc2, nm2);
                            float2 pr;
                            // The polynomial pairs are spread evenly: MUFU and FMA work alternate.
                            // (Terms may hide a key; those take MUFU, whose 2^-inf is exactly 0.)
                            if (kMask != 1 && (e * P::kPolyPairs) % 8 < P::kPolyPairs) {
                                pr = exp2_poly2(y);
                            } else {
                                pr.x = fast_exp2(y.x);
                                pr.y = fast_exp2(y.y);
                            }
                            l2[e & 1] = __fadd2_rn(l2[e & 1], pr);
                            wv[e] = pack_bf16(pr.x, pr.y);
                        }
                        if (c == 0) wait_p_free();
                        if (c == 2) end_turn();   // (the rest of this block runs beside the other's start)
                        tmem_st16(p_addr + c * 16, wv);
                        if (P::kPOverS && (c == 1 || (kMask == 1 && c == 0 && stored == 1))) {
                            // P V may start on the first half of the keys.
                            tmem_wait_st();
                            tc_fence_before();
                            mbar_arrive_warp(bar(P::bPFull + 2 * t));
                        }
                    }
                } else {
                    // (Idle warps wait too: one that did not could get a whole item ahead and find a
                    // barrier's parity right for the wrong reason.)
                    wait_p_free();
#pragma unroll 1
                    for (int c = 0; c < stored; ++c) {
                        uint32_t wv[16];
                        if (c < chunks) {
                            float x[32];
                            tmem_ld32(s_addr + c * 32, x);
                            tmem_wait_ld();
#pragma unroll
                            for (int e = 0; e < 16; ++e) {
                                const float2 y = __fadd2_rn(make_float2(x[2 * e], x[2 * e + 1]), nm2);
                                const float2 pr = make_float2(fast_exp2(y.x), fast_exp2(y.y));
                                l2[e & 1] = __fadd2_rn(l2[e & 1], pr);
                                wv[e] = pack_bf16(pr.x, pr.y);
                            }
                        } else {
#pragma unroll
                            for (int e = 0; e < 16; ++e) wv[e] = 0u;
                        }
                        tmem_st16(p_addr + c * 16, wv);
                    }
                    end_turn();
                    tmem_wait_st();
                    tc_fence_before();
                    mbar_arrive_warp(bar(P::kPOverS ? P::bPFull + 2 * t : P::bSFree + t));
                }
                if (!ok) break;
                tmem_wait_st();
                tc_fence_before();
                mbar_arrive_warp(bar(P::bPFull + 2 * t + (P::kPOverS ? 1 : 0)));
            }
            if (!ok) break;

            // ---- the item's end: O / l to memory ----
            // (The item is read from the queue again: its numbers would not fit beside the scores.)
            const Item* e = queue + n % P::kQueue;
            const bool halves = kMixed ? e->dual != 0 : all_dual;
            const int nb_other = e->n[1], e_b = e->b, e_h = e->h[halves ? 0 : t], e_q0 = e->q0[halves ? 0 : t], e_lq = e->si.lq, e_off = e->si.q_off;
            const int last = blk + nb - 1;
            blk += nb;
            turns += taking;
            float l_row = (l2[0].x + l2[0].y) + (l2[1].x + l2[1].y), m_row = m_ref;
            float f_mine = 1.f, f_other = 0.f;
            const bool merge = halves && nb_other > 0;
            if (merge) {
                wait_for(P::bPVDone + t, last & 1, 330 + t);
                if (!ok) break;
                tc_fence_after();
                float2* part = reinterpret_cast<float2*>(smem + P::kPartial);
                if (t == 1) {
                    // Tile A's threads take this half out of tensor memory and free it.
                    part[row] = make_float2(m_row, l_row);
                    tc_fence_before();
                    mbar_arrive_warp(bar(P::bPartial));
                    give_item(n);
                    continue;
                }
                wait_for(P::bPartial, shared & 1, 380);
                ++shared;
                if (!ok) break;
                tc_fence_after();
                const float2 other = part[row];
                const float m_all = fmaxf(m_row, other.x);
                const float base_m = (m_all == -INFINITY) ? 0.f : m_all;
                f_mine = fast_exp2(m_row - base_m);
                f_other = fast_exp2(other.x - base_m);
                l_row = fmaf(other.y, f_other, l_row * f_mine);
                m_row = m_all;
            }
            const float inv = l_row > 0.f ? 1.f / l_row : 0.f;
            // (Without a merge the statistics leave while the last P V runs.)
            if (p.lse && e_q0 + row < e_lq) {
                p.lse[e_b * p.ls[0] + e_h * p.ls[1] + (e_off + e_q0 + row) * p.ls[2]] = l_row > 0.f ? kLn2 * (m_row + log2f(l_row)) : -INFINITY;
            }
            if (!merge) {
                wait_for(P::bPVDone + t, last & 1, 332 + t);
                if (!ok) break;
                tc_fence_after();
            }
            // A warp's 32 rows, 32 columns at a time. Four lanes exchange their rows' 16-byte pieces
            // first, so that a store writes 64 bytes of each of eight rows (a thread's own row straight
            // to memory is a line of its own for every piece: 4,300 clk for 128 rows of 80, now 3,100).
            const int r0 = e_q0 + (warp & 3) * 32 + (lane & ~3);
            __nv_bfloat16* og = p.out + e_b * p.os[0] + e_h * p.os[1] + static_cast<int64_t>(e_off + r0) * p.os[2] + (lane & 3) * 8;
#pragma unroll 1
            for (int c = 0; c * 32 < p.dv; ++c) {
                float o[32];
                tmem_ld32(o_addr + c * 32, o);
                if (merge) {
                    float o1[32];
                    tmem_ld32(tmem + lane_addr + P::kO + DP + c * 32, o1);
                    tmem_wait_ld();
#pragma unroll
                    for (int e = 0; e < 32; ++e) o[e] = fmaf(o1[e], f_other, o[e] * f_mine);
                } else {
                    tmem_wait_ld();
                }
                if (c * 32 + 32 >= p.dv) {
                    // O is in registers: the next item's P V may overwrite it.
                    tc_fence_before();
                    mbar_arrive_warp(bar(P::bOFree + t));
                    if (merge) mbar_arrive_warp(bar(P::bOFree + 1));
                }
                uint32_t w[4][4];   // [piece][word]; after the exchange [row][word] of piece lane & 3
#pragma unroll
                for (int e = 0; e < 16; ++e) w[e >> 2][e & 3] = pack_bf16(o[2 * e] * inv, o[2 * e + 1] * inv);
#pragma unroll
                for (int x = 1; x < 4; x <<= 1) {
                    const bool odd = lane & x;
#pragma unroll
                    for (int a = 0; a < 4; ++a) {
                        if (a & x) continue;
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? w[a][i] : w[a + x][i], x);
                            if (odd) w[a][i] = got; else w[a + x][i] = got;
                        }
                    }
                }
                const bool inside = c * 32 + (lane & 3) * 8 < p.dv;
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    if (inside && r0 + a < e_lq) *reinterpret_cast<uint4*>(og + a * p.os[2] + c * 32) = make_uint4(w[a][0], w[a][1], w[a][2], w[a][3]);
                }
            }
            give_item(n);
        }
    }

    // Teardown: everyone arrives (all waits above are bounded), then the allocating warp frees
    // tensor memory.
    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        if (*abort_flag) {
            if (lane == 0) atomicCAS_system(tp.status, 0, *abort_flag);
            const long long t0 = clock64();
            while (clock64() - t0 < 2000000) {
            }
        }
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// ---- masks with a row per query ----------------------------------------------------------
//
// One CTA per 32 query rows of a plane walks the keys once, a warp per row, four blocks of 128
// keys at a time. It is not bound by reading the mask once (2 x 2048 x 2048 bf16 terms: 2.6 us of the
// copy bandwidth; DRAM 12 % busy) but by what it does per term in the few CTAs there are: the ALU
// pipes of 128 SMs are 71 % busy, and each of four rounds ends at a barrier (16.7 us under ncu with
// cold caches, about 8 in a stream). Pieces without values to apply cost nothing further, and what
// the attention kernel reads back is the bits or values of the pieces that have any. The code is kept
// small (a type per instance, one row per warp): with four rows per warp and the type looked up per
// load it was 85 to 106 KB of straight-line instructions that every pass fetched again; that call (2 x
// 16 heads, D 64) 103 -> 75 us.
//
// A block is hidden from a group when every term of it is at the floor (-5e5): its weights are
// exactly 0 as long as each row of the group keeps a key well above the floor. A group with a
// row that does not (a row that sees nothing) has none of its blocks left out.
constexpr float kSafeTerm = 0.5f * kMaskedLogit;
constexpr int kPlanUnroll = 4, kPlanThreads = 1024;

// The term at `idx`.
template <int kType>
__device__ __forceinline__ float mask_term(const void* mask, int64_t idx) {
    if constexpr (kType == KTT_B200_MASK_BOOL) return __ldg(static_cast<const uint8_t*>(mask) + idx) ? 0.f : kMaskedLogit;
    if constexpr (kType == KTT_B200_MASK_BF16) return __uint_as_float(static_cast<uint32_t>(__ldg(static_cast<const uint16_t*>(mask) + idx)) << 16);
    if constexpr (kType == KTT_B200_MASK_F16) return __half2float(__ldg(static_cast<const __half*>(mask) + idx));
    return __ldg(static_cast<const float*>(mask) + idx);
}
// The four terms from `idx`, in one load.
template <int kType>
__device__ __forceinline__ void mask_terms(const void* mask, int64_t idx, float (&v)[4]) {
    if constexpr (kType == KTT_B200_MASK_BOOL) {
        const uint32_t x = __ldg(reinterpret_cast<const uint32_t*>(static_cast<const uint8_t*>(mask) + idx));
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = (x >> (8 * e)) & 0xffu ? 0.f : kMaskedLogit;
    } else if constexpr (kType == KTT_B200_MASK_F32) {
        const float4 x = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(mask) + idx));
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    } else {
        const uint2 x = __ldg(reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(mask) + idx));
        if constexpr (kType == KTT_B200_MASK_BF16) {
            v[0] = __uint_as_float(x.x << 16); v[1] = __uint_as_float(x.x & 0xffff0000u);
            v[2] = __uint_as_float(x.y << 16); v[3] = __uint_as_float(x.y & 0xffff0000u);
        } else {
            const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&x.x)), hi = __half22float2(*reinterpret_cast<const __half2*>(&x.y));
            v[0] = lo.x; v[1] = lo.y; v[2] = hi.x; v[3] = hi.y;
        }
    }
}

// `vec`: the keys are contiguous and every row of the mask starts on a multiple of four terms, so
// that a lane reads its four keys in one load.
template <int kType>
__global__ void __launch_bounds__(kPlanThreads) mask_plan_kernel(const AttnParams p, const MaskPlan m, int32_t* header, const bool vec) {
    __shared__ uint32_t seen[kMaxPlanBlocks];   // per block: 1 floor, 2 zero, 4 anything else
    __shared__ int unsafe;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int plane = blockIdx.x, g = blockIdx.y;   // (x: there may be more planes than the 65,535 of y)
    const int pb = plane / m.heads, ph = plane - pb * m.heads;
    const int rr = threadIdx.x >> 5, lane = threadIdx.x & 31;   // row of the group, position in the row
    for (int i = threadIdx.x; i < m.blocks; i += kPlanThreads) seen[i] = 0;
    if (threadIdx.x == 0) unsafe = 0;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // The attention kernel's work counters: this launch comes first in the stream.
    if (g == 0 && plane == 0 && threadIdx.x < 2) header[threadIdx.x] = 0;
    __syncthreads();
    const int64_t piece0 = (static_cast<int64_t>(plane) * m.groups + g) * m.blocks;
    const int row = g * 32 + rr;
    const bool real = row < p.sq;
    const int64_t at = pb * p.ms[0] + ph * p.ms[1] + static_cast<int64_t>(min(row, p.sq - 1)) * p.ms[2];
    float best = -INFINITY;   // the row's largest term so far
#pragma unroll 1
    for (int b0 = 0; b0 < m.blocks; b0 += kPlanUnroll) {
        float v[kPlanUnroll][4];
#pragma unroll
        for (int u = 0; u < kPlanUnroll; ++u) {
            const int col = (b0 + u) * 128 + lane * 4;
#pragma unroll
            for (int e = 0; e < 4; ++e) v[u][e] = kMaskedLogit;
            if (vec && col + 3 < p.sk) mask_terms<kType>(p.mask, at + col, v[u]);
        }
        if (!vec || (b0 + kPlanUnroll) * 128 > p.sk) {   // terms apart, and the last ones of a row
#pragma unroll
            for (int u = 0; u < kPlanUnroll; ++u) {
                const int col = (b0 + u) * 128 + lane * 4;
                if (vec && col + 3 < p.sk) continue;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    if (col + e < p.sk) v[u][e] = mask_term<kType>(p.mask, at + (col + e) * p.ms[3]);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kPlanUnroll; ++u) {
            uint32_t flags = 0;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                // Columns past the last key count as hidden; they decide nothing.
                const float x = v[u][e];
                const uint32_t f = !(x > kMaskedLogit) ? 1u : x == 0.f ? 2u : 4u;
                if ((b0 + u) * 128 + lane * 4 + e < p.sk) flags |= f;
                if (f != 1u) best = fmaxf(best, x);
            }
            flags = __reduce_or_sync(0xffffffffu, flags);
            if (lane == 0 && b0 + u < m.blocks && real) atomicOr(&seen[b0 + u], flags);
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kPlanUnroll; ++u) {
            if (b0 + u >= m.blocks) break;
            const uint32_t f = seen[b0 + u];
            const int64_t piece = piece0 + b0 + u;
            if (f & 4u) {
                if (m.wide) {
                    reinterpret_cast<float4*>(m.values)[(piece * 32 + lane) * 32 + rr] = make_float4(v[u][0], v[u][1], v[u][2], v[u][3]);
                } else {
                    // bf16 in, bf16 out: the upper halves, two lanes to a 16-byte chunk
                    uint2 w;
                    w.x = __byte_perm(__float_as_uint(v[u][0]), __float_as_uint(v[u][1]), 0x7632);
                    w.y = __byte_perm(__float_as_uint(v[u][2]), __float_as_uint(v[u][3]), 0x7632);
                    reinterpret_cast<uint2*>(m.values + (piece * 16 + (lane >> 1)) * 32 + rr)[lane & 1] = w;
                }
            } else if (f == 3u) {
                // Four bits per lane; eight lanes make a word, four words a row.
                uint32_t x = 0;
#pragma unroll
                for (int e = 0; e < 4; ++e) x |= (v[u][e] > kMaskedLogit ? 1u : 0u) << (4 * (lane & 7) + e);
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) x |= __shfl_xor_sync(0xffffffffu, x, o);
                if ((lane & 7) == 0) reinterpret_cast<uint32_t*>(m.bits + piece * 32 + rr)[lane >> 3] = x;
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
    if (lane == 0 && real && !(best > kSafeTerm)) unsafe = 1;
    __syncthreads();
    for (int i = threadIdx.x; i < m.blocks; i += kPlanThreads) {
        const uint32_t f = seen[i];
        m.kind[piece0 + i] = (f & 4u) ? kValues : f == 3u ? kYesNo : f == 2u ? kNoEffect : unsafe ? kAllFloor : kHidden;
    }
    if (rr < m.words) {   // (at most 1,024 blocks: 32 words, a warp each)
        const int i = rr * 32 + lane;
        const uint32_t bits = __ballot_sync(0xffffffffu, i < m.blocks && (unsafe || seen[i] != 1u));
        if (lane == 0) m.active[(static_cast<int64_t>(plane) * m.groups + g) * m.words + rr] = bits;
    }
}

// ---- host side ---------------------------------------------------------------------------

bool mask_needs_plan(const AttnParams& p) { return p.mask_dtype != KTT_B200_MASK_NONE && p.ms[2] != 0 && p.sq > 1; }

int64_t up256(int64_t x) { return (x + 255) / 256 * 256; }

// Sizes of a plan and its place in `base` (null: sizes only); returns its bytes.
int64_t plan_layout(const AttnParams& p, unsigned char* base, MaskPlan* m) {
    m->groups = (p.sq + 31) / 32;
    m->blocks = (p.sk + kBN - 1) / kBN;
    m->words = (m->blocks + 31) / 32;
    m->heads = p.ms[1] != 0 ? p.heads : 1;
    m->batched = p.ms[0] != 0 ? 1 : 0;
    m->wide = (p.mask_dtype == KTT_B200_MASK_F32 || p.mask_dtype == KTT_B200_MASK_F16) ? 1 : 0;
    const int64_t planes = static_cast<int64_t>(m->heads) * (m->batched ? p.batch : 1);
    const int64_t pieces = planes * m->groups * m->blocks;
    const int64_t active = up256(planes * m->groups * m->words * 4), kind = up256(pieces), bits = up256(pieces * 32 * 16);
    const int64_t values = p.mask_dtype == KTT_B200_MASK_BOOL ? 0 : pieces * 32 * 128 * (m->wide ? 4 : 2);
    m->active = reinterpret_cast<uint32_t*>(base);
    m->kind = base + active;
    m->bits = reinterpret_cast<uint4*>(base + active + kind);
    m->values = reinterpret_cast<uint4*>(base + active + kind + bits);
    return active + kind + bits + values;
}

// A plan is written a part of the call at a time - batch entries, then heads, then query rows - so that it
// takes at most this much memory however large the mask is.
constexpr int64_t kMostPlan = 1ll << 30;
struct PlanPart {
    int batch, heads, rows;
};

int64_t plan_bytes(const AttnParams& p, const PlanPart& part) {
    AttnParams s = p;
    MaskPlan m;
    s.batch = part.batch;
    s.heads = part.heads;
    s.sq = part.rows;
    return plan_layout(s, nullptr, &m);
}

// The smallest part there is: a query tile of one plane.
PlanPart least_part(const AttnParams& p) { return {p.ms[0] ? 1 : p.batch, p.ms[1] ? 1 : p.heads, p.sq < kBM ? p.sq : kBM}; }

int sm_count() {
    static int sms[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (!sms[dev]) {
        int n = 148;
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        sms[dev] = n;
    }
    return sms[dev];
}

// The parts to plan at a time so that a plan fits `room` bytes (or the smallest ones).
PlanPart plan_part(const AttnParams& p, int64_t room) {
    PlanPart part = {p.batch, p.heads, p.sq};
    if (plan_bytes(p, part) <= room) return part;
    auto cut = [&](int& n, int step) {
        if (n <= step || plan_bytes(p, part) <= room) return;
        const int64_t whole = n;
        n = step;
        int64_t fit = room / plan_bytes(p, part);   // steps (rounding makes several no larger than their sum)
        if (fit < 1) fit = 1;
        // Of the upper half of what fits, the size whose parts leave the fewest SMs idle: 32 heads of 4096 x
        // 4096 fp32 terms, D 64, at 1 GB in parts of 11 heads 3,292 us, of 9 2,715 (whole 2,570).
        float least = 0.f;
        int64_t best = fit;
        for (int i = 0; i < 16; ++i) {
            const int64_t steps = fit - fit * i / 32;
            n = static_cast<int>(steps * step < whole ? steps * step : whole);
            const int64_t units = static_cast<int64_t>((part.rows + kBM - 1) / kBM) * part.heads * part.batch, sms = sm_count();
            const float rounds = units <= sms && p.sk > kBN ? 0.5f : static_cast<float>((units + 2 * sms - 1) / (2 * sms));
            const float cost = rounds * static_cast<float>((whole + n - 1) / n);
            if (i == 0 || cost < least) {
                least = cost;
                best = n;
            }
        }
        n = static_cast<int>(best);
    };
    const int group = p.heads / p.kv_heads;
    if (p.ms[0]) cut(part.batch, 1);
    if (p.ms[1]) cut(part.heads, group);
    if (p.ms[1] && part.heads == group) cut(part.heads, 1);   // within the heads of one K / V head
    cut(part.rows, kBM);
    return part;
}

constexpr int64_t kMostTiles = 0x3fffffff;   // (query tile, head) pairs of a call
constexpr int64_t kHeaderBytes = 256;   // {int32 next item, int32 producers finished}

template <typename Kernel, typename... Args>
int launch_dependent(Kernel kernel, dim3 grid, int threads, int smem, cudaStream_t stream, const char* what, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return check_cuda(cudaLaunchKernelEx(&cfg, kernel, args...), what);
}

template <int DP>
int launch_pair(const AttnParams& p, const CUtensorMap (&maps)[3], PairParams& tp, int grid, cudaStream_t stream) {
    using P = PairPlan<DP>;
    const bool none = p.mask_dtype == KTT_B200_MASK_NONE, mixed = tp.cut > 0;
    auto kernel = mask_needs_plan(p) ? fwd_pair_kernel<DP, 2, false, false>
                : none ? (mixed ? fwd_pair_kernel<DP, 0, false, true> : fwd_pair_kernel<DP, 0, false, false>)
                       : (mixed ? fwd_pair_kernel<DP, 1, false, true> : fwd_pair_kernel<DP, 1, false, false>);
    if constexpr (P::kPOverS) {
        // Turns, without a mask, for pairs from five blocks of keys on: with three, their waits and the code for them
        // weigh more. Measured, us without and with: D 80, 16 heads x 4096 167 -> 153; D 96, 48 x 1025 52.5 ->
        // 49.3; D 80, 32 x 2048 causal 46.9 -> 45.0; 128 x 577 44.4 -> 43.3, 128 x 640 42.3 -> 40.4; but 256 x
        // 257 34.9 -> 35.9, D 128, 10 x 2048 queries x 300 keys 12.7 -> 13.4, and halves, D 80, 8 x 935 14.3 -> 14.6. (Head dims up to 64, whose scores
        // are ready in any case: 157 both, 20 x 4096. Masks with a row per query, D 128, 32 x 2048: 68.7 -> 71.1.)
        if (none && tp.duals > 0 && p.sk > 4 * kBN) kernel = mixed ? fwd_pair_kernel<DP, 0, true, true> : fwd_pair_kernel<DP, 0, true, false>;
    }
    if (int rc = ensure_smem(kernel, P::kBytes, "cudaFuncSetAttribute(fwd_pair)")) return rc;
    return launch_dependent(kernel, dim3(grid), kPairThreads, P::kBytes, stream, "fwd_pair launch", maps[0], maps[1], maps[2], tp);
}

}  // namespace

bool forward_pair_takes(const AttnParams& p) {
    if (p.d > 128 || p.dv > 128 || p.d % 8 || p.dv % 8) return false;
    // A plan covers the keys whatever a sequence's length, and 131,072 of them.
    if (mask_needs_plan(p) && (p.cu_q || p.key_lengths || p.sk > kMaxPlanBlocks * kBN)) return false;
    if (reinterpret_cast<uintptr_t>(p.out) & 15 || p.os[0] % 8 || p.os[1] % 8 || p.os[2] % 8) return false;
    // Items are counted in int32; a plan has its 32-row groups in y of its grid.
    if (static_cast<int64_t>((p.sq + kBM - 1) / kBM) * p.heads * p.batch > kMostTiles) return false;
    if (mask_needs_plan(p) && (p.sq + 31) / 32 > 65535) return false;
    const int64_t tq = p.cu_q ? p.total_q : p.sq, tk = p.cu_q ? p.total_k : p.sk;
    const int64_t bq = p.cu_q ? 1 : p.batch;
    int64_t s[3];
    const char* why;
    return operand_layout(p.q, tq, p.heads, bq, p.qs, s, &why) && operand_layout(p.k, tk, p.kv_heads, bq, p.ks, s, &why) &&
           operand_layout(p.v, tk, p.kv_heads, bq, p.vs, s, &why);
}

namespace {
// Pairs of equal length in rounds of one per SM, the last of which leaves half of the SMs or more without one:
// its tiles run as halves, each on an SM of its own.
bool last_round_in_halves(const AttnParams& p) {
    if (p.causal || p.cu_q || p.key_lengths || mask_needs_plan(p) || p.sk <= kBN) return false;
    const int64_t sms = sm_count(), group = p.heads / p.kv_heads, planes = static_cast<int64_t>(p.batch) * p.kv_heads;
    const int64_t per_plane = (p.sq + kBM - 1) / kBM * group, pairs = (per_plane + 1) / 2 * planes, over = pairs % sms;
    return per_plane * planes > sms && pairs > sms && over > 0 && 2 * over <= sms;
}
}  // namespace

namespace {
// Dense calls of head dim 64 or 128 without a mask: whether this kernel's pairs of tiles fill their rounds so
// much better than the other kernel's tiles (D 64: two halves of a tile's keys at a time, from six tiles per SM
// on whole tiles in two streams; D 128: whole tiles) that it ends sooner by the estimate below. What a call, an
// item, a block and, causal, a diagonal cost (us) is fitted to 490 calls of 20 to 1,200 tiles (D 64 within 5 %
// rms, D 128 within 4 and 6.5): prompts of 1 to 16 sequences, 100 to 4,096 rows, and non-causal ones of 200 to
// 4,608. The fit is of the kernels without halves in a last round and without turns, which the estimate has only the
// first of: at D 128 from five blocks of keys on a block is 1.90 us, not 2.20, so that calls stay with the other kernel there
// that this one would take as fast. The line is 8 % because none of 610 calls on this side of it, timed in a graph, was
// slower here (at 3 % four were, by up to 5 %). Timed as calls, 145 sizes on this side are 1.11 times as fast in the
// mean, at worst 0.98: 8 x 14 heads over 2 x 512, D 64, causal 19.7 and 15.7 us, 2 x 32 over 8 x 1024 27.7 and 21.8, 20
// heads x 1024 20.7 and 18.4, x 4096 144 and 131; the other way 1 x 14 over 2 x 2048 causal 19.7 and 30.8.
bool pair_rounds_better(const AttnParams& p) {
    struct Fit { float call, item, block, diagonal; };
    static constexpr Fit kOther[2] = {{2.59f, 2.36f, 1.66f, 0.07f}, {3.62f, 2.55f, 0.95f, 0.42f}};
    static constexpr Fit kPair[2] = {{2.78f, 2.54f, 1.56f, 0.36f}, {3.55f, 2.43f, 2.20f, 0.67f}};
    const int wide = p.d == 128 ? 1 : 0, tiles = (p.sq + kBM - 1) / kBM, group = p.heads / p.kv_heads;
    const int64_t sms = sm_count(), planes = static_cast<int64_t>(p.batch) * p.kv_heads, heads = planes * group, all = heads * tiles;
    if (all <= sms) return false;                             // one round either way
    if (tiles > kMostLevels || all > 8 * sms) return false;   // many rounds: the two are even
    const Fit &o = kOther[wide], &m = kPair[wide];
    const int shift = p.causal == KTT_B200_CAUSAL_BOTTOM_RIGHT ? p.sk - p.sq : 0;
    auto blocks_of = [&](int back) {   // of the tile `back` tiles from the last
        int kend = p.sk;
        if (p.causal) {
            const int last = (tiles - back) * kBM;
            kend = (last < p.sq ? last : p.sq) + shift;
            kend = kend < 0 ? 0 : kend < p.sk ? kend : p.sk;
        }
        return (kend + kBN - 1) / kBN;
    };
    float cost[2 * kMostLevels];
    int64_t count[2 * kMostLevels];
    const bool halves = !wide && all <= 6 * sms, dual = p.sk > kBN && all <= sms;
    auto add = [&](const Fit& f, int& n, int blocks, int64_t items) {
        const float c = f.item + (p.causal ? f.diagonal : 0.f) + f.block * static_cast<float>(blocks);
        if (n > 0 && cost[n - 1] == c) {
            count[n - 1] += items;
            return;
        }
        cost[n] = c;
        count[n++] = items;
    };
    int n = 0;
    for (int t = 0; t < tiles; ++t) add(o, n, halves ? (blocks_of(t) + 1) / 2 : blocks_of(t), heads);
    const float other = o.call + makespan(cost, count, n, wide || halves ? sms : 2 * sms);
    n = 0;
    if (dual) {
        for (int t = 0; t < tiles; ++t) add(m, n, (blocks_of(t) + 1) / 2, heads);
    } else {
        // An item is two neighbours in a plane's list of (tile, head), last rows first.
        for (int t = 0; t < tiles; ++t) {
            const int items = ((t + 1) * group + 1) / 2 - (t * group + 1) / 2;   // those whose first tile is one of these
            if (items > 0) add(m, n, blocks_of(t), planes * items);
        }
        if (last_round_in_halves(p)) {   // (all of them are alike)
            const int64_t over = count[0] % sms;
            count[0] -= over;
            add(m, n, (blocks_of(0) + 1) / 2, 2 * over);
        }
    }
    const float pair = m.call + makespan(cost, count, n, sms);
    return pair < 0.92f * other;
}
}  // namespace

// Head dims 64 and 128 without a mask or with one row of it per (batch, head) have kernels of their
// own, with one tile per work item and two items at a time on an SM. This one is faster where its
// pairs fill whole rounds and the keys are few: what it leaves out of a block (columns past the last
// key, the item arithmetic of all roles but one) weighs most there. Measured on B200, other kernel
// -> this one: D 64, 520 tiles, 64 keys 17.1 -> 13.0 us, 300 keys 25.1 -> 19.6, 1024 keys 38.4 ->
// 34.5; D 128, 220 tiles, 256 keys 13.5 -> 11.9, 64 keys 11.1 -> 9.3. The lines:
//  - as many rounds as the others need, up to three (from the fourth on it is even or slower), and
//    no last round in which a single tile per SM would run alone and faster (of three rounds that
//    one weighs less);
//  - D 64: 1024 keys, with mask terms 320 (at 1024 keys 26.9 -> 27.9);
//  - D 128: 320 keys in the first round or with mask terms, else 96 (at 200 keys 20.9 -> 21.9).
// Without a mask also where its rounds are the better filled ones (pair_rounds_better). Not while a trace or a dump is
// asked for, which the other kernels write.
bool forward_pair_preferred(const AttnParams& p) {
    if (get_trace_buffer() || (p.d == 64 && get_dump_request().buffer)) return false;
    if (p.cu_q || p.key_lengths || mask_needs_plan(p) || p.d != p.dv || (p.d != 64 && p.d != 128)) return false;
    if (p.mask_dtype == KTT_B200_MASK_NONE && pair_rounds_better(p) && forward_pair_takes(p)) return true;
    if (p.causal) return false;
    const int64_t sms = sm_count(), group = p.heads / p.kv_heads, planes = static_cast<int64_t>(p.batch) * p.kv_heads;
    const int64_t per_plane = (p.sq + kBM - 1) / kBM * group, tiles = per_plane * planes, pairs = (per_plane + 1) / 2 * planes;
    const int64_t rounds = (tiles + 2 * sms - 1) / (2 * sms), last = tiles - (rounds - 1) * 2 * sms;
    if (rounds > 3 || pairs > rounds * sms || (rounds < 3 && last <= sms)) return false;
    const bool masked = p.mask_dtype != KTT_B200_MASK_NONE;
    const int most = p.d == 64 ? (masked ? 320 : 1024) : (rounds == 1 || masked ? 320 : 96);
    return p.sk <= most && forward_pair_takes(p);
}

// Head dims and masks that only this kernel and the warp-MMA one take: this one unless the estimate below
// has the other 10 % faster. This one has one CTA of two 128-row tiles per SM, and in front of a mask with
// a row per query its plan; warp-MMA has four 64-row CTAs per SM. With few rows per (batch, head), or a
// plan that few heads share, that is the better. Measured on B200, this kernel and warp-MMA, us:
//   16 x 49 rows and keys, D 32            5.7    4.2     8,192 x 64, D 32                   173    86
//   512 x 64, a bf16 mask each, D 32      61.3    9.4     8,192 x 64, a bf16 mask each, D 32 920   147
//   2,048 x 64, D 80                      54     75       512 x 128, D 80                     19    54
//   512 x 197, one bool mask, D 64        46    124       48 x 520, a bf16 mask each, D 64    85    74
// The constants are fitted to 13,600 such pairs of times (2 to 3,000 rows, 8 to 2,500 keys, 1 to 65,000
// (batch, head) pairs, every kind of mask, D 8 to 128): within 10 to 25 % rms of each side. On 1,213 fresh
// sizes the choice is within 0.5 % of the better side on average, 36 % faster than always this kernel; at
// worst 1.55 times the better side's time.
bool forward_pair_pays(const AttnParams& p) {
    // us. Warp-MMA, a 64-key block of a CTA, by padded head dim (32, 64, 128): when it runs alone on
    // its SM, and its share of a full one (of the CTA, of 64 rows). This kernel, by padded head dim (64,
    // 128): a call, an item, a 128-key block of it; a plan's CTA, four blocks of it.
    // Masks: none, one row, bool, values.
    struct Warp { float alone, cta, rows; };
    static constexpr Warp kWarp[3][4] = {{{1.8f, 0.7f, 0.f}, {4.3f, 1.4f, 0.f}, {5.1f, 1.3f, 0.3f}, {5.8f, 1.2f, 1.f}},
                                         {{3.2f, 1.2f, 0.f}, {5.7f, 1.8f, 0.f}, {6.2f, 1.6f, 0.5f}, {7.1f, 1.7f, 0.9f}},
                                         {{4.5f, 2.7f, 0.5f}, {7.1f, 3.8f, 0.6f}, {7.6f, 3.6f, 1.3f}, {8.3f, 3.8f, 2.1f}}};
    struct Pair { float call, item, block, plan, plan_blocks; };
    static constexpr Pair kPair[2][4] = {{{3.1f, 1.7f, 1.6f, 0.f, 0.f}, {2.6f, 1.5f, 2.5f, 0.f, 0.f}, {4.1f, 3.8f, 1.4f, 1.2f, 3.7f}, {3.6f, 0.f, 5.5f, 0.f, 6.2f}},
                                         {{3.5f, 1.5f, 2.5f, 0.f, 0.f}, {3.f, 1.6f, 3.1f, 0.f, 0.f}, {4.3f, 4.f, 2.1f, 1.4f, 3.7f}, {3.8f, 0.f, 6.6f, 0.f, 6.2f}}};
    const bool planned = mask_needs_plan(p);
    const int kind = p.mask_dtype == KTT_B200_MASK_NONE ? 0 : !planned ? 1 : p.mask_dtype == KTT_B200_MASK_BOOL ? 2 : 3;
    const int dim = p.d > p.dv ? p.d : p.dv;
    // (Packed: sequences of the average length.)
    const int64_t sq = p.cu_q ? p.total_q / p.batch + 1 : p.sq, sk = p.cu_q ? p.total_k / p.batch + 1 : p.sk;
    const int64_t group = p.heads / p.kv_heads, kv_pairs = static_cast<int64_t>(p.batch) * p.kv_heads;
    const float sms = static_cast<float>(sm_count());

    const int64_t warp_tiles = (sq + 63) / 64;
    const Warp& w = kWarp[dim <= 32 ? 0 : dim <= 64 ? 1 : 2][kind];
    const bool beyond_l2 = 2 * kv_pairs * (group * sq + sk) * (p.d + p.dv) > (96ll << 20);   // then its loads are what it waits for
    const float share = (w.cta + w.rows * static_cast<float>(sq) / static_cast<float>(64 * warp_tiles)) * (beyond_l2 ? 1.4f : 1.f);
    const float per_sm = ceilf(static_cast<float>(warp_tiles * group * kv_pairs) / sms), full = ceilf(per_sm / 4.f) - 1.f;
    const float warp_us = 2.f + static_cast<float>((sk + 63) / 64) * (full * fmaxf(w.alone, 4.f * share) + fmaxf(w.alone, (per_sm - 4.f * full) * share));

    auto rounds = [&](int64_t n) {   // of one per SM; uneven ones overlap
        const float x = static_cast<float>(n) / sms;
        return x <= 3.f ? ceilf(x) : x + 0.5f;
    };
    const Pair& c = kPair[dim <= 64 ? 0 : 1][kind];
    const int64_t tiles = (sq + kBM - 1) / kBM * group, blocks = (sk + kBN - 1) / kBN;
    const bool dual = sk > kBN && tiles * kv_pairs <= sm_count();
    float pair_us = c.call + rounds((dual ? tiles : (tiles + 1) / 2) * kv_pairs) * (c.item + c.block * static_cast<float>(dual ? (blocks + 1) / 2 : blocks));
    if (planned) {
        const int64_t planes = static_cast<int64_t>(p.ms[0] ? p.batch : 1) * (p.ms[1] ? p.heads : 1);
        pair_us += rounds(planes * ((sq + 31) / 32)) * (c.plan + c.plan_blocks * static_cast<float>((blocks + 3) / 4));
    }
    return warp_us > 0.9f * pair_us;
}

int64_t forward_pair_workspace(const AttnParams& p) {
    return kHeaderBytes + (mask_needs_plan(p) ? plan_bytes(p, plan_part(p, kMostPlan)) : 0);
}

namespace {

int launch_whole(const AttnParams& p, void* workspace, int64_t workspace_bytes, cudaStream_t stream) {
    const char* why = "";
    const int64_t tq = p.cu_q ? p.total_q : p.sq, tk = p.cu_q ? p.total_k : p.sk;
    const int64_t bq = p.cu_q ? 1 : p.batch;
    const void* base[3] = {p.q, p.k, p.v};
    const int64_t rows[3] = {tq, tk, tk}, heads[3] = {p.heads, p.kv_heads, p.kv_heads};
    const int64_t* strides[3] = {p.qs, p.ks, p.vs};
    const int width[3] = {p.d, p.d, p.dv};
    PairParams tp;
    CUtensorMap maps[3];
    for (int o = 0; o < 3; ++o) {
        int64_t s[3];
        if (!operand_layout(base[o], rows[o], heads[o], bq, strides[o], s, &why)) return fail(KTT_B200_ERR_UNSUPPORTED, "tcgen05 forward: %s", why);
        const DimOrder order = order_of(s);
        if (!encode_map(&maps[o], base[o], width[o], rows[o], heads[o], bq, s, order, kBM, &why)) return fail(KTT_B200_ERR_UNSUPPORTED, "tcgen05 forward: %s", why);
        for (int i = 0; i < 3; ++i) tp.dim_of[o][i] = order.slot_of[i];
    }
    tp.a = p;
    int* host_status = status_word(&tp.status);
    if (!host_status || !tp.status) return fail(KTT_B200_ERR_LAUNCH, "tcgen05 forward: no status word");
    if (*host_status != 0) {
        const int code = *host_status;
        *host_status = 0;
        note_call(5);
        return fail(KTT_B200_ERR_DEVICE_WAIT, "an earlier tcgen05 launch gave up waiting (code %d)", code);
    }

    const int group = p.heads / p.kv_heads;
    const int q_tiles = (p.sq + kBM - 1) / kBM;
    const int64_t units = static_cast<int64_t>(q_tiles) * group * p.kv_heads * p.batch;   // (query tile, head)
    if (units > kMostTiles) return fail(KTT_B200_ERR_UNSUPPORTED, "tcgen05 forward: too many query tiles");
    const int sms = sm_count();
    // Dual halves a tile's chain of blocks but adds a merge and doubles the items: it pays where
    // tiles would leave SMs without one. (Up to six tiles per SM it cost more than it gave, when it was
    // tried: 16 x 16 heads x 257, D 80: 43 -> 37 us without it, 4 x 16 heads 19 -> 13; 2 x 16 heads x
    // 2048, D 64, causal mask: 71 -> 58. At 8 heads x 2 x 1024, D 80, 128 tiles, it gives 25 -> 16.)
    const bool dual = p.sk > kBN && units <= sms;
    const int levels = dual ? q_tiles * group : (q_tiles * group + 1) / 2;
    tp.work = levels * p.kv_heads * p.batch;
    tp.duals = dual ? 0 : tp.work;
    tp.cut = 0;
    const int over = last_round_in_halves(p) ? tp.work % sms : 0;
    if (over) {
        tp.cut = tp.duals = tp.work - over;
        tp.work += over;
    }
    tp.by_batch = divisor_of(p.batch);
    tp.by_kv_heads = divisor_of(p.kv_heads);
    tp.by_group = divisor_of(group);
    tp.by_levels = divisor_of(levels);

    const bool planned = mask_needs_plan(p);
    const bool usable = workspace && (reinterpret_cast<uintptr_t>(workspace) & 15) == 0;
    if (planned) {
        plan_layout(p, static_cast<unsigned char*>(workspace) + kHeaderBytes, &tp.plan);
        const MaskPlan& m = tp.plan;
        const int64_t planes = static_cast<int64_t>(m.heads) * (m.batched ? p.batch : 1);
        const int size = p.mask_dtype == KTT_B200_MASK_BOOL ? 1 : p.mask_dtype == KTT_B200_MASK_F32 ? 4 : 2;
        const bool vec = p.ms[3] == 1 && (reinterpret_cast<uintptr_t>(p.mask) % (4 * size)) == 0 && p.ms[0] % 4 == 0 && p.ms[1] % 4 == 0 && p.ms[2] % 4 == 0;
        auto plan = p.mask_dtype == KTT_B200_MASK_BOOL ? mask_plan_kernel<KTT_B200_MASK_BOOL> : p.mask_dtype == KTT_B200_MASK_BF16 ? mask_plan_kernel<KTT_B200_MASK_BF16>
                  : p.mask_dtype == KTT_B200_MASK_F16  ? mask_plan_kernel<KTT_B200_MASK_F16>  : mask_plan_kernel<KTT_B200_MASK_F32>;
        if (int rc = launch_dependent(plan, dim3(static_cast<unsigned>(planes), m.groups), kPlanThreads, 0, stream, "mask_plan launch", p, tp.plan,
                                      static_cast<int32_t*>(workspace), vec)) return rc;
    }
    // K / V beyond what L2 keeps (126 MB on B200): the grouped order, which needs the counter.
    const int64_t kv_bytes = (p.cu_q ? p.total_k : static_cast<int64_t>(p.batch) * p.sk) * p.kv_heads * (p.d + p.dv) * 2;
    const bool large = kv_bytes > (96ll << 20);
    // The counter pays when a CTA gets several items; with one or two the fixed deal (longest
    // first, snake order) is as even and saves the trip to the counter before each item's first
    // load. A workspace of 4 to 255 bytes is one int32 the caller zeroes before every call; not at head
    // dim 64, where a caller cannot know which kernel takes the call, and the other one has no
    // use for less than the whole header, 16-byte aligned.
    const bool narrow = p.d == 64 && p.dv == 64;
    const bool words = workspace && (reinterpret_cast<uintptr_t>(workspace) & 3) == 0;
    const bool header = (narrow ? usable : words) && workspace_bytes >= kHeaderBytes;
    const bool drawn = header ? tp.work > 2 * static_cast<int64_t>(sms) : !narrow && words && workspace_bytes >= 4;
    tp.work_counter = drawn ? static_cast<int*>(workspace) : nullptr;
    tp.done_counter = drawn && header ? static_cast<int*>(workspace) + 1 : nullptr;
    tp.grouped = drawn && large ? 1 : 0;
    const int grid = tp.work < sms ? tp.work : sms;
    if (p.d <= 64 && p.dv <= 64) return launch_pair<64>(p, maps, tp, grid, stream);
    return launch_pair<128>(p, maps, tp, grid, stream);
}

}  // namespace

int launch_forward_pair(const AttnParams& p, void* workspace, int64_t workspace_bytes, cudaStream_t stream) {
    if (!mask_needs_plan(p)) return launch_whole(p, workspace, workspace_bytes, stream);
    const int64_t room = workspace_bytes - kHeaderBytes;
    if (!workspace || (reinterpret_cast<uintptr_t>(workspace) & 15) || room < plan_bytes(p, least_part(p))) {
        return fail(KTT_B200_ERR_BAD_ARGUMENT, "tcgen05 forward: a mask with a row per query needs %lld bytes of workspace, 16-byte aligned",
                    static_cast<long long>(forward_pair_workspace(p)));
    }
    // One part in nearly every call. The next one's plan waits for this one's attention, as it does for
    // whatever is before it in the stream. (Causal calls take no mask: rows do not depend on the others.)
    const PlanPart part = plan_part(p, room);
    const int group = p.heads / p.kv_heads;
    const int64_t size = p.mask_dtype == KTT_B200_MASK_BOOL ? 1 : p.mask_dtype == KTT_B200_MASK_F32 ? 4 : 2;
    for (int b = 0; b < p.batch; b += part.batch) {
        for (int h = 0, heads; h < p.heads; h += heads) {
            heads = part.heads < p.heads - h ? part.heads : p.heads - h;
            if (part.heads < group && heads > group - h % group) heads = group - h % group;
            const int64_t hk = h / group;
            for (int r = 0; r < p.sq; r += part.rows) {
                AttnParams s = p;
                s.batch = part.batch < p.batch - b ? part.batch : p.batch - b;
                s.heads = heads;
                s.kv_heads = heads < group ? 1 : heads / group;
                s.sq = part.rows < p.sq - r ? part.rows : p.sq - r;
                auto at = [&](const int64_t (&st)[3], int64_t head, int64_t row) { return b * st[0] + head * st[1] + row * st[2]; };
                s.q += at(p.qs, h, r);
                s.k += at(p.ks, hk, 0);
                s.v += at(p.vs, hk, 0);
                s.out += at(p.os, h, r);
                if (s.lse) s.lse += at(p.ls, h, r);
                s.mask = static_cast<const unsigned char*>(p.mask) + (b * p.ms[0] + h * p.ms[1] + r * p.ms[2]) * size;
                if (int rc = launch_whole(s, workspace, workspace_bytes, stream)) return rc;
            }
        }
    }
    return 0;
}

}  // namespace ktt
