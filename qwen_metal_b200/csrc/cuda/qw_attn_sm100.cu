// Block-causal (prefix-visible) flash-attention forward for sm_100a.
//
// One CTA owns 256 query rows of one (batch, head): two 128-row sub-tiles that
// ping-pong on the tensor pipe.  Q/K/V tiles arrive through TMA (128B swizzle)
// into shared memory; S = Q K^T and O += P V run as tcgen05.mma with fp32
// accumulators in tensor memory (TMEM); the softmax is fp32 in the exp2 domain,
// one thread per query row, and writes P back to TMEM as bf16 over the S
// columns so P V reads its A operand straight from TMEM.
//
// Warp roles (384 threads = 3 warpgroups; registers are moved from the third
// warpgroup to the two softmax warpgroups with setmaxnreg):
//   warps 0-3   softmax + epilogue of sub-tile 0 (TMEM lanes 0..127)
//   warps 4-7   softmax + epilogue of sub-tile 1
//   warp  8     MMA issue (all lanes run the loop, one is elected per issue), TMEM allocation
//   warp  9     TMA producer (one elected lane)
//   warps 10-11 idle (they only complete the third warpgroup)
//
// Mask: every row has an integer key limit (prefix) and the batch item may have
// a key-padding window.  Key tiles past the largest limit of a sub-tile are
// never issued, key tiles that lie completely inside the padding window are
// skipped by all roles, interior tiles run without a compare, boundary tiles have their
// scores masked (see mask_scores).
//
// Epilogue: O / l is rounded to bf16 and goes through the (by then dead) Q tile in shared
// memory to global memory, every warp its own 32 rows (write_rows).  When the heads
// are sharded over several GPUs the rows go to this rank's head columns of a
// full-width output (the kernel can address several such destinations, peer-
// mapped ones included); the multi-GPU group writes the rank's own buffer here
// and carries the columns to the peers with a push kernel under the next layer,
// because with a single wave of CTAs all peer stores would leave at the kernel's
// end as one exposed burst.  At its start the kernel then opens the output slot's
// next epoch for the peers' pushes.
//
// Softmax.  Callers that promise bounded row norms (the DiT layer's QK-norm) get
// P = exp2(score*c - bound) against one fixed exponent: no row maximum, no
// rescaling, scores streamed out of TMEM in 32-column chunks.  Other callers get the
// running maximum with lazy rescaling.
//
// Wave tail.  The grid is one CTA per (batch, head, 256-row block), heaviest
// blocks first, and rarely a multiple of the SM count.  The units that would
// form the last, partly filled wave are therefore run in split form, two CTAs per
// unit: a CTA takes 128 of the rows and gives each of its two sub-tiles half of
// the key tiles; at the end warpgroup 0 merges the two accumulators (both sit in
// the same TMEM lanes) with the usual exp2 reweighting.  Twice the CTAs of half
// the length fill the idle SMs, and nothing leaves the CTA unmerged.
//
// Every wait is bounded: when one runs out the CTA records where in the status
// words, raises a shared abort flag that the other waits poll, drains its TMA
// loads, frees its TMEM and returns.  (The MMA warp's waits do not poll it: they count
// probes, and end within the same budget.)
//
// Semantics follow the reference prefix kernel (h3_shaders.metal:3061-3272):
// scale applied to fp32 scores, P rounded to bf16 before P V, fp32 accumulate,
// output acc / l rounded to bf16; rows without a visible key store zeros.

#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <type_traits>

#include "qw_sm100.cuh"

namespace {

using namespace sm100;

constexpr int kHeadDim = 128;
constexpr int kTileM = 128;  // query rows per sub-tile (= TMEM lanes)
constexpr int kTileN = 128;  // keys per tile
constexpr int kStages = 4;   // K/V ring slots
constexpr int kTileBytes = kTileN * kHeadDim * 2;  // 32 KiB
constexpr int kHalfTileBytes = kTileBytes / 2;     // one 64-column TMA box
constexpr int kThreads = 384;
// setmaxnreg only redistributes the registers the CTA got at launch
// (kThreads * 168 = 64512): 2 * 128 * 224 + 128 * 56 = 64512.  Asking for more
// would block the second softmax warpgroup forever.
constexpr int kLaunchRegs = 168;
constexpr int kSoftmaxRegs = 224;
constexpr int kOtherRegs = 56;
static_assert(2 * 128 * kSoftmaxRegs + 128 * kOtherRegs <= kThreads * kLaunchRegs,
              "setmaxnreg budget exceeds the launch allocation");
// P of a tile is published in two parts, the first kPart * 16 keys and the rest: P V of
// the first part runs under the softmax of the rest, which takes it out of the chain
// S -> softmax -> P V -> next S that bounds the kernel (eight layers of six heads, 4352 keys, with
// a bound: 528 us with 4, 513 us with 6; 8188 x 8211 keys without one: 966 and 945 us).
constexpr int kPart = 6;
constexpr int kSoftmaxThreads = 256;
constexpr int kMmaWarp = 8;
constexpr int kTmaWarp = 9;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kTmemS0 = 0, kTmemS1 = 128, kTmemO0 = 256, kTmemO1 = 384;
// Lazy rescale threshold in the exp2 domain: P may grow to 2^8 before O and l
// are brought back to the running maximum.
constexpr float kRescaleThreshold = 8.0f;

enum Barrier : int {
    kBarQFull = 0,                        // 2: Q sub-tile i landed
    kBarKvFull = 2,                       // kStages
    kBarKvEmpty = kBarKvFull + kStages,   // kStages
    kBarSFull = kBarKvEmpty + kStages,    // 2: S_i complete in TMEM
    kBarPFirst = kBarSFull + 2,           // 2: first part of P_i written (one arrival per warp)
    kBarPFull = kBarPFirst + 2,           // 2: the rest of P_i written
    kBarOFinal = kBarPFull + 2,           // 2: last P V of sub-tile i complete
    kBarMerge = kBarOFinal + 2,           // split form: sub-tile 1 published its exponent and row sum
    kBarCount = kBarMerge + 1
};

struct __align__(16) SharedControl {
    Mbar bars[kBarCount];
    uint32_t tmem_base;
    volatile uint32_t abort_flag;
    long long wait_cycles;  // budget of every bounded wait of this CTA but the MMA warp's
    int n_tiles[2];      // key tiles each sub-tile needs (by its largest limit)
    int warp_max[8];     // per softmax warp: largest limit
    int skip_lo, skip_hi;  // key tiles [skip_lo, skip_hi) lie inside the padding window
    // Visited key tiles (the padding window taken out) are numbered 0, 1, ...;
    // sub-tile i walks tile_count[i] of them from tile_first[i].  Whole form: both
    // from 0.  Split form: the two halves of one list.
    int tile_first[2], tile_count[2];
    float merge_m[kTileM];  // split form: sub-tile 1's reference exponent and row sum
    float merge_l[kTileM];
};

constexpr size_t kSmemData = (size_t)(2 + kStages) * kTileBytes;
constexpr size_t kSmemBytes = kSmemData + sizeof(SharedControl) + 1024;  // +1024: manual alignment

struct KernelParams {
    const int32_t *kv_limit;
    uint32_t *status;
#ifdef QW_ATTN_TRACE
    unsigned long long *trace;  // event log of block (0,0,0), dumped to $QW_CUDA_ATTN_TRACE
#endif
    int per_batch_limits;
    int causal;
    uint32_t causal_offset;
    uint32_t batch, q_rows, kv_rows, heads, kv_heads;
    uint32_t text_len[8];
    uint32_t text_pad;
    float scale_log2;  // scale * log2(e)
    // Optional promise by the caller (two floats in device memory): every query row
    // has a 2-norm of at most score_bound[0] and every key row of at most
    // score_bound[1], so |q.k| <= their product and the softmax can use one fixed
    // reference exponent instead of a running row maximum.
    const float *score_bound;
    int head_major_out;
    // Sharded runs: the rows are stored at this rank's head columns of n_out
    // full-width outputs (peer-mapped pointers allowed).  out_heads_total is the
    // head count of the destination rows and out_head_offset this rank's first head.
    __nv_bfloat16 *out_peers[8];
    uint32_t n_out, out_heads_total, out_head_offset;
    // Launch geometry: CTA c < total_units - tail_units runs unit c whole; the
    // last tail_units units run in split form, two CTAs each.
    uint32_t n_qblocks, total_units, tail_units;
    // Gather by a separate push: epoch counter of the output slot and the peers'
    // flag words that receive the new epoch when this kernel starts.
    uint32_t *slot_use;
    uint32_t *freed_peer[8];
    uint32_t n_freed;
    // Bounded-wait exercise (tests only): budget in SM cycles (0 = the default) and
    // the first visited key tile the producer does NOT load (< 0: loads everything),
    // so that the waits downstream of it run out and the CTA takes its clean exit.
    long long wait_cycles;
    int withhold_from;
    int mma_probes;  // the same budget for the MMA warp's waits, in probes
};

// Shared address of a barrier.  (The roles keep the first one's and add: a conversion from a pointer
// at every wait and commit cost 1 % with six heads and 4352 keys, 2 % with 24 heads of two.)
__device__ __forceinline__ uint32_t bar_at(uint32_t bars, uint32_t which) {
    return bars + which * (uint32_t)sizeof(Mbar);
}

// A wait ran out: the first one of the launch leaves its place in the status words, and the other
// waits of the CTA end.
__device__ __noinline__ void record_expiry(SharedControl *ctl, uint32_t *status, uint32_t where,
                                           uint32_t tile) {
    ctl->abort_flag = 1;
    if (atomicCAS(status, 0u, (uint32_t)QWCU_STATUS_WAIT_TIMEOUT) == 0u) {
        status[1] = where;
        status[2] = tile;
        status[3] = blockIdx.x;
    }
    __threadfence();
}

// Bounded wait.  Returns false when the budget ran out here (recorded) or another thread
// of the CTA already gave up.  (The GEMM's, out of line after a few probes, is not used
// here: the softmax waits with its registers full.)
__device__ __forceinline__ bool mbar_wait_slow(SharedControl *ctl, uint32_t bar,
                                            uint32_t parity, uint32_t *status, uint32_t where,
                                            uint32_t tile) {
    long long start = clock64();
    for (;;) {
        for (int i = 0; i < 32; ++i)
            if (mbar_try(bar, parity)) return true;
        if (ctl->abort_flag) return false;
        if (clock64() - start > ctl->wait_cycles) {
            record_expiry(ctl, status, where, tile);
            return false;
        }
    }
}

__device__ __forceinline__ bool mbar_wait(SharedControl *ctl, uint32_t bar,
                                          uint32_t parity, uint32_t *status, uint32_t where,
                                          uint32_t tile) {
    if (mbar_try(bar, parity)) return true;
    return mbar_wait_slow(ctl, bar, parity, status, where, tile);
}

// The wait of the MMA warp, for all its lanes at once, bounded by a number of probes that the host
// makes of the budget.  The warp issues every MMA of the CTA and each of its clocks is on the chain
// of both sub-tiles, so the loop holds nothing else: with the clock and the abort flag of the wait
// above behind 32 probes, in line or called, layers of six heads, 4352 keys, took 11 to 15 % longer,
// of 24 heads of two 6 to 10 %.  A probe that fails suspends the warp for a time that the hardware sets: 400 000 of them took 1.58 s, 7800 clocks each.
constexpr long long kProbeCycles = 10000;
__device__ __forceinline__ bool mbar_wait_warp(const KernelParams &p, uint32_t bar, uint32_t parity) {
    bool ok = false;
#pragma unroll 1
    for (int i = 0; i < p.mma_probes && !ok; ++i) ok = mbar_try(bar, parity);
    return __all_sync(0xffffffffu, ok) != 0;
}

// What the MMA warp does when one ran out, before it leaves.  It waits for what stayed away itself,
// the softmax only for the scores behind it, so its record is the one that names the ring slot.  Out
// of line, so that the loop around the waits does not grow.
__device__ __noinline__ void mma_gave_up(SharedControl *ctl, uint32_t *status, uint32_t bar,
                                         uint32_t tile) {
    record_expiry(ctl, status, (2u << 16) | bar, tile);
}

// A value the compiler knows to be the same in all lanes of the (converged) warp.
template <typename T>
__device__ __forceinline__ T uniform(T v) {
    return __shfl_sync(0xffffffffu, v, 0);
}
// Instruction descriptors, M = 128, N = 128.
constexpr uint32_t kIdescQK = instr_desc(kTileM, kTileN, false);
constexpr uint32_t kIdescPV = instr_desc(kTileM, kTileN, true);

#define QW_TMEM_LD32(taddr, r)                                                                  \
    asm volatile(                                                                               \
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "                                               \
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "              \
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, "    \
        "[%32];"                                                                                \
        : "=r"((r)[0]), "=r"((r)[1]), "=r"((r)[2]), "=r"((r)[3]), "=r"((r)[4]), "=r"((r)[5]),   \
          "=r"((r)[6]), "=r"((r)[7]), "=r"((r)[8]), "=r"((r)[9]), "=r"((r)[10]), "=r"((r)[11]), \
          "=r"((r)[12]), "=r"((r)[13]), "=r"((r)[14]), "=r"((r)[15]), "=r"((r)[16]),            \
          "=r"((r)[17]), "=r"((r)[18]), "=r"((r)[19]), "=r"((r)[20]), "=r"((r)[21]),            \
          "=r"((r)[22]), "=r"((r)[23]), "=r"((r)[24]), "=r"((r)[25]), "=r"((r)[26]),            \
          "=r"((r)[27]), "=r"((r)[28]), "=r"((r)[29]), "=r"((r)[30]), "=r"((r)[31])             \
        : "r"(taddr))

#define QW_TMEM_ST32(taddr, r)                                                                  \
    asm volatile(                                                                               \
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "                                         \
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "             \
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"     \
        ::"r"(taddr), "r"((r)[0]), "r"((r)[1]), "r"((r)[2]), "r"((r)[3]), "r"((r)[4]),          \
          "r"((r)[5]), "r"((r)[6]), "r"((r)[7]), "r"((r)[8]), "r"((r)[9]), "r"((r)[10]),        \
          "r"((r)[11]), "r"((r)[12]), "r"((r)[13]), "r"((r)[14]), "r"((r)[15]), "r"((r)[16]),   \
          "r"((r)[17]), "r"((r)[18]), "r"((r)[19]), "r"((r)[20]), "r"((r)[21]), "r"((r)[22]),   \
          "r"((r)[23]), "r"((r)[24]), "r"((r)[25]), "r"((r)[26]), "r"((r)[27]), "r"((r)[28]),   \
          "r"((r)[29]), "r"((r)[30]), "r"((r)[31])                                              \
        : "memory")

#define QW_TMEM_ST16(taddr, r)                                                                  \
    asm volatile(                                                                               \
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "                                         \
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"             \
        ::"r"(taddr), "r"((r)[0]), "r"((r)[1]), "r"((r)[2]), "r"((r)[3]), "r"((r)[4]),          \
          "r"((r)[5]), "r"((r)[6]), "r"((r)[7]), "r"((r)[8]), "r"((r)[9]), "r"((r)[10]),        \
          "r"((r)[11]), "r"((r)[12]), "r"((r)[13]), "r"((r)[14]), "r"((r)[15])                  \
        : "memory")

// tcgen05.wait::ld that names the 32 registers of an earlier load as read-write
// operands: no use of them can be scheduled ahead of the wait.
#define QW_TMEM_WAIT_LD32(r)                                                                    \
    asm volatile(                                                                               \
        "tcgen05.wait::ld.sync.aligned;"                                                        \
        : "+r"((r)[0]), "+r"((r)[1]), "+r"((r)[2]), "+r"((r)[3]), "+r"((r)[4]), "+r"((r)[5]),   \
          "+r"((r)[6]), "+r"((r)[7]), "+r"((r)[8]), "+r"((r)[9]), "+r"((r)[10]), "+r"((r)[11]), \
          "+r"((r)[12]), "+r"((r)[13]), "+r"((r)[14]), "+r"((r)[15]), "+r"((r)[16]),            \
          "+r"((r)[17]), "+r"((r)[18]), "+r"((r)[19]), "+r"((r)[20]), "+r"((r)[21]),            \
          "+r"((r)[22]), "+r"((r)[23]), "+r"((r)[24]), "+r"((r)[25]), "+r"((r)[26]),            \
          "+r"((r)[27]), "+r"((r)[28]), "+r"((r)[29]), "+r"((r)[30]), "+r"((r)[31])             \
        :                                                                                       \
        : "memory")

__device__ __forceinline__ void tmem_wait_ld() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Packed fp32 pairs (one issue slot for two lanes of work on sm_100).
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
        "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ float2 fadd2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "add.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Pipeline event log, compiled in only with -DQW_ATTN_TRACE (a debugging build).
#ifdef QW_ATTN_TRACE
// Event log for pipeline analysis: (role, event, tile) and the SM clock, written
// by one thread per role of block (0, 0, 0) when a trace buffer is attached.
constexpr int kTraceSlots = 4096;
__device__ __forceinline__ void trace_event(const KernelParams &p, int role, int event, int tile,
                                            uint32_t &cursor) {
    // One private region per role and a register cursor: a plain store, no
    // round trip, so the log barely perturbs what it measures.  (The MMA warp runs its
    // loop with all lanes: one writes.)
    if (p.trace && (threadIdx.x & 31) == 0 && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && cursor < 1000) {
        p.trace[1 + role * 1024 + cursor] =
            ((unsigned long long)(role << 20 | event << 12 | (tile & 0xfff)) << 40) |
            ((unsigned long long)clock64() & 0xffffffffffull);
        ++cursor;
    }
}
#define QW_TRACE(role, event, tile) trace_event(p, role, event, tile, trace_cursor)
#else
#define QW_TRACE(role, event, tile) ((void)0)
#endif

__device__ __forceinline__ int row_limit(const KernelParams &p, uint32_t b, uint32_t r) {
    if (r >= p.q_rows) return 0;
    if (p.text_pad && r >= p.text_len[b] && r < p.text_pad) return 0;  // padding query row
    int limit;
    if (p.kv_limit) {
        limit = p.kv_limit[p.per_batch_limits ? (size_t)b * p.q_rows + r : r];
        limit = max(limit, 0);
    } else if (p.causal) {
        unsigned long long c = (unsigned long long)r + 1ull + p.causal_offset;
        limit = (int)min(c, (unsigned long long)p.kv_rows);
    } else {
        limit = (int)p.kv_rows;
    }
    return min(limit, (int)p.kv_rows);
}

// Visited tile u -> key tile index, and how many of `tiles` key tiles are visited.
__device__ __forceinline__ int phys_tile(const SharedControl *ctl, int u) {
    return u < ctl->skip_lo ? u : u + (ctl->skip_hi - ctl->skip_lo);
}
__device__ __forceinline__ int visited_tiles(int tiles, int lo, int hi) {
    if (tiles <= lo) return tiles;
    if (tiles >= hi) return tiles - (hi - lo);
    return lo;
}

// ---------------------------------------------------------------------------
// Softmax + epilogue role: 128 threads per sub-tile, one query row each.
// ---------------------------------------------------------------------------
// The first part of P: published before the exponentials of the rest are begun, so that its P V
// runs under them.
__device__ __forceinline__ void publish_p_first(uint32_t bar, int tid_in_group) {
    tmem_wait_st();
    tc_fence_before();
    if ((tid_in_group & 31) == 0) mbar_arrive(bar);
}

// Bits 0 .. n - 1 (none for n <= 0, all for n >= 32).
__device__ __forceinline__ uint32_t low_bits(int n) {
    uint32_t r;
    asm("bmsk.clamp.b32 %0, %1, %2;" : "=r"(r) : "r"(0), "r"(max(n, 0)));
    return r;
}
// 32 scores of keys key0 .. key0 + 31: those the row does not see become -infinity.  The
// row's mask is made once for the 32 keys and a score costs a bit test and a select, where
// comparing its key with the limit and the padding window took three compares and a select.
// (When every 32 keys carried the masks in line, that took a quarter off a launch of six heads
// and 4352 rows, 64 of them text.)
//
// Where text rows, which see few keys, share a block with image rows, their warps mask every tile
// and the launch waits for them.  Tiles without a mask must not pay for it either: 256 text rows
// have a block of their own.  Six heads, 4352 rows, 64 / 256 of them text, a launch's time over
// that of the present form, and the present form's us:
//                                        with a bound      without
//   a branch in every 32 keys              1.16 / 1.07    1.10 / 1.07
//   every masked tile by mask_tile         1.25 / 1.00    1.19 / 1.00
//   as now                            us   65.3 / 59.2    71.4 / 62.1
// With a bound a tile's softmax stands twice in the code, with the masks in line and without.
// Without one the 128 scores are in registers at once: rows that see nothing of a tile take one
// select per score, and only tiles that some row sees a part of go through mask_tile.  A second
// copy there is slower where launches are short, since each reads the code anew (six launches of
// 412 text rows: 4 %), and so are the bits of all masks in registers (1 %, 5 % with 64 text rows).
__device__ __forceinline__ void mask_scores(uint32_t *s, int key0, int limit, int pad_lo, int pad_hi) {
    const uint32_t visible =
        low_bits(limit - key0) & ~(low_bits(pad_hi - key0) & ~low_bits(pad_lo - key0));
#pragma unroll
    for (int i = 0; i < 32; ++i)
        s[i] = (visible & (1u << i)) ? s[i] : 0xff800000u;
}

// The masks of a tile, as a pass of their own over its scores in TMEM: a small loop.
__device__ __forceinline__ void mask_tile(uint32_t tmem_s, int key0, int limit, int pad_lo, int pad_hi) {
#pragma unroll 1
    for (int i = 0; i < kTileN; i += 32) {
        uint32_t s[32];
        QW_TMEM_LD32(tmem_s + i, s);
        QW_TMEM_WAIT_LD32(s);
        mask_scores(s, key0 + i, limit, pad_lo, pad_hi);
        QW_TMEM_ST32(tmem_s + i, s);
    }
    tmem_wait_st();
}

// 32 output rows of a warp, one destination: out = (w_own * O_own + w_other * O_other) * inv,
// rounded to bf16.  A thread has a row in TMEM; 32 columns at a time go through a box of 32 rows
// x 64 bytes in shared memory (16-byte pieces XOR-swizzled by the row, two boxes in turn) and from
// there to global memory with four lanes per row.  (tmem_own, tmem_other: kNoTmem where there is
// none.  Every lane takes part in the warp-collective TMEM loads.)
//
// Plain stores end with the instruction; a TMA store of the tile had to be waited for until it
// had read shared memory, 1100 clocks at the end of every CTA.  And a function of its own: its
// registers in one allocation with the softmax loop's cost that loop more than all of this (in
// line, 8188 x 8211 keys took 7 % longer).  Against the TMA stores layers of 33 to 412 text rows
// gained 6 to 2 %, of six heads, 4352 keys, 3 %.  (A function's registers beyond some 60 are saved
// on the stack at its call: all 128 columns at once cost half a microsecond a launch, 64 at a time
// 1 % of a layer of 1500 text rows.)
constexpr uint32_t kNoTmem = 0xffffffffu;
__device__ __noinline__ void write_rows(uint32_t tmem_own, uint32_t tmem_other, float w_own,
                                        float w_other, float inv, uint32_t box, __nv_bfloat16 *out,
                                        uint32_t row_stride, uint32_t rows) {
    const uint32_t lane = threadIdx.x & 31u, first = lane >> 2, piece = lane & 3u;
    out += (size_t)first * row_stride + piece * 8u;
#pragma unroll 1
    for (uint32_t c = 0; c < (uint32_t)kHeadDim; c += 32, out += 32) {
        const uint32_t at = box + (c & 32u) * 64u;  // (the second box 2 KB behind the first)
        uint32_t o[32];
        if (tmem_own != kNoTmem) {
            QW_TMEM_LD32(tmem_own + c, o);
            QW_TMEM_WAIT_LD32(o);
        } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = 0u;
        }
        if (tmem_other != kNoTmem) {
            uint32_t x[32];
            QW_TMEM_LD32(tmem_other + c, x);
            QW_TMEM_WAIT_LD32(x);
#pragma unroll
            for (int i = 0; i < 32; ++i)
                o[i] = __float_as_uint(
                    fmaf(__uint_as_float(x[i]), w_other, __uint_as_float(o[i]) * w_own));
        } else if (w_own != 1.0f) {
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * w_own);
        }
#pragma unroll
        for (uint32_t c16 = 0; c16 < 4; ++c16) {
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                w[i] = pack_bf16(__uint_as_float(o[8 * c16 + 2 * i]) * inv,
                                 __uint_as_float(o[8 * c16 + 2 * i + 1]) * inv);
            st_shared16(at + lane * 64u + ((c16 ^ ((lane >> 1) & 3u)) << 4), w[0], w[1], w[2], w[3]);
        }
        __syncwarp();  // (the box before is read while this one is written: one barrier is enough)
        __nv_bfloat16 *to = out;
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i, to += 8 * (size_t)row_stride) {
            const uint32_t r = 8u * i + first;
            const uint4 x = ld_shared16(at + r * 64u + ((piece ^ ((r >> 1) & 3u)) << 4));
            if (r < rows) *reinterpret_cast<uint4 *>(to) = x;
        }
    }
}

// kBounded: the caller promised |score * scale * log2(e)| <= bound (see
// KernelParams::score_bound), so P = exp2(score*c - bound) needs no row maximum:
// the scores stream out of TMEM 32 columns at a time, each chunk's exponentials
// run under the next chunk's load, and O is never rescaled.
template <bool kBounded>
__device__ __forceinline__ void softmax_role(const KernelParams &p, SharedControl *ctl,
                                             uint8_t *stage, int sub, int tid_in_group,
                                             int my_limit, uint32_t b, uint32_t h,
                                             uint32_t tile_row0, bool split, float bound) {
    const int warp_in_group = tid_in_group >> 5;
    const uint32_t lane_base = (uint32_t)(warp_in_group * 32) << 16;
    const uint32_t tmem = ctl->tmem_base;
    const uint32_t tmem_s = tmem + lane_base + (sub ? kTmemS1 : kTmemS0);
    const uint32_t tmem_o = tmem + lane_base + (sub ? kTmemO1 : kTmemO0);
    const uint32_t bars = smem_u32(ctl->bars) + (uint32_t)sub * (uint32_t)sizeof(Mbar);
    const uint32_t bar_s = bar_at(bars, kBarSFull), bar_p = bar_at(bars, kBarPFull);
    const uint32_t bar_p_first = bar_at(bars, kBarPFirst);
    const int pad_lo = p.text_pad ? (int)p.text_len[b] : 0;
    const int pad_hi = (int)p.text_pad;
    const float c = p.scale_log2;  // positive (the host sends other scales elsewhere)

    [[maybe_unused]] uint32_t trace_cursor = 0;
    float m_run = -INFINITY;  // running maximum of the raw scores
    float m_ref = -INFINITY;  // maximum the stored exponents refer to
    float l_run = 0.0f;
    uint32_t phase = 0;
    bool ok = true;
    int processed = 0;

    const int u_first = ctl->tile_first[sub], u_end = u_first + ctl->tile_count[sub];
    if constexpr (kBounded) {
        const float2 cs2 = make_float2(c, c), bias2 = make_float2(-bound, -bound);
        float2 sum_a = make_float2(0.0f, 0.0f), sum_b = make_float2(0.0f, 0.0f);
        for (int u = u_first; u < u_end && ok; ++u) {
            const int j = phys_tile(ctl, u);
            ok = mbar_wait(ctl, bar_s, phase, p.status, (1u << 16) | (uint32_t)(kBarSFull + sub),
                           (uint32_t)j);
            if (!ok) break;
            phase ^= 1u;
            tc_fence_after();
            if (tid_in_group == 0) QW_TRACE(sub, 0, j);
            const int key0 = j * kTileN;
            const bool pad_hit = pad_hi > pad_lo && key0 < pad_hi && key0 + kTileN > pad_lo;
            const bool boundary = __any_sync(0xffffffffu, key0 + kTileN > my_limit) || pad_hit;
            const auto softmax_tile = [&](auto masked) __attribute__((always_inline)) {
                uint32_t sa[32], sb[32];
                QW_TMEM_LD32(tmem_s, sa);
#pragma unroll
                for (int chunk = 0; chunk < 4; ++chunk) {
                    uint32_t(&cur)[32] = (chunk & 1) ? sb : sa;
                    uint32_t(&nxt)[32] = (chunk & 1) ? sa : sb;
                    if (chunk == kPart / 2) publish_p_first(bar_p_first, tid_in_group);
                    QW_TMEM_WAIT_LD32(cur);
                    if (chunk == 0 && tid_in_group == 0) QW_TRACE(sub, 1, j);
                    if (chunk < 3) QW_TMEM_LD32(tmem_s + 32 * (chunk + 1), nxt);
                    if constexpr (decltype(masked)::value)
                        mask_scores(cur, key0 + chunk * 32, my_limit, pad_lo, pad_hi);
                    uint32_t pk[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        float2 x = ffma2(make_float2(__uint_as_float(cur[2 * i]),
                                                     __uint_as_float(cur[2 * i + 1])),
                                         cs2, bias2);
                        const float2 pr = make_float2(fast_exp2(x.x), fast_exp2(x.y));
                        if (i & 1) sum_b = fadd2(sum_b, pr);
                        else sum_a = fadd2(sum_a, pr);
                        pk[i] = pack_bf16(pr.x, pr.y);
                    }
                    // P chunk c lands on columns [16c, 16c+16): scores already consumed.
                    QW_TMEM_ST16(tmem_s + chunk * 16, pk);
                    if (chunk == 1 && tid_in_group == 0) QW_TRACE(sub, 2, j);
                }
            };
            if (boundary) softmax_tile(std::true_type());
            else softmax_tile(std::false_type());
            if (tid_in_group == 0) QW_TRACE(sub, 3, j);
            tmem_wait_st();
            tc_fence_before();
            if ((tid_in_group & 31) == 0) mbar_arrive(bar_p);
            if (tid_in_group == 0) QW_TRACE(sub, 4, j);
            ++processed;
        }
        sum_a = fadd2(sum_a, sum_b);
        l_run = sum_a.x + sum_a.y;
    } else
    for (int u = u_first; u < u_end && ok; ++u) {
        const int j = phys_tile(ctl, u);
        ok = mbar_wait(ctl, bar_s, phase, p.status, (1u << 16) | (uint32_t)(kBarSFull + sub),
                       (uint32_t)j);
        if (!ok) break;
        phase ^= 1u;
        tc_fence_after();
        if (tid_in_group == 0) QW_TRACE(sub, 0, j);

        const int key0 = j * kTileN;
        const bool pad_hit = pad_hi > pad_lo && key0 < pad_hi && key0 + kTileN > pad_lo;
        const bool boundary = __any_sync(0xffffffffu, key0 + kTileN > my_limit) || pad_hit;
        // A row sees all of the tile, part of it (its limit or the padding window cuts it) or,
        // like a text row beside image rows, nothing.
        const bool cut =
            __any_sync(0xffffffffu, (uint32_t)(my_limit - key0 - 1) < (uint32_t)(kTileN - 1)) || pad_hit;
        if (cut) mask_tile(tmem_s, key0, my_limit, pad_lo, pad_hi);
        uint32_t s[128];
        QW_TMEM_LD32(tmem_s + 0, s + 0);
        QW_TMEM_LD32(tmem_s + 32, s + 32);
        QW_TMEM_LD32(tmem_s + 64, s + 64);
        QW_TMEM_LD32(tmem_s + 96, s + 96);
        tmem_wait_ld();
        if (boundary && !cut) {
            const bool unseen = key0 >= my_limit;
#pragma unroll
            for (int i = 0; i < kTileN; ++i) s[i] = unseen ? 0xff800000u : s[i];
        }
        if (tid_in_group == 0) QW_TRACE(sub, 1, j);

        // Row maximum (four independent chains).
        float e0 = -INFINITY, e1 = -INFINITY, e2 = -INFINITY, e3 = -INFINITY;
#pragma unroll
        for (int i = 0; i < 128; i += 8) {
            e0 = fmax3(e0, __uint_as_float(s[i]), __uint_as_float(s[i + 1]));
            e1 = fmax3(e1, __uint_as_float(s[i + 2]), __uint_as_float(s[i + 3]));
            e2 = fmax3(e2, __uint_as_float(s[i + 4]), __uint_as_float(s[i + 5]));
            e3 = fmax3(e3, __uint_as_float(s[i + 6]), __uint_as_float(s[i + 7]));
        }
        const float m_tile = fmaxf(fmaxf(e0, e1), fmaxf(e2, e3));
        const float m_new = fmaxf(m_run, m_tile);
        m_run = m_new;
        // Does the reference point have to move?  (first finite value, or drift > threshold)
        const bool move = (m_new != -INFINITY) &&
                          (m_ref == -INFINITY || (m_new - m_ref) * c > kRescaleThreshold);
        const bool any_move = __any_sync(0xffffffffu, move && processed > 0 && m_ref != -INFINITY);
        float alpha = 1.0f;
        if (move) {
            alpha = (m_ref == -INFINITY) ? 0.0f : fast_exp2((m_ref - m_new) * c);
            m_ref = m_new;
        }
        if (any_move) {
            // s_full of this tile was committed after the previous P V of this
            // sub-tile, so O is quiescent until P of this tile is published.
#pragma unroll 1
            for (int chunk = 0; chunk < 4; ++chunk) {
                uint32_t o[32];
                QW_TMEM_LD32(tmem_o + chunk * 32, o);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                QW_TMEM_ST32(tmem_o + chunk * 32, o);
            }
            tmem_wait_st();
        }
        l_run *= alpha;
        if (tid_in_group == 0) QW_TRACE(sub, 2, j);

        // P = exp2(score*c - m_ref*c) as bf16 pairs, written over S 32 keys (16 packed
        // columns) at a time.
        const float bias = (m_ref == -INFINITY) ? 0.0f : -m_ref * c;
        const float2 cs2 = make_float2(c, c), bias2 = make_float2(bias, bias);
        float2 sum_a = make_float2(0.0f, 0.0f), sum_b = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int chunk = 0; chunk < 4; ++chunk) {
            uint32_t pk[16];
            if (chunk == kPart / 2) {
                publish_p_first(bar_p_first, tid_in_group);
                QW_TMEM_WAIT_LD32(s + 32 * (kPart / 2));  // (nothing is loading: the rest stays behind)
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int e = chunk * 32 + 2 * i;
                float2 x = ffma2(make_float2(__uint_as_float(s[e]), __uint_as_float(s[e + 1])),
                                 cs2, bias2);
                const float2 pr = make_float2(fast_exp2(x.x), fast_exp2(x.y));
                if (i & 1) sum_b = fadd2(sum_b, pr);
                else sum_a = fadd2(sum_a, pr);
                pk[i] = pack_bf16(pr.x, pr.y);
            }
            QW_TMEM_ST16(tmem_s + chunk * 16, pk);
        }
        if (tid_in_group == 0) QW_TRACE(sub, 3, j);
        tmem_wait_st();  // warp-collective: every lane's stores have landed
        tc_fence_before();
        if ((tid_in_group & 31) == 0) mbar_arrive(bar_p);
        if (tid_in_group == 0) QW_TRACE(sub, 4, j);
        sum_a = fadd2(sum_a, sum_b);
        l_run += sum_a.x + sum_a.y;
        ++processed;
    }

    // Epilogue: O / l -> bf16.
    if (!ok || tile_row0 >= p.q_rows) return;  // gave up, or this sub-tile holds no rows
    if (processed > 0) {
        ok = mbar_wait(ctl, bar_at(bars, kBarOFinal), 0, p.status,
                       (1u << 16) | (uint32_t)(kBarOFinal + sub), 0xffffu);
        if (!ok) return;
        tc_fence_after();
    }
    // Scale factors of the accumulators that make up the output rows: O_sub alone,
    // or in split form O_0 and O_1 brought to a common reference exponent.
    // out = (w_own * O_own + w_other * O_other) * inv: the weights are exactly 1 when
    // the reference exponents agree, so a split block of equal-score rows merges
    // exactly like the whole block would have summed.
    float w_own = 1.0f, w_other = 0.0f, inv = l_run > 0.0f ? 1.0f / l_run : 0.0f;
    bool use_own = processed > 0, use_other = false;
    if (split) {
        const float m_own = kBounded ? (processed > 0 ? bound : -INFINITY)
                            : (processed > 0 && m_ref != -INFINITY) ? m_ref * c
                                                                    : -INFINITY;
        if (sub == 1) {
            // Publish exponent and row sum; warpgroup 0 reads O_1 itself (same lanes).
            ctl->merge_m[tid_in_group] = m_own;
            ctl->merge_l[tid_in_group] = l_run;
            __syncwarp();
            if ((tid_in_group & 31) == 0) mbar_arrive(&ctl->bars[kBarMerge]);
            return;
        }
        ok = mbar_wait(ctl, bar_at(bars, kBarMerge), 0, p.status, (1u << 16) | (uint32_t)kBarMerge,
                       0xfffbu);
        if (!ok) return;
        use_other = ctl->tile_count[1] > 0;
        if (use_other) {
            ok = mbar_wait(ctl, bar_at(bars, kBarOFinal + 1), 0, p.status,
                           (1u << 16) | (uint32_t)(kBarOFinal + 1), 0xfffeu);
            if (!ok) return;
            tc_fence_after();
        }
        const float m_other = ctl->merge_m[tid_in_group], l_other = ctl->merge_l[tid_in_group];
        const float m_all = fmaxf(m_own, m_other);
        const float a_own = m_own == -INFINITY ? 0.0f : fast_exp2(m_own - m_all);
        const float a_other = m_other == -INFINITY ? 0.0f : fast_exp2(m_other - m_all);
        const float l_all = a_own * l_run + a_other * l_other;
        inv = l_all > 0.0f ? 1.0f / l_all : 0.0f;
        w_own = a_own;
        w_other = a_other;
    } else if (processed == 0) {
        // Nothing was computed for this sub-tile (zeros go out), but its Q load may
        // still be in flight into the staging area: let it land first.
        ok = mbar_wait(ctl, bar_at(bars, kBarQFull), 0, p.status,
                       (1u << 16) | (uint32_t)(kBarQFull + sub), 0xfffdu);
        if (!ok) return;
    }
    if (split && !use_own) {
        // (same reason: the shared Q tile is the staging area)
        ok = mbar_wait(ctl, bar_at(bars, kBarQFull), 0, p.status,
                       (1u << 16) | (uint32_t)(kBarQFull + 0), 0xfffdu);
        if (!ok) return;
    }
    const uint32_t warp_row0 = tile_row0 + (uint32_t)warp_in_group * 32u;
    if (warp_row0 >= p.q_rows) return;
    const uint32_t row_stride = (p.head_major_out ? 1u : p.out_heads_total) * kHeadDim;
    const size_t first = p.head_major_out
                             ? (((size_t)b * p.heads + h) * p.q_rows + warp_row0) * kHeadDim
                             : ((size_t)b * p.q_rows + warp_row0) * row_stride +
                                   (size_t)(p.out_head_offset + h) * kHeadDim;
    const uint32_t tmem_own = use_own ? tmem_o : kNoTmem;
    const uint32_t tmem_other = use_other ? tmem + lane_base + kTmemO1 : kNoTmem;
#pragma unroll 1
    for (uint32_t d = 0; d < p.n_out; ++d)
        write_rows(tmem_own, tmem_other, w_own, w_other, inv,
                   smem_u32(stage + warp_in_group * (32 * 128)), p.out_peers[d] + first, row_stride,
                   min(32u, p.q_rows - warp_row0));
}

// ---------------------------------------------------------------------------
// MMA issue role: one warp.  All lanes run the loop and one is elected around the
// instructions (always the same one, so its commits cover its MMAs): the operands of
// the MMAs then stay in uniform registers, where in a one-lane branch each of them is
// moved there first, more clocks per MMA than the 64 it executes in.
// ---------------------------------------------------------------------------
// Low descriptor words, everything but the start address; V's two 64-column halves lie half
// a tile apart.
constexpr uint32_t kDescLoVMajor = desc_lo(kHalfTileBytes);

__device__ __forceinline__ void issue_qk(uint32_t d_tmem, uint32_t q_lo, uint32_t k_lo) {
    // K-major operands, 128B swizzle: 8-row groups 1024 B apart; the second
    // 64-column box sits one half tile further; 16 columns = 32 B per step.
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
        const uint32_t off = ((uint32_t)(kk >> 2) * kHalfTileBytes + (uint32_t)(kk & 3) * 32u) >> 4;
        mma_ss<1>(d_tmem, q_lo + off, k_lo + off, kIdescQK, kk > 0 ? 1u : 0u);
    }
}

// Keys 16 * kFrom .. 16 * kTo - 1 of P V.
template <int kFrom, int kTo>
__device__ __forceinline__ void issue_pv_keys(uint32_t d_tmem, uint32_t p_tmem, uint32_t v_lo,
                                              bool accumulate) {
    // A = P from TMEM (16 keys = 8 packed columns per step).  B = V, MN-major:
    // 16 keys = 2 groups of 8 rows (1024 B apart), the two 64-wide column
    // halves one half tile apart.
#pragma unroll
    for (int kk = kFrom; kk < kTo; ++kk) {
        mma_ts(d_tmem, p_tmem + (uint32_t)kk * 8u, v_lo + (uint32_t)(kk * 2048 >> 4), kIdescPV,
               (accumulate || kk > 0) ? 1u : 0u);
    }
}

__device__ __forceinline__ void mma_role(const KernelParams &p, SharedControl *ctl,
                                         uint8_t *smem_q, uint8_t *smem_kv) {
    // Whole form: both sub-tiles walk the visited tiles from 0; u counts them.
    const int n0 = uniform(ctl->tile_count[0]), n1 = uniform(ctl->tile_count[1]);
    const int n_max = max(n0, n1);
    int j = 0;
    if (j >= n_max) return;
    const uint32_t tmem = uniform(ctl->tmem_base), bars = uniform(smem_u32(ctl->bars));
    // Low descriptor words: start address in 16-byte units plus the fixed LBO field.
    const uint32_t q_lo = (smem_u32(smem_q) >> 4) | kDescKMajor;  // sub-tile 1's is one tile further
    const uint32_t kv_lo = smem_u32(smem_kv) >> 4;  // slot s starts (s * kTileBytes) >> 4 further
    uint32_t t = 0;  // ring position (K and V tiles alternate)
    [[maybe_unused]] uint32_t trace_cursor = 0;

    {
        const uint32_t slot = t++ % kStages;
        if (!mbar_wait_warp(p, bar_at(bars, kBarKvFull + slot), 0))
            return mma_gave_up(ctl, p.status, kBarKvFull + slot, (uint32_t)j);
        const uint32_t k_lo = (kv_lo + slot * (kTileBytes >> 4)) | kDescKMajor;
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
            if (j >= (i ? n1 : n0)) continue;
            if (!mbar_wait_warp(p, bar_at(bars, kBarQFull + i), 0))
                return mma_gave_up(ctl, p.status, kBarQFull + i, 0);
            tc_fence_after();
            if (elect_one()) {
                issue_qk(tmem + kTmemS0 + (uint32_t)i * kTileN,
                         q_lo + (uint32_t)i * (kTileBytes >> 4), k_lo);
                tc_commit<1>(bar_at(bars, kBarSFull + i));
            }
            __syncwarp();
        }
        if (elect_one()) tc_commit<1>(bar_at(bars, kBarKvEmpty + slot));
        __syncwarp();
    }
    uint32_t v_slot = t++ % kStages;
    if (!mbar_wait_warp(p, bar_at(bars, kBarKvFull + v_slot), 0))
        return mma_gave_up(ctl, p.status, kBarKvFull + v_slot, (uint32_t)j);
    // The tensor cores take four MMAs ahead, about 150 clocks of work, and a wait costs this warp 60
    // to 110 even where nothing is left to wait for.  So the next tiles of K and of V are waited
    // for behind the first parts of P V, where the warp waits for the rest of P anyway, and not both
    // in front of the step; and the two sub-tiles take turns in one loop, whose code is half as long.
    // Layers of six heads, 4352 keys, gained 1.4 %, and 2.7 % more with the epilogue's registers out
    // of the softmax's way (see write_rows).
    while (j < n_max) {
        const int jn = j + 1;
        const bool more = jn < n_max;
        const uint32_t k_slot = t % kStages, k_par = (t / kStages) & 1u;
        const uint32_t v_lo = (kv_lo + v_slot * (kTileBytes >> 4)) | kDescLoVMajor;
        const uint32_t k_lo = (kv_lo + k_slot * (kTileBytes >> 4)) | kDescKMajor;
        bool have_k = !more;
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
            const int n_i = i ? n1 : n0;
            const uint32_t s_i = tmem + kTmemS0 + (uint32_t)i * kTileN;
            const uint32_t o_i = tmem + kTmemO0 + (uint32_t)i * kTileN;
            if (j < n_i) {
                if (!mbar_wait_warp(p, bar_at(bars, kBarPFirst + i), (uint32_t)j & 1u))
                    return mma_gave_up(ctl, p.status, kBarPFirst + i, (uint32_t)j);
                tc_fence_after();
                QW_TRACE(2, i, j);
                if (elect_one())
                    issue_pv_keys<0, kPart>(o_i, s_i, v_lo, j > 0);
                __syncwarp();
                if (i == 1 && more) {
                    const uint32_t tv = t + 1;
                    if (!mbar_wait_warp(p, bar_at(bars, kBarKvFull + tv % kStages), (tv / kStages) & 1u))
                        return mma_gave_up(ctl, p.status, kBarKvFull + tv % kStages, (uint32_t)jn);
                }
                if (!have_k) {
                    if (!mbar_wait_warp(p, bar_at(bars, kBarKvFull + k_slot), k_par))
                        return mma_gave_up(ctl, p.status, kBarKvFull + k_slot, (uint32_t)jn);
                    have_k = true;
                }
                if (!mbar_wait_warp(p, bar_at(bars, kBarPFull + i), (uint32_t)j & 1u))
                    return mma_gave_up(ctl, p.status, kBarPFull + i, (uint32_t)j);
                tc_fence_after();
                if (elect_one()) {
                    issue_pv_keys<kPart, 8>(o_i, s_i, v_lo, true);
                    if (i == 1 && more) tc_commit<1>(bar_at(bars, kBarKvEmpty + v_slot));
                    if (jn < n_i) {
                        issue_qk(s_i, q_lo + (uint32_t)i * (kTileBytes >> 4), k_lo);
                        tc_commit<1>(bar_at(bars, kBarSFull + i));
                    } else {
                        tc_commit<1>(bar_at(bars, kBarOFinal + i));
                    }
                }
                __syncwarp();
                QW_TRACE(2, 2 + i, jn);
            }
        }
        if (more) {
            if (elect_one()) {
                if (j >= n1) tc_commit<1>(bar_at(bars, kBarKvEmpty + v_slot));
                tc_commit<1>(bar_at(bars, kBarKvEmpty + k_slot));
            }
            __syncwarp();
            ++t;
            v_slot = t % kStages;
            if (j >= n1 && !mbar_wait_warp(p, bar_at(bars, kBarKvFull + v_slot), (t / kStages) & 1u))
                return mma_gave_up(ctl, p.status, kBarKvFull + v_slot, (uint32_t)jn);
            ++t;
        }
        j = jn;
    }
}

// Split form: sub-tile 0 walks visited tiles [0, la), sub-tile 1 [la, la + lb),
// both against the one Q tile.  K/V pairs are loaded in the order a0 b0 a1 b1 ...
// (pair = K then V, one ring slot each); slot_of() gives the ring position of a
// pair's K, its V follows.
__device__ __forceinline__ uint32_t pair_a(int s, int lb) { return 2u * (uint32_t)(s + min(s, lb)); }
__device__ __forceinline__ uint32_t pair_b(int s) { return 2u * (uint32_t)(2 * s + 1); }

__device__ __forceinline__ void mma_role_split(const KernelParams &p, SharedControl *ctl,
                                               uint8_t *smem_q, uint8_t *smem_kv) {
    const int la = uniform(ctl->tile_count[0]), lb = uniform(ctl->tile_count[1]);
    if (la <= 0) return;
    const uint32_t tmem = uniform(ctl->tmem_base), bars = uniform(smem_u32(ctl->bars));
    const uint32_t q_lo = (smem_u32(smem_q) >> 4) | kDescKMajor;
    const uint32_t kv_lo = smem_u32(smem_kv) >> 4;

    // Waits for ring position t, returns the low descriptor word of its slot.
#define QW_RING_WAIT(t_, lo_fixed_, out_)                                                       \
    {                                                                                           \
        const uint32_t slot_ = (t_) % kStages, par_ = ((t_) / kStages) & 1u;                    \
        if (!mbar_wait_warp(p, bar_at(bars, kBarKvFull + slot_), par_))                         \
            return mma_gave_up(ctl, p.status, kBarKvFull + slot_, (t_));                        \
        tc_fence_after();                                                                       \
        out_ = (kv_lo + slot_ * (kTileBytes >> 4)) | (lo_fixed_);                               \
    }
#define QW_RING_FREE(t_) tc_commit<1>(bar_at(bars, kBarKvEmpty + ((t_) % kStages)))

    if (!mbar_wait_warp(p, bar_at(bars, kBarQFull + 0), 0))
        return mma_gave_up(ctl, p.status, kBarQFull + 0, 0);
    uint32_t desc;
    QW_RING_WAIT(pair_a(0, lb), kDescKMajor, desc);
    if (elect_one()) {
        issue_qk(tmem + kTmemS0, q_lo, desc);
        tc_commit<1>(bar_at(bars, kBarSFull + 0));
        QW_RING_FREE(pair_a(0, lb));
    }
    __syncwarp();
    if (lb > 0) {
        QW_RING_WAIT(pair_b(0), kDescKMajor, desc);
        if (elect_one()) {
            issue_qk(tmem + kTmemS1, q_lo, desc);
            tc_commit<1>(bar_at(bars, kBarSFull + 1));
            QW_RING_FREE(pair_b(0));
        }
        __syncwarp();
    }
    for (int s = 0; s < la; ++s) {
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
            const uint32_t s_i = tmem + kTmemS0 + (uint32_t)i * kTileN;
            const uint32_t o_i = tmem + kTmemO0 + (uint32_t)i * kTileN;
            const int count = i ? lb : la;
            if (s >= count) continue;
            const uint32_t t_now = i ? pair_b(s) : pair_a(s, lb);
            QW_RING_WAIT(t_now + 1, kDescLoVMajor, desc);
            if (!mbar_wait_warp(p, bar_at(bars, kBarPFirst + i), (uint32_t)s & 1u))
                return mma_gave_up(ctl, p.status, kBarPFirst + i, (uint32_t)s);
            tc_fence_after();
            if (elect_one()) issue_pv_keys<0, kPart>(o_i, s_i, desc, s > 0);
            __syncwarp();
            if (!mbar_wait_warp(p, bar_at(bars, kBarPFull + i), (uint32_t)s & 1u))
                return mma_gave_up(ctl, p.status, kBarPFull + i, (uint32_t)s);
            tc_fence_after();
            if (elect_one()) {
                issue_pv_keys<kPart, 8>(o_i, s_i, desc, true);
                QW_RING_FREE(t_now + 1);
            }
            __syncwarp();
            if (s + 1 < count) {
                const uint32_t t_next = i ? pair_b(s + 1) : pair_a(s + 1, lb);
                QW_RING_WAIT(t_next, kDescKMajor, desc);
                if (elect_one()) {
                    issue_qk(s_i, q_lo, desc);
                    tc_commit<1>(bar_at(bars, kBarSFull + i));
                    QW_RING_FREE(t_next);
                }
                __syncwarp();
            }
        }
    }
#undef QW_RING_WAIT
#undef QW_RING_FREE
    if (elect_one()) {
        tc_commit<1>(bar_at(bars, kBarOFinal + 0));
        tc_commit<1>(bar_at(bars, kBarOFinal + 1));
    }
}

// ---------------------------------------------------------------------------
// TMA producer role (one thread).
// ---------------------------------------------------------------------------
__device__ void tma_role(const KernelParams &p, SharedControl *ctl, uint8_t *smem_kv,
                         const CUtensorMap *map_k, const CUtensorMap *map_v, uint32_t b,
                         uint32_t kvh, bool split) {
    const uint32_t where = 3u << 16;
    // K and V of the first visited tile are already on their way (ring slots 0, 1):
    // the kernel body issued them before the row limits were known.
    uint32_t t = 2;
    bool ok = true;
    const int col = (int)(kvh * kHeadDim);
    // One (K, V) pair of visited tile u into the next two ring slots.
    auto load_pair = [&](int u) {
        if (p.withhold_from >= 0 && u >= p.withhold_from) {
            ok = false;  // the tile stays away: nothing is issued, nothing is in flight
            return;
        }
        const int j = phys_tile(ctl, u);
        for (int which = 0; which < 2 && ok; ++which) {
            uint32_t slot = t % kStages, par = ((t / kStages) & 1u) ^ 1u;
            ok = mbar_wait(ctl, smem_u32(&ctl->bars[kBarKvEmpty + slot]), par, p.status,
                           where | (kBarKvEmpty + slot), (uint32_t)j);
            if (!ok) break;
            ++t;
            uint8_t *dst = smem_kv + (size_t)slot * kTileBytes;
            Mbar *bar = &ctl->bars[kBarKvFull + slot];
            mbar_expect_tx(bar, kTileBytes);
            const CUtensorMap *map = which ? map_v : map_k;
            tma_load_3d(dst, map, bar, col, j * kTileN, (int)b);
            tma_load_3d(dst + kHalfTileBytes, map, bar, col + 64, j * kTileN, (int)b);
        }
    };
    if (!split) {
        const int n_max = max(ctl->tile_count[0], ctl->tile_count[1]);
        for (int u = 1; u < n_max && ok; ++u) load_pair(u);
    } else {
        // pairs in the order a0 (under way), b0, a1, b1, ...
        const int la = ctl->tile_count[0], lb = ctl->tile_count[1];
        for (int s = 0; s < la && ok; ++s) {
            if (s > 0) load_pair(s);
            if (s < lb && ok) load_pair(la + s);
        }
    }
    // Leave no copy in flight: every issued load must have landed before the
    // CTA may release its shared memory (bounded like every other wait).
    uint32_t first = t > (uint32_t)kStages ? t - kStages : 0;
    for (uint32_t u = first; u < t; ++u) {
        uint32_t slot = u % kStages, par = (u / kStages) & 1u;
        long long start = clock64();
        while (!mbar_try(&ctl->bars[kBarKvFull + slot], par))
            if (clock64() - start > ctl->wait_cycles) break;
    }
}

__device__ __forceinline__ void issue_q_loads(const KernelParams &p, SharedControl *ctl,
                                              uint8_t *smem_q, const CUtensorMap *map_q, uint32_t b,
                                              uint32_t h, uint32_t row0, int tiles) {
    for (int i = 0; i < tiles; ++i) {
        uint32_t r = row0 + (uint32_t)i * kTileM;
        if (r >= p.q_rows) continue;  // inactive sub-tile: n_tiles is 0, nobody waits
        Mbar *bar = &ctl->bars[kBarQFull + i];
        mbar_expect_tx(bar, kTileBytes);
        uint8_t *dst = smem_q + (size_t)i * kTileBytes;
        tma_load_3d(dst, map_q, bar, (int)(h * kHeadDim), (int)r, (int)b);
        tma_load_3d(dst + kHalfTileBytes, map_q, bar, (int)(h * kHeadDim) + 64, (int)r, (int)b);
    }
}

template <bool kMayBound>
__global__ void __launch_bounds__(kThreads, 1)
qw_attn_sm100_kernel(const __grid_constant__ CUtensorMap map_q,
                     const __grid_constant__ CUtensorMap map_k,
                     const __grid_constant__ CUtensorMap map_v, const KernelParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *smem_q = smem;
    uint8_t *smem_kv = smem + 2 * kTileBytes;
    SharedControl *ctl = reinterpret_cast<SharedControl *>(smem + kSmemData);

    const int tid = threadIdx.x;
    const int warp = warp_index();
    const int lane = tid & 31;
    // CTA -> unit.  Units are numbered batch-major, then head, then query block
    // with the heaviest blocks first (rows late in the joint sequence see the most
    // keys).  The last tail_units units run in split form, two CTAs each.
    const uint32_t whole_units = p.total_units - p.tail_units;
    const bool split = blockIdx.x >= whole_units;
    const uint32_t unit = split ? whole_units + ((blockIdx.x - whole_units) >> 1) : blockIdx.x;
    const uint32_t half = split ? (blockIdx.x - whole_units) & 1u : 0u;
    const uint32_t bh = unit / p.n_qblocks;
    const uint32_t b = bh / p.heads;
    const uint32_t h = bh - b * p.heads;
    const uint32_t kvh = (uint32_t)((unsigned long long)h * p.kv_heads / p.heads);
    const uint32_t qblock = p.n_qblocks - 1 - (unit - bh * p.n_qblocks);
    const uint32_t row0 = qblock * (2 * kTileM) + half * kTileM;

    // The producer thread sets the barriers up itself and starts Q and the first
    // K/V tile at once, under the row-limit loads of the softmax threads.
    if (warp == kTmaWarp && lane == 0) {
        for (int i = 0; i < 2; ++i) mbar_init(&ctl->bars[kBarQFull + i], 1);
        for (int i = 0; i < kStages; ++i) {
            mbar_init(&ctl->bars[kBarKvFull + i], 1);
            mbar_init(&ctl->bars[kBarKvEmpty + i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&ctl->bars[kBarSFull + i], 1);
            mbar_init(&ctl->bars[kBarPFirst + i], kTileM / 32);
            mbar_init(&ctl->bars[kBarPFull + i], kTileM / 32);
            mbar_init(&ctl->bars[kBarOFinal + i], 1);
        }
        mbar_init(&ctl->bars[kBarMerge], kTileM / 32);
        ctl->abort_flag = 0;
        ctl->wait_cycles = p.wait_cycles > 0 ? p.wait_cycles : kWaitCycles;
        int lo = 0, hi = 0;
        if (p.text_pad && p.text_len[b] < p.text_pad) {
            lo = ((int)p.text_len[b] + kTileN - 1) / kTileN;
            hi = (int)p.text_pad / kTileN;
            if (hi < lo) hi = lo;
        }
        ctl->skip_lo = lo;
        ctl->skip_hi = hi;
        mbar_init_fence();
    }
    if (warp == kMmaWarp) {
        tmem_alloc<1>(&ctl->tmem_base, kTmemCols);
    }
    // What stands above may run under the tail of the kernel before this one; all that
    // reads or writes global memory stands below.
    grid_launch_dependents();
    grid_wait();
    if (warp == kTmaWarp && lane == 0) {
        const int lo = ctl->skip_lo, hi = ctl->skip_hi;
        issue_q_loads(p, ctl, smem_q, &map_q, b, h, row0, split ? 1 : 2);
        // First visited key tile, assuming the unit has one (if it has none the
        // tile is simply never consumed; the producer drains it before exit).
        const int j0 = lo == 0 ? hi : 0;
        for (int which = 0; which < 2; ++which) {
            uint8_t *dst = smem_kv + (size_t)which * kTileBytes;
            Mbar *bar = &ctl->bars[kBarKvFull + which];
            mbar_expect_tx(bar, kTileBytes);
            const CUtensorMap *map = which ? &map_v : &map_k;
            const int col = (int)(kvh * kHeadDim);
            tma_load_3d(dst, map, bar, col, j0 * kTileN, (int)b);
            tma_load_3d(dst + kHalfTileBytes, map, bar, col + 64, j0 * kTileN, (int)b);
        }
    }
    if (blockIdx.x == 0 && warp == 10 && lane == 0 && p.slot_use) {
        // Sharded heads: whatever read this output slot's previous contents was
        // enqueued before this kernel, so the peers may store the new epoch now.
        const uint32_t epoch = *p.slot_use + 1u;
        *p.slot_use = epoch;
        __threadfence_system();
        for (uint32_t d = 0; d < p.n_freed; ++d)
            asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p.freed_peer[d]), "r"(epoch)
                         : "memory");
    }

    // Row limits: each softmax thread owns one row; the largest limit of a
    // sub-tile bounds its key-tile loop.
    int my_limit = 0;
    int sub = 0, tid_in_group = 0;
    // Fixed reference exponent (log2 units, an integer so that P is the exact
    // power-of-two multiple of what any other reference would give), or < 0 for
    // the running-maximum softmax: no promise given, or one too loose to keep
    // exp2(score*c - bound) >= 2^-2*bound inside the normal fp32 range.
    float bound = -1.0f;
    if (kMayBound && p.score_bound) {  // every role needs to know which softmax runs
        const float limit = ceilf(p.score_bound[0] * p.score_bound[1] * p.scale_log2);
        if (limit >= 0.0f && limit <= 60.0f) bound = limit;
    }
    if (tid < kSoftmaxThreads) {
        sub = tid >> 7;
        tid_in_group = tid & 127;
        // (split form: both warpgroups work on the same 128 rows)
        const uint32_t my_row = row0 + (split ? 0u : (uint32_t)sub * kTileM) + (uint32_t)tid_in_group;
        my_limit = row_limit(p, b, my_row);
        int warp_max = my_limit;
        // A row past the end is computed like its neighbours and never stored: with a
        // limit of 0 it would send its whole warp through the masked path on every tile
        // (600 -> 1500 clocks a tile for the row maximum alone).
        if (my_row >= p.q_rows) my_limit = 0x7fffffff;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
            warp_max = max(warp_max, __shfl_xor_sync(0xffffffffu, warp_max, off));
        if (lane == 0) ctl->warp_max[warp] = warp_max;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (tid < 2) {
        int m = 0;
        for (int w = 0; w < 4; ++w) m = max(m, ctl->warp_max[tid * 4 + w]);
        const int tiles = (m + kTileN - 1) / kTileN;
        ctl->n_tiles[tid] = tiles;
        const int visited = visited_tiles(tiles, ctl->skip_lo, ctl->skip_hi);
        if (!split) {
            ctl->tile_first[tid] = 0;
            ctl->tile_count[tid] = visited;
        } else {
            // both warpgroups saw the same rows: the first half (rounded up) and the rest
            const int first_half = (visited + 1) / 2;
            ctl->tile_first[tid] = tid ? first_half : 0;
            ctl->tile_count[tid] = tid ? visited - first_half : first_half;
        }
    }
    __syncthreads();

    if (tid < kSoftmaxThreads) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSoftmaxRegs));
        uint8_t *stage = smem_q + (size_t)sub * kTileBytes;
        const uint32_t tile_row0 = split ? row0 : row0 + (uint32_t)sub * kTileM;
        if (kMayBound && bound >= 0.0f)
            softmax_role<kMayBound>(p, ctl, stage, sub, tid_in_group, my_limit, b, h, tile_row0, split,
                                    bound);
        else
            softmax_role<false>(p, ctl, stage, sub, tid_in_group, my_limit, b, h, tile_row0, split, 0.0f);
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
    }
    if (tid < kSoftmaxThreads) {
    } else if (warp == kMmaWarp) {
        if (split) mma_role_split(p, ctl, smem_q, smem_kv);
        else mma_role(p, ctl, smem_q, smem_kv);
    } else if (warp == kTmaWarp && lane == 0) {
        tma_role(p, ctl, smem_kv, &map_k, &map_v, b, kvh, split);
        // Q loads of active sub-tiles must have landed as well.
        for (int i = 0; i < (split ? 1 : 2); ++i) {
            if (row0 + (uint32_t)i * kTileM >= p.q_rows) continue;
            long long start = clock64();
            while (!mbar_try(&ctl->bars[kBarQFull + i], 0))
                if (clock64() - start > ctl->wait_cycles) break;
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        tc_fence_after();
        tmem_dealloc<1>(ctl->tmem_base, kTmemCols);
    }
}

// [batch][rows][heads*128] bf16, boxes of 128 rows x 64 columns.
int make_map_3d(CUtensorMap *map, const void *base, uint32_t batch, uint32_t rows, uint32_t heads) {
    const cuuint64_t dims[3] = {(cuuint64_t)heads * kHeadDim, rows, batch};
    const cuuint64_t strides[2] = {(cuuint64_t)heads * kHeadDim * 2,
                                   (cuuint64_t)rows * heads * kHeadDim * 2};
    return make_map(map, base, 3, dims, strides, kTileN);
}

#ifdef QW_ATTN_TRACE
// QW_CUDA_ATTN_TRACE=<file>: attach an event log to every launch and dump it after
// each one (synchronous; a debugging aid, never set in production runs).
unsigned long long *trace_buffer() {
    static unsigned long long *buffer = nullptr;
    static bool looked = false;
    if (!looked) {
        looked = true;
        const char *path = getenv("QW_CUDA_ATTN_TRACE");
        if (path && *path) {
            if (cudaMalloc(&buffer, kTraceSlots * 8) != cudaSuccess) buffer = nullptr;
            else cudaMemset(buffer, 0, kTraceSlots * 8);
        }
    }
    return buffer;
}

void trace_dump(cudaStream_t stream) {
    unsigned long long *buffer = trace_buffer();
    if (!buffer) return;
    static unsigned long long host[kTraceSlots];
    cudaStreamSynchronize(stream);
    cudaMemcpy(host, buffer, sizeof(host), cudaMemcpyDeviceToHost);
    cudaMemset(buffer, 0, kTraceSlots * 8);
    FILE *f = fopen(getenv("QW_CUDA_ATTN_TRACE"), "a");
    if (!f) return;
    fprintf(f, "launch\n");
    for (int i = 1; i < kTraceSlots; ++i) {
        unsigned long long w = host[i];
        if (!w) continue;
        unsigned tag = (unsigned)(w >> 40);
        fprintf(f, "%u %u %u %llu\n", tag >> 20, (tag >> 12) & 0xff, tag & 0xfff,
                w & 0xffffffffffull);
    }
    fclose(f);
}
#endif

typedef void (*AttnKernel)(const CUtensorMap, const CUtensorMap, const CUtensorMap,
                           const KernelParams);

int sm_count_of_current_device() {
    static int sms[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return 148;
    if (!sms[dev]) {
        cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
        if (sms[dev] <= 0) sms[dev] = 148;
    }
    return sms[dev];
}

// QW_CUDA_ATTN_TAIL=whole: never split the last wave's units (comparison runs).
bool whole_units_forced() {
    static int forced = -1;
    if (forced < 0) {
        const char *env = getenv("QW_CUDA_ATTN_TAIL");
        forced = env && !strcmp(env, "whole") ? 1 : 0;
    }
    return forced != 0;
}

// The kernel with or without the fixed-exponent softmax, for callers that pass a score
// bound or not.  The opt-in to ~197 KB of dynamic shared memory is a per-device
// attribute: it is set on first use on every device a process drives.
AttnKernel pick_kernel(bool may_bound) {
    static bool ready[64][2];
    AttnKernel chosen = may_bound ? qw_attn_sm100_kernel<true> : qw_attn_sm100_kernel<false>;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    const bool tracked = dev >= 0 && dev < 64;
    if (!tracked || !ready[dev][may_bound ? 1 : 0]) {
        if (cudaFuncSetAttribute(chosen, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kSmemBytes) != cudaSuccess)
            return nullptr;
        if (tracked) ready[dev][may_bound ? 1 : 0] = true;
    }
    return chosen;
}

}  // namespace

// Units of the last, partly filled wave that run in split form: all of them when
// the doubled CTAs still fit the SMs (a sixteenth over is tolerated: block-causal
// layouts always have a few near-empty units that retire at once), none otherwise
// -- two half-length waves would take as long as the one they replace.
extern "C" uint32_t qwcu_attn_sm100_tail_units(uint32_t units, uint32_t sm_count) {
    if (!sm_count) return 0;
    const uint32_t rest = units % sm_count;
    return rest && 2 * rest <= sm_count + sm_count / 16 ? rest : 0u;
}

extern "C" int qwcu_attn_sm100_launch(const qwcu_attn_args *a, qwcu_stream stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (a->batch == 0 || a->batch > 8 || !a->q_rows || !a->kv_rows || !a->heads || !a->kv_heads)
        return (int)cudaErrorInvalidValue;
    // TMA needs 16-byte aligned bases; cudaMalloc gives 256.
    if (((uintptr_t)a->q | (uintptr_t)a->k | (uintptr_t)a->v | (uintptr_t)a->out) & 15u)
        return (int)cudaErrorMisalignedAddress;
    AttnKernel kernel = pick_kernel(a->score_bound != nullptr);
    if (!kernel) return (int)cudaGetLastError();
    CUtensorMap map_q, map_k, map_v;
    int rc;
    if ((rc = make_map_3d(&map_q, a->q, a->batch, a->q_rows, a->heads))) return rc;
    if ((rc = make_map_3d(&map_k, a->k, a->batch, a->kv_rows, a->kv_heads))) return rc;
    if ((rc = make_map_3d(&map_v, a->v, a->batch, a->kv_rows, a->kv_heads))) return rc;
    KernelParams p;
    p.kv_limit = a->kv_limit;
    p.status = a->status;
#ifdef QW_ATTN_TRACE
    p.trace = trace_buffer();
#endif
    p.per_batch_limits = a->per_batch_limits;
    p.causal = a->causal;
    p.causal_offset = a->causal_offset;
    p.batch = a->batch;
    p.q_rows = a->q_rows;
    p.kv_rows = a->kv_rows;
    p.heads = a->heads;
    p.kv_heads = a->kv_heads;
    for (int i = 0; i < 8; ++i) p.text_len[i] = a->text_len[i];
    p.text_pad = a->text_pad;
    p.scale_log2 = a->scale * 1.4426950408889634f;
    p.score_bound = a->score_bound;
    p.head_major_out = a->head_major_out;
    if (a->n_out_peers > 0) {
        if (a->n_out_peers > 8 || a->head_major_out) return (int)cudaErrorInvalidValue;
        p.n_out = a->n_out_peers;
        for (uint32_t d = 0; d < p.n_out; ++d) {
            if ((uintptr_t)a->out_peers[d] & 15u) return (int)cudaErrorMisalignedAddress;
            p.out_peers[d] = static_cast<__nv_bfloat16 *>(a->out_peers[d]);
        }
        p.out_heads_total = a->out_heads_total;
        p.out_head_offset = a->out_head_offset;
    } else {
        p.n_out = 1;
        p.out_peers[0] = static_cast<__nv_bfloat16 *>(a->out);
        p.out_heads_total = a->heads;
        p.out_head_offset = 0;
    }
    p.wait_cycles = a->wait_cycles;
    // (At least 32 probes, like the other waits.  kProbeCycles is more than a probe takes: this
    // role, which waits for the cause itself, gives up before those that wait behind it.)
    const long long budget = p.wait_cycles > 0 ? p.wait_cycles : kWaitCycles;
    p.mma_probes = 32 + (int)min(budget / kProbeCycles, 1ll << 30);
    p.withhold_from = a->withhold_from > 0 ? a->withhold_from : -1;
    p.slot_use = a->slot_use;
    p.n_freed = a->slot_use ? a->n_freed : 0;
    if (p.n_freed > 8) return (int)cudaErrorInvalidValue;
    for (uint32_t d = 0; d < 8; ++d) p.freed_peer[d] = d < p.n_freed ? a->freed_peer[d] : nullptr;
    // One CTA per unit; the units of the last, partly filled wave run split in two
    // (half the rows each, the key tiles divided between the sub-tiles) when the
    // doubled CTAs still fit the idle SMs, give or take a few light units.
    const unsigned long long units =
        (unsigned long long)((a->q_rows + 2 * kTileM - 1) / (2 * kTileM)) * a->heads * a->batch;
    if (units > 0x3fffffffull) return (int)cudaErrorInvalidValue;
    p.n_qblocks = (a->q_rows + 2 * kTileM - 1) / (2 * kTileM);
    p.total_units = (uint32_t)units;
    p.tail_units = (a->whole_units || whole_units_forced())
                       ? 0u
                       : qwcu_attn_sm100_tail_units(p.total_units,
                                                    (uint32_t)sm_count_of_current_device());
    const unsigned grid = p.total_units + p.tail_units;
    rc = launch(kernel, grid, kThreads, kSmemBytes, 1, stream, map_q, map_k, map_v, p);
#ifdef QW_ATTN_TRACE
    if (p.trace && !rc) trace_dump(stream);
#endif
    return rc;
}
