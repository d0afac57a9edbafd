// bf16 linear layers of the DiT block on the tensor cores of sm_100a:
//   C[M, N] = A[M, K] * W[N, K]^T (+ bias), fp32 accumulate, one rounding to bf16
// (reference h3_gpu_linear_bf16: h3_gpu.m:2697-2812, h3_shaders.metal:788-822), and
// the fused q/k/v projection, three such products sharing A in one launch
// (reference qw_gpu_qkv_bf16: h3_gpu.m:2918-3018, called qwen_dit.m:1270).  The
// weights keep the checkpoint's [out, in] layout, which is the K-major B operand.
//
// Persistent CTAs.  Large problems run on CTA pairs (tcgen05 cta_group::2): a pair owns
// a 256 (M) x 256 (N) tile, each CTA holds 128 rows of A and half of the W rows, so a
// K step of 64 costs a CTA 32 KB of shared memory instead of 48 KB and the tensor
// cores read each W row once per pair.  Problems that do not fill the pairs take pairs of
// 128 columns or, where the CTAs of one wave do what pairs need two for, single CTAs of
// 128 (M) x 256 (N) (choose() below).
//   warp 0     : TMA producer  (128B-swizzled boxes of 64 columns)
//   warp 1     : MMA issuer    (of the pair's first CTA)
//   warps 2..9 : epilogue      (TMEM -> registers -> bf16 -> a staging box of 32 rows x
//                               64 columns per warp -> TMA store; a warp waits for
//                               nobody but its own last store)
// Two TMEM accumulators let the epilogue of tile i run under the main loop of i + 1.
//
// Optional fused epilogue (q and k of the DiT block): a thread owns one row of a head
// of 128 columns, so the per-head RMSNorm needs no exchange between threads and
// follows the reference's serial fma order exactly; the interleaved RoPE follows with
// the rows' cos/sin.  The bf16 roundings the reference has between its three kernels
// are reproduced, which makes the result the same as GEMM -> h3_gpu_head_rms_norm_bf16
// -> qw_gpu_qk_rope_bf16 without the two extra passes over q and k.
//
// Where a CTA has one tile, nothing hides its epilogue, and most of that was latency: of
// cos/sin, which every thread read for its own row (32 lines a load, twice what L1 holds),
// and of code that each launch reads anew.  So the rotation runs on the staged box, where
// eight lanes share a row's line and the loads are issued under the main loop, the
// loops are rolled (a row's columns are read from TMEM twice instead of being held), and the
// last tile's second box is staged in the ring instead of waiting for the first one's store.
// 320 rows of 3072, clocks from complete accumulator to stores issued: 12700 -> 3700; chains of
// four layers, 256^2 279 -> 262 us, 512^2 477 -> 460 us.
//
// Every wait is bounded (status words, abort flag).  A CTA leaves nothing in flight, also
// after a wait has run out: see the end of the kernel.

#include <string.h>

#include "qw_sm100.cuh"

namespace {

using namespace sm100;

constexpr int kTileK = 64;                   // one 128-byte swizzle row of bf16
constexpr int kRows = 128;                   // rows of a CTA's accumulator (TMEM lanes)
constexpr int kABytes = kRows * kTileK * 2;  // 16 KB
constexpr int kBoxBytes = 64 * kTileK * 2;   // 8 KB, 64 rows of W
constexpr int kEpilogueWarps = 8;
constexpr int kThreads = 64 + kEpilogueWarps * 32;
constexpr int kStoreBytes = 32 * 128;  // a warp's staging box: 32 rows x 64 columns
constexpr int kMaxSmem = 227 * 1024;
constexpr int kMaxStages = 8;
constexpr int kMaxOutputs = 3;
constexpr int kBand = 2048;  // rows of A whose tiles run side by side (L2 reuse of W)

enum Barrier : int {
    kBarFull = 0,                          // stage landed (in both CTAs of a pair)
    kBarEmpty = kBarFull + kMaxStages,     // stage consumed
    kBarAccFull = kBarEmpty + kMaxStages,  // 2: accumulator complete
    kBarAccEmpty = kBarAccFull + 2,        // 2: accumulator drained
    kBarCount = kBarAccEmpty + 2
};

struct __align__(16) Control {
    Mbar bars[kBarCount];
    uint32_t tmem_base;
    volatile uint32_t abort_flag;
    uint32_t issued[2];  // of the pair's CTAs: K steps loaded, kGaveUp when a wait ran out
    alignas(16) float norm_w[2][128];
};
constexpr uint32_t kGaveUp = 0x80000000u;

template <int kGroup, int kN>
struct Config {
    static constexpr int kBBytes = kN / kGroup * kTileK * 2;  // a CTA's share of W
    static constexpr int kStageBytes = kABytes + kBBytes;
    static constexpr int kFixed = kEpilogueWarps * kStoreBytes + (int)sizeof(Control) + 1024;
    static constexpr int kFit = (kMaxSmem - kFixed) / kStageBytes;
    static constexpr int kStages = kFit < kMaxStages ? kFit : kMaxStages;
    static constexpr int kSmem = kFixed + kStages * kStageBytes;
    static constexpr uint32_t kTmemCols = 2 * kN;
    static_assert(kStages >= 3, "too few stages");
};

struct Params {
    uint32_t m, k;
    uint32_t n_each;             // columns of every output
    uint32_t tiles_per_output;   // ceil(n_each / kN)
    uint32_t m_tiles, n_tiles;   // n_tiles over all outputs
    uint32_t n_outputs;
    uint32_t band;               // M tiles that run side by side
    uint32_t whole, items;       // items [0, whole) are tiles, the rest half tiles (kN / 2 columns)
    const uint16_t *bias[kMaxOutputs];  // bf16 [n_each] or null
    uint32_t *status;
    // Optional fused epilogue for outputs 0 and 1 (q and k of the DiT block): per-head
    // RMSNorm over 128 columns and interleaved RoPE, with the reference's bf16
    // roundings between the stages (GEMM result -> bf16 -> norm -> bf16 -> rotation).
    const uint16_t *norm_weight[2];    // bf16 [128] each, null = plain output
    const float *rope_cos, *rope_sin;  // f32 [table_rows][64]
    uint32_t table_rows, table_step;   // table row = output row % table_rows; 4 % table_rows
    float epsilon;
    float *bound_out;  // optional: [0], [1] = bounds of the 2-norm of any q row, k row
    // Bounded-wait exercise (tests only): budget in SM cycles, and the K step (counted over
    // its items) from which a CTA of the pair loads nothing.
    long long wait_cycles;
    uint32_t withhold_from[2];
};

struct Maps {
    CUtensorMap a;
    CUtensorMap w[kMaxOutputs];
    CUtensorMap c[kMaxOutputs];
};

struct Item {
    uint32_t tm;     // M tile
    uint32_t which;  // output
    uint32_t col0;   // first column of the output
    uint32_t cols;   // kN, or half of it
};

// Tiles in bands of `band` M tiles, M fastest: the CTAs running side by side cover a
// block of the output about as high as it is wide, so they share A and W through L2.
template <int kN>
__device__ __forceinline__ Item item_at(const Params &p, uint32_t i) {
    Item it;
    uint32_t half = 0, tile = i;
    it.cols = kN;
    if (i >= p.whole) {
        half = (i - p.whole) & 1u;
        tile = p.whole + ((i - p.whole) >> 1);
        it.cols = kN / 2;
    }
    const uint32_t per_band = p.band * p.n_tiles;
    const uint32_t b = tile / per_band, rest = tile - b * per_band;
    const uint32_t height = min(p.band, p.m_tiles - b * p.band);
    const uint32_t tn = rest / height;
    it.tm = b * p.band + (rest - tn * height);
    it.which = tn / p.tiles_per_output;
    it.col0 = (tn - it.which * p.tiles_per_output) * kN + half * (kN / 2);
    return it;
}

// How many of a warp's `boxes` (64 columns each, the first from column col0 on) hold columns of
// an output of n: the last tile may reach past it, with a box or with both.
__host__ __device__ constexpr int boxes_inside(int boxes, uint32_t col0, uint32_t n) {
    return col0 >= n ? 0 : boxes == 2 && col0 + 64u >= n ? 1 : boxes;
}
static_assert(boxes_inside(2, 2688, 2688) == 0 && boxes_inside(2, 2752, 2688) == 0 &&
                  boxes_inside(2, 2624, 2688) == 1 && boxes_inside(2, 2560, 2688) == 2 &&
                  boxes_inside(2, 2560, 2632) == 2 && boxes_inside(1, 2624, 2688) == 1 &&
                  boxes_inside(1, 2688, 2688) == 0 && boxes_inside(0, 0, 2688) == 0,
              "a warp's boxes at the end of an output");

// 32 columns of one row out of the accumulator, as packed bf16 pairs: the GEMM result
// (plus bias) rounded to bf16.
__device__ __forceinline__ void row_from_tmem(uint32_t (&pk)[16], uint32_t taddr, const uint16_t *bias,
                                              uint32_t bias_cols) {
    uint32_t o[32];
    tmem_ld32(o, taddr);
    tmem_wait_ld32(o);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        float lo = __uint_as_float(o[2 * i]), hi = __uint_as_float(o[2 * i + 1]);
        if (bias && (uint32_t)(2 * i) < bias_cols) {  // (column counts are even)
            const uint32_t b2 = *reinterpret_cast<const uint32_t *>(bias + 2 * i);
            lo = __fadd_rn(lo, bf16_lo(b2));
            hi = __fadd_rn(hi, bf16_hi(b2));
        }
        pk[i] = pack_bf16(lo, hi);
    }
}

template <int kGroup, int kN>
__global__ void __launch_bounds__(kThreads, 1)
qw_linear_sm100_kernel(const __grid_constant__ Maps maps, const Params p) {
    using C = Config<kGroup, kN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *ring = reinterpret_cast<uint8_t *>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *staging = ring + C::kStages * C::kStageBytes;
    Control *ctl = reinterpret_cast<Control *>(staging + kEpilogueWarps * kStoreBytes);
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const uint32_t rank = kGroup == 2 ? cluster_rank() : 0u;
    const uint32_t first = blockIdx.x / kGroup, step = gridDim.x / kGroup;
    const uint32_t k_steps = (p.k + kTileK - 1) / kTileK;
    const Waiter wait = {&ctl->abort_flag, p.status, p.wait_cycles};

    if (threadIdx.x == 0) {
        for (int i = 0; i < C::kStages; ++i) {
            mbar_init(&ctl->bars[kBarFull + i], 1);
            mbar_init(&ctl->bars[kBarEmpty + i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&ctl->bars[kBarAccFull + i], 1);
            mbar_init(&ctl->bars[kBarAccEmpty + i], kEpilogueWarps * kGroup);
        }
        ctl->abort_flag = 0;
        mbar_init_fence();
    }
    // (parameters, not memory that a kernel before this one writes)
    if (warp == 2) {
        if (lane == 0) tma_prefetch(&maps.a);
        else if ((uint32_t)lane <= p.n_outputs) tma_prefetch(&maps.w[lane - 1]);
        else if ((uint32_t)lane <= 2 * p.n_outputs) tma_prefetch(&maps.c[lane - 1 - p.n_outputs]);
    }
    // The producer may start as soon as the barriers exist, the peer's too, to which it
    // reports; the others wait for TMEM as well.
    __syncwarp();
    if constexpr (kGroup == 2) cluster_sync();
    else __syncthreads();
    uint32_t tmem = 0;
    if (warp != 0) {
        if (warp == 1) tmem_alloc<kGroup>(&ctl->tmem_base, C::kTmemCols);
        tc_fence_before();
        asm volatile("bar.sync 2, %0;" ::"n"(kThreads - 32) : "memory");
        tc_fence_after();
        tmem = ctl->tmem_base;
    }
    grid_launch_dependents();
    grid_wait();

    // This CTA's loads of K step ks of an item, the t-th step it loads: its rows of A and
    // its share of the W rows.
    const auto load_step = [&](const Item &it, uint32_t ks, uint32_t t) {
        const uint32_t slot = t % C::kStages, share = it.cols / kGroup;  // (in boxes of 64)
        const int a_row = (int)((it.tm * kGroup + rank) * kRows);
        const int w_row = (int)(it.col0 + rank * share);
        Mbar *bar = &ctl->bars[kBarFull + slot];
        const uint32_t bar_at = kGroup == 2 ? map_to_rank(bar, 0) : smem_u32(bar);
        uint8_t *dst = ring + slot * C::kStageBytes;
        const int k0 = (int)(ks * kTileK);
        if (elect_one()) {
            if (rank == 0) mbar_expect_tx(bar, (kABytes + share * (kTileK * 2)) * kGroup);
            tma_load_2d<kGroup>(dst, &maps.a, bar_at, k0, a_row);
#pragma unroll
            for (int box = 0; box < C::kBBytes / kBoxBytes; ++box)
                if ((uint32_t)box * 64u < share)
                    tma_load_2d<kGroup>(dst + kABytes + box * kBoxBytes, &maps.w[it.which], bar_at, k0,
                                        w_row + box * 64);
        }
        __syncwarp();
    };

    if (warp == 0) {
        // ---- producer
        uint32_t t = 0;
        bool ok = true;
        for (uint32_t i = first; i < p.items && ok; i += step) {
            const Item it = item_at<kN>(p, i);
            for (uint32_t ks = 0; ks < k_steps; ++ks, ++t) {
                const uint32_t slot = t % C::kStages, par = ((t / C::kStages) & 1u) ^ 1u;
                ok = t < p.withhold_from[rank] &&
                     mbar_wait_warp(wait, &ctl->bars[kBarEmpty + slot], par, (3u << 16) | slot, i);
                if (!ok) break;
                load_step(it, ks, t);
            }
        }
        // Wait until the last steps are consumed: then their loads (the peer's too) have
        // landed and the commits that report here, those of the pair's first CTA among
        // them, have arrived.
        for (uint32_t u = t > (uint32_t)C::kStages ? t - C::kStages : 0; u < t && ok; ++u)
            ok = mbar_wait_warp(wait, &ctl->bars[kBarEmpty + u % C::kStages], (u / C::kStages) & 1u,
                                (3u << 16) | (u % C::kStages), p.items);
        if (lane < kGroup) {
            const uint32_t word = ok ? t : t | kGaveUp;
            if constexpr (kGroup == 2) st_at(map_to_rank(&ctl->issued[rank], (uint32_t)lane), word);
            else ctl->issued[0] = word;
        }
    } else if (warp == 1 && rank == 0) {
        // ---- MMA issuer (for both CTAs of a pair)
        uint32_t t = 0, local = 0;
        const uint32_t ring_lo = (smem_u32(ring) >> 4) | kDescKMajor;
        constexpr uint32_t idesc_whole = instr_desc(kRows * kGroup, kN, false);
        constexpr uint32_t idesc_half = instr_desc(kRows * kGroup, kN / 2, false);
        for (uint32_t i = first; i < p.items; i += step, ++local) {
            const uint32_t acc = local & 1u;
            // the epilogue must have drained this accumulator (used two tiles ago)
            if (local >= 2 &&
                !mbar_wait_warp(wait, &ctl->bars[kBarAccEmpty + acc], ((local >> 1) - 1u) & 1u,
                                (2u << 16) | (kBarAccEmpty + acc), i))
                break;
            tc_fence_after();
            const uint32_t d_tmem = tmem + acc * kN;
            const uint32_t idesc = i < p.whole ? idesc_whole : idesc_half;
            bool ok = true;
            for (uint32_t ks = 0; ks < k_steps; ++ks, ++t) {
                const uint32_t slot = t % C::kStages, par = (t / C::kStages) & 1u;
                ok = mbar_wait_warp(wait, &ctl->bars[kBarFull + slot], par, (2u << 16) | slot, i);
                if (!ok) break;
                tc_fence_after();
                const uint32_t a_lo = ring_lo + slot * (uint32_t)(C::kStageBytes >> 4);
                const uint32_t b_lo = a_lo + (kABytes >> 4);
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        mma_ss<kGroup>(d_tmem, a_lo + (uint32_t)(kk * 32 >> 4),
                                       b_lo + (uint32_t)(kk * 32 >> 4), idesc, (ks | kk) ? 1u : 0u);
                    tc_commit<kGroup>(&ctl->bars[kBarEmpty + slot]);
                    if (ks + 1 == k_steps) tc_commit<kGroup>(&ctl->bars[kBarAccFull + acc]);
                }
                __syncwarp();
            }
            if (!ok) break;
        }
        // Nothing that was issued runs on into the release of TMEM and shared memory (all of
        // it is done already, unless a wait has run out).
        if (t) mbar_drain(&ctl->bars[kBarEmpty + (t - 1) % C::kStages], ((t - 1) / C::kStages) & 1u, p.wait_cycles);
    } else if (warp >= 2) {
        // ---- epilogue: warp w reads TMEM lanes 32 * (w % 4) ..., thread = one row; the
        // warps of the second group take the second half of a wide tile's columns
        const int ew = warp - 2, group = ew >> 2;
        const uint32_t quarter = (uint32_t)(warp & 3);
        const uint32_t lanes = tmem + ((quarter * 32u) << 16);
        uint8_t *stage = staging + ew * kStoreBytes;
        const uint32_t sw = (uint32_t)lane & 7u;
        if (p.norm_weight[0] || p.norm_weight[1]) {
            // norm weights of q and k as floats, shared by all rows
            const int t = threadIdx.x - 64;
            const uint16_t *w = p.norm_weight[t >> 7];
            ctl->norm_w[t >> 7][t & 127] = w ? __uint_as_float((uint32_t)w[t & 127] << 16) : 0.0f;
            asm volatile("bar.sync 1, %0;" ::"n"(kEpilogueWarps * 32) : "memory");
            if (blockIdx.x == 0 && warp == 2 && p.bound_out) {
                // A normalised head has sum (x*inv)^2 <= 128, so after the weight its
                // 2-norm is at most sqrt(128) * max|w|; the rotation preserves it and
                // the two bf16 roundings add well under 1 %.
                for (int which = 0; which < 2; ++which) {
                    float wmax = 0.0f;
                    for (int i = lane; i < 128; i += 32) wmax = fmaxf(wmax, fabsf(ctl->norm_w[which][i]));
#pragma unroll
                    for (int off = 16; off > 0; off >>= 1)
                        wmax = fmaxf(wmax, __shfl_xor_sync(0xffffffffu, wmax, off));
                    if (lane == 0) p.bound_out[which] = 11.313708499f * 1.01f * wmax;
                }
            }
        }
        uint32_t local = 0;
        for (uint32_t i = first; i < p.items; i += step, ++local) {
            const Item it = item_at<kN>(p, i);
            const uint32_t acc = local & 1u;
            const bool fused = it.which < 2 && p.norm_weight[it.which] != nullptr;
            // columns of this warp: 128 of a 256-column tile; a narrower one is shared out
            // in boxes of 64, except that a head to be normalised stays in one thread
            const bool wide = it.cols == 256 || (fused && it.cols == 128);
            const uint32_t off = (uint32_t)group * (wide ? 128u : 64u);
            const uint32_t col0 = it.col0 + off;
            const uint32_t row0 = (it.tm * kGroup + rank) * kRows + quarter * 32u;
            // The second box of a CTA's last tile is staged in the ring, which is done with.
            uint8_t *const spare = i + step < p.items ? stage : ring + ew * kStoreBytes;
            const int boxes = off >= it.cols || row0 >= p.m ? 0 : wide ? 2 : 1;
            const int live = boxes_inside(boxes, col0, p.n_each);
            // The rotation's entries of a box: lane l takes four pairs (16 bytes of cos and of
            // sin) of rows l / 8, l / 8 + 4, ..., so that a load touches four rows' lines and not
            // 32.  The first box's are on their way while the accumulator is still filling.
            float4 cs[8], sn[8];
            uint32_t table_row = 0;
            const auto load_table = [&](int i, int box) {
                const size_t at =
                    (size_t)(row0 + 4u * i + ((uint32_t)lane >> 3) < p.m ? table_row : 0u) * 64 + box * 32 +
                    4 * (lane & 7);
                cs[i] = __ldg(reinterpret_cast<const float4 *>(p.rope_cos + at));
                sn[i] = __ldg(reinterpret_cast<const float4 *>(p.rope_sin + at));
                table_row += p.table_step;
                if (table_row >= p.table_rows) table_row -= p.table_rows;
            };
            if (fused && live) {
                table_row = (row0 + ((uint32_t)lane >> 3)) % p.table_rows;
#pragma unroll
                for (int i = 0; i < 8; ++i) load_table(i, 0);
            }
            if (!mbar_wait_warp(wait, &ctl->bars[kBarAccFull + acc], (local >> 1) & 1u,
                                (1u << 16) | (kBarAccFull + acc), i))
                break;
            tc_fence_after();
            const uint32_t src = lanes + acc * kN + off;
            const uint16_t *bias = live && p.bias[it.which] ? p.bias[it.which] + col0 : nullptr;
            float inverse = 0.0f;
            if (fused && live) {  // serial fma over the bf16 values, element order 0..127
                float ss = 0.0f;
#pragma unroll 1
                for (int c = 0; c < 4; ++c) {
                    uint32_t pk[16];
                    row_from_tmem(pk, src + (uint32_t)(c * 32), bias ? bias + c * 32 : nullptr, 32);
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        ss = fmaf(bf16_lo(pk[j]), bf16_lo(pk[j]), ss);
                        ss = fmaf(bf16_hi(pk[j]), bf16_hi(pk[j]), ss);
                    }
                }
                inverse = 1.0f / sqrtf(__fadd_rn(ss / 128.0f, p.epsilon));
            }
#pragma unroll 1
            for (int box = 0; box < live; ++box) {
                uint8_t *const staged = box ? spare : stage;
                if (staged == stage) {
                    if (lane == 0) tma_store_wait_read<0>();
                    __syncwarp();
                }
#pragma unroll 1
                for (int half = 0; half < 2; ++half) {
                    const uint32_t at = (uint32_t)(box * 64 + half * 32);
                    uint32_t pk[16];
                    row_from_tmem(pk, src + at, bias ? bias + at : nullptr,
                                  col0 + at < p.n_each ? p.n_each - col0 - at : 0u);
                    if (fused) {  // bf16(x * inv * w), stored as bf16 between norm and rotation
                        const float4 *w4 = reinterpret_cast<const float4 *>(&ctl->norm_w[it.which][at]);
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float4 w = w4[j];
                            pk[2 * j] = pack_bf16(__fmul_rn(__fmul_rn(bf16_lo(pk[2 * j]), inverse), w.x),
                                                  __fmul_rn(__fmul_rn(bf16_hi(pk[2 * j]), inverse), w.y));
                            pk[2 * j + 1] =
                                pack_bf16(__fmul_rn(__fmul_rn(bf16_lo(pk[2 * j + 1]), inverse), w.z),
                                          __fmul_rn(__fmul_rn(bf16_hi(pk[2 * j + 1]), inverse), w.w));
                        }
                    }
#pragma unroll
                    for (int c16 = 0; c16 < 4; ++c16)
                        *reinterpret_cast<uint4 *>(staged + lane * 128 +
                                                   (((uint32_t)(half * 4 + c16) ^ sw) << 4)) =
                            make_uint4(pk[4 * c16], pk[4 * c16 + 1], pk[4 * c16 + 2], pk[4 * c16 + 3]);
                }
                if (fused) {
                    // The rotation, in place: a lane has the pairs its table entries are for.
                    __syncwarp();
                    if (box == 0 && live == 2) table_row = (row0 + ((uint32_t)lane >> 3)) % p.table_rows;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const uint32_t r = 4u * i + ((uint32_t)lane >> 3);
                        uint4 *at = reinterpret_cast<uint4 *>(
                            staged + r * 128 + ((((uint32_t)lane & 7u) ^ (r & 7u)) << 4));
                        const uint4 x = *at;
                        const uint32_t n[4] = {x.x, x.y, x.z, x.w};
                        const float cc[4] = {cs[i].x, cs[i].y, cs[i].z, cs[i].w};
                        const float ss[4] = {sn[i].x, sn[i].y, sn[i].z, sn[i].w};
                        uint32_t y[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const float e = bf16_lo(n[j]), o = bf16_hi(n[j]);
                            y[j] = pack_bf16(__fsub_rn(__fmul_rn(e, cc[j]), __fmul_rn(o, ss[j])),
                                             __fadd_rn(__fmul_rn(e, ss[j]), __fmul_rn(o, cc[j])));
                        }
                        *at = make_uint4(y[0], y[1], y[2], y[3]);
                        if (box + 1 < live) load_table(i, box + 1);
                    }
                }
                fence_async_shared();
                __syncwarp();
                if (lane == 0) {
                    tma_store_2d(&maps.c[it.which], staged, (int)(col0 + box * 64), (int)row0);
                    tma_store_commit();
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {  // this warp's part of the accumulator has left TMEM
                if constexpr (kGroup == 2) mbar_arrive_at(map_to_rank(&ctl->bars[kBarAccEmpty + acc], 0));
                else mbar_arrive(&ctl->bars[kBarAccEmpty + acc]);
            }
        }
        if (lane == 0) tma_store_wait_read<0>();
    }
    const auto sync_all = [&]() {
        tc_fence_before();
        __syncwarp();
        if constexpr (kGroup == 2) cluster_sync();
        else __syncthreads();
        tc_fence_after();
    };
    sync_all();
    if ((ctl->issued[0] | (kGroup == 2 ? ctl->issued[1] : 0u)) & kGaveUp) {
        // A wait has run out somewhere, and loads may be in flight.  Only the first CTA's
        // barriers count them, both CTAs' bytes of a step together, so the CTA that got less
        // far loads the steps it is behind (their slots are free: the other one has seen
        // them consumed) and the first CTA waits for the last step of every slot.
        const uint32_t t0 = ctl->issued[0] & ~kGaveUp;
        const uint32_t t1 = kGroup == 2 ? ctl->issued[1] & ~kGaveUp : t0, most = max(t0, t1);
        if (warp == 0) {
            for (uint32_t t = rank ? t1 : t0; t < most; ++t)
                load_step(item_at<kN>(p, first + t / k_steps * step), t % k_steps, t);
            if (rank == 0)
                for (uint32_t t = most > (uint32_t)C::kStages ? most - C::kStages : 0; t < most; ++t)
                    mbar_drain(&ctl->bars[kBarFull + t % C::kStages], (t / C::kStages) & 1u, p.wait_cycles);
        }
        sync_all();
    }
    if (warp == 1) tmem_dealloc<kGroup>(tmem, C::kTmemCols);
}

typedef void (*LinearKernel)(const Maps, const Params);

struct Variant {
    LinearKernel kernel;
    int group, n, smem;
    // Measured nanoseconds of one K step of 64 on a tile, and of one on a half tile.  The
    // 256-column pair is bound by the tensor cores, the others by the 70 bytes a clock
    // that L2 delivers to an SM (24 KB a step for 128 columns, 48 KB on a single CTA).  A half
    // tile moves what a 128-column pair does through a shorter ring: 12288 x 3072 columns at
    // 128 rows 46.5 us as halves, 40.8 us as 128-column tiles, 4096 x 4096 at 64 rows 20.1 and
    // 17.3 us, so halves are for a last wave behind whole tiles only.
    int step_ns, half_ns;
};

const Variant kVariants[] = {
    {qw_linear_sm100_kernel<2, 256>, 2, 256, Config<2, 256>::kSmem, 250, 240},
    {qw_linear_sm100_kernel<2, 128>, 2, 128, Config<2, 128>::kSmem, 215, 0},
    {qw_linear_sm100_kernel<1, 256>, 1, 256, Config<1, 256>::kSmem, 360, 0},
};
constexpr int kVariantCount = sizeof(kVariants) / sizeof(kVariants[0]);

struct Choice {
    const Variant *v;
    uint32_t tiles_per_output, m_tiles, n_tiles, whole, items;
};

// The variant whose waves take the least time per K step.  The tiles of a last, partly
// filled wave are cut in two along N when the halves still fit one wave (256-column
// tiles of pairs only).
bool choose(Choice *best, uint32_t m, uint32_t n, uint32_t n_outputs, uint32_t sms) {
    uint64_t best_cost = 0;
    best->v = nullptr;
    for (int i = 0; i < kVariantCount; ++i) {
        const Variant *v = &kVariants[i];
        const uint64_t slots = sms / (uint32_t)v->group;
        const uint64_t m_tiles = (m + kRows * v->group - 1) / (kRows * v->group);
        const uint64_t per_output = (n + v->n - 1) / v->n, n_tiles = per_output * n_outputs;
        const uint64_t tiles = m_tiles * n_tiles;
        if (tiles > 0x3fffffffull || !slots) continue;
        const uint64_t rest = tiles % slots;
        const bool halves = v->half_ns && rest && 2 * rest <= slots;
        const uint64_t last = !rest ? 0 : (uint64_t)(halves ? v->half_ns : v->step_ns);
        const uint64_t cost = tiles / slots * (uint64_t)v->step_ns + last;
        if (best->v && cost >= best_cost) continue;
        best_cost = cost;
        *best = {v, (uint32_t)per_output, (uint32_t)m_tiles, (uint32_t)n_tiles,
                 (uint32_t)(halves ? tiles - rest : tiles), (uint32_t)(halves ? tiles + rest : tiles)};
    }
    return best->v != nullptr;
}

// The opt-in to more than 48 KB of dynamic shared memory is a per-device attribute.  The
// first launch sets it for all variants: a size that takes another one may follow inside a
// graph capture.
bool kernels_ready() {
    static bool ready[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    const bool tracked = dev >= 0 && dev < 64;
    if (tracked && ready[dev]) return true;
    for (const Variant &v : kVariants)
        if (cudaFuncSetAttribute(v.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, v.smem) !=
            cudaSuccess)
            return false;
    if (tracked) ready[dev] = true;
    return true;
}

uint32_t usable_sms(int sm_count) { return (uint32_t)(sm_count > 1 ? sm_count : 148); }

}  // namespace

extern "C" int qwcu_linear_sm100_plan(uint32_t m, uint32_t n, uint32_t n_outputs, int sm_count,
                                      qwcu_linear_plan *plan) {
    Choice choice;
    if (!m || !n || !n_outputs || !choose(&choice, m, n, n_outputs, usable_sms(sm_count)))
        return (int)cudaErrorInvalidValue;
    *plan = {(uint32_t)choice.v->group, (uint32_t)choice.v->n, choice.whole, choice.items};
    return 0;
}

extern "C" int qwcu_linear_sm100_launch(const qwcu_linear_args *a, int sm_count,
                                        qwcu_stream stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (!a->m || !a->k || !a->n || !a->n_outputs || a->n_outputs > (uint32_t)kMaxOutputs ||
        a->k % 8 || a->n % 8 || !a->a || !a->status)
        return (int)cudaErrorInvalidValue;
    const bool fused = a->norm_weight[0] || a->norm_weight[1];
    if (fused && (a->n % 128 || !a->rope_cos || !a->rope_sin || !a->table_rows))
        return (int)cudaErrorInvalidValue;
    if (a->bound_out && !(a->norm_weight[0] && a->norm_weight[1])) return (int)cudaErrorInvalidValue;
    const uint32_t sms = usable_sms(sm_count);
    Choice choice;
    if (!choose(&choice, a->m, a->n, a->n_outputs, sms)) return (int)cudaErrorInvalidValue;
    const Variant *v = choice.v;
    if (!kernels_ready()) return (int)cudaGetLastError();
    Maps maps;
    memset(&maps, 0, sizeof(maps));
    int rc;
    if (((uintptr_t)a->a & 15u)) return (int)cudaErrorMisalignedAddress;
    if ((rc = make_map_2d(&maps.a, a->a, a->m, a->k, kRows))) return rc;
    Params p;
    memset(&p, 0, sizeof(p));
    for (uint32_t i = 0; i < a->n_outputs; ++i) {
        if (!a->w[i] || !a->c[i]) return (int)cudaErrorInvalidValue;
        if (((uintptr_t)a->w[i] | (uintptr_t)a->c[i]) & 15u) return (int)cudaErrorMisalignedAddress;
        if ((rc = make_map_2d(&maps.w[i], a->w[i], a->n, a->k, 64))) return rc;
        if ((rc = make_map_2d(&maps.c[i], a->c[i], a->m, a->n, 32))) return rc;
        p.bias[i] = static_cast<const uint16_t *>(a->bias[i]);
    }
    p.m = a->m;
    p.k = a->k;
    p.n_each = a->n;
    p.n_outputs = a->n_outputs;
    p.tiles_per_output = choice.tiles_per_output;
    p.m_tiles = choice.m_tiles;
    p.n_tiles = choice.n_tiles;
    p.band = (uint32_t)(kBand / (kRows * v->group));
    p.whole = choice.whole;
    p.items = choice.items;
    p.status = a->status;
    p.norm_weight[0] = static_cast<const uint16_t *>(a->norm_weight[0]);
    p.norm_weight[1] = static_cast<const uint16_t *>(a->norm_weight[1]);
    p.rope_cos = a->rope_cos;
    p.rope_sin = a->rope_sin;
    p.table_rows = a->table_rows ? a->table_rows : 1;
    p.table_step = 4u % p.table_rows;
    p.epsilon = a->epsilon;
    p.bound_out = a->bound_out;
    p.wait_cycles = a->wait_cycles > 0 ? a->wait_cycles : kWaitCycles;
    for (int r = 0; r < 2; ++r) p.withhold_from[r] = a->withhold_from[r] ? a->withhold_from[r] : UINT32_MAX;
    const uint32_t slots = sms / (uint32_t)v->group;
    const uint32_t clusters = choice.items < slots ? choice.items : slots;
    return launch(v->kernel, clusters * (uint32_t)v->group, kThreads, (size_t)v->smem, v->group, stream,
                  maps, p);
}
