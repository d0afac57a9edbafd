// The sm_100a instructions the tensor-core kernels share: mbarriers (also a peer
// CTA's of the cluster), TMA tile loads and stores, tcgen05 MMA / TMEM, for one CTA
// (cta_group::1) and for a pair (cta_group::2).
#ifndef QW_SM100_CUH
#define QW_SM100_CUH

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../qw_cuda.h"

namespace sm100 {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// The warp's index as a value the compiler knows to be the same in all lanes, and one
// lane of a converged warp.  The issuing warps run their loops with all lanes and elect
// one only around the instruction itself: descriptors and coordinates then live in
// uniform registers.  (Inside a one-lane branch every operand of every MMA is moved
// there first: 140 clocks per MMA instead of the 32 to 128 it executes in.)
__device__ __forceinline__ int warp_index() {
    return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
}
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile(
        "{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(pred));
    return pred != 0;
}

// ---- programmatic dependent launch ------------------------------------------
// A kernel launched with launch() below may start (barriers, TMEM, descriptors) under the
// tail of the one before it; it waits for that one's results before it touches global
// memory.
__device__ __forceinline__ void grid_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void grid_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ---- mbarriers ----------------------------------------------------------------
typedef unsigned long long Mbar;

__device__ __forceinline__ void mbar_init(Mbar *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_init_fence() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// (By pointer or by shared address: a loop that keeps the address of its barriers as one word
// saves the conversion at each of them.)
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive(Mbar *bar) { mbar_arrive(smem_u32(bar)); }
__device__ __forceinline__ void mbar_expect_tx(Mbar *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
// (The arrivals may come from the peer CTA: what they order is TMEM and TMA traffic,
// which carries fences of its own.)
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ bool mbar_try(Mbar *bar, uint32_t parity) {
    return mbar_try(smem_u32(bar), parity);
}

// ---- cluster --------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// Address of this CTA's shared variable as CTA `rank` of the cluster has it.
__device__ __forceinline__ uint32_t map_to_rank(const void *p, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_at(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr)
                 : "memory");
}
__device__ __forceinline__ void st_at(uint32_t cluster_addr, uint32_t value) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(value) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// ---- TMA ------------------------------------------------------------------------
// The barrier is a shared::cluster address: with cta_group::2 a CTA's load may report
// to the pair's leader.
template <int kGroup>
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, uint32_t bar, int c0,
                                            int c1) {
    if constexpr (kGroup == 2)
        asm volatile(
            "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile."
            "mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
            "l"(map), "r"(bar), "r"(c0), "r"(c1)
            : "memory");
    else
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
            "[%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
            "l"(map), "r"(bar), "r"(c0), "r"(c1)
            : "memory");
}
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, Mbar *bar, int c0, int c1,
                                            int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap *map, const void *src, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map),
        "r"(smem_u32(src)), "r"(c0), "r"(c1)
        : "memory");
}
__device__ __forceinline__ void tma_store_commit() {
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// Until at most kPending committed stores have still to read their shared memory.
template <int kPending>
__device__ __forceinline__ void tma_store_wait_read() {
    asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(kPending) : "memory");
}
__device__ __forceinline__ void tma_prefetch(const CUtensorMap *map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}
__device__ __forceinline__ void st_shared16(uint32_t at, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(a), "r"(b), "r"(c), "r"(d)
                 : "memory");
}
__device__ __forceinline__ uint4 ld_shared16(uint32_t at) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(at)
                 : "memory");
    return v;
}
__device__ __forceinline__ void fence_async_shared() {  // generic writes -> TMA reads
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---- tcgen05 --------------------------------------------------------------------
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
template <int kGroup>
__device__ __forceinline__ void tmem_alloc(uint32_t *slot, uint32_t cols) {
    if constexpr (kGroup == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(slot)),
                     "r"(cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(slot)),
                     "r"(cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
}
template <int kGroup>
__device__ __forceinline__ void tmem_dealloc(uint32_t tmem, uint32_t cols) {
    if constexpr (kGroup == 2)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols)
                     : "memory");
    else
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols)
                     : "memory");
}
// The barrier is signalled when every MMA issued so far by this thread is done; for a
// pair the same barrier of both CTAs.
template <int kGroup>
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    if constexpr (kGroup == 2)
        asm volatile(
            "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 "
            "[%0], %1;" ::"r"(bar),
            "h"((unsigned short)3)
            : "memory");
    else
        asm volatile(
            "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
            : "memory");
}
template <int kGroup>
__device__ __forceinline__ void tc_commit(Mbar *bar) {
    tc_commit<kGroup>(smem_u32(bar));
}

// Shared-memory matrix descriptor as two words: start address >> 4 in bits 0-13,
// leading byte offset >> 4 in bits 16-29 (low word), stride byte offset >> 4 in bits
// 0-13, version 1 in bit 14, 128B swizzle = 2 in bits 29-31 (high word).  Stepping
// through a tile only changes the start address, one add on the issuing thread.
__host__ __device__ constexpr uint32_t desc_hi(uint32_t sbo_bytes) {
    return ((sbo_bytes >> 4) & 0x3FFFu) | (1u << 14) | (2u << 29);
}
__host__ __device__ constexpr uint32_t desc_lo(uint32_t lbo_bytes) { return ((lbo_bytes >> 4) & 0x3FFFu) << 16; }
constexpr uint32_t kDescHi = desc_hi(1024);  // 8 rows of 128 bytes
constexpr uint32_t kDescKMajor = desc_lo(16);  // (LBO is unused: one swizzle row wide)

// Instruction descriptor, kind::f16: bf16 x bf16 -> fp32, A K-major.
__host__ __device__ constexpr uint32_t instr_desc(uint32_t m, uint32_t n, bool b_mn_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn_major ? 1u : 0u) << 16) | ((n >> 3) << 17) |
           ((m >> 4) << 24);
}

template <int kGroup>
__device__ __forceinline__ void mma_ss(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                       uint32_t accumulate) {
    if constexpr (kGroup == 2)
        asm volatile(
            "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
            "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\tsetp.ne.b32 p, %5, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %4, p;\n\t}" ::"r"(d_tmem),
            "r"(a_lo), "r"(b_lo), "r"(kDescHi), "r"(idesc), "r"(accumulate)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
            "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\tsetp.ne.b32 p, %5, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}" ::"r"(d_tmem),
            "r"(a_lo), "r"(b_lo), "r"(kDescHi), "r"(idesc), "r"(accumulate)
            : "memory");
}
// A from TMEM.
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc,
                                       uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
        "mov.b64 db, {%2, %3};\n\tsetp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "r"(b_lo), "r"(kDescHi), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t (&r)[32], uint32_t taddr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
// tcgen05.wait::ld that names the registers of an earlier load as read-write operands:
// no use of them can be scheduled ahead of the wait.
__device__ __forceinline__ void tmem_wait_ld32(uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.wait::ld.sync.aligned;"
        : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
          "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]),
          "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]),
          "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]),
          "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
        :
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// ---- arithmetic -------------------------------------------------------------------
__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// ---- bounded waits ------------------------------------------------------------------
// A wait that runs out records where in the status words and raises the CTA's abort
// flag, which the other waits of the CTA poll (the attention's MMA warp counts probes
// instead); the roles then leave in order.
constexpr long long kWaitCycles = 400000000LL;  // about 0.2 s; a healthy wait is microseconds

struct Waiter {
    volatile uint32_t *abort_flag;  // shared memory
    uint32_t *status;
    long long budget;
};

static __device__ __noinline__ bool mbar_wait_slow(const Waiter w, Mbar *bar, uint32_t parity,
                                                   uint32_t where, uint32_t tile) {
    const long long start = clock64();
    for (;;) {
        for (int i = 0; i < 32; ++i)
            if (mbar_try(bar, parity)) return true;
        if (*w.abort_flag) return false;
        if (clock64() - start > w.budget) {
            *w.abort_flag = 1;
            if (atomicCAS(w.status, 0u, (uint32_t)QWCU_STATUS_WAIT_TIMEOUT) == 0u) {
                w.status[1] = where;
                w.status[2] = tile;
                w.status[3] = blockIdx.x;
            }
            __threadfence_system();
            return false;
        }
    }
}
__device__ __forceinline__ bool mbar_wait(const Waiter &w, Mbar *bar, uint32_t parity, uint32_t where,
                                          uint32_t tile) {
    for (int i = 0; i < 4; ++i)
        if (mbar_try(bar, parity)) return true;
    return mbar_wait_slow(w, bar, parity, where, tile);
}
// The same for all lanes of a warp at once: true when every lane saw the phase complete.
__device__ __forceinline__ bool mbar_wait_warp(const Waiter &w, Mbar *bar, uint32_t parity,
                                               uint32_t where, uint32_t tile) {
    return __all_sync(0xffffffffu, mbar_wait(w, bar, parity, where, tile)) != 0;
}

// Wait without reporting, for what is in flight when the roles leave.
__device__ __forceinline__ void mbar_drain(Mbar *bar, uint32_t parity, long long budget) {
    const long long start = clock64();
    while (!mbar_try(bar, parity))
        if (clock64() - start > budget) break;
}

// ---- host: tensor maps ----------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static inline EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) ==
                cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(sym);
    }
    return fn;
}

// Dense bf16 tensor of `rank` dimensions (innermost first), boxes of 64 columns (one
// 128-byte swizzle row) x box_rows x 1; reads past an extent deliver zeros, writes past
// it are dropped.
static inline int make_map(CUtensorMap *map, const void *base, int rank, const cuuint64_t *dims,
                           const cuuint64_t *stride_bytes, uint32_t box_rows) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return (int)cudaErrorNotSupported;
    const cuuint32_t box[3] = {64, box_rows, 1}, elem[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void *>(base),
                    dims, stride_bytes, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}
static inline int make_map_2d(CUtensorMap *map, const void *base, uint32_t rows, uint32_t cols,
                              uint32_t box_rows) {
    const cuuint64_t dims[2] = {cols, rows}, strides[1] = {(cuuint64_t)cols * 2};
    return make_map(map, base, 2, dims, strides, box_rows);
}

// Launch behind the stream's last kernel with the programmatic dependency described at
// grid_wait(), in clusters of `cluster` CTAs.
template <typename... Params, typename... Args>
static inline int launch(void (*kernel)(Params...), unsigned grid, unsigned threads, size_t smem,
                         int cluster, cudaStream_t stream, const Args &...args) {
    cudaLaunchConfig_t config = {};
    cudaLaunchAttribute attrs[2];
    config.gridDim = dim3(grid);
    config.blockDim = dim3(threads);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = attrs;
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    config.numAttrs = 1;
    if (cluster > 1) {
        attrs[1].id = cudaLaunchAttributeClusterDimension;
        attrs[1].val.clusterDim.x = (unsigned)cluster;
        attrs[1].val.clusterDim.y = attrs[1].val.clusterDim.z = 1;
        config.numAttrs = 2;
    }
    const cudaError_t code = cudaLaunchKernelEx(&config, kernel, args...);
    const cudaError_t last = cudaGetLastError();
    return (int)(code != cudaSuccess ? code : last);
}

}  // namespace sm100

#endif
