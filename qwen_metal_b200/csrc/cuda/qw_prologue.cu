// Fused per-head QK RMSNorm + interleaved 3-axis RoPE (HBM-bound prologue).
//
// A head is 128 bf16 = 256 B = sixteen 16-byte vectors, so a half-warp owns one
// head at a time: one 16-byte load per lane (8 elements = 4 whole RoPE pairs), a
// 4-step shuffle reduction for the sum of squares, then the rotation, one
// 16-byte store.  Each half-warp walks all heads of one (row, tensor) strip with
// its slice of the norm weight and of the row's cos/sin held in registers, four
// heads in flight at a time.  Q and K each cross HBM exactly once in each
// direction.  The kernel was instruction-bound before it was HBM-bound, so the
// bf16 roundings use cvt.rn.bf16x2.f32 and the inverse norm uses rsqrtf.
//
// Arithmetic follows the reference's three separate kernels including the bf16
// store between norm and rotation: n = bf16(x * inv * w) (h3_shaders.metal:
// 4309-4329; bf16(bf16(x*inv)*w) for the double-rounding variant :4975-4997),
// then (e, o) <- bf16(e*c - o*s), bf16(e*s + o*c) (h3_shaders.metal:4864-4890),
// products and sums as separate fp32 operations.  The sum of squares is reduced
// as a tree and 1/sqrt is within 2 ulp, where the reference shader runs a serial
// fma chain and its own rsqrt: a normalised value differs from a serial CPU
// restatement by one bf16 step in about 1 element in 10^5.

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "qw_sm100.cuh"

namespace {

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// Round-to-nearest-even by the integer trick the reference uses on every
// path (h3_shaders.metal:15-19); NaN handling is irrelevant here.
__device__ __forceinline__ uint32_t f32_to_bf16_bits(float v) {
    uint32_t bits = __float_as_uint(v);
    bits += 0x7fffu + ((bits >> 16) & 1u);
    return bits >> 16;
}

struct Params {
    const uint4 *q_in;
    const uint4 *k_in;
    uint4 *q_out;
    uint4 *k_out;
    const uint4 *v_in;  // optional third tensor: copied as is (K/V cache update)
    uint4 *v_out;
    const uint4 *wq;
    const uint4 *wk;
    const float4 *cos_t;
    const float4 *sin_t;
    uint32_t rows, table_rows, heads;
    float eps;
    int double_round;
    uint32_t groups, group_heads;  // few strips: a row's heads in groups
    uint32_t strips;  // rows * tensors: one half-warp walks the heads of one (row, tensor)
    int tensors;
    float *bound_out;  // optional: [0], [1] = upper bounds of the 2-norm of any q row, k row
};

// Two floats -> packed bf16 pair, round to nearest even in one instruction
// (the same rounding as the integer trick for every finite value).
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// Heads a half-warp has in flight at once (independent 16-byte loads; the
// kernel is HBM-bound once the instruction count is small enough).
constexpr int kHeadsPerTrip = 4;

// One head: lane l of a half-warp holds elements [8l, 8l+8) = RoPE pairs 4l..4l+3.
__device__ __forceinline__ uint4 finish_head(const Params &p, const uint4 &x, bool norm, bool rotate,
                                             const float (&wf)[8], const float (&cc)[4],
                                             const float (&sn)[4], uint32_t half_mask) {
    float v[8] = {bf16_lo(x.x), bf16_hi(x.x), bf16_lo(x.y), bf16_hi(x.y),
                  bf16_lo(x.z), bf16_hi(x.z), bf16_lo(x.w), bf16_hi(x.w)};
    uint32_t y[4] = {x.x, x.y, x.z, x.w};
    if (norm) {
        float ss = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) ss = fmaf(v[i], v[i], ss);
#pragma unroll
        for (int off = 8; off > 0; off >>= 1)
            ss += __shfl_xor_sync(half_mask, ss, off, 16);
        // mean = ss / 128 exactly; 1/sqrt to within 2 ulp of the reference's rsqrt
        const float inv = rsqrtf(__fadd_rn(ss * 0.0078125f, p.eps));
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
            float n0 = __fmul_rn(v[i], inv), n1 = __fmul_rn(v[i + 1], inv);
            if (p.double_round) {
                const uint32_t r = pack_bf16x2(n0, n1);
                n0 = bf16_lo(r);
                n1 = bf16_hi(r);
            }
            y[i >> 1] = pack_bf16x2(__fmul_rn(n0, wf[i]), __fmul_rn(n1, wf[i + 1]));
        }
        if (rotate) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {  // the bf16 store between norm and rotation
                v[2 * i] = bf16_lo(y[i]);
                v[2 * i + 1] = bf16_hi(y[i]);
            }
        }
    }
    if (rotate) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float e = v[2 * i], o = v[2 * i + 1];
            y[i] = pack_bf16x2(__fsub_rn(__fmul_rn(e, cc[i]), __fmul_rn(o, sn[i])),
                               __fadd_rn(__fmul_rn(e, sn[i]), __fmul_rn(o, cc[i])));
        }
    }
    return make_uint4(y[0], y[1], y[2], y[3]);
}

// The bound of a normalised head's 2-norm (the first strips are row 0 of q and of k): sum
// (x*inv)^2 <= 128, so after the weight it is at most sqrt(128) * max|w|; the two bf16 roundings
// (norm, rotation) and the f32 tables add well under 1 %.  The rotation itself preserves it.
__device__ __forceinline__ void write_bound(const Params &p, uint32_t which, const float (&wf)[8],
                                            uint32_t half_mask, int lane16) {
    float wmax = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) wmax = fmaxf(wmax, fabsf(wf[i]));
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) wmax = fmaxf(wmax, __shfl_xor_sync(half_mask, wmax, off, 16));
    if (lane16 == 0) p.bound_out[which] = 11.313708499f * 1.01f * wmax;
}

// A half-warp owns one (row, tensor) strip: it keeps its 8-element slice of the
// norm weight and of the row's cos/sin in registers and walks the heads, four at
// a time.  Lane l holds elements [8l, 8l+8) of every head = RoPE pairs 4l..4l+3.
// The two half-warps of a warp may hold different tensors (a normed key strip
// next to a copied value strip), so the reductions name their own 16 lanes.
__global__ void __launch_bounds__(256) qw_prologue_kernel(const Params p) {
    sm100::grid_launch_dependents();
    sm100::grid_wait();
    const int lane16 = threadIdx.x & 15;
    const uint32_t half_mask = (threadIdx.x & 16) ? 0xffff0000u : 0x0000ffffu;
    const uint32_t half_warps = (gridDim.x * blockDim.x) >> 4;
    // Both half-warps of a warp run the same number of trips (the strip count is
    // padded to an even number by the host): the shuffles need the whole warp.
    for (uint32_t strip = (blockIdx.x * blockDim.x + threadIdx.x) >> 4; strip < p.strips;
         strip += half_warps) {
        const uint32_t row = strip / (uint32_t)p.tensors;
        const uint32_t which = strip - row * (uint32_t)p.tensors;  // 0 query, 1 key, 2 value
        const bool live = row < p.rows;
        const uint4 *src = (which == 0 ? p.q_in : which == 1 ? p.k_in : p.v_in) +
                           (size_t)row * p.heads * 16 + lane16;
        uint4 *dst = (which == 0 ? p.q_out : which == 1 ? p.k_out : p.v_out) +
                     (size_t)row * p.heads * 16 + lane16;
        const uint4 *w = which == 0 ? p.wq : which == 1 ? p.wk : nullptr;
        const bool rotate = p.cos_t && which < 2;
        float wf[8], cc[4], sn[4];
        if (w) {
            const uint4 wv = w[lane16];
            wf[0] = bf16_lo(wv.x); wf[1] = bf16_hi(wv.x); wf[2] = bf16_lo(wv.y); wf[3] = bf16_hi(wv.y);
            wf[4] = bf16_lo(wv.z); wf[5] = bf16_hi(wv.z); wf[6] = bf16_lo(wv.w); wf[7] = bf16_hi(wv.w);
        }
        if (p.bound_out && strip < 2u && w) write_bound(p, which, wf, half_mask, lane16);
        if (rotate) {
            const size_t t = (size_t)((live ? row : 0u) % p.table_rows) * 16 + lane16;
            const float4 c = p.cos_t[t], s4 = p.sin_t[t];
            cc[0] = c.x; cc[1] = c.y; cc[2] = c.z; cc[3] = c.w;
            sn[0] = s4.x; sn[1] = s4.y; sn[2] = s4.z; sn[3] = s4.w;
        }
        for (uint32_t head0 = 0; head0 < p.heads; head0 += kHeadsPerTrip) {
            uint4 x[kHeadsPerTrip];
#pragma unroll
            for (int u = 0; u < kHeadsPerTrip; ++u)
                x[u] = (live && head0 + u < p.heads) ? src[(size_t)(head0 + u) * 16]
                                                     : make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int u = 0; u < kHeadsPerTrip; ++u) {
                const uint4 y = finish_head(p, x[u], w != nullptr, rotate, wf, cc, sn, half_mask);
                if (live && head0 + u < p.heads)
                    dst[(size_t)(head0 + u) * 16] = y;
            }
        }
    }
}

// The same for few strips, where a strip's time is a chain of memory round trips and not
// bandwidth: its first loads all leave together, a trip's loads run under the trip before, and
// the heads of a row are dealt out to p.groups half-warps of p.group_heads each, as long as that
// finds SMs with room.  Two heads a trip (and the next two in flight) fit the registers of four
// CTAs per SM, which is the largest grid it is for; four heads a trip fit three.  us a launch of
// q and k:
//                         form above   trips of four   trips of two
//   24 heads,  320 rows       9.7            4.9            5.1
//   24 heads, 1152 rows      12.2            7.5            7.0
//   32 heads, 2351 rows      18.2           15.5           13.7
//   24 heads, 3500 rows      17.0           15.8           16.3
//    6 heads, 4352 rows       8.1            9.8            6.9
//   24 heads, 4352 rows      21.0           22.9           20.7
// Two waves of it are no better than the form above (24 heads, 8704 rows 39.4 and 39.4, 16896
// rows 72.1 and 73.5).
constexpr int kFewTrip = 2, kFewPerSm = 4;
constexpr uint32_t kFewGroup = 4;  // heads are dealt out by the four
__global__ void __launch_bounds__(256, kFewPerSm) qw_prologue_few_kernel(const Params p) {
    sm100::grid_launch_dependents();
    sm100::grid_wait();
    const int lane16 = threadIdx.x & 15;
    const uint32_t half_mask = (threadIdx.x & 16) ? 0xffff0000u : 0x0000ffffu;
    const uint32_t strip = (blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    const uint32_t per_row = (uint32_t)p.tensors * p.groups;
    const uint32_t row = strip / per_row, rest = strip - row * per_row;
    if (row >= p.rows) return;  // (the reductions name their own 16 lanes)
    const uint32_t group = rest / (uint32_t)p.tensors;
    const uint32_t which = rest - group * (uint32_t)p.tensors;  // 0 query, 1 key, 2 value
    const size_t at = (size_t)row * p.heads * 16 + lane16;
    const uint4 *src = (which == 0 ? p.q_in : which == 1 ? p.k_in : p.v_in) + at;
    uint4 *dst = (which == 0 ? p.q_out : which == 1 ? p.k_out : p.v_out) + at;
    const uint4 *w = which == 0 ? p.wq : which == 1 ? p.wk : nullptr;
    const bool rotate = p.cos_t && which < 2;
    const uint32_t begin = group * p.group_heads, end = min(p.heads, begin + p.group_heads);
    const auto load_trip = [&](uint4 (&x)[kFewTrip], uint32_t head0) {
#pragma unroll
        for (int u = 0; u < kFewTrip; ++u)
            x[u] = head0 + u < end ? src[(size_t)(head0 + u) * 16] : make_uint4(0, 0, 0, 0);
    };
    uint4 x[kFewTrip];
    load_trip(x, begin);
    float4 c4 = make_float4(0, 0, 0, 0), s4 = c4;
    if (rotate) {
        const size_t t = (size_t)(row % p.table_rows) * 16 + lane16;
        c4 = p.cos_t[t];
        s4 = p.sin_t[t];
    }
    const uint4 wv = w ? w[lane16] : make_uint4(0, 0, 0, 0);
    const float cc[4] = {c4.x, c4.y, c4.z, c4.w}, sn[4] = {s4.x, s4.y, s4.z, s4.w};
    const float wf[8] = {bf16_lo(wv.x), bf16_hi(wv.x), bf16_lo(wv.y), bf16_hi(wv.y),
                         bf16_lo(wv.z), bf16_hi(wv.z), bf16_lo(wv.w), bf16_hi(wv.w)};
    for (uint32_t head0 = begin; head0 < end; head0 += kFewTrip) {
        uint4 next[kFewTrip];
        load_trip(next, head0 + kFewTrip);
#pragma unroll
        for (int u = 0; u < kFewTrip; ++u) {
            const uint4 y = finish_head(p, x[u], w != nullptr, rotate, wf, cc, sn, half_mask);
            if (head0 + u < end) dst[(size_t)(head0 + u) * 16] = y;
        }
#pragma unroll
        for (int u = 0; u < kFewTrip; ++u) x[u] = next[u];
    }
    if (p.bound_out && row == 0 && group == 0 && w) write_bound(p, which, wf, half_mask, lane16);
}

__global__ void qw_scale_bf16_kernel(__nv_bfloat16 *out, const __nv_bfloat16 *in, size_t n,
                                     float scale) {
    sm100::grid_launch_dependents();
    sm100::grid_wait();
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (; i < n; i += stride) {
        float v = __uint_as_float((uint32_t)__bfloat16_as_ushort(in[i]) << 16);
        out[i] = __ushort_as_bfloat16((unsigned short)f32_to_bf16_bits(__fmul_rn(v, scale)));
    }
}

// SM count of the current device (a process may drive several devices).
int sm_count_cached() {
    static int sms[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (!sms[dev]) {
        cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
        if (sms[dev] <= 0) sms[dev] = 148;
    }
    return sms[dev];
}

// Dynamic shared memory with which `per_sm` CTAs fit an SM (228 KB, 1 KB of it taken per
// CTA) and one more does not.
constexpr size_t spread_smem(unsigned per_sm) { return 227 * 1024 / (per_sm + 1) + 1024; }

// More than 48 KB of it needs a per-device attribute (set by the first launch of any size:
// a later one may be captured).
bool spread_ready() {
    static bool ready[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    const bool tracked = dev >= 0 && dev < 64;
    if (tracked && ready[dev]) return true;
    if (cudaFuncSetAttribute(qw_prologue_few_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)spread_smem(1)) != cudaSuccess)
        return false;
    if (tracked) ready[dev] = true;
    return true;
}

}  // namespace

extern "C" int qwcu_prologue_launch(const qwcu_prologue_args *a, qwcu_stream stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (!a->rows || !a->heads || !a->q_in || !a->q_out) return (int)cudaErrorInvalidValue;
    Params p;
    p.q_in = static_cast<const uint4 *>(a->q_in);
    p.k_in = static_cast<const uint4 *>(a->k_in);
    p.q_out = static_cast<uint4 *>(a->q_out);
    p.k_out = static_cast<uint4 *>(a->k_out);
    p.wq = static_cast<const uint4 *>(a->norm_weight_q);
    p.wk = static_cast<const uint4 *>(a->norm_weight_k);
    p.cos_t = reinterpret_cast<const float4 *>(a->rope_cos);
    p.sin_t = reinterpret_cast<const float4 *>(a->rope_sin);
    p.rows = a->rows;
    p.table_rows = a->table_rows ? a->table_rows : a->rows;
    p.heads = a->heads;
    p.eps = a->epsilon;
    p.double_round = a->double_round;
    p.v_in = static_cast<const uint4 *>(a->v_in);
    p.v_out = static_cast<uint4 *>(a->v_out);
    p.bound_out = a->bound_out;
    if (a->bound_out && (!a->k_in || a->v_in || !a->norm_weight_q || !a->norm_weight_k))
        return (int)cudaErrorInvalidValue;
    if (a->v_in && (!a->k_in || !a->v_out)) return (int)cudaErrorInvalidValue;
    p.tensors = a->v_in ? 3 : a->k_in ? 2 : 1;
    unsigned long long strips = (unsigned long long)a->rows * p.tensors;
    strips = (strips + 1ull) & ~1ull;  // whole warps iterate together
    if (strips > 0xffffffffull) return (int)cudaErrorInvalidValue;
    p.strips = (uint32_t)strips;
    const unsigned threads = 256, sms = (unsigned)sm_count_cached();
    if (!spread_ready()) return (int)cudaGetLastError();
    const unsigned long long room = (unsigned long long)kFewPerSm * sms * (threads / 16);  // half-warps
    const unsigned long long plain = (unsigned long long)a->rows * p.tensors;
    if (plain <= room) {
        const uint32_t parts = (a->heads + kFewGroup - 1) / kFewGroup;
        unsigned long long groups = room / plain;
        if (groups > parts) groups = parts;
        p.group_heads = (uint32_t)((parts + groups - 1) / groups) * kFewGroup;
        p.groups = (a->heads + p.group_heads - 1) / p.group_heads;
        const unsigned blocks = (unsigned)((plain * p.groups * 16 + threads - 1) / threads);
        // Started under the tail of the kernel before it (sm100::launch), a grid of half a CTA to
        // three CTAs per SM would pile up on the SMs that are free first.  Shared memory that
        // nobody uses holds every SM to its even share (32 heads, 700 rows 7.8 -> 6.8 us; 24 heads,
        // 1152 rows 7.9 -> 7.0, 3500 rows 18.3 -> 16.3; 2351 rows of 32 heads 13.7, 320 of 24 heads
        // 5.1 either way).  A smaller grid finds an SM for every CTA, a larger one fills all of them.
        const bool spread = 2 * blocks > sms && blocks <= 3 * sms;
        const size_t smem = spread ? spread_smem((blocks + sms - 1) / sms) : 0;
        return sm100::launch(qw_prologue_few_kernel, blocks, threads, smem, 1, stream, p);
    }
    const unsigned long long want = (strips * 16 + threads - 1) / threads;
    // Grid: at most 8 resident CTAs per SM, a multiple of the SM count when capped.
    const unsigned long long cap = sms * 8ull;
    const unsigned blocks = (unsigned)(want < cap ? want : cap);
    return sm100::launch(qw_prologue_kernel, blocks, threads, 0, 1, stream, p);
}

extern "C" int qwcu_scale_bf16_launch(void *out, const void *in, size_t elements, float scale,
                                      qwcu_stream stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (!elements) return 0;
    size_t want = (elements + 255) / 256;
    size_t cap = (size_t)sm_count_cached() * 16;
    unsigned int blocks = (unsigned int)(want < cap ? want : cap);
    return sm100::launch(qw_scale_bf16_kernel, blocks, 256, 0, 1, stream,
                         static_cast<__nv_bfloat16 *>(out), static_cast<const __nv_bfloat16 *>(in),
                         elements, scale);
}

extern "C" int qwcu_device_sm_count(int device) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
    return sms;
}

extern "C" int qwcu_device_cc(int device) {
    int major = 0, minor = 0;
    if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, device) != cudaSuccess)
        return 0;
    return major * 10 + minor;
}
