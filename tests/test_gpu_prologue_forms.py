"""The norm and rotation of few rows run in a kernel of their own, which deals the heads of a row
out to several half-warps.  The arithmetic is the other kernel's, so the same rows must give the
same bits in either: few rows by themselves, and as part of a call that is too long for it."""
import numpy as np
import pytest

from qwen_metal_b200 import workloads

pytestmark = pytest.mark.gpu
MANY = 9600  # rows: more strips than four CTAs per SM hold (148 SMs of 64 strips)


@pytest.mark.parametrize("rows", [1, 5, 33, 320, 2351])
@pytest.mark.parametrize("heads", [1, 3, 4, 5, 24, 32])
def test_few_rows_give_the_bits_of_many(gpu, rows, heads):
    if rows * heads > 40000:
        heads = 6
    lib, rng = gpu.lib, np.random.default_rng(rows * 100 + heads)
    q, k = (workloads.normal_bf16(rng, (rows, heads, 128)) for _ in range(2))
    wq, wk = (workloads.normal_bf16(rng, (128,), 1.0, 0.1) for _ in range(2))
    angle = rng.uniform(-3, 3, (rows, 64))
    cos, sin = np.cos(angle).astype(np.float32), np.sin(angle).astype(np.float32)
    reps = -(-MANY // rows)
    held = []

    def dev(make, a):
        held.append(make(a))
        return held[-1]

    wqt, wkt = dev(gpu.bf16, wq), dev(gpu.bf16, wk)
    got = {}
    for name, times in (("few", 1), ("many", reps)):
        n = rows * times
        tile = lambda a: np.tile(a, (times,) + (1,) * (a.ndim - 1))  # noqa: E731
        src = [dev(gpu.bf16, tile(q)), dev(gpu.bf16, tile(k))]
        norm = dev(gpu.bf16, tile(q))
        twice = dev(gpu.bf16, tile(q))
        cache_k, cache_v = (dev(gpu.bf16, np.zeros(n * heads * 128, np.uint16)) for _ in range(2))
        out = [dev(gpu.new_bf16, n * heads * 128) for _ in range(3)]
        ct, st, bt = dev(gpu.f32, tile(cos)), dev(gpu.f32, tile(sin)), dev(gpu.new_f32, 2)
        gpu.begin()
        gpu.check(lib.qw_gpu_qk_norm_rope_bound_bf16(gpu.handle, *out[:2], *src, wqt, wkt, ct, st, bt, 1, n,
                                                     heads, 128, 1e-6), "norm rope bound")
        gpu.check(lib.qw_gpu_qk_norm_rope_cache_bf16(gpu.handle, out[2], cache_k, cache_v, src[1], src[0],
                                                     wqt, wkt, ct, st, n, 0, n, heads, 128, 1e-6), "cache")
        gpu.check(lib.h3_gpu_head_rms_norm_bf16(gpu.handle, norm, wqt, n, heads, 128, 1e-6), "norm")
        gpu.check(lib.qw_gpu_head_rms_norm_bf16(gpu.handle, twice, wkt, n, heads, 128, 1e-6), "norm twice")
        gpu.check(lib.qw_gpu_qk_rope_bf16(gpu.handle, *src, *src, ct, st, n, heads, 128), "rope in place")
        gpu.submit()
        got[name] = [gpu.read_bf16(t, rows * heads * 128) for t in
                     (*out[:2], cache_k, cache_v, norm, twice, *src)] + [gpu.read_f32(bt, 2)]
    for few, many in zip(got["few"], got["many"]):
        assert np.array_equal(few, many)
    assert np.array_equal(got["few"][3], q.ravel())  # V goes into the cache as it is
    for t in held:
        gpu.free(t)
