"""Run by test_gpu_linear_tiles.py in a process of its own: a small linear layer first, then a
graph capture of sizes whose kernels the process has not launched before."""
import sys

import numpy as np

import conftest  # noqa: F401  (puts the repository on the path)
from qwen_metal_b200 import abi

gpu = abi.Gpu()
lib, rng = gpu.lib, np.random.default_rng(5)


def normal(*shape):
    return gpu.bf16(abi.f32_to_bf16(rng.standard_normal(shape).astype(np.float32)))


k = 128
x, w = normal(4096, k), normal(12288, k)
outs = [gpu.new_bf16(m * n) for m, n in ((16, 128), (384, 12288), (4096, 3072))]
calls = [lambda m=m, n=n, o=o: lib.h3_gpu_linear_bf16(gpu.handle, o, x, w, None, m, k, n)
         for (m, n), o in zip(((16, 128), (384, 12288), (4096, 3072)), outs)]
gpu.begin()
gpu.check(calls[0](), "first size")
gpu.submit()
gpu.begin()
gpu.check(lib.qw_gpu_graph_begin(gpu.handle), "graph begin")
for call in calls:
    gpu.check(call(), "captured")
graph = lib.qw_gpu_graph_end(gpu.handle)
gpu.check(graph, "graph end")
gpu.check(lib.qw_gpu_graph_launch(gpu.handle, graph), "replay")
gpu.submit()
sizes = (16 * 128, 384 * 12288, 4096 * 3072)
replayed = [gpu.read_bf16(o, n) for o, n in zip(outs, sizes)]
gpu.begin()
for call in calls:
    gpu.check(call(), "eager")
gpu.submit()
lib.qw_gpu_graph_free(graph)
assert all(r.any() and np.array_equal(r, gpu.read_bf16(o, n)) for r, o, n in zip(replayed, outs, sizes))
gpu.close()
sys.exit(0)
