"""GPU parity of the GEMM's tile shapes: every variant of the dispatch at the edges of
its tiles (first, last and ragged rows and columns, a K tail, several tiles per CTA
pair, the half tiles of a partly filled last wave), against the CPU oracle on the rows
around the tile borders.  Tolerance as for the GEMM elsewhere: fp32 sums in another
order, one rounding to bf16."""
import numpy as np
import pytest

import oracle_lib as O
from qwen_metal_b200 import workloads
from test_gpu_linear import check_gemm, weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,k,n,bias", [
    (1, 8, 8, True),            # the smallest: one row, one 16-byte column group
    (257, 136, 264, True),      # 128-column pair tiles, one row and 8 columns over
    (513, 72, 5120, False),     # 256-column pair tiles, one wave
    (300, 72, 11520, True),     # 90 pair tiles on 74 pairs: 16 of them as halves
    (384, 200, 12288, False),   # single CTAs of 128 x 256: one wave where pairs need two
    (4097, 64, 3072, False),    # several tiles per pair: both accumulators, both phases
    (200, 1160, 520, True),     # W rows of 2320 bytes: prefetched in whole and partial pieces
])
def test_every_tile_shape_matches_oracle(gpu, rows, k, n, bias):
    rng = np.random.default_rng(rows + k + n)
    x, w = workloads.normal_bf16(rng, (rows, k)), weights(rng, n, k)
    b = workloads.normal_bf16(rng, (n,)) if bias else None
    xt, wt, ot = gpu.bf16(x), gpu.bf16(w), gpu.new_bf16(rows * n)
    bt = gpu.bf16(b) if bias else None
    gpu.begin()
    gpu.check(gpu.lib.h3_gpu_linear_bf16(gpu.handle, ot, xt, wt, bt, rows, k, n), "linear")
    gpu.submit()
    got = gpu.read_bf16(ot, rows * n).reshape(rows, n)
    edges = {r + d for r in range(0, rows, 128) for d in (-1, 0, 1, 31, 32)} | {rows - 1}
    sample = np.array(sorted(r for r in edges if 0 <= r < rows), np.uint32)
    check_gemm(got[sample], O.linear(x, w, b, rows, k, n, sample)[sample], f"{rows}x{k}x{n}")
    for t in [xt, wt, ot] + ([bt] if bias else []):
        gpu.free(t)
