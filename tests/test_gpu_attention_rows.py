"""The attention kernel writes its output 32 rows per warp, several lanes to a row: row counts
around a warp's, a sub-tile's and a block's rows, in both forms, token- and head-major, against
the CPU oracle, with rows that see nothing and with what lies behind the output left as it was.
Tolerances as for the attention elsewhere."""
import numpy as np
import pytest

import oracle_lib as O
from qwen_metal_b200 import workloads
from test_gpu_parity import SCALE, gates

pytestmark = pytest.mark.gpu
BEHIND = 4096  # elements behind the output


@pytest.mark.parametrize("form", ["sm100", "sm100-whole"])
@pytest.mark.parametrize("rows", [1, 31, 32, 33, 97, 128, 129, 160, 255, 289])
def test_output_rows_at_the_edges_of_warps_and_blocks(gpu, rows, form):
    lib, heads, keys = gpu.lib, 2, 200
    rng = np.random.default_rng(rows)
    q = workloads.normal_bf16(rng, (rows, heads, 128))
    k, v = (workloads.normal_bf16(rng, (max(rows, keys), heads, 128)) for _ in range(2))
    limits = rng.integers(0, rows + 1, rows).astype(np.uint32)
    limits[: min(rows, 5)] = 0                       # rows that see nothing
    if rows > 128:
        limits[128:160] = 0                          # a warp whose rows see nothing
    qt, kt, vt, lt = gpu.bf16(q), gpu.bf16(k), gpu.bf16(v), gpu.u32(limits)
    behind = workloads.normal_bf16(rng, (q.size + BEHIND,))
    assert lib.qw_gpu_set_attention_kernel(gpu.handle, form.encode())
    try:
        for name in ("full", "head-major", "limits"):
            ot = gpu.bf16(behind)
            gpu.begin()
            if name == "full":
                gpu.check(lib.qw_gpu_sdpa_rect_bf16(gpu.handle, ot, qt, kt, vt, rows, keys, heads, 128,
                                                    SCALE), name)
                ref, _ = O.sdpa(q, k[:keys], v[:keys], None, 1, rows, keys, heads, heads, SCALE)
            elif name == "head-major":
                gpu.check(lib.h3_gpu_sdpa_bf16_head_major_output(gpu.handle, ot, qt, kt, vt, rows, heads,
                                                                 128, SCALE), name)
                ref, _ = O.sdpa(q, k[:rows], v[:rows], None, 1, rows, rows, heads, heads, SCALE)
                ref = np.asarray(ref).reshape(rows, heads, 128).transpose(1, 0, 2)
            else:
                gpu.check(lib.qw_gpu_attn_block_causal_bf16(gpu.handle, ot, qt, kt, vt, lt, 1, rows, heads,
                                                            heads, 128, None, 0, SCALE), name)
                ref, _ = O.sdpa(q, k[:rows], v[:rows], limits, 1, rows, rows, heads, heads, SCALE)
            gpu.submit()
            got = gpu.read_bf16(ot, q.size + BEHIND)
            if np.abs(np.asarray(ref, np.float64)).max() > 0:
                gates(got[: q.size], ref, f"{name}, {rows} rows, {form}")
            if name == "limits":
                rows_out = got[: q.size].reshape(rows, heads, 128)
                assert not (rows_out[limits == 0] & 0x7FFF).any()
            assert np.array_equal(got[q.size:], behind[q.size:]), name
            gpu.free(ot)
    finally:
        assert lib.qw_gpu_set_attention_kernel(gpu.handle, b"sm100")
    for t in (qt, kt, vt, lt):
        gpu.free(t)
