"""GPU parity of the GEMM's tile shapes: every variant of the dispatch at the edges of
its tiles (first, last and ragged rows and columns, a K tail, several tiles per CTA
pair, the half tiles of a partly filled last wave), against the CPU oracle on the rows
around the tile borders.  Tolerance as for the GEMM elsewhere: fp32 sums in another
order, one rounding to bf16.  linear_plans.py holds what each size is dispatched to on
148 SMs; the tests fail where it is something else."""
import ctypes as C

import numpy as np
import pytest

import linear_plans as P
import oracle_lib as O
from qwen_metal_b200 import abi, workloads
from test_gpu_linear import check_gemm, weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,k,n,bias", [
    (1, 8, 8, True),            # the smallest: one row, one 16-byte column group
    (257, 136, 264, True),      # 128-column pair tiles, one row and 8 columns over
    (513, 72, 5120, False),     # 256-column pair tiles, one wave
    (300, 72, 11520, True),     # single CTAs: one wave where pairs need a whole one and a half one
    (384, 200, 12288, False),   # single CTAs of 128 x 256: one wave where pairs need two
    (4097, 64, 3072, False),    # several tiles per pair: both accumulators, both phases
    (200, 1160, 520, True),     # 128-column pair tiles, 18 K steps and 8 columns
    (5000, 64, 384, True),      # 128-column pair tiles in one wave where 256 columns leave half a tile
    (1100, 72, 5120, True),     # 256-column pair tiles, the last wave as halves
    (1152, 64, 9216, False),    # the same behind two tiles per pair
])
def test_every_tile_shape_matches_oracle(gpu, rows, k, n, bias):
    P.check(gpu, rows, n, 1)
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


@pytest.mark.parametrize("batch,table,dim", [
    (1, 200, 512),    # 128-column pair tiles: a head per tile
    (1, 300, 4096),   # single CTAs: two heads per tile, the second by the second warp group
    (1, 1152, 3072),  # pairs: two whole tiles on either accumulator, then halves of one head
    (1, 513, 2688),   # 21 heads: the last tile of every output holds one
    # the same with a rotation table that begins again between, inside and many times in the boxes
    # of 32 rows, in 256-column tiles and halves, on a first and a last tile of a CTA
    (100, 2, 512), (60, 5, 4096), (4, 75, 4096), (9, 128, 3072), (384, 3, 3072), (12, 96, 3072), (19, 27, 2688),
])
def test_fused_epilogue_on_every_tile_shape(gpu, batch, table, dim):
    """q/k/v with the norm and the rotation in the epilogue: the plain projection against
    the oracle on a row sample, the fused one bit for bit against the oracle's norm and
    rotation of the plain one's bf16 output, v equal to the plain one's."""
    seq = batch * table
    P.check(gpu, seq, dim, 3)
    rng = np.random.default_rng(seq + dim)
    lib, heads = gpu.lib, dim // 128
    x = workloads.normal_bf16(rng, (seq, dim))
    ws = [weights(rng, dim, dim) for _ in range(3)]
    wq, wk = (workloads.normal_bf16(rng, (128,), 1.0, 0.1) for _ in range(2))
    if batch == 1:
        cos, sin = abi.rope_tables(seq - 144, 12, 12)
    else:
        angle = rng.uniform(-3, 3, (table, 64))
        cos, sin = np.cos(angle).astype(np.float32), np.sin(angle).astype(np.float32)
    xt, wts = gpu.bf16(x), [gpu.bf16(w) for w in ws]
    plain, fused = ([gpu.new_bf16(seq * dim) for _ in range(3)] for _ in range(2))
    wqt, wkt, ct, st, bt = gpu.bf16(wq), gpu.bf16(wk), gpu.f32(cos), gpu.f32(sin), gpu.new_f32(2)
    gpu.begin()
    gpu.check(lib.qw_gpu_qkv_bf16(gpu.handle, *plain, xt, *wts, seq, dim), "qkv")
    gpu.check(lib.qw_gpu_qkv_norm_rope_bf16(gpu.handle, *fused, xt, *wts, wqt, wkt, ct, st, bt, batch,
                                            table, dim, 1e-6), "qkv norm rope")
    gpu.submit()
    got = [gpu.read_bf16(t, seq * dim).reshape(seq, dim) for t in plain]
    sample = np.array([0, 31, 32, 127, 128, seq // 2, seq - 1], np.uint32)
    for name, g, w in zip("qkv", got, ws):
        check_gemm(g[sample], O.linear(x, w, None, seq, dim, dim, sample)[sample], f"{name} {seq}x{dim}")
    normed = [O.head_rms_norm(g.reshape(seq, heads, 128), w, seq, heads, 1e-6)
              for g, w in zip(got, (wq, wk))]
    want_q, want_k = O.qk_rope(*normed, np.tile(cos, (batch, 1)), np.tile(sin, (batch, 1)), seq, heads)
    fq, fk, fv = (gpu.read_bf16(t, seq * dim).reshape(seq, heads, 128) for t in fused)
    assert np.array_equal(fq, want_q.reshape(fq.shape)), float((fq != want_q.reshape(fq.shape)).mean())
    assert np.array_equal(fk, want_k.reshape(fk.shape)), float((fk != want_k.reshape(fk.shape)).mean())
    assert np.array_equal(fv.reshape(seq, dim), got[2])
    for t in [xt, wqt, wkt, ct, st, bt] + wts + plain + fused:
        gpu.free(t)


class LinearArgs(C.Structure):
    """qwcu_linear_args."""
    _fields_ = [("a", C.c_void_p), ("w", C.c_void_p * 3), ("c", C.c_void_p * 3), ("bias", C.c_void_p * 3),
                ("n_outputs", C.c_uint32), ("m", C.c_uint32), ("k", C.c_uint32), ("n", C.c_uint32),
                ("norm_weight", C.c_void_p * 2), ("rope_cos", C.c_void_p), ("rope_sin", C.c_void_p),
                ("table_rows", C.c_uint32), ("epsilon", C.c_float), ("bound_out", C.c_void_p),
                ("status", C.c_void_p), ("wait_cycles", C.c_longlong), ("withhold_from", C.c_uint32 * 2)]


@pytest.mark.parametrize("rows,dim", [(200, 512), (513, 2688)])  # (21 heads: half a tile past each output)
def test_fused_epilogue_takes_a_bias(gpu, rows, dim):
    """The launch takes a bias together with the norm and the rotation, which no op asks for: bit
    for bit the projection with a bias, then the oracle's norm and rotation."""
    P.check(gpu, rows, dim, 3)
    rng = np.random.default_rng(rows)
    lib, heads, k = gpu.lib, dim // 128, 72
    ptr = lib.qw_gpu_tensor_device_ptr
    x = gpu.bf16(workloads.normal_bf16(rng, (rows, k)))
    ws = [gpu.bf16(weights(rng, dim, k)) for _ in range(3)]
    bs = [gpu.bf16(workloads.normal_bf16(rng, (dim,))) for _ in range(3)]
    norms = [workloads.normal_bf16(rng, (128,), 1.0, 0.1) for _ in range(2)]
    angle = rng.uniform(-3, 3, (rows, 64))
    cos, sin = np.cos(angle).astype(np.float32), np.sin(angle).astype(np.float32)
    rest = [gpu.bf16(norms[0]), gpu.bf16(norms[1]), gpu.f32(cos), gpu.f32(sin), gpu.u32(np.zeros(16, np.uint32))]
    plain, fused = ([gpu.new_bf16(rows * dim) for _ in range(3)] for _ in range(2))
    args = LinearArgs(a=ptr(x), n_outputs=3, m=rows, k=k, n=dim, rope_cos=ptr(rest[2]), rope_sin=ptr(rest[3]),
                      table_rows=rows, epsilon=1e-6, status=ptr(rest[4]))
    for i in range(3):
        args.w[i], args.c[i], args.bias[i] = ptr(ws[i]), ptr(fused[i]), ptr(bs[i])
    for i in range(2):
        args.norm_weight[i] = ptr(rest[i])
    launch = lib.qwcu_linear_sm100_launch
    launch.restype, launch.argtypes = C.c_int, [C.POINTER(LinearArgs), C.c_int, C.c_void_p]
    gpu.begin()
    for i in range(3):
        gpu.check(lib.h3_gpu_linear_bf16(gpu.handle, plain[i], x, ws[i], bs[i], rows, k, dim), "linear")
    assert launch(C.byref(args), lib.qwcu_device_sm_count(0), lib.qw_gpu_stream(gpu.handle)) == 0
    gpu.submit()
    got = [gpu.read_bf16(t, rows * dim).reshape(rows, heads, 128) for t in plain]
    normed = [O.head_rms_norm(g, w, rows, heads, 1e-6) for g, w in zip(got, norms)]
    want = [*O.qk_rope(*normed, cos, sin, rows, heads), got[2]]
    for t, w in zip(fused, want):
        assert np.array_equal(gpu.read_bf16(t, rows * dim).reshape(w.shape), w)
    for t in [x] + ws + bs + rest + plain + fused:
        gpu.free(t)


@pytest.mark.parametrize("rows,k,n", [
    (200, 1024, 520),    # 128-column pair tiles, one per pair
    (1100, 1024, 5120),  # 256-column pair tiles, whole and half
    (300, 1024, 11520),  # single CTAs
])
@pytest.mark.parametrize("withheld", [(5, 5), (5, 7), (7, 5), (3, 0), (0, 4)])
def test_expired_waits_leave_nothing_in_flight(gpu, rows, k, n, withheld):
    """The GEMM's waits run out cleanly.  With a budget of about a millisecond and
    producers that leave out every K step from some point on -- the same for both CTAs of a
    pair, or one earlier than the other, so that the copies of the other are in flight for
    steps that never become complete -- the kernel records where, brings every copy it
    issued to its end, frees its TMEM and returns; h3_gpu_submit reports it, and the next
    launch on the context gives the bits it gave before."""
    P.check(gpu, rows, n, 1)
    if P.plan(gpu, rows, n, 1).ctas == 1 and not withheld[0]:
        pytest.skip("a single CTA has no second producer")
    lib = gpu.lib
    rng = np.random.default_rng(rows)
    xt, wt = gpu.bf16(workloads.normal_bf16(rng, (rows, k))), gpu.bf16(weights(rng, n, k))
    ot = gpu.new_bf16(rows * n)

    def launch():
        gpu.begin()
        assert lib.h3_gpu_linear_bf16(gpu.handle, ot, xt, wt, None, rows, k, n) == 1
        return lib.h3_gpu_submit(gpu.handle)

    assert launch() == 1
    want = gpu.read_bf16(ot, rows * n)
    try:
        assert lib.qw_gpu_debug_linear_waits(gpu.handle, 2_000_000, *withheld)
        assert launch() == 0
        assert "wait ran out" in gpu.error(), gpu.error()
    finally:
        assert lib.qw_gpu_debug_linear_waits(gpu.handle, 0, 0, 0)
    assert launch() == 1
    assert np.array_equal(gpu.read_bf16(ot, rows * n), want)
    for t in (xt, wt, ot):
        gpu.free(t)


def test_a_tile_shape_met_first_inside_a_capture():
    """The op has run before the capture, but at a size that takes another kernel."""
    import os
    import subprocess
    import sys
    worker = os.path.join(os.path.dirname(os.path.abspath(__file__)), "capture_worker.py")
    done = subprocess.run([sys.executable, worker], capture_output=True, text=True, timeout=240)
    assert done.returncode == 0, done.stdout[-2000:] + done.stderr[-2000:]
