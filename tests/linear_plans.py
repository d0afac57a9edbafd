"""What the GEMM's dispatch makes of the sizes the tests use, on the 148 SMs of a B200:
(rows, columns of an output, outputs) -> CTAs per tile, columns of a tile, whole tiles,
whole and half tiles together.  A change of the dispatch's costs that sends a size
elsewhere fails here, instead of leaving a tile shape without a test."""
import ctypes as C

SMS = 148
PLANS = {
    (1, 8, 1): (2, 128, 1, 1),
    (257, 264, 1): (2, 128, 6, 6),
    (200, 520, 1): (2, 128, 5, 5),
    (5000, 384, 1): (2, 128, 60, 60),
    (513, 5120, 1): (2, 256, 60, 60),
    (4097, 3072, 1): (2, 256, 204, 204),
    (1100, 5120, 1): (2, 256, 74, 126),
    (1152, 9216, 1): (2, 256, 148, 212),
    (300, 11520, 1): (1, 256, 135, 135),
    (384, 12288, 1): (1, 256, 144, 144),
    (200, 512, 3): (2, 128, 12, 12),
    (300, 4096, 3): (1, 256, 144, 144),
    (1152, 3072, 3): (2, 256, 148, 212),
    (513, 2688, 3): (2, 256, 74, 124),
}


class Plan(C.Structure):
    _fields_ = [(f, C.c_uint32) for f in ("ctas", "columns", "whole", "items")]

    def fields(self):
        return tuple(getattr(self, f) for f, _ in self._fields_)


def plan_on(lib, rows, columns, outputs, sms=SMS):
    fn = lib.qwcu_linear_sm100_plan
    fn.restype = C.c_int
    fn.argtypes = [C.c_uint32] * 3 + [C.c_int, C.POINTER(Plan)]
    p = Plan()
    assert fn(rows, columns, outputs, sms, C.byref(p)) == 0
    return p


def plan(gpu, rows, columns, outputs):
    """The dispatch's choice on this GPU."""
    return plan_on(gpu.lib, rows, columns, outputs, gpu.lib.qwcu_device_sm_count(0))


def check(gpu, rows, columns, outputs):
    assert plan(gpu, rows, columns, outputs).fields() == PLANS[rows, columns, outputs]
