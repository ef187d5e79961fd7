"""Which 2-D calls take the kernel of several steps per launch: the rule is host
arithmetic on the run's constants."""
import ctypes as C

import pytest

FP64, FP32 = 0, 1


def steps_per_launch(n, dx, prec, left, sums):
    import coolbubble_b200 as cb
    from coolbubble_b200 import _lib as L

    class Constants(C.Structure):
        _fields_ = [("bytes", C.c_ubyte * 208)]   # StepConst

    make = L.lib["_ZN2cb10make_constEPK9cb_params"]
    make.restype, make.argtypes = Constants, [C.POINTER(L.cb_params)]
    rule = L.lib["_ZN2cb13step2tb_stepsERKNS_9StepConstEiib"]
    rule.restype, rule.argtypes = C.c_int, [C.POINTER(Constants), C.c_int, C.c_int, C.c_bool]
    k = make(C.byref(cb.make_params(2, n, n * dx, 2.0, 0.1 * dx, precision="fp64" if prec == FP64 else "fp32c")))
    return rule(C.byref(k), prec, left, sums)


@pytest.mark.parametrize("n,dx,prec,left,here", [
    (288, 0.125, FP64, 1, False), (292, 0.125, FP64, 1, True), (64, 0.125, FP64, 2, False), (68, 0.125, FP64, 2, True),
    (1024, 0.125, FP32, 1, False), (1024, 0.125, FP32, 2, False), (1024, 0.125, FP32, 3, True),   # one strip a row
    (1024, 0.125, FP64, 1, True), (1028, 0.125, FP32, 1, True),
    (3584, 0.125, FP32, 1, True), (4096, 0.125, FP32, 1, False), (8192, 0.125, FP32, 1, False),
    (4097, 0.125, FP32, 1, True),                                   # rows the strips do not take
    (4096, 0.125, FP32, 2, True), (4096, 0.125, FP64, 1, True), (4096, 0.1, FP64, 1, True),
    (3584, 0.17, FP64, 1, True), (4096, 0.17, FP64, 1, False), (4096, 0.17, FP64, 2, True)])   # the compiler's division
def test_calls_of_one_or_two_steps_with_a_line(n, dx, prec, left, here):
    got = steps_per_launch(n, dx, prec, left, True)
    assert (got > 0) == here and got <= left


def test_plain_single_steps_stay_on_the_one_step_kernels():
    for n in (64, 512, 1024, 4096):
        for prec in (FP64, FP32):
            assert steps_per_launch(n, 0.125, prec, 1, False) == 0
            assert steps_per_launch(n, 0.125, prec, 2, False) == 2
