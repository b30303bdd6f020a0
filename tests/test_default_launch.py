"""Which launch shape a mesh has by default, on GPUs of several sizes (host
side, no GPU): the smallest FP64 meshes take a block per quad as long as all
of their blocks are resident at once, one per SM (16x16) or two (8x8)."""
import ctypes as C

import pytest

FP64, FP32 = 0, 1


def shape(ag, form, n, nquad, sms):
    v = [C.c_int() for _ in range(3)]
    assert ag.lib().amrgpu_default_launch(form, n, nquad, sms, *[C.byref(x) for x in v]) == 0
    return tuple(x.value for x in v)


@pytest.mark.parametrize("sms", [148, 132, 64])
@pytest.mark.parametrize("n,small", [(16, (1, 288, 1)), (8, (1, 160, 2))])
def test_small_fp64_meshes_are_resident_at_once(ag, n, small, sms):
    limit = small[0] * small[2] * sms
    assert shape(ag, FP64, n, 1, sms) == small
    assert shape(ag, FP64, n, limit, sms) == small
    assert shape(ag, FP64, n, limit + 1, sms) != small
    assert shape(ag, FP32, n, limit, sms) != small


@pytest.mark.parametrize("form,n,sweep", [(FP64, 16, (4, 128, 3)), (FP64, 8, (8, 128, 3))])
def test_large_meshes_take_the_row_sweep(ag, form, n, sweep):
    quads_of_1024_warps = 1024 * (2 if n == 8 else 1)
    assert shape(ag, form, n, quads_of_1024_warps, 148) == sweep
    assert shape(ag, form, n, quads_of_1024_warps - 2, 148) != sweep


def test_unknown_arguments_are_refused(ag):
    f = ag.lib().amrgpu_default_launch
    for form, n, nquad, sms in ((2, 16, 1, 148), (0, 5, 1, 148), (0, 16, -1, 148), (0, 16, 1, 0)):
        assert f(form, n, nquad, sms, None, None, None) != 0
