"""The rule that gives a mesh its one-launch PCG form and row ranges (host only)."""
import ctypes as C

import pytest


def parts(n, e, nv=4, vsize=4, sms=148, cap=0, two_level=1, after=0):
    from sors_b200 import _lib
    fn = _lib.load().sors_pcg_parts
    fn.restype = None
    fn.argtypes = [C.c_int32] * 8 + [C.POINTER(C.c_int32)]
    out = (C.c_int32 * 3)()
    fn(n, e, nv, vsize, sms, cap, two_level, after, out)
    return tuple(out)


@pytest.mark.parametrize("n,e,nv", [(8, 5, 4), (525, 1536, 4), (2744, 13182, 4), (5000, 24000, 4), (891, 640, 8)])
@pytest.mark.parametrize("vsize", [4, 8])
@pytest.mark.parametrize("cap", [1, 2, 7, 8, 15, 16, 148])
def test_grid_cap_holds_for_the_cluster(n, e, nv, vsize, cap):
    """max_blocks is the largest grid of any kernel of the handle, below 16 blocks too."""
    form, g, _ = parts(n, e, nv, vsize, cap=cap)
    assert form == 0 or 1 <= g <= cap
    if form:  # every range within a block's rows
        assert n <= g * 512
    if cap >= 16:
        assert (form, g) == parts(n, e, nv, vsize)[:2] or form != 1


@pytest.mark.parametrize("cap", [1184, 14_510_025, 2**31 - 1])
def test_cap_above_the_whole_gpu_changes_nothing(cap):
    assert parts(9856, 52488, cap=cap) == parts(9856, 52488)


@pytest.mark.parametrize("n,e,nv,vsize,forms", [(525, 1536, 4, 8, [1, 2, 3]), (9856, 52488, 4, 4, [2, 3]),
                                                (39304, 215622, 4, 8, [2, 3]), (101000, 576000, 4, 4, [3]),
                                                (18921, 15680, 8, 8, [2])])
def test_a_refused_form_goes_on_to_the_next(n, e, nv, vsize, forms):
    """Forms in their order, each at most once, down to none (the rings of FP64 hex rows are too
    large to stream); the streamed one needs the coarse correction."""
    seen, form = [], 0
    while True:
        form = parts(n, e, nv, vsize, after=form)[0]
        if not form:
            break
        seen.append(form)
    assert seen == forms
    assert 3 not in [parts(n, e, nv, vsize, two_level=0, after=k)[0] for k in range(4)]


@pytest.mark.parametrize("n", [8, 81, 525, 2000, 9856])
@pytest.mark.parametrize("after", [0, 1, 2])
def test_ranges_have_enough_rows_for_their_rigid_modes(n, after):
    form, g, a = parts(n, 5 * n, after=after)
    assert form and n > 16 * (g * a - 1)
