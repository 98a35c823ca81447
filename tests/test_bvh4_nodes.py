"""The quantised four-child node (pack_bvh4): every plane it decodes to lies on
or outside its child's box, whatever the boxes' size and place, and not more
than a few quanta outside; axes without a finite grid bound nothing. Checked
in exact rational arithmetic, no GPU needed."""
import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

from oxideav_render_b200 import native


def pack(lo, hi, ref):
    out = np.zeros(16, np.uint32)
    ref = np.asarray(ref, np.int32)
    lo, hi = np.ascontiguousarray(lo, np.float32), np.ascontiguousarray(hi, np.float32)
    rc = native.load().pt_debug_pack_node4(lo.ctypes.data_as(native.fp), hi.ctypes.data_as(native.fp),
                                           ref.ctypes.data_as(C.POINTER(C.c_int32)), out.ctypes.data_as(native.u32p))
    assert rc == 0
    f = out.view(np.float32)
    base, step = f[0:3], (f[3], f[4], f[5])
    words = ((out[6], out[7]), (out[8], out[9]), (out[10], out[11]))
    assert np.array_equal(out[12:16].view(np.int32), ref)
    return base, step, words


def planes(base, step, words, axis, child):
    q = [(int(w) >> (8 * child)) & 0xFF for w in words[axis]]
    b, s = Fraction(float(base[axis])), Fraction(float(step[axis]))
    return [b + s + s * x / 32768 for x in q], s / 32768


@pytest.mark.parametrize("size", [1e-35, 1e-12, 1.0, 7e4, 1e30])
@pytest.mark.parametrize("offset", [0.0, 1.0, -3e3])
@pytest.mark.parametrize("children", [1, 2, 3, 4])
def test_planes_enclose_the_boxes(size, offset, children):
    rng = np.random.default_rng(int(children * 100 + abs(offset) % 7))
    for _ in range(20):
        a = (rng.normal(size=(3, 4)) * size + offset).astype(np.float32)
        b = (a + np.abs(rng.normal(size=(3, 4))) * size * rng.choice([0.0, 1e-3, 1.0])).astype(np.float32)
        ref = [5, -7, 9, 11][:children] + [-1] * (4 - children)
        base, step, words = pack(a, np.maximum(a, b), ref)
        for ax in range(3):
            m, e = np.frexp(step[ax])
            assert m == 0.5  # a power of two
            lo, hi = a[ax, :children], np.maximum(a, b)[ax, :children]
            grid = max(float(hi.max()) - float(lo.min()), 0.0)
            for c in range(4):
                (pl, ph), quantum = planes(base, step, words, ax, c)
                if c >= children:
                    assert pl > ph  # an unused slot is missed
                    continue
                tl, th = Fraction(float(lo[c])), Fraction(float(hi[c]))
                assert pl <= tl and ph >= th
                assert pl >= tl - 2 * quantum and ph <= th + 2 * quantum
            # Eight bits over the node's extent, plus what the rounding of the
            # base to f32 needs at this distance from zero.
            assert quantum <= max(Fraction(grid) / 63, Fraction(float(np.abs(a[ax]).max())) / 2 ** 22,
                                  Fraction(2) ** -99)


# Bounds next to zero against the grid, whose distance from the grid's origin
# f64 cannot hold: -1e-30 below an extent of 1, 1e-30 above one, and both
# next to a plane inside.
@pytest.mark.parametrize("lo,hi", [(-1e-30, 1.0), (-1.0, 1e-30), (-1e-30, 1e-30), (-1e-38, 3.0), (-7e4, 1e-20),
                                   (-1e-45, 1e9), (1e-30, 2.0), (-3.0, -1e-30)])
def test_planes_enclose_bounds_next_to_zero(lo, hi):
    inner = np.float32((lo + hi) / 2)
    a = np.array([[lo, lo, np.float32(-1e-30) if lo < -1e-30 < hi else lo, inner]] * 3, np.float32)
    b = np.array([[hi, inner, hi, np.float32(1e-30) if inner < 1e-30 < hi else hi]] * 3, np.float32)
    base, step, words = pack(a, b, [1, 2, 3, 4])
    for ax in range(3):
        for c in range(4):
            (pl, ph), _ = planes(base, step, words, ax, c)
            assert pl <= Fraction(float(a[ax, c])) and ph >= Fraction(float(b[ax, c])), (ax, c)


@pytest.mark.parametrize("bad", [np.inf, np.nan, 3e38])
def test_axes_without_a_grid_bound_nothing(bad):
    lo = np.zeros((3, 4), np.float32)
    hi = np.ones((3, 4), np.float32)
    lo[1, 2], hi[1, 2] = -bad, bad
    base, step, words = pack(lo, hi, [1, 2, 3, -4])
    if np.isnan(bad):  # an empty box: the node's own bounds for it
        (pl, ph), _ = planes(base, step, words, 1, 2)
        assert pl <= 0 and ph >= 1
    else:
        # base + step * f is -inf + inf: NaN, which min / max pass over.
        assert np.isneginf(base[1]) and np.isposinf(step[1])
    for ax in (0, 2):
        (pl, ph), _ = planes(base, step, words, ax, 2)
        assert pl <= 0 and ph >= 1
