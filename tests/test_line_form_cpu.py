"""Which plans the segmented line kernel takes, and how it cuts their lines: the
host side of the choice, without a device."""
import ctypes as C
import time

import pytest

import compactles_b200 as cl
from compactles_b200 import abi


def _form(ng, scheme, dim=1, periodic=False, dtype=abi.CLES_F64, count=6):
    per = tuple(1 if (k != dim - 1 or periodic) else 0 for k in range(3))
    info = (C.c_int * 4)()
    cl.api._check(cl.lib().cles_selftest_line_form(C.byref(cl.grid(ng, per)), C.byref(scheme), dim, dtype, count, info))
    return tuple(info)


SCHEMES = {"c6": cl.lele_d1_6, "c10": cl.lele_d1_10, "filter": lambda: cl.compact_filter(0.45), "pade": cl.pade_d1_4}


def _check(ng, scheme, periodic):
    n = ng[0]
    _, S, tile, blocks = _form(ng, scheme, periodic=periodic)
    assert 2 <= S <= 512 and n // S >= 9 and -(-n // S) <= tile <= 32, (ng, S, tile)
    assert n // S >= tile - 8 and 1 <= blocks <= 8, (ng, S, tile, blocks)


@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("periodic", [False, True])
def test_short_lines(scheme, periodic):
    """x lines from 18 points up, one line and some: at most 512 segments of nine
    points or more, within the register tile."""
    for n in range(18, 130):
        for lines in (1, 31):
            _check((n, lines, 1), SCHEMES[scheme](), periodic)


@pytest.mark.parametrize("n", [4096, 5712, 7936, 7937, 8191, 8192, 8193, 9001, 12288, 12289, 12800])
def test_long_lines(n):
    """Up to the longest x line a plan may have (a C10 plan's dense inverse takes
    seconds on the host there)."""
    for scheme in ("c6", "filter", "pade") + (("c10",) if n in (7937, 8192, 8193) else ()):
        for lines in (1, 3, 16, 31, 32):
            if scheme != "c10" or lines == 1:
                _check((n, lines, 1), SCHEMES[scheme](), False)


def test_lines_of_y_and_z():
    for dim in (2, 3):
        for n in (18, 35, 161, 8192, 8193, 12800):
            ng = tuple(n if k == dim - 1 else 1 for k in range(3))
            _, S, tile, _ = _form((3,) + ng[1:], cl.lele_d1_6(), dim=dim)
            assert 2 <= S <= 512 and n // S >= 9 and -(-n // S) <= tile <= 32


def test_long_tubes_spread_over_eight_blocks():
    assert _form((8192, 1, 1), cl.lele_d1_6())[1:] == (512, 16, 8)
    assert _form((5712, 1, 1), cl.lele_d1_6())[3] == 6


def test_what_other_kernels_serve():
    assert _form((17, 40, 1), cl.lele_d1_6())[1] == 0                        # too short for two segments
    assert _form((1000, 9, 9), cl.compact_filter(0.4995))[1] == 0            # decays too slowly
    assert _form((300, 9, 9), cl.compact_filter(0.4995))[1] > 0              # the window holds the line
    assert _form((256, 64, 64), cl.lele_d1_6(), periodic=True)[0] == 1       # warp per line


def test_schemes_without_a_line_form_are_refused_early():
    """A window past its limit ends the search for one: planning a filter that decays over
    thousands of points takes no longer than planning any other on the same lines (both
    spend 0.1 s on the generic form's interface inverse; the search used to go on to the
    inverse of the whole line, 1 s)."""
    def seconds(alpha, expect):
        best = 1e9
        for _ in range(3):
            t = time.perf_counter()
            form = _form((8192, 1, 1), cl.compact_filter(alpha), periodic=True)
            best = min(best, time.perf_counter() - t)
        assert (form[1] > 0) == expect
        return best
    assert seconds(0.49999, False) < 3 * seconds(0.45, True)


def test_bad_arguments_are_refused():
    info = (C.c_int * 4)()
    g, s = cl.grid((64, 1, 1), (0, 1, 1)), cl.lele_d1_6()
    call = cl.lib().cles_selftest_line_form
    assert call(None, C.byref(s), 1, abi.CLES_F64, 1, info) == abi.CLES_EINVAL
    assert call(C.byref(g), C.byref(s), 4, abi.CLES_F64, 1, info) == abi.CLES_EINVAL
    assert call(C.byref(g), C.byref(s), 1, abi.CLES_F64, 0, info) == abi.CLES_EINVAL
    assert call(C.byref(g), C.byref(s), 1, 7, 1, info) == abi.CLES_EINVAL
