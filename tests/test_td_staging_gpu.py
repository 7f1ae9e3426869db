"""GPU tests of the small host calls that move their inputs and their outputs
in one staged copy each (up to 32,768 doubles): the sizes on both sides of
each limit against one large, unstaged call; without pinned memory the same
results."""
import ctypes

import numpy as np
import pytest

from helpers import assert_parity

pytestmark = pytest.mark.gpu
N = 8
IN, OUT = 10890, 151   # last M with 3M + 12N <= 32768, and with 27 N M <= 32768


@pytest.fixture(scope="module")
def data():
    rng = np.random.default_rng(5)
    P = [rng.uniform([-1, -1, -2], [1, 1, -1], (N, 3)) for _ in range(3)]
    pts = rng.uniform([-3, -3, -3], [3, 3, -0.1], (IN + 1, 3))
    return P, rng.uniform(-1, 1, (3, N)), pts


def _inf(cad, data, M, disp=1, strain=1, hs=1):
    P, sl, pts = data
    S, U = cad.TD(*pts[:M].T, *P, *sl, 0.25, 1.0, disp, strain, hs)
    return list(S) * (strain == 1) + list(U) * (disp == 1)


@pytest.mark.parametrize("M", [1, OUT, OUT + 1, IN])
def test_influence_around_the_limits(cad, data, M):
    for flags in ((1, 1), (0, 1), (1, 0)):
        for a, b in zip(_inf(cad, data, M, *flags), _inf(cad, data, IN + 1, *flags)):
            assert a.shape == (M, N) and np.array_equal(a, b[:M])


@pytest.mark.parametrize("M", [1, 3640, 3641, IN])   # 9 M doubles out: staged up to 3640
def test_sums_around_the_limits(cad, data, M):
    P, sl, pts = data

    def run(M, disp=1, strain=1):
        S, U = cad.TD(*pts[:M].T, *P, *sl, 0.25, 1.0, disp, strain, 0, cad.Strains(), cad.Disps())
        return list(S) * (strain == 1) + list(U) * (disp == 1)

    # other numbers of points sum the triangles in other chunks, and the
    # kernels of one kind of field round otherwise than those of both
    whole = [b[:M] for b in run(IN + 1)]
    for part in (run(M), run(M, disp=0) + run(M, strain=0)):
        assert_parity(np.stack(part[:6]), np.stack(whole[:6]))
        assert_parity(np.stack(part[6:]), np.stack(whole[6:]))


def test_without_pinned_memory(cad, data, fresh_context):
    from cutanddisplacejulia_b200 import _lib
    L = _lib.load()
    want = _inf(cad, data, OUT)                # with it, in the test's own context
    other = ctypes.c_void_p()
    _lib.check(L.cad_init(0, ctypes.byref(other)), None)
    _lib._ctx[0] = other
    try:
        _lib.check(L.cad_fail_allocation(other, 3), other)   # after the inputs' and the outputs' workspaces
        got = _inf(cad, data, OUT)
    finally:
        _lib._ctx[0] = fresh_context
        L.cad_destroy(other)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
