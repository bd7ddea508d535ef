"""dg_set_observers on offsets that do not ascend: ranges that end where or
before they start hold nothing (their samples are 0/0), ranges beyond the lists are refused,
and the observers set before stay."""
import ctypes as C

import numpy as np
import pytest

from conftest import smooth_state
from test_gpu_bernstein import _sized
from test_gpu_parity import _phys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [64, -1])
@pytest.mark.parametrize("offsets,empty", [([0, -1], [True]), ([3, 0, -2], [True, True]), ([0, 4, 2, 4], [False, True, False]),
                                           ([2, 4], [False]), ([0, 5, 4], None), ([-1, 4], None), ([-3, -1, 2], None)])
def test_offsets(pkg, variant, offsets, empty):
    mesh = _sized(pkg, 2, 2, 5)
    S = pkg.gpu.Solver(mesh, precision=pkg.gpu.DG_FP64, **_phys(2))
    S.tune(variant)
    S.set_state(smooth_state(mesh, seed=2))
    S.set_observers([[7, 8]], [[1.0, 3.0]])
    want = S.run(2, 1e-30)[1]
    off = np.array(offsets, dtype=np.int64)
    dofs, w = np.array([7, 8, 7, 8, 9], dtype=np.int64), np.array([1.0, 3.0, 1.0, 3.0, 1.0])
    p = lambda a, t: a.ctypes.data_as(C.POINTER(t))  # noqa: E731
    n = len(off) - 1
    rc = pkg.gpu.lib().dg_set_observers(S.h, n, p(off, C.c_int64), p(dofs, C.c_int64), p(w, C.c_double))
    assert rc == (1 if empty is None else 0)
    if empty is not None:
        S.n_obs = n
    got = S.run(2, 1e-30)[1]
    if empty is None:
        assert np.array_equal(got, want)
    else:
        for o in range(n):
            if empty[o]:
                assert np.all(np.isnan(got[:, o]))
            else:  # the pair of the same nodes and weights, once or more often
                np.testing.assert_allclose(got[:, o], want[:, 0], rtol=1e-14, atol=0)
    S.close()
