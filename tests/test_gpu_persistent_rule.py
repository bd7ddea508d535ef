"""Which FP64 meshes run in the many-steps kernel: those whose tiles of 32 elements
have a place on the GPU at once, but at order 3 in 3-D only up to a tile per SM (with
two on some SMs it is the slower one). Its residuals are summed tile by tile, so that
they end in other bits than those of the launches per stage."""
import numpy as np
import pytest

from conftest import smooth_state
from test_gpu_bernstein import BB, _sized
from test_gpu_parity import _phys
from test_gpu_persistent import PERSIST

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,per_sm,taken", [(3, 0.9, True), (3, 1.5, False), (2, 1.5, True), (1, 2.5, True)])
def test_run_by_tiles_per_sm(pkg, p, per_sm, taken):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    k = 9
    mesh = _sized(pkg, 3, p, (k, k, max(1, int(per_sm * sms * 32 // (6 * k * k)))))
    assert ((mesh["elem_nodes"].shape[0] + 31) // 32 > sms) == (per_sm > 1)
    S = pkg.gpu.Solver(mesh, precision=pkg.gpu.DG_FP64, **_phys(3))
    v, u0 = S.info()["kernel_variant"], smooth_state(mesh, seed=1)
    assert v >= PERSIST
    out = []
    for variant in (v, v - PERSIST + BB):
        S.tune(variant)
        S.set_state(u0)
        S.snapshot()
        S.step = 0
        out.append((S.run(20, 1e-6)[0], S.get_state()))
    S.close()
    assert np.array_equal(out[0][0], out[1][0]) == (not taken)
    np.testing.assert_allclose(out[0][0], out[1][0], rtol=1e-10)
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=0, atol=1e-12)
