"""Which FP64 meshes take the many-steps kernel by themselves: those whose tiles of
32 elements have a place on the GPU at once, at order 3 in 3-D an SM each (with two
on some SMs it is the slower one)."""
import pytest

from test_gpu_bernstein import _sized
from test_gpu_parity import _phys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,per_sm,taken", [(3, 0.9, True), (3, 1.5, False), (2, 1.5, True), (1, 2.5, True)])
def test_selection_by_tiles_per_sm(pkg, p, per_sm, taken):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    k = 9
    layers = max(1, int(per_sm * sms * 32 // (6 * k * k)))
    mesh = _sized(pkg, 3, p, (k, k, layers))
    tiles = (mesh["elem_nodes"].shape[0] + 31) // 32
    assert (tiles > sms) == (per_sm > 1)
    S = pkg.gpu.Solver(mesh, precision=pkg.gpu.DG_FP64, **_phys(3))
    assert (S.info()["kernel_variant"] >= 80) == taken
    assert (S.kernel_info(80)[0] > 0) == taken
    S.close()
