"""Nearest-bin forward projections of images at most two lines of tiles across give the same bits every time: a bin of a
pulse gets one sum from each line, and two terms add up the same in either order.  Geometries that put most samples near a
rounding boundary, whose bins are decided again, from 100 km (flat wave fronts), with strip and with ring windows, and a
spotlight."""
import numpy as np
import pytest
import torch

from cases import crandn, rel_l2, spotlight
from sarsolver_gb300 import SarPlan
from sarsolver_gb300.geometry import C, GridSarScene, NumpySimpleSarAperture

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def cuda_required():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def repeated(scene, ap, upsample, rings):
    plan = SarPlan(scene, ap, upsample_ratio=upsample, interp="nearest_ref", path="grid")
    assert (plan.scatter_ring_half > 0) == rings and plan.scatter_lattice is None
    x = torch.from_numpy(crandn(np.random.default_rng(5), scene.num_scatterers)).cuda()
    first = plan.forward(x).clone()
    assert all(torch.equal(plan.forward(x), first) for _ in range(30))
    general = SarPlan(scene, ap, upsample_ratio=upsample, interp="nearest_ref", path="points")
    assert rel_l2(first.cpu().numpy(), general.forward(x).cpu().numpy()) < 1.0e-5 and plan.device_flags() == 0


@pytest.mark.parametrize("look,distance,shape,upsample,step,rings", [
    ((1, 0), 1.0e5, (700, 40), 8.0, (2, 0), False), ((0, 1), 1.0e5, (40, 700), 8.0, (0, 3), False),
    ((1, 0), 1.0e5, (500, 64), 128.0, (33, 0), False),
    ((1, 1), 1.0e6, (200, 64), 128.0, (21, 20), True), ((1, 1), 1.0e6, (64, 200), 128.0, (20, 21), True)])
def test_many_bins_decided_again(look, distance, shape, upsample, step, rings):
    """Pixels whole numbers of bins apart (x, y) along the look direction, 4 mm across it."""
    fs, n, pulses = 200.0e6, 512, 64
    bin_m = C / (2.0 * fs * upsample)
    u = np.array([look[0], look[1], 0.0]) / np.hypot(*look)
    tx = np.tile(distance * u, (pulses, 1))
    off = np.where(np.arange(pulses) % 2, 0.5 + 1.0e-5, 0.5 - 5.0e-5) * bin_m
    ap = NumpySimpleSarAperture(tx, tx.copy(), off[:, None] * u[None, :], 10.0e9, fs, num_freqs=n)
    sx, sy = (step[d] * bin_m / u[d] if step[d] else 0.004 for d in range(2))
    repeated(GridSarScene([1] + list(shape), [0.0, sy * (shape[0] - 1), sx * (shape[1] - 1)]), ap, upsample, rings)


@pytest.mark.parametrize("az,shape,upsample,pulses,rings", [(0.0, (1500, 33), 8.0, 600, False), (17.0, (2000, 50), 128.0, 300, True)])
def test_spotlight(az, shape, upsample, pulses, rings):
    tx = spotlight(pulses, 5.0, centre_az_deg=az)
    ap = NumpySimpleSarAperture(tx, tx.copy(), np.zeros((pulses, 3)), 10.0e9, 200.0e6, num_freqs=1024)
    repeated(GridSarScene([1] + list(shape), [0.0, 0.25 * (shape[0] - 1), 0.25 * (shape[1] - 1)]), ap, upsample, rings)
