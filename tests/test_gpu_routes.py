"""Which kernels a plan runs, and the tile kernels behind the plans that walk no lattice along iso-range lines, against
the per-pixel path (1e-5 relative L2, the operator's own tolerance)."""
import numpy as np
import pytest
import torch

from cases import crandn, rel_l2, spotlight
from sarsolver_gb300 import SarPlan
from sarsolver_gb300.geometry import GridSarScene, NumpySimpleSarAperture

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def cuda_required():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def make(pulses, shape, spacing, upsample, interp, az=0.0, samples=512, path="grid"):
    tx = spotlight(pulses, 3.0, centre_az_deg=az)
    ap = NumpySimpleSarAperture(tx, tx.copy(), np.zeros((pulses, 3)), 10.0e9, 200.0e6, num_freqs=samples)
    scene = GridSarScene([1] + list(shape), [0.0, spacing * (shape[0] - 1), spacing * (shape[1] - 1)])
    return SarPlan(scene, ap, upsample_ratio=upsample, interp=interp, path=path)


def test_lattices_are_reported():
    plan = make(64, (160, 160), 0.25, 8.0, "linear")
    assert plan.gather_lattice == ((1, 0), (0, 1)) and plan.scatter_lattice == ((1, 0), (0, 1))   # lines along y
    plan = make(64, (160, 160), 0.25, 8.0, "linear", az=90.0)
    assert plan.gather_lattice == ((0, 1), (1, 0)) and plan.scatter_lattice == ((0, 1), (1, 0))
    plan = make(64, (160, 160), 0.25, 8.0, "nearest_ref")   # lanes along the lines, no lattice forwards
    assert plan.gather_lattice == ((0, 1), (1, 0)) and plan.scatter_lattice is None
    assert make(8, (40, 50), 0.25, 8.0, "linear", path="points").gather_lattice is None


@pytest.mark.parametrize("shape,spacing,upsample,interp,gather", [
    ((40, 300), 0.25, 8.0, "linear", True),          # two tile strips across: the forward's tile kernel
    ((90, 70), 3.0, 128.0, "nearest_ref", False),    # fourth-order terms of the range: the backprojection's too
    ((70, 90), 3.0, 64.0, "linear", False)])
def test_tile_kernels(shape, spacing, upsample, interp, gather):
    rng = np.random.default_rng(shape[0])
    # shown along an axis across the short side: the scatter's strips run along the long one
    plan = make(40, shape, spacing, upsample, interp, az=90.0, samples=1024)
    general = make(40, shape, spacing, upsample, interp, az=90.0, samples=1024, path="points")
    assert plan.is_grid and plan.scatter_lattice is None and (plan.gather_lattice is not None) == gather
    x = torch.from_numpy(crandn(rng, shape[0] * shape[1]))
    y = torch.from_numpy(crandn(rng, 40, 1024))
    assert rel_l2(plan.forward(x).cpu().numpy(), general.forward(x).cpu().numpy()) < 1.0e-5
    assert rel_l2(plan.adjoint(y).cpu().numpy(), general.adjoint(y).cpu().numpy()) < 1.0e-5
    assert plan.device_flags() == 0


@pytest.mark.parametrize("side,pulses,spacing,upsample,az,gather,scatter", [
    # (v, w): no runs along any line, so short windows of many lines, and lanes whose loads fall on few bins, come first
    (512, 1024, 0.5, 8.0, 50.0, ((0, 1), (1, 0)), ((1, 0), (-1, 1))),
    (512, 1024, 0.25, 8.0, 18.0, ((0, 1), (1, 0)), ((1, 0), (0, 1))),
    (512, 1024, 0.3, 16.0, 22.0, ((0, 1), (1, 0)), ((0, 1), (-1, 2))),
    (192, 400, 0.5, 8.0, 42.0, ((1, 0), (-1, 1)), ...),   # (forward: within 5 % on either kernel)
    (192, 400, 0.3, 16.0, 14.0, ((1, 0), (0, 1)), None)])   # the tile kernel: 46 us against 70
def test_lattices_of_oblique_looks(side, pulses, spacing, upsample, az, gather, scatter):
    """Measured with every lattice forced: with others the first forward projection took 2083 us for 429, the second
    backprojection 387 us for 286, the third 706 us for 334, the fourth 74 us for 48."""
    plan = make(pulses, (side, side), spacing, upsample, "linear", az=az, samples=1024)
    assert plan.gather_lattice == gather and scatter in (plan.scatter_lattice, ...)


@pytest.mark.parametrize("interp", ["linear", "nearest_ref"])
@pytest.mark.parametrize("az,pulses", [(22.0, 33), (30.0, 33), (22.0, 1030), (30.0, 1030), (0.0, 1030)])
def test_ring_windows(interp, az, pulses):
    """Ring windows with padding and without (22 and 30 degrees, where either spares most bank conflicts), 8 and 16 pulses
    a CTA (few pulses and many)."""
    rng = np.random.default_rng(pulses + int(az))
    plan = make(pulses, (100, 130), 0.3, 24.0 if az else 128.0, interp, az=az)
    general = make(pulses, (100, 130), 0.3, 24.0 if az else 128.0, interp, az=az, path="points")
    assert plan.scatter_ring_half > 0 and plan.scatter_lattice is None
    x = torch.from_numpy(crandn(rng, 13000))
    assert rel_l2(plan.forward(x).cpu().numpy(), general.forward(x).cpu().numpy()) < 1.0e-5
    assert plan.device_flags() == 0
