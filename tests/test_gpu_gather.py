"""The gather along iso-range lines (linear sampling) against the FP64 oracle: every lattice direction, ragged
images and pulse counts (odd last stages), several planes, bistatic pulses, wide windows, runs of 16 pixels down to
single pixels, one part and several; bitwise reproducible, also in pulse blocks that add onto the image.
Tolerance: the operator's own, 1e-5 relative L2."""
import numpy as np
import pytest
import torch

import oracle
from cases import Case, crandn, rel_l2, spotlight
from sarsolver_gb300 import SarPlan
from sarsolver_gb300.geometry import GridSarScene, NumpySimpleSarAperture

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def cuda_required():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("az,shape,spacing,pulses,degrees,bistatic,radius", [
    (0.0, (1, 33, 97), 0.25, 33, 3.0, False, 10.0e3), (90.0, (1, 97, 33), 0.25, 31, 3.0, False, 10.0e3),
    (27.0, (1, 65, 81), 0.25, 65, 2.0, False, 10.0e3), (45.0, (1, 70, 70), 0.25, 40, 2.0, False, 10.0e3),
    (63.0, (1, 200, 77), 0.25, 129, 2.0, False, 10.0e3), (117.0, (1, 77, 90), 0.25, 10, 2.0, False, 10.0e3),
    (135.0, (1, 17, 90), 0.25, 1, 2.0, False, 10.0e3), (153.0, (2, 31, 98), 0.25, 64, 2.0, False, 10.0e3),
    (14.0, (1, 84, 74), 0.3, 50, 4.0, True, 10.0e3),    # no lattice direction near: short runs, single pixels
    (0.0, (3, 16, 16), 0.5, 1, 0.0, False, 10.0e3), (0.0, (1, 1, 1), 0.5, 3, 1.0, False, 10.0e3),
    (20.0, (1, 1, 200), 0.5, 5, 1.0, False, 10.0e3), (70.0, (1, 200, 1), 0.5, 300, 1.0, False, 10.0e3),
    (33.0, (1, 70, 80), 0.75, 20, 3.0, False, 10.0e3),   # wide windows
    (10.0, (1, 78, 88), 0.25, 40, 60.0, False, 2.0e3)])  # a wide aperture at short range
def test_gather_matches_oracle(az, shape, spacing, pulses, degrees, bistatic, radius):
    rng = np.random.default_rng(int(az) + pulses)
    tx = spotlight(pulses, degrees, radius, 0.5 * radius, az)
    rx = spotlight(pulses, 0.5 * degrees, 0.8 * radius, 0.3 * radius, az + 20.0) if bistatic else tx.copy()
    ap = NumpySimpleSarAperture(tx, rx, np.zeros((pulses, 3)), 10.0e9, 200.0e6, num_freqs=512,
                                slow_time_weighting=np.exp(1j * rng.uniform(-3, 3, pulses)))
    dims = [2.0 * (shape[0] - 1), spacing * (shape[1] - 1), spacing * (shape[2] - 1)]
    case = Case(GridSarScene(list(shape), dims), ap, 8.0, {})
    plan = SarPlan(case.scene, ap, upsample_ratio=8.0, interp="linear", path="grid")
    y = crandn(rng, pulses, 512)
    yd = torch.from_numpy(y).to(torch.complex64).cuda()
    got = plan.adjoint(yd)
    assert rel_l2(got.cpu().numpy(), oracle.adjoint(case.problem(), y, "linear", threads=8)) < 1.0e-5
    assert torch.equal(plan.adjoint(yd), got)
    blocks = plan.adjoint_streamed(yd.cpu().pin_memory(), block=max(1, pulses // 3))
    assert rel_l2(blocks.cpu().numpy(), got.cpu().numpy()) < 5.0e-6
    assert torch.equal(plan.adjoint_streamed(yd.cpu().pin_memory(), block=max(1, pulses // 3)), blocks)
    assert plan.device_flags() == 0


@pytest.mark.parametrize("az,shape,spacing,pulses,degrees,bistatic,radius,n,upsample", [
    (62.0, (2, 200, 23), 0.8, 192, 20.0, False, 10.0e3, 1000, 3.0), (34.0, (1, 153, 248), 0.8, 165, 19.0, True, 50.0e3, 256, 1.0)])
def test_coarse_bins(az, shape, spacing, pulses, degrees, bistatic, radius, n, upsample):
    """Tiles of 128 pixels that span 140 bins and more, at an upsample where neighbouring bins differ by their own size: a
    bin's rounding counts in full.  Held in FP32 to the sub-tile's 16 bins at most it is 1e-6 (half a unit of 2^-20) at
    worst and half of that in the mean, as much as phases of up to two and a half turns (0.6e-6); to the tile's, four
    times as much.  Bound: 1.3e-6."""
    rng = np.random.default_rng(pulses)
    tx = spotlight(pulses, degrees, radius, 0.5 * radius, az)
    rx = spotlight(pulses, 0.5 * degrees, 0.8 * radius, 0.3 * radius, az + 20.0) if bistatic else tx.copy()
    ap = NumpySimpleSarAperture(tx, rx, 0.1 * rng.normal(size=(pulses, 3)), 10.0e9, 200.0e6, num_freqs=n)
    case = Case(GridSarScene(list(shape), [2.0 * (shape[0] - 1), spacing * (shape[1] - 1), spacing * (shape[2] - 1)]), ap, upsample, {})
    plan = SarPlan(case.scene, ap, upsample_ratio=upsample, interp="linear", path="grid")
    y = crandn(rng, pulses, n)
    got = plan.adjoint(torch.from_numpy(y)).cpu().numpy()
    assert rel_l2(got, oracle.adjoint(case.problem(), y, "linear", threads=8)) < 1.3e-6
    assert plan.device_flags() == 0


@pytest.mark.parametrize("az,shape,spacing,pulses,degrees,n,upsample", [
    (204.0, (2, 162, 251), 0.25, 86, 8.0, 256, 1.0), (16.0, (1, 151, 35), 0.25, 168, 30.0, 512, 3.0)])
def test_expansions_of_long_steps(az, shape, spacing, pulses, degrees, n, upsample):
    """Blocks of lattices with longer steps than the image's are not taken at a range (1.7 km) where their third-order
    expansions leave 6e-6 rad in a corner, 1.5e-6 of a block in the mean.  Without: phases of up to two and a half turns
    (0.6e-6), bins (0.5e-6) and the image's own blocks (0.7e-6), 1.1e-6 in all, and the forward scatter's sums (0.8e-6),
    1.4e-6."""
    rng = np.random.default_rng(pulses)
    tx = spotlight(pulses, degrees, 2.0e3, 1.0e3, az)
    rx = spotlight(pulses, 0.5 * degrees, 1.6e3, 0.6e3, az + 20.0)
    ap = NumpySimpleSarAperture(tx, rx, 0.1 * rng.normal(size=(pulses, 3)), 10.0e9, 200.0e6, num_freqs=n)
    case = Case(GridSarScene(list(shape), [2.0 * (shape[0] - 1), spacing * (shape[1] - 1), spacing * (shape[2] - 1)]), ap, upsample, {})
    plan = SarPlan(case.scene, ap, upsample_ratio=upsample, interp="linear", path="grid")
    x, y = crandn(rng, case.scene.num_scatterers), crandn(rng, pulses, n)
    got = plan.adjoint(torch.from_numpy(y)).cpu().numpy()
    assert rel_l2(got, oracle.adjoint(case.problem(), y, "linear", threads=8)) < 1.1e-6 * 1.2
    got = plan.forward(torch.from_numpy(x)).cpu().numpy()
    assert rel_l2(got, oracle.forward(case.problem(), x, "linear", threads=8)) < 1.4e-6 * 1.2
    assert plan.device_flags() == 0
