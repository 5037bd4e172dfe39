"""Nearest-bin sampling on the grid kernels (and linear sampling with bins split into integer and fraction, which
shares the gather) against the per-pixel path, which decides every bin exactly: narrow and
wide windows (upsample 8 and 128), looks along the grid axes and between them, ragged images and pulse counts, several
planes, bistatic pulses, short range, and geometries that put every sample within 5e-5 bins of a rounding boundary
(every note of the exact re-decision queues taken, and overflowing).  Tolerance: the operator's own, 1e-5 relative
L2; a single other bin would show as 1e-4 or more."""
import numpy as np
import pytest
import torch

from cases import Case, crandn, rel_l2, spotlight
from sarsolver_gb300 import SarPlan
from sarsolver_gb300.geometry import C, GridSarScene, NumpySimpleSarAperture

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def cuda_required():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def check(case, upsample, rng, interp="nearest_ref"):
    plan = SarPlan(case.scene, case.aperture, upsample_ratio=upsample, interp=interp, path="grid")
    general = SarPlan(case.scene, case.aperture, upsample_ratio=upsample, interp=interp, path="points")
    x = crandn(rng, case.scene.num_scatterers)
    y = crandn(rng, case.aperture.num_slow_times, case.aperture.num_freqs)
    x, y = torch.from_numpy(x), torch.from_numpy(y)
    assert rel_l2(plan.forward(x).cpu().numpy(), general.forward(x).cpu().numpy()) < 1.0e-5
    assert rel_l2(plan.adjoint(y).cpu().numpy(), general.adjoint(y).cpu().numpy()) < 1.0e-5
    assert plan.device_flags() == 0


@pytest.mark.parametrize("interp,upsample", [("nearest_ref", 8.0), ("nearest_ref", 128.0), ("linear", 64.0)])
@pytest.mark.parametrize("az,shape,spacing,pulses,degrees,bistatic,radius", [
    (0.0, (1, 33, 97), 0.25, 33, 3.0, False, 10.0e3), (90.0, (1, 97, 33), 0.25, 31, 3.0, False, 10.0e3),
    (45.0, (1, 70, 70), 0.25, 40, 2.0, False, 10.0e3), (63.0, (1, 100, 177), 0.25, 129, 2.0, False, 10.0e3),
    (153.0, (2, 31, 98), 0.25, 64, 2.0, False, 10.0e3), (14.0, (1, 84, 74), 0.3, 50, 4.0, True, 10.0e3),
    (20.0, (1, 1, 200), 0.5, 5, 1.0, False, 10.0e3), (70.0, (3, 66, 1), 0.5, 1, 1.0, False, 10.0e3),
    (33.0, (1, 70, 80), 0.9, 20, 3.0, False, 10.0e3), (10.0, (1, 78, 88), 0.25, 40, 60.0, False, 2.0e3),
    (0.0, (1, 150, 140), 0.3, 530, 3.0, False, 10.0e3),
    (33.0, (1, 260, 140), 0.3, 37, 3.0, False, 10.0e3), (60.0, (1, 140, 290), 0.5, 21, 3.0, True, 10.0e3),   # wide windows
    (5.0, (1, 300, 40), 0.15, 90, 2.0, False, 10.0e3)])
def test_grid_matches_points(az, shape, spacing, pulses, degrees, bistatic, radius, interp, upsample):
    rng = np.random.default_rng(int(az) + pulses)
    tx = spotlight(pulses, degrees, radius, 0.5 * radius, az)
    rx = spotlight(pulses, 0.5 * degrees, 0.8 * radius, 0.3 * radius, az + 20.0) if bistatic else tx.copy()
    ap = NumpySimpleSarAperture(tx, rx, np.zeros((pulses, 3)), 10.0e9, 200.0e6, num_freqs=512,
                                slow_time_weighting=np.exp(1j * rng.uniform(-3, 3, pulses)))
    dims = [2.0 * (shape[0] - 1), spacing * (shape[1] - 1), spacing * (shape[2] - 1)]
    check(Case(GridSarScene(list(shape), dims), ap, upsample, {}), upsample, rng, interp)


@pytest.mark.parametrize("upsample,step", [(8.0, 1), (8.0, 3), (128.0, 16), (128.0, 37)])
@pytest.mark.parametrize("along", [0, 1])
def test_every_sample_near_a_boundary(along, upsample, step):
    """Pixels a whole number of bins apart along the look direction, seen from 100 km, where the wave fronts are
    flat to 3e-5 bins across the image; the reference ranges put the image's pixels 1e-5 to 5e-5 bins above or below
    a boundary (the grid kernels' double-float ranges resolve 2e-7 bins there)."""
    rng = np.random.default_rng(step)
    fs, n, pulses = 200.0e6, 512, 20
    bin_m = C / (2.0 * fs * upsample)
    look = np.zeros(3)
    look[along] = 1.0
    tx = np.tile(1.0e5 * look, (pulses, 1))
    off = np.where(np.arange(pulses) % 2, 0.5 + 1.0e-5, 0.5 - 5.0e-5) * bin_m
    srp = off[:, None] * look[None, :]
    ap = NumpySimpleSarAperture(tx, tx.copy(), srp, 10.0e9, fs, num_freqs=n,
                                slow_time_weighting=np.exp(1j * rng.uniform(-3, 3, pulses)))
    spacing = [0.004, 0.004]
    spacing[along] = step * bin_m
    scene = GridSarScene([1, 65, 97], [0.0, spacing[1] * 64, spacing[0] * 96])
    check(Case(scene, ap, upsample, {}), upsample, rng)


@pytest.mark.parametrize("interp,upsample,pulses,az,shape,degrees,n", [
    ("linear", 3.0, 159, 309.0, (1, 241, 184), 28.5, 512), ("linear", 64.0, 53, 22.0, (1, 50, 92), 13.1, 256),
    ("nearest_ref", 4.0, 45, 124.0, (2, 225, 52), 10.7, 500)])
def test_coarse_pixels_at_short_range(interp, upsample, pulses, az, shape, degrees, n):
    """0.8 m pixels at 2 km, where third-order expansions about 16 x 16 pixels leave up to d^4 / (4 R^3) = 1.9e-6 m of
    range (d = 8 x 1.6 m, R = 1.5 km), 4e-4 rad, a twentieth of it (2e-5) in the mean over a block: lattices with longer
    steps would leave more, and are not taken there."""
    rng = np.random.default_rng(pulses)
    tx = spotlight(pulses, degrees, 2.0e3, 1.0e3, az)
    rx = spotlight(pulses, 0.5 * degrees, 1.6e3, 0.6e3, az + 20.0)
    ap = NumpySimpleSarAperture(tx, rx, 0.1 * rng.normal(size=(pulses, 3)), 10.0e9, 200.0e6, num_freqs=n)
    scene = GridSarScene(list(shape), [2.0 * (shape[0] - 1), 0.8 * (shape[1] - 1), 0.8 * (shape[2] - 1)])
    plan, general = (SarPlan(scene, ap, upsample_ratio=upsample, interp=interp, path=p) for p in ("grid", "points"))
    x = torch.from_numpy(crandn(rng, scene.num_scatterers))
    y = torch.from_numpy(crandn(rng, pulses, n))
    assert rel_l2(plan.forward(x).cpu().numpy(), general.forward(x).cpu().numpy()) < 2.0e-5
    assert rel_l2(plan.adjoint(y).cpu().numpy(), general.adjoint(y).cpu().numpy()) < 2.0e-5
    assert plan.device_flags() == 0


@pytest.mark.parametrize("spacing", [0.1, 0.107, 0.114, 0.121, 0.128, 0.135, 0.142, 0.149])
@pytest.mark.parametrize("shape,az", [((1, 241, 53), 355.0), ((2, 127, 38), 44.0)])
def test_narrow_windows(shape, az, spacing):
    """Fine pixels seen from afar, where the host's bound of a tile's bins is tight: windows that end wherever the
    spacing has it, at up to a whole bin from the bound, hold every nearest bin of pulses with any range offset."""
    rng = np.random.default_rng(round(1000 * spacing))
    tx = spotlight(200, 17.0, 5.0e4, 2.5e4, az)
    rx = spotlight(200, 8.5, 4.0e4, 1.5e4, az + 20.0)
    ap = NumpySimpleSarAperture(tx, rx, rng.normal(size=(200, 3)), 10.0e9, 200.0e6, num_freqs=256)
    scene = GridSarScene(list(shape), [2.0 * (shape[0] - 1), spacing * (shape[1] - 1), spacing * (shape[2] - 1)])
    check(Case(scene, ap, 1.0, {}), 1.0, rng)
