"""The forward scatter with a pulse per lane (linear sampling) against the FP64 oracle: every lattice direction,
ragged images and pulse counts, several planes, bistatic pulses, blocks of 16 to 2 lines, and runs of 16
pixels down to single pixels.  Tolerance: the operator's own, 1e-5 relative L2."""
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
    (63.0, (1, 100, 77), 0.25, 129, 2.0, False, 10.0e3), (117.0, (1, 77, 90), 0.25, 10, 2.0, False, 10.0e3),
    (135.0, (1, 17, 90), 0.25, 32, 2.0, False, 10.0e3), (153.0, (2, 31, 98), 0.25, 64, 2.0, False, 10.0e3),
    (14.0, (1, 84, 74), 0.3, 50, 4.0, True, 10.0e3),    # no lattice direction near: short runs, single pixels
    (0.0, (3, 16, 66), 0.5, 1, 0.0, False, 10.0e3), (20.0, (1, 1, 200), 0.5, 5, 1.0, False, 10.0e3),
    (70.0, (1, 200, 1), 0.5, 5, 1.0, False, 10.0e3),
    (33.0, (1, 70, 80), 0.75, 20, 3.0, False, 10.0e3),   # wide blocks: fewer lines
    (10.0, (1, 78, 88), 0.25, 40, 60.0, False, 2.0e3),   # a wide aperture at short range
    (0.0, (1, 40, 64), 0.25, 20, 3.0, False, 10.0e3)])   # two strips across: the tile kernel
def test_scatter_matches_oracle(az, shape, spacing, pulses, degrees, bistatic, radius):
    rng = np.random.default_rng(int(az) + pulses)
    tx = spotlight(pulses, degrees, radius, 0.5 * radius, az)
    rx = spotlight(pulses, 0.5 * degrees, 0.8 * radius, 0.3 * radius, az + 20.0) if bistatic else tx.copy()
    ap = NumpySimpleSarAperture(tx, rx, np.zeros((pulses, 3)), 10.0e9, 200.0e6, num_freqs=512,
                                slow_time_weighting=np.exp(1j * rng.uniform(-3, 3, pulses)))
    dims = [2.0 * (shape[0] - 1), spacing * (shape[1] - 1), spacing * (shape[2] - 1)]
    case = Case(GridSarScene(list(shape), dims), ap, 8.0, {})
    plan = SarPlan(case.scene, ap, upsample_ratio=8.0, interp="linear", path="grid")
    x = crandn(rng, case.scene.num_scatterers)
    got = plan.forward(torch.from_numpy(x)).cpu().numpy()
    assert rel_l2(got, oracle.forward(case.problem(), x, "linear", threads=8)) < 1.0e-5
    assert plan.device_flags() == 0


@pytest.mark.parametrize("interp", ["linear", "nearest_ref"])
@pytest.mark.parametrize("spacing,az", [(0.5, 0.0), (0.4, 20.0), (0.3, 45.0)])
def test_wide_tiles_forward(spacing, az, interp):
    """Tiles of more than 2048 bins at upsample 128: the forward projection runs per pixel, with phases in double-float
    that are rounded once (1e-7 rad of at most 2 pi: 1.8e-7 in the mean over random phases with the fold's and the
    transform's 1.5e-7 and the sums' 2e-7: 3e-7).  Bound: twice that; block expansions in FP32 leave 8e-7 and more."""
    rng = np.random.default_rng(int(az))
    tx = spotlight(60, 3.0, 1.0e4, 5.0e3, az)
    ap = NumpySimpleSarAperture(tx, tx.copy(), 0.1 * rng.normal(size=(60, 3)), 10.0e9, 200.0e6, num_freqs=1024)
    scene = GridSarScene([1, 110, 150], [0.0, spacing * 109, spacing * 149])
    case = Case(scene, ap, 128.0, {})
    plan = SarPlan(scene, ap, upsample_ratio=128.0, interp=interp, path="grid")
    x = crandn(rng, scene.num_scatterers)
    got = plan.forward(torch.from_numpy(x)).cpu().numpy()
    assert rel_l2(got, oracle.forward(case.problem(), x, interp, threads=8)) < 6.0e-7
    assert plan.device_flags() == 0
    streamed = SarPlan(scene, ap, upsample_ratio=128.0, interp=interp, path="grid", block_pulses=25)   # ring windows
    assert streamed.scatter_ring_half > 0 == plan.scatter_ring_half
    xd = torch.from_numpy(x).to(torch.complex64).cuda()
    assert rel_l2(streamed.forward(xd).cpu().numpy(), got) < 1.0e-5
    assert streamed.device_flags() == 0
