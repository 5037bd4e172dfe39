"""Unstructured scatterers with the pulses shared out over CTAs (point_parts) against the FP64 oracle: one pulse,
a stage, one more, several uneven shares; partial blocks of points; both samplings.  Tolerance: the operator's own."""
import numpy as np
import pytest
import torch

import oracle
from cases import Case, crandn, rel_l2, spotlight
from sarsolver_gb300 import SarPlan
from sarsolver_gb300.geometry import NumpySimpleSarAperture, SimpleSarScene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def cuda_required():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("mode", ["linear", "nearest_ref"])
@pytest.mark.parametrize("pulses,points", [(1, 1), (64, 257), (65, 256), (200, 300), (129, 5)])
def test_points_match_oracle(mode, pulses, points):
    rng = np.random.default_rng(pulses + points)
    tx = spotlight(pulses, 3.0)
    ap = NumpySimpleSarAperture(tx, tx.copy(), np.zeros((pulses, 3)), 10.0e9, 200.0e6, num_freqs=512,
                                slow_time_weighting=np.exp(1j * rng.uniform(-3, 3, pulses)))
    case = Case(SimpleSarScene(rng.uniform(-40.0, 40.0, (points, 3))), ap, 16.0, {})
    plan = SarPlan(case.scene, ap, upsample_ratio=16.0, interp=mode)
    y, x = crandn(rng, pulses, 512), crandn(rng, points)
    yd = torch.from_numpy(y).to(torch.complex64).cuda()
    got = plan.adjoint(yd)
    assert torch.equal(plan.adjoint(yd), got)
    assert rel_l2(got.cpu().numpy(), oracle.adjoint(case.problem(), y, mode, threads=8)) < 1.0e-5
    assert rel_l2(plan.forward(torch.from_numpy(x)).cpu().numpy(), oracle.forward(case.problem(), x, mode, threads=8)) < 1.0e-5
