"""Collections of more than 65535 pulses, the largest gridDim.y, through the transforms whose kernels take a row each
there (sample counts off the fused lengths), against the FP64 oracle; the operator's tolerance, 1e-5."""
import numpy as np
import pytest
import torch

import oracle
from cases import crandn, rel_l2, spotlight_case
from sarsolver_gb300 import SarPlan

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def cuda_required():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("pulses,samples,U,block", [(70001, 100, 8, 0), (65536, 96, 4, 0), (66000, 64, 2, 0), (65600, 33, 3, 0),
                                                    (70001, 100, 8, 66000)])
def test_operator_beyond_grid_limit(pulses, samples, U, block):
    rng = np.random.default_rng(pulses + samples)
    case = spotlight_case(pulses, samples, 10, 0.5, 3.0, upsample=float(U))
    plan = SarPlan(case.scene, case.aperture, upsample_ratio=float(U), interp="linear", path="grid", block_pulses=block)
    y = crandn(rng, pulses, samples)
    assert rel_l2(plan.adjoint(torch.from_numpy(y)).cpu().numpy(), oracle.adjoint(case.problem(), y, "linear", threads=8)) < 1.0e-5
    x = crandn(rng, case.scene.num_scatterers)
    assert rel_l2(plan.forward(torch.from_numpy(x)).cpu().numpy(), oracle.forward(case.problem(), x, "linear", threads=8)) < 1.0e-5
    assert plan.device_flags() == 0
