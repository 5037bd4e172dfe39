"""Range profiles through the base grid (2 N points and a ten-tap filter, sar_fir.cu) against the FP64
oracle: phases per base step that are and are not powers of two, odd and non-smooth sample counts, one
step and many, and the factors that stay on the other transforms (odd, or below 4).

Tolerance of the profiles: the filter passes 7e-10 of the images and FP32 rounds the base transform
and the ten-term sum to 2e-7 or so (2-norm); 1e-6 leaves a factor of five.  Projections: 1e-5, the
operator's own tolerance.
"""
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


@pytest.mark.parametrize("mode,pulses,samples,U,n,spacing", [
    ("linear", 5, 512, 4, 33, 0.5), ("nearest_ref", 3, 512, 6, 40, 0.5), ("linear", 1, 1024, 10, 64, 0.25),
    ("linear", 4, 2048, 34, 32, 0.5), ("nearest_ref", 7, 4096, 32, 50, 1.0), ("linear", 3, 8192, 16, 64, 0.5),
    ("linear", 9, 251, 8, 48, 0.5), ("nearest_ref", 6, 251, 128, 40, 0.25), ("linear", 5, 1000, 12, 65, 0.5),
    ("linear", 2, 333, 22, 20, 0.5), ("nearest_ref", 4, 2000, 128, 96, 0.3), ("linear", 3, 120, 8, 16, 0.1),
    ("linear", 4, 512, 5, 40, 0.5), ("linear", 4, 300, 7, 40, 0.5), ("linear", 4, 512, 2, 40, 0.5)])
def test_range_filter_matches_oracle(mode, pulses, samples, U, n, spacing):
    rng = np.random.default_rng(samples + U)
    case = spotlight_case(pulses, samples, n, spacing, 3.0, upsample=float(U),
                          weights=np.exp(1j * rng.uniform(-3, 3, pulses)))
    plan = SarPlan(case.scene, case.aperture, upsample_ratio=float(U), interp=mode, path="grid")
    y = crandn(rng, pulses, samples)
    full = oracle.upsample(case.problem(), y)
    bins = (plan.profile_first_bin + np.arange(plan.profile_length)) % full.shape[1]
    assert rel_l2(plan.profiles(torch.from_numpy(y)).cpu().numpy(), full[:, bins]) < 1.0e-6
    back = plan.adjoint(torch.from_numpy(y)).cpu().numpy()
    assert rel_l2(back, oracle.adjoint(case.problem(), y, mode, threads=8)) < 1.0e-5
    x = crandn(rng, case.scene.num_scatterers)
    ahead = plan.forward(torch.from_numpy(x)).cpu().numpy()
    assert rel_l2(ahead, oracle.forward(case.problem(), x, mode, threads=8)) < 1.0e-5
    assert plan.device_flags() == 0
