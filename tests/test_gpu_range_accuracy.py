"""Rounding error of the range-profile transforms against the FP64 oracle, on data that complex64 holds exactly."""
import numpy as np
import pytest
import torch

import oracle
from cases import rel_l2, spotlight_case
from sarsolver_gb300 import SarPlan

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def cuda_required():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def upsampling_error(samples, U, n, spacing, pulses=6):
    case = spotlight_case(pulses, samples, n, spacing, 3.0, upsample=float(U))
    plan = SarPlan(case.scene, case.aperture, upsample_ratio=float(U), interp="linear", path="grid")
    rng = np.random.default_rng(samples)
    y = (rng.standard_normal((pulses, samples)) + 1j * rng.standard_normal((pulses, samples))).astype(np.complex64)
    full = oracle.upsample(case.problem(), y.astype(np.complex128))
    bins = (plan.profile_first_bin + np.arange(plan.profile_length)) % full.shape[1]
    return rel_l2(plan.profiles(torch.from_numpy(y)).cpu().numpy(), full[:, bins])


def downsampling_error(samples, U, n, spacing, pulses=6):
    """One pixel and nearest bins: a pulse's accumulator row holds one value, and what that value's own error does (one
    factor a row) is taken out."""
    case = spotlight_case(pulses, samples, n, spacing, 3.0, upsample=float(U))
    plan = SarPlan(case.scene, case.aperture, upsample_ratio=float(U), interp="nearest_ref", path="grid")
    x = np.zeros(n * n, np.complex64)
    x[n * n // 3] = 1.0
    got = plan.forward(torch.from_numpy(x)).cpu().numpy().astype(np.complex128)
    want = oracle.forward(case.problem(), x.astype(np.complex128), "nearest_ref", threads=8)
    scale = (want.conj() * got).sum(axis=1) / (np.abs(want) ** 2).sum(axis=1)
    return rel_l2(got, scale[:, None] * want)


@pytest.mark.parametrize("samples,U", [(512, 8), (512, 128), (1024, 8), (2048, 8), (4096, 8), (8192, 8), (8192, 16), (2048, 34)])
def test_fused_upsampling(samples, U):
    """Some 4.5e-8 a level of independent roundings (an addition, half a twiddle), 14 levels at most: 1.7e-7."""
    assert upsampling_error(samples, U, 64 if U < 34 else 32, 0.5 if U < 100 else 0.25) < 2.0e-7


@pytest.mark.parametrize("samples", [512, 1024, 2048, 4096, 8192])
def test_fused_downsampling(samples):
    """Few values to add; a dozen twiddles and products of 3e-8 each: 1.0e-7."""
    assert downsampling_error(samples, 8, 64, 0.5) < 1.1e-7


DOUBLE = [(251, 8, 48, 0.5), (251, 128, 40, 0.25), (333, 22, 20, 0.5), (300, 22, 40, 0.5), (999, 4, 64, 0.5), (1999, 8, 64, 0.5),
          (1999, 128, 33, 0.25), (500, 26, 33, 0.5)]


@pytest.mark.parametrize("samples,U,n,spacing", DOUBLE + [(512, 22, 40, 0.5), (512, 22, 1200, 0.25), (2048, 34, 32, 0.5)])
def test_complex128_upsampling(samples, U, n, spacing):
    """Lengths U N with a prime factor above 7: transformed and filtered in 64 bits and rounded once, 2.5e-8 rms (uniform
    in a unit of the last place of 6e-8 to 1.2e-7 relative); 4e-8 leaves room for the window's 1e-9 and nothing more.  Also
    where N has a fused kernel, which only the projections use."""
    assert upsampling_error(samples, U, n, spacing) < 4.0e-8


@pytest.mark.parametrize("samples,U,n,spacing", DOUBLE)
def test_complex128_downsampling(samples, U, n, spacing):
    """The same in the other direction: one rounding of the result (the pulse factors are 1)."""
    assert downsampling_error(samples, U, n, spacing) < 4.0e-8
