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


@pytest.mark.parametrize("S,N,fast", [(65542, 64, 1.7), (140000, 31, 1.0), (66000, 512, 8.0)])
def test_resampling_beyond_grid_limit(S, N, fast):
    """More than 65535 output pulses: several chunks of work rows, and the fused kernel.  2e-6 as the other resampling
    tests (rounding of two FP32 transforms)."""
    from oracle import resample as ora
    from sarsolver_gb300 import resample as rs
    from sarsolver_gb300.geometry import NumpySimpleSarAperture, NumpySimpleSarDataset
    rng = np.random.default_rng(S + N)
    tx = np.stack([np.full(S, 9e3), np.linspace(-300, 300, S), np.full(S, 4e3)], axis=-1)
    ph = crandn(rng, S, N).astype(np.complex64)
    ap = NumpySimpleSarAperture(tx, tx.copy(), np.zeros((S, 3)), 10e9, 200e6, num_freqs=N)
    new = np.array([20.0, -10.0, 0.0])
    out = rs.resample_dataset(NumpySimpleSarDataset(ap, ph), fast, 1, new_srp=new).phase_history()
    taps = ora.downsample_kernel(1)
    T = S - len(taps) - 1
    moved = ora.move_srps(ph, np.zeros((S, 3)), new, tx, tx, 10e9, 200e6)
    down = ora.fast_freq_downsample(moved, min(int(1.0 + N / fast), N), 1.2)
    want = sum(taps[k] * down[k:k + T] for k in range(len(taps)))
    assert out.shape == want.shape and T > 65535
    assert rel_l2(out, want) < 2.0e-6
