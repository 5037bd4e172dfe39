"""GPU dataset resampling against the reference's own outputs (tests/golden/resample_*.npz,
made by tests/golden/make_resample_golden.py from the reference's utils and
NumpySimpleSarDataset.from_resampling): SRP rephasing, fast-frequency downsampling, the full
resampling with a slow-time filter, odd N, sign -1, and a pulse with non-finite positions."""
import os

import numpy as np
import pytest
import torch

from sarsolver_gb300 import resample as rs
from sarsolver_gb300.geometry import NumpySimpleSarAperture, NumpySimpleSarDataset

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


@pytest.fixture(scope="module", autouse=True)
def cuda_required():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(np.asarray(b)))


@pytest.mark.parametrize("name", ["a", "b", "c"])
def test_resampling_matches_reference(name):
    d = dict(np.load(os.path.join(GOLDEN, f"resample_{name}.npz")))
    fc, fs, sign = float(d["centre_frequency"]), float(d["sample_frequency"]), float(d["sign_multiplier"])
    moved = rs.move_srps(d["ph"], d["srps"], d["new_srp"], d["tx"], d["rx"], fc, fs, sign)
    ok = np.isfinite(d["moved"]).all(axis=1)
    assert rel(moved[ok], d["moved"][ok]) < 1e-6
    ffd = rs.fast_freq_downsample(d["ph"], int(d["n_new"]), 1.2)
    assert rel(ffd, d["ffd"]) < 1e-6
    np.testing.assert_allclose(rs.get_downsample_kernel(max(int(d["slow_factor"]), 1)), d["kernel"], rtol=1e-6, atol=1e-7)
    ap = NumpySimpleSarAperture(d["tx"], d["rx"], d["srps"], fc, fs, waveform_fft=d["wave"],
                                slow_time_weighting=d["wt"], sign_multiplier=sign)
    amb = {}
    if float(d["range_amb"]) > 0:   # the reference chose the factors from ambiguous extents
        amb = dict(range_amb=float(d["range_amb"]), cross_range_amb=float(d["cross_range_amb"]))
    out = rs.resample_dataset(NumpySimpleSarDataset(ap, d["ph"]), fast_downsample_factor=float(d["fast_factor"]) or 1.0,
                              slow_downsample_factor=int(d["slow_factor"]) or 1, new_srp=d["new_srp"],
                              safety_factor=1.2, **amb)
    oap = out.aperture
    assert out.phase_history().shape == d["out_ph"].shape
    assert rel(out.phase_history(), d["out_ph"]) < 1e-5
    np.testing.assert_array_equal(oap.transmitter_positions, d["out_tx"])
    np.testing.assert_array_equal(oap.receiver_positions, d["out_rx"])
    np.testing.assert_allclose(oap.stab_ref_posns, d["out_srps"])
    np.testing.assert_allclose(oap.slow_time_weighting, d["out_wt"], rtol=1e-6)
    assert rel(oap.waveform_fft, d["out_wave"]) < 1e-6


def test_large_phase_ramps_stay_accurate():
    """Hundreds of turns of phase per pulse (a 600 m SRP move at 10 GHz): the device phase keeps
    FP64-level accuracy (split slope, FP64-reduced constant)."""
    rng = np.random.default_rng(3)
    S, N = 64, 2048
    az = np.deg2rad(np.linspace(-2, 2, S))
    tx = np.stack([10e3 * np.cos(az), 10e3 * np.sin(az), np.full(S, 5e3)], axis=-1)
    ph = (rng.standard_normal((S, N)) + 1j * rng.standard_normal((S, N))) / np.sqrt(2)
    old = np.zeros((S, 3))
    new = np.array([400.0, 450.0, 0.0])
    got = rs.move_srps(ph, old, new, tx, tx, 10e9, 200e6, 1.0)
    dr = rs.range_changes(old, new, tx, tx)[:, None]
    bb = np.fft.fftshift(np.fft.fftfreq(N, 1.0 / 200e6))[None, :]
    ref = ph * np.exp(2j * np.pi * dr / 299792458.0 * (bb - 10e9))
    assert np.abs(dr).max() > 300.0
    assert rel(got, ref) < 2e-6


def test_resampling_throughput_report():
    """8192 pulses x 8192 samples (0.5 GB complex64) resampled by 2 in both dimensions; prints the
    device time and the effective bandwidth of the HBM-bound passes."""
    import time
    rng = np.random.default_rng(5)
    S, N = 8192, 8192
    az = np.deg2rad(np.linspace(-3, 3, S))
    tx = np.stack([10e3 * np.cos(az), 10e3 * np.sin(az), np.full(S, 5e3)], axis=-1)
    ap = NumpySimpleSarAperture(tx, tx, np.zeros((S, 3)), 10e9, 200e6, num_freqs=N)
    ph = torch.complex(torch.randn(S, N, device="cuda"), torch.randn(S, N, device="cuda"))
    ds = NumpySimpleSarDataset(ap, ph)
    out = rs.resample_dataset(ds, 2.0, 2, new_srp=np.array([5.0, 5.0, 0.0]), keep_on_device=True)   # warm-up
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    out = rs.resample_dataset(ds, 2.0, 2, new_srp=np.array([5.0, 5.0, 0.0]), keep_on_device=True)
    e1.record()
    torch.cuda.synchronize()
    dt = time.perf_counter() - t0
    dev_ms = e0.elapsed_time(e1)
    T, n = out.phase_history().shape
    # passes over HBM: read S*N, write S*N, FFT S*N (read+write), crop read S*n + write S*n, FFT S*n,
    # filter reads 10 taps per output row (L2-resident rows) and writes T*n.
    moved = 8.0 * (2 * S * N + 2 * S * N + 2 * S * n + 2 * S * n + T * n)
    print(f"resample {S}x{N} -> {T}x{n}: {dt * 1e3:.2f} ms wall ({dev_ms:.2f} ms between events on the stream), "
          f"{moved / dt / 1e9:.0f} GB/s over the main passes")
    assert T > 0 and n == 4097


@pytest.mark.parametrize("S,N,fast,slow,move", [
    (16, 512, 1.7, 1, True), (40, 1024, 3.0, 3, True), (25, 2048, 1.0, 2, False), (12, 4096, 2.9, 1, True),
    (30, 8192, 2.0, 2, True), (33, 511, 1.3, 2, True), (20, 1000, 2.5, 1, True), (9, 17, 1.0, 1, True),
    (200, 300, 2.0, 12, True), (5000, 1200, 4.0, 1, True)])   # a filter of 60 taps; several chunks of work rows
def test_resampling_matches_oracle(S, N, fast, slow, move):
    """The filter before the transforms (fused for N = 512 ... 8192, chunked work rows otherwise) against the
    FP64 restatement: rounding of two FP32 transforms and L products, a few 1e-7; 2e-6 leaves a factor of five."""
    from oracle import resample as ora
    rng = np.random.default_rng(S + N)
    tx = np.stack([np.full(S, 9e3), np.linspace(-300, 300, S), np.full(S, 4e3)], axis=-1) + 0.1 * rng.standard_normal((S, 3))
    srps = rng.standard_normal((S, 3)) if move else np.zeros((S, 3))
    new = np.array([20.0, -10.0, 0.0]) if move else np.zeros(3)
    ph = rng.standard_normal((S, N)) + 1j * rng.standard_normal((S, N))
    wave, wt = rng.standard_normal(N) + 1j * rng.standard_normal(N), rng.standard_normal(S) + 0j
    ap = NumpySimpleSarAperture(tx, tx.copy(), srps, 10e9, 200e6, waveform_fft=wave, slow_time_weighting=wt)
    out = rs.resample_dataset(NumpySimpleSarDataset(ap, ph), fast, slow, new_srp=new)
    n = min(int(1.0 + N / fast), N)
    moved = ora.move_srps(ph, srps, new, tx, tx, 10e9, 200e6)
    down, taps = ora.fast_freq_downsample(moved, n, 1.2), ora.downsample_kernel(slow)
    L = len(taps)
    T = (S - L) // slow - 1
    want = np.stack([(taps[:, None] * down[slow * t:slow * t + L]).sum(axis=0) for t in range(T)])
    assert rel(out.phase_history(), want) < 2e-6
    assert rel(out.aperture.waveform_fft, ora.fast_freq_downsample(wave[None], n, 1.2)[0]) < 1e-6


@pytest.mark.parametrize("S,N,fast,slow", [(300, 1999, 1.9, 2), (300, 3000, 1.0, 2), (400, 1024, 1.9, 1), (200, 512, 1.3, 1),
                                           (300, 700, 2.0, 3), (300, 4096, 1.9, 2)])
def test_fused_rephasing_is_as_accurate_as_each_sample_rephased(S, N, fast, slow):
    """The filter's phase factors, products of two, against move_srps, which forms each sample's phase by itself, followed by
    the same resampling without a move: the error to the FP64 restatement may be no larger."""
    from oracle import resample as ora
    rng = np.random.default_rng(N)
    az = np.deg2rad(np.linspace(-2, 2, S))
    tx = np.stack([10e3 * np.cos(az), 10e3 * np.sin(az), np.full(S, 5e3)], axis=-1)
    old, new = 3.0 * rng.standard_normal((S, 3)), np.array([40.0, -25.0, 0.0])
    ph = ((rng.standard_normal((S, N)) + 1j * rng.standard_normal((S, N))) / np.sqrt(2)).astype(np.complex64)
    make = lambda srps, p: NumpySimpleSarDataset(NumpySimpleSarAperture(tx, tx.copy(), srps, 10e9, 200e6, num_freqs=N), p)
    news = np.repeat(new[None], S, axis=0)
    fused = rs.resample_dataset(make(old, ph), fast, slow, new_srp=new).phase_history()
    moved = rs.move_srps(torch.from_numpy(ph).cuda(), old, new, tx, tx, 10e9, 200e6)
    apart = rs.resample_dataset(make(news, moved), fast, slow, new_srp=new).phase_history()
    n, taps = min(int(1.0 + N / fast), N), ora.downsample_kernel(slow)
    down = ora.fast_freq_downsample(ora.move_srps(ph.astype(np.complex128), old, new, tx, tx, 10e9, 200e6), n, 1.2)
    T = (S - len(taps)) // slow - 1
    want = np.stack([(taps[:, None] * down[slow * t:slow * t + len(taps)]).sum(axis=0) for t in range(T)])
    assert rel(fused, want) <= rel(apart, want)
