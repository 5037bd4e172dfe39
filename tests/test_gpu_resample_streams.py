"""Resampling of one shape on several streams and from several threads at a time: the transforms of a shape share a
cuFFT plan with one work area, which lengths with a large prime factor use.  Results are the bits of calls that wait
for each other."""
import ctypes
import threading

import numpy as np
import pytest
import torch

from sarsolver_gb300 import _lib
from sarsolver_gb300 import resample as rs
from sarsolver_gb300.geometry import NumpySimpleSarAperture, NumpySimpleSarDataset

pytestmark = pytest.mark.gpu
SHAPES = [(400, 4096, 2039), (700, 1201, 601), (300, 1999, 1999)]   # pulses, samples, kept samples (primes)


@pytest.fixture(scope="module", autouse=True)
def cuda_required():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def history(S, N, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.complex(torch.randn(S, N, device="cuda", generator=g), torch.randn(S, N, device="cuda", generator=g))


@pytest.mark.parametrize("S,N,n", SHAPES)
def test_two_streams_queued_together(S, N, n):
    lib = _lib.load()
    taps = rs.get_downsample_kernel(1)
    ktab = np.ascontiguousarray(np.stack([taps.real, taps.imag], axis=-1).astype(np.float64))
    win = rs.downsample_window(n, 1.2)
    row0 = np.arange(S - len(taps), dtype=np.int32)
    dr = np.linspace(-3.0, 3.0, S)
    need = lib.sar_resample_workspace(S, N, n, len(taps), len(row0))
    as_p = lambda a: a.ctypes.data_as(ctypes.c_void_p)

    def call(x, out, work, stream):
        _lib.check(lib.sar_resample_phase_history_ws(
            ctypes.c_void_p(x.data_ptr()), S, N, as_p(dr), 10.0e9, 200.0e6, 1.0, 299792458.0, n, as_p(win), as_p(ktab),
            len(taps), as_p(row0), len(row0), ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(work.data_ptr()), need,
            ctypes.c_void_p(stream.cuda_stream)), "sar_resample_phase_history_ws")

    streams = [torch.cuda.Stream() for _ in range(2)]
    xs = [history(S, N, 11 + k) for k in range(2)]
    outs, want = ([torch.zeros((len(row0), n), dtype=torch.complex64, device="cuda") for _ in range(2)] for _ in range(2))
    works = [torch.empty(need, dtype=torch.uint8, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    for k in range(2):
        call(xs[k], want[k], works[k], streams[k])
        torch.cuda.synchronize()
    for _ in range(20):
        for k in range(2):
            call(xs[k], outs[k], works[k], streams[k])
    torch.cuda.synchronize()
    assert all(torch.equal(outs[k], want[k]) for k in range(2))


def test_two_threads():
    S, N, n = SHAPES[1]
    az = np.deg2rad(np.linspace(-2, 2, S))
    tx = np.stack([10e3 * np.cos(az), 10e3 * np.sin(az), np.full(S, 5e3)], axis=-1)
    ap = NumpySimpleSarAperture(tx, tx.copy(), np.zeros((S, 3)), 10.0e9, 200.0e6, num_freqs=N)
    sets = [NumpySimpleSarDataset(ap, history(S, N, 21 + k)) for k in range(2)]
    fast = N / (n - 0.5)   # int(1 + N / fast) = n
    step = lambda k: rs.resample_dataset(sets[k], fast, 1, new_srp=np.array([5.0, 5.0, 0.0]), keep_on_device=True).phase_history()
    want = [step(k).clone() for k in range(2)]
    torch.cuda.synchronize()
    assert want[0].shape[1] == n
    bad = []

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                got = step(k)
                torch.cuda.current_stream().synchronize()
                if not torch.equal(got, want[k]):
                    bad.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_result_on_device_is_finished():
    """The tensor that resample_dataset leaves on the device can be read on any stream once the call has returned."""
    S = N = 8192   # milliseconds of device work, against some 0.3 ms of host work after its launch
    tx = np.stack([np.full(S, 9e3), np.linspace(-300, 300, S), np.full(S, 4e3)], axis=-1)
    ap = NumpySimpleSarAperture(tx, tx.copy(), np.zeros((S, 3)), 10.0e9, 200.0e6, num_freqs=N)
    ds = NumpySimpleSarDataset(ap, history(S, N, 31))
    with torch.cuda.stream(torch.cuda.Stream()):
        for _ in range(3):
            rs.resample_dataset(ds, 1.0, 1, new_srp=np.array([5.0, 5.0, 0.0]), keep_on_device=True)
            assert torch.cuda.current_stream().query()
