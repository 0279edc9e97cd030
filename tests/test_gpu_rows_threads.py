"""One GPUAAK handle on several threads: GetWaveform after a batch turns the
packed rows into half spectra in place, once, and neither runs beside a batch."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from test_gpu_packed_rows import _setup  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _together(fs):
    gate, errors = threading.Barrier(len(fs)), []

    def go(f):
        gate.wait()
        try:
            f()
        except Exception as e:
            errors.append(e)

    ts = [threading.Thread(target=go, args=(f,)) for f in fs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors


def test_threads_read_the_same_half_spectrum():
    g, X, _, _, _ = _setup(1 << 17, 4)
    out = g.likelihood_batch(X)
    want = g.GetWaveform(is_Fourier=True)[1:]
    got = [None] * 4

    def read(k):
        got[k] = g.GetWaveform(is_Fourier=True)[1:]

    for _ in range(10):
        assert np.array_equal(g.likelihood_batch(X), out)
        _together([lambda k=k: read(k) for k in range(4)])
        for h in got:
            assert np.array_equal(h[0], want[0]) and np.array_equal(h[1], want[1])


def test_reading_beside_a_batch_leaves_its_products():
    g, X, _, _, _ = _setup(1 << 17, 8)
    out = g.likelihood_batch(X, max_batch=2)
    got = [None]

    def batch():
        got[0] = g.likelihood_batch(X, max_batch=2)

    for _ in range(10):
        _together([batch] + [lambda: g.GetWaveform(is_Fourier=True)] * 2)
        assert np.array_equal(got[0], out)
