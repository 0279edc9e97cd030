"""A likelihood batch that runs out of device memory, at every point where that
can happen: the call says so, and what GetWaveform returns afterwards is never a
spectrum in place of a waveform (or half-written rows)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from test_gpu_packed_rows import INJ, _setup  # noqa: E402

from emri_kludge_suite_b200._lib import AAKError  # noqa: E402
from emri_kludge_suite_b200.gpuAAK import GPUAAK  # noqa: E402

LENGTH, B = 1 << 18, 16


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _handle(w, D):
    g = GPUAAK(1.0, 100, LENGTH, 100.0, 10.0, True, False)
    g.input_data(D[0], D[1], w[0], w[1])
    return g


def test_rows_after_a_call_without_memory():
    g, X, w, D, _ = _setup(LENGTH, B)
    torch.cuda.synchronize()
    g2 = _handle(w, D)
    before = torch.cuda.mem_get_info()[0]
    full = g2.likelihood_batch(X, max_batch=B)
    used = before - torch.cuda.mem_get_info()[0]
    g2.gpu_gen_AAK(*X[0])
    h = g2.GetWaveform()[1:]
    spec = [np.fft.rfft(a[:LENGTH]) for a in h]
    del g, g2
    failed = 0
    for k in range(24):
        g = _handle(w, D)
        free = torch.cuda.mem_get_info()[0]
        hog = torch.empty(max(free - used * k // 24, 1), dtype=torch.uint8, device="cuda")
        try:
            out = g.likelihood_batch(X, max_batch=B)
        except AAKError:
            failed += 1
            out = None
        del hog
        torch.cuda.empty_cache()
        if out is not None:
            assert np.max(np.abs(out - full)) <= 1e-9 * full[:, 1].max(), k
        try:
            got = g.GetWaveform()[1:]
        except AAKError:
            assert out is None  # no template in the rows
            got = None
        for c in range(2) if got is not None else ():
            s = got[c][0::2] + 1j * got[c][1::2]
            is_spec = np.max(np.abs(s - spec[c])) <= 1e-10 * np.sum(np.abs(h[c]))
            if out is None:
                assert np.max(np.abs(got[c] - h[c])[:LENGTH]) <= 1e-10 * np.max(np.abs(h[c][:LENGTH])), (k, is_spec)
            else:
                assert is_spec, k
        # the handle goes on: a template of its own, and the batch
        g.gpu_gen_AAK(*INJ)
        assert np.array_equal(g.likelihood_batch(X, max_batch=B), full), k
    assert failed >= 3
