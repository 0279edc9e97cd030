"""FP64 batches, phase products and likelihood batches on a device that has memory
for their outputs and tables but none for the polynomial segments: the in-tile
kernels take every source, with the values that the segments give."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import emri_kludge_suite_b200 as E  # noqa: E402
from emri_kludge_suite_b200 import workloads  # noqa: E402
from test_gpu_packed_rows import _setup  # noqa: E402
from test_gpu_rows_no_memory import _handle  # noqa: E402

MB = 1 << 20


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    yield
    torch.cuda.empty_cache()


def _leave(nbytes):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info()[0] - int(nbytes), dtype=torch.uint8, device="cuda")


def _batch():
    """Ten sources of 2e6 samples (19540 tiles, 30 harmonics), one of them plunging, and a small one."""
    rng = np.random.default_rng(5)
    src = []
    for i, n in enumerate([2000003] * 10 + [5000]):
        p = workloads.draw_source(rng)
        rr = (p["M"] * workloads.MSUN_SEC) ** 2 / (p["mu"] * workloads.MSUN_SEC)
        end = 10.0 + 3.0 * p["e"]
        late = 0.5 if i == 3 else 2.0
        p.update(length=n, T=n * p["dt"] / workloads.YEAR,
                 p=max((end**4 + late * (256.0 / 5.0) * n * p["dt"] / rr) ** 0.25, 7.0))
        src.append(p)
    wb = E.WaveBatch(0)
    wb.plan(src, nmodes=[30] * len(src))
    assert np.all(wb.status == 0)
    wb.upload()
    return wb


def test_waveforms_without_memory_for_the_segments():
    want, wb = _batch(), _batch()
    N, tiles = wb.total_samples, sum(-(-int(n) // 1024) for n in np.diff(wb.offsets))
    a, b = (torch.empty((2, N), dtype=torch.float64, device="cuda") for _ in range(2))
    want.run(a[0].data_ptr(), a[1].data_ptr())
    assert want.launches() == 5  # the small source, segments, carries, direct tiles, waveform
    want.close()
    hog = _leave(tiles * 5 // 4 * (8160 + 64) + 40 * MB)  # tables and tile records, not 70 MB of segments
    wb.run(b[0].data_ptr(), b[1].data_ptr())
    torch.cuda.synchronize()
    assert wb.launches() == 1 and wb.device_status() == 0
    del hog
    torch.cuda.empty_cache()
    # the two FP64 kernels (the bar of the launch shapes' test)
    assert torch.max(torch.abs(a - b)) <= 1e-10 * torch.max(torch.abs(a))
    wb.upload()  # there is room again
    wb.run(b[0].data_ptr(), b[1].data_ptr())
    torch.cuda.synchronize()
    assert wb.launches() == 5 and torch.equal(a, b)


def test_phases_without_memory_for_the_segments():
    want, wb = _batch(), _batch()
    N = wb.total_samples
    a, b = (torch.empty((8, N), dtype=torch.float64, device="cuda") for _ in range(2))
    want.run_phase(a.data_ptr(), N)
    torch.cuda.synchronize()
    want.close()
    hog = _leave(20 * MB)  # tile records, not 40 MB of segments
    wb.run_phase(b.data_ptr(), N)
    torch.cuda.synchronize()
    assert wb.launches() == 3 and wb.device_status() == 0
    del hog
    torch.cuda.empty_cache()
    o = wb.offsets
    for s in range(wb.nsrc):  # the bars of the phase product against the oracle
        x, y = a[:, o[s]:o[s + 1]], b[:, o[s]:o[s + 1]]
        assert torch.equal(x[0], y[0])
        for k in (1, 2, 3):
            assert torch.max(torch.abs(x[k] - y[k])) <= 1e-11 * max(1.0, float(torch.max(torch.abs(x[k])))), (s, k)
        for k in (4, 5, 6, 7):
            assert torch.max(torch.abs(x[k] - y[k]) / torch.abs(x[k])) < 1e-12, (s, k)


def test_likelihoods_without_memory_for_the_segments():
    length, n = 1 << 18, 16
    g, X, w, D, _ = _setup(length, n)
    want = g.likelihood_batch(X, max_batch=n)
    g = _handle(w, D)
    before = torch.cuda.mem_get_info()[0]
    g.likelihood_batch(X, max_batch=n)
    used = before - torch.cuda.mem_get_info()[0]
    g = _handle(w, D)
    hog = _leave(used - n * (length // 1024) * 3600 * 5 // 4)
    out = g.likelihood_batch(X, max_batch=n)
    out2 = g.likelihood_batch(X, max_batch=n)
    del hog
    torch.cuda.empty_cache()
    assert np.max(np.abs(out - want)) <= 1e-9 * want[:, 1].max()  # as every launch shape
    assert np.max(np.abs(out2 - want)) <= 1e-9 * want[:, 1].max()
