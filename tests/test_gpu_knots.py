"""The two solves of a batch's spline coefficients (FP64 and split): launches of both
precisions on one upload, in any order, uncaptured or in a graph of the caller's, give
the samples of an upload of their own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import emri_kludge_suite_b200 as E  # noqa: E402
from emri_kludge_suite_b200 import workloads  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _batch():
    """Fast inspirals (M = 1e4 to 1e5) that run into their plunge, where a spline's curvature is large and the last bits
    of the two solves show in samples; a slow source, a small one."""
    rng = np.random.default_rng(2)
    src = []
    for n, M, mu in [(100000, 1e5, 100.0)] * 6 + [(150000, 1e4, 10.0)] * 3 + [(150000, 1e6, 10.0), (9000, 1e6, 10.0)]:
        p = workloads.draw_source(rng)
        p.update(M=M, mu=mu)
        rr = (M * workloads.MSUN_SEC) ** 2 / (mu * workloads.MSUN_SEC)
        end = 10.0 + 3.0 * p["e"]
        p.update(length=n, T=n * p["dt"] / workloads.YEAR,
                 p=min(max((end**4 + 0.9 * (256.0 / 5.0) * n * p["dt"] / rr) ** 0.25, 9.0), 80.0))
        src.append(p)
    wb = E.WaveBatch(0)
    wb.plan(src, nmodes=[12] * len(src))
    assert np.all(wb.status == 0)
    return wb


def _same(a, b):
    return torch.equal(torch.nan_to_num(a), torch.nan_to_num(b))


def _wave(wb, precision, graph=False, out=None):
    h = torch.empty((2, wb.total_samples), dtype=torch.float64, device="cuda") if out is None else out
    st = torch.cuda.current_stream().cuda_stream
    (wb.run_graph if graph else wb.run)(h[0].data_ptr(), h[1].data_ptr(), precision=precision, stream=st)
    return h


def _phase(wb):
    r = torch.empty((8, wb.total_samples), dtype=torch.float64, device="cuda")
    wb.run_phase(r.data_ptr(), wb.total_samples, stream=torch.cuda.current_stream().cuda_stream)
    return r


@pytest.fixture(scope="module")
def alone():
    """Each product from an upload of its own."""
    out = []
    for f in (lambda w: _wave(w, 0), lambda w: _wave(w, 1), _phase):
        wb = _batch()
        wb.upload()
        out.append(f(wb))
        torch.cuda.synchronize()
        assert wb.device_status() == 0
    return out


def test_precisions_in_turn_on_one_upload(alone):
    wb = _batch()
    wb.upload()
    for what in (0, 1, 0, 2, 1, 2, 0, 1):
        got = _phase(wb) if what == 2 else _wave(wb, what)
        assert _same(got, alone[what]), what
    for precision in (1, 0, 1):
        assert _same(_wave(wb, precision, graph=True), alone[precision])
        assert _same(_wave(wb, 1 - precision), alone[1 - precision])
    assert wb.device_status() == 0


def test_other_streams(alone):
    """Small and large sources beside one another on a stream that is not the default one."""
    wb = _batch()
    s = torch.cuda.Stream()
    wb.upload(s.cuda_stream)
    with torch.cuda.stream(s):
        got = [_wave(wb, 0), _wave(wb, 1), _phase(wb), _wave(wb, 0, graph=True)]
        s.synchronize()
    for g, w in zip(got, alone + alone[:1]):
        assert _same(g, w)


@pytest.mark.parametrize("precision", [0, 1])
def test_graphs_of_the_caller(alone, precision):
    wb = _batch()
    wb.upload()
    h = torch.empty((2, wb.total_samples), dtype=torch.float64, device="cuda")
    for p in (0, 1, 1 - precision):  # every buffer made; the next upload solves for the other precision
        _wave(wb, p, out=h)
    _phase(wb)
    wb.upload()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):  # the first launch in this precision since the upload
        _wave(wb, precision, out=h)
    # nothing of the capture has run: a launch beside it
    assert _same(_wave(wb, precision), alone[precision])
    for other in (None, 1 - precision, precision):
        if other is not None:
            assert _same(_wave(wb, other), alone[other])
        h.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert _same(h, alone[precision]), other
    # captured with its coefficients there, replayed after the other precision's launches
    g2 = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g2):
        _wave(wb, precision, out=h)
    assert _same(_wave(wb, 1 - precision), alone[1 - precision])
    h.zero_()
    g2.replay()
    torch.cuda.synchronize()
    assert _same(h, alone[precision])
