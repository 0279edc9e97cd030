"""FP64 tiles that the polynomial segments do not serve (long time steps, the end of
a fast inspiral, phases past a plunge), against the oracle: as few of them as run
in quarters, as many as run in halves or whole, those without a Bessel table, and
rows of tiles whose Phidot clamp reaches back over tiles without a positive rate."""
import numpy as np
import pytest

from conftest import mismatch

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import emri_kludge_suite_b200 as E  # noqa: E402
from emri_kludge_suite_b200 import workloads  # noqa: E402
from oracle import oracle as O  # noqa: E402
from test_gpu_segments import BASE, _mapped  # noqa: E402

LONG = dict(dt=1000.0, p=18.0, mu=2.0)  # at 1000 s the response is not a polynomial of degree 7 over 256 samples


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    O.set_threads(8)
    yield
    O.set_threads(1)


def _fast(k):
    """Source k of a draw of fast inspirals (M = 1e5, mu = 100) that plunge before their span ends."""
    rng = np.random.default_rng(2)
    for _ in range(k + 1):
        q = workloads.draw_source(rng)
    q.update(M=1e5, mu=100.0)
    n, rr, end = 100000, (1e5 * workloads.MSUN_SEC) ** 2 / (100.0 * workloads.MSUN_SEC), 10.0 + 3.0 * q["e"]
    q.update(length=n, T=n * 10.0 / workloads.YEAR,
             p=min(max((end**4 + 0.9 * (256.0 / 5.0) * n * 10.0 / rr) ** 0.25, 9.0), 80.0))
    return q


def _run(pars, nm, phase=True):
    maps = [E.front_end(p) for p in pars]
    wb = E.WaveBatch(0)
    wb.plan(pars, nmodes=nm, mapped=maps)
    assert np.all(wb.status == 0)
    N = wb.total_samples
    h = torch.full((2, N), 7.0, dtype=torch.float64, device="cuda")
    rows = torch.full((8, N), 7.0, dtype=torch.float64, device="cuda")
    wb.upload()
    wb.run(h[0].data_ptr(), h[1].data_ptr())
    if phase:
        wb.run_phase(rows.data_ptr(), N)
    torch.cuda.synchronize()
    assert wb.device_status() == 0
    return wb, maps, h.cpu().numpy(), rows.cpu().numpy()


def _check_wave(pars, mp, nm, h):
    oI, oII = O.oracle_genwave(pars, _mapped(mp), nm)[1:3]
    scale = max(np.abs(oI).max(), np.abs(oII).max())
    # the bars of the FP64 path against the oracle (test_gpu_waveform.py)
    assert np.abs(h[0] - oI).max() <= 1e-8 * scale and np.abs(h[1] - oII).max() <= 1e-8 * scale
    assert mismatch(h[0], h[1], oI, oII) < 1e-12


def _check_phase(pars, mp, rows):
    ref = O.oracle_genphase(pars, _mapped(mp))
    assert np.array_equal(rows[0], ref[0])
    # the bars of the phase product (test_gpu_phase.py), the rates' of the largest: they pass through zero
    for k in (1, 2, 3):
        assert np.max(np.abs(rows[k] - ref[k])) <= 1e-11 * max(1.0, np.abs(ref[k]).max()), k
    for k in (4, 5, 6):
        assert np.max(np.abs(rows[k] - ref[k])) <= 1e-12 * np.abs(ref[k]).max(), k


# direct tiles in all: 60 a source, cut in quarters (at most 111 of them on 444 CTAs), halves (222), or whole
@pytest.mark.parametrize("nsrc,backint", [(1, False), (1, True), (3, False), (10, False)])
def test_long_steps(nsrc, backint):
    rng = np.random.default_rng(nsrc)
    pars = []
    for _ in range(nsrc):
        p = dict(BASE, **LONG, length=60 * 1024 - 77, backint=backint)
        p.update(T=p["length"] * p["dt"] / O.YEAR, theta_S=rng.uniform(0.3, 2.8), phi_S=rng.uniform(0.0, 6.0))
        pars.append(p)
    wb, maps, h, rows = _run(pars, [5] * nsrc)
    o = wb.offsets
    for s in sorted({0, nsrc // 2, nsrc - 1}):
        _check_wave(pars[s], maps[s], 5, h[:, o[s]:o[s + 1]])
        _check_phase(pars[s], maps[s], rows[:, o[s]:o[s + 1]])


def test_whole_and_quartered_entries_give_the_same_samples():
    """A source's samples do not depend on how many direct tiles come with it."""
    pars = dict(BASE, **LONG, length=60 * 1024 - 77)
    pars["T"] = pars["length"] * pars["dt"] / O.YEAR
    _, _, h1, r1 = _run([pars], [5])
    _, _, h, r = _run([pars] * 9, [5] * 9)
    n = pars["length"]
    for s in range(9):
        assert np.array_equal(h[:, s * n:(s + 1) * n], h1) and np.array_equal(r[:, s * n:(s + 1) * n], r1)


# k = 2: knots closer than the samples, so that only sample 0 is in the spline's boundary layer
@pytest.mark.parametrize("k", [2, 7])
def test_phases_past_a_plunge(k):
    """Plunges at sample 85679 and 88272 of 100000, and the tiles past them."""
    pars = _fast(k)
    _, maps, _, rows = _run([pars], [3])
    _check_phase(pars, maps[0], rows)


def test_end_of_a_fast_inspiral():
    """Tiles without a Bessel table (e changes too far in them), beside ordinary ones."""
    pars = dict(BASE, p=12.0, M=1e5, mu=50.0, e=0.5, length=60 * 1024 - 5, dt=10.0)
    pars["T"] = pars["length"] * pars["dt"] / O.YEAR
    wb, maps, h, rows = _run([pars], [12])
    _check_wave(pars, maps[0], 12, h)
    _check_phase(pars, maps[0], rows)
