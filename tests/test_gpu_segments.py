"""The FP64 polynomial segments (sources of more than 24 tiles of 1024 samples)
against the oracle, at the sizes where they can go wrong: the line to the
in-tile kernel, ragged last tiles and segments, t = 0 inside a tile, the end of
a plunge (direct tiles, frozen phases), the response switched off, harmonic
counts past the tables."""
import numpy as np
import pytest

from conftest import load_golden, mismatch

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import emri_kludge_suite_b200 as E  # noqa: E402
from oracle import oracle as O  # noqa: E402

BASE = dict(backint=False, LISA=True, dt=10.0, p=9.0, T=0.25, f=2e-3, T_fit=1.0, mu=10.0, M=1e6, s=0.5, e=0.3,
            iota=0.785, gamma=0.1, psi=0.2, theta_S=0.5, phi_S=1.0, theta_K=0.8, phi_K=2.0, alpha=0.4, D=1.0)
PLUNGE = dict(p=6.0, mu=100.0, e=0.2, gamma=0.3)

CASES = {
    "last_small": dict(length=24 * 1024, nmodes=6),
    "first_segments": dict(length=24 * 1024 + 1, nmodes=6),
    "ragged_255": dict(length=25 * 1024 + 255, nmodes=7),
    "ragged_256": dict(length=25 * 1024 + 256, nmodes=8, LISA=False, iota=2.2),
    "ragged_257": dict(length=25 * 1024 + 257, nmodes=9, e=0.6, p=12.0),
    "many_modes": dict(length=26 * 1024 - 1, nmodes=130, e=0.65, p=14.0),
    "plunge": dict(PLUNGE, length=40000, nmodes=10),
    "plunge_backint": dict(PLUNGE, length=40000, nmodes=10, backint=True),
    "long_steps": dict(length=30011, dt=120.0, p=14.0, nmodes=5, backint=True),
    "dense_knots": dict(length=30011, dt=120.0, p=20.0, T_fit=0.003, nmodes=5),
}


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    O.set_threads(8)
    yield
    O.set_threads(1)


def _pars(name):
    p = dict(BASE, **CASES[name])
    nm = p.pop("nmodes")
    p["T"] = p["length"] * p["dt"] / O.YEAR
    return p, nm


def _mapped(m):
    return O.MappedTrajectory(m.steps, m.e_traj, m.v_map, m.M_map, m.s_map, m.dt_map, m.Phi0, 2)


@pytest.mark.parametrize("name", sorted(CASES))
def test_waveform_and_phases_match_oracle(name):
    pars, nm = _pars(name)
    m = E.front_end(pars)
    wb = E.WaveBatch(0)
    wb.plan([pars], nmodes=nm, mapped=[m])
    assert wb.status[0] == 0
    N = wb.total_samples
    h = torch.full((2, N), 7.0, dtype=torch.float64, device="cuda")
    t = torch.zeros(N, dtype=torch.float64, device="cuda")
    rows = torch.full((8, N), 7.0, dtype=torch.float64, device="cuda")
    wb.upload()
    wb.run(h[0].data_ptr(), h[1].data_ptr(), t_ptr=t.data_ptr())
    wb.run_phase(rows.data_ptr(), N)
    torch.cuda.synchronize()
    assert wb.device_status() == 0
    h, rows = h.cpu().numpy(), rows.cpu().numpy()
    oI, oII = O.oracle_genwave(pars, _mapped(m), nm)[1:3]
    scale = max(np.abs(oI).max(), np.abs(oII).max())
    # the bars of the FP64 path against the oracle (test_gpu_waveform.py)
    assert np.abs(h[0] - oI).max() <= 1e-8 * scale and np.abs(h[1] - oII).max() <= 1e-8 * scale
    assert mismatch(h[0], h[1], oI, oII) < 1e-12
    ref = O.oracle_genphase(pars, _mapped(m))
    assert np.array_equal(t.cpu().numpy(), ref[0]) and np.array_equal(rows[0], ref[0])
    # the bars of the phase product (test_gpu_phase.py)
    for k in (1, 2, 3):
        assert np.max(np.abs(rows[k] - ref[k])) <= 1e-11 * max(1.0, np.abs(ref[k]).max()), k
    for k in (4, 5, 6):
        assert np.max(np.abs(rows[k] - ref[k]) / np.abs(ref[k])) < 1e-12, k
    assert np.max(np.abs(rows[7] - ref[7]) / np.abs(ref[7])) < 1e-13
    first = max(int(ref[8]) + int(ref[9]) + 2, 1)
    if first < N:
        assert np.all(rows[1:4, first:] == rows[1:4, int(ref[8]), None])


def test_mixed_batch_equals_single_sources_bit_for_bit():
    """Small and large sources in one batch, one of them invalid: every source's samples and phases are those of a
    call of its own, and a CUDA-graph replay's are the same."""
    names = sorted(CASES)
    pars = [_pars(n)[0] for n in names]
    nm = [_pars(n)[1] for n in names]
    pars.insert(3, dict(load_golden("cfg0_short")["pars"], e=-0.2, length=30000))
    nm.insert(3, 4)

    def run(p, n, graph):
        wb = E.WaveBatch(0)
        wb.plan(p, nmodes=n)
        h = torch.full((2, wb.total_samples), 7.0, dtype=torch.float64, device="cuda")
        rows = torch.full((8, wb.total_samples), 7.0, dtype=torch.float64, device="cuda")
        wb.upload()
        (wb.run_graph if graph else wb.run)(h[0].data_ptr(), h[1].data_ptr())
        wb.run_phase(rows.data_ptr(), wb.total_samples)
        torch.cuda.synchronize()
        assert wb.device_status() == 0
        return wb, h.cpu().numpy(), rows.cpu().numpy()

    wb, h, rows = run(pars, nm, False)
    _, hg, _ = run(pars, nm, True)
    assert np.array_equal(h, hg)
    o = wb.offsets
    assert wb.status[3] != 0 and np.all(h[:, o[3]:o[4]] == 0.0) and np.all(rows[:, o[3]:o[4]] == 0.0)
    for s in range(len(pars)):
        if s == 3:
            continue
        _, h1, r1 = run([pars[s]], [nm[s]], False)
        assert np.array_equal(h1, h[:, o[s]:o[s + 1]]), names[s - (s > 3)]
        assert np.array_equal(r1, rows[:, o[s]:o[s + 1]]), names[s - (s > 3)]
