"""The device spline solve (short blocks, four lanes each) against the oracle's
dense trajectory, over knot counts from one block to many and both ends of a
block's last, ragged window."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import emri_kludge_suite_b200 as E  # noqa: E402
from oracle import oracle as O  # noqa: E402

BASE = dict(backint=False, LISA=True, dt=10.0, p=12.0, T=0.25, f=2e-3, T_fit=1.0, mu=10.0, M=1e6, s=0.5, e=0.3,
            iota=0.785, gamma=0.1, psi=0.2, theta_S=0.5, phi_S=1.0, theta_K=0.8, phi_K=2.0, alpha=0.4, D=1.0)


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


# knots of a source: about (steps - 1) max(1, span / (T_fit M^2 / mu)); the spans below give 40 to 20000 of them
@pytest.mark.parametrize("length,dt,T_fit", [(900, 10.0, 1.0), (1500, 25.0, 0.02), (4001, 40.0, 0.02), (4001, 41.0, 0.02),
                                             (9000, 60.0, 0.01), (20011, 120.0, 0.003)])
def test_spline_trajectory_matches_oracle(length, dt, T_fit):
    pars = dict(BASE, length=length, dt=dt, T_fit=T_fit)
    m = E.front_end(pars)
    ref, _, _ = O.oracle_pnevolution(pars, O.MappedTrajectory(m.steps, m.e_traj, m.v_map, m.M_map, m.s_map, m.dt_map, m.Phi0, 2))
    wb = E.WaveBatch(0)
    wb.plan([pars], nmodes=4, mapped=[m])
    assert wb.status[0] == 0
    N = wb.total_samples
    h = torch.zeros((2, N), dtype=torch.float64, device="cuda")
    traj = torch.zeros((9, N), dtype=torch.float64, device="cuda")
    wb.upload()
    wb.run(h[0].data_ptr(), h[1].data_ptr(), traj_ptr=traj.data_ptr(), traj_stride=N)
    torch.cuda.synchronize()
    tr = traj.cpu().numpy()
    n = min(N, int(wb.i_plunge[0]) + int(wb.i_buffer[0]))
    # the same knots on both sides: e, v, M, S agree to rounding (1e-13, as in the fixture comparison)
    for row, k in enumerate(["e", "v", "M", "S"]):
        want = ref[1 + row][:n]  # the oracle's rows start with t
        assert np.max(np.abs(tr[row, :n] - want) / np.abs(want)) < 1e-13, k
