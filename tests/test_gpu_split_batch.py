"""The split-precision waveform kernel of a batch (tiles taken one after
another, the next one's data requested ahead) against the kernel that does
everything inside the tile: ragged and single-tile sources, failed ones, tiles
after the taper, t = 0 inside a tile, knot windows too long to stage, harmonic
counts past the tables, and more tiles than resident CTAs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import emri_kludge_suite_b200 as E  # noqa: E402

BASE = dict(backint=False, LISA=True, dt=10.0, p=9.0, T=0.25, f=2e-3, T_fit=1.0, mu=10.0, M=1e6, s=0.5, e=0.3,
            iota=0.785, gamma=0.1, psi=0.2, theta_S=0.5, phi_S=1.0, theta_K=0.8, phi_K=2.0, alpha=0.4, D=1.0)
PLUNGE = dict(p=6.0, mu=100.0, e=0.2, gamma=0.3)

CASES = {
    "ragged": [dict(length=n, nmodes=7 + k) for k, n in enumerate((2, 255, 1023, 1024, 1025, 2047, 5000, 70001))],
    "failed": [dict(length=3000, nmodes=9), dict(length=3000, nmodes=9, e=-0.1), dict(length=9000, nmodes=8, p=2.0),
               dict(length=9000, nmodes=8)],
    "plunge": [dict(PLUNGE, length=40000, nmodes=10), dict(PLUNGE, length=40000, nmodes=11, backint=True),
               dict(PLUNGE, length=33000, nmodes=6, LISA=False)],
    "backward": [dict(length=30011, dt=120.0, p=14.0, nmodes=5, backint=True)] * 2,
    "dense_knots": [dict(length=30011, dt=120.0, p=20.0, T_fit=0.003, nmodes=5), dict(length=7000, nmodes=4)],
    "many_modes": [dict(length=3001, nmodes=130, e=0.65, p=14.0), dict(length=5003, nmodes=128, e=0.6, p=14.0)],
    "queue": [dict(length=8000 + 37 * k, nmodes=4 + k % 3, gamma=0.01 * k) for k in range(160)],
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_matches_the_kernel_inside_the_tile(name):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    src = [dict(BASE, **c) for c in CASES[name]]
    nm = [p.pop("nmodes") for p in src]
    wb = E.WaveBatch(0)
    wb.plan(src, nmodes=nm)
    wb.upload()
    N = wb.total_samples
    out = []
    for v in (1, 0):  # inside the tile, then the batch kernel
        h = torch.full((3, N), 7.0, dtype=torch.float64, device="cuda")
        wb.set_variant(1, v)
        wb.run(h[0].data_ptr(), h[1].data_ptr(), t_ptr=h[2].data_ptr(), precision=1)
        torch.cuda.synchronize()
        out.append(h.cpu().numpy())
    assert wb.device_status() == 0
    assert np.array_equal(out[0][2], out[1][2])
    # the same phases and tables; the FP32 sums may contract multiply-adds differently: 1e-5 of the largest sample, as
    # for any two launch shapes
    for ch in (0, 1):
        for a, b in zip(wb.offsets[:-1], wb.offsets[1:]):
            want, got = out[0][ch][a:b], out[1][ch][a:b]
            if len(want):
                assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max(), (name, ch)
