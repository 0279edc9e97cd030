"""The packed transforms of FP64 likelihood and Fisher batches (even lengths)
against numpy's rfft of the same templates, at lengths where the pairing of
bins can go wrong, and what the rows hold afterwards."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from oracle import oracle as O  # noqa: E402

from emri_kludge_suite_b200.gpuAAK import GPUAAK  # noqa: E402

INJ = np.array([0.785, 0.5, 8.0, 0.2, 1e6, 10.0, 0.3, 0.2, 0.4, 0.5, 1.0, 0.8, 2.0, 1.0])


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _setup(length, n):
    rng = np.random.default_rng(length)
    nb = length // 2 + 1
    w = [rng.uniform(0.5, 2.0, nb) * 1e18 for _ in range(2)]
    D = [rng.standard_normal(nb) + 1j * rng.standard_normal(nb) for _ in range(2)]
    g = GPUAAK(1.0, 100, length, 100.0, 10.0, True, False)
    g.input_data(D[0], D[1], w[0], w[1])
    X = np.tile(INJ, (n, 1))
    X[:, 6:11] += 0.3 * rng.standard_normal((n, 5))
    X[:, 2] += 0.01 * rng.standard_normal(n)
    waves = []
    for x in X:
        g.gpu_gen_AAK(*x)
        _, hI, hII = g.GetWaveform()
        waves.append((hI[:length].copy(), hII[:length].copy()))
    return g, X, w, D, waves


# odd (unpacked), M odd, M even, M = 2 mod 4, a ragged last chunk, large prime factor
@pytest.mark.parametrize("length", [9001, 9002, 9004, 10000, 12346, 4 * 4099])
def test_batches_match_numpy_on_the_same_templates(length):
    n = 7
    g, X, w, D, waves = _setup(length, n)
    out = g.likelihood_batch(X, max_batch=3)
    ref = np.array([O.inner_products(a, b, D[0], D[1], w[0], w[1]) for a, b in waves])
    # sums of ~1e4 terms in FP64, both sides: 1e-12 of <h|h>'s scale
    scale = np.abs(ref[:, 1]).max() + np.abs(ref[:, 0]).max()
    assert np.max(np.abs(out - ref)) <= 1e-12 * scale
    # the batch again after a Fisher call, a plan of each size kept
    Xf = np.repeat(X[:1], 6, axis=0)
    for i in range(3):
        Xf[2 * i + 1, 6 + i] += 1e-3
    G = g.fisher_gram(Xf, 10.0)
    W = []
    for x in Xf:
        g.gpu_gen_AAK(*x)
        _, hI, hII = g.GetWaveform()
        W.append((np.fft.rfft(hI[:length]) * w[0], np.fft.rfft(hII[:length]) * w[1]))
    for c in range(2):
        d = np.array([10.0 * (W[2 * i + 1][c] - W[2 * i][c]) for i in range(3)])
        want = 4.0 * np.real(d.conj() @ d.T)
        assert np.max(np.abs(G[c] - want)) <= 1e-9 * np.abs(want).max()  # differences of 1e-3: FFT rounding over 1e-3
    assert np.array_equal(g.likelihood_batch(X, max_batch=3), out)


@pytest.mark.parametrize("length", [9001, 9004])
def test_rows_after_a_batch_hold_half_spectra(length):
    """GetWaveform after a batch returns the half spectrum of the last chunk's
    first template, and Likelihood() on those rows its products."""
    g, X, w, D, waves = _setup(length, 4)
    g.likelihood_batch(X, max_batch=4)
    _, sI, sII = g.GetWaveform(is_Fourier=True)
    nb = length // 2 + 1
    for s, h in ((sI, waves[0][0]), (sII, waves[0][1])):
        spec = s[0:2 * nb:2] + 1j * s[1:2 * nb:2]
        want = np.fft.rfft(h)
        assert np.max(np.abs(spec - want)) <= 1e-13 * np.sum(np.abs(h))
    # a new template after that: time-domain rows again
    g.gpu_gen_AAK(*X[1])
    _, hI, _ = g.GetWaveform()
    assert np.array_equal(hI[:length], waves[1][0])
    assert np.max(np.abs(g.Likelihood() - O.inner_products(*waves[1], D[0], D[1], w[0], w[1]))) <= 1e-12 * abs(
        O.inner_products(*waves[1], D[0], D[1], w[0], w[1])[1])
