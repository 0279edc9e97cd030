"""The warm-start network's kernels at the edges of their tiles and groups
(128 rows a tile, four tiles a CTA, one CTA an SM), and with pre-activations
far outside the range where the sigmoid changes, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from oracle import mlp_oracle as O  # noqa: E402

from emri_kludge_suite_b200 import parmap_mlp as P  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _points(n, seed):
    rng = np.random.default_rng(seed)
    x = np.stack([rng.uniform(6.5, 20, n), rng.uniform(0.01, 0.7, n), rng.uniform(0, np.pi, n), rng.uniform(0, 0.95, n)], 1)
    y = np.stack([1 + 0.3 / x[:, 0], 1 - 0.8 / x[:, 0], 0.1 * x[:, 1] * x[:, 3]], 1)
    return x.astype(np.float32), y.astype(np.float32)


def _model(scale=1.0):
    x, y = _points(4096, 1)
    m = P.ParMapMLP(0, params=(scale * P.init_params(3)).astype(np.float32))
    m.fit_norm(x.astype(np.float64), y.astype(np.float64))
    return m


def _norm64(m):
    return {k: np.asarray(v, dtype=np.float64) for k, v in m.norm.items()}


# a row, ragged tiles, one tile more than CTAs, one more than the groups of all CTAs
@pytest.mark.parametrize("n", [1, 127, 128, 129, 148 * 128 + 1, 4 * 148 * 128 + 130])
def test_forward_rows(n):
    m = _model()
    x, _ = _points(n, n)
    xd = torch.tensor(x, device="cuda")
    yd = torch.full((n + 1, 3), 7.0, dtype=torch.float32, device="cuda")
    m.forward_device(xd.data_ptr(), yd.data_ptr(), n)
    y = yd.cpu().numpy()
    assert np.all(y[n] == 7.0)
    pick = np.unique(np.r_[0, n - 1, np.random.default_rng(0).integers(0, n, 2000)])
    ref = O.predict(m.params().astype(np.float64), x[pick].astype(np.float64), _norm64(m))
    # the bar of the forward kernel (test_gpu_parmap_mlp.py)
    assert np.max(np.abs(y[pick] - ref) / m.norm["out_scale"]) < 5e-3


@pytest.mark.parametrize("n", [1, 127, 128, 129, 16384])
def test_gradient_rows(n):
    m = _model()
    x, y = _points(n, 5)
    perm = np.random.default_rng(2).permutation(n).astype(np.int32)
    d = [torch.tensor(v, device="cuda") for v in (x, y, perm)]
    grad = torch.full((P.n_params() + 1,), 7.0, dtype=torch.float32, device="cuda")
    loss = m.gradients_device(d[0].data_ptr(), d[1].data_ptr(), n, grad.data_ptr(), perm_ptr=d[2].data_ptr())
    g = grad.cpu().numpy().astype(np.float64)
    assert g[-1] == 7.0
    lref, gref = O.loss_and_grad(m.params().astype(np.float64), x.astype(np.float64), y.astype(np.float64), _norm64(m))
    # the bars of the gradient kernel (test_gpu_parmap_mlp.py)
    assert abs(loss - lref) <= 1e-4 * lref
    for k, (o, s) in O.OFFSETS.items():
        sz = int(np.prod(s))
        assert np.linalg.norm(g[o:o + sz] - gref[o:o + sz]) < 2e-2 * np.linalg.norm(gref[o:o + sz]), k


@pytest.mark.parametrize("scale", [30.0, 1000.0])
def test_saturated_activations(scale):
    """Pre-activations up to 1e2 .. 1e8: the sigmoid is 0 or 1 to rounding, and nothing overflows."""
    m = _model(scale)
    x, _ = _points(500, 8)
    got = m.predict(x.astype(np.float64))
    with np.errstate(over="ignore"):
        ref = O.predict(m.params().astype(np.float64), x.astype(np.float64), _norm64(m))
    assert np.all(np.isfinite(got))
    # FP32 sums whose terms are the BF16 oracle's: flips of a BF16 rounding move a term by 2^-8 of itself
    assert np.max(np.abs(got - ref)) <= 1e-2 * np.max(np.abs(ref))
