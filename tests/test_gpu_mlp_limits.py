"""Inference with pre-activations far below the sigmoid's range: silu goes to its
limit there, 0 (down to -1e20), and a NaN stays one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from oracle import mlp_oracle as O  # noqa: E402
from test_gpu_mlp_tiles import _model, _norm64, _points  # noqa: E402

from emri_kludge_suite_b200 import parmap_mlp as P  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _with_bias(layer, value, every):
    base = _model()
    d = O.unpack(base.params())
    d[layer] = d[layer].copy()
    d[layer][::every] = value
    m = P.ParMapMLP(0, params=O.pack(d).astype(np.float32))
    m.set_norm(*[base.norm[k] for k in ("in_shift", "in_scale", "out_shift", "out_scale")])
    return m


# pairs of units share a reciprocal: both of a pair (every 1), one of it (every 2), the other layers' epilogues
@pytest.mark.parametrize("layer", ["b1", "b2", "b3"])
@pytest.mark.parametrize("value,every", [(-1e20, 1), (-1e20, 2), (-1e18, 3), (-45.0, 1), (-75.0, 1), (-60.0, 2)])
def test_silu_far_below_zero(layer, value, every):
    m = _with_bias(layer, value, every)
    x, _ = _points(300, 4)
    with np.errstate(over="ignore"):
        ref = O.predict(m.params().astype(np.float64), x.astype(np.float64), _norm64(m))
    got = m.predict(x.astype(np.float64))
    # the bar of the forward kernel (test_gpu_parmap_mlp.py)
    assert np.max(np.abs(got - ref) / m.norm["out_scale"]) < 5e-3


def test_nan_stays():
    m = _with_bias("b2", np.nan, 128)
    x, _ = _points(300, 4)
    assert np.all(np.isnan(m.predict(x.astype(np.float64))))
