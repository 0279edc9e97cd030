"""A tuning-cache entry names the table of launch shapes that its index was
chosen from: an entry of another table, or of a file that named none, is timed
again and not taken."""
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from test_gpu_autotune import _batch  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("precision", [0, 1])
def test_entries_of_another_table_are_not_used(precision, tmp_path):
    wb = _batch()
    a, b = (torch.zeros(wb.total_samples, dtype=torch.float64, device="cuda") for _ in range(2))
    cache = tmp_path / "tune.txt"
    wb.autotune(a.data_ptr(), b.data_ptr(), precision=precision, cache_path=str(cache))
    entry = cache.read_text().strip()
    key = entry.split()[0]
    table = int(re.search(r"\|t(\d+)\|", key).group(1))
    others = [key.replace(f"|t{table}|", "|"), key.replace(f"|t{table}|", f"|t{table - 1}|")]
    cache.write_text("".join(f"{k} {v} {np.ones(6)}\n" for k in others for v in range(6)))
    v, ms = wb.autotune(a.data_ptr(), b.data_ptr(), precision=precision, cache_path=str(cache))
    assert all(m > 0 for m in ms) and ms[v] == min(ms)
    assert wb.autotune(a.data_ptr(), b.data_ptr(), precision=precision, cache_path=str(cache))[0] == v
