"""Sources of one plan call that share an inspiral (masses, spin, orbit, span)
share its front end.  Each source's plan must stay that of the source planned
alone: status, samples, plunge index, buffer length and Newton counts, with
sources that fail among those that share (host-only context, no GPU)."""
import numpy as np
import pytest

import emri_kludge_suite_b200 as E
from emri_kludge_suite_b200.workloads import config1


def _sources(kinds):
    base, _ = config1(29, 64)
    out = []
    for i, (src, change) in enumerate(kinds):
        q = dict(base[src])
        q["length"] = min(int(q["length"]), 300000)
        q.update(gamma=0.1 + 0.01 * i, psi=0.4 + 0.3 * i, alpha=1.0 + 0.02 * i, D=1.0 + 0.1 * i)
        q.update(change)
        out.append(q)
    return out


CASES = {
    # three inspirals, sky and phase angles all different
    "extrinsic": [(0, {})] * 4 + [(1, {})] * 3 + [(2, {})],
    # failures: of the source alone (angles), of the shared inspiral itself
    # (below the separatrix), and a first source that is invalid
    "failing": [(0, {"theta_K": 0.0}), (0, {}), (0, {"psi": float("nan")}), (0, {}), (3, {"p": 3.0}), (3, {"p": 3.0}),
                (3, {}), (3, {})],
    # the same orbit over other spans, spacings and directions is another inspiral
    "spans": [(4, {}), (4, {"length": 200000}), (4, {"dt": 7.0}), (4, {"backint": True}), (4, {"backint": True}),
              (4, {"T_fit": 0.3}), (4, {}), (4, {}), (4, {"length": 200000}), (4, {"dt": 7.0})],
    # too few shared to be worth it: each source its own
    "distinct": [(i, {}) for i in range(7)] + [(0, {})],
    "pair": [(5, {}), (5, {})],
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("threads", [1, 3])
def test_shared_front_ends_equal_single_plans(name, threads):
    params = _sources(CASES[name])
    wb = E.WaveBatch(-1)
    wb.plan(params, nmodes=30, nthreads=threads)
    batch = (wb.status.copy(), np.diff(wb.offsets), wb.i_plunge.copy(), wb.i_buffer.copy())
    points = iters = 0
    for s, p in enumerate(params):
        one = E.WaveBatch(-1)
        one.plan([p], nmodes=30, nthreads=1)
        for b, x in zip(batch, (one.status, np.diff(one.offsets), one.i_plunge, one.i_buffer)):
            assert b[s] == x[0], (name, s)
        n = one.newton_stats()
        points += n["points"]
        iters += n["iterations"]
    n = wb.newton_stats()
    assert (n["points"], n["iterations"]) == (points, iters)
