"""The constant matrices of the polynomial segments (csrc/segment_fit.hpp)
against their definitions, by brute force on the host: interpolation at the
Chebyshev points and the Adams-Bashforth sums of a polynomial rate."""
import os
import re

import numpy as np

HPP = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "emri_kludge_suite_b200", "csrc",
                   "segment_fit.hpp")


def _tables():
    out = {}
    for name, body in re.findall(r"constexpr double (kSeg\w+)(?:\[\w+\])+ = \{(.*?)\};", open(HPP).read(), re.S):
        rows = re.findall(r"\{([^{}]*)\}", body) or [body]
        out[name] = np.array([[float(v) for v in r.split(",") if v.strip()] for r in rows])
    return out


TAB = _tables()
MID, HALF = 127.5, 128.5


def _x(m):
    return (np.asarray(m, dtype=np.float64) - MID) / HALF


def _poly(c, x):
    return np.polynomial.polynomial.polyval(x, c)


def test_fit_and_tail_reproduce_polynomials():
    nodes = TAB["kSegNode"][0]
    np.testing.assert_allclose(nodes, -np.cos((2 * np.arange(8) + 1) * np.pi / 16), atol=1e-16)
    rng = np.random.default_rng(1)
    for _ in range(20):
        c7 = rng.standard_normal(8)
        np.testing.assert_allclose(TAB["kSegFit7"] @ _poly(c7, nodes), c7, atol=2e-12)  # rows sum to ~100 in magnitude
        np.testing.assert_allclose(TAB["kSegFit4"] @ _poly(c7[:5], nodes), c7[:5], atol=1e-13)
        ch = np.polynomial.chebyshev.poly2cheb(c7)
        np.testing.assert_allclose(TAB["kSegTail"] @ _poly(c7, nodes), ch[5:], atol=1e-14)
        # the cut fit is the interpolant without its last three Chebyshev terms
        cut = np.polynomial.chebyshev.cheb2poly(ch[:5])
        np.testing.assert_allclose(TAB["kSegFit4"] @ _poly(c7, nodes), cut, atol=1e-13)


def test_sums_reproduce_the_adams_bashforth_recurrence():
    nodes = TAB["kSegNode"][0]
    rng = np.random.default_rng(2)
    m = np.arange(-1, 257)
    for D in (4, 7):
        for _ in range(10):
            c = np.concatenate([rng.standard_normal(1), 1e-2 * rng.standard_normal(D)])
            r = _poly(c, _x(m)).astype(np.longdouble)  # r[j + 1]: sample j
            fwd = np.concatenate([[0], np.cumsum(1.5 * r[1:257] - 0.5 * r[0:256])]).astype(np.float64)  # j < m, m = 0..256
            inc = (1.5 * r[1:257] - 0.5 * r[2:258])[::-1]
            bwd = np.concatenate([[0], np.cumsum(inc)])[::-1].astype(np.float64)  # j > m, m = -1..255
            ref = _poly(c, nodes)[4]
            dv = _poly(c, nodes) - ref
            pf, pb = TAB[f"kSegFwd{D}"] @ dv, TAB[f"kSegBwd{D}"] @ dv
            pf[:2] += ref * np.array([MID, HALF])
            pb[:2] += ref * np.array([MID, -HALF])
            # 256 terms of order 1: 256 x 2e-16 x the fit's amplification of about ten
            np.testing.assert_allclose(_poly(pf, _x(np.arange(0, 257))), fwd, atol=1e-11)
            np.testing.assert_allclose(_poly(pb, _x(np.arange(-1, 256))), bwd, atol=1e-11)
