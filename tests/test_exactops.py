"""Rewritten FP64 collisions give the results of the printed code."""
import math
import re

import numpy as np
import pytest

from pylbm_gb300 import workloads as W
from pylbm_gb300.codegen import SchemeSource
from pylbm_gb300.exactops import rewrite
from pylbm_gb300.scheme import Scheme


def _fma(a, b, c):
    assert abs(math.frexp(a)[0]) == 0.5   # the product is exact, so this rounds once
    return a * b + c


def _run(lines, env):
    for line in lines:
        text = line.strip().rstrip(";").replace("const R ", "").replace("lbm_scaled_add<R>", "_fma").replace("lbm_neg<R>", "-")
        exec(re.sub(r"LBM_R\(([^()]*)\)", r"(\1)", text), {"_fma": _fma, "pow": math.pow}, env)


def _statements(dico):
    ref = SchemeSource(Scheme(dico), False, None, style="reference").reference_forms()
    return ref.moments_pull("g", "m") + ref.relaxation("m") + ref.populations("m", "g")


@pytest.mark.parametrize("dico, most", [(lambda: W.cavity(n=16), 127), (lambda: W.tgv3d(n=8), 401)])
def test_rewritten_collision_is_exact(dico, most):
    statements = _statements(dico())
    lines, count = rewrite(statements, "g")
    assert sum(count.values()) <= most
    q = sum(s.strip().startswith("g[") for s in statements)
    rng = np.random.default_rng(3)
    for scale in (1.0, 1e-3, 1e100):
        for _ in range(20):
            g = (rng.normal(size=q) * scale).tolist()
            a, b = {"g": list(g), "m": [0.0] * q}, {"g": list(g), "m": [0.0] * q}
            _run(statements, a)
            _run(lines, b)
            assert np.array_equal(a["g"], b["g"])


def test_special_values_pass_through():
    statements = _statements(W.cavity(n=16))
    lines, _ = rewrite(statements, "g")
    for bad in (math.inf, -math.inf, math.nan):
        g = [0.1] * 9
        g[5] = bad
        a, b = {"g": list(g), "m": [0.0] * 9}, {"g": list(g), "m": [0.0] * 9}
        _run(statements, a)
        _run(lines, b)
        assert np.array_equal(a["g"], b["g"], equal_nan=True)


def test_scales_and_shared_prefixes():
    lines, count = rewrite(["m[0] = g[0] + g[1] - g[2];", "m[1] = -2.0*g[0] - 2.0*g[1] + 3.0*g[2];",
                            "g[0] = m[0] + 0.25*m[1];", "g[1] = m[1];"], "g")
    # g0 + g1 once; 3 g2 once; m1 = fma(-2, s, 3 g2); g0' = fma(0.25, m1, m0)
    assert count == {"add": 2, "mul": 1, "fma": 2}
    env = {"g": [0.3, 0.7, 1.1], "m": [0.0, 0.0]}
    _run(lines, env)
    m0, m1 = 0.3 + 0.7 - 1.1, -2.0 * 0.3 - 2.0 * 0.7 + 3.0 * 1.1
    assert env["g"][0] == m0 + 0.25 * m1 and env["g"][1] == m1
