"""The precision form in two dimensions, where four elements share a CTA, at
element counts on both sides of a full group: tendency, steps and transpose
against the FP64 form, inviscid and viscous, axis-aligned and tilted.  The
winds are random per node, so an element that takes another's values or is
left out moves the result by its own size; FP32 rounding stays within the
form's 1e-5 (relative L2; of the sum of the magnitudes for the transpose)."""
import numpy as np
import pytest

import nebulasem_gb300 as ng
from conftest import VARS, rel_l2
from nebulasem_gb300 import mesh as ngmesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("visc", [0.0, 1.5])
@pytest.mark.parametrize("tilt", [0.0, 30.0])
@pytest.mark.parametrize("n,order", [((1, 1), 4), ((1, 2), 3), ((3, 1), 4), ((2, 2), 3), ((5, 1), 4),
                                     ((7, 1), 3)])
def test_against_fp64(n, order, tilt, visc):
    length = (n[0] * 62.5, 62.5, n[1] * 80.0)
    m = ngmesh.box_mesh((n[0], 1, n[1]), order, length, dim=2, tilt=tilt)
    u, m["p_ref"], m["rho_ref"], m["gh"] = ngmesh.bubble_state(
        m, 0.5, [x / 2 for x in length], (80.0,) * 3)
    rng = np.random.default_rng(order)
    for c in (1, 3):
        u[c] = u[0] * rng.uniform(-1.0, 1.0, len(u[0]))
    m.update(P0=1e5, T0=300.0, cp=1004.5, cv=717.5, gravity=np.array([0.0, 0.0, -9.81]), Pr=0.9,
             viscosity=visc)
    s = ng.Solver(m, dt=0.02 / order ** 2)
    s.set_state(u)
    L64 = s.tendency(prec=ng.FP64)
    top = max(np.linalg.norm(x) for x in L64)
    for a, b, v in zip(s.tendency(prec=ng.MIXED), L64, VARS):
        if np.linalg.norm(b) >= 1e-8 * top:
            assert rel_l2(a, b) <= 1e-5, (v, rel_l2(a, b))
    w = [rng.standard_normal(len(u[0])) for _ in range(5)]
    du = [rng.standard_normal(len(u[0])) * sc for sc in (1e-3, 1e-1, 0.0, 1e-1, 1e-1)]
    g64 = [np.asarray(x).copy() for x in s.vjp(w, prec=ng.FP64)]
    g32 = s.vjp(w, prec=ng.MIXED)
    diff = abs(sum(np.dot(a - b, d) for a, b, d in zip(g32, g64, du)))
    assert diff <= 1e-5 * sum(np.abs(a * d).sum() for a, d in zip(g64, du))
    got = {}
    for prec in (ng.FP64, ng.MIXED):
        s.set_state(u)
        s.step(3, prec=prec)
        got[prec] = [np.asarray(x).copy() for x in s.get_state()]
    s.close()
    for c in (0, 4):
        assert rel_l2(got[ng.MIXED][c], got[ng.FP64][c]) <= 1e-5, VARS[c]
    assert rel_l2(np.stack(got[ng.MIXED][1:4]), np.stack(got[ng.FP64][1:4])) <= 1e-5
