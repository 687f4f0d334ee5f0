"""The order-7 kernels' packed background rows: every node and every face slot
must get the background of its own node and of the node across the face.  In a
stratified box with walls on all sides the perturbed state's tendency, steps
and transpose follow the FP64 form's to the form's 1e-5.  A value from a wrong
node is off by the change of pressure over an element, orders above."""
import numpy as np
import pytest

import nebulasem_gb300 as ng
from conftest import VARS, rel_l2
from nebulasem_gb300 import mesh as ngmesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(1, 1, 1), (2, 1, 3), (3, 2, 2)])
def test_order7_background(n):
    length = (n[0] * 200.0, n[1] * 250.0, n[2] * 300.0)
    m = ngmesh.box_mesh(n, 7, length)
    u, m["p_ref"], m["rho_ref"], m["gh"] = ngmesh.bubble_state(
        m, 0.5, [x / 2 for x in length], (150.0,) * 3)
    rng = np.random.default_rng(7)
    for c in (1, 2, 3):
        u[c] = u[0] * rng.uniform(-1.0, 1.0, len(u[0]))
    m.update(P0=1e5, T0=300.0, cp=1004.5, cv=717.5, gravity=np.array([0.0, 0.0, -9.81]), Pr=0.9,
             viscosity=0.0)
    s = ng.Solver(m, dt=1e-3)
    s.set_state(u)
    L64 = s.tendency(prec=ng.FP64)
    for a, b, v in zip(s.tendency(prec=ng.MIXED), L64, VARS):
        assert rel_l2(a, b) <= 1e-5, (v, rel_l2(a, b))
    w = [rng.standard_normal(len(u[0])) for _ in range(5)]
    du = [rng.standard_normal(len(u[0])) * sc for sc in (1e-3, 1e-1, 1e-1, 1e-1, 1e-1)]
    g64 = [np.asarray(x).copy() for x in s.vjp(w, prec=ng.FP64)]
    g32 = s.vjp(w, prec=ng.MIXED)
    diff = abs(sum(np.dot(a - b, d) for a, b, d in zip(g32, g64, du)))
    assert diff <= 1e-5 * sum(np.abs(a * d).sum() for a, d in zip(g64, du))
    s.set_state(u)
    s.step(3, prec=ng.FP64)
    ref = [np.asarray(x).copy() for x in s.get_state()]
    s.set_state(u)
    s.step(3, prec=ng.MIXED)
    for c, (a, b) in enumerate(zip(s.get_state(), ref)):
        if c in (0, 4):
            assert rel_l2(a, b) <= 1e-5, VARS[c]
    s.close()
