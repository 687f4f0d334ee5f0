"""The precision form's viscous gradients, formed line by line, at even and odd
node counts, in two dimensions, on single elements (walls on every side) and
with the full metric of tilted boxes: the tendency against the FP64 form's.
The winds are random per node and the lengths differ per direction, so a value
taken from a wrong line or a wrong face moves it by its own size; FP32 rounding
stays within the form's 1e-5 of the relative L2 norm."""
import numpy as np
import pytest

import nebulasem_gb300 as ng
from conftest import VARS, rel_l2
from nebulasem_gb300 import mesh as ngmesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tilt", [0.0, 30.0])
@pytest.mark.parametrize("n,dim,order", [((2, 3, 2), 3, 3), ((3, 2, 4), 3, 4), ((2, 2, 3), 3, 7),
                                         ((1, 1, 1), 3, 4), ((1, 1, 1), 3, 7), ((4, 1, 3), 2, 3),
                                         ((3, 1, 5), 2, 4)])
def test_tendency_against_fp64(n, dim, order, tilt):
    length = (n[0] * 62.5, n[1] * 80.0, n[2] * 100.0)
    m = ngmesh.box_mesh(n, order, length, dim=dim, tilt=tilt)
    u, m["p_ref"], m["rho_ref"], m["gh"] = ngmesh.bubble_state(
        m, 0.5, [x / 2 for x in length], (80.0,) * 3)
    rng = np.random.default_rng(order)
    for c in (1, 2, 3) if dim == 3 else (1, 3):
        u[c] = u[0] * rng.uniform(-1.0, 1.0, len(u[0]))
    m.update(P0=1e5, T0=300.0, cp=1004.5, cv=717.5, gravity=np.array([0.0, 0.0, -9.81]), Pr=0.9,
             viscosity=1.5)
    s = ng.Solver(m, dt=0.02 / order ** 2)
    s.set_state(u)
    L64 = s.tendency(prec=ng.FP64)
    L32 = s.tendency(prec=ng.MIXED)
    s.close()
    top = max(np.linalg.norm(x) for x in L64)
    for a, b, v in zip(L32, L64, VARS):
        if np.linalg.norm(b) >= 1e-8 * top:
            assert rel_l2(a, b) <= 1e-5, (v, rel_l2(a, b))
