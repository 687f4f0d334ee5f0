"""The precision form's last stage converts its increments and the new state on
the integer pipes, with a fast path for values in range.  Exact zeros, values
below FP32's smallest normal and non-finite ones: hydrostatic rest stays exact
with a momentum of 1e-42 added (which FP32 drops, FP64 keeps), and a NaN or an
increment that overflows is reported, on both geometries."""
import numpy as np
import pytest

import nebulasem_gb300 as ng
from nebulasem_gb300 import mesh as ngmesh

pytestmark = pytest.mark.gpu


def _setup(tilt, dim):
    n = (3, 1 if dim == 2 else 2, 3)
    length = tuple(100.0 * x for x in n)
    m = ngmesh.box_mesh(n, 4, length, dim=dim, tilt=tilt)
    u, m["p_ref"], m["rho_ref"], m["gh"] = ngmesh.bubble_state(m, 0.0, (0.0,) * 3, (1.0,) * 3)
    m.update(P0=1e5, T0=300.0, cp=1004.5, cv=717.5, gravity=np.array([0.0, 0.0, -9.81]), Pr=0.9,
             viscosity=0.0)
    return m, [np.asarray(x, dtype=np.float64).copy() for x in u]


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("tilt", [0.0, 30.0])
def test_zero_tiny_and_nonfinite(tilt, dim):
    m, u = _setup(tilt, dim)
    s = ng.Solver(m, dt=1e-3)
    tiny = np.zeros_like(u[1])
    tiny[::7] = 1e-42
    u[1], u[3] = tiny.copy(), -tiny
    s.set_state(u)
    s.step(1, prec=ng.MIXED)
    got = s.get_state()
    assert all(np.array_equal(a, b) for a, b in zip(got, u))
    mid = len(tiny) // 2
    for v, x in ((4, np.nan), (1, np.inf), (3, 1e38)):
        bad = [a.copy() for a in u]
        bad[v][mid] = x
        s.set_state(bad)
        with pytest.raises(ng.NsemError):
            s.step(1, prec=ng.MIXED)
    # and the form recovers with the next state
    s.set_state(u)
    s.step(1, prec=ng.MIXED)
    assert all(np.array_equal(a, b) for a, b in zip(s.get_state(), u))
    s.close()
