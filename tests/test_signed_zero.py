"""Momenta of -0: a node without a tendency keeps its zero's sign through a
step, as in the plain products' update (a zero product there has the sign of
its factors).  Compared with the oracle as bit patterns."""
import numpy as np
import pytest

import nebulasem_gb300 as ng
from nebulasem_gb300 import mesh as ngmesh

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a, dtype=np.float64).reshape(-1).view(np.uint64)


@pytest.mark.parametrize("visc", [0.0, 1.5])
@pytest.mark.parametrize("zero", [(2,), (1, 2, 3)])
def test_sign_of_a_zero_momentum(visc, zero):
    import oracle

    h, n = 62.5, (4, 1, 3)
    m = ngmesh.box_mesh(n, 4, tuple(h * x for x in n), dim=2)
    u, m["p_ref"], m["rho_ref"], m["gh"] = ngmesh.bubble_state(m, 0.5, [h * x / 2 for x in n], (80.0,) * 3)
    rng = np.random.default_rng(11)
    for c in (1, 3):
        u[c] = u[0] * rng.uniform(-1.0, 1.0, len(u[0]))
    for c in zero:
        u[c] = np.where(rng.uniform(size=len(u[0])) < 0.5, -0.0, 0.0)
    m.update(P0=1e5, T0=300.0, cp=1004.5, cv=717.5, gravity=np.array([0.0, 0.0, -9.81]), Pr=0.9,
             viscosity=visc)
    dt = 1e-3
    o = oracle.OracleMesh(dict(m, dt=dt))
    s = ng.Solver(m, dt=dt)
    oracle.set_pow(1)
    try:
        for steps in (1, 2):
            s.set_state(u)
            s.step(steps, prec=ng.FP64)
            want = o.ssprk3(u, dt, steps)
            assert np.signbit(want[2]).any()
            for a, b in zip(s.get_state(), want):
                assert np.array_equal(_bits(a), _bits(b))
    finally:
        oracle.set_pow(0)
    s.close()
