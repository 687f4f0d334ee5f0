"""The FP64 form where its volume kernel starts beside the face kernel and where
it starts after it: the same bits as the oracle on every side of the rule's
lines (2.5 elements, 8 and 32 warps per SM; 152 SMs)."""
import numpy as np
import pytest

import nebulasem_gb300 as ng
from nebulasem_gb300 import mesh as ngmesh

pytestmark = pytest.mark.gpu


# elements and warps per SM: 2.4 and 2.4, 2.6 and 2.6, 7.9 and 7.9, 8.1 and 8.1,
# 31.6 and 31.6, 32.3 and 32.3 (order 2, one warp); 0.6 and 4.3 (order 5)
@pytest.mark.parametrize("n,order,visc", [((8, 5, 9), 2, 0.0), ((8, 5, 10), 2, 1.5), ((10, 10, 12), 2, 0.0),
                                          ((11, 7, 16), 2, 1.5), ((20, 12, 20), 2, 0.0), ((17, 17, 17), 2, 0.0),
                                          ((4, 5, 5), 5, 1.5)])
def test_equal_to_the_oracle(n, order, visc):
    import oracle

    h = 62.5
    m = ngmesh.box_mesh(n, order, tuple(h * x for x in n))
    u, m["p_ref"], m["rho_ref"], m["gh"] = ngmesh.bubble_state(m, 0.5, [h * x / 2 for x in n], (80.0,) * 3)
    rng = np.random.default_rng(order)
    for c in (1, 2, 3):
        u[c] = u[0] * rng.uniform(-1.0, 1.0, len(u[0]))
    m.update(P0=1e5, T0=300.0, cp=1004.5, cv=717.5, gravity=np.array([0.0, 0.0, -9.81]), Pr=0.9,
             viscosity=visc)
    dt = 0.02 / order ** 2
    s = ng.Solver(m, dt=dt)
    s.set_state(u)
    s.step(3, prec=ng.FP64)
    got = s.get_state()
    s.close()
    oracle.set_pow(1)
    try:
        want = oracle.OracleMesh(dict(m, dt=dt)).ssprk3(u, dt, 3)
    finally:
        oracle.set_pow(0)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
