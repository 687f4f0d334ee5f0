"""Results copied to the host together through a pinned buffer and one by one
(larger results; arrays that are pinned themselves): the same bytes on both
sides of the limit and from both kinds of arrays, the FP64 tendency's pressure
among them, and a non-finite state is still reported."""
import numpy as np
import pytest
import torch

import nebulasem_gb300 as ng
from nebulasem_gb300 import mesh as ngmesh

pytestmark = pytest.mark.gpu


# five arrays of 5, 320 and 400 KB together, with the pressure 6, 384 (10^3) and 480: the limit is 393216 bytes
@pytest.mark.parametrize("n", [(1, 1, 1), (4, 4, 4), (5, 4, 4)])
def test_same_results(n):
    m = ngmesh.box_mesh(n, 4, tuple(62.5 * x for x in n))
    u, m["p_ref"], m["rho_ref"], m["gh"] = ngmesh.bubble_state(
        m, 0.5, [31.25 * x for x in n], (80.0,) * 3)
    m.update(P0=1e5, T0=300.0, cp=1004.5, cv=717.5, gravity=np.array([0.0, 0.0, -9.81]), Pr=0.9,
             viscosity=0.0)
    s = ng.Solver(m, dt=1e-3)
    s.set_state(u)
    L, p = s.tendency(ng.FP64, return_p=True)
    assert np.array_equal(p, s.get_pressure())
    s.step(2, prec=ng.FP64)
    got = s.get_state()
    size = len(u[0])
    out = tuple(torch.zeros(k * size, dtype=torch.float64).pin_memory().numpy().reshape(-1, k)
                for k in (1, 3, 1))
    s.get_state_raw(*out)
    assert np.array_equal(got[0], out[0][:, 0]) and np.array_equal(got[4], out[2][:, 0])
    for c in range(3):
        assert np.array_equal(got[1 + c], out[1][:, c])
    s.set_state(u)
    again = s.tendency(ng.FP64)
    assert all(np.array_equal(a, b) for a, b in zip(L, again))
    bad = [x.copy() for x in u]
    bad[4][size // 2] = np.nan
    s.set_state(bad)
    with pytest.raises(ng.NsemError):
        s.step(1, prec=ng.FP64)
        s.get_state()
    s.close()
