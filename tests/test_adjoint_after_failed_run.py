"""The reverse sweep belongs to the last checkpointed run: after one that failed
there is nothing to differentiate, also where an earlier run of the other form
had ended well; a call that is refused before it starts leaves that run."""
import numpy as np
import pytest

import nebulasem_gb300 as ng
from nebulasem_gb300 import mesh as ngmesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first,failing", [(ng.MIXED, ng.FP64), (ng.FP64, ng.MIXED), (ng.FP64, ng.FP64),
                                           (ng.MIXED, ng.MIXED)])
def test_no_gradient_of_an_older_run(first, failing):
    h, n = 125.0, (2, 2, 2)
    m = ngmesh.box_mesh(n, 4, tuple(h * x for x in n))
    u, m["p_ref"], m["rho_ref"], m["gh"] = ngmesh.bubble_state(m, 0.5, [h] * 3, (120.0,) * 3)
    rng = np.random.default_rng(7)
    lam = [rng.standard_normal(len(u[0])) for _ in range(5)]
    s = ng.Solver(m, dt=0.01)
    s.set_state(u)
    s.forward_checkpointed(3, 2, first)
    want, _ = s.adjoint(lam)
    with pytest.raises(ng.NsemError):      # refused: the run before stands
        s.forward_checkpointed(0, 2, failing)
    got, _ = s.adjoint(lam)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
    bad = [x.copy() for x in u]
    bad[4][len(u[0]) // 2] = np.nan
    s.set_state(bad)
    with pytest.raises(ng.NsemError):
        s.forward_checkpointed(3, 2, failing)
    with pytest.raises(ng.NsemError):
        s.adjoint(lam)
    s.set_state(u)
    s.forward_checkpointed(3, 2, first)
    got, _ = s.adjoint(lam)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
    s.close()
