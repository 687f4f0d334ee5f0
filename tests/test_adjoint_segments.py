"""The reverse sweep's segments: the last one's stage states are kept from the
forward run, the others recomputed.  The recomputed states are the same bits,
so the gradient does not depend on the checkpoint interval, on a second call,
or on what other calls did to the storage in between."""
import numpy as np
import pytest

import nebulasem_gb300 as ng
from nebulasem_gb300 import mesh as ngmesh

pytestmark = pytest.mark.gpu


def _solver(visc=0.0):
    h, n = 125.0, (3, 2, 3)
    m = ngmesh.box_mesh(n, 4, tuple(h * x for x in n))
    u, m["p_ref"], m["rho_ref"], m["gh"] = ngmesh.bubble_state(
        m, 0.5, [h * x / 2 for x in n], (120.0,) * 3)
    rng = np.random.default_rng(5)
    for c in (1, 2, 3):
        u[c] = u[0] * rng.uniform(-0.5, 0.5, len(u[0]))
    lam = [rng.standard_normal(len(u[0])) for _ in range(5)]
    return ng.Solver(m, dt=0.01, viscosity=visc), u, lam


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("visc", [0.0, 1.5])
@pytest.mark.parametrize("prec", [ng.FP64, ng.MIXED])
def test_gradient_independent_of_the_interval(prec, visc):
    s, u, lam = _solver(visc)
    s.set_state(u)
    s.forward_checkpointed(7, 7, prec)     # one segment: nothing recomputed
    end = s.get_state()
    want, _ = s.adjoint(lam)
    for every in (1, 2, 3, 6, 7, 50):
        s.set_state(u)
        s.forward_checkpointed(7, every, prec)
        got, _ = s.adjoint(lam)
        assert _same(got, want), every
        assert _same(s.get_state(), end), every
        again, _ = s.adjoint(lam)          # the storage now holds the first segment
        assert _same(again, want), every
    s.close()


@pytest.mark.parametrize("prec", [ng.FP64, ng.MIXED])
def test_other_calls_between_forward_and_adjoint(prec):
    s, u, lam = _solver()
    s.set_state(u)
    s.forward_checkpointed(5, 2, prec)
    want, _ = s.adjoint(lam)
    s.set_state(u)
    s.forward_checkpointed(5, 2, prec)
    s.step(2, prec=ng.FP64)
    s.step(3, prec=ng.MIXED)
    s.vjp(lam, prec)
    s.tlm(2, lam)                          # uses the FP64 stage-state storage
    got, _ = s.adjoint(lam)
    assert _same(got, want)
    # a longer run after a shorter one, and a shorter one after it
    for nsteps, every in ((9, 4), (3, 2)):
        s.set_state(u)
        s.forward_checkpointed(nsteps, every, prec)
        a, _ = s.adjoint(lam)
        s.set_state(u)
        s.forward_checkpointed(nsteps, nsteps, prec)
        b, _ = s.adjoint(lam)
        assert _same(a, b)
    s.close()
