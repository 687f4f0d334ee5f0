"""FP64 forms at the limits of the integer products' range: on walls whose
weight and normal, and fields whose density, gradients and viscosity, are each
small, the viscous face flux is subnormal though none of its factors is; and
viscous states with momenta of every size.  The same bits as the oracle's."""
import numpy as np
import pytest

import nebulasem_gb300 as ng
from nebulasem_gb300 import mesh as ngmesh

pytestmark = pytest.mark.gpu

CONST = dict(P0=1e5, T0=300.0, cp=1004.5, cv=717.5, gravity=np.array([0.0, 0.0, -9.81]))


def _box(n, order, tilt=0.0):
    h = 62.5
    m = ngmesh.box_mesh(n, order, tuple(h * x for x in n), tilt=tilt)
    u, m["p_ref"], m["rho_ref"], m["gh"] = ngmesh.bubble_state(m, 0.5, [h * x / 2 for x in n], (80.0,) * 3)
    return m, u


def _same(a, b):
    return all(np.array_equal(np.asarray(x).reshape(-1), np.asarray(y).reshape(-1), equal_nan=True)
               for x, y in zip(a, b))


# exponents of the wall's fI, with the normals at 2^-195: products of fI, n, nu,
# 1 / Pr, rho and the gradient from 2^-985 (normal) to 2^-1045 (subnormal)
@pytest.mark.parametrize("weight", [1.0, 2.0 ** -30, 2.0 ** -60])
def test_subnormal_viscous_wall_flux(weight):
    import oracle

    m, u = _box((2, 2, 2), 3)
    rng = np.random.default_rng(3)
    size = len(u[0])
    u[0] = 1e-60 * rng.uniform(1.0, 2.0, size)
    for c in (1, 2, 3):
        u[c] = np.zeros(size)
    u[4] = u[0] * (1e-57 * rng.uniform(1.0, 2.0, size))
    m["fN"] = m["fN"] * 1e-60
    m["fI"] = np.where(m["fI"] == 0.0, weight, m["fI"])
    m.update(CONST, viscosity=1e-60, Pr=1e60)
    s = ng.Solver(m, dt=1e-3)
    s.set_state(u)
    got = s.tendency(ng.FP64)
    s.close()
    oracle.set_pow(1)
    try:
        want = oracle.OracleMesh(dict(m, dt=1e-3)).tendency(u)
    finally:
        oracle.set_pow(0)
    assert _same(got, want)


@pytest.mark.parametrize("tilt", [0.0, 30.0])
@pytest.mark.parametrize("scale", [1e-40, 1e-100, 1e-155, 1e-300, 1e50])
def test_viscous_momenta_of_every_size(scale, tilt):
    import oracle

    m, u = _box((3, 2, 2), 4, tilt)
    rng = np.random.default_rng(4)
    for c in (1, 2, 3):
        u[c] = u[0] * rng.uniform(-1.0, 1.0, len(u[0]))
        u[c][125:250] *= scale          # the second element
    m.update(CONST, viscosity=1.5, Pr=0.9)
    dt = 1e-3
    o = oracle.OracleMesh(dict(m, dt=dt))
    s = ng.Solver(m, dt=dt)
    oracle.set_pow(1)
    try:
        s.set_state(u)
        assert _same(s.tendency(ng.FP64), o.tendency(u))
        if scale < 1:
            s.step(2)
            assert _same(s.get_state(), o.ssprk3(u, dt, 2))
            U, T = np.stack([u[c] / u[0] for c in (1, 2, 3)], axis=1), u[4] / u[0] - CONST["T0"]
            s.set_fields(u[0], U, T)
            s.step(2, scheme=ng.REF_SEGREGATED)
            assert _same(s.get_fields(), o.segregated(u[0], U, T, dt, 2))
    finally:
        oracle.set_pow(0)
    s.close()
