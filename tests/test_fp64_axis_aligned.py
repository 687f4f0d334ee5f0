"""The FP64 forms on elements whose metric is diagonal and on faces whose
normal lies along an axis, against the oracle bit for bit: the kernels leave
out products with the metric's and normal's zeros there.  Also an element
with a full metric among diagonal ones, and non-finite states, which must
spread to the same nodes as in the full products."""
import numpy as np
import pytest

import nebulasem_gb300 as ng
from nebulasem_gb300 import mesh as ngmesh

pytestmark = pytest.mark.gpu

CONST = dict(P0=1e5, T0=300.0, cp=1004.5, cv=717.5, gravity=np.array([0.0, 0.0, -9.81]), Pr=0.9)


def _setup(n, order, dim, visc, tilt=0.0):
    h = 62.5
    m = ngmesh.box_mesh(n, order, tuple(h * x for x in n), dim=dim, tilt=tilt)
    n_int = int(m["meta"][7])
    centre = [h * x / 2 for x in n]
    u, m["p_ref"], m["rho_ref"], m["gh"] = ngmesh.bubble_state(m, 0.5, centre, (80.0,) * 3)
    rng = np.random.default_rng(order)
    for c in (1, 2, 3) if dim == 3 else (1, 3):
        u[c] = u[0] * rng.uniform(-1.0, 1.0, n_int)
    m.update(CONST, viscosity=visc)
    return m, u, 0.02 / order ** 2


def _oracle(m, dt):
    import oracle
    return oracle, oracle.OracleMesh(dict(m, dt=dt))


def _same(a, b):
    return all(np.array_equal(np.asarray(x).reshape(-1), np.asarray(y).reshape(-1), equal_nan=True)
               for x, y in zip(a, b))


@pytest.mark.parametrize("visc", [0.0, 1.5])
@pytest.mark.parametrize("n,dim,order", [((2, 1, 1), 3, 9), ((3, 2, 4), 3, 2), ((2, 3, 2), 3, 4), ((2, 2, 3), 3, 7),
                                         ((1, 1, 1), 3, 5), ((5, 1, 3), 2, 1), ((4, 1, 5), 2, 6)])
def test_forms_equal_oracle(n, dim, order, visc):
    if order == 9 and visc:
        pytest.skip("the gradient kernel's registers hold up to order 8")
    m, u, dt = _setup(n, order, dim, visc)
    oracle, o = _oracle(m, dt)
    s = ng.Solver(m, dt=dt)
    U = np.stack([u[1] / u[0], u[2] / u[0], u[3] / u[0]], axis=1)
    T = u[4] / u[0] - CONST["T0"]
    wind = U + np.array([6.0, -4.0, 5.0])
    oracle.set_pow(1)
    try:
        s.set_state(u)
        assert _same(s.tendency(ng.FP64), o.tendency(u))
        s.step(3)
        assert _same(s.get_state(), o.ssprk3(u, dt, 3))
        s.set_fields(u[0], U, T)
        s.step(3, scheme=ng.REF_SEGREGATED)
        assert _same(s.get_fields(), o.segregated(u[0], U, T, dt, 3))
    finally:
        oracle.set_pow(0)
    s.convection_set(wind, T)
    s.convection_step(3)
    assert _same([s.convection_get()], [o.convection(wind, T, dt, 3)])
    s.close()


@pytest.mark.parametrize("tilt", [0.0, 30.0])
@pytest.mark.parametrize("scale", [1e-40, 1e-100, 1e-155, 1e-300, 1e50, 1e70])
def test_values_outside_the_integer_products_range(scale, tilt):
    """Momenta of every size, in one element and in all: products, squares and
    fluxes that are subnormal or zero take the FP64 products."""
    for one in (True, False):
        m, u, dt = _setup((3, 2, 2), 4, 3, 0.0, tilt)
        at = slice(125, 250) if one else slice(None)
        for c in (1, 2, 3):
            u[c][at] *= scale
        oracle, o = _oracle(m, dt)
        s = ng.Solver(m, dt=dt)
        U = np.stack([u[1] / u[0], u[2] / u[0], u[3] / u[0]], axis=1)
        T = u[4] / u[0] - CONST["T0"]
        oracle.set_pow(1)
        try:
            s.set_state(u)
            assert _same(s.tendency(ng.FP64), o.tendency(u))
            if scale < 1:
                s.step(2)
                assert _same(s.get_state(), o.ssprk3(u, dt, 2))
                s.set_fields(u[0], U, T)
                s.step(2, scheme=ng.REF_SEGREGATED)
                assert _same(s.get_fields(), o.segregated(u[0], U, T, dt, 2))
        finally:
            oracle.set_pow(0)
        s.close()


@pytest.mark.parametrize("visc", [0.0, 1.5])
def test_full_metric_among_diagonal_elements(visc):
    m, u, dt = _setup((3, 2, 2), 4, 3, visc)
    J = m["Jinv"].reshape(-1, 9)
    J[125:250, 3:] = 1e-4          # one element with every component set
    J[400, 5] = -1e-9              # one node of another
    m["fN"].reshape(-1, 3)[40:60] += 1e-3
    oracle, o = _oracle(m, dt)
    s = ng.Solver(m, dt=dt)
    oracle.set_pow(1)
    try:
        s.set_state(u)
        s.step(2)
        assert _same(s.get_state(), o.ssprk3(u, dt, 2))
    finally:
        oracle.set_pow(0)
    s.close()


@pytest.mark.parametrize("visc", [0.0, 1.5])
@pytest.mark.parametrize("var,value", [(0, np.nan), (1, np.inf), (2, -np.inf), (4, np.inf), (3, 1e250)])
def test_non_finite_values_spread_as_in_the_full_products(var, value, visc):
    m, u, dt = _setup((3, 2, 2), 4, 3, visc)
    u[var][300] = value            # a node on a face of the third element
    oracle, o = _oracle(m, dt)
    s = ng.Solver(m, dt=dt)
    oracle.set_pow(1)
    try:
        s.set_state(u)
        got, want = s.tendency(ng.FP64), o.tendency(u)
    finally:
        oracle.set_pow(0)
    s.close()
    for a, b in zip(got, want):
        assert np.array_equal(np.isfinite(a), np.isfinite(b))
        assert np.array_equal(a[np.isfinite(b)], b[np.isfinite(b)])


@pytest.mark.parametrize("n,dim,order,visc,tilt", [((3, 2, 2), 3, 4, 0.0, 0.0), ((2, 2, 3), 3, 3, 1.5, 0.0),
                                                   ((4, 1, 3), 2, 5, 0.0, 0.0), ((2, 2, 2), 3, 4, 0.0, 30.0)])
def test_transpose_of_the_tangent(n, dim, order, visc, tilt):
    """<w, J dv> = <J^T w, dv>: each side sums n_int products of rounding error
    below 1e-14 of its terms, so 1e-12 of the sum of magnitudes bounds it."""
    m, u, dt = _setup(n, order, dim, visc, tilt)
    rng = np.random.default_rng(3)
    s = ng.Solver(m, dt=dt)
    s.set_state(u)
    dv = [a * rng.standard_normal(len(a)) * 1e-3 + (1e-3 if c in (1, 3) else 0.0) for c, a in enumerate(u)]
    w = [rng.standard_normal(len(u[0])) for _ in range(5)]
    Jd, Jw = s.jvp(dv), s.vjp(w)
    s.close()
    lhs = sum(np.dot(a, b) for a, b in zip(w, Jd))
    rhs = sum(np.dot(a, b) for a, b in zip(Jw, dv))
    scale = sum(np.abs(a * b).sum() for a, b in zip(w, Jd))
    assert abs(lhs - rhs) <= 1e-12 * scale
