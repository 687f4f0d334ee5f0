"""The adjoint's density row: with no wind and weights on the momentum rows
alone, rho acts through the gravity source only (the pressure depends on
rho theta, every other term has a factor U), so J^T w there is g . w.  The
kernel forms it as (w / cV) g cV: three roundings of 2^-53, and zeros; 4 are
allowed.  The pressure's adjoint must not pass through that row, where shares
of gamma p / rho would cancel and leave their rounding."""
import numpy as np
import pytest

import nebulasem_gb300 as ng
from nebulasem_gb300 import mesh as ngmesh
from conftest import load_golden

pytestmark = pytest.mark.gpu

G = np.array([0.0, 0.0, -9.81])


def _check(m, u, visc):
    rng = np.random.default_rng(1)
    size = len(u[0])
    zero = np.zeros(size)
    u = [u[0], zero, zero, zero, u[4]]
    w = [zero] + [rng.standard_normal(size) for _ in range(3)] + [zero]
    s = ng.Solver(m, dt=1e-3, gravity=G, viscosity=visc, Pr=0.9)
    s.set_state(u)
    got = s.vjp(w)[0]
    s.close()
    want = G[2] * w[3]
    assert np.all(np.abs(got - want) <= 4 * 2.0 ** -53 * np.abs(want))


@pytest.mark.parametrize("visc", [0.0, 1.5])
@pytest.mark.parametrize("n,order,dim,tilt", [((2, 2, 2), 3, 3, 0.0), ((2, 3, 2), 4, 3, 30.0), ((4, 1, 3), 4, 2, 0.0),
                                              ((1, 1, 2), 7, 3, 0.0)])
def test_boxes(n, order, dim, tilt, visc):
    h = 125.0
    m = ngmesh.box_mesh(n, order, tuple(h * x for x in n), dim=dim, tilt=tilt)
    u, m["p_ref"], m["rho_ref"], m["gh"] = ngmesh.bubble_state(m, 0.5, [h * x / 2 for x in n], (120.0,) * 3)
    _check(m, u, visc)


@pytest.mark.parametrize("visc", [0.0, 1.5])
@pytest.mark.parametrize("name", ["amr_g3_4n3", "amr_hill_2d_visc"])
def test_refined_meshes(name, visc):
    g = load_golden(name)
    _check(g, [g[f"u0_{v}"] for v in ("rho", "rhou", "rhov", "rhow", "rhotheta")], visc)
