"""What the float-pair kernels must hand over to FP64: windows whose smoothness terms leave
the pairs' range beside constant states.

Tolerance: the path's 1e-12 relative L2 per right-hand side against the oracle, each
component by itself."""
import numpy as np
import pytest

import oracle as O
from hypar_gb300 import cases as C
from hypar_gb300.solver import Solver

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
RHS_TOL = 1e-12


def conserved(rho, vel, p):
    e = p / 0.4 + 0.5 * rho * sum(v * v for v in vel)
    return np.stack([rho] + [rho * v for v in vel] + [e], axis=-1).reshape(-1, len(vel) + 2)


def build_case(size, interp, upw, state, weights="js", scheme="weno5"):
    """`state`: (rho, velocities, p) over the grid coordinates [0, 1) per dimension."""
    base = {1: C.sod(16, n_iter=1), 2: C.vortex(16, n_iter=1), 3: C.tgv(8, n_iter=1)}[len(size)]
    base.interp, base.upwinding, base.weights, base.Re, base.hyp_scheme = interp, upw, weights, None, scheme
    base.size = list(size)
    base.x = [np.arange(n) / n for n in size]
    x = list(reversed(np.meshgrid(*[np.arange(n) / n for n in reversed(size)], indexing="ij")))
    base.u = conserved(*state(x))
    return base


def both(case, tmp_path):
    """The right-hand side of the oracle and of the kernels, (points, components)."""
    d = str(tmp_path / "deck")
    case.write(d)
    s = Solver.from_dir(d)
    P = O.Problem(case)
    u0 = P.u0()
    ref = O.interior(P.rhs(u0), case.size, case.nvars, 3).reshape(-1, case.nvars)
    u = torch.from_numpy(u0).cuda()
    out = torch.zeros_like(u)
    s.rhs(out, u)
    return ref, O.interior(out.cpu().numpy(), case.size, case.nvars, 3).reshape(-1, case.nvars)


def check(case, tmp_path):
    ref, got = both(case, tmp_path)
    for v in range(case.nvars):
        n = np.linalg.norm(ref[:, v])
        assert np.linalg.norm(got[:, v] - ref[:, v]) <= RHS_TOL * n, v


@pytest.mark.parametrize("size,interp,upw,weights,scheme", [
    ((90,), "components", "roe", "js", "weno5"), ((90,), "characteristic", "llf-char", "js", "weno5"),
    ((48, 30), "components", "roe", "js", "weno5"), ((48, 30), "characteristic", "roe", "mapped", "weno5"),
    ((48, 30), "components", "llf-char", "none", "weno5"), ((16, 14, 12), "components", "roe", "mapped", "weno5"),
    ((16, 14, 12), "characteristic", "rf-char", "js", "weno5"), ((48, 30), "components", "roe", "js", "crweno5")])
@pytest.mark.parametrize("p", [4e18, 8e18, 1e19])
def test_constant_states_beside_a_large_jump(built_lib, oracle_lib, tmp_path, size, interp, upw, weights, scheme, p):
    """Two constant states at rest whose jump squared leaves the FP32 range: the constant
    sub-stencils keep the weights' sum in range."""

    def state(x):
        left = x[0] < 0.5
        for xi in x[1:]:
            left = left ^ (xi < 0.5)
        one = np.ones_like(x[0])
        return np.where(left, 1.0, 0.4) * one, [0.0 * one for _ in x], np.where(left, p, 0.3 * p) * one

    check(build_case(size, interp, upw, state, weights, scheme), tmp_path)


@pytest.mark.parametrize("size,interp,upw,weights,scheme", [
    ((128,), "components", "roe", "js", "weno5"), ((128,), "characteristic", "roe", "js", "weno5"),
    ((64, 20), "components", "roe", "js", "weno5"), ((64, 20), "characteristic", "llf-char", "mapped", "weno5"),
    ((64, 20), "components", "rf-char", "borges", "weno5"), ((64, 8, 9), "components", "rusanov", "yc", "weno5"),
    ((64, 8, 9), "characteristic", "roe", "js", "weno5"), ((64, 20), "components", "roe", "yc", "crweno5")])
@pytest.mark.parametrize("rho0,a", [(1e-24, 1e6), (1e-12, 1e-3), (1e-15, 1.0), (1e-12, 1e10), (1e18, 1e-15), (1e-9, 1e3)])
def test_density_and_speed_far_apart(built_lib, oracle_lib, tmp_path, size, interp, upw, weights, scheme, rho0, a):
    """Small waves in units whose density and speed differ widely: the differences of the
    states may lie below what pairs hold where the fluxes do not.

    Tolerance: a flux is a dozen roundings of its scale (density, momentum, energy times the
    speed), in the kernel and in the oracle: 32 units of 2^-53 of it over the spacing; the
    line solves of the compact scheme add up the roundings of a few neighbours: 4 times that."""

    def state(x):
        w = 1e-5 * np.sin(2 * np.pi * x[0])
        return rho0 * (1 + w), [a * (0.3 + w) for _ in x], rho0 * a * a / 1.4 * (1 + 1.4 * w)

    case = build_case(size, interp, upw, state, weights, scheme)
    ref, got = both(case, tmp_path)
    u = case.u
    vel = u[:, 1:-1] / u[:, :1]
    p = 0.4 * (u[:, -1] - 0.5 * u[:, 0] * (vel ** 2).sum(1))
    lam = (np.abs(vel).max(1) + np.sqrt(1.4 * p / u[:, 0])).max()
    if upw == "roe":
        lam = max(lam, 5e-7)  # the entropy fix's least dissipation speed (Harten, delta = 1e-6)
    scale = u[:, 0].max() * lam * np.array([1.0] + [lam] * vel.shape[1] + [((u[:, -1] + p) / u[:, 0]).max()])
    tol = 32 * (4 if scheme == "crweno5" else 1) * 2.0 ** -53 * scale * max(size)
    assert (np.abs(got - ref).max(0) <= tol).all(), np.abs(got - ref).max(0) / tol
