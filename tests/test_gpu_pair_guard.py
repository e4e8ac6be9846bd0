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
