"""The float-pair direction kernels at the edges of their blocks: lines shorter than the
halo, around one and two pieces of a line, around the lines a block takes, with smooth and
discontinuous data in the same warp (pairs and the FP64 evaluation side by side), in units
that leave the pairs' range, and for every weight formulation.

Tolerance: the path's 1e-12 relative L2 per right-hand side against the oracle."""
import numpy as np
import pytest

import oracle as O
from hypar_gb300 import cases as C
from hypar_gb300.solver import Solver

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
RHS_TOL = 1e-12


def state(size, jump, unit):
    """Waves of a few cells' to a line's length; `jump`: a block of denser, hotter gas."""
    nd = len(size)
    grids = np.meshgrid(*[np.arange(n) / max(n, 12) for n in reversed(size)], indexing="ij")
    x = list(reversed(grids))
    ph = sum((k + 1.0) * xi for k, xi in enumerate(x)) * 2 * np.pi
    rho, p = 1.0 + 0.1 * np.sin(ph), 1.0 + 0.1 * np.cos(ph + 0.3)
    vel = [0.3 + 0.1 * np.sin(ph + d) for d in range(nd)]
    if jump:
        box = np.ones_like(rho, dtype=bool)
        for xi, n in zip(x, size):
            box &= (xi * max(n, 12) >= n // 3) & (xi * max(n, 12) < n // 3 + max(2, n // 4))
        rho, p = np.where(box, rho + 1.0, rho), np.where(box, p + 2.0, p)
    rho, p = rho * unit, p * unit
    e = p / 0.4 + 0.5 * rho * sum(v * v for v in vel)
    return np.stack([rho] + [rho * v for v in vel] + [e], axis=-1).reshape(-1, nd + 2)


def build_case(size, interp, upw, weights="js", jump=False, unit=1.0):
    nd = len(size)
    base = {1: C.sod(16, n_iter=1), 2: C.vortex(16, n_iter=1), 3: C.tgv(8, n_iter=1)}[nd]
    base.interp, base.upwinding, base.weights, base.Re = interp, upw, weights, None
    base.size = list(size)
    base.x = [np.arange(n) / max(n, 12) for n in size]
    base.u = state(size, jump, unit)
    return base


def check(case, tmp_path, block=None):
    d = str(tmp_path / "deck")
    case.write(d)
    s = Solver.from_dir(d)
    if block:
        for dd in range(len(case.size)):
            s.set_launch(dd, 0, block)
    P = O.Problem(case)
    u0 = P.u0()
    ref = O.interior(P.rhs(u0), case.size, case.nvars, 3)
    u = torch.from_numpy(u0).cuda()
    out = torch.zeros_like(u)
    s.rhs(out, u)
    got = O.interior(out.cpu().numpy(), case.size, case.nvars, 3)
    assert np.linalg.norm(got - ref) <= RHS_TOL * np.linalg.norm(ref)


SIZES = [(3,), (7,), (57,), (58,), (59,), (117,), (251,), (3, 130), (59, 5), (250, 4), (61, 33), (5, 7, 66), (31, 3, 26)]


@pytest.mark.parametrize("jump", [False, True], ids=["smooth", "jump"])
@pytest.mark.parametrize("interp", ["components", "characteristic"])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
def test_block_edges(built_lib, oracle_lib, tmp_path, size, interp, jump):
    check(build_case(size, interp, "roe", jump=jump), tmp_path)


@pytest.mark.parametrize("block", [32, 64, 96])
@pytest.mark.parametrize("upw", ["llf-char", "rf-char"])
@pytest.mark.parametrize("size", [(130,), (61, 33), (13, 9, 31)], ids=lambda s: "x".join(map(str, s)))
def test_block_sizes(built_lib, oracle_lib, tmp_path, size, upw, block):
    check(build_case(size, "characteristic", upw, jump=True), tmp_path, block)


@pytest.mark.parametrize("weights", ["mapped", "borges", "yc", "none"])
@pytest.mark.parametrize("interp", ["components", "characteristic"])
def test_weights_with_jumps(built_lib, oracle_lib, tmp_path, interp, weights):
    check(build_case((61, 33), interp, "roe", weights, jump=True), tmp_path)


@pytest.mark.parametrize("unit", [1e-30, 1e-6, 1e9, 1e30])
@pytest.mark.parametrize("model", [(90,), (40, 30), (12, 14, 9)], ids=["1d", "2d", "3d"])
def test_units(built_lib, oracle_lib, tmp_path, model, unit):
    """Densities and pressures far from 1: the pairs' range check hands over to FP64."""
    check(build_case(model, "components", "roe", jump=True, unit=unit), tmp_path)


@pytest.mark.parametrize("Re", [0.5, 20.0, 1600.0])
def test_viscous_regimes(built_lib, oracle_lib, tmp_path, Re):
    """Viscous fluxes from dominant (FP64 throughout) to small (pairs) against the convective ones."""
    case = C.tgv(12, n_iter=1, dt=1e-3, perturb=0.05)
    case.Re = Re
    check(case, tmp_path)
