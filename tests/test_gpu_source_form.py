"""The well-balanced source as a difference of two evaluations of the hyperbolic term: an
interface takes the same form (float pairs or FP64) in both, so that the components without a
source come out as exactly zero.  (Component-wise: the FP64 form of the characteristic
reconstruction rounds differently with and without a source.)"""
import numpy as np
import pytest

from hypar_gb300 import cases as C
from hypar_gb300.solver import Solver

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", ["navierstokes3d", "euler1d"])
def test_components_without_a_source_are_zero(built_lib, tmp_path, model):
    """Pressure far below RT rho_ref and a hydrostatic field with waves of ten cells: the source's
    terms are not small against the flux where the flux's own are."""
    if model == "euler1d":
        case = C.stratified_1d(200, n_iter=1)
        n, yd, g = 200, 0, 3
    else:
        case = C.rising_thermal_bubble(20, n_iter=1)
        n, yd, g = 20, 1, 3
    nd = len(case.size)
    rho = case.u[:, 0]
    vel = 0.1 * np.sqrt(case.u[:, -1:] / rho[:, None]) * np.ones((1, nd))
    e = case.u[:, -1] / 300.0
    vel = vel / np.sqrt(300.0)
    case.u = np.concatenate([rho[:, None], rho[:, None] * vel, (e + 0.5 * rho * (vel ** 2).sum(1))[:, None]], axis=1)
    d = str(tmp_path / "deck")
    case.write(d)
    s = Solver.from_dir(d)
    y = np.arange(-g, n + g) * 2.0 * np.pi / 10.0
    gg = 1.0 + 0.02 * np.sin(y)
    shape = [m + 2 * g for m in reversed(case.size)]
    gg = np.broadcast_to(gg.reshape([-1 if k == nd - 1 - yd else 1 for k in range(nd)]), shape).reshape(-1)
    s.set_gravity_field(np.concatenate([1.0 / gg, gg]))
    u = torch.zeros(shape + [case.nvars], dtype=torch.float64, device="cuda")
    inner = tuple(slice(g, -g) for _ in range(nd))
    u[inner] = torch.from_numpy(case.u.reshape([m for m in reversed(case.size)] + [case.nvars]).copy()).cuda()
    s.apply_bc(u)
    src = torch.zeros_like(u)
    s.source(src, u)
    src = src[inner].reshape(-1, case.nvars)
    assert float(src[:, 1 + yd].abs().max()) > 0.0
    for v in range(case.nvars):
        if v not in (1 + yd, case.nvars - 1):
            assert float(src[:, v].abs().max()) == 0.0, v
