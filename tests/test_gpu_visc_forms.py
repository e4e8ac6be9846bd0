"""Which form the viscous term takes in a right-hand side (float pairs or FP64), and that it
makes no difference beyond the rounding of the fluxes.

gb_ParabolicFunction is FP64 throughout, and a right-hand side subtracts the hyperbolic term
from the viscous one, so that the right-hand side equals parabolic - hyperbolic bit for bit if
and only if its viscous term was formed in FP64."""
import numpy as np
import pytest

from hypar_gb300 import cases as C
from hypar_gb300.solver import Solver

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def terms(case, tmp_path):
    """(right-hand side, parabolic - hyperbolic), interior points by components."""
    d = str(tmp_path / "deck")
    case.write(d)
    s = Solver.from_dir(d)
    shape = [n + 6 for n in reversed(case.size)] + [5]
    u = torch.zeros(shape, dtype=torch.float64, device="cuda")
    u[3:-3, 3:-3, 3:-3] = torch.from_numpy(case.u.reshape(list(reversed(case.size)) + [5]).copy()).cuda()
    rhs, hyp, par = (torch.zeros_like(u) for _ in range(3))
    s.rhs(rhs, u)
    s.apply_bc(u)
    s.hyperbolic(hyp, u)
    s.parabolic(par, u)
    return tuple(q[3:-3, 3:-3, 3:-3].reshape(-1, 5).cpu().numpy() for q in (rhs, par - hyp))


def flux_scale(case):
    u = case.u
    v = u[:, 1:4] / u[:, :1]
    p = 0.4 * (u[:, 4] - 0.5 * u[:, 0] * (v ** 2).sum(1))
    lam = np.abs(v).max(1) + np.sqrt(1.4 * p / u[:, 0])
    rl = u[:, 0] * lam
    return np.stack([rl, rl * lam, rl * lam, rl * lam, lam * (u[:, 4] + p)], 1).max(0) / (case.x[0][1] - case.x[0][0])


def scaled(case, rho, a, h):
    """The case in units of rho, a and h, its viscosity 1/100 of the least that FP64 is taken for."""
    case.u = case.u * rho * np.array([1.0, a, a, a, a * a])
    case.x = [x * h for x in case.x]
    dx = case.x[0][1] - case.x[0][0]
    case.Minf, case.Re = 1.0, 100.0 * 32.0 * (a * a) ** 0.76 / dx / (rho * a)
    return case


@pytest.mark.parametrize("rho,a,h", [(1.0, 1.0, 1.0), (1e-16, 1e-8, 1.0), (1e-17, 1e-3, 1e3), (1.2, 340.0, 1e-2),
                                     (1e14, 1e4, 1e-14), (1e-6, 1e-2, 1e6), (1e6, 1e5, 1e-6)])
def test_viscous_term_in_any_units(built_lib, tmp_path, rho, a, h):
    """Tolerance: the pairs are held to a quarter of the rounding of the convective flux, the sum
    rounds twice: 2 units of 2^-53 of the flux scale over the spacing."""
    case = scaled(C.tgv(12, n_iter=1, perturb=0.05), rho, a, h)
    rhs, ref = terms(case, tmp_path)
    tol = 2.0 * 2.0 ** -53 * flux_scale(case)
    assert (np.abs(rhs - ref).max(0) <= tol).all(), np.abs(rhs - ref).max(0) / tol


def test_forms_of_the_periodic_box(built_lib, tmp_path):
    case = C.tgv(12, n_iter=1, perturb=0.05)
    (tmp_path / "a").mkdir()
    (tmp_path / "b").mkdir()
    rhs, ref = terms(case, tmp_path / "a")
    assert not np.array_equal(rhs, ref)  # pairs
    case.Re = 0.5
    rhs, ref = terms(case, tmp_path / "b")
    assert np.array_equal(rhs, ref)  # FP64


@pytest.mark.parametrize("wall", ["slip-wall", "noslip-wall"])
@pytest.mark.parametrize("dims", [(0, 1), (1, 2), (0, 1, 2)], ids=["duct-z", "duct-x", "box"])
def test_forms_between_walls(built_lib, tmp_path, dims, wall):
    """Walls in two or three directions: the edges' ghost points, which no wall fills, do not
    decide the form."""
    case = C.tgv(12, n_iter=1, perturb=0.05)
    case.bcs = {(d, f): (wall, [0.0, 0.0, 0.0]) for d in dims for f in (1, -1)}
    rhs, ref = terms(case, tmp_path)
    assert np.isfinite(rhs).all()
    assert not np.array_equal(rhs, ref)  # pairs
    tol = 2.0 * 2.0 ** -53 * flux_scale(case)
    assert (np.abs(rhs - ref).max(0) <= tol).all(), np.abs(rhs - ref).max(0) / tol


def test_replays_of_a_captured_step_do_not_depend_on_history(built_lib, tmp_path):
    """A captured step gives the same bits for the same state after a replay whose state was
    refused the pairs (thin gas: the viscous term is not small)."""
    case = C.tgv(12, n_iter=1, perturb=0.05)
    d = str(tmp_path / "deck")
    case.write(d)
    s = Solver.from_dir(d)
    stream = torch.cuda.Stream()
    s.set_stream(stream.cuda_stream)
    s.step(1)
    s.sync()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        s.step(1)

    def replay(u):
        s.set_state(u.reshape(-1))
        with torch.cuda.stream(stream):
            graph.replay()
        stream.synchronize()
        return s.get_state()

    first = replay(case.u)
    thin = replay(case.u * 1e-4)
    assert np.isfinite(thin).all()
    assert np.array_equal(replay(case.u), first)
    s.set_state(case.u.reshape(-1))
    s.step(1)
    assert np.array_equal(s.get_state(), first)
