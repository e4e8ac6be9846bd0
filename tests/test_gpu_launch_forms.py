"""The forms a launch shape selects: float pairs (seg = GB_SEG_AUTO, the default, `block` the most threads
of a block) and the FP64 kernels (segments, tiles), on solvers and ensembles; and the
autotuner's choice between them.

Tolerances: steps agree with the oracle to 1e-10 relative L2, as everywhere; two forms of one
step differ by rounding, so that equal bits mean that the same form ran."""
import numpy as np
import pytest

import oracle as O
from hypar_gb300 import cases as C
from hypar_gb300.adjoint import Adjoint
from hypar_gb300.solver import Ensemble, Inputs, Solver

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
AUTO = 1 << 30  # GB_SEG_AUTO


def solver_for(case, tmp_path, name="deck"):
    d = str(tmp_path / name)
    case.write(d)
    return Solver.from_dir(d)


def rough(case, a, seed=5):
    """Noise of relative amplitude a on density, velocity (of the speed of sound) and pressure."""
    r = np.random.default_rng(seed)
    u, nd, n = case.u, len(case.size), len(case.u)
    vel = u[:, 1:1 + nd] / u[:, :1]
    p = 0.4 * (u[:, -1] - 0.5 * u[:, 0] * (vel ** 2).sum(1))
    c = np.sqrt(1.4 * p / u[:, 0])
    rho, p = u[:, 0] * (1 + a * r.uniform(-1, 1, n)), p * (1 + a * r.uniform(-1, 1, n))
    vel = vel + a * c[:, None] * r.uniform(-1, 1, (n, nd))
    case.u = np.concatenate([rho[:, None], rho[:, None] * vel,
                             (p / 0.4 + 0.5 * rho * (vel ** 2).sum(1))[:, None]], 1)
    return case


def with_scheme(case, scheme):
    case.hyp_scheme = scheme
    return case


MAKE = {"euler1d": lambda: C.sod(128, n_iter=2), "euler2d": lambda: C.vortex(40, n_iter=2),
        "navierstokes3d": lambda: C.isotropic_turbulence(14, n_iter=2),
        "gravity": lambda: C.rising_thermal_bubble(16, n_iter=2),
        "crweno5": lambda: with_scheme(C.vortex(40, n_iter=2), "crweno5")}


@pytest.mark.parametrize("shape", [(16, 64), (-32, 0), (-128, 0)], ids=["walker", "tile32", "tile128"])
@pytest.mark.parametrize("interp", ["components", "characteristic"])
@pytest.mark.parametrize("model", list(MAKE))
def test_shapes_select_the_fp64_forms(built_lib, oracle_lib, tmp_path, model, interp, shape):
    case = rough(MAKE[model](), 0.002)
    case.interp = interp
    s = solver_for(case, tmp_path)
    nd = len(case.size)
    u0 = s.get_state()

    def steps():
        s.set_state(u0)
        s.step(2)
        return s.get_state()

    pairs = steps()
    for d in range(nd):
        s.set_launch(d, *shape)
        assert s.get_launch(d)[0] == shape[0]
    fp64 = steps()
    assert not np.array_equal(pairs, fp64)
    for d in range(nd):
        s.set_launch(d, AUTO, 32)
        assert s.get_launch(d) == (AUTO, 32)
    assert np.array_equal(steps(), pairs)
    P = O.Problem(case)
    ref = O.interior(P.rk(P.u0(), 2), case.size, case.nvars, 3).reshape(-1)
    for got in (pairs, fp64):
        assert np.linalg.norm(got - ref) <= 1e-10 * np.linalg.norm(ref)


def test_autotuner_takes_fp64_for_a_rough_field(built_lib, tmp_path):
    """Noise of 20 %: nearly every interface leaves the pairs' bound, and the FP64 kernels are three
    times as fast; on a smooth field the pairs are."""
    case = rough(C.vortex(128, n_iter=1, dt=1e-9, interp="characteristic"), 0.2)
    assert all(seg < AUTO for seg, _ in solver_for(case, tmp_path, "rough").autotune(2))
    case = C.vortex(128, n_iter=1, interp="characteristic")
    assert all(seg >= AUTO for seg, _ in solver_for(case, tmp_path, "smooth").autotune(2))


@pytest.mark.parametrize("n", [64, 256])
def test_tuned_solver_shape_on_an_adjoint(built_lib, tmp_path, n):
    """A program that hands the tuned shape of a forward solver to the adjoint leaves its taped
    steps in tiles (segment walkers of 32 interfaces leave most SMs without a warp)."""
    case, _ = C.adjoint_problem(n, 4)
    d = str(tmp_path / "deck")
    case.write(d)
    inp = Inputs(d)
    s = Solver(inp.config, inp.dxinv)
    s.set_state(case.u)
    adj = Adjoint(inp.config, inp.dxinv, 4)
    for k, (seg, block) in enumerate(s.autotune(1)):
        adj.set_launch(k, seg, block)
        assert adj.get_launch(k)[0] in (-32, -64, -128)


@pytest.mark.parametrize("block", [0, 32, 64, 128])
@pytest.mark.parametrize("interp", ["components", "characteristic"])
def test_ensemble_of_mixed_sizes_equals_solvers(built_lib, tmp_path, interp, block):
    """Float pairs: members of mixed sizes, whose blocks have shapes of their own in one launch, and
    whose interfaces are partly evaluated in FP64 (noise), equal single solvers bit for bit."""
    members = C.ensemble_vortex(6, sizes=[16, 70, 41, 136, 25, 33], n_iter=3, seed=19, interp=interp, scheme="ssprk3")
    for k, m in enumerate(members):
        if k % 2:
            rough(m, 0.02, k)
    d = str(tmp_path / "ens")
    C.write_ensemble(members, d)
    e = Ensemble.from_dir(d)
    for dd in range(2):
        assert e.get_launch(dd) == (AUTO, 128)
        e.set_launch(dd, 0, block)
        assert e.get_launch(dd) == (AUTO, block or 128)
    e.step(3)
    for k, case in enumerate(members):
        s = solver_for(case, tmp_path, f"m{k}")
        s.step(3)
        assert np.array_equal(e.get_state(k), s.get_state()), k
