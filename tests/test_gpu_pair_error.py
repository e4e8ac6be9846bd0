"""How far the right-hand side of the float-pair kernels is from one in extended precision:
no further than FP64 arithmetic leaves it.

Unit: 2^-53 of an interface's flux scale (rho lam, rho lam^2, rho lam H with lam = |u| + a)
over the spacing.  A cell's flux takes some six roundings, each of 0.29 units rms of the
quantity it rounds, and of these quantities the mass flux is exact, the momentum flux and its
pressure about half the scale, the energy flux about a third; the differences of the scheme
weigh neighbouring fluxes by sqrt(2 (2/3)^2 + 2/12^2) = 0.95.  That gives 0.3 to 0.4 units
rms over the components for FP64 arithmetic; 0.45 is held."""
import numpy as np
import pytest

from hypar_gb300 import cases as C
from hypar_gb300.solver import Solver

torch = pytest.importorskip("torch")
LD = np.longdouble
GAMMA, EPS = LD(1.4), LD(1e-6)


def weno5(m):
    m0, m1, m2, m3, m4 = m
    t = LD(13) / 12
    b = [t * (m0 - 2 * m1 + m2) ** 2 + (m0 - 4 * m1 + 3 * m2) ** 2 / 4,
         t * (m1 - 2 * m2 + m3) ** 2 + (m1 - m3) ** 2 / 4, t * (m2 - 2 * m3 + m4) ** 2 + (3 * m2 - 4 * m3 + m4) ** 2 / 4]
    a = [LD(c) / 10 / (EPS + bk) ** 2 for c, bk in zip((1, 6, 3), b)]
    f = [(2 * m0 - 7 * m1 + 11 * m2) / 6, (-m1 + 5 * m2 + 2 * m3) / 6, (2 * m2 + 5 * m3 - m4) / 6]
    return sum(ak * fk for ak, fk in zip(a, f)) / sum(a)


def primitive(u):
    v = u[:, 1] / u[:, 0]
    return u[:, 0], v, (GAMMA - 1) * (u[:, 2] - u[:, 0] * v * v / 2)


def eigen(uL, uR):
    """Roe average of the cells: eigenvalues, left and right eigenvectors (u - c, u, u + c) in
    HyPar's scaling (euler1d.h: the acoustic fields are velocities), which the weights see."""
    (rl, vl, pl), (rr, vr, pr) = primitive(uL), primitive(uR)
    a, b = np.sqrt(rl), np.sqrt(rr)
    v = (a * vl + b * vr) / (a + b)
    H = (a * (uL[:, 2] + pl) / rl + b * (uR[:, 2] + pr) / rr) / (a + b)
    c = np.sqrt((GAMMA - 1) * (H - v * v / 2))
    one, g = np.ones_like(v), (GAMMA - 1) / (c * c)
    R = np.array([[one, one, one], [v - c, v, v + c], [H - v * c, v * v / 2, H + v * c]])
    L = np.array([[(g * v * v / 2 + v / c) / 2, -(g * v + 1 / c) / 2, g / 2], [1 - g * v * v / 2, g * v, -g],
                  [(g * v * v / 2 - v / c) / 2, -(g * v - 1 / c) / 2, g / 2]])
    k = 2 * c / (a * b)
    L[0], L[2], R[:, 0], R[:, 2] = L[0] * k, L[2] * k, R[:, 0] / k, R[:, 2] / k
    return np.array([v - c, v, v + c]), L, R


def exact_rhs(u64, dxinv, characteristic):
    """-dF/dx of periodic data in extended precision: WENO5 (Jiang-Shu) + Roe."""
    u = u64.astype(LD)
    rho, v, p = primitive(u)
    f = np.stack([u[:, 1], u[:, 1] * v + p, (u[:, 2] + p) * v], 1)
    lam, L, R = eigen(u, np.roll(u, -1, 0))  # interface i + 1/2
    mul = lambda A, x: np.einsum("ijn,nj->ni", A, x)  # noqa: E731
    win = lambda q, k: np.roll(q, -k, 0)  # noqa: E731
    proj = (lambda q: mul(L, q)) if characteristic else (lambda q: q)
    back = (lambda q: mul(R, q)) if characteristic else (lambda q: q)
    side = lambda q, ks: back(weno5([proj(win(q, k)) for k in ks]))  # noqa: E731
    left, right = (-2, -1, 0, 1, 2), (3, 2, 1, 0, -1)
    d = mul(R, np.abs(lam).T * mul(L, side(u, right) - side(u, left)))
    F = (side(f, left) + side(f, right) - d) / 2
    return -(F - np.roll(F, 1, 0)) * dxinv.astype(LD)[:, None]


def wave(cells, noise, n=1200, seed=3):
    r = np.random.default_rng(seed)
    ph = np.arange(n) * 2 * np.pi / cells
    rho, v, p = 1 + 0.1 * np.sin(ph), 0.3 + 0.1 * np.sin(ph), 1 + 0.1 * np.cos(ph + 0.3)
    if noise:
        rho, v, p = rho * (1 + noise * r.uniform(-1, 1, n)), v + noise * r.uniform(-1, 1, n), p * (1 + noise * r.uniform(-1, 1, n))
    return np.stack([rho, rho * v, p / 0.4 + 0.5 * rho * v * v], 1)


def case_of(u, interp):
    c = C.sod(16, n_iter=1)
    c.size, c.bc, c.interp, c.upwinding, c.u = [len(u)], "periodic", interp, "roe", u
    c.x = [np.arange(len(u)) / len(u)]
    return c


CASES = [(6, 0.0), (8, 0.0), (12, 0.0), (30, 0.0), (100, 0.0), (60, 0.003), (60, 0.01), (60, 0.02), (60, 0.06)]


@pytest.mark.parametrize("interp", ["components", "characteristic"])
@pytest.mark.parametrize("cells,noise", [(8, 0.0), (60, 0.02)])
def test_extended_precision_restates_the_oracle(oracle_lib, interp, cells, noise):
    """The extended-precision restatement against the oracle's 64 bits (its own rounding, some
    ten units)."""
    import oracle as O
    case = case_of(wave(cells, noise), interp)
    P = O.Problem(case)
    ref = O.interior(P.rhs(P.u0()), case.size, 3, 3).reshape(-1, 3)
    got = exact_rhs(case.u, P.dxinv[3:-3], interp == "characteristic")
    assert np.abs(got - ref).max() <= 1e-11 * np.abs(ref).max()


@pytest.mark.gpu
@pytest.mark.parametrize("interp", ["components", "characteristic"])
@pytest.mark.parametrize("cells,noise", CASES)
def test_rounding_of_a_right_hand_side(built_lib, tmp_path, interp, cells, noise):
    u0 = wave(cells, noise)
    case = case_of(u0, interp)
    d = str(tmp_path / "deck")
    case.write(d)
    s = Solver.from_dir(d)
    u = torch.zeros(len(u0) + 6, 3, dtype=torch.float64, device="cuda")
    u[3:-3] = torch.from_numpy(u0)
    out = torch.zeros_like(u)
    s.rhs(out, u)
    dxinv = s.dxinv[3:-3]
    err = np.abs(out[3:-3].cpu().numpy() - exact_rhs(u0, dxinv, interp == "characteristic"))
    rho, v, p = (q.astype(np.float64) for q in primitive(u0.astype(LD)))
    lam = np.abs(v) + np.sqrt(1.4 * p / rho)
    unit = np.stack([rho * lam, rho * lam * lam, lam * (u0[:, 2] + p)], 1) * dxinv[:, None] * 2.0 ** -53
    rms = float(np.sqrt(((err / unit) ** 2).mean()))
    assert rms <= 0.45, rms
