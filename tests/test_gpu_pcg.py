"""Pressure solve by preconditioned conjugate gradients (Solver = 2).

The solution of div(C grad P) = RHS does not depend on the solver, so the
bars are: the PCG solution satisfies the discrete equation to its two-norm
tolerance, agrees with the converged Richardson solution (Solver = 0) and with
steps taken with it, gets further than Richardson for the same number of FFT
solves at a large density ratio, and is bit-identical between eager and
graph-replayed steps.
"""
import numpy as np
import pytest

from conftest import rel_err
from tpm import inputs, params as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    from tpm import build, capi

    build.build()
    return capi


def variable_density_problem(N=32, ratio=20.0, seed=1):
    p = P.physical(N, 1, nu=0.02, A=0.0, tau_p=0.1, mass_loading=0.1)
    z, y, x = np.meshgrid(*(np.arange(N) * (p.Lx / N),) * 3, indexing="ij")
    a = (ratio - 1) / (ratio + 1)
    Rho = 1.0 + a * np.sin(x) * np.sin(y) * np.cos(z)
    C3 = np.stack([1.0 / ((Rho + np.roll(Rho, 1, axis=ax)) * 0.5) for ax in (2, 1, 0)])
    rng = np.random.default_rng(seed)
    RHS = rng.standard_normal((N, N, N))
    RHS -= RHS.mean()
    return p, C3, RHS


def div_c_grad(p, C3, Pf):
    h = (p.Lx / p.Nx, p.Ly / p.Ny, p.Lz / p.Nz)
    out = np.zeros_like(Pf)
    for d, ax in enumerate((2, 1, 0)):
        hi = np.roll(C3[d], -1, axis=ax) * (np.roll(Pf, -1, axis=ax) - Pf)
        lo = C3[d] * (Pf - np.roll(Pf, 1, axis=ax))
        out += (hi - lo) / h[d] ** 2
    return out


@pytest.mark.parametrize("prec,tol", [(P.PREC_FP64, 1e-11), (P.PREC_MIXED, 1e-8)])
def test_pcg_solves_variable_coefficient_problem(capi, prec, tol):
    p, C3, RHS = variable_density_problem()
    P0 = np.zeros_like(RHS)
    pcg = capi.Context(p.replace(Solver=2, precision=prec), 1)
    x_pcg, it_pcg, err_pcg = pcg.poisson_solve(C3, P0, RHS, 500, tol)
    rel = np.linalg.norm(div_c_grad(p, C3, x_pcg) - RHS) / np.linalg.norm(RHS)
    assert rel <= 3 * tol, rel  # the recursive residual tracks the true one
    assert err_pcg <= tol and it_pcg < 500
    rich = capi.Context(p.replace(Solver=0), 1)
    x_r, it_r, _ = rich.poisson_solve(C3, P0, RHS, 1000, 1e-14)
    rel_r = np.linalg.norm(div_c_grad(p, C3, x_r) - RHS) / np.linalg.norm(RHS)
    if rel_r <= 1e-9:  # Richardson converged: same solution up to a constant
        d = (x_pcg - x_pcg.mean()) - (x_r - x_r.mean())
        assert np.abs(d).max() <= 1e3 * max(rel, rel_r) * np.abs(x_r - x_r.mean()).max()
    # for the same number of preconditioner applications (one FFT solve each),
    # conjugate gradients get further than Richardson at this density ratio
    x_k, it_k, _ = rich.poisson_solve(C3, P0, RHS, it_pcg, 0.0)
    rel_k = np.linalg.norm(div_c_grad(p, C3, x_k) - RHS) / np.linalg.norm(RHS)
    assert it_k == it_pcg and rel < rel_k, (it_pcg, rel, rel_k)


def case(solver, prec=P.PREC_FP64, N=32, seed=3):
    p = P.physical(N, 5000, nu=0.02, A=0.1, tau_p=0.1, mass_loading=0.5, heating_Q=0.5,
                   iterations=60, epsilon=1e-13, precision=prec)
    s = inputs.make_state(p, 5000, seed=seed)
    z, y, x = np.meshgrid(*((np.arange(N) + 0.5) * (p.Lx / N),) * 3, indexing="ij")
    s.Rho = 1.0 + 0.6 * np.sin(x) * np.cos(y) * np.sin(z)  # density ratio 4
    s.RU = s.RU * ((s.Rho + np.roll(s.Rho, 1, axis=2)) * 0.5)[None]
    return p.replace(dt=inputs.cfl_dt(p, s.RU), Solver=solver), s


def run(capi, p, s, nsteps, graph=False):
    ctx = capi.Context(p, s.npart)
    ctx.load(s)
    ctx.initialize()
    if graph:
        ctx.set_graph(True)
    ctx.run(nsteps)
    ctx.sync()
    return ctx


def test_pcg_steps_match_richardson_steps(capi):
    p0, s = case(0)
    p2, _ = case(2)
    a, b = run(capi, p0, s, 3), run(capi, p2, s, 3)
    for f in ("RU", "RHO", "C", "Q"):
        assert rel_err(b.download_field(f), a.download_field(f)) <= 1e-9, f
    # P is defined up to a constant: the Richardson update dp = M^-1(cc r) keeps
    # the mean of cc*r, conjugate gradients do not move the mean
    Pa, Pb = a.download_field("P"), b.download_field("P")
    assert rel_err(Pb - Pb.mean(), Pa - Pa.mean()) <= 1e-9
    pa, pb = a.download_particles(), b.download_particles()
    for q in inputs.PQ:
        assert rel_err(pb[q], pa[q]) <= 1e-9, q


def test_pcg_graph_bit_identical_and_mixed_close(capi):
    p2, s = case(2, seed=4)
    eager = run(capi, p2, s, 3)
    graph = run(capi, p2, s, 3, graph=True)
    for f in ("RU", "RHO", "P", "C", "Q"):
        assert np.array_equal(graph.download_field(f), eager.download_field(f)), f
    assert graph.scalars()["total_poisson_iterations"] == eager.scalars()["total_poisson_iterations"]
    mixed = run(capi, p2.replace(precision=P.PREC_MIXED), s, 3)
    for f in ("RU", "RHO", "P"):
        assert rel_err(mixed.download_field(f), eager.download_field(f)) <= 1e-5, f


def test_heated_pcg_box_does_not_depend_on_batch_or_tiles(capi):
    """A heated FP64 box solved by conjugate gradients gives the same bits alone,
    in a batch and with other transform tiles: r.z is summed by groups of rows
    that only the grid decides."""
    from test_gpu_graph import assert_same, state

    p, s = case(2)
    want = state(run(capi, p, s, 2))
    b = capi.Batch([p, p], [s.npart, s.npart])
    for box in b.boxes:
        box.load(s)
        box.initialize()
    b.run(2)
    b.sync()
    got = [state(box) for box in b.boxes]
    b.close()
    for tiles in ([1, 2, 4, 64, 96, 160], [8, 4, 8, 128, 64, 128]):
        ctx = capi.Context(p, s.npart)
        ctx.load(s)
        ctx.set_fft_tiles(tiles)
        ctx.initialize()
        ctx.run(2)
        got.append(state(ctx))
    for g in got:
        assert_same(g, want)


@pytest.mark.parametrize("heat,prec", [(0.0, P.PREC_FP64), (0.5, P.PREC_MIXED)])
def test_pcg_box_does_not_depend_on_tiles(capi, heat, prec):
    """The same of the FP64 and the mixed passes: tiles that an autotuner might pick
    leave every bit of a conjugate-gradient solve alone."""
    from test_gpu_graph import assert_same, state

    p, s = case(2, prec)
    p = p.replace(I01=heat * p.I01, I02=heat * p.I02)
    want = state(run(capi, p, s, 2))
    for tiles in ([1, 2, 4, 64, 96, 160], [8, 4, 8, 128, 64, 128]):
        ctx = capi.Context(p, s.npart)
        ctx.load(s)
        ctx.set_fft_tiles(tiles)
        ctx.initialize()
        ctx.run(2)
        assert_same(state(ctx), want)
