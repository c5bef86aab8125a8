"""Diagnostics on the device (tpm_statistics, tpm_spectrum, tpm_rdf) against
the oracle and the reference's own stat files.

Bars: grid::Statistics scalars and the extensions within 1e-12 relative of
the oracle (extrema exact); the reference's stat files to their 6 printed
digits; spectrum shells within 1e-12 of the total energy; RDF pair counts
identical to the O(Np^2) count.
"""
import numpy as np
import pytest

from conftest import rel_err
from golden import STATS_NAMES, load
from tpm import inputs, params as P

pytestmark = pytest.mark.gpu

TOL = 1e-12
TOL_PRINTED = 6e-6
EXACT = ("Rho_max", "Rho_min", "C_max", "C_min", "u_max", "Gas_CFL_Max", "Vp_max", "Tp_max",
         "P0", "T_cur", "num_timestep", "Gas_Max_Diff_CFL")


@pytest.fixture(scope="module")
def capi():
    from tpm import build, capi

    build.build()
    return capi


def case(N=32, npart=10_000, seed=7, heat=0.5, **kw):
    p = P.physical(N, npart, nu=0.02, A=0.1, tau_p=0.1, mass_loading=0.5, heating_Q=heat,
                   iterations=20, epsilon=1e-13, **kw)
    s = inputs.make_state(p, npart, seed=seed)
    return p.replace(dt=inputs.cfl_dt(p, s.RU)), s


def compare_stats(g, o, tol=TOL):
    for k, want in o.items():
        got = g[k]
        if k == "num_iteration":
            # with epsilon = 1e-13 at the roundoff floor of max|dp| the stopping
            # iteration depends on FFT rounding; the fields agree either way
            assert (got == 0) == (want == 0) and got <= 20
        elif k in EXACT:
            assert got == want, (k, got, want)
        else:
            assert abs(got - want) <= tol * max(abs(want), 1e-300), (k, got, want)


@pytest.mark.parametrize("nsteps", [0, 2])
def test_statistics_match_oracle(capi, oracle_lib, nsteps):
    p, s = case()
    ctx = capi.Context(p, s.npart)
    ctx.load(s)
    ctx.initialize()
    o = oracle_lib.Oracle(p, s.npart)
    o.load(s)
    o.initialize()
    for _ in range(nsteps):
        ctx.step()
        o.step()
    g = ctx.statistics()
    compare_stats(g, o.statistics())
    assert ctx.statistics() == g  # bit-reproducible


@pytest.mark.parametrize("name", STATS_NAMES)
def test_statistics_match_reference_stat_files(capi, name):
    p, s, ref, nsteps, _ = load(name)
    ctx = capi.Context(p, s.npart)
    ctx.load(s)
    ctx.initialize()
    for st in range(nsteps):
        ctx.step()
        got = ctx.statistics()
        for key, vals in ref["stats"].items():
            r = float(vals[st])
            assert abs(got[key] - r) <= TOL_PRINTED * abs(r) + 1e-300, (st, key, got[key], r)


def test_statistics_need_a_step_boundary(capi):
    p, s = case(N=16, npart=100)
    ctx = capi.Context(p, s.npart)
    ctx.load(s)
    ctx.initialize()
    ctx.substep(0)
    with pytest.raises(capi.TpmError):
        ctx.statistics()


def test_mixed_statistics_close_to_fp64(capi):
    p, s = case(N=32, npart=10_000, seed=8)
    out = []
    for prec in (P.PREC_FP64, P.PREC_MIXED):
        ctx = capi.Context(p.replace(precision=prec), s.npart)
        ctx.load(s)
        ctx.initialize()
        ctx.run(3)
        out.append(ctx.statistics())
    for k in ("TKE", "TKE2", "dissipation", "C_var", "Tg_mean", "Tp_mean", "u_rms"):
        assert abs(out[1][k] - out[0][k]) <= 1e-5 * abs(out[0][k]), k


@pytest.mark.parametrize("dims", [(32, 32, 32), (24, 30, 16)])
def test_spectrum_matches_numpy(capi, oracle_lib, dims):
    nx, ny, nz = dims
    p, s = case(N=nx, npart=2000, seed=9)
    if (ny, nz) != (nx, nx):
        p = p.replace(Ny=ny, Nz=nz, Ly=p.Lx * ny / nx, Lz=p.Lx * nz / nx)
        s = inputs.make_state(p, 2000, seed=9)
        p = p.replace(dt=inputs.cfl_dt(p, s.RU))
    ctx = capi.Context(p, s.npart)
    ctx.load(s)
    ctx.initialize()
    ctx.run(2)
    E, dk = ctx.spectrum()
    want, dk_w = oracle_lib.spectrum(p, ctx.download_field("RU"), ctx.download_field("RHO"))
    assert dk == dk_w and E.shape == want.shape
    assert np.abs(E - want).max() <= TOL * want.sum()
    U = oracle_lib.face_velocity(ctx.download_field("RU"), ctx.download_field("RHO"))
    assert abs(E.sum() - 0.5 * np.mean(U ** 2) * 3) <= TOL * E.sum()


def test_spectrum_large_box_parseval(capi):
    p, s = case(N=128, npart=100_000, seed=10, heat=0.1)
    ctx = capi.Context(p, s.npart)
    ctx.load(s)
    ctx.initialize()
    ctx.step()
    E, _ = ctx.spectrum()
    st = ctx.statistics()
    assert abs(E.sum() - 1.5 * st["u_rms"] ** 2) <= 1e-12 * E.sum()
    # the initial spectrum peaks near k = 4 and is negligible in the top shells
    assert 2 <= int(np.argmax(E)) <= 6
    assert E[-5:].sum() <= 1e-6 * E.sum()


@pytest.mark.parametrize("clustered", [False, True])
def test_rdf_pairs_match_brute_force(capi, oracle_lib, clustered):
    p, s = case(N=32, npart=20_000, seed=11)
    if clustered:  # most particles in a few cells, some on the boundary planes
        rng = np.random.default_rng(11)
        for q, L in zip(("x", "y", "z"), (p.Lx, p.Ly, p.Lz)):
            s.part[q] = np.where(rng.random(s.npart) < 0.7, 0.3 + 0.05 * rng.random(s.npart),
                                 s.part[q])
        s.part["x"][:50] = 0.0
        s.part["y"][50:100] = p.Ly
    ctx = capi.Context(p, s.npart)
    ctx.load(s)
    ctx.initialize()
    for r_max, nb in ((0.5, 50), (p.Lx / 3, 64)):
        pairs, g = ctx.rdf(r_max, nb)
        base = ctx.download_particles("base")
        want = oracle_lib.rdf_pairs(base["x"], base["y"], base["z"], (p.Lx, p.Ly, p.Lz), r_max, nb)
        assert np.array_equal(pairs, want)
        assert np.array_equal(ctx.rdf(r_max, nb)[0], pairs)
    if not clustered:  # uniform random positions: g ~ 1 away from r = 0
        assert abs(g[nb // 2:].mean() - 1.0) < 0.02


@pytest.mark.parametrize("share", [3, 4])
def test_rdf_pairs_at_bin_edges(capi, oracle_lib, share):
    """Separations on and within rounding of bin edges (a lattice of the bin
    width, along the axes and across the boundary), where single precision
    cannot tell the bin."""
    p, s = case(N=24, npart=4000, seed=12)
    rng = np.random.default_rng(12)
    nb, r_max = 32, p.Lx / share
    w = r_max / nb
    for q in ("x", "y", "z"):
        v = w * rng.integers(0, share * nb, s.npart)
        v[::3] = np.nextafter(v[::3], p.Lx)
        v[1::5] = p.Lx * rng.random(v[1::5].size)
        s.part[q] = np.minimum(v, p.Lx)
    ctx = capi.Context(p, s.npart)
    ctx.load(s)
    ctx.initialize()
    base = ctx.download_particles("base")
    pairs, _ = ctx.rdf(r_max, nb)
    want = oracle_lib.rdf_pairs(base["x"], base["y"], base["z"], (p.Lx, p.Ly, p.Lz), r_max, nb)
    assert np.array_equal(pairs, want)


@pytest.mark.parametrize("units", [2.0 / 3.0, 0.4, 1.0])
def test_rdf_pairs_of_bins_finer_than_the_integer_positions(capi, oracle_lib, units):
    """Bins of about 2^-32 of the box, finer than single precision and integer
    positions tell apart: every pair is binned in FP64, those half a bin from the
    edges too."""
    p, s = case(N=24, npart=4000, seed=13)
    p = p.replace(Lx=1.0, Ly=1.0, Lz=1.0)
    rng = np.random.default_rng(13)
    for q in ("x", "y", "z"):
        s.part[q] = np.repeat(0.1 + 0.8 * rng.random(s.npart // 20), 20)
    s.part["x"] += 8 * 2.0 ** -32 * rng.random(s.npart)
    nb = 12
    r_max = nb * units * 2.0 ** -32
    ctx = capi.Context(p, s.npart)
    ctx.load(s)
    ctx.initialize()
    base = ctx.download_particles("base")
    pairs, _ = ctx.rdf(r_max, nb)
    want = oracle_lib.rdf_pairs(base["x"], base["y"], base["z"], (1.0, 1.0, 1.0), r_max, nb)
    assert want.sum() > 1000
    assert np.array_equal(pairs, want)


@pytest.mark.parametrize("L", [3e-20, 1.0, 1e20])
def test_rdf_pairs_in_any_unit_of_length(capi, oracle_lib, L):
    """The single-precision form of the pairs counts in bins: a box whose squared
    lengths leave the range of single precision gets the same counts."""
    p, s = case(N=24, npart=3000, seed=14)
    rng = np.random.default_rng(14)
    for q in ("x", "y", "z"):
        s.part[q] = L * rng.random(s.npart)
    p = p.replace(Lx=L, Ly=L, Lz=L)
    ctx = capi.Context(p, s.npart)
    ctx.load(s)
    ctx.initialize()
    base = ctx.download_particles("base")
    pairs, _ = ctx.rdf(L / 3, 32)
    want = oracle_lib.rdf_pairs(base["x"], base["y"], base["z"], (L, L, L), L / 3, 32)
    assert np.array_equal(pairs, want)


def test_rdf_rejects_r_max_beyond_a_third_of_the_box(capi):
    p, s = case(N=16, npart=100)
    ctx = capi.Context(p, s.npart)
    ctx.load(s)
    ctx.initialize()
    with pytest.raises(capi.TpmError):
        ctx.rdf(p.Lx / 2, 10)
