"""The 8-lanes-per-walker kernels at the numbers of walkers that they serve (on 148 SMs more than 2368 for DMC and
T-moves, 2072 for Gaussian moves, 4736 for the E_L of a mixed-precision sweep), walker by walker against the oracle
and against the kernels with a warp per walker."""
import dataclasses

import numpy as np
import pytest

from champ_b200 import system as S

pytestmark = pytest.mark.gpu


def system(k):
    return S.c2_bfd_example(10) if k == "c2bfd" else S.c2_dimer()


@pytest.mark.parametrize("k", ["dimer", "c2bfd"])
@pytest.mark.parametrize("variant", [1, 2])
def test_tmoves_follow_the_oracle(oracle_mod, k, variant):
    """Draws are keyed by the walker, so the first walkers of many move as the oracle moves them: to the
    same points, but for a draw tied at the last bit.  What the moves leave for the next proposals (inverse, pair
    table, distances, power sums) gives the ratios that a state built from the new positions gives."""
    from champ_b200.engine import Engine
    s = system(k)
    nw, nor, tau = 2500, 100, 0.1
    eng = Engine(s, nw, "fp64")
    eng.set_walkers(S.initial_walkers(s, nw, seed=23))
    eng.vmc_sweeps(20, seed=4, sweep0=0, step=s.step, stats=False)
    x = eng.get_walkers()
    eng.set_walkers(x)
    moved = eng.tmoves(seed=31, step=7, tau=tau, variant=variant)
    xg = eng.get_walkers()
    assert np.array_equal(moved > 0, np.any(xg != x, axis=(1, 2)))
    orc = oracle_mod.Oracle(s)
    same = 0
    for w in range(nor):
        xo, n = orc.tmoves(x[w], seed=31, iw=w, step=7, tau=tau, variant=variant)
        same += np.allclose(xg[w], xo, rtol=0, atol=1e-9) and n == moved[w]
    assert same >= nor - 1
    assert moved.sum() > 0
    xn = xg[:, 3] + s.step * np.random.default_rng(2).standard_normal((nw, 3))
    r0, g0 = eng.propose_1e(3, xn, grad=True)
    eng.set_walkers(xg)
    r1, g1 = eng.propose_1e(3, xn, grad=True)
    near = np.abs(r1).max()  # updated against new inverses: the updates' conditioning, 1e-9 as in the parity tests
    assert np.all(np.abs(r0 - r1) <= 1e-9 * np.maximum(np.abs(r1), 1e-3 * min(near, 1e3)))
    assert np.all(np.abs(g0 - g1) <= 1e-7 * np.abs(g1).max(axis=1, keepdims=True))
    eng.close()


def dmc(s, prec, nw, steps, **options):
    from champ_b200.engine import Engine
    eng = Engine(s, 2 * nw, prec)
    for name, v in options.items():
        eng.set_option(name, v)
    eng.set_walkers(S.initial_walkers(s, nw, seed=9))
    eng.vmc_sweeps(10, seed=9, sweep0=0, step=0.4, stats=False)
    eng.dmc_init(nw, 0.01)
    out = np.vstack([eng.dmc_steps(n, seed=31 + n) for n in steps]), eng.get_walkers()
    eng.close()
    return out


@pytest.mark.parametrize("k,prec,nw", [("dimer", "fp64", 2600), ("c2bfd", "fp64", 2600), ("dimer", "mixed", 5000)])
def test_dmc_steps_match_a_warp_per_walker(k, prec, nw):
    """FP64 steps, and the FP64 half of mixed steps, against the persistent kernel (a warp per walker): the same
    populations and walkers, weights and energies to the order of sums."""
    a, xa = dmc(system(k), prec, nw, (5,), dmc_persistent=0)
    b, xb = dmc(system(k), prec, nw, (5,), dmc_persistent=1)
    assert np.array_equal(a[:, 0], b[:, 0])
    assert np.allclose(a[:, 1:], b[:, 1:], rtol=1e-10, atol=1e-10)
    assert np.allclose(xa, xb, rtol=0, atol=1e-10)


@pytest.mark.parametrize("tmoves", [0, 2])
def test_dmc_graph_replay(tmoves):
    """Captured steps, an odd number of them and a change of seed, against steps launched one by one: the same
    kernels, so the same population and walkers; weight sums to the order of the atomic additions."""
    s = system("dimer")
    a, xa = dmc(s, "fp64", 2600, (5, 4), dmc_graph=0, tmoves=tmoves)
    b, xb = dmc(s, "fp64", 2600, (5, 4), dmc_graph=1, tmoves=tmoves)
    assert np.array_equal(a[:, 0], b[:, 0])
    assert np.allclose(a[:, 1:], b[:, 1:], rtol=1e-10, atol=1e-10)
    assert np.allclose(xa, xb, rtol=0, atol=1e-12)


def test_mixed_sweeps_of_few_among_many():
    """The FP32 move tables that the small evaluation leaves: the first walkers of many against the same walkers
    alone, three sweeps.  A table entry may round the other way, so a decision may tie: at most one walker of 60."""
    from champ_b200.engine import Engine
    s = system("dimer")
    x = S.initial_walkers(s, 60, seed=12)
    out = []
    for y in (x, np.resize(x, (4801,) + x.shape[1:])):
        eng = Engine(s, len(y), "mixed")
        eng.set_walkers(y)
        st = eng.vmc_sweeps(3, seed=19, sweep0=1, step=s.step)
        out.append((eng.get_walkers()[:60], st["accept"][:60], st["elast"][:60]))
        eng.close()
    same = np.abs(out[0][0] - out[1][0]).max(axis=(1, 2)) == 0
    assert same.sum() >= 59
    assert np.array_equal(out[0][1][same], out[1][1][same])
    assert np.allclose(out[0][2][same], out[1][2][same], rtol=1e-9, atol=1e-9)


def test_singular_walkers_leave_their_matrix():
    """Up electrons so far out that every orbital is zero there: the walker is flagged, its energy NaN, and the evaluation
    leaves the zero matrix in the inverse's place, so that the ratio of a move back is zero whatever the
    walkers beside it are; the others are as without it."""
    from champ_b200.engine import Engine
    s = system("dimer")
    nw, bad = 4801, [0, 7, 13, 16, 100, 2000, 4800]
    x = S.initial_walkers(s, nw, seed=15)
    y = x.copy()
    y[bad, :s.nup] += 1e4 * np.arange(1, s.nup + 1)[:, None]
    out = []
    for z in (x, y):
        eng = Engine(s, nw, "mixed")
        eng.set_walkers(z)
        st = eng.vmc_sweeps(1, seed=21, sweep0=0, step=s.step)  # FP32 moves, then the small kernel's E_L
        r = eng.propose_1e(0, np.broadcast_to(s.cent[0] + 0.4, (nw, 3)).copy())
        out.append((st["elast"], eng.get_walkers(), eng.walker_status(), r))
        eng.close()
    good = np.setdiff1d(np.arange(nw), bad)
    for a, b in zip(*out):
        assert np.array_equal(a[good], b[good])
    assert np.all(np.isnan(out[1][0][bad])) and np.all(out[1][2][bad] & 1) and not out[1][2][good].any()
    assert np.array_equal(out[1][3][bad], np.zeros(len(bad)))


def test_exponential_of_the_shell_tables(oracle_mod):
    """Local energies of one electron in three contracted s shells about a bare nucleus, from 1e-3 bohr to where the
    tightest primitives are not formed and on: a ratio of sums of the tables' exponentials.  A primitive's relative
    error is 2 ulp of its argument z r^2 (below 70 where it counts) and 2 of its own, 4e-14 at most; a term of the
    Laplacian is up to 6 z + 4 z^2 r^2 times the function."""
    from champ_b200.engine import Engine
    base = S.cluster128(ncent=1, box=3.5, norb=1)
    z = np.array([0.05, 0.9, 12.0, 0.08, 2.0, 0.3, 6.0, 40.0])
    one = np.zeros(3, np.int32)
    s = dataclasses.replace(
        base, nelec=1, nup=1, cent=np.zeros((1, 3)), shell_cent=one, shell_n=one + 1, shell_l=one, shell_kind=one + 1,
        shell_nprim=np.array([3, 2, 3], np.int32), prim_zeta=z, prim_coef=np.array([0.4, 0.7, 0.3, 0.8, -0.2, 0.5, 0.4, 0.6]),
        basis_shell=np.arange(3, dtype=np.int32), basis_m=one, coef=np.array([[0.6, 0.5, 0.7]]), det_orb=np.zeros((1, 1), np.int32),
        nloc=0, nordc=0, een_cusp=0, c=np.zeros((1, 0)), a4=np.zeros_like(base.a4), b=np.zeros_like(base.b))
    rng = np.random.default_rng(6)
    r = np.exp(np.linspace(np.log(1e-3), np.log(25.0), 3000))
    u = rng.standard_normal((3000, 3))
    x = (r[:, None] * u / np.linalg.norm(u, axis=1, keepdims=True))[:, None, :]
    eng = Engine(s, 3000, "fp64")
    eng.set_walkers(x)
    st = eng.vmc_sweeps(1, seed=3, sweep0=0, step=1e-6)
    y = eng.get_walkers()
    eng.close()
    orc = oracle_mod.Oracle(s)
    e = np.array([orc.eval(p)["energy"] for p in y])
    rr = np.linalg.norm(y[:, 0], axis=1)
    zmax = np.minimum(40.0, 70.0 / rr ** 2 + 0.05)  # the tightest exponent that counts
    bound = 1e-13 * (6 * zmax + 4 * zmax ** 2 * rr ** 2 + s.znuc[0] / rr)
    assert np.all(np.abs(st["elast"] - e) <= bound)
