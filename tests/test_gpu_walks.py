"""Walks whose every step depends on the last bits of the one before.

Where psi nearly vanishes the inverse Slater matrix magnifies a rounding of the orbital rows by the matrix's
condition number, and the accelerated mover, whose proposals follow the drift, magnifies it again with every
sweep: two orders of the same sums walk apart within a few sweeps of a large molecule.  The tiled evaluation
therefore forms the rows and inverses that the moves start from to the bits of the warp-per-electron
kernels.  These tests hold it to that: against ratios and walks recorded from those kernels, and against
the oracle as far as the walk itself allows.  (The recordings are the walks of commit 305d744 on a B200.)"""
import dataclasses
import os

import numpy as np
import pytest

from champ_b200 import system as S

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "accelerated_walks.npz")


def cluster(n, nup, ncent, nordc):
    s = S.cluster128(ncent=ncent, box=14.0 * (max(ncent, 4) / 32) ** (1 / 3), norb=max(nup, n - nup))
    j = S._jastrow(np.random.default_rng(3), 1, 5, 5, nordc)
    return dataclasses.replace(s, nelec=n, nup=nup, nordc=nordc, een_cusp=j["een_cusp"], c=j["c"],
                               det_orb=np.array([list(range(nup)) + list(range(n - nup))], np.int32))


# electrons, up electrons, centres, e-e-n order: 3 to 64 orbitals of a spin, in and across the classes of
# interleaved sums (up to 16) and of tiles of 32 electrons
SHAPES = [(12, 9, 6, 0), (13, 8, 3, 4), (13, 9, 3, 4), (17, 9, 3, 4), (26, 16, 5, 5), (34, 17, 9, 4), (65, 33, 17, 4),
          (80, 40, 20, 4), (128, 64, 32, 4)]


def near_node(shape, idx=None):
    """Of 400 unequilibrated walkers those of idx, or the 8 with the largest drifts, whose psi nearly vanishes."""
    from champ_b200.engine import Engine
    s = cluster(*shape)
    x = S.initial_walkers(s, 400, seed=shape[0] + shape[1])
    if idx is None:
        eng = Engine(s, 400, "fp64")
        eng.set_walkers(x)
        idx = np.argsort(-np.abs(eng.eval_full()["velocity"]).max(axis=(1, 2)))[:8]
        eng.close()
    eng = Engine(s, len(idx), "fp64")
    assert eng.get_option("staged_eval")
    eng.set_walkers(x[idx])
    return s, idx, x[idx], eng


def ratios(shape, idx=None):
    """Ratios and gradients of three electrons' moves from walkers near a node."""
    s, idx, x, eng = near_node(shape, idx)
    n, nup = shape[:2]
    dx = s.step * np.random.default_rng(n).standard_normal((n, 400, 3))
    out = [eng.propose_1e(e, np.ascontiguousarray(x[:, e] + dx[e, idx]), grad=True) for e in (0, nup - 1, n - 1)]
    eng.close()
    return idx, np.array([r for r, _ in out]), np.array([g for _, g in out])


@pytest.mark.parametrize("shape", SHAPES)
def test_ratios_as_recorded(shape):
    """The rows and inverses are those recorded, so a ratio differs by the rounding of its N + C Jastrow terms
    (2e-14 for the largest molecule), a gradient not even by that."""
    ref = np.load(GOLDEN)
    key = "ratio_%d_%d_" % shape[:2]
    _, r, g = ratios(shape, ref[key + "idx"])
    assert np.all(np.abs(r - ref[key + "r"]) <= 1e-13 * np.abs(ref[key + "r"]))
    assert np.all(np.abs(g - ref[key + "g"]) <= 1e-13 * np.abs(ref[key + "g"]).max(axis=2, keepdims=True))


@pytest.mark.parametrize("shape", SHAPES)
def test_energies_as_recorded(shape):
    """E_L near a node, where lap psi / psi and |grad psi / psi|^2 grow as 1 / d and cancel: it keeps the last bits of
    their sums, and those are the recorded ones.  What may differ is the rounding of N^2 Jastrow terms of order 1
    and of the pseudopotential's sum (1e-13 of its largest points)."""
    ref = np.load(GOLDEN)
    key = "energy_%d_%d" % shape[:2]
    eng = near_node(shape, ref["ratio_%d_%d_idx" % shape[:2]])[3]
    r = eng.eval_full()
    eng.close()
    print(np.abs(r["energy"] - ref[key]).max(), np.abs(ref[key]).max(), np.abs(r["pe_nonloc"]).max(), np.square(r["velocity"]).sum(axis=(1, 2)).max())
    assert np.all(np.abs(r["energy"] - ref[key]) <= 1e-16 * shape[0] ** 2 + 1e-13 * (np.abs(ref[key]) + 10 * np.abs(r["pe_nonloc"])))


RECORDED = [(9, 5, 2, 4, "fp64"), (13, 9, 3, 4, "fp64"), (20, 10, 5, 5, "fp64"), (34, 17, 9, 4, "fp64"), (51, 26, 13, 5, "fp64"),
            (128, 64, 32, 4, "fp64"), (34, 17, 9, 4, "mixed"), (128, 64, 32, 4, "mixed")]


def accelerated_walk(case):
    from champ_b200.engine import Engine
    s = cluster(*case[:4])
    eng = Engine(s, 3, case[4])
    eng.set_walkers(S.initial_walkers(s, 3, seed=case[0]))
    eng.set_mover(6)
    st = eng.vmc_sweeps(4, seed=31, sweep0=2, step=s.step)
    x = eng.get_walkers()
    eng.close()
    return x, st["accept"]


@pytest.mark.parametrize("case", RECORDED)
def test_accelerated_walk_as_recorded(case):
    """Four accelerated sweeps against the positions recorded from the evaluation by a warp per walker and
    electron.  Rounding alone takes the largest molecule's electrons 1e-2 bohr apart in as many sweeps."""
    x, accept = accelerated_walk(case)
    ref = np.load(GOLDEN)
    key = "%d_%d_%s" % (case[0], case[3], case[4])
    assert np.abs(x - ref[key]).max() <= 1e-12
    assert np.array_equal(accept, ref[key + "_accept"])


@pytest.mark.parametrize("n,nup,ncent,nordc", [(24, 13, 6, 5), (40, 20, 10, 4)])
def test_accelerated_sweep_follows_the_oracle(oracle_mod, n, nup, ncent, nordc):
    """One accelerated sweep of equilibrated walkers in HBM, electron by electron, against the oracle.  How far
    the two may come apart is the walk's own: the oracle's sweeps from positions moved by 1e-13 bohr (rounding
    of a 10-bohr coordinate is 1e-15, of the drift 1e-15 of it) show its magnification, electron by electron."""
    from champ_b200.engine import Engine
    s = cluster(n, nup, ncent, nordc)
    nw = 4
    eng = Engine(s, nw, "fp64")
    eng.set_walkers(S.initial_walkers(s, nw, seed=n))
    eng.vmc_sweeps(20, seed=3, sweep0=0, step=s.step, stats=False)
    x = eng.get_walkers()
    eng.set_walkers(x)
    eng.set_mover(6, deltar=5.0, deltat=1.0, fbias=1.0)
    st = eng.vmc_sweeps(1, seed=777, sweep0=0, step=0.5)
    xg = eng.get_walkers()
    eng.close()
    orc = oracle_mod.Oracle(s)
    run = lambda y: orc.vmc_accel(y, 1, seed=777, sweep0=0, deltar=5.0, deltat=1.0, fbias=1.0, nthreads=4)  # noqa: E731
    ref = run(x)
    rng = np.random.default_rng(n)
    grown = np.zeros((nw, n))
    for _ in range(3):
        grown = np.maximum(grown, np.abs(run(x + 1e-13 * rng.choice([-1.0, 1.0], x.shape))["x"] - ref["x"]).max(axis=2))
    # an electron's magnification, with those moved before it
    bound = 10 * np.maximum.accumulate(grown, axis=1) + 1e-12
    d = np.abs(xg - ref["x"]).max(axis=2)
    print(f"{n} electrons: first {d[:, 0].max():.1e}, all {d.max():.1e} bohr; allowed {bound[:, 0].max():.1e} {bound.max():.1e}")
    assert np.all(d <= bound)
    assert np.array_equal(st["accept"], ref["accept"])


@pytest.mark.parametrize("case", ["dimer", "dimer, order 5", "dimer, no e-e-n", "mixed", "be", "c2bfd"])
def test_accelerated_walk_of_few_among_many(case):
    """A small walker's evaluation and accelerated walk do not depend on how many walk beside it, although other kernels
    serve many: to the bit for Gaussian shells (over 15 sweeps, the inverses formed anew at sweep 13 only), and for
    the Slater and numerical ones to what their walks make of rounding (1e-9 bohr after 15 sweeps)."""
    from champ_b200.engine import Engine
    s = {"c2bfd": lambda: S.c2_bfd_example(10), "be": S.be_atom}.get(case, S.c2_dimer)()
    nord = {"dimer, order 5": 5, "dimer, no e-e-n": 0}.get(case, s.nordc)
    if nord != s.nordc:
        j = S._jastrow(np.random.default_rng(3), 1, 5, 5, nord)
        s = dataclasses.replace(s, nordc=nord, een_cusp=j["een_cusp"], c=j["c"])
    x = S.initial_walkers(s, 40, seed=11)
    out = []
    for y in (x, np.resize(x, (5003,) + x.shape[1:])):
        eng = Engine(s, len(y), "mixed" if case == "mixed" else "fp64")
        eng.set_walkers(y)
        r = eng.eval_full()
        eng.set_mover(6)
        st = eng.vmc_sweeps(15, seed=19, sweep0=1, step=s.step)
        out.append((r["energy"][:40], r["velocity"][:40], eng.get_walkers()[:40], st["accept"][:40], st["elast"][:40]))
        eng.close()
    (e0, v0, x0, a0, l0), (e1, v1, x1, a1, l1) = out
    assert np.array_equal(e0, e1) and np.array_equal(v0, v1) and np.array_equal(a0, a1)
    if case in ("be", "c2bfd"):
        assert np.abs(x0 - x1).max() <= 1e-9
        assert np.allclose(l0, l1, rtol=1e-7, atol=1e-7)
    else:
        assert np.array_equal(x0, x1)
        assert np.allclose(l0, l1, rtol=1e-10, atol=1e-10)  # E_L in another order of sums


@pytest.mark.parametrize("shape", [(1, 1, 1, 0), (2, 1, 1, 0), (3, 2, 2, 4), (4, 4, 1, 4), (5, 3, 2, 5), (7, 4, 3, 4), (3, 2, 12, 4), (2, 1, 20, 5)])
def test_accelerated_sweeps_at_the_edges_of_the_small_kernel(oracle_mod, shape):
    """One electron to a spin, one spin, 1 to 4 orbitals (32 to 8 interleaved sums), more centres than lanes: the
    first of many against the same walkers alone, to the bit, and one sweep against the oracle."""
    from champ_b200.engine import Engine
    s = cluster(*shape)
    x = S.initial_walkers(s, 24, seed=sum(shape))
    out = []
    for y in (x, np.resize(x, (1200,) + x.shape[1:])):
        eng = Engine(s, len(y), "fp64")
        eng.set_walkers(y)
        eng.set_mover(6, deltar=5.0, deltat=1.0, fbias=1.0)
        walk = []
        for k in range(6):
            st = eng.vmc_sweeps(1, seed=5, sweep0=k, step=s.step)
            walk.append((eng.get_walkers()[:24], st["accept"][:24], st["elast"][:24]))
        out.append(walk)
        eng.close()
    for (xa, aa, ea), (xb, ab, eb) in zip(*out):
        assert np.array_equal(xa, xb) and np.array_equal(aa, ab)
        assert np.allclose(ea, eb, rtol=1e-9, atol=1e-9)
    ref = oracle_mod.Oracle(s).vmc_accel(x, 1, seed=5, sweep0=0, deltar=5.0, deltat=1.0, fbias=1.0)
    same = np.abs(out[1][0][0] - ref["x"]).max(axis=(1, 2)) <= 1e-9
    assert same.sum() >= 23  # a draw may tie at the last bit
    assert np.array_equal(out[1][0][1][same], ref["accept"][same])
