"""The staged evaluation's tensor-core parts at the edges of their tiles, against the CPU oracle:
electrons around multiples of 8 and 32, one centre to more than a tile of them, both e-e-n orders, spins
of unequal size.  Every sum is FP64 in both, so the tolerance is the parity tests' 1e-9 relative."""
import dataclasses

import numpy as np
import pytest

from champ_b200 import system as S

pytestmark = pytest.mark.gpu

CASES = [  # electrons, up electrons, centres, e-e-n order
    (13, 7, 1, 4), (16, 8, 2, 5), (17, 9, 3, 4), (31, 16, 5, 5), (32, 16, 4, 4), (33, 17, 9, 4), (40, 24, 7, 5),
    (51, 26, 13, 5), (64, 32, 33, 4), (65, 33, 17, 4), (72, 40, 12, 0), (127, 64, 32, 4), (128, 64, 40, 5),
]


def cluster(n, nup, ncent, nordc):
    s = S.cluster128(ncent=ncent, box=14.0 * (max(ncent, 4) / 32) ** (1 / 3), norb=max(nup, n - nup))
    j = S._jastrow(np.random.default_rng(3), 1, 5, 5, nordc)
    return dataclasses.replace(s, nelec=n, nup=nup, nordc=nordc, een_cusp=j["een_cusp"], c=j["c"],
                               det_orb=np.array([list(range(nup)) + list(range(n - nup))], np.int32))


@pytest.mark.parametrize("n,nup,ncent,nordc", CASES)
def test_evaluation_matches_oracle(oracle_mod, n, nup, ncent, nordc):
    from champ_b200.engine import Engine
    s = cluster(n, nup, ncent, nordc)
    nw = 3
    x = S.initial_walkers(s, nw, seed=n)
    orc = oracle_mod.Oracle(s)
    for prec in ("fp64", "mixed"):
        eng = Engine(s, nw, prec)
        eng.set_walkers(x)
        r = eng.eval_full()
        for w in range(nw):
            o = orc.eval(x[w])
            scale = max(1.0, abs(o["energy"]), abs(o["d2lnpsi"]))
            assert abs(r["lnpsi"][w] - o["lnpsi"]) <= 1e-9 * max(1.0, abs(o["lnpsi"]))
            assert abs(r["psij"][w] - o["psij"]) <= 1e-9 * max(1.0, abs(o["psij"]))
            assert r["sign"][w] == o["sign"]
            assert abs(r["pe_nonloc"][w] - o["pe_nonloc"]) <= 1e-9 * scale
            assert abs(r["energy"][w] - o["energy"]) <= 1e-9 * scale
            assert abs(r["d2lnpsi"][w] - o["d2lnpsi"]) <= 1e-9 * scale
            vs = np.abs(o["vel"]).max()
            assert np.abs(r["velocity"][w] - o["vel"]).max() <= 1e-9 * vs
            assert np.abs(r["div_v"][w] - o["div_v"]).max() <= 1e-9 * max(scale, np.abs(o["div_v"]).max())
        eng.close()


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n,nup,ncent,nordc", [c for c in CASES if c[0] > 16])
def test_batched_moves_walk_as_single_moves(n, nup, ncent, nordc, prec):
    """Two sweeps of batched moves against the same sweeps move by move (staged evaluation off): the
    same decisions, so the same positions.  The two differ in the order of FP64 sums (and with it now
    and then in an FP32 table's last bit), 1e-7 of a decision's probability at most: of 64 walkers and
    256 decisions each, one walker may differ."""
    from champ_b200.engine import Engine
    s = cluster(n, nup, ncent, nordc)
    x = S.initial_walkers(s, 64, seed=n + 1)
    out = []
    for staged in (1, 0):
        eng = Engine(s, 64, prec)
        eng.set_walkers(x)
        if not eng.get_option("staged_eval"):
            pytest.skip("walker state of this system is resident in shared memory")
        if not staged:
            eng.set_option("staged_eval", 0)
            eng.set_option("reinvert_every", 1)
        st = eng.vmc_sweeps(2, seed=5, sweep0=3, step=s.step)
        out.append((eng.get_walkers(), st["accept"]))
        eng.close()
    same = np.abs(out[0][0] - out[1][0]).max(axis=(1, 2)) <= 1e-12
    assert same.sum() >= 63, same.sum()
    assert np.array_equal(out[0][1][same], out[1][1][same])
    assert 0 < out[0][1].sum() < 64 * 2 * n


SMALL = [(1, 1, 1, 0), (2, 1, 1, 0), (3, 2, 2, 4), (4, 4, 1, 4), (5, 3, 2, 5), (7, 4, 3, 4), (8, 4, 2, 5)]


@pytest.mark.parametrize("n,nup,ncent,nordc", SMALL)
def test_small_walkers_match_oracle(oracle_mod, n, nup, ncent, nordc):
    """The 8-lanes-per-walker kernels at the edges of their range (one electron, one spin only, up to 8
    electrons and 4 of a spin): evaluation, and two sweeps walked as the oracle walks them.  The kernels serve
    many walkers only, so the oracle's 19 are the first of 4801 (not a multiple of the walkers of a block) that
    repeat them; 19 alone take the warp-per-walker kernels, to the same bounds."""
    from champ_b200.engine import Engine
    s = cluster(n, nup, ncent, nordc)
    nw = 19
    x = S.initial_walkers(s, nw, seed=n)
    many = np.resize(x, (4801,) + x.shape[1:])
    orc = oracle_mod.Oracle(s)
    for prec, y in (("fp64", many), ("mixed", many), ("fp64", x)):
        eng = Engine(s, len(y), prec)
        eng.set_walkers(y)
        r = eng.eval_full()
        assert np.array_equal(r["energy"], np.resize(r["energy"][:nw], len(y)))
        for w in range(nw):
            o = orc.eval(x[w])
            scale = max(1.0, abs(o["energy"]), abs(o["d2lnpsi"]))
            assert abs(r["lnpsi"][w] - o["lnpsi"]) <= 1e-9 * max(1.0, abs(o["lnpsi"]))
            assert r["sign"][w] == o["sign"]
            assert abs(r["pe_nonloc"][w] - o["pe_nonloc"]) <= 1e-9 * scale
            assert abs(r["energy"][w] - o["energy"]) <= 1e-9 * scale
            assert np.abs(r["velocity"][w] - o["vel"]).max() <= 1e-9 * np.abs(o["vel"]).max()
            assert np.abs(r["div_v"][w] - o["div_v"]).max() <= 1e-9 * max(scale, np.abs(o["div_v"]).max())
        if prec == "fp64":
            st = eng.vmc_sweeps(2, seed=11, sweep0=4, step=s.step)
            ref = orc.vmc(x, 2, seed=11, sweep0=4, step=s.step)
            assert np.abs(eng.get_walkers()[:nw] - ref["x"]).max() <= 1e-12
            scale = np.array([max(1.0, abs(e), abs(orc.eval(y)["d2lnpsi"])) for e, y in zip(ref["elast"], ref["x"])])
            assert np.all(np.abs(st["elast"][:nw] - ref["elast"]) <= 1e-9 * scale)
            assert np.array_equal(st["accept"][:nw], ref["accept"])
        eng.close()


@pytest.mark.parametrize("n,nup,ncent,nordc", [c for c in CASES if c[3] in (4, 5) and c[0] < 70])
def test_parameter_gradient_matches_single_kernels(n, nup, ncent, nordc):
    """Tiled forward pass and reverse sweep against the warp-per-walker kernels (staged evaluation off), FP64."""
    from champ_b200.engine import Engine
    s = cluster(n, nup, ncent, nordc)
    x = S.initial_walkers(s, 5, seed=n + 2)
    out = []
    for staged in (1, 0):
        eng = Engine(s, 5, "fp64")
        if not eng.get_option("staged_eval"):
            pytest.skip("walker state of this system is resident in shared memory")
        if not staged:
            eng.set_option("staged_eval", 0)
        eng.set_walkers(x)
        out.append(eng.param_grad())
        eng.close()
    for a, b in zip(*out):
        # per walker: sums of terms as large as the walker's largest derivative
        scale = np.abs(b).reshape(len(b), -1).max(axis=1).reshape((-1,) + (1,) * (b.ndim - 1))
        assert np.all(np.abs(a - b) <= 1e-9 * np.maximum(1.0, scale))


@pytest.mark.parametrize("first", [0, 1])
def test_gradient_passes_with_the_option_changed_between(first):
    """A tape of the single kernels swept in reverse after the staged evaluation is switched on (its distances were
    never formed), and a tiled tape after it is switched off: the derivatives of either pair of passes."""
    from champ_b200.engine import Engine
    s = cluster(40, 24, 7, 5)
    x = S.initial_walkers(s, 5, seed=42)
    ref = Engine(s, 5, "fp64")
    ref.set_option("staged_eval", 0)
    ref.set_walkers(x)
    dl0, de0, _ = ref.param_grad()
    ref.close()
    eng = Engine(s, 5, "fp64")
    eng.set_option("staged_eval", first)
    eng.set_walkers(x)
    eng.param_grad_fwd()
    eng.set_option("staged_eval", 1 - first)
    dl, de = eng.param_grad_bwd()
    eng.close()
    for a, b in ((dl, dl0), (de, de0)):
        assert np.all(np.abs(a - b) <= 1e-9 * np.maximum(1.0, np.abs(b).max(axis=1, keepdims=True)))


@pytest.mark.parametrize("n,nup,ncent,nordc", [(33, 17, 9, 4), (51, 26, 13, 5), (65, 33, 17, 4), (72, 40, 33, 4)])
def test_parameter_gradient_with_virtual_orbitals(n, nup, ncent, nordc):
    """As above with three orbitals to a centre, so that the points' coefficients have room and the tiles serve
    beyond 32 and 64 electrons and 32 centres, and orbital rotations into virtual orbitals are among the parameters."""
    from champ_b200.engine import Engine
    s = cluster(n, nup, ncent, nordc)
    s = dataclasses.replace(s, coef=S.cluster128(ncent=ncent, box=14.0 * (max(ncent, 4) / 32) ** (1 / 3), norb=3 * ncent).coef)
    x = S.initial_walkers(s, 3, seed=n + 2)
    out = []
    for staged in (1, 0):
        eng = Engine(s, 3, "fp64")
        eng.set_option("staged_eval", staged)
        eng.set_walkers(x)
        out.append(eng.param_grad())
        eng.close()
    assert not all(np.array_equal(a, b) for a, b in zip(*out))  # two kernels
    for a, b in zip(*out):
        scale = np.abs(b).reshape(len(b), -1).max(axis=1).reshape((-1,) + (1,) * (b.ndim - 1))
        assert np.all(np.abs(a - b) <= 1e-9 * np.maximum(1.0, scale))
