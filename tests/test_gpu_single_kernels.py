"""The kernels that serve where the tiles do not, on systems and options that reach them: several centre types
with e-e-n terms (k_el_jas, k_el_fin), one or two and more than 64 orbitals of a spin (k_el_orb), the moves with a shared
coefficient stream and with delayed inverse updates, and the gradient's passes by a warp per walker."""
import dataclasses

import numpy as np
import pytest

from champ_b200 import system as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw", [256, 254])
def test_cooperative_moves_without_batches(nw):
    """Staged evaluation off: the FP32 moves run electron by electron, with the block's coefficient stream shared or
    not.  The same sums in the same order, so the same walk, bit for bit."""
    from champ_b200.engine import Engine
    s = S.cluster128(ncent=8)
    x = S.initial_walkers(s, nw, seed=17)
    out = {}
    for coop in (1, 0):
        eng = Engine(s, nw, "mixed")
        eng.set_option("staged_eval", 0)
        eng.set_option("move_coop", coop)
        eng.set_walkers(x)
        st = eng.vmc_sweeps(3, seed=23, sweep0=0, step=s.step)
        out[coop] = (eng.get_walkers(), st)
        eng.close()
    assert np.array_equal(out[0][0], out[1][0])
    for k in ("accept", "esum", "elast"):
        assert np.array_equal(out[0][1][k], out[1][1][k]), k
    assert out[1][1]["accept"].mean() > 0.1


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_delayed_updates_without_batches(prec):
    """Staged evaluation off: delayed against immediate updates of the inverse.  Ratios agree to rounding, so a
    walker splits off only where a decision ties: at most 1 of 20."""
    from champ_b200.engine import Engine
    s = S.get_system(5)
    nw = 64
    x = S.initial_walkers(s, nw, seed=13)
    out = []
    for rank in (4, 0):
        eng = Engine(s, nw, prec)
        eng.set_option("staged_eval", 0)
        eng.set_option("delay_rank", rank)
        eng.set_walkers(x)
        st = eng.vmc_sweeps(2, seed=17, sweep0=0, step=s.step)
        out.append((eng.get_walkers(), st))
        eng.close()
    (xa, sa), (xb, sb) = out
    same = np.all(np.abs(xa - xb) <= 1e-12, axis=(1, 2))
    assert same.mean() >= 0.95, same.mean()
    assert np.array_equal(sa["accept"][same], sb["accept"][same])
    assert 0 < sa["accept"].sum() < 2 * nw * s.nelec


def test_gradient_pair_matches_one_pass_by_single_kernels():
    """Staged evaluation off, 128 electrons, FP64: forward and reverse pass against the one-pass kernel."""
    from champ_b200.engine import Engine
    s = S.get_system(5)
    x = S.initial_walkers(s, 8, seed=90)
    eng = Engine(s, 8, "fp64")
    eng.set_option("staged_eval", 0)
    eng.set_walkers(x)
    eng.set_option("param_grad_mode", 1)
    dl1, de1, el1 = eng.param_grad()
    eng.set_option("param_grad_mode", 0)
    el0 = eng.param_grad_fwd()
    dl0, de0 = eng.param_grad_bwd()
    eng.close()
    assert np.allclose(el0, el1, rtol=1e-12, atol=1e-12)
    assert np.all(np.abs(dl0 - dl1) <= 1e-9 * np.maximum(1.0, np.abs(dl1)))
    assert np.all(np.abs(de0 - de1) <= 1e-9 * np.maximum(1.0, np.abs(el1))[:, None])


def molecule(n, nup, ncent, nordc, nct=1, norb=None):
    """A cluster of nct elements, each with its own e-n and e-e-n parameters and pseudopotential."""
    s = S.cluster128(ncent=ncent, box=14.0 * (max(ncent, 4) / 32) ** (1 / 3), norb=norb or max(nup, n - nup))
    rng = np.random.default_rng(7)
    s = dataclasses.replace(s, nelec=n, nup=nup, iwctype=np.arange(ncent, dtype=np.int32) % nct,
                            det_orb=np.array([list(range(nup)) + list(range(n - nup))], np.int32),
                            **S._jastrow(rng, nct, 5, 5, nordc))
    return s if nct == 1 else dataclasses.replace(s, znuc=np.array([4.0, 3.0]), **S._gaussian_ecp(rng, nct))


def excitations(s, norb):
    """The determinant of s and every single excitation of its first up electron into the orbitals up to norb."""
    ref = list(s.det_orb[0])
    det = [ref] + [[k] + ref[1:] for k in range(s.nup, norb)]
    m = len(det) - 1
    return dataclasses.replace(s, det_orb=np.array(det, np.int32), csf_coef=np.array([1.0, 0.05]), csf_ndet=np.array([1, m], np.int32),
                               csf_det=np.arange(m + 1, dtype=np.int32), csf_det_coef=np.cos(np.arange(m + 1.0)))


def check_evaluation(orc, x, r):
    """The parity tests' bounds, as in the tests of the tiles."""
    for w in range(len(x)):
        o = orc.eval(x[w])
        scale = max(1.0, abs(o["energy"]), abs(o["d2lnpsi"]))
        assert abs(r["lnpsi"][w] - o["lnpsi"]) <= 1e-9 * max(1.0, abs(o["lnpsi"]))
        assert r["sign"][w] == o["sign"]
        assert abs(r["pe_nonloc"][w] - o["pe_nonloc"]) <= 1e-9 * scale
        assert abs(r["energy"][w] - o["energy"]) <= 1e-9 * scale
        assert np.abs(r["velocity"][w] - o["vel"]).max() <= 1e-9 * np.abs(o["vel"]).max()
        assert np.abs(r["div_v"][w] - o["div_v"]).max() <= 1e-9 * max(scale, np.abs(o["div_v"]).max())


SYSTEMS = {
    "two elements, order 4": lambda: molecule(33, 17, 9, 4, nct=2),
    "two elements, order 5": lambda: molecule(20, 11, 5, 5, nct=2),
    "two elements, no e-e-n": lambda: molecule(36, 18, 6, 0, nct=2),
    "two orbitals and one": lambda: molecule(3, 2, 44, 4),
    "76 orbitals of a spin": lambda: excitations(molecule(20, 10, 8, 4, norb=80), 76),
    "250 orbitals of a spin": lambda: excitations(molecule(16, 8, 32, 4, norb=256), 250),
}


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("name", SYSTEMS)
def test_evaluation_and_sweep_follow_the_oracle(oracle_mod, name, prec):
    from champ_b200.engine import Engine
    s = SYSTEMS[name]()
    x = S.initial_walkers(s, 3, seed=s.nelec)
    orc = oracle_mod.Oracle(s)
    eng = Engine(s, 3, prec)
    assert eng.get_option("staged_eval")
    eng.set_walkers(x)
    check_evaluation(orc, x, eng.eval_full())
    st = eng.vmc_sweeps(1, seed=11, sweep0=4, step=s.step)
    y = eng.get_walkers()
    check_evaluation(orc, y, eng.eval_full())
    if prec == "fp64":
        ref = orc.vmc(x, 1, seed=11, sweep0=4, step=s.step)
        assert np.abs(y - ref["x"]).max() <= 1e-12
        assert np.array_equal(st["accept"], ref["accept"])
    assert 0 < st["accept"].sum() < 3 * s.nelec
    eng.close()


def test_autotune_times_what_the_sweeps_read(tmp_path):
    """Options without effect on the batched Gaussian sweeps keep their values, also in the cache; the accelerated
    mover's delayed updates are timed."""
    from champ_b200.engine import Engine
    s = S.cluster128(ncent=8)
    eng = Engine(s, 64, "mixed")
    eng.set_walkers(S.initial_walkers(s, 64, seed=3))
    eng.set_option("delay_rank", 8)
    eng.set_option("orb_coop", 0)
    cache = tmp_path / "tune.txt"
    rep = eng.autotune(nsweep=1, cache=str(cache))
    assert "staged_eval ms/sweep" in rep
    assert eng.get_option("staged_eval") == 1  # several times faster
    for name in ("delay_rank", "move_coop", "orb_coop"):
        assert name + " ms/sweep" not in rep, rep
    assert (eng.get_option("delay_rank"), eng.get_option("move_coop"), eng.get_option("orb_coop")) == (8, 1, 0)
    assert "delay_rank=8 move_coop=1 orb_coop=0" in cache.read_text()
    eng.set_mover(6)
    rep = eng.autotune(nsweep=1)
    assert "delay_rank ms/sweep" in rep and "move_coop ms/sweep" not in rep, rep
    eng.close()
