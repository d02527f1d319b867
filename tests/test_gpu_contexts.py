"""Several contexts in one process: what one sets for its kernels takes nothing from another."""
import dataclasses

import numpy as np
import pytest

from champ_b200 import system as S

pytestmark = pytest.mark.gpu


def cluster(n, ncent, nordc):
    s = S.cluster128(ncent=ncent, box=14.0 * (max(ncent, 4) / 32) ** (1 / 3), norb=3 * ncent)
    j = S._jastrow(np.random.default_rng(3), 1, 5, 5, nordc)
    nup = (n + 1) // 2
    return dataclasses.replace(s, nelec=n, nup=nup, nordc=nordc, een_cusp=j["een_cusp"], c=j["c"],
                               det_orb=np.array([list(range(nup)) + list(range(n - nup))], np.int32))


@pytest.mark.parametrize("large,small", [("cluster", "cluster"), ("cluster", "dimer"), ("dimer", "be")])
@pytest.mark.parametrize("prec", ["fp64", "mixed", "fp32"])
def test_a_smaller_context_leaves_a_larger_one_alone(large, small, prec):
    """Kernels' shared-memory limits are per process: every call of the larger context runs as before after a
    smaller one of the same e-e-n order is made, to the same bits."""
    from champ_b200.engine import Engine
    big = cluster(70, 18, 4) if large == "cluster" else dataclasses.replace(S.c2_dimer(), nordc=0, een_cusp=0, c=np.zeros((1, 0)))
    little = cluster(20, 5, 4) if small == "cluster" else S.c2_dimer() if small == "dimer" else S.be_atom()
    x = S.initial_walkers(big, 40, seed=3)

    def calls(eng):
        eng.set_mover(1)
        eng.set_walkers(x)
        out = [eng.eval_full()["energy"], *eng.param_grad()]
        r, g = eng.propose_1e(1, x[:, 1] + 0.1, grad=True)
        eng.accept_1e(1, np.ones(len(x), np.uint8))
        out += [r, g]
        for mover in (1, 6):
            eng.set_mover(mover)
            st = eng.vmc_sweeps(1, seed=4, sweep0=1, step=big.step)
            out += [st["elast"], eng.get_walkers()]
        return out

    eng = Engine(big, 40, prec)
    before = calls(eng)
    other = Engine(little, 8, prec)
    other.set_walkers(S.initial_walkers(little, 8, seed=2))
    other.vmc_sweeps(1, seed=1, sweep0=0, step=little.step)
    after = calls(eng)
    for a, b in zip(before, after):
        assert np.allclose(a, b, rtol=1e-12, atol=0, equal_nan=True)
    eng.close()
    other.close()
