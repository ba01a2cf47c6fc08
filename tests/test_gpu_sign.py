"""The initial sign of HBM walkers (one CTA per spin, the next pivot found while the column updates
run) against numpy's determinants of the same G, at sides around the warp's width and its multiples,
one and two spins."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dq():
    import __graft_entry__ as g

    g.build()
    import dqmc_gb300

    return dqmc_gb300


@pytest.mark.parametrize("model", [0, 1])
@pytest.mark.parametrize("L", [2, 3, 5, 6, 8, 11, 16])
def test_sign_against_numpy(dq, model, L):
    descs = [dq.WalkerDesc(model=model, L=L, U=4.0, mu=-0.4 if model else 0.3, beta=1.0, Lt=10, pace=5, seed=60 + w)
             for w in range(4)]
    b = dq.Batch(descs, rng=dq.RNG_MINSTD, hbm=True)
    for w in range(4):
        b.fields_random(w)
    b.init_greens()
    for w in range(4):
        s = np.prod([np.linalg.slogdet(b.green(w, k))[0] for k in (0, 1)])
        assert b.config_sign(w) == s
    b.close()
