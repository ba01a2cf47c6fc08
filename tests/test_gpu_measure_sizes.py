"""The equal-time measurement of HBM walkers (a cluster of 1, 2, 4 or 8 CTAs a walker over pairs of
32-site tiles) against the shared-memory kernels' on the same chains, where tiles end and where the
cluster size changes: one site past a tile, one and two tiles, odd sides (whose Fourier table is
not even), one and two spins, cubes; and against the oracle above 64 sites."""
import numpy as np
import pytest

from test_gpu_parity import _run_pair, dq  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", [0, 1])
@pytest.mark.parametrize("L,lattice", [(2, 0), (3, 0), (5, 0), (6, 0), (7, 0), (8, 0), (3, 1), (4, 1)])
def test_hbm_measurement_against_shared_memory(dq, model, L, lattice):  # noqa: F811
    d = dq.WalkerDesc(model=model, L=L, U=4.0, mu=-0.3 if model else 0.0, beta=1.0, Lt=10, pace=5, seed=500 + L,
                      lattice=lattice)
    out = []
    for hbm in (False, True):
        b = dq.Batch([d], rng=dq.RNG_MINSTD, hbm=hbm)
        b.fields_random(0)
        b.init_greens()
        b.sweep_0_to_beta(measure=True)
        b.sweep_beta_to_0(measure=True)
        assert b.status(0) == 0
        out.append((b.fields(0), *b.observables(0)))
        b.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][2], out[1][2])
    np.testing.assert_allclose(out[1][1], out[0][1], rtol=1e-10, atol=1e-10)


@pytest.mark.parametrize("model,L,lattice", [(0, 9, 0), (1, 10, 0), (0, 5, 1), (1, 12, 0)])
def test_hbm_measurement_against_oracle(dq, oracle_mod, model, L, lattice):  # noqa: F811
    d = dq.WalkerDesc(model=model, L=L, U=4.0, mu=-0.3 if model else 0.0, beta=0.8, Lt=8, pace=4, seed=520 + L,
                      lattice=lattice)
    _run_pair(dq, oracle_mod, [d], sweeps=1)


@pytest.mark.parametrize("L", [5, 7, 9])
def test_measured_sums_do_not_depend_on_the_batch(dq, L):  # noqa: F811
    """Beside a larger walker the cluster is that one's; a walker's sums stay the same to the bit."""
    out = []
    for others in ([], [12], [16]):
        b = dq.Batch([dq.WalkerDesc(model=0, L=x, U=4.0, beta=1.0, Lt=10, pace=5, seed=560 + x) for x in [L, *others]],
                     rng=dq.RNG_PHILOX, hbm=True)
        for w in range(1 + len(others)):
            b.fields_random(w)
        b.init_greens()
        b.sweep_0_to_beta(measure=True)
        b.sweep_beta_to_0(measure=True)
        out.append((b.fields(0), b.green(0, 0), *b.observables(0)))
        b.close()
    for o in out[1:]:
        for a, c in zip(out[0], o):
            np.testing.assert_array_equal(a, c)
