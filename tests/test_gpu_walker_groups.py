"""Uneven batches in walker groups: each group launches only what its own walkers need.

A group's largest N, slices per block, number of blocks, spins, kind of exp(-dtau K) and kind
of stabilization size its launches.  The groups here differ in each of them, and one holds
shared-memory walkers only.  One group and four give the same fields and Green's functions bit
for bit; the measured sums may be added in another order (the number of CTAs follows the
group's largest N), so they agree within 1e-12.
"""
import numpy as np
import pytest

from test_gpu_parity import dq  # noqa: F401

pytestmark = pytest.mark.gpu

# (model, L, Lt, pace, checkerboard), two walkers a group
SHAPES = [(0, 4, 10, 5, False), (1, 6, 9, 3, False),      # FP64: shared-memory walkers only
          (1, 10, 12, 4, True), (1, 12, 8, 8, True),      # one spin, plaquettes
          (0, 9, 10, 5, False), (0, 5, 20, 5, False),     # two spins, dense
          (1, 17, 6, 2, False), (0, 12, 7, 7, True)]      # N = 289 beside N = 144


@pytest.mark.parametrize("mixed", [False, True])
def test_uneven_groups_give_identical_walkers(dq, monkeypatch, mixed):  # noqa: F811
    descs = [dq.WalkerDesc(model=m, L=L, U=4.0, mu=-0.4 * m, beta=0.1 * Lt, Lt=Lt, pace=pace, checkerboard=cb,
                           seed=700 + i) for i, (m, L, Lt, pace, cb) in enumerate(SHAPES)]
    monkeypatch.setenv("DQMC_METROPOLIS_KIND", "2")  # both runs the same, whatever the tuner times
    n, res = len(descs), []
    for groups in ("1", "4"):
        monkeypatch.setenv("DQMC_STREAM_GROUPS", groups)
        b = dq.Batch(descs, rng=dq.RNG_PHILOX, precision=dq.MIXED if mixed else dq.FP64)
        for w in range(n):
            b.fields_random(w)
        b.init_greens()
        b.sweep_0_to_beta(measure=True)
        b.sweep_beta_to_0(measure=True)
        b.sweep_dynamic([0, 3, 5])
        res.append(([b.fields(w) for w in range(n)], [b.green(w, 0) for w in range(n)],
                    [b.dynamic(w)[0] for w in range(n)], b.observables_all(), [b.status(w) for w in range(n)]))
        b.close()
    (f1, g1, d1, o1, s1), (f4, g4, d4, o4, s4) = res
    assert s1 == s4 == [0] * n
    for w in range(n):
        np.testing.assert_array_equal(f1[w], f4[w])
        np.testing.assert_array_equal(g1[w], g4[w])
        np.testing.assert_allclose(d1[w], d4[w], rtol=1e-12, atol=1e-12)
    np.testing.assert_allclose(o1[0], o4[0], rtol=1e-12, atol=1e-12)
    np.testing.assert_array_equal(o1[1], o4[1])


def test_uneven_groups_with_the_split_kernels(dq, monkeypatch):  # noqa: F811
    """The split Metropolis kernels' grids (128-line blocks, column tiles, spins) follow the group's
    largest walker: one group and four, to the bit."""
    monkeypatch.setenv("DQMC_METROPOLIS_KIND", "3")
    descs = [dq.WalkerDesc(model=m, L=L, U=4.0, mu=-0.4 * m, beta=0.1 * Lt, Lt=Lt, pace=pace, checkerboard=cb,
                           seed=720 + i) for i, (m, L, Lt, pace, cb) in enumerate(SHAPES)]
    res = []
    for groups in ("1", "4"):
        monkeypatch.setenv("DQMC_STREAM_GROUPS", groups)
        b = dq.Batch(descs, rng=dq.RNG_PHILOX, precision=dq.MIXED)
        for w in range(len(descs)):
            b.fields_random(w)
        b.init_greens()
        assert b.tuning()["tc_flush"] == 3
        b.sweep_0_to_beta(measure=True)
        b.sweep_beta_to_0(measure=True)
        res.append([x for w in range(len(descs)) for x in (b.fields(w), b.green(w, 0), b.status(w))])
        b.close()
    for a, c in zip(*res):
        np.testing.assert_array_equal(a, c)
