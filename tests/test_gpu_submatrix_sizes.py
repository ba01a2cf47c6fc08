"""The split submatrix kernels (decisions, preparation per spin and 128 lines, flush per spin and
column tiles) against the fused kernel, bit for bit, where their tiles and blocks end: less than a
32-site block's neighbour, one and two 128-line blocks with ragged ends, odd column tiles, one and
two spins.  Both forms run the same arithmetic, so G is equal to the bit, and the decisions are the
FP64 path's."""
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
@pytest.mark.parametrize("L,lattice", [(5, 0), (6, 0), (11, 0), (12, 0), (13, 0), (16, 0), (5, 1)])
def test_split_equals_fused(dq, monkeypatch, model, L, lattice):
    descs = [dq.WalkerDesc(model=model, L=L, U=4.0, mu=-0.3 if model else 0.0, beta=0.6, Lt=6, pace=3,
                           seed=700 + 10 * L + w, lattice=lattice) for w in range(2)]
    out = []
    for kind in ("2", "3", None):
        if kind:
            monkeypatch.setenv("DQMC_METROPOLIS_KIND", kind)
        else:
            monkeypatch.delenv("DQMC_METROPOLIS_KIND")
        b = dq.Batch(descs, rng=dq.RNG_PHILOX, precision=dq.MIXED if kind else dq.FP64, hbm=True)
        r = np.random.default_rng(L)
        for w, d in enumerate(descs):
            b.set_fields(w, (2 * r.integers(0, 2, size=(d.Lt, d.N)) - 1).astype(np.int8))
        b.init_greens()
        if kind:
            assert b.tuning()["tc_flush"] == int(kind)
        b.sweep_0_to_beta()
        b.sweep_beta_to_0()
        out.append(([b.fields(w) for w in (0, 1)], [b.green(w, s) for w in (0, 1) for s in (0, 1)],
                    [b.accept_count(w) for w in (0, 1)], [b.status(w) for w in (0, 1)]))
        b.close()
    fused, split, plain = out
    for k in (0, 1):
        np.testing.assert_array_equal(fused[0][k], split[0][k])
        np.testing.assert_array_equal(fused[0][k], plain[0][k])
    for a, c in zip(fused[1], split[1]):
        np.testing.assert_array_equal(a, c)
    assert fused[2] == split[2] == plain[2]
    assert fused[3] == split[3] == plain[3] == [0, 0]


@pytest.mark.parametrize("model", [0, 1])
def test_blocks_without_accepts(dq, monkeypatch, model):
    """Strong coupling on fields that have settled: most 32-site blocks accept nothing, so the fused
    kernel's warps go from block to block meeting at one barrier only, and the blocks that do accept
    lie at every parity.  Equal to the split kernels to the bit."""
    descs = [dq.WalkerDesc(model=model, L=12, U=10.0, beta=8.0, Lt=16, pace=1, seed=60 + w) for w in range(4)]
    out = []
    for kind in ("2", "3"):
        monkeypatch.setenv("DQMC_METROPOLIS_KIND", kind)
        b = dq.Batch(descs, rng=dq.RNG_PHILOX, precision=dq.MIXED)
        r = np.random.default_rng(model)
        for w, d in enumerate(descs):
            b.set_fields(w, (2 * r.integers(0, 2, size=(d.Lt, d.N)) - 1).astype(np.int8))
        b.init_greens()
        accepts = []
        for _ in range(6):
            before = [b.accept_count(w) for w in range(4)]
            b.sweep_0_to_beta()
            b.sweep_beta_to_0()
            accepts.append([b.accept_count(w) - x for w, x in enumerate(before)])
        out.append(([b.fields(w) for w in range(4)], [b.green(w, 0) for w in range(4)], accepts,
                    [b.status(w) for w in range(4)]))
        b.close()
    (f2, g2, a2, s2), (f3, g3, a3, s3) = out
    # 160 blocks a walker and pair of half-sweeps, 154 to 177 accepts in the last pair of a chain of the
    # oracle: every third block or so has none
    assert min(a2[-1]) < 320
    assert a2 == a3 and s2 == s3 == [0] * 4
    for a, c in zip(f2 + g2, f3 + g3):
        np.testing.assert_array_equal(a, c)
