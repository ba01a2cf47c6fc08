"""The factored exp(-+dtau K) products of HBM walkers (kin_op_kernel: whole columns or rows of about
2048 elements a CTA) against the shared-memory kernels' on the same chains: every side from 2 to 8,
both kinds of factors, two and three directions (and the FP64 submatrix updates); the last tile of columns or rows is ragged at
most sides.  Identical decisions and G within 1e-10, the bar of the FP64 paths."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dq():
    import __graft_entry__ as g

    g.build()
    import dqmc_gb300

    return dqmc_gb300


@pytest.mark.parametrize("L,cb,lattice", [(L, False, 0) for L in range(2, 9)] + [(4, True, 0), (6, True, 0), (8, True, 0)]
                         + [(2, False, 1), (3, False, 1), (4, False, 1)])
def test_hbm_products_against_shared_memory(dq, L, cb, lattice):
    descs = [dq.WalkerDesc(model=m, L=L, U=4.0, mu=-0.4 if m else 0.0, beta=1.2, Lt=13, pace=5, checkerboard=cb,
                           seed=900 + 10 * L + m, lattice=lattice) for m in (0, 1)]
    out = []
    for hbm in (False, True):
        b = dq.Batch(descs, rng=dq.RNG_MINSTD, hbm=hbm)
        for w in (0, 1):
            b.fields_random(w)
        b.init_greens()
        b.sweep_0_to_beta()
        b.sweep_beta_to_0()
        b.sweep_dynamic([0, 3, 12])
        out.append(([b.fields(w) for w in (0, 1)], [b.green(w, s) for w in (0, 1) for s in (0, 1)],
                    [b.green_dynamic(w, k, s) for w in (0, 1) for k in (0, 1) for s in (0, 1)],
                    [b.status(w) for w in (0, 1)]))
        b.close()
    small, large = out
    assert small[3] == large[3] == [0, 0]
    for a, c in zip(small[0], large[0]):
        np.testing.assert_array_equal(a, c)
    for a, c in zip(small[1] + small[2], large[1] + large[2]):
        assert abs(a - c).max() <= 1e-10 * max(1.0, abs(a).max())


@pytest.mark.parametrize("mixed", [False, True])
def test_many_slices_on_few_sites(dq, mixed):
    """Lt N bytes of fields are more than the scratch of a 2 x 2 walker's matrices holds: the set-up
    trials of HBM walkers leave the stacks and the fields as they are."""
    out = []
    for hbm in (False, True):
        b = dq.Batch([dq.WalkerDesc(model=1, L=2, U=4.0, mu=-0.3, beta=4.0, Lt=400, pace=200, seed=8)], rng=dq.RNG_MINSTD,
                     hbm=hbm, precision=dq.MIXED if mixed and hbm else dq.FP64)
        b.fields_random(0)
        b.init_greens()
        b.sweep_0_to_beta()
        b.sweep_beta_to_0()
        out.append((b.fields(0), b.green(0, 0), b.status(0), b.wrap_error(0)))
        b.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    assert out[0][2] == out[1][2] == 0
    # two ways to wrap 200 slices: their distance from a fresh G bounds how far apart they may be
    assert abs(out[0][1] - out[1][1]).max() <= 1e-10 + out[0][3] + out[1][3]
