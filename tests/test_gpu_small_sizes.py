"""Shared-memory FP64 walkers at every size where their kernels change shape, against the oracle.

The block products give a thread 1, 3, 6, 10 or 16 outputs (N up to 16, 27, 39, 50, 64), the
rank-1 update takes two columns a warp up to N = 16, the chain lives beside G up to N = 50, and
the Metropolis scan takes windows of 16 sites (both spins) or 32 (one): sides 2 to 8 with each
model, the plaquette passes at even sides, and the small cubes.  Identical decisions, G and
observables within 1e-10, the bar of tests/test_gpu_parity.py.
"""
import pytest

from test_gpu_parity import _run_pair, dq  # noqa: F401

pytestmark = pytest.mark.gpu

SHAPES = ([(m, L, False, 0) for m in (0, 1) for L in range(2, 9)]
          + [(m, L, True, 0) for m in (0, 1) for L in (4, 6, 8)]
          + [(0, 2, False, 1), (1, 3, False, 1), (0, 3, False, 1), (0, 4, False, 1)])


@pytest.mark.parametrize("model,L,cb,lattice", SHAPES)
def test_small_walker_against_oracle(dq, oracle_mod, model, L, cb, lattice):  # noqa: F811
    d = dq.WalkerDesc(model=model, L=L, U=4.0, mu=-0.3 if model else 0.0, beta=1.5, Lt=15, pace=6, checkerboard=cb,
                      seed=300 + L, lattice=lattice)
    _run_pair(dq, oracle_mod, [d], sweeps=1)


def test_mixed_small_sizes_share_a_batch(dq, oracle_mod):  # noqa: F811
    """The largest walker of a batch (N = 64) decides where every walker's chain lives."""
    descs = [dq.WalkerDesc(model=L % 2, L=L, U=4.0, beta=1.0, Lt=10, pace=5, seed=40 + L) for L in (3, 7, 8)]
    _run_pair(dq, oracle_mod, descs, sweeps=1)
