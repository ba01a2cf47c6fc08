"""Device memory of a walker: its state, the buffers that every path needs, and no more.

The bytes are those of two batches of different numbers of walkers, taken apart, so that what a batch
or the device holds once does not count.  The bound lists the arrays of a walker: G, the chain's two
buffers, a product temporary, the factorization's matrix and right-hand sides, the stacks, the fields;
on the mixed path also the slices of one wrap operand, the Metropolis updates' slices and room for the
slices of two N x N operands of the stabilization (one up to 127 sites, where it has none).  128 KB
for the allocations' granularity (2 MB over 30 walkers) and the small arrays.
"""
import pytest

from test_gpu_parity import dq  # noqa: F401

pytestmark = pytest.mark.gpu


def _bound(d, mixed):
    n, s, up = d.N, 1 if d.model else 2, lambda x, m: -(-x // m) * m
    levels = -(-d.Lt // d.pace)
    total = 8 * n * n * (2 + 2 * s + s + 2 * s) + 8 * 2 * s * levels * up(2 * n * n + n, 32) + d.Lt * n
    if mixed:
        lines = up(n, 128)
        total += 2 * s * 8 * lines * up(n, 16)             # eight slices of a wrap operand
        total += 2 * s * 6 * 32 * (128 + 3 * lines)        # six slices of Gamma and three N x 32 operands
        total += 2 * s * 9 * lines * up(n, 32) * (2 if n >= 128 else 1)
    return total + 128 * 1024


@pytest.mark.parametrize("mixed,L,model", [(True, 10, 0), (True, 12, 0), (True, 16, 1), (True, 24, 0), (False, 10, 0),
                                           (False, 16, 1)])
def test_walker_fits_its_arrays(dq, mixed, L, model):  # noqa: F811
    import torch

    def used(walkers):
        before = torch.cuda.mem_get_info()[0]
        b = dq.Batch([dq.WalkerDesc(model=model, L=L, U=4.0, beta=1.0, Lt=10, pace=5, seed=w) for w in range(walkers)],
                     rng=dq.RNG_PHILOX, precision=dq.MIXED if mixed else dq.FP64)
        after = torch.cuda.mem_get_info()[0]
        b.close()
        return before - after

    used(2)  # what the first batch of a process loads
    few, many = used(4), used(34)
    d = dq.WalkerDesc(model=model, L=L, U=4.0, beta=1.0, Lt=10, pace=5)
    assert (many - few) / 30 <= _bound(d, mixed), ((many - few) / 30, _bound(d, mixed))
