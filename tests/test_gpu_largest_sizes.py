"""HBM walkers above 24 x 24, up to the largest (N = 1024), and the line at N = 768 between the
blocked stabilization and the column-at-a-time one.  Checkerboard walkers of even sides, whose
set-up needs no diagonalisation on the host; a few slices, one walker of a kind.  FP64 on both sides
of the line against numpy's inverse on the walker's last fields (1e-10), both kinds in one batch
against batches of their own to the bit, and the tensor-core path against FP64 at the bar of
tests/test_gpu_mixed.py (identical decisions, 1e-6).
"""
import numpy as np
import pytest

from test_gpu_parity import dq  # noqa: F401

pytestmark = pytest.mark.gpu


def _walker(dq, L, model):  # noqa: F811
    return dq.WalkerDesc(model=model, L=L, U=4.0, mu=-0.3 if model else 0.0, beta=0.4, Lt=4, pace=2, checkerboard=True,
                         seed=800 + L)


def _greens(d, fields):
    """G = (1 + B_Lt ... B_1)^-1 with B = diag(exp(alpha s)) A B, the plaquette layers multiplied out
    (well conditioned at this beta)."""
    L, dtau = d.L, d.beta / d.Lt
    alpha = np.arccosh(np.exp(0.5 * dtau * d.U))
    ch, sh = np.cosh(dtau * d.t), np.sinh(dtau * d.t)
    plaq = np.exp(0.5 * dtau * d.mu) * np.kron([[ch, sh], [sh, ch]], [[ch, sh], [sh, ch]])

    def layer(parity):
        k = np.zeros((d.N, d.N))
        for x in range(parity, L, 2):
            for y in range(parity, L, 2):
                x1, y1 = (x + 1) % L, (y + 1) % L
                at = [x + L * y, x1 + L * y, x + L * y1, x1 + L * y1]
                k[np.ix_(at, at)] = plaq
        return k

    hop, p = layer(0) @ layer(1), np.eye(d.N)
    for f in fields:
        p = np.exp(alpha * f)[:, None] * (hop @ p)
    return np.linalg.inv(np.eye(d.N) + p)


def _run(dq, descs, **kw):  # noqa: F811
    b = dq.Batch(descs, rng=dq.RNG_MINSTD, **kw)
    for w in range(len(descs)):
        b.fields_random(w)
    b.init_greens()
    b.sweep_0_to_beta(measure=True)
    b.sweep_beta_to_0(measure=True)
    green = [b.green(w, 0) for w in range(len(descs))]  # at t = 0
    b.sweep_dynamic([0, 1, 3])
    out = [(b.fields(w), green[w], b.green_dynamic(w, 0, 0), b.dynamic(w)[0], b.observables(w)[0], b.status(w))
           for w in range(len(descs))]
    b.close()
    return out


def test_both_stabilizations_in_one_batch(dq):  # noqa: F811
    descs = [_walker(dq, L, m) for L, m in ((26, 0), (28, 1), (32, 1))]
    together = _run(dq, descs)
    for d, a in zip(descs, together):
        c, = _run(dq, [d])
        assert a[-1] == c[-1] == 0
        for x, y in zip(a, c):
            np.testing.assert_array_equal(x, y)
        assert abs(a[1] - _greens(d, a[0])).max() <= 1e-10


@pytest.mark.parametrize("L", [26, 32])
def test_mixed_against_fp64(dq, L):  # noqa: F811
    (mixed,), (plain,) = (_run(dq, [_walker(dq, L, 1)], precision=p) for p in (dq.MIXED, dq.FP64))
    assert mixed[-1] == plain[-1] == 0
    np.testing.assert_array_equal(mixed[0], plain[0])
    for k in (1, 2, 3):
        assert abs(mixed[k] - plain[k]).max() <= 1e-6
