"""How far a freshly assembled G of the FP64 walkers above shared memory is from its exact value.

G at a stabilization in the middle of a half-sweep is built from both stacks, each a chain of
graded products; a QR that does not pivot on the columns as they stand loses digits there, more
with beta, U and the size.  The reference is the same stack in numpy's long double (80 or 113
bits, at least 2000 times finer), the yardstick the same stack in 64 bits with a pivot per column.

Two equally accurate forms differ by a factor of e or so on one matrix (the shared-memory kernels,
which pivot, against numpy at 8 x 8: 1.3 in the geometric mean of twelve, 0.5 to 8 on single ones),
so on the geometric mean of n matrices by exp(3 / sqrt(n)) at three deviations: 2.9 at the eight
taken here.  4 leaves room for the factors of exp(-dtau K), which differ from numpy's by rounding.
"""
import numpy as np
import pytest

from test_gpu_parity import dq  # noqa: F401

pytestmark = pytest.mark.gpu


def _kinetic(L):
    k, i = np.zeros((L * L, L * L)), np.arange(L * L)
    for n in ((i + 1) % L + L * (i // L), (i + L) % (L * L)):
        k[i, n] -= 1.0
        k[n, i] -= 1.0
    return k


def _householder(x):
    """v (v_0 = 1), tau and beta of the reflector that takes x to beta e_0."""
    v, s = x.copy(), (x[1:] ** 2).sum()
    v[0] = 1
    if s == 0:
        return v, x[0] * 0, x[0]
    beta = -np.copysign(np.sqrt(x[0] ** 2 + s), x[0])
    v[1:] /= x[0] - beta
    return v, (beta - x[0]) / beta, beta


def _pivoted_qr(a):
    a, n = a.copy(), len(a)
    perm, v, tau = np.arange(n), np.zeros_like(a), np.zeros(n, a.dtype)
    for k in range(n):
        p = k + int(np.argmax((a[k:, k:] ** 2).sum(0)))
        a[:, [k, p]] = a[:, [p, k]]
        perm[[k, p]] = perm[[p, k]]
        v[k:, k], tau[k], beta = _householder(a[k:, k])
        a[k:, k + 1:] -= tau[k] * np.outer(v[k:, k], v[k:, k] @ a[k:, k + 1:])
        a[k, k], a[k + 1:, k] = beta, 0
    q = np.eye(n, dtype=a.dtype)
    for k in range(n - 1, -1, -1):
        q[k:, k:] -= tau[k] * np.outer(v[k:, k], v[k:, k] @ q[k:, k:])
    return q, a, perm


def _stack(slices, transposed, pace):
    """U, D, F of a product of slices (diagonal, exp(-dtau K)), the first one innermost."""
    n, dt = len(slices[0][0]), slices[0][0].dtype
    u, d, f = np.eye(n, dtype=dt), np.ones(n, dt), np.eye(n, dtype=dt)
    for a in range(0, len(slices), pace):
        c = u * d
        for e, k in slices[a:a + pace]:
            c = k @ (e[:, None] * c) if transposed else e[:, None] * (k @ c)
        u, r, perm = _pivoted_qr(c)
        d = abs(np.diag(r))
        f = (np.triu(r) / d[:, None]) @ f[perm]
    return u, d, f


def _solve(m, y):
    m, y = m.copy(), y.copy()
    for k in range(len(m)):
        v, tau, _ = _householder(m[k:, k])
        m[k:, k:] -= tau * np.outer(v, v @ m[k:, k:])
        y[k:] -= tau * np.outer(v, v @ y[k:])
    for k in range(len(m) - 1, -1, -1):
        y[k] = (y[k] - m[k, k + 1:] @ y[k + 1:]) / m[k, k]
    return y


def _green(fields, l, spin, U, beta, pace, expk):
    """G after slice l, 0 < l < Lt (the stabilized form that both stacks give)."""
    dt, Lt = expk.dtype.type, len(fields)
    alpha = np.arccosh(np.exp(dt(0.5) * dt(beta / Lt) * dt(U))) * (1 - 2 * spin)
    s = [(np.exp(alpha * f.astype(dt)), expk) for f in fields]
    ul, dl, fl = _stack(s[:l], False, pace)
    ur, dr, fr = _stack(s[:l - 1:-1], True, pace)
    m = (ul.T @ ur) / np.maximum(dl, 1)[:, None] / np.maximum(dr, 1)
    m += np.minimum(dl, 1)[:, None] * (fl @ fr.T) * np.minimum(dr, 1)
    return (ur / np.maximum(dr, 1)) @ _solve(m, ul.T / np.maximum(dl, 1)[:, None])


@pytest.mark.parametrize("L,U,beta,walkers,levels", [(8, 6.0, 6.0, 2, (2, 3)), (10, 6.0, 6.0, 2, (2, 3))])
def test_assembled_green_is_as_accurate_as_a_pivoted_stack(dq, L, U, beta, walkers, levels):  # noqa: F811
    Lt, pace = 60, 10
    w_, v_ = np.linalg.eigh(_kinetic(L))
    expk = (v_ * np.exp(-beta / Lt * w_)) @ v_.T
    b = dq.Batch([dq.WalkerDesc(model=0, L=L, U=U, beta=beta, Lt=Lt, pace=pace, seed=700 + w) for w in range(walkers)],
                 trace=True, hbm=True)
    old = [np.where(np.random.default_rng(w).random((Lt, L * L)) < 0.5, 1, -1).astype(np.int8) for w in range(walkers)]
    for w in range(walkers):
        b.set_fields(w, old[w])
    b.init_greens()
    b.trace_clear()
    b.sweep_0_to_beta()
    device, plain = [], []
    for w in range(walkers):
        new, trace = b.fields(w), b.trace(w)
        for j in levels:
            l = (j + 1) * pace
            fields = np.vstack([new[:l], old[w][l:]])
            for spin in (0, 1):
                exact = _green(fields, l, spin, U, beta, pace, expk.astype(np.longdouble))
                scale = abs(exact).max()
                device.append(float(abs(trace[j, spin] - exact).max() / scale))
                plain.append(float(abs(_green(fields, l, spin, U, beta, pace, expk) - exact).max() / scale))
    b.close()
    gm = lambda x: float(np.exp(np.mean(np.log(x))))  # noqa: E731
    assert gm(device) <= 4 * gm(plain), (gm(device), gm(plain), device, plain)


@pytest.mark.parametrize("L,model", [(6, 0), (7, 1), (10, 0), (13, 1)])
def test_pivoted_qr_does_not_depend_on_its_cluster(dq, L, model):  # noqa: F811
    """The CTAs of a matrix follow from the number of matrices and the size (one to eight, columns
    ragged over warps and CTAs); a column's sums are one warp's, so G is the same to the bit."""
    out = []
    for n in (2, 16, 36, 80) if L < 13 else (2, 60):
        b = dq.Batch([dq.WalkerDesc(model=model, L=L, U=5.0, mu=-0.2 if model else 0.0, beta=2.0, Lt=10, pace=5,
                                    seed=40 + w) for w in range(n)], rng=dq.RNG_PHILOX, hbm=True)
        for w in range(n):
            b.fields_random(w)
        b.init_greens()
        b.sweep_0_to_beta()
        b.sweep_beta_to_0()
        out.append([b.fields(w) for w in (0, 1)] + [b.green(w, s) for w in (0, 1) for s in (0, 1)])
        assert b.status(0) == 0
        b.close()
    for o in out[1:]:
        for a, c in zip(out[0], o):
            np.testing.assert_array_equal(a, c)
