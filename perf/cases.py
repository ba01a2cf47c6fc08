"""The work that is timed on a GPU: what a DQMC program has the library do.

Each case is one call, or the few calls that belong together, through the Python binding or
the C-ABI.  A simulation spends its life in forth-and-back pairs of half-sweeps with equal-time
measurements ("pair"); it bins them ("bins"), measures time-displaced functions ("dynamic"),
and starts from fields that it was given ("init").  "product" is the exact-slice matrix product
that the library offers on device buffers.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "dqmc-framework_gb300"))
import dqmc_gb300 as dq  # noqa: E402
from dqmc_gb300 import workloads  # noqa: E402


def _case(kind, walkers, model, L, beta, Lt, pace, precision, *, lattice="square", U=4.0, mu=0.0, cb=False,
          hbm=False, rng="philox"):
    return {"kind": kind, "walkers": walkers, "model": model, "lattice": lattice, "L": L, "U": U, "mu": mu,
            "beta": beta, "Lt": Lt, "pace": pace, "cb": cb, "precision": precision, "hbm": hbm, "rng": rng}


def listed():
    rep, att = "repulsive", "attractive"
    c = {
        # one chain with the reference's random stream, its default way to run: latency of one CTA
        "single_4x4": _case("pair", 1, rep, 4, 4.0, 80, 10, "fp64", rng="minstd"),
        # the throughput batch of the plain method: checkerboard walkers that live in shared memory
        "chains_8x8_checkerboard": _case("pair", 256, rep, 8, 8.0, 160, 10, "fp64", cb=True),
        # a short production loop with binning on the device, chains of a small lattice
        "bins_6x6": dict(_case("bins", 64, rep, 6, 4.0, 40, 10, "fp64"), nbins=2, bin_size=2, between=2),
        # the plain method just above the shared-memory limit, an odd side
        "fp64_9x9": _case("pair", 32, rep, 9, 2.0, 20, 10, "fp64"),
        # the plain method on the lattice of the large batches, few walkers
        "fp64_16x16": _case("pair", 16, att, 16, 1.6, 8, 8, "fp64", mu=-0.5),
        # the large production batch on the tensor cores, the benchmark's default
        "mixed_16x16": _case("pair", 128, att, 16, 10.0, 100, 8, "mixed", mu=-0.5),
        # the same lattice with both spins and few walkers: latency of the tensor-core path
        "mixed_16x16_few": _case("pair", 6, rep, 16, 2.0, 20, 10, "mixed"),
        # chains of different sides, U and beta in one batch (a parameter scan)
        "mixed_uneven": {"kind": "uneven", "per_side": 16, "precision": "mixed"},
        # a cubic lattice on the tensor cores
        "mixed_cubic_6": _case("pair", 24, rep, 6, 2.0, 20, 5, "mixed", lattice="cubic"),
        # time-displaced measurement and the updating sweep back, the largest lattice of the benchmark
        "dynamic_24x24": dict(_case("dynamic", 8, rep, 24, 1.2, 12, 6, "mixed"), stride=3),
        # a warm start: fields handed in, stacks and G built
        "init_12x12": _case("init", 48, rep, 12, 4.0, 40, 10, "mixed"),
        # one product on the caller's device buffers
        "product_256": {"kind": "product", "n": 256},
    }
    return [dict(v, name=k) for k, v in c.items()]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _sites(c):
    return c["L"] ** (3 if c["lattice"] == "cubic" else 2)


def draw(rng):
    kind = rng.choice(["small", "small", "hbm", "mixed", "mixed", "mixed", "dynamic", "init", "bins", "product", "uneven"])
    if kind == "product":
        return {"kind": "product", "n": _log_int(rng, 8, 256)}
    if kind == "uneven":
        return {"kind": "uneven", "per_side": rng.randint(3, 15), "precision": "mixed"}
    model = rng.choice(["repulsive", "attractive"])
    mu = round(rng.uniform(-0.8, 0.0), 2) if model == "attractive" else 0.0
    U = round(rng.uniform(2.0, 6.0), 2)
    pace = rng.randint(5, 10)
    dtau = rng.choice([0.05, 0.1])
    if kind in ("small", "bins"):
        L = rng.randint(2, 8)
        Lt = _log_int(rng, 10, 160 if kind == "small" else 40)
        c = _case("pair" if kind == "small" else "bins", _log_int(rng, 1, 256), model, L, round(Lt * dtau / 2, 3), Lt, pace, "fp64",
                  U=U, mu=mu, cb=(L % 2 == 0 and L > 2 and rng.random() < 0.5), rng=rng.choice(["philox", "minstd"]))
        return c if kind == "small" else dict(c, nbins=rng.randint(1, 3), bin_size=2, between=2 * rng.randint(0, 1))
    lattice, L = "square", rng.randint(9, 16)
    if kind == "hbm":
        Lt = _log_int(rng, 5, 20 if L <= 12 else 8)
        return _case("pair", _log_int(rng, 1, 16), model, L, round(Lt * dtau, 3), Lt, pace, "fp64", U=U, mu=mu,
                     cb=(L % 2 == 0 and rng.random() < 0.4))
    if kind == "init":
        Lt = _log_int(rng, 10, 40)
        return _case("init", _log_int(rng, 1, 48), model, L, round(Lt * dtau, 3), Lt, pace, "mixed", U=U, mu=mu)
    if rng.random() < 0.25:
        lattice, L = "cubic", rng.randint(4, 7)
    else:
        L = rng.randint(6, 24)
    n = L ** (3 if lattice == "cubic" else 2)
    Lt = _log_int(rng, 10, 100 if n <= 100 else 40 if n <= 256 else 12)
    if kind == "dynamic":
        Lt = min(Lt, 12)
    pace = min(pace, Lt)
    walkers = max(1, min(_log_int(rng, 1, 128), int(128 * 100 * 256.0 ** 2 / (6 * Lt * float(n) ** 2))))
    if kind == "dynamic":
        walkers = min(walkers, 8)
    c = _case("pair" if kind == "mixed" else "dynamic", walkers, model, L, round(Lt * dtau, 3), Lt, pace, "mixed",
              lattice=lattice, U=U, mu=mu,
              cb=(lattice == "square" and L % 2 == 0 and rng.random() < 0.15))
    return c if kind == "mixed" else dict(c, stride=rng.randint(1, 4))


def _descs(case, seed):
    if case["kind"] == "uneven":
        return workloads.uneven_batch(dq, per_size=case["per_side"], seed0=100000 + 1000 * (seed % 100000))
    return [dq.WalkerDesc(model=dq.REPULSIVE if case["model"] == "repulsive" else dq.ATTRACTIVE, L=case["L"],
                          U=case["U"], mu=case["mu"], beta=case["beta"], Lt=case["Lt"], pace=case["pace"],
                          checkerboard=case["cb"], seed=1 + (1009 * seed + w) % 2000000000,
                          lattice=dq.CUBIC if case["lattice"] == "cubic" else dq.SQUARE)
            for w in range(case["walkers"])]


def _fields(descs, seed):
    """Random starting fields, as a cold start has them."""
    r = np.random.default_rng(seed)
    return [(2 * r.integers(0, 2, size=(d.Lt, d.N), dtype=np.int8) - 1).astype(np.int8) for d in descs]


def _product_inputs(case, seed):
    """Entries of a Green's function's range: order 1 with rows of different scale."""
    n = case["n"]
    g = np.random.default_rng(seed)
    a = g.standard_normal((n, n)) * np.exp(g.uniform(-3, 3, size=(n, 1)))
    return np.asfortranarray(a), np.asfortranarray(g.standard_normal((n, n)))


def _taus(case):
    return list(range(0, case["Lt"], case["stride"]))


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    if case["kind"] == "product":
        a, b = _product_inputs(case, seed)
        # column-major on the device: the transposed array's C order
        s.a, s.b = (torch.from_numpy(np.ascontiguousarray(x.T)).cuda() for x in (a, b))
        s.c = torch.empty_like(s.a)
        return s
    d = _descs(case, seed)
    s.descs, s.fields = d, _fields(d, seed)
    s.batch = dq.Batch(d, rng=dq.RNG_MINSTD if case.get("rng") == "minstd" else dq.RNG_PHILOX,
                       precision=dq.MIXED if case["precision"] == "mixed" else dq.FP64, hbm=case.get("hbm", False))
    for w, f in enumerate(s.fields):
        s.batch.set_fields(w, f)
    s.batch.init_greens()
    return s


def _spins(d):
    return 1 if d.model == dq.ATTRACTIVE else 2  # the attractive model's two G are equal


def _greens(s):
    """G of every walker and spin, one flat array (walkers of a batch may differ in size)."""
    return np.concatenate([s.batch.green(w, sp).ravel(order="F")
                           for w, d in enumerate(s.descs) for sp in range(_spins(d))])


def _new_fields(s):
    return np.concatenate([s.batch.fields(w).ravel() for w in range(len(s.descs))])


def _bin(batch):
    """One bin per walker, as MeasureHandler normalises it (the sign's own scale divided out)."""
    sums, counts = batch.observables_all()
    return np.array([dq.write_bin(a, n) for a, n in zip(sums, counts)])


def run(s):
    case = s.case
    if case["kind"] == "product":
        st = torch.cuda.current_stream().cuda_stream
        rc = dq.load().dqmc_product_device_noalloc(case["n"], s.a.data_ptr(), s.b.data_ptr(), s.c.data_ptr(),
                                                   ctypes.c_void_p(st))
        if rc:
            raise RuntimeError(dq.load().dqmc_last_error().decode())
        return s.c
    b = s.batch
    if case["kind"] == "init":
        for w, f in enumerate(s.fields):
            b.set_fields(w, f)
        b.init_greens()
        return {"green": _greens(s)}
    if case["kind"] == "bins":
        bins = b.measure_bins(case["nbins"], case["bin_size"], case["between"])
        return {"bins": bins, "fields": _new_fields(s), "green": _greens(s)}
    if case["kind"] == "dynamic":
        b.clear_observables()
        b.clear_dynamic()
        b.sweep_dynamic(_taus(case))
        n = range(len(s.descs))
        sign = np.array([b.config_sign(w) for w in n])
        gk = np.array([b.dynamic(w)[0] for w in n]) * sign[:, None]
        obs = np.array([b.dynamic_obs(w) for w in n]) * sign[:, None, None]
        gr = np.array([b.dynamic_r(w) for w in n]) * sign[:, None, None]
        b.sweep_beta_to_0(measure=True)
        return {"gk": gk, "dos": obs[:, 0], "chi": obs[:, 1], "rho": obs[:, 2], "gr": gr, "bins": _bin(b),
                "fields": _new_fields(s), "green": _greens(s)}
    b.clear_observables()
    b.sweep_0_to_beta(measure=True)
    b.sweep_beta_to_0(measure=True)
    return {"bins": _bin(b), "fields": _new_fields(s), "green": _greens(s)}


def _half_sweeps(case):
    """(updating half-sweeps, dynamic half-sweeps) of one pass."""
    if case["kind"] == "bins":
        return 2 * case["nbins"] * (case["bin_size"] // 2 + case["between"] // 2), 0
    return (1, 1) if case["kind"] == "dynamic" else (0, 0) if case["kind"] == "init" else (2, 0)


def work(case):
    """Per walker and spin: a wrap is two N x N products and a step of the B-chain one (34 N^2 and 17 N^2
    with checkerboard factors), half of the N flips of a slice cost 2 N^2 each, a stabilization is a
    factorization with its factors (4 N^3) and the assembly of G (8 N^3); the time-displaced functions add
    two products a slice and 4 N^3 a stabilization.  Bytes: fields, G and the stacks' levels, in and out once."""
    if case["kind"] == "product":
        return {"bytes": 3 * 8 * case["n"] ** 2, "flops": 2 * case["n"] ** 3}
    up, dyn = _half_sweeps(case)
    flops = bytes_ = 0.0
    for d in _descs(case, 0):
        n, S = float(d.N), _spins(d)
        ns = -(-d.Lt // d.pace)
        chain = 17 * n * n if d.checkerboard else 2 * n ** 3
        per_slice = 3 * chain
        flops += S * up * (d.Lt * (per_slice + 0.5 * n * 2 * n * n) + ns * 12 * n ** 3)
        flops += S * dyn * (d.Lt * (per_slice + 2 * chain) + ns * 16 * n ** 3)
        if case["kind"] == "init":
            flops += S * (d.Lt * chain + ns * 4 * n ** 3 + 8 * n ** 3)
        bytes_ += (up + dyn) * (2 * d.Lt * d.N + S * 8 * n * n * (2 + 2 * 2 * ns)) + (S * 8 * n * n * (1 + 2 * ns) + d.Lt * d.N)
    return {"bytes": bytes_, "flops": flops}


# ---------------------------------------------------------------------------------------------
# The same results in 64 bits by plain torch: dense or plaquette factors multiplied out, QR stacks,
# one rank-1 update per accepted flip.  All walkers of a batch at once (they have one shape).
# ---------------------------------------------------------------------------------------------
def _philox(seeds, walkers, sweep, attempts):
    """Philox4x32-10 (Salmon et al., SC'11), 53 bits of (counter = attempt, sweep, walker; key = seed)."""
    m = np.uint64(0xFFFFFFFF)
    c = [np.broadcast_to(attempts.astype(np.uint64)[None, :], (len(seeds), len(attempts))),
         np.uint64(sweep & 0xFFFFFFFF), np.uint64(sweep >> 32), np.asarray(walkers, dtype=np.uint64)[:, None]]
    k0, k1 = (np.asarray(seeds, dtype=np.uint64)[:, None] >> np.uint64(s) & m for s in (0, 32))
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ k0, p1 & m, (p0 >> np.uint64(32)) ^ c[3] ^ k1, p0 & m]
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & m, (k1 + np.uint64(0xBB67AE85)) & m
    bits = ((c[0] >> np.uint64(5)) << np.uint64(26)) | (c[1] >> np.uint64(6))
    return bits.astype(np.float64) * 2.0 ** -53


class _Minstd:
    """minstd_rand0, two draws to a 53-bit uniform (std::generate_canonical)."""

    def __init__(self, seeds):
        self.x = np.array([s % 2147483647 or 1 for s in seeds], dtype=np.int64)

    def _next(self):
        self.x = self.x * 16807 % 2147483647
        return (self.x - 1).astype(np.float64)

    def uniforms(self, n):
        out = np.empty((len(self.x), n))
        r = 2147483646.0
        for k in range(n):
            out[:, k] = (self._next() + self._next() * r) / (r * r)
        return np.minimum(out, np.nextafter(1.0, 0.0))


class _Exact:
    def __init__(self, case, descs, fields, seed):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        d = descs[0]
        self.d, self.W, self.N, self.Lt, self.pace = d, len(descs), d.N, d.Lt, d.pace
        self.dim = 3 if d.lattice == dq.CUBIC else 2
        self.att = d.model == dq.ATTRACTIVE
        self.S = 1 if self.att else 2
        self.seeds = [x.seed for x in descs]
        self.philox = case["rng"] != "minstd"
        self.minstd, self.sweep = _Minstd(self.seeds), 0
        dtau = d.beta / d.Lt
        self.alpha = math.acosh(math.exp(0.5 * dtau * abs(d.U)))
        self.s = torch.tensor(np.stack(fields), dtype=torch.float64, device=self.dev)  # [W][Lt][N]
        L, N = d.L, d.N
        i = np.arange(N)
        self.xyz = np.stack([i % L, (i // L) % L, i // (L * L)][: self.dim])
        self.nn = [self._site((self.xyz[a] + 1) % L, a) for a in range(self.dim)]
        if d.checkerboard:
            ch, sh = math.cosh(dtau * d.t), math.sinh(dtau * d.t)
            P = math.exp(0.5 * dtau * d.mu) * np.kron([[ch, sh], [sh, ch]], [[ch, sh], [sh, ch]])
            Q = math.exp(-0.5 * dtau * d.mu) * np.kron([[ch, -sh], [-sh, ch]], [[ch, -sh], [-sh, ch]])
            even, odd = self._layer(P, 0), self._layer(P, 1)
            K, Ki = even @ odd, self._layer(Q, 1) @ self._layer(Q, 0)
        else:
            T = np.zeros((N, N))
            for n_ in self.nn:
                np.add.at(T, (i, n_), -d.t)
                np.add.at(T, (n_, i), -d.t)
            w, v = np.linalg.eigh(T + d.mu * np.eye(N))
            K, Ki = (v * np.exp(-dtau * w)) @ v.T, (v * np.exp(dtau * w)) @ v.T
        self.K, self.Ki = self._t(K), self._t(Ki)
        self.eye = torch.eye(N, dtype=torch.float64, device=self.dev).expand(self.W, self.S, N, N)
        # transposed walk of a plaquette product: its factors in the order in which B^T takes them
        self.KT = self._t(self._layer(P, 1) @ self._layer(P, 0)) if d.checkerboard else self.K
        k = math.pi  # the last k star, (pi, pi) or (pi, pi, pi)
        disp = (self.xyz[:, None, :] - self.xyz[:, :, None]) % L  # [dim][i][j]: j - i
        self.ff = self._t(np.cos(-k * disp.sum(0)))
        self.disp = torch.tensor(sum(disp[a] * L ** a for a in range(self.dim)), device=self.dev)
        half = (L + 1) // 2
        first = [(a, b) for a in range(half, L + 1) for b in range(half, a + 1)]
        k1 = first[1][0] / L * 2 * math.pi - math.pi if len(first) > 1 else 0.0
        self.ffxy = self._t(np.cos(-disp[0] * k1) - np.cos(-disp[1] * k1))
        self.left, self.right = [], []
        self.clear()

    def _t(self, x):
        return torch.tensor(x, dtype=torch.float64, device=self.dev)

    def _site(self, moved, a):
        c = [x.copy() for x in self.xyz]
        c[a] = moved
        return sum(c[b] * self.d.L ** b for b in range(self.dim))

    def _layer(self, P, parity):
        L, m = self.d.L, np.eye(self.N)
        for x in range(parity, L, 2):
            for y in range(parity, L, 2):
                at = [(x + a) % L + L * ((y + b) % L) for b in (0, 1) for a in (0, 1)]
                m[at, :] = P @ m[at, :]
        return m

    def clear(self):
        self.acc = torch.zeros(self.W, 9, dtype=torch.float64, device=self.dev)
        self.cnt = 0

    def _v(self, t):
        """exp(alpha s) of slice t per walker, spin and site."""
        e = torch.exp(self.alpha * self.s[:, t - 1])
        return e[:, None] if self.att else torch.stack([e, 1 / e], 1)

    def B(self, t, m):
        return self._v(t)[..., None] * (self.K @ m)

    def BT(self, t, m):
        return self.KT @ (self._v(t)[..., None] * m)

    def wrap(self, t):  # G(t-1) -> G(t)
        self.G = (self.B(t, self.G) @ self.Ki) / self._v(t)[..., None, :]

    def unwrap(self, t):  # G(t) -> G(t-1)
        self.G = self.Ki @ ((self.G * self._v(t)[..., None, :]) @ self.K / self._v(t)[..., None])

    def push(self, stack, chain):
        if stack:
            U, D, F = stack[-1]
            chain = (chain @ U) * D[..., None, :]
        else:
            F = self.eye
        at = torch.argsort(torch.linalg.vector_norm(chain, dim=-2), dim=-1, descending=True)
        Q, R = torch.linalg.qr(torch.gather(chain, -1, at[..., None, :].expand_as(chain)))
        D = torch.diagonal(R, dim1=-2, dim2=-1).abs()
        F = (R / D[..., None]) @ torch.gather(F, -2, at[..., None].expand_as(F))
        stack.append((Q, D, F))

    def assemble(self, what="tt"):
        one = torch.ones(self.W, self.S, self.N, dtype=torch.float64, device=self.dev)
        UL, DL, FL = self.left[-1] if self.left else (self.eye, one, self.eye)
        UR, DR, FR = self.right[-1] if self.right else (self.eye, one, self.eye)
        lM, lm, rM, rm = DL.clamp(min=1.0), DL.clamp(max=1.0), DR.clamp(min=1.0), DR.clamp(max=1.0)
        M = (UL.mT @ UR) / lM[..., None] / rM[..., None, :] + lm[..., None] * (FL @ FR.mT) * rm[..., None, :]
        X = torch.linalg.solve(M, UL.mT / lM[..., None])
        G = (UR / rM[..., None, :]) @ X
        if what == "tt":
            return G
        X2 = torch.linalg.solve(M, lm[..., None] * FL)
        return G, (UR / rM[..., None, :]) @ X2, -(FR.mT * rm[..., None, :]) @ X

    def init(self):
        chain = self.eye
        for t in range(self.Lt, 0, -1):
            chain = self.BT(t, chain)
            if (t - 1) % self.pace == 0:
                self.push(self.right, chain)
                chain = self.eye
        self.G = self.assemble()

    def metropolis(self, t, u):
        a = self.alpha
        for i in range(self.N):
            s = self.s[:, t - 1, i]
            du = torch.exp(-2 * a * s) - 1
            D = du[:, None] if self.att else torch.stack([du, torch.exp(2 * a * s) - 1], 1)
            q = 1 + (1 - self.G[:, :, i, i]) * D
            r = torch.exp(2 * a * s) * q[:, 0] ** 2 if self.att else q[:, 0] * q[:, 1]
            ok = u[:, i] < r.abs().clamp(max=1.0)
            f = torch.where(ok[:, None], D / q, torch.zeros_like(q))
            col = self.G[:, :, :, i] * f[..., None]
            row = -self.G[:, :, i, :]
            row[..., i] += 1
            self.G -= col[..., None] * row[..., None, :]
            self.s[:, t - 1, i] = torch.where(ok, -s, s)

    def _draws(self, order):
        """Uniforms of one half-sweep, {slice: [W][N]}."""
        if not self.philox:
            u = self._t(self.minstd.uniforms(self.Lt * self.N))
            return {t: u[:, k * self.N:(k + 1) * self.N] for k, t in enumerate(order)}
        self.sweep += 1
        u = self._t(_philox(self.seeds, range(self.W), self.sweep, np.arange(self.Lt * self.N)))
        return {t: u[:, (t - 1) * self.N:t * self.N] for t in order}

    def measure(self, G):
        N, S = self.N, self.S
        up, dn = G[:, 0], G[:, S - 1]
        a, b = (torch.diagonal(g, dim1=-2, dim2=-1) for g in (up, dn))
        kin = sum((up[:, range(N), n_] + dn[:, range(N), n_]).sum(-1) for n_ in self.nn)
        eye = self.eye[0, 0]
        cu, cd, na, nb = eye - up.mT, eye - dn.mT, 1 - a, 1 - b
        same = na[:, :, None] * na[:, None, :] + cu * up + nb[:, :, None] * nb[:, None, :] + cd * dn
        cross = nb[:, :, None] * na[:, None, :] + na[:, :, None] * nb[:, None, :]
        self.acc += torch.stack([
            2 - (a + b).sum(-1) / N, (na * nb).sum(-1) / N, 2 * self.d.t * kin / N,
            1 - 0.5 * ((up + dn).mT * self.ff).sum((-1, -2)) / N, (a + b - 2 * a * b).sum(-1) / N,
            (self.ff * (same - cross)).sum((-1, -2)) / N ** 2, (self.ff * (same + cross)).sum((-1, -2)) / N ** 2,
            (cu * cd).sum((-1, -2)) / N, torch.ones(self.W, dtype=torch.float64, device=self.dev)], 1)
        self.cnt += 1

    def forth(self, measure=True):
        u, chain = self._draws(range(1, self.Lt + 1)), self.eye
        self.left = []
        for t in range(1, self.Lt + 1):
            self.wrap(t)
            self.metropolis(t, u[t])
            chain = self.B(t, chain)
            if t % self.pace == 0 or t == self.Lt:
                self.right.pop()
                self.push(self.left, chain)
                self.G, chain = self.assemble(), self.eye
            if measure:
                self.measure(self.G)

    def back(self, measure=True):
        u, chain = self._draws(range(self.Lt, 0, -1)), self.eye
        self.right = []
        for t in range(self.Lt, 0, -1):
            if t % self.pace == 0 and t != self.Lt:
                self.left.pop()
                self.push(self.right, chain)
                self.G, chain = self.assemble(), self.eye
            self.metropolis(t, u[t])
            if measure and t < self.Lt:
                self.measure(self.G)
            chain = self.BT(t, chain)
            self.unwrap(t)
        self.left.pop()
        self.push(self.right, chain)
        self.G = self.assemble()
        if measure:
            self.measure(self.G)

    def dynamic(self, taus):
        self.left, chain = [], self.eye
        gt0, g0t, seen = self.G, self.G - self.eye, {}
        for t in range(1, self.Lt + 1):
            self.wrap(t)
            gt0 = self.B(t, gt0)
            g0t = (g0t @ self.Ki) / self._v(t)[..., None, :]
            chain = self.B(t, chain)
            if t % self.pace == 0 or t == self.Lt:
                self.right.pop()
                self.push(self.left, chain)
                self.G, gt0, g0t = self.assemble("all")
                chain = self.eye
            if t in taus or t == self.Lt:
                seen[t % self.Lt] = self.G, gt0, g0t
        N, out = self.N, {"gk": [], "dos": [], "chi": [], "rho": [], "gr": []}
        g00 = seen[0][0]
        both = lambda f: f(0) + f(self.S - 1)  # noqa: E731
        diag = lambda g: torch.diagonal(g, dim1=-2, dim2=-1)  # noqa: E731
        px = torch.tensor(self.nn[0], device=self.dev)
        for tau in taus:
            gtt, t0, ot = seen[tau]
            g = gtt if tau == 0 else t0
            mean = 0.5 * both(lambda q: g[:, q]).mT / N  # [i][j]: G(j, i)
            out["gk"].append((mean * self.ff).sum((-1, -2)))
            out["gr"].append(torch.zeros(self.W, N, dtype=torch.float64, device=self.dev).index_add_(
                1, self.disp.reshape(-1), mean.reshape(self.W, -1)))
            out["dos"].append(0.5 * both(lambda q: diag(g[:, q]).sum(-1)) / N)
            ct, c0 = ([1 - diag(x[:, q]) for q in (0, self.S - 1)] for x in (gtt, g00))
            out["chi"].append(0.25 / N * ((ct[0] - ct[1]) * (c0[0] - c0[1])
                                          - both(lambda q: diag(ot[:, q]) * diag(t0[:, q]))).sum(-1))
            cur = lambda x: both(lambda q: x[:, q, range(N), px] - x[:, q, px, range(N)])  # noqa: E731
            con = both(lambda q: -ot[:, q][:, px][:, :, px] * t0[:, q].mT + ot[:, q][:, :, px] * t0[:, q][:, :, px].mT
                       + ot[:, q][:, px] * t0[:, q][:, px].mT - ot[:, q] * t0[:, q][:, px][:, :, px].mT)
            rho = (self.ffxy * (-cur(g00)[:, :, None] * cur(gtt)[:, None, :] + con)).sum((-1, -2))
            out["rho"].append(0.25 * self.d.t ** 2 / N ** 2 * (rho if self.dim == 2 else 0 * rho))
        return {k: torch.stack(v, 1) for k, v in out.items()}

    def bin(self):
        return self.acc / self.cnt

    def state(self):
        return {"fields": self.s.to(torch.int8).reshape(-1), "green": self.G.mT.reshape(-1)}


def _exact_seconds(case):
    """What the plain computation takes, about: one step a flip attempt, one QR a stabilization, walker and spin."""
    n, S = _sites(case), 1 if case["model"] == "attractive" else 2
    up, dyn = _half_sweeps(case)
    qrs = case["walkers"] * S * -(-case["Lt"] // case["pace"]) * (up + dyn + 1)
    flips = up * case["Lt"] * n * (2.5e-4 + case["walkers"] * S * n * n * 24 / 3e12)
    return flips + qrs * (3e-4 + 3e-3 * (n / 256) ** 2)


def exact(case, seed):
    if case["kind"] == "product":
        a, b = _product_inputs(case, seed)
        return torch.from_numpy(np.ascontiguousarray((a @ b).T))
    # walkers of several shapes, and runs of many steps: too long by plain means
    if case["kind"] == "uneven" or _exact_seconds(case) > 15:
        return None
    d = _descs(case, seed)
    x = _Exact(case, d, _fields(d, seed), seed)
    x.init()
    if case["kind"] == "init":
        return {"green": x.state()["green"]}
    if case["kind"] == "bins":
        bins = []
        for _ in range(case["nbins"]):
            x.clear()
            for _ in range(case["bin_size"] // 2):
                x.forth()
                x.back()
            bins.append(x.bin())
            for _ in range(case["between"] // 2):
                x.forth(False)
                x.back(False)
        return dict(x.state(), bins=torch.stack(bins, 1))
    if case["kind"] == "dynamic":
        out = x.dynamic(_taus(case))
        x.back()
        return dict(x.state(), bins=x.bin(), **out)
    x.forth()
    x.back()
    return dict(x.state(), bins=x.bin())
