"""Performance cases of the DQMC library: the calls that users make, with their inputs.

A case is a dict of plain values.  `listed()` gives the fixed cases, `draw(rng)`
one more of the same ranges, `prepare(case, seed)` what a program holds before
the call (chains with their field, initialised; streams and matrices),
`run(state)` one pass through the public API with its outputs, `work(case)` the
bytes and flops a pass cannot do without, and `exact(case, seed)` the outputs
in plain 64-bit numpy (None where that takes too long).

Kinds of work:
  update    one update() call (propagate + local updates of one slice) with its
            determinant ratios: the smallest step of a run, and the debugging call
  sweep     n_calls update() calls from pre-generated streams in host memory,
            then G and the field, as a run does between two measurements
  batch     the same on independent chains of uneven L sharing the GPU, streams
            in device memory
  greens    from-scratch G and log|det G| of one slice (validation, restarts)
  gradient  log-weight and its reverse rule: a Langevin or HMC step
  tdgf      time-displaced Green's functions of all slices
  measure   the measurement hook and the equal-time correlators
  udt       the pivoted UDT decomposition of one matrix

Precisions: "fp64" (immediate rank-4 updates by default, or delayed with
`delay` = k) and "mixed" (split-BF16 products, delayed updates).  Lattices L in
4..16, so n = 4 L^2 is 64..1024, mostly not a multiple of a tile.  The model is
that of the library's tests and benchmark: lambda = r = c = u = 1,
mu = -0.5, dtau = 0.1, box 0.2, fields i.i.d. uniform in [-1, 1].
"""
import numpy as np
import torch

from dqmc_gb300 import api

DTAU, LAM, MU, BOX = 0.1, 1.0, -0.5, 0.2
TX, TY = (1.0, -0.5), (0.5, -1.0)   # horizontal and vertical hopping of bands x, y
SIZES = (4, 6, 8, 10, 12, 14, 16)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # smallest lattice of the test suite, one call: latency and launches
        dict(name="update L4 fp64", kind="update", L=4, slices=40, safe_mult=10, precision="fp64", delay=0),
        # the same lattice, one full pass over its 40 slices (beta = 4)
        dict(name="sweep L4 fp64", kind="sweep", L=4, slices=40, safe_mult=10, precision="fp64", delay=0, calls=40),
        # a production lattice of moderate size in the mixed form (beta = 8)
        dict(name="sweep L8 mixed", kind="sweep", L=8, slices=80, safe_mult=10, precision="mixed", delay=16,
             calls=80),
        # the plain FP64 workload with delayed rank-4 updates, k = 16 (beta = 10); n = 400 is no multiple of a tile
        dict(name="sweep L10 fp64 delayed", kind="sweep", L=10, slices=100, safe_mult=10, precision="fp64", delay=16,
             calls=100),
        # the headline lattice in the default form (FP64, immediate updates): two stabilisation intervals
        dict(name="sweep L16 fp64", kind="sweep", L=16, slices=200, safe_mult=10, precision="fp64", delay=0,
             calls=20),
        # the headline workload: one full pass of the mixed form (beta = 20)
        dict(name="sweep L16 mixed", kind="sweep", L=16, slices=200, safe_mult=10, precision="mixed", delay=16,
             calls=200),
        # independent chains of uneven L on one GPU (beta = 8)
        dict(name="batch 16 chains mixed", kind="batch", chains=16, slices=80, safe_mult=10, precision="mixed",
             delay=16, calls=80),
        # validation: G of one slice from scratch
        dict(name="greens L6 fp64", kind="greens", L=6, slices=40, safe_mult=10, precision="fp64", delay=0, slice=17),
        # forward and reverse rule of the log-weight on the adjoint-force workload (beta = 10)
        dict(name="gradient L12 fp64", kind="gradient", L=12, slices=100, safe_mult=10, precision="fp64", delay=0),
        # time-displaced measurement
        dict(name="tdgf L6 mixed", kind="tdgf", L=6, slices=40, safe_mult=10, precision="mixed", delay=16),
        # measurement hook and equal-time correlators
        dict(name="measure L8 fp64", kind="measure", L=8, slices=80, safe_mult=10, precision="fp64", delay=0),
        # one pivoted UDT decomposition, ragged size n = 784
        dict(name="udt L14 fp64", kind="udt", L=14, slices=10, safe_mult=10, precision="fp64", delay=0),
    ]


def draw(rng):
    kind = rng.choice(["sweep"] * 5 + ["update", "batch", "greens", "gradient", "tdgf", "measure", "udt"])
    s = rng.choice([5, 8, 10])
    prec = rng.choice(["fp64", "mixed"])
    delay = rng.choice([8, 16, 32]) if prec == "mixed" else rng.choice([0, 0, 8, 16])
    c = dict(kind=kind, slices=s * rng.randint(2, 20), safe_mult=s, precision=prec, delay=delay)
    if kind == "batch":
        c.update(chains=rng.randint(3, 16), slices=s * rng.randint(2, 8), precision="mixed",
                 delay=rng.choice([8, 16, 32]))
        c["calls"] = rng.randint(s, c["slices"])
        return c
    if kind == "gradient":
        c["L"] = rng.choice([4, 6, 8, 10, 12])
        c["slices"] = s * rng.randint(2, 10)
    elif kind == "tdgf":
        c["L"] = rng.choice([4, 6, 8, 10])
        c["slices"] = 2 * s * rng.randint(1, 3)
    else:
        c["L"] = rng.choice(SIZES)
    if kind == "udt":
        c["slices"] = s
    if kind == "greens":
        c["slice"] = rng.randint(1, c["slices"])
        c["slices"] = min(c["slices"], 10 * s) if c["L"] > 12 else c["slices"]
        c["slice"] = min(c["slice"], c["slices"])
    if kind == "sweep":
        # a pass of the largest lattices stays below the largest listed one
        n = 4 * c["L"] ** 2
        most = 200 if n <= 600 else (120 if prec == "mixed" else 30)
        c["calls"] = rng.randint(min(s, 8), min(most, c["slices"]))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _params(case, L):
    return api.ModelParams(L=L, slices=case["slices"], safe_mult=case["safe_mult"], delta_tau=DTAU, lambda_=LAM,
                           r=1.0, c=1.0, u=1.0, mu1=MU, mu2=MU, hoppings=(TX[0], TY[0], TX[1], TY[1]), box=BOX,
                           precision=case["precision"], delay=case["delay"])


def _field(rng, N, M):
    return rng.uniform(-1.0, 1.0, size=(3, N, M))


def _streams(rng, N, calls):
    return rng.uniform(-BOX, BOX, size=(calls, 3, N)), rng.uniform(size=(calls, N))


def _matrix(rng, n):
    """A column-graded matrix, as a chain of slices times U D hands to the UDT decomposition."""
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    return a * np.logspace(5.0, -5.0, n)[rng.permutation(n)][None, :]


def _lattices(case):
    """L of each chain of a batch: cycled over 6, 8, 10, 12."""
    return [(6, 8, 10, 12)[i % 4] for i in range(case["chains"])]


def _inputs(case, seed):
    """Everything drawn from the seed: fields and streams of each chain, or the matrix."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "batch":
        return [(_field(rng, L * L, case["slices"]), *_streams(rng, L * L, case["calls"])) for L in _lattices(case)]
    L = case["L"]
    phi = _field(rng, L * L, case["slices"])
    if kind == "update":
        return phi, *_streams(rng, L * L, 1)
    if kind == "sweep":
        return phi, *_streams(rng, L * L, case["calls"])
    if kind == "udt":
        return phi, _matrix(rng, 4 * L * L)
    return (phi,)


def prepare(case, seed):
    inp = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batch":
        ps = [_params(case, L) for L in _lattices(case)]
        b = api.Batch(ps, [x[0] for x in inp])
        b.init()
        # per call the (3, N) block of a stream is component fastest
        d = [torch.from_numpy(np.ascontiguousarray(x[1].transpose(0, 2, 1))).cuda() for x in inp]
        u = [torch.from_numpy(x[2]).cuda() for x in inp]
        return dict(case=case, batch=b, delta=d, unif=u)
    chain = api.DQMC(_params(case, case["L"]), inp[0])
    if kind != "udt":
        chain.init()
    return dict(case=case, chain=chain, inputs=inp)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        b = state["batch"]
        st = b.sweep_device(case["calls"], [x.data_ptr() for x in state["delta"]],
                            [x.data_ptr() for x in state["unif"]])
        return dict(accepted=np.array([s["accepted"] for s in st]), greens=[c.greens for c in b.chains],
                    field=[c.get_field() for c in b.chains])
    c, inp = state["chain"], state["inputs"]
    if kind == "update":
        rate, acc, det, pacc = c.update(inp[1][0], inp[2][0], return_details=True)
        return dict(accepted=acc, rate=rate, detratio=det, p_acc=pacc)
    if kind == "sweep":
        res = c.sweep(case["calls"], inp[1], inp[2], return_accepted=True)
        return dict(accepted=res["accepted_mask"], count=res["accepted"], greens=c.greens, field=c.get_field())
    if kind == "greens":
        G, ld = c.calc_greens_and_logdet(case["slice"])
        return dict(greens=G, logdet=ld)
    if kind == "gradient":
        y, pullback = c.rrule_log_weight(inp[0])
        return dict(log_weight=y, gradient=pullback(1.0))
    if kind == "tdgf":
        gt0, g0t = c.measure_tdgfs()
        return dict(gt0=gt0, g0t=g0t)
    if kind == "measure":
        m = c.measure()
        etpc_p, etpc_m, etcdc_p, etcdc_m = c.measure_equal_time()
        return dict(greens=m["greens"], occupation=m["occupation"], e_kin=m["e_kin"], etpc_plus=etpc_p,
                    etpc_minus=etpc_m, etcdc_plus=etcdc_p, etcdc_minus=etcdc_m)
    U, D, T = c.decompose_udt(inp[1])
    return dict(U=U, D=D, T=T)


def work(case):
    """Bytes: the pass's inputs and outputs once (a sweep's G is read and
    written once per call).  Flops: real FP64 flops of the method (checkerboard
    slices 74 n^2, rank-4 updates 32 n^2 at the typical acceptance 0.6, pivoted
    QR 16/3 n^3 and its Q 16/3 n^3, one LU 8/3 n^3, products 8 n^3, two
    triangular solves 4 n^3 each)."""
    M, s = case["slices"], case["safe_mult"]

    def per(n):
        udt = 32.0 / 3.0 * n ** 3 + s * 74.0 * n ** 2
        greens = 24.0 * n ** 3 + 8.0 / 3.0 * n ** 3 + 8.0 * n ** 3
        return udt, greens

    def sweep(n, calls):
        udt, greens = per(n)
        N = n // 4
        return (calls * (148.0 * n ** 2 + 0.6 * N * 32.0 * n ** 2) + calls / s * (udt + 8.0 * n ** 3 + greens),
                calls * (32.0 * n ** 2 + 33.0 * N) + 16.0 * n ** 2)
    kind = case["kind"]
    if kind == "batch":
        w = [sweep(4 * L * L, case["calls"]) for L in _lattices(case)]
        return dict(flops=sum(x[0] for x in w), bytes=sum(x[1] for x in w))
    n = 4 * case["L"] ** 2
    udt, greens = per(n)
    if kind == "update":
        fl, by = sweep(n, 1)
    elif kind == "sweep":
        fl, by = sweep(n, case["calls"])
    elif kind == "greens":
        fl, by = M / s * (udt + 8.0 * n ** 3) + greens, 24.0 * n // 4 * M + 16.0 * n ** 2
    elif kind == "gradient":
        fl, by = 2 * M / s * (udt + 8.0 * n ** 3) + M / s * greens + M * 148.0 * n ** 2, 48.0 * n // 4 * M
    elif kind == "tdgf":
        fl, by = M / s * (4 * (udt + 8.0 * n ** 3) + 2 * (2 * udt + greens)) + 2 * M * 74.0 * n ** 2, 32.0 * M * n ** 2
    elif kind == "measure":
        fl, by = (148.0 + 64.0) * n ** 2 + 40.0 * 6 * n ** 2 / 16, 32.0 * n ** 2
    else:
        fl, by = 32.0 / 3.0 * n ** 3, 64.0 * n ** 2
    return dict(flops=float(fl), bytes=float(by))


# ---------------------------------------------------------------------------
# the same in plain numpy
# ---------------------------------------------------------------------------
class _Model:
    """The O(3) model on an L x L lattice in numpy: slice matrices, G from
    scratch by column-sorted QR chains, local updates."""

    def __init__(self, L, M, s, phi):
        self.L, self.N, self.n, self.M, self.s = L, L * L, 4 * L * L, M, s
        self.phi = np.array(phi)
        self.H, self.Hinv, self.E, self.Einv = [], [], [], []
        for b in range(2):
            hb, ha = self._layer(b, 1, 0.5), self._layer(b, 0, 1.0)
            hbi, hai = self._layer(b, 1, -0.5), self._layer(b, 0, -1.0)
            mu = np.exp(DTAU * MU)
            self.H.append(hb @ ha @ hb * mu)
            self.Hinv.append(hbi @ hai @ hbi / mu)
            # effective -> true transformation
            self.E.append(hb @ self._layer(b, 0, 0.5))
            self.Einv.append(self._layer(b, 0, -0.5) @ hbi)

    def _layer(self, b, group, pre):
        """exp(-pre dtau T) of one plaquette group of band b (N x N)."""
        L, N = self.L, self.N
        h, v = pre * DTAU * TX[b], pre * DTAU * TY[b]
        ch, sh, cv, sv = np.cosh(h), np.sinh(h), np.cosh(v), np.sinh(v)
        X = np.eye(N)
        for x in range(group, L, 2):
            for y in range(group, L, 2):
                x1, y1 = (x + 1) % L, (y + 1) % L
                q = [y + L * x, y1 + L * x, y + L * x1, y1 + L * x1]
                P = np.kron(np.array([[ch, sh], [sh, ch]]), np.array([[cv, sv], [sv, cv]]))
                X[q] = P @ X[q]
        return X

    def ev(self, l, power):
        """(N, 4, 4) interaction blocks exp(-power dtau V) of slice l (0-based)."""
        p = self.phi[:, :, l]
        nrm = np.sqrt((p * p).sum(0))
        sh = power * np.sinh(LAM * DTAU * nrm) / nrm
        return self._blocks(np.cosh(LAM * DTAU * nrm), (1j * p[1] - p[0]) * sh, -p[2] * sh)

    @staticmethod
    def _blocks(C, S, R):
        z = np.zeros(C.shape + (4, 4), dtype=complex)
        for i in range(4):
            z[..., i, i] = C
        z[..., 0, 1] = z[..., 3, 2] = S
        z[..., 1, 0] = z[..., 2, 3] = np.conj(S)
        z[..., 0, 3] = z[..., 3, 0] = R
        z[..., 1, 2] = z[..., 2, 1] = -R
        return z

    def _hop(self, mats, A):
        N = self.N
        return np.concatenate([mats[f & 1] @ A[f * N:(f + 1) * N] for f in range(4)])

    def _site(self, z, A):
        B = A.reshape(4, self.N, -1)
        return np.matmul(z, B.transpose(1, 0, 2)).transpose(1, 0, 2).reshape(A.shape)

    def left(self, l, A):          # B_l A
        return self._hop(self.H, self._site(self.ev(l, 1.0), A))

    def left_inv(self, l, A):
        return self._site(self.ev(l, -1.0), self._hop(self.Hinv, A))

    def left_dag(self, l, A):      # B_l^dag A (hops symmetric, blocks Hermitian)
        return self._site(self.ev(l, 1.0), self._hop([h.T for h in self.H], A))

    def right(self, l, A):         # A B_l
        return self.left_dag(l, A.conj().T).conj().T

    def right_inv(self, l, A):
        e = self.ev(l, -1.0)
        return self._hop([h.T for h in self.Hinv], self._site(e, A.conj().T)).conj().T

    @staticmethod
    def udt(A, T0):
        """A T0 = U diag(D) T by QR with the columns sorted by norm."""
        order = np.argsort(-np.linalg.norm(A, axis=0), kind="stable")
        Q, R = np.linalg.qr(A[:, order])
        D = np.abs(np.diag(R))
        T = np.empty_like(A)
        T[:, order] = R / D[:, None]
        return Q, D, T if T0 is None else T @ T0

    def chain(self, slices, step):
        """UDT of step(l_k) ... step(l_1), re-decomposed every s slices."""
        U, D, T = np.eye(self.n, dtype=complex), np.ones(self.n), None
        out = []
        for k, l in enumerate(slices):
            U = step(l, U)
            if (k + 1) % self.s == 0 or k == len(slices) - 1:
                U, D1, T = self.udt(U * D[None, :], T)
                D = D1
                out.append((U, D, T))
        return out

    def from_udts(self, left, right):
        """[1 + Ul Dl Tl (Ur Dr Tr)^dag]^-1 and log|det| of it."""
        n = self.n
        one = (np.eye(n, dtype=complex), np.ones(n), np.eye(n, dtype=complex))
        Ul, Dl, Tl = left or one
        Ur, Dr, Tr = right or one
        lp, lm, rp, rm = np.maximum(Dl, 1), np.minimum(Dl, 1), np.maximum(Dr, 1), np.minimum(Dr, 1)
        X = (Ul.conj().T @ Ur) / lp[:, None] / rp[None, :] + lm[:, None] * (Tl @ Tr.conj().T) * rm[None, :]
        G = (Ur / rp[None, :]) @ np.linalg.solve(X, Ul.conj().T / lp[:, None])
        return G, -(np.linalg.slogdet(X)[1] + np.log(lp).sum() + np.log(rp).sum())

    def greens(self, slice1):
        """[1 + B(slice-1) ... B(1) B(M) ... B(slice)]^-1 and log|det G|."""
        left = self.chain(range(slice1 - 1), self.left) if slice1 > 1 else None
        right = self.chain(range(self.M - 1, slice1 - 2, -1), self.left_dag)
        return self.from_udts(left[-1] if left else None, right[-1])

    def true(self, G):
        """Effective to true G: E^-1 G E with the half hopping layers."""
        A = self._hop(self.Einv, G)
        return self._hop([e.T for e in self.E], A.conj().T).conj().T

    def action(self):
        h = self.phi.reshape((3, self.L, self.L, self.M), order="F")
        d = [h - np.roll(h, -1, axis=a) for a in (1, 2, 3)]
        sq = (self.phi ** 2).sum(0)
        return 0.5 / DTAU * (d[2] ** 2).sum() + 0.5 * DTAU * ((d[0] ** 2).sum() + (d[1] ** 2).sum()) + \
            DTAU * (0.5 * sq + 0.25 * sq * sq).sum()

    def action_gradient(self):
        h = self.phi.reshape((3, self.L, self.L, self.M), order="F")
        g = (2 * h - np.roll(h, -1, 3) - np.roll(h, 1, 3)) / DTAU
        g += DTAU * (4 * h - sum(np.roll(h, k, a) for a in (1, 2) for k in (1, -1)))
        g += DTAU * (1.0 + (h * h).sum(0)[None]) * h
        return g.reshape((3, self.N, self.M), order="F")

    def update_slice(self, G, l, delta, unif):
        """Metropolis visits of all sites of slice l (0-based) in order; G is
        taken through pending rank-4 factors that are applied every 16."""
        L, N, M, n, phi = self.L, self.N, self.M, self.n, self.phi
        acc, det, pac = np.zeros(N, bool), np.zeros(N, complex), np.zeros(N)
        X, Y = np.zeros((n, 0), complex), np.zeros((0, n), complex)
        for i in range(N):
            ix = i + N * np.arange(4)
            old = phi[:, i, l].copy()
            new = old + delta[:, i]
            d = new - old
            y, x = i % L, i // L
            nb = [(y + 1) % L + L * x, y + L * ((x + 1) % L), (y - 1) % L + L * x, y + L * ((x - 1) % L)]
            so, sn = old @ old, new @ new
            t = phi[:, i, (l + 1) % M] + phi[:, i, (l - 1) % M]
            dS = (sn - so - t @ d) / DTAU + 0.5 * DTAU * (4 * (sn - so) - 2 * phi[:, nb, l].sum(1) @ d) + \
                DTAU * (0.5 * (sn - so) + 0.25 * (sn * sn - so * so))
            z = []
            for v, pw in ((old, -1.0), (new, 1.0)):
                r = np.sqrt(v @ v)
                sh = pw * np.sinh(LAM * DTAU * r) / r
                z.append(self._blocks(np.cosh(LAM * DTAU * r), (1j * v[1] - v[0]) * sh, -v[2] * sh))
            D = z[0] @ z[1] - np.eye(4)
            Mx = np.eye(4) + D @ (np.eye(4) - G[np.ix_(ix, ix)] - X[ix] @ Y[:, ix])
            det[i] = np.linalg.det(Mx)
            pac[i] = np.exp(-dS) * det[i].real
            if pac[i] > 1.0 or unif[i] < pac[i]:
                acc[i] = True
                phi[:, i, l] = new
                a = G[:, ix] + X @ Y[:, ix]
                a[ix, np.arange(4)] -= 1.0
                b = np.linalg.solve(Mx, D) @ (G[ix] + X[ix] @ Y)
                X, Y = np.concatenate([X, a], 1), np.concatenate([Y, b], 0)
                if X.shape[1] == 64:
                    G, X, Y = G + X @ Y, X[:, :0], Y[:0]
        return G + X @ Y, acc, det, pac

    def sweep(self, calls, delta, unif):
        """update() calls from the state (slice M, down) that a fresh chain has."""
        l, down, G = self.M, True, None
        accs, dets, pacs = [], [], []
        for c in range(calls):
            if down and l == 1:
                down = False          # the turnaround visits the end slice twice
            elif not down and l == self.M:
                down = True
            else:
                if G is not None:
                    k = l - 2 if down else l - 1
                    G = self.right(k, self.left_inv(k, G)) if down else self.right_inv(k, self.left(k, G))
                l += -1 if down else 1
            if G is None or c % self.s == 0:
                G = self.greens(l)[0]
            G, a, d, p = self.update_slice(G, l - 1, delta[c], unif[c])
            accs.append(a), dets.append(d), pacs.append(p)
        return l, np.array(accs), np.array(dets), np.array(pacs)


def _equal_time(L, G):
    """Pairing and charge-density correlators of a true G, [y, x] by displacement."""
    N = L * L
    g = G.reshape(4, N, 4, N)
    y, x = np.arange(N) % L, np.arange(N) // L
    pp, pm = np.zeros((L, L)), np.zeros((L, L))
    cp, cm = np.zeros((L, L), complex), np.zeros((L, L), complex)
    r0 = np.arange(N)
    js = ((2, 0, 0, 2), (2, 0, 3, 1), (1, 3, 0, 2), (1, 3, 3, 1))
    for dx in range(L):
        for dy in range(L):
            ri = (y + dy) % L + L * ((x + dx) % L)
            e = [(g[a, ri, d, r0] * g[b, ri, c, r0] - g[a, ri, c, r0] * g[b, ri, d, r0]).real.sum()
                 for a, b, c, d in js]
            pp[dy, dx], pm[dy, dx] = (e[0] + e[1] + e[2] + e[3]) / N, (e[0] - e[1] - e[2] + e[3]) / N
            for a in range(4):
                for b in range(4):
                    t = ((1 - g[a, ri, a, ri]) * (1 - g[b, r0, b, r0]) +
                         (((ri == r0) & (a == b)) - g[b, r0, a, ri]) * g[a, ri, b, r0]).sum() / N
                    cp[dy, dx] += t
                    cm[dy, dx] += t if (a & 1) == (b & 1) else -t
    return pp, pm, cp, cm


def _gradient(m):
    """d log|det M| / d phi from G of every slice: G at the block ends from UDT
    chains, wrapped inside the blocks."""
    M, s, N = m.M, m.s, m.N
    lefts = [None] + m.chain(range(M), m.left)
    rights = [None] + m.chain(range(M - 1, -1, -1), m.left_dag)
    nb = M // s
    grad = np.zeros((3, N, M))
    logdet = 0.0
    for b in range(nb):
        # G at slice 1 + b s
        G, ld = m.from_udts(lefts[b], rights[nb - b])
        if b == 0:
            logdet = -ld
        for l in range(b * s, (b + 1) * s):
            blk = np.array([G[i::N, i::N] for i in range(N)])
            p = m.phi[:, :, l]
            nrm = np.sqrt((p * p).sum(0))
            x = LAM * DTAU * nrm
            sh, C = np.sinh(x) / nrm, np.cosh(x)
            dsh = (LAM * DTAU * C - sh) / nrm ** 2
            Einv = m.ev(l, -1.0)
            for a in range(3):
                dS = (1j * p[1] - p[0]) * dsh * p[a] + (1j * (a == 1) - 1.0 * (a == 0)) * sh
                dE = m._blocks(LAM * DTAU * p[a] * sh, dS, -p[2] * dsh * p[a] - (a == 2) * sh)
                grad[a, :, l] = -np.einsum("nij,nji->n", blk, Einv @ dE).real
            if l + 1 < (b + 1) * s:
                G = m.right_inv(l, m.left(l, G))
    return logdet, grad


def _tdgf(m):
    """G(tau, 0) and -G(0, tau) of all slices: the stabilised ones from the
    space-time system, the others as fill_tdgf does."""
    n, M = m.n, m.M
    A = np.zeros((n * M, n * M), complex)
    B = [m.left(l, np.eye(n, dtype=complex)) for l in range(M)]
    for t in range(M):
        A[t * n:(t + 1) * n, t * n:(t + 1) * n] = np.eye(n)
        if t:
            A[t * n:(t + 1) * n, (t - 1) * n:t * n] = -B[t - 1]
    A[:n, (M - 1) * n:] += B[M - 1]
    e = np.zeros((n * M, n), complex)
    e[:n] = np.eye(n)
    # the inverse's first block column is G(tau, 0); its first block row is
    # (G0, -G0 B_M ... B_2, ...): (1 - G0) B(tau-1, 1)^-1 = G0 B_M ... B_tau
    col = np.linalg.solve(A, e)
    row = np.linalg.solve(A.T, e).T
    gt0, g0t = [None] * M, [None] * M
    for t in range(0, M, m.s):
        gt0[t] = m.true(col[t * n:(t + 1) * n])
        g0t[t] = m.true(row[:, t * n:(t + 1) * n] - (np.eye(n) if t == 0 else 0.0))
    # the slices in between are filled from the stabilised ones of each half
    for t in range(M // 2, M):
        if t % m.s:
            gt0[t], g0t[t] = m.left(t, gt0[t - 1]), m.right_inv(t, g0t[t - 1])
    for t in range(M // 2 - 1, -1, -1):
        if t % m.s:
            gt0[t], g0t[t] = m.left_inv(t + 1, gt0[t + 1]), m.right(t + 1, g0t[t + 1])
    return np.array(gt0), np.array(g0t)


def _udt_pivoted(A):
    """Householder QR, at every step the first column of largest remaining norm."""
    R = np.array(A)
    n = len(R)
    order, vs, beta = np.arange(n), [], np.zeros(n)
    for k in range(n):
        p = k + int(np.argmax(np.einsum("ij,ij->j", R[k:, k:].real, R[k:, k:].real) +
                              np.einsum("ij,ij->j", R[k:, k:].imag, R[k:, k:].imag)))
        R[:, [k, p]], order[[k, p]] = R[:, [p, k]], order[[p, k]]
        v = R[k:, k].copy()
        a, nr = v[0], np.linalg.norm(v)
        if k == n - 1 and a.imag == 0.0:
            vs.append(None)
            beta[k] = a.real
            continue
        beta[k] = -nr if a.real >= 0 else nr
        tau = (beta[k] - a) / beta[k]
        v = v / (a - beta[k])
        v[0] = 1.0
        R[k:, k + 1:] -= np.outer(np.conj(tau) * v, v.conj() @ R[k:, k + 1:])
        R[k + 1:, k], R[k, k] = 0.0, beta[k]
        vs.append((tau, v))
    Q = np.eye(n, dtype=complex)
    for k in range(n - 1, -1, -1):
        if vs[k] is not None:
            tau, v = vs[k]
            Q[k:, k:] -= np.outer(tau * v, v.conj() @ Q[k:, k:])
    D = np.abs(beta)
    T = np.empty_like(R)
    T[:, order] = R / D[:, None]
    return Q, D, T


def exact(case, seed):
    kind, M, s = case["kind"], case["slices"], case["safe_mult"]
    if kind == "batch":
        return None
    L = case["L"]
    n, N = 4 * L * L, L * L
    inp = _inputs(case, seed)
    if kind == "udt":
        if n > 600:
            return None
        U, D, T = _udt_pivoted(inp[1])
        return dict(U=U, D=D, T=T)
    m = _Model(L, M, s, inp[0])
    if kind in ("update", "sweep"):
        # seconds of the from-scratch G's and of the site visits
        calls = case.get("calls", 1)
        if (calls / s + 2) * M / s * (n / 576) ** 3 * 0.25 + calls * N * 4e-4 * (1 + n / 300) > 20:
            return None
        l, acc, det, pac = m.sweep(calls, inp[1], inp[2])
        if kind == "update":
            return dict(accepted=acc[0], rate=float(acc.mean()), detratio=det[0], p_acc=pac[0])
        return dict(accepted=acc, count=int(acc.sum()), greens=m.greens(l)[0], field=m.phi)
    if kind == "greens":
        G, ld = m.greens(case["slice"])
        return dict(greens=G, logdet=ld) if n <= 800 else None
    if kind == "gradient":
        ld, g = _gradient(m)
        return dict(log_weight=ld + m.action(), gradient=g + m.action_gradient())
    if kind == "tdgf":
        if n * M > 6000:
            return None
        gt0, g0t = _tdgf(m)
        return dict(gt0=gt0, g0t=g0t)
    # measure: the chain stands at slice M after the first G; the hook wraps it one slice up
    if n > 600:
        return None
    G = m.true(m.greens(1)[0])
    T = []
    for b in range(2):
        t = np.diag(np.full(N, -MU))
        for x in range(L):
            for y in range(L):
                for q, v in (((y + 1) % L + L * x, TY[b]), ((y - 1) % L + L * x, TY[b]),
                             (y + L * ((x + 1) % L), TX[b]), (y + L * ((x - 1) % L), TX[b])):
                    t[q, y + L * x] -= v
        T.append(t)
    occ = float(np.mean(1 - np.diag(G).real))
    ek = sum(float((T[f & 1] * (np.eye(N) - G[f * N:(f + 1) * N, f * N:(f + 1) * N].T.real)).sum())
             for f in range(4))
    pp, pm, cp, cm = _equal_time(L, G)
    return dict(greens=G, occupation=occ, e_kin=ek, etpc_plus=pp, etpc_minus=pm, etcdc_plus=cp, etcdc_minus=cm)
