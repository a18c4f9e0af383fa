"""The workloads this library is measured on, through its Python entry points.

A case names a call (`kind`) and its sizes: n electrons in r oscillator
shells (m = r (r + 1) single-particle states).  Inputs are synthetic and come
from the seed alone: dense random operators for the commutator benchmark, and
for everything that belongs to a flow a Hartree-Fock-like Hamiltonian
(oscillator energies with a gap at the Fermi level, two-body elements that
fall off with the shells, a nearly vanishing particle-hole one-body part).

exact() states the same quantities on plain torch tensors in float64, written
from the textbook formulas block by block of (M_L, M_S).
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import qd_imsrg_b200 as qd
from qd_imsrg_b200 import warmstart

CLOSED = (2, 6, 12, 20)  # electrons that fill whole shells
STEP = float(np.float32(0.7))  # Magnus step of the flow
COF = (1.0, 0.5, 0.166666666666666666, 0.04166666666666666, 0.0083333333333333333, .001388888888888, 1.984126984e-4,
       2.48015873e-5, 2.755731922e-6, 2.755731922e-7, 2.505210839e-8)  # the BCH series' coefficients
NPARAM = 70401  # parameters of the warm-start network


def listed():
    return [
        # The smallest useful dot with the particle-hole channel: only launches and latency.
        {"name": "commutator_n2_r3", "kind": "commutator", "n": 2, "r": 3, "gen": False, "pandya": True, "split": 0},
        # One commutator of two dense operators, all terms, at an ordinary size.
        {"name": "commutator_n6_r10", "kind": "commutator", "n": 6, "r": 10, "gen": False, "pandya": True, "split": 0},
        # The commutator microbenchmark at the largest basis (bench.py --workload commutator).
        {"name": "commutator_n20_r20", "kind": "commutator", "n": 20, "r": 20, "gen": False, "pandya": True, "split": 0},
        # The same call with the block contractions in the split form, four slices (bench.py --split 4).
        {"name": "commutator_split_n20_r16", "kind": "commutator", "n": 20, "r": 16, "gen": False, "pandya": True,
         "split": 4},
        # The term a Magnus flow evaluates over and over: [Omega, X], Omega generator-like, ladders only.
        {"name": "commutator_gen_n20_r20", "kind": "commutator", "n": 20, "r": 20, "gen": True, "pandya": False,
         "split": 0},
        # Right-hand side of the ODE form of the flow, as the host's Adams integrator calls it.
        {"name": "dgam_n12_r15", "kind": "dgam", "n": 12, "r": 15},
        # One BCH expansion with the particle-hole channel, odd shell count.
        {"name": "bch_ph_n12_r13", "kind": "bch", "n": 12, "r": 13, "pandya": True},
        # A whole ground-state flow of a small dot (the N = 6, R = 10 configuration).
        {"name": "flow_n6_r10", "kind": "flow", "n": 6, "r": 10, "pandya": False},
        # The headline: a converged Magnus IM-SRG(2) flow of N = 20 in R = 20 shells.
        {"name": "flow_n20_r20", "kind": "flow", "n": 20, "r": 20, "pandya": False},
        # A scan over dots: eight flows of mixed sizes in lockstep (bench.py --workload batch).
        {"name": "batch8_r8", "kind": "batch", "count": 8, "r": 8},
        # One Lanczos step's matrix-vector product for a non-scalar (dipole) target.
        {"name": "eom_n12_r10", "kind": "eom", "n": 12, "r": 10, "ml": 1, "ms": 0},
        # Forward and backward pass of the warm-start network on one minibatch of its training.
        {"name": "mlp_grad_8192", "kind": "mlp", "rows": 8192},
    ]


def _closed(rng, r, most=20):
    """An electron number whose shells leave at least two empty ones in r."""
    return rng.choice([n for k, n in enumerate(CLOSED, 1) if k + 2 <= r and n <= most])


def draw(rng):
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    kind = rng.choice(["commutator", "commutator", "commutator", "dgam", "bch", "flow", "flow", "batch", "eom", "mlp"])
    if kind == "commutator":
        r = log(3, 20)
        gen = rng.random() < 0.5
        return {"kind": kind, "n": _closed(rng, r), "r": r, "gen": gen, "pandya": rng.random() < 0.5,
                "split": rng.choice([0, 0, 0, 3, 4, 6])}
    if kind == "dgam":
        r = rng.randint(4, 18)
        return {"kind": kind, "n": _closed(rng, r), "r": r}
    if kind == "bch":
        r = rng.randint(4, 16)
        return {"kind": kind, "n": _closed(rng, r), "r": r, "pandya": rng.random() < 0.5}
    if kind == "flow":
        pandya = rng.random() < 0.3
        r = rng.randint(4, 11 if pandya else 18)
        return {"kind": kind, "n": _closed(rng, r), "r": r, "pandya": pandya}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(2, 10), "r": rng.randint(5, 9)}
    if kind == "eom":
        r = rng.randint(5, 12)
        ml, ms = rng.choice([(0, 0), (1, 0), (-1, 0), (2, 0), (1, 2), (0, 2), (3, 0)])
        return {"kind": kind, "n": _closed(rng, r, 12), "r": r, "ml": ml, "ms": ms}
    return {"kind": kind, "rows": 32 * log(8, 4096)}


# ---- the basis: states, pairs and blocks in the library's vectorize order ----
class Basis:
    """States by shell, then m_l, then m_s; two-body blocks by (M_S, M_L);
    pairs a < b of a block classed hh, ph, pp.  An operator is one vector: E0,
    fhh, fpp, fph, then per block Vhhhh, Vpppp, Vpphh, Vphph, Vppph, Vphhh,
    each column-major."""

    def __init__(self, n: int, r: int):
        self.n, self.r, self.m = n, r, r * (r + 1)
        n, m = self.n, self.m
        sh, ml, ms = zip(*[(s, l, z) for s in range(r) for l in range(-s, s + 1, 2) for z in (-1, 1)])
        self.shell, self.ml, self.ms = np.array(sh), np.array(ml), np.array(ms)
        a, b = np.triu_indices(m, 1)
        q = (self.ms[a] + self.ms[b] + 2) // 2 * (4 * r - 3) + self.ml[a] + self.ml[b] + 2 * r - 2
        cls = (a >= n).astype(np.int64) + (b >= n)
        order = np.argsort(3 * q + cls, kind="stable")
        a, b = a[order], b[order]
        self.nblock = 12 * r - 9
        cnt = np.bincount((3 * q + cls), minlength=3 * self.nblock).reshape(-1, 3)
        start = np.concatenate([[0], np.cumsum(cnt.sum(1))])
        o = 1
        self.one = []
        for rows, cols in ((n, n), (m - n, m - n), (m - n, n)):
            self.one.append((o, rows, cols))
            o += rows * cols
        self.blocks = []  # (first states, second states, (nh, nb, np), [(offset, row class, column class)])
        for k in range(self.nblock):
            parts = []
            for rc, cc in ((0, 0), (2, 2), (2, 0), (1, 1), (2, 1), (1, 0)):
                parts.append((o, rc, cc))
                o += int(cnt[k, rc] * cnt[k, cc])
            s = slice(start[k], start[k + 1])
            self.blocks.append((a[s], b[s], tuple(int(x) for x in cnt[k]), parts))
        self.neq = o

    def energies(self):
        """Single-particle energies: the oscillator's, with a gap of 2 at the Fermi level."""
        return self.shell + 1.0 - 1.0 * (np.arange(self.m) < self.n)

    def same(self):
        """m x m: states of one (m_l, m_s)."""
        return (self.ml[:, None] == self.ml[None, :]) & (self.ms[:, None] == self.ms[None, :])


@functools.lru_cache(maxsize=32)
def _basis(n, r):
    return Basis(n, r)


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _normals(n, seed):
    return torch.randn(n, dtype=torch.float64, device=_device(),
                       generator=torch.Generator(device=_device()).manual_seed(int(seed)))


def _one_body(B, v, scale, same=True):
    """Scales the one-body parts of v and clears what does not conserve (m_l, m_s)."""
    ok = torch.from_numpy(B.same()).to(v.device)
    sl = (slice(0, B.n), slice(B.n, B.m))
    for (o, rows, cols), (x, y) in zip(B.one, ((0, 0), (1, 1), (1, 0))):
        M = v[o:o + rows * cols].view(cols, rows).T
        M *= scale * ok[sl[x], sl[y]]


def _symmetric(B, v, herm):
    """The diagonal-class parts (X + herm X^T) / 2."""
    for o, k, _ in B.one[:2]:
        M = v[o:o + k * k].view(k, k)
        M.copy_((M + herm * M.T) / 2)
    for _, _, cnt, parts in B.blocks:
        for o, rc, cc in parts:
            if rc == cc and cnt[rc]:
                M = v[o:o + cnt[rc] ** 2].view(cnt[rc], cnt[rc])
                M.copy_((M + herm * M.T) / 2)


def _dense_operator(B, herm, seed):
    """Every part N(0, 0.1^2), (m_l, m_s)-conserving, E0 = 0."""
    v = _normals(B.neq, seed) * 0.1
    v[0] = 0.0
    _symmetric(B, v, herm)
    _one_body(B, v, 1.0)
    return v


def _hamiltonian(B, seed):
    """Hartree-Fock-like: energies on the diagonal, tiny one-body remainder,
    two-body elements 0.75 / (shells), about one unit of correlation energy, E0 = 0."""
    v = _normals(B.neq, seed)
    v[0] = 0.0
    fall = 1.0 / (1.0 + torch.from_numpy(B.shell.astype(np.float64)).to(v.device))
    for a, b, cnt, parts in B.blocks:
        w = fall[torch.from_numpy(a).to(v.device)] * fall[torch.from_numpy(b).to(v.device)]
        at = (0, cnt[0], cnt[0] + cnt[1], sum(cnt))
        for o, rc, cc in parts:
            if cnt[rc] and cnt[cc]:
                M = v[o:o + cnt[rc] * cnt[cc]].view(cnt[cc], cnt[rc])
                M *= 0.75 * w[at[cc]:at[cc + 1], None].sqrt() * w[None, at[rc]:at[rc + 1]].sqrt()
    _symmetric(B, v, 1)
    _one_body(B, v, 1e-6)
    e = torch.from_numpy(B.energies()).to(v.device)
    for (o, k, _), s in zip(B.one[:2], (slice(0, B.n), slice(B.n, B.m))):
        v[o:o + k * k].view(k, k).diagonal().copy_(e[s])
    return v


def _generator(B, v, scale):
    """A Magnus-like operator from v: only fph and Vpphh, scaled."""
    g = torch.zeros_like(v)
    o, rows, cols = B.one[2]
    g[o:o + rows * cols] = scale * v[o:o + rows * cols]
    for _, _, cnt, parts in B.blocks:
        o, rc, cc = parts[2]
        g[o:o + cnt[rc] * cnt[cc]] = scale * v[o:o + cnt[rc] * cnt[cc]]
    return g


def _operators(case, seed):
    """The operators of a case as vectors: [(vector, herm), ...]."""
    B = _basis(case["n"], case["r"])
    if case["kind"] == "commutator":
        if case["gen"]:
            return [(_generator(B, _dense_operator(B, -1, 2 * seed), 1.0), -1), (_hamiltonian(B, 2 * seed + 1), 1)]
        return [(_dense_operator(B, -1, 2 * seed), -1), (_dense_operator(B, 1, 2 * seed + 1), 1)]
    H = _hamiltonian(B, 2 * seed + 1)
    if case["kind"] == "bch":  # Omega after one step of the flow, near enough: 0.7 V / (energy denominator)
        return [(_generator(B, H, STEP / 6.0), -1), (H, 1)]
    return [(H, 1)]


# ---- what a program holds ----------------------------------------------------
@functools.lru_cache(maxsize=1)
def _stream():
    """One stream for all work of this program, as one that mixes torch and the library uses."""
    return torch.cuda.Stream()


class _State:
    def __init__(self, case):
        self.case = case


def _new_layout(n, r, own_stream=False):
    P = qd.Layout(n, r, eig=_basis(n, r).energies())
    if not own_stream:
        P.set_stream(_stream().cuda_stream)
    return P


def _view(op):
    """The operator's device array as a tensor that keeps the operator alive."""
    view = qd.DeviceView(op)
    view.op = op
    return torch.as_tensor(view, device="cuda")


def _ham(P, v, herm):
    return qd.FullHam(P, herm, v.cpu().numpy())


def _batch_sizes(case):
    return [(CLOSED[i % 3], case["r"] + i % 4) for i in range(case["count"])]


def _mlp_data(case, seed):
    """Features and targets like the warm start's rows, and the network's parameters."""
    g = torch.Generator(device=_device()).manual_seed(int(seed))
    kw = {"generator": g, "device": _device(), "dtype": torch.float32}
    X = torch.randn((case["rows"], 16), **kw)
    X[:, 4:8] = (X[:, 4:8] > 0).float()
    T = torch.tanh(X[:, 0] - 0.5 * X[:, 8]) + 0.1 * torch.randn(case["rows"], **kw)
    P = torch.randn(NPARAM, **kw) / 16.0
    P[:256 * 16] *= 4.0
    return X, T, P


def prepare(case, seed):
    s = _State(case)
    kind = case["kind"]
    if kind == "mlp":
        s.X, s.T, p = _mlp_data(case, seed)
        s.net = warmstart.MLP()
        s.net.set_params(p.cpu().numpy())
        s.g = torch.empty(NPARAM, dtype=torch.float32, device="cuda")
        return s
    if kind == "batch":
        s.pairs, s.keep = [], []
        for i, (n, r) in enumerate(_batch_sizes(case)):
            P = _new_layout(n, r, own_stream=True)
            s.keep.append(P)
            s.pairs.append((_ham(P, _hamiltonian(_basis(n, r), 100 * seed + i), 1), qd.FullHam(P, 1)))
        s.out = [_view(hs) for _, hs in s.pairs]
        return s
    s.P = _new_layout(case["n"], case["r"])
    s.ops = [_ham(s.P, v, h) for v, h in _operators(case, seed)]
    if kind == "eom":
        n1, n2 = qd.eom_dim(s.P, case["ml"], case["ms"])
        s.v = _normals(n1 + n2, 7 * seed + 3)
        s.v /= s.v.norm()
        return s
    s.C = qd.FullHam(s.P, 1)
    s.out = _view(s.C)
    if kind == "commutator":
        s.P.split = case["split"]
    if kind == "bch":
        s.ws = [qd.FullHam(s.P, 1) for _ in range(5)]
        s.cc = [qd.CCMat(s.P, 1.0), qd.CCMat(s.P, -1.0)]
    s.P.synchronize()
    return s


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "commutator":
        qd.commutator(s.ops[0], s.ops[1], s.C, pandya=case["pandya"])
        return s.out
    if kind == "dgam":
        qd.dgam(s.ops[0], s.C)
        return s.out
    if kind == "bch":
        terms = qd.bch_expand(s.C, s.ops[0], s.ops[1], *s.ws, *s.cc, pandya=case["pandya"])
        return {"HS": s.out, "terms": terms}
    if kind == "flow":
        _, res = qd.magnus_flow(s.ops[0], s.C, pandya=case["pandya"])
        return {"HS": s.out, "steps": res.iterations, "commutators": res.commutators}
    if kind == "batch":
        res, _ = qd.magnus_flow_batch(s.pairs)
        return {"HS": s.out, "commutators": [r.commutators for r in res]}
    if kind == "eom":
        return qd.eom_matvec_target(s.ops[0], case["ml"], case["ms"], s.v)
    loss = s.net.grad(s.X, s.T, s.g)
    return {"grad": s.g, "loss": loss}


# ---- work of one pass ----------------------------------------------------------
def _commutator_flops(B, gen, pandya):
    """FP64 operations of [A, B]: ladders, one particle-hole product per
    cross-coupled block, and two operations per term of the one-body legs."""
    size = {}
    for key in zip(B.ml, B.ms):
        size[key] = size.get(key, 0) + 1
    legs = np.array([size[key] for key in zip(B.ml, B.ms)], np.float64)
    fl = 0.0
    for a, b, (nh, nb, npp), _ in B.blocks:
        d = nh + nb + npp
        if gen:  # A holds only Vpphh: pp and hh rows meet it over hh and pp pairs
            fl += 2.0 * npp * nh * (npp + nh + 2 * nb + npp + nh)
        else:  # the six stored parts, contracted over hh and pp pairs, for both orders
            stored = nh * nh + npp * npp + npp * nh + nb * nb + npp * nb + nb * nh
            fl += 2.0 * stored * (nh + npp)
            fl += 4.0 * d * float((legs[a] + legs[b]).sum()) if d else 0.0
    if pandya:
        key = (B.ml[:, None] - B.ml[None, :]) * 8 + B.ms[:, None] - B.ms[None, :]
        ks, inv = np.unique(key, return_inverse=True)
        inv = inv.reshape(key.shape)
        rows = np.bincount(inv.ravel(), minlength=len(ks)).astype(float)
        cols = np.bincount(inv[:B.n, B.n:].ravel(), minlength=len(ks)).astype(float)
        fl += float((2.0 * rows * rows * cols).sum())
    return fl


def work(case):
    kind = case["kind"]
    if kind == "mlp":
        per = 2.0 * (16 * 256 + 256 * 256 + 256)
        return {"bytes": 4.0 * (case["rows"] * 17 + 2 * NPARAM + 1), "flops": 3.0 * per * case["rows"]}
    if kind == "batch":
        w = [work({"kind": "flow", "n": n, "r": r, "pandya": False}) for n, r in _batch_sizes(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    B = _basis(case["n"], case["r"])
    gen_entries = B.one[2][1] * B.one[2][2] + sum(c[2] * c[0] for _, _, c, _ in B.blocks)
    if kind == "commutator":
        a = gen_entries if case["gen"] else B.neq
        return {"bytes": 8.0 * (a + 2 * B.neq), "flops": _commutator_flops(B, case["gen"], case["pandya"])}
    if kind == "dgam":
        return {"bytes": 16.0 * B.neq, "flops": _commutator_flops(B, True, True)}
    if kind == "bch":  # about six terms until the series is cut
        return {"bytes": 8.0 * (gen_entries + 2 * B.neq), "flops": 6 * _commutator_flops(B, True, case["pandya"])}
    if kind == "flow":  # about fourteen steps of six terms
        return {"bytes": 16.0 * B.neq, "flops": 80 * _commutator_flops(B, True, case["pandya"])}
    n, p = B.n, B.m - B.n  # eom: every stored element of H read once, each amplitude meets a row of H
    nv = sum(len(x) for x in _targets(B, case["ml"], case["ms"]))
    return {"bytes": 8.0 * (B.neq + 2 * nv), "flops": 2.0 * nv * (4.0 * p + p * p / (2.0 * B.r) + 4.0 * n * p / B.r)}


# ---- the same in 64 bits, on plain tensors -------------------------------------
class _Dense:
    """Block matrices of operators on one basis (all pairs of a block, both triangles)."""

    def __init__(self, B):
        self.B, self.dev = B, _device()
        t = lambda x: torch.as_tensor(x, device=self.dev)  # noqa: E731
        m = B.m
        self.hole = torch.arange(m, device=self.dev) < B.n
        self.pairs = [(t(a), t(b)) for a, b, _, _ in B.blocks]
        self.d = [len(a) for a, _, _, _ in B.blocks]
        self.off = t(np.concatenate([[0], np.cumsum([x * x for x in self.d])]))
        blk = np.full((m, m), -1)
        pos = np.zeros((m, m), np.int64)
        sgn = np.zeros((m, m))
        for q, (a, b, _, _) in enumerate(B.blocks):
            for x, y, s in ((a, b, 1.0), (b, a, -1.0)):
                blk[x, y], pos[x, y], sgn[x, y] = q, np.arange(len(a)), s
        self.blk, self.pos, self.sgn, self.dim = t(blk), t(pos), t(sgn), t(np.array(self.d))
        self.same = t(B.same())

    def unpack(self, v, herm):
        """(f, [block matrices]) of a vector."""
        B, n = self.B, self.B.n
        f = torch.zeros((B.m, B.m), dtype=torch.float64, device=self.dev)
        part = lambda o, rows, cols: v[o:o + rows * cols].view(cols, rows).T  # noqa: E731
        f[:n, :n], f[n:, n:], f[n:, :n] = (part(*x) for x in B.one)
        f[:n, n:] = herm * f[n:, :n].T
        V = []
        for d, (_, _, cnt, parts) in zip(self.d, B.blocks):
            M = torch.zeros((d, d), dtype=torch.float64, device=self.dev)
            at = (0, cnt[0], cnt[0] + cnt[1], d)
            for o, rc, cc in parts:
                if cnt[rc] and cnt[cc]:
                    X = part(o, cnt[rc], cnt[cc])
                    M[at[rc]:at[rc + 1], at[cc]:at[cc + 1]] = X
                    if rc != cc:
                        M[at[cc]:at[cc + 1], at[rc]:at[rc + 1]] = herm * X.T
            V.append(M)
        return f, V

    def pack(self, e0, f, V):
        B, n = self.B, self.B.n
        v = torch.empty(B.neq, dtype=torch.float64, device=self.dev)
        v[0] = e0
        for (o, rows, cols), X in zip(B.one, (f[:n, :n], f[n:, n:], f[n:, :n])):
            v[o:o + rows * cols] = X.T.reshape(-1)
        for M, d, (_, _, cnt, parts) in zip(V, self.d, B.blocks):
            at = (0, cnt[0], cnt[0] + cnt[1], d)
            for o, rc, cc in parts:
                v[o:o + cnt[rc] * cnt[cc]] = M[at[rc]:at[rc + 1], at[cc]:at[cc + 1]].T.reshape(-1)
        return v

    def element(self, flat, a, b, c, d):
        """V_abcd from concatenated block matrices, for broadcast index tensors."""
        q, s = self.blk[a, b], self.sgn[a, b] * self.sgn[c, d]
        ok = (q >= 0) & (q == self.blk[c, d])
        at = self.off[q.clamp(min=0)] + self.pos[a, b] * self.dim[q.clamp(min=0)] + self.pos[c, d]
        return torch.where(ok, s * flat[torch.where(ok, at, 0)], 0.0)

    def _one_times_pair(self, q, f):
        """f on either leg of the block's pairs: f_ac d_bd - f_ad d_bc + d_ac f_bd - d_ad f_bc."""
        i, j = self.pairs[q]
        eq = lambda x, y: (x[:, None] == y[None, :]).double()  # noqa: E731
        g = lambda x, y: f[x][:, y]  # noqa: E731
        return g(i, i) * eq(j, j) - g(i, j) * eq(j, i) + eq(i, i) * g(j, j) - eq(i, j) * g(j, i)

    def commutator(self, a, ha, b, hb, pandya):
        B, n = self.B, self.B.n
        fa, VA = self.unpack(a, ha)
        fb, VB = self.unpack(b, hb)
        w1 = self.hole.double()[:, None] - self.hole.double()[None, :]
        e0 = float((w1 * fa * fb.T).sum())
        f = fa @ fb - fb @ fa
        V = []
        for q, (_, _, cnt, _) in enumerate(B.blocks):
            A, X, nh, lo = VA[q], VB[q], cnt[0], cnt[0] + cnt[1]
            e0 += float((A[:nh, lo:] * X[lo:, :nh].T).sum() - (X[:nh, lo:] * A[lo:, :nh].T).sum())
            w = torch.zeros(self.d[q], dtype=torch.float64, device=self.dev)
            w[:nh], w[lo:] = -1.0, 1.0
            FA, FB = self._one_times_pair(q, fa), self._one_times_pair(q, fb)
            V.append((FA + A * w) @ X - X @ (FA + w[:, None] * A) - FB @ A + A @ FB)
            if self.d[q] == 0:
                continue
            # one-body: sum over c of W_cicj, intermediate pp pairs for a hole c, hh pairs for a particle c
            Wpp = A[:, lo:] @ X[lo:, :] - X[:, lo:] @ A[lo:, :]
            Whh = A[:, :nh] @ X[:nh, :] - X[:, :nh] @ A[:nh, :]
            i, j = self.pairs[q]
            for c, x, c2, y, s in ((i, j, i, j, 1.0), (j, i, j, i, 1.0), (i, j, j, i, -1.0), (j, i, i, j, -1.0)):
                r, k = torch.nonzero(c[:, None] == c2[None, :], as_tuple=True)
                val = s * torch.where(self.hole[c[r]], Wpp[r, k], Whh[r, k])
                f.index_put_((x[r], y[k]), val, accumulate=True)
        FA, FB = (torch.cat([M.reshape(-1) for M in U]) for U in (VA, VB))
        # one-body: sum_ab (n_a - n_b) (fA_ab VB_biaj - fB_ab VA_biaj)
        sa, sb = torch.nonzero(self.same & (w1 != 0), as_tuple=True)
        ti, tj = torch.nonzero(self.same, as_tuple=True)
        for at in range(0, len(ti), 1024):
            i, j = ti[at:at + 1024, None], tj[at:at + 1024, None]
            x = (w1 * fa)[sa, sb] * self.element(FB, sb[None], i, sa[None], j)
            x -= (w1 * fb)[sa, sb] * self.element(FA, sb[None], i, sa[None], j)
            f[i[:, 0], j[:, 0]] += x.sum(1)
        if pandya:
            self._particle_hole(FA, FB, w1, V)
        return self.pack(e0, f, V)

    def _particle_hole(self, FA, FB, w1, V):
        """V -= (1 - P12)(1 - P34) G, G_ijkl = sum_ab (n_a - n_b) VA_bjal VB_aibk, by the
        transfer (m_l, m_s)_i - (m_l, m_s)_k."""
        B = self.B
        key = (B.ml[:, None] - B.ml[None, :]) * 8 + B.ms[:, None] - B.ms[None, :]
        ks, inv = np.unique(key, return_inverse=True)  # symmetric about zero: class k has transfer -class[-1 - k]
        inv = inv.reshape(key.shape)
        rows = [np.nonzero(inv == k) for k in range(len(ks))]
        pos = np.zeros((B.m, B.m), np.int64)
        for x, y in rows:
            pos[x, y] = np.arange(len(x))
        t = lambda x: torch.as_tensor(x, device=self.dev)  # noqa: E731
        cnt = np.array([len(x) for x, _ in rows])
        size = cnt * cnt[::-1]
        goff, G = t(np.concatenate([[0], np.cumsum(size)])), []
        for k in range(len(ks)):
            i, c = (t(x)[:, None] for x in rows[k])
            j, l = (t(x)[:, None] for x in rows[-1 - k])
            b, a = (t(x)[None] for x in rows[k])
            keep = (w1[a[0], b[0]] != 0)
            a, b = a[:, keep], b[:, keep]
            XB = self.element(FB, a, i, b, c) * w1[a[0], b[0]]
            G.append((XB @ self.element(FA, b, j, a, l).T).reshape(-1))
        G, tinv, tpos, tcnt = torch.cat(G), t(inv), t(pos), t(cnt[::-1].copy())

        def g(i, j, k, l):
            q = tinv[i, k]
            return G[goff[q] + tpos[i, k] * tcnt[q] + tpos[j, l]]

        for q, (x, y) in enumerate(self.pairs):
            i, j, k, l = x[:, None], y[:, None], x[None], y[None]
            V[q] -= g(i, j, k, l) - g(j, i, k, l) - g(i, j, l, k) + g(j, i, l, k)

    def white(self, h):
        """The generator V / (energy denominator with the diagonal two-body elements), as a vector."""
        B, n = self.B, self.B.n
        f, V = self.unpack(h, 1)
        flat = torch.cat([M.reshape(-1) for M in V])
        e = f.diagonal()
        s = torch.arange(B.m, device=self.dev)
        dd = self.element(flat, s[:, None], s[None], s[:, None], s[None])  # V_abab
        g = torch.zeros_like(h)
        o, rows, cols = B.one[2]
        g[o:o + rows * cols] = (f[n:, :n] / (e[n:, None] - e[None, :n] - dd[n:, :n])).T.reshape(-1)
        for M, (x, y), (_, _, cnt, parts) in zip(V, self.pairs, B.blocks):
            nh, lo = cnt[0], cnt[0] + cnt[1]
            if nh and cnt[2]:
                a, b, i, j = x[lo:, None], y[lo:, None], x[None, :nh], y[None, :nh]
                den = e[a] + e[b] - e[i] - e[j] + dd[a, b] + dd[i, j] - dd[a, i] - dd[a, j] - dd[b, i] - dd[b, j]
                g[parts[2][0]:parts[2][0] + nh * cnt[2]] = (M[lo:, :nh] / den).T.reshape(-1)
        return g

    def mbpt2(self, h):
        f, V = self.unpack(h, 1)
        e, tot = f.diagonal(), 0.0
        for M, (x, y), (_, _, cnt, _) in zip(V, self.pairs, self.B.blocks):
            nh, lo = cnt[0], cnt[0] + cnt[1]
            a, b, i, j = x[lo:, None], y[lo:, None], x[None, :nh], y[None, :nh]
            tot += float((M[lo:, :nh] ** 2 / (e[i] + e[j] - e[a] - e[b])).sum())
        return tot

    def bch(self, g, h, pandya):
        hs, ad, terms = h.clone(), h, 0
        for cof in COF:
            ad = self.commutator(g, -1, ad, 1, pandya)
            n1, n2 = float(hs[1:].norm()), float(ad[1:].norm())
            hs = hs + cof * ad
            terms += 1
            if n2 * cof / n1 < float(np.float32(1e-5)):
                break
        return hs, terms

    def flow(self, h, pandya):
        g, hs, eta = torch.zeros_like(h), h, self.white(h)
        step, crit, total, steps, nrm1 = STEP, abs(self.mbpt2(h)), 0, 0, float(eta[1:].norm())
        while crit > float(np.float32(1e-9)):
            g2 = g + step * eta
            hs2, terms = self.bch(g2, h, pandya)
            total += terms
            eta2 = self.white(hs2)
            if nrm1 * 1.5 < float(eta2[1:].norm()):  # the step is rejected
                step = step / 2.0 + float(np.float32(1e-3))
            else:
                g, hs, eta, steps = g2, hs2, eta2, steps + 1
                crit = abs(self.mbpt2(hs))
        return {"HS": hs, "steps": steps, "commutators": total}


def _targets(B, ml, ms):
    """Index arrays (a, i) and (a, b, i, j) of an excitation by (ml, ms), in the library's vector order."""
    n, m = B.n, B.m
    a, i = (x.ravel() for x in np.meshgrid(np.arange(n, m), np.arange(n), indexing="ij"))
    ok = (B.ml[a] - B.ml[i] == ml) & (B.ms[a] - B.ms[i] == ms)
    one = np.stack([a[ok], i[ok]], 1)
    a, b = (x + n for x in np.triu_indices(m - n, 1))
    i, j = np.triu_indices(n, 1)
    x, y = np.nonzero(((B.ml[a] + B.ml[b])[:, None] - (B.ml[i] + B.ml[j])[None] == ml) &
                      ((B.ms[a] + B.ms[b])[:, None] - (B.ms[i] + B.ms[j])[None] == ms))
    return one, np.stack([a[x], b[x], i[y], j[y]], 1)


def _eom(D, h, case, v):
    """[H, Q] for Q = sum Q_ai a+i + 1/4 sum Q_abij a+b+ji on full index ranges."""
    B, n, m = D.B, D.B.n, D.B.m
    f, V = D.unpack(h, 1)
    flat = torch.cat([M.reshape(-1) for M in V])
    P, H = slice(n, m), slice(0, n)
    s = torch.arange(m, device=D.dev)

    def el(*r):
        r = [s[x] for x in r]
        return D.element(flat, r[0][:, None, None, None], r[1][:, None, None], r[2][:, None], r[3])

    one, two = (torch.as_tensor(x, device=D.dev) for x in _targets(B, case["ml"], case["ms"]))
    p = m - n
    q1 = torch.zeros((p, n), dtype=torch.float64, device=D.dev)
    q2 = torch.zeros((p, p, n, n), dtype=torch.float64, device=D.dev)
    q1[one[:, 0] - n, one[:, 1]] = v[:len(one)]
    a, b, i, j = two[:, 0] - n, two[:, 1] - n, two[:, 2], two[:, 3]
    x = v[len(one):]
    q2[a, b, i, j], q2[b, a, i, j], q2[a, b, j, i], q2[b, a, j, i] = x, -x, -x, x
    fp, fh, fhp = f[P, P], f[H, H], f[H, P]
    ee = torch.einsum
    phph = el(P, H, P, H)  # V_akci
    r1 = fp @ q1 - q1 @ fh + ee("jb,abij->ai", fhp, q2) - ee("bj,ajbi->ai", q1, phph)
    r1 += 0.5 * ee("cbij,ajcb->ai", q2, el(P, H, P, P)) - 0.5 * ee("abkj,kjib->ai", q2, el(H, H, H, P))
    r2 = ee("ac,cbij->abij", fp, q2) + ee("bc,acij->abij", fp, q2)
    r2 += -ee("abkj,ki->abij", q2, fh) + ee("abki,kj->abij", q2, fh)
    t = ee("ci,abcj->abij", q1, el(P, P, P, H))
    r2 += t - t.transpose(2, 3)
    t = ee("akji,bk->abij", el(P, H, H, H), q1)
    r2 += t - t.transpose(0, 1)
    r2 += 0.5 * (el(P, P, P, P).reshape(p * p, p * p) @ q2.reshape(p * p, n * n)).reshape(p, p, n, n)
    r2 += 0.5 * ee("klij,abkl->abij", el(H, H, H, H), q2)
    t = ee("akci,bckj->abij", phph, q2)
    t = t - t.transpose(0, 1)
    r2 += t - t.transpose(2, 3)
    return torch.cat([r1[one[:, 0] - n, one[:, 1]], r2[a, b, i, j]])


def _mlp(X, T, P):
    X, T = X.double(), T.double()
    P = P.double().requires_grad_(True)
    W1, b1, W2, b2, w3, b3 = torch.split(P, (256 * 16, 256, 256 * 256, 256, 256, 1))
    gelu = torch.nn.functional.gelu
    y = gelu(gelu(X @ W1.view(256, 16).T + b1) @ W2.view(256, 256).T + b2) @ w3 + b3
    loss = ((y - T) ** 2).mean()
    loss.backward()
    return {"grad": P.grad, "loss": float(loss)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        return _mlp(*_mlp_data(case, seed))
    # whole flows take hundreds of commutators, full index ranges m^4 values
    if kind == "batch" or (kind == "flow" and case["r"] > 5) or (kind == "eom" and case["r"] > 10):
        return None
    if kind == "bch" and case["r"] > 14:
        return None
    D = _Dense(_basis(case["n"], case["r"]))
    ops = _operators(case, seed)
    if kind == "commutator":
        return D.commutator(*ops[0], *ops[1], case["pandya"])
    h = ops[-1][0]
    if kind == "dgam":
        return D.commutator(D.white(h), -1, h, 1, True)
    if kind == "bch":
        hs, terms = D.bch(ops[0][0], h, case["pandya"])
        return {"HS": hs, "terms": terms}
    if kind == "flow":
        return D.flow(h, case["pandya"])
    v = _normals(sum(len(x) for x in _targets(D.B, case["ml"], case["ms"])), 7 * seed + 3)
    return _eom(D, h, case, v / v.norm())
