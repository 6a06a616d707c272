"""The work that programs have this library do, as cases that can be timed and compared.

A case names one of the kinds below with its sizes.  Every system has the synthetic integrals of
shci_gb300/synthetic.py (random, no symmetry, orbitals in order of energy), n orbitals and n_up /
n_dn electrons; its determinants are the first `dets` of the library's own heat-bath schedule, as
they are in a user's run.

  elems      Hamiltonian elements of pairs of determinants (the plugin API's matrix elements)
  connected  connected determinants of a list (the plugin API's find_connected_dets)
  variation  the whole variational stage: selection, Hamiltonian updates, Davidson
  step       one Hamiltonian build + Davidson + energy on a list that comes from host memory
  hv         one product H v of a Hamiltonian that is built (device vectors)
  dtm        deterministic PT2 of a wavefunction
  pt2        the three PT2 stages: deterministic, pseudo-stochastic, stochastic
  rdm        1- and 2-RDM of a wavefunction (the adjoint of its energy)
  batch      many small systems solved at a time, from their FCIDUMP files
"""
import math
import os
import tempfile

import numpy as np
import torch

import shci_gb300
from shci_gb300 import synthetic

SCHEDULE = (1e-3, 5e-4, 2e-4, 1e-4, 5e-5, 2e-5)
TARGET = 5e-5  # target_error: the library's default
PREC = {"fp64": shci_gb300.PREC_FP64, "mixed": shci_gb300.PREC_MIXED}


def listed():
    return [
        # a few pairs' elements: the smallest call, all of it latency
        dict(name="elems_n16", kind="elems", n=16, n_up=5, n_dn=5, dets=600, count=200),
        # every connection of some dets through the plugin API (a window without a threshold)
        dict(name="connected_n26", kind="connected", n=26, n_up=7, n_dn=7, dets=600, count=16),
        # a small molecule's whole variational run, all FP64 (the n = 16 workload)
        dict(name="variation_n16_fp64", kind="variation", n=16, n_up=5, n_dn=5, eps_var=1e-4,
             prec="fp64", room=1 << 15),
        # the n = 26 workload's variational run, mixed storage
        dict(name="variation_n26_mixed", kind="variation", n=26, n_up=7, n_dn=7, eps_var=1e-4,
             prec="mixed", room=1 << 17),
        # the benchmark's step (n = 40) at the size of its eps_var = 5e-5 iteration: the largest
        dict(name="step_n40_mixed", kind="step", n=40, n_up=10, n_dn=10, dets=1200000, prec="mixed"),
        # a product H v as an eigensolver of the user's own calls it, mixed storage
        dict(name="hv_n40_mixed", kind="hv", n=40, n_up=10, n_dn=10, dets=400000, prec="mixed"),
        # the same in FP64 on an odd-sized open-shell system
        dict(name="hv_n23_fp64", kind="hv", n=23, n_up=7, n_dn=5, dets=50001, prec="fp64"),
        # deterministic PT2 of the n = 26 workload's wavefunction
        dict(name="dtm_n26", kind="dtm", n=26, n_up=7, n_dn=7, dets=30000, eps_pt=1e-6),
        # semistochastic PT2 of the n = 40 workload: three stages, 64 stochastic batches
        dict(name="pt2_n40", kind="pt2", n=40, n_up=10, n_dn=10, dets=40000, eps_pt=1e-6,
             samples=20000),
        # gradients with respect to the integrals (n = 26 adjoint workload)
        dict(name="rdm_n26", kind="rdm", n=26, n_up=7, n_dn=7, dets=80000, prec="mixed"),
        # both RDMs of an open-shell system with an odd orbital count
        dict(name="rdm_n19_fp64", kind="rdm", n=19, n_up=6, n_dn=4, dets=9999, prec="fp64"),
        # a queue of small instances through the batch runner
        dict(name="batch_16", kind="batch", count=16, eps_var=1e-4, eps_pt=1e-6),
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choice(["elems", "connected", "variation", "variation", "step", "step", "hv", "hv",
                       "dtm", "pt2", "rdm", "batch"])
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 16), eps_var=float("%.3g" % _log(rng, 1e-4, 1e-3)),
                    eps_pt=1e-6)
    n = rng.randint(12, 40)
    n_up = rng.randint(3, min(10, n // 4 + 1))
    n_dn = rng.randint(max(2, n_up - 2), n_up)
    if kind in ("dtm", "rdm"):  # (their 64-bit values pack a determinant into one word)
        n = min(n, 30)
        n_up, n_dn = min(n_up, 8), min(n_dn, 8)
    c = dict(kind=kind, n=n, n_up=n_up, n_dn=n_dn)
    most = space(n, n_up + n_dn, 1e-4)
    if kind == "variation":
        c["eps_var"] = float("%.3g" % _log(rng, 1.5e-4, 2e-3))
        c["prec"] = rng.choice(["fp64", "mixed"])
        c["room"] = 1 << int(math.log2(4 * space(n, n_up + n_dn, c["eps_var"])) + 1)
        return c
    limit = {"elems": 1000, "connected": 1000, "dtm": 20000, "pt2": 30000}.get(kind, 500000)
    least = 5000 if kind == "hv" else 100
    c["dets"] = int(_log(rng, least, max(2 * least, min(limit, most / 4))))
    if kind == "elems":
        c["count"] = int(_log(rng, 1, 200000))
    elif kind == "connected":
        c["count"] = int(_log(rng, 1, 30))
    elif kind in ("dtm", "pt2"):
        c["eps_pt"] = float("%.3g" % _log(rng, 1e-6, 1e-5))
        if kind == "pt2":
            c["samples"] = int(_log(rng, 500, 20000))
    else:
        c["prec"] = rng.choice(["fp64", "mixed"])
    return c


# ---- inputs ---------------------------------------------------------------------------------


def integrals(n, n_occ, seed):
    """Synthetic integrals with the orbitals in order of their energies in the lowest filling, as
    reading an FCIDUMP leaves them."""
    rng = np.random.default_rng(synthetic.BASE_SEED + 7919 * seed + n)
    a = rng.standard_normal((n, n))
    h = np.diag(-2.0 + 4.0 * np.arange(n) / n) + 0.05 * (a + a.T) / 2.0
    p = np.arange(n)
    decay = np.exp(-np.abs(p[:, None] - p[None, :]) / 4.0) * 0.3 / np.sqrt(2.0 * n)
    u = rng.standard_normal((2 * n, n, n))
    b = (np.triu(u) + np.triu(u, 1).transpose(0, 2, 1)) * decay
    f = b.reshape(2 * n, n * n)
    g = (f.T @ f).reshape(n, n, n, n)
    low = np.argsort(np.diag(h))[:n_occ]
    e = np.diag(h) + 2 * np.einsum("ppqq->pq", g)[:, low].sum(1) - np.einsum("pqqp->pq", g)[:, low].sum(1)
    o = np.argsort(e, kind="stable")
    h = np.ascontiguousarray(h[np.ix_(o, o)])
    g = np.ascontiguousarray(g[np.ix_(o, o, o, o)])
    pq = np.maximum.outer(p, p) * n + np.minimum.outer(p, p)  # (exactly symmetric, as a file is)
    i, j = np.divmod(pq, n)
    g = g[i, j][:, :, i, j]
    k = pq.ravel()
    m = g.reshape(n * n, n * n)
    m = np.where(k[:, None] >= k[None, :], m, m.T)
    return np.ascontiguousarray(h), np.ascontiguousarray(m.reshape(n, n, n, n))


def context(case, seed):
    n, nu, nd = case["n"], case["n_up"], case["n_dn"]
    h, g = integrals(n, (nu + nd) // 2, seed)
    ctx = shci_gb300.Context(0)
    ctx.set_integrals(h, g, nu, nd, (1 << nu) - 1, (1 << nd) - 1)
    ctx.build_queues()
    return ctx, h, g


def schedule(eps):
    return [e for e in SCHEDULE if e > eps * 1.0001]


def determinants(ctx, case):
    """The first `dets` determinants of the schedule with the coefficients that its last selection
    leaves (new ones at 1e-16)."""
    eps = list(SCHEDULE)
    while True:
        e = eps.pop(0) if eps else e / 2
        ctx.select(e)
        n = ctx.n_dets()
        if n >= case["dets"] or e < 1e-7:
            break
        ctx.update_hamiltonian(PREC["mixed"])
        ctx.davidson(TARGET / 50)
    m = min(n, case["dets"])
    return [np.ascontiguousarray(v[:m]) for v in ctx.dets()]


def wavefunction(ctx, case):
    ctx.set_dets(*determinants(ctx, case))
    ctx.update_hamiltonian(PREC[case.get("prec", "mixed")])
    ctx.davidson(1e-10)


def prepare(case, seed):
    if case["kind"] == "batch":
        d = tempfile.TemporaryDirectory(prefix="shci_batch_")
        rng = np.random.default_rng(seed)
        inst = []
        for i in range(case["count"]):
            n = int(rng.integers(12, 21))
            ne = int(rng.integers(3, n // 2))
            h, g = integrals(n, ne, 1000 * seed + i)
            path = os.path.join(d.name, "FCIDUMP_%d" % i)
            synthetic.write_fcidump(path, h, g, 2 * ne)
            inst.append((path, ne, ne))
        return dict(case=case, dir=d, inst=inst)
    ctx, _, _ = context(case, seed)
    s = dict(case=case, ctx=ctx)
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind in ("elems", "connected"):
        up, dn, _ = determinants(ctx, case)
        if kind == "connected":
            k = rng.integers(0, len(up), case["count"])
            s["args"] = (up[k], dn[k], 1e100, 0.0)
        else:  # half of the pairs are near one another in the list, which connects many of them
            i = rng.integers(0, len(up), case["count"])
            j = rng.integers(0, len(up), case["count"])
            j[::2] = (i[::2] + rng.integers(0, 4, len(i[::2]))) % len(up)
            s["args"] = (up[i], dn[i], up[j], dn[j])
    elif kind == "step":
        s["dets"] = determinants(ctx, case)
    elif kind == "hv":
        wavefunction(ctx, case)
        c = ctx.dets()[2]
        # an eigensolver's vector: the wavefunction and a correction over all determinants
        g = torch.Generator(device="cuda").manual_seed(seed)
        r = torch.randn(len(c), generator=g, device="cuda", dtype=torch.float64)
        s["x"] = torch.from_numpy(c).cuda() + r * (0.1 / math.sqrt(len(c)))
        s["y"] = torch.empty_like(s["x"])
    elif kind in ("dtm", "pt2", "rdm"):
        wavefunction(ctx, case)
        s["e"] = ctx.energy_fp64()
    torch.cuda.synchronize()
    return s


def run(s):
    case, ctx = s["case"], s.get("ctx")
    kind = case["kind"]
    if kind == "elems":
        return ctx.h_elems(*s["args"])
    if kind == "connected":
        off, u, d, nx = ctx.find_connected(*s["args"])
        return [off.view(np.int64), u.view(np.int64), d.view(np.int64), nx]
    if kind == "variation":
        one = np.ones(1, np.uint64)
        ctx.set_dets((one << case["n_up"]) - one, (one << case["n_dn"]) - one, np.ones(1))
        e = ctx.run_variation([case["eps_var"]], schedule(case["eps_var"]), TARGET, PREC[case["prec"]])
        up, dn, c = ctx.dets()
        room = case["room"]  # (of one length for every seed)
        return [e, len(c)] + [np.pad(v, (0, room - len(v))) for v in (up.view(np.int64), dn.view(np.int64), c)]
    if kind == "step":
        up, dn, c = s["dets"]
        ctx.set_dets(up, dn, c)
        nnz, _ = ctx.update_hamiltonian(PREC[case["prec"]])
        ctx.davidson(1e-10)
        return [ctx.energy_fp64(), nnz, ctx.dets()[2]]
    if kind == "hv":
        ctx.hv_dev(s["x"].data_ptr(), s["y"].data_ptr())
        return s["y"]
    if kind == "dtm":
        value, _, count = ctx.pt2_dtm(s["e"], case["eps_pt"], 0)
        return [value, count]
    if kind == "pt2":
        e, eps = s["e"], case["eps_pt"]
        dtm, _, n_dtm = ctx.pt2_dtm(e, eps, 0)
        psto, u, n_psto, done = ctx.pt2_psto(e, eps, eps / 5, 16, TARGET / 10, eps / 20)
        sto, su, loops = ctx.pt2_sto(e, eps / 5, eps / 20, 64, case["samples"], 347634253, 20, TARGET, u)
        return [dtm, n_dtm, psto, u, n_psto, done, sto, su, loops]
    if kind == "rdm":
        return [ctx.rdm1(), ctx.rdm2_half()]
    res, _ = shci_gb300._lib.batch_solve(s["inst"], [case["eps_var"]], (), (case["eps_pt"], 0.0, 0.0))
    return [np.array([r[k] for r in res], t) for k, t in
            (("energy_hf", float), ("energy_var", float), ("correction_pt", float), ("n_dets", np.int64),
             ("n_pt_dets", np.int64))]


# ---- the work of a pass -----------------------------------------------------------------------


def space(n, ne, eps):
    """Determinants of the space at eps_var: a fit to runs of these systems (within about a factor
    of two)."""
    return 2270.0 * (1e-3 / eps) ** 1.75 * (n / 26) ** 1.77 * (ne / 14) ** 1.53


def row(n, ne, dets):
    """Stored (upper) elements of a determinant: a fit, as above."""
    return min(dets / 2, 177.0 * (dets / 1e4) ** 0.166 * (n / 26) * (ne / 14) ** 0.31)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        dets = space(16, 11, case["eps_var"])
        one = dets * row(16, 11, dets) * 12
        return dict(bytes=case["count"] * one * 30, flops=case["count"] * one * 20)
    n, nu, nd = case["n"], case["n_up"], case["n_dn"]
    ne = nu + nd
    if kind == "elems":  # four strings read and a value written; about 2 ne terms of a single
        return dict(bytes=case["count"] * 40.0, flops=case["count"] * 2.0 * ne)
    if kind == "connected":  # both strings and a byte written
        u, d = nu * (n - nu), nd * (n - nd)
        pairs = u + d + u * d + (u * (nu - 1) * (n - nu - 1) + d * (nd - 1) * (n - nd - 1)) / 4
        return dict(bytes=case["count"] * (32 + 17.0 * pairs), flops=0)
    dets = case["dets"] if "dets" in case else space(n, ne, case["eps_var"])
    nnz = dets * row(n, ne, dets)
    value = 8 if case.get("prec") == "fp64" else 4
    if kind == "hv":  # columns and values once, both vectors
        return dict(bytes=nnz * (4 + value) + 24 * dets, flops=4 * nnz)
    if kind == "step":  # the list in; elements written (with the residual); 9 products; the correction
        return dict(bytes=24 * dets + nnz * 12 + 9 * (nnz * (4 + value) + 80 * dets) + nnz * 8, flops=40 * nnz)
    if kind == "variation":  # the last list's elements once, four Davidson calls' products
        return dict(bytes=nnz * 12 + 30 * nnz * (4 + value) + 40 * dets, flops=130 * nnz)
    if kind == "rdm":  # columns once, both strings and a coefficient of each determinant, the RDMs
        return dict(bytes=nnz * 4 + 24 * dets + 8 * n ** 2 + 4 * n ** 4, flops=10 * nnz)
    # PT2: the candidates in each window, 24 bytes (key and value) each, and the determinants
    cand = dets * ne * ne * 4.0 * (1e-6 / case["eps_pt"]) ** 0.5 * (12 if kind == "pt2" else 1)
    return dict(bytes=24.0 * (cand + dets), flops=0)


# ---- the same values in 64 bits, in plain torch -------------------------------------------------


def _popc(x):
    x = x - ((x >> 1) & 0x5555555555555555)
    x = (x & 0x3333333333333333) + ((x >> 2) & 0x3333333333333333)
    x = (x + (x >> 4)) & 0x0F0F0F0F0F0F0F0F
    x = x + (x >> 8)
    x = x + (x >> 16)
    return (x + (x >> 32)) & 0x7F


def _low(x):
    """Index of the lowest set bit."""
    return torch.log2((x & -x).double()).round().long()


def _between(s, a, b):
    """Parity of the electrons of s strictly between orbitals a and b."""
    lo, hi = torch.minimum(a, b), torch.maximum(a, b)
    one = torch.ones_like(lo)
    return _popc(s & ((one << hi) - 1) & ~((one << (lo + 1)) - 1)) & 1


def _occ(x, n):
    return ((x[:, None] >> torch.arange(n, device=x.device)) & 1).double()


class Exact:
    """Slater-Condon elements in FP64 (torch, on the GPU)."""

    def __init__(self, h, g):
        self.n = len(h)
        self.h, self.g = torch.from_numpy(h).cuda(), torch.from_numpy(g).cuda()
        self.D = torch.einsum("ijoo->ijo", self.g).contiguous()
        self.X = torch.einsum("iooj->ijo", self.g).contiguous()
        self.J = torch.einsum("aabb->ab", self.g)
        self.K = torch.einsum("abba->ab", self.g)

    def diag(self, u, d):
        a, b = _occ(u, self.n), _occ(d, self.n)
        e = (a + b) @ torch.diagonal(self.h) + ((a @ self.J) * b).sum(1)
        return e + 0.5 * (((a @ (self.J - self.K)) * a).sum(1) + ((b @ (self.J - self.K)) * b).sum(1))

    def single(self, same, oppo, p, q):
        s = _occ(same, self.n)
        s[torch.arange(len(p), device=p.device), p] = 0
        e = self.h[p, q] + ((self.D[p, q] - self.X[p, q]) * s).sum(1) + (self.D[p, q] * _occ(oppo, self.n)).sum(1)
        return e * (1 - 2 * _between(same, p, q)).double()

    def pair(self, s, t):
        """Two electrons of one string moved: s -> t."""
        x = s ^ t
        l, r = s & x, t & x
        l0, r0 = _low(l), _low(r)
        l1, r1 = _low(l & (l - 1)), _low(r & (r - 1))
        one = torch.ones_like(l0)
        par = sum(_popc(v & ((one << k) - 1)) for v, k in ((s, l0), (s, l1), (t, r0), (t, r1))) & 1
        return (self.g[l0, r0, l1, r1] - self.g[l0, r1, l1, r0]) * (1 - 2 * par).double()

    def elems(self, ui, di, uj, dj):
        xu, xd = ui ^ uj, di ^ dj
        nu, nd = _popc(xu), _popc(xd)
        out = torch.zeros(len(ui), dtype=torch.float64, device=ui.device)

        def put(mask, f):
            k = mask.nonzero()[:, 0]
            if len(k):
                out[k] = f(ui[k], di[k], uj[k], dj[k])

        put((nu + nd) == 0, lambda a, b, c, d: self.diag(a, b))
        put((nu == 2) & (nd == 0), lambda a, b, c, d: self.single(a, b, _low(a & ~c), _low(c & ~a)))
        put((nu == 0) & (nd == 2), lambda a, b, c, d: self.single(b, a, _low(b & ~d), _low(d & ~b)))
        put((nu == 4) & (nd == 0), lambda a, b, c, d: self.pair(a, c))
        put((nu == 0) & (nd == 4), lambda a, b, c, d: self.pair(b, d))

        def mixed(a, b, c, d):
            p, q, r, t = _low(a & ~c), _low(c & ~a), _low(b & ~d), _low(d & ~b)
            return self.g[p, q, r, t] * (1 - 2 * (_between(a, p, q) ^ _between(b, r, t))).double()

        put((nu == 2) & (nd == 2), mixed)
        return out


def _dev(x):
    return torch.from_numpy(np.ascontiguousarray(x).view(np.int64)).cuda()


def _connected(u, d, n, common):
    """Row, column of every ordered pair that shares at least `common` electrons, in blocks."""
    o = torch.cat([_occ(u, n), _occ(d, n)], 1).half()
    m = len(u)
    step = max(1, min(m, 400_000_000 // m))
    for b in range(0, m, step):
        k = (o[b:b + step] @ o.T >= common).nonzero()
        yield k[:, 0] + b, k[:, 1]


def _exact_hv(E, u, d, x, ne):
    y = E.diag(u, d) * x
    for i, j in _connected(u, d, E.n, ne - 2):
        k = i != j
        i, j = i[k], j[k]
        y.index_add_(0, i, E.elems(u[i], d[i], u[j], d[j]) * x[j])
    return y


def _exact_rdm(u, d, c, n, ne):
    # 1-RDM from the pairs one move apart
    o = _occ(u, n) + _occ(d, n)
    one = torch.diag((c * c) @ o).reshape(-1).clone()
    for i, j in _connected(u, d, n, ne - 1):
        k = i != j
        i, j = i[k], j[k]
        up = u[i] != u[j]
        s, t = torch.where(up, u[i], d[i]), torch.where(up, u[j], d[j])
        p, r = _low(s & ~t), _low(t & ~s)
        one.index_add_(0, p * n + r, c[i] * c[j] * (1 - 2 * _between(s, p, r)).double())
    # 2-RDM from Phi_PQ = a_Q a_P Psi over the spin orbitals P < Q (alpha ones first)
    w = 2 * n
    det = u | (d << n)
    orbs = _occ(det, w).nonzero()[:, 1].reshape(len(u), ne)
    core, pair, amp = [], [], []
    for a in range(ne):
        for b in range(a + 1, ne):
            p, q = orbs[:, a], orbs[:, b]
            bit = torch.ones_like(p)
            core.append(det ^ (bit << p) ^ (bit << q))
            pair.append(p * w + q)
            # a_P passes a electrons, then a_Q passes b - 1
            amp.append(c * (-1.0) ** (a + b - 1))
    core, pair, amp = torch.cat(core), torch.cat(pair), torch.cat(amp)
    core, k = core.sort()
    pair, amp = pair[k], amp[k]
    phi = torch.zeros(w * w, w * w, dtype=torch.float64, device=u.device).reshape(-1)
    at = torch.arange(len(core), device=u.device)
    phi.index_add_(0, pair * (w * w) + pair, amp * amp)
    shift = 1
    while len(at):
        at = at[at + shift < len(core)]
        at = at[core[at] == core[at + shift]]
        v = amp[at] * amp[at + shift]
        phi.index_add_(0, pair[at] * (w * w) + pair[at + shift], v)
        phi.index_add_(0, pair[at + shift] * (w * w) + pair[at], v)
        shift += 1
    t = phi.reshape(w, w, w, w)
    t = t - t.transpose(0, 1)
    t = t - t.transpose(2, 3)
    # Gamma(p, q, r, s) = sum over spins of <a+_p a+_q a_r a_s> = <Phi_pq, Phi_sr>
    t = t.reshape(2, n, 2, n, 2, n, 2, n)
    gam = sum(t[a, :, b, :, a, :, b, :] for a in (0, 1) for b in (0, 1))  # [p, q, s, r]
    gam = gam.permute(0, 2, 1, 3).reshape(n * n, n * n)  # [(p, s), (q, r)]
    i, j = torch.tril_indices(n * n, n * n, device=u.device)
    return one.reshape(n, n), gam[i, j]


def _exact_dtm(E, u, d, c, e_var, eps, n, nu, nd):
    dev = u.device
    known = (u | (d << n)).sort()[0]
    orb = torch.arange(n, device=dev)

    def moves(s, ns):
        """Single moves of each string: from, to, new string, sign; [len(s), ns (n - ns)]."""
        o = _occ(s, n)
        f, t = o.nonzero()[:, 1].reshape(-1, ns), (1 - o).nonzero()[:, 1].reshape(-1, n - ns)
        f = f[:, :, None].expand(-1, -1, n - ns).reshape(len(s), -1)
        t = t[:, None, :].expand(-1, ns, -1).reshape(len(s), -1)
        b = torch.ones_like(f)
        return f, t, s[:, None] ^ (b << f) ^ (b << t), (1 - 2 * _between(s[:, None].expand_as(f), f, t)).double()

    keys, vals = [], []

    def keep(cu, cd, hc):
        k = hc.abs() >= eps
        key = (cu | (cd << n))[k]
        at = torch.searchsorted(known, key).clamp_(max=len(known) - 1)
        new = known[at] != key
        keys.append(key[new])
        vals.append(hc[k][new])

    step = max(1, 20_000_000 // (nu * (n - nu) * nd * (n - nd)))
    for b in range(0, len(u), step):
        a, q, ci = u[b:b + step], d[b:b + step], c[b:b + step]
        fa, ta, sa, ga = moves(a, nu)
        fb, tb, sb, gb = moves(q, nd)
        m, ka, kb = len(a), fa.shape[1], fb.shape[1]
        A, Q = a[:, None], q[:, None]
        for s, o, f, t, new, k, alpha in ((A, Q, fa, ta, sa, ka, True), (Q, A, fb, tb, sb, kb, False)):
            s2, o2 = s.expand(m, k).reshape(-1), o.expand(m, k).reshape(-1)
            hc = E.single(s2, o2, f.reshape(-1), t.reshape(-1)) * ci[:, None].expand(m, k).reshape(-1)
            keep(*((new.reshape(-1), o2) if alpha else (o2, new.reshape(-1))), hc)
        # one electron of each spin
        hc = E.g[fa[:, :, None], ta[:, :, None], fb[:, None, :], tb[:, None, :]]
        hc = hc * ga[:, :, None] * gb[:, None, :] * ci[:, None, None]
        k = (hc.abs() >= eps).nonzero()
        keep(sa[k[:, 0], k[:, 1]], sb[k[:, 0], k[:, 2]], hc[k[:, 0], k[:, 1], k[:, 2]])
        # two electrons of one string
        for s, o, ns, alpha in ((a, q, nu, True), (q, a, nd, False)):
            if ns < 2:
                continue
            oc = _occ(s, n)
            f, t = oc.nonzero()[:, 1].reshape(m, ns), (1 - oc).nonzero()[:, 1].reshape(m, n - ns)
            i, j = torch.triu_indices(ns, ns, 1, device=dev)
            x, y = torch.triu_indices(n - ns, n - ns, 1, device=dev)
            bit = torch.ones((), dtype=torch.int64, device=dev)
            out = (bit << f[:, i]) | (bit << f[:, j])
            put = (bit << t[:, x]) | (bit << t[:, y])
            new = (s[:, None, None] ^ out[:, :, None]) | put[:, None, :]
            shape = new.shape
            s2 = s[:, None, None].expand(shape).reshape(-1)
            hc = E.pair(s2, new.reshape(-1)) * ci[:, None, None].expand(shape).reshape(-1)
            o2 = o[:, None, None].expand(shape).reshape(-1)
            keep(*((new.reshape(-1), o2) if alpha else (o2, new.reshape(-1))), hc)
    key, inv = torch.unique(torch.cat(keys), return_inverse=True)
    tot = torch.zeros(len(key), dtype=torch.float64, device=dev).index_add_(0, inv, torch.cat(vals))
    full = (1 << n) - 1
    total = 0.0
    for b in range(0, len(key), 1 << 22):
        k = key[b:b + (1 << 22)]
        total += float((tot[b:b + (1 << 22)] ** 2 / (e_var - E.diag(k & full, k >> n))).sum())
    return total


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("elems", "hv", "rdm", "dtm"):
        return None  # lists and samples, or the end of an iteration that stops at a tolerance
    n, nu, nd = case["n"], case["n_up"], case["n_dn"]
    s = prepare(case, seed)
    h, g = integrals(n, (nu + nd) // 2, seed)
    E = Exact(h, g)
    if kind == "elems":
        return E.elems(*(_dev(v) for v in s["args"]))
    up, dn, c = s["ctx"].dets()
    u, d, c = _dev(up), _dev(dn), torch.from_numpy(c).cuda()
    s["ctx"].close()
    if kind == "hv":
        return _exact_hv(E, u, d, s["x"], nu + nd) if len(u) < 900_000 else None
    if kind == "rdm":
        if 2 * n > 62 or len(u) > 400_000:
            return None
        return list(_exact_rdm(u, d, c, n, nu + nd))
    if 2 * n > 62 or len(u) * (nu * (n - nu) + nd * (n - nd)) ** 2 > 2e10:
        return None
    return [_exact_dtm(E, u, d, c, s["e"], case["eps_pt"], n, nu, nd), None]
