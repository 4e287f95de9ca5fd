"""The work whose speed counts: cutoff steps of pf-FRG flows through the package's public entry points.

A case is a stretch of a flow as a user's program runs it: the state goes to the GPU, the flow takes a few
cutoff steps (right-hand side, measurement, divergence check, Euler update) and the correlations at every
cutoff and the final state come back.  The cases cover the SU(2), XYZ and TRI cores, a batch of SU(2) flows and
the FP64 flow; from flows of a few sites and frequencies, where launches count, to the largest served ones.

`exact` restates the flow equations, the measurement and the Euler step in 64 bits with plain torch.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import spinparser_gb300 as spn
from spinparser_gb300.driver import run_flow

# lattice -> (resource model, its couplings); the tables of a flow depend on both and on the range
MODELS = {
    "square": ("square-j1j2heisenberg", {"j1": "1", "j2": "0.5"}),
    "cubic": ("cubic-j1j2heisenberg", {"j1": "1", "j2": "0.25"}),
    "pyrochlore": ("pyrochlore-j1j2heisenberg", {"j1": "1", "j2": "0.25"}),
    "kitaev": ("honeycomb-kitaev", {"j": "0.1", "k": "-1.0"}),
    "gamma": ("honeycomb-kitaev-gamma", {"j": "0.2", "k": "1.0", "g": "-0.1"}),
}
LATTICE = {"kitaev": "honeycomb", "gamma": "honeycomb"}


def _case(name, core, lattice, rng, n, fmin, fmax, cutoff, ratio, steps, **more):
    return dict(name=name, core=core, lattice=lattice, range=rng, n_freq=n, fmin=fmin, fmax=fmax, cutoff=cutoff,
                ratio=ratio, steps=steps, **more)


def listed():
    return [
        # one step of a very small flow: what an interactive user or a test runs, all latency
        _case("su2 square r2 n16", "su2", "square", 2, 16, 0.05, 50.0, 2.0, 0.95, 1),
        # the whole flow of the square-lattice Heisenberg antiferromagnet, from the bare couplings
        _case("su2 square r3 n32 whole flow", "su2", "square", 3, 32, 0.005, 50.0, 50.0, 0.98, 341, bare=True),
        # the single large flow, in its precision form (FP64 self-energy), in the middle of the flow
        _case("su2 cubic r6 n64", "su2", "cubic", 6, 64, 0.005, 100.0, 2.24, 0.98, 6, fp64_sigma=True),
        # the precision-stress flow, late in the flow, where most loop frequencies count
        _case("su2 pyrochlore r5 n64 late", "su2", "pyrochlore", 5, 64, 0.002, 100.0, 0.02, 0.99, 4),
        # a ragged size: an odd frequency count and 49 sites, early in the flow
        _case("su2 square r12 n47 early", "su2", "square", 12, 47, 0.005, 50.0, 12.0, 0.98, 4),
        # the largest request of the serving mix (70 sites)
        _case("su2 pyrochlore r7 n64", "su2", "pyrochlore", 7, 64, 0.005, 50.0, 0.5, 0.98, 3),
        # a parameter scan's flows advanced together
        _case("batch square scan", "batch", "square", 0, 0, 0.005, 50.0, 1.0, 0.98, 12, flows=12),
        # Heisenberg-Kitaev flow, and a small one of odd sizes
        _case("xyz honeycomb r9 n48", "xyz", "kitaev", 9, 48, 0.005, 50.0, 1.0, 0.98, 4),
        _case("xyz honeycomb r4 n21", "xyz", "kitaev", 4, 21, 0.02, 40.0, 0.4, 0.97, 2),
        # Heisenberg-Kitaev-Gamma flow, and a small one of odd sizes
        _case("tri honeycomb r9 n32", "tri", "gamma", 9, 32, 0.005, 50.0, 0.5, 0.98, 3),
        _case("tri honeycomb r4 n15", "tri", "gamma", 4, 15, 0.05, 40.0, 1.0, 0.97, 2),
        # the double-precision flow that the others' errors are stated against
        _case("su2 fp64 square r5 n32", "f64", "square", 5, 32, 0.005, 50.0, 0.7, 0.98, 2),
    ]


def draw(rng):
    core = rng.choice(["su2"] * 6 + ["batch", "xyz", "xyz", "tri", "tri", "f64"])
    n = int(round(math.exp(rng.uniform(math.log(8), math.log({"tri": 32, "xyz": 48, "f64": 24}.get(core, 64))))))
    lattice = {"xyz": "kitaev", "tri": "gamma", "batch": "square", "f64": "square"}.get(core) or rng.choice(
        ["square", "cubic", "pyrochlore"])
    top = {"square": 18, "cubic": 9, "pyrochlore": 7, "kitaev": 10, "gamma": 9}[lattice]
    r = 0 if core == "batch" else rng.randint(2, 6 if core == "f64" else top)
    fmin = math.exp(rng.uniform(math.log(0.002), math.log(0.05)))
    fmax = rng.uniform(20.0, 100.0)
    cutoff = math.exp(rng.uniform(math.log(4 * fmin), math.log(0.4 * fmax)))
    steps = {"batch": rng.randint(4, 12), "f64": 1, "tri": rng.randint(1, 3)}.get(core, rng.randint(1, 5))
    more = {"flows": rng.randint(2, 12), "seed": rng.randrange(1 << 20)} if core == "batch" else {}
    if core == "su2":
        more["fp64_sigma"] = rng.random() < 0.4
    case = _case(None, core, lattice, r, 0 if core == "batch" else n, round(fmin, 5), round(fmax, 2), round(cutoff, 4),
                 rng.choice([0.95, 0.98, 0.99]), steps, **more)
    del case["name"]
    return case


# ---------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _lattice(lattice, rng):
    model, params = MODELS[lattice]
    lat = spn.Lattice(LATTICE.get(lattice, lattice), rng, model, params)
    return lat.tables(), lat.spin_tables()


def _members(case):
    """The (range, frequency count) of each flow of a case; a scan's flows draw both."""
    if case["core"] != "batch":
        return [(case["range"], case["n_freq"])]
    g = np.random.RandomState(case.get("seed", 20261203))
    return [(int(g.choice([3, 5, 7])), int(g.choice([32, 48, 64]))) for _ in range(case["flows"])]


def _cutoffs(case):
    c = np.float32(case["cutoff"])
    out = [c]
    for _ in range(case["steps"]):
        c = np.float32(c * np.float32(case["ratio"]))
        out.append(c)
    return np.array(out, np.float32)


def _mesh(case, n):
    return spn.frequency_exponential(case["fmin"], case["fmax"], n)


def _vertex(g, mesh, comps, nl, scale, antisym, bare):
    """A vertex as flows have it: couplings that fall off with the distance, dressed by smooth functions of the
    three transfer frequencies (symmetric, or for `antisym` components antisymmetric, in s and u)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n = len(mesh)
    w = torch.tensor(mesh.astype(np.float64), device=dev)
    si = torch.tensor([s for s in range(n) for u in range(s + 1)], device=dev)
    ui = torch.tensor([u for s in range(n) for u in range(s + 1)], device=dev)
    fall = np.exp(-np.arange(nl) / (0.2 * nl + 1.0))
    out = []
    for c in range(comps):
        amp = torch.tensor(scale[c] * fall * g.uniform(0.5, 1.0, nl) * g.choice([-1.0, 1.0], nl), device=dev)
        v = torch.zeros(n * (n + 1) // 2, n, nl, dtype=torch.float64, device=dev)
        if bare:
            v += 0.0 if antisym[c] else amp * torch.tensor(np.arange(nl) == 1, device=dev)
        else:
            for _ in range(2):
                b = g.uniform(0.2, 5.0, 3)
                site = amp * torch.tensor(g.uniform(0.3, 1.0, nl), device=dev)
                f, h = b[0] ** 2 / (w ** 2 + b[0] ** 2), b[1] / (w + b[1])
                su = f[si] * h[ui] - h[si] * f[ui] if antisym[c] else f[si] * f[ui] + 0.5 * (h[si] + h[ui])
                v += su[:, None, None] * (1.0 + b[2] / (w + b[2]))[None, :, None] * site
        out.append(v.reshape(-1, nl).float())
    return torch.stack(out)


def _inputs(case, seed):
    """Per flow: lattice tables, spin tables, mesh, self-energy and vertex (components first)."""
    found = []
    for k, (rng, n) in enumerate(_members(case)):
        tab, spin = _lattice(case["lattice"], rng)
        g = np.random.RandomState((seed * 1009 + k) % (1 << 32))
        mesh = _mesh(case, n)
        w = mesh.astype(np.float64)
        b, bare = g.uniform(0.3, 1.5), case.get("bare", False)
        v2 = np.zeros(n, np.float32) if bare else (g.uniform(0.1, 0.3) * w / (w * w + b * b)).astype(np.float32)
        if case["core"] == "tri":
            scale = [0.3 if a == b else 0.02 for a in range(4) for b in range(4)]
            antisym = [b == 3 for a in range(4) for b in range(4)]
        elif case["core"] == "xyz":
            scale, antisym = [0.3, 0.25, 0.35, 0.1], [False, False, False, True]
        else:
            scale, antisym = [0.9 if bare else 0.3, 0.1], [False, True]
        found.append((tab, spin, mesh, v2, _vertex(g, mesh, len(scale), tab.n_sites, scale, antisym, bare)))
    return found


def _host(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=torch.cuda.is_available())
    h.copy_(t)
    return h.numpy()


def prepare(case, seed):
    core, cut = case["core"], _cutoffs(case)
    flows = _inputs(case, seed)
    if core == "batch":
        members = [(tab, mesh, v2, *_host(v).reshape(2, -1)) for tab, _, mesh, v2, v in flows]
        return {"core": core, "cut": cut, "batch": spn.Su2Batch(), "flows": members}
    tab, spin, mesh, v2, v = flows[0]
    st = {"core": core, "cut": cut, "v2": v2}
    if core == "su2":
        st["flow"] = spn.Su2Flow(tab, mesh, flags=spn.FP64_SELF_ENERGY if case.get("fp64_sigma") else 0)
        st["v4"] = _host(v).reshape(2, -1)
        st["out"] = [_host(torch.zeros(k)) for k in (len(mesh), v[0].numel(), v[0].numel())]
    elif core == "f64":
        st["flow"] = spn.Su2Flow(tab, mesh, flags=spn.FP64)
        st["v2"], st["v4"] = v2.astype(np.float64), v.cpu().numpy().astype(np.float64).reshape(2, -1)
    elif core == "xyz":
        st["flow"], st["v4"] = spn.XyzFlow(tab, spin, mesh), _host(v).reshape(4, -1)
    else:  # the TRI vertex is one array [F_N][16][Nl]
        st["flow"], st["v4"] = spn.TriFlow(tab, spin, mesh), _host(v.transpose(0, 1).contiguous()).reshape(-1)
    return st


def run(st):
    core, cut = st["core"], st["cut"]
    if core == "batch":
        b = st["batch"]
        ids = [b.add(tab, mesh, cut, (v2, ss, dd)) for tab, mesh, v2, ss, dd in st["flows"]]
        b.run()
        out = []
        for i in ids:
            r = b.result(i)
            _, v2, ss, dd = b.state(i)
            out.append({"zz": r.zz, "dd": r.dd, "v2": v2, "v4ss": ss, "v4dd": dd})
            b.remove(i)
        return out
    f = st["flow"]
    if core == "su2":
        _, zz, dd, chi_zz, chi_dd, _ = run_flow(f, cut, (st["v2"], *st["v4"]))
        _, v2, ss, den = f.get_state(*st["out"])
        return {"zz": zz, "dd": dd, "chi_zz": chi_zz, "chi_dd": chi_dd, "v2": v2, "v4ss": ss, "v4dd": den}
    if core == "f64":
        f.set_state_f64(float(cut[0]), st["v2"], *st["v4"])
        zz, dd = [], []
        for c in cut[1:]:
            f.compute_step()
            z, d, _, _ = f.measure_correlation_f64()
            zz.append(z), dd.append(d)
            f.finalize_step(float(c))
        z, d, _, _ = f.measure_correlation_f64()
        zz.append(z), dd.append(d)
        _, v2, ss, den = f.get_state_f64()
        return {"zz": np.array(zz), "dd": np.array(dd), "v2": v2, "v4ss": ss, "v4dd": den}
    _, corr, _ = f.run(cut, st["v2"], st["v4"])
    _, v2, v4 = f.get_state()
    return {"corr": corr, "v2": v2, "v4": v4}


# ---------------------------------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------------------------------
def _node_counts(mesh, cut):
    """Loop frequencies of each transfer frequency's integrals, summed over the cutoffs."""
    w = mesh.astype(np.float64)
    return sum(np.array([len(_nodes(w, x, float(c))[0]) for x in w]) for c in cut)


def work(case):
    cut, n_bytes, flops = _cutoffs(case), 0.0, 0.0
    comps = {"xyz": 4, "tri": 16}.get(case["core"], 2)
    # per site and loop frequency of a triple: 16 supports read for the s and u channels of two triples
    # and 8 for the t channel, and the channels' products; per loop frequency, the lattice sum's products
    site = {2: 24 * 4 + 60, 4: 24 * 8 + 140, 16: 24 * 32 + 4096}[comps]
    pair = {2: 4, 4: 8, 16: 256}[comps]
    for rng, n in _members(case):
        tab, _ = _lattice(case["lattice"], rng)
        mesh = _mesh(case, n)
        some = cut[:-1] if len(cut) < 40 else cut[:-1:10]
        nodes = _node_counts(mesh, some).sum() * (len(cut) - 1) / len(some)
        nl, fn = tab.n_sites, n * n * (n + 1) // 2
        pairs = len(np.unique(np.stack([np.repeat(np.arange(nl), np.diff(tab.overlap_ptr)), tab.overlap_rid1,
                                        tab.overlap_rid2]), axis=1).T)
        pairs = min(pairs, nl * nl) if comps == 2 else len(tab.overlap_rid1)
        flops += nodes * n * (n + 1) / 2 * (nl * site + pairs * pair)
        n_bytes += (8 if case["core"] == "f64" else 4) * comps * fn * nl * (2.0 + 3.0 * (len(cut) - 1))
    return {"bytes": n_bytes, "flops": flops}


# ---------------------------------------------------------------------------------------------------
# the flow in 64 bits
# ---------------------------------------------------------------------------------------------------
PERMS = [[0, 1, 2], [0, 2, 1], [1, 0, 2], [1, 2, 0], [2, 0, 1], [2, 1, 0]]


def _trapezoid(points):
    p = np.asarray(points)
    w = np.zeros(len(p))
    d = np.diff(p)
    w[:-1] += 0.5 * d
    w[1:] += 0.5 * d
    return p, w


def _nodes(w, x, cut):
    """(frequency, weight) of the trapezoid rules of transfer frequency x: the three ranges of the loop frequency
    in which it and its sum with x lie above the cutoff in magnitude.  The rules end at the mesh's last point."""
    full = np.concatenate([-w[::-1], w])
    p, q = [], []

    def add(points):
        a, b = _trapezoid(points)
        p.append(a), q.append(b)

    lo, hi = cut, cut + x
    if hi < w[-1]:
        add(np.append(full[full < -hi], -hi))
    if x - lo > lo:
        add(np.concatenate([[lo - x], full[(full > lo - x) & (full < -lo)], [-lo]]))
    if lo < w[-1]:
        add(np.append(lo, full[full > lo]))
    return (np.concatenate(p), np.concatenate(q)) if p else (np.zeros(0), np.zeros(0))


class _Exact:
    """One flow in 64 bits: V[s(s+1)/2 + u, t, component, site], on the mesh w."""

    def __init__(self, core, tab, spin, mesh, v2, v4):
        self.core = core
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        T = functools.partial(torch.as_tensor, device=self.dev)
        self.w = mesh.astype(np.float64)
        self.n, self.nl, self.C = len(mesh), tab.n_sites, v4.shape[0]
        n, nl, C = self.n, self.nl, self.C
        self.mesh = T(self.w)
        self.v2 = v2.astype(np.float64)
        self.V = v4.double().to(self.dev).reshape(C, n * (n + 1) // 2, n, nl).permute(1, 2, 0, 3).contiguous()
        second = [c == 1 for c in range(2)] if C == 2 else [c == 3 for c in range(4)] if C == 4 else [c % 4 == 3 for c in range(16)]
        first = second if C < 16 else [c // 4 == 3 for c in range(16)]
        self.swap = T(np.where(second, -1.0, 1.0))        # s and u exchanged: by the stored second component
        self.swap_first = T(np.where(first, -1.0, 1.0))
        mixed = [C == 16 and (c // 4 == 3) != (c % 4 == 3) for c in range(C)]
        self.tu = T(np.where(mixed, -1.0, 1.0))           # exactly one of t and u negated

        def bundle(site, perm, exchange):
            m = np.empty((C, nl), np.int64)
            for c in range(C):
                for j in range(nl):
                    pc = PERMS[perm[j]] + [3]
                    if C == 2:
                        k = c
                    elif C == 4:
                        k = pc[c]
                    else:
                        a, b = (c % 4, c // 4) if exchange else (c // 4, c % 4)
                        k = 4 * pc[a] + pc[b]
                    m[c, j] = k * nl + site[j]
            return T(m.reshape(-1))

        self.plain = bundle(tab.sites_rid, spin.sites_perm, False)
        self.exch = bundle(tab.inv_sites_rid, spin.inv_sites_perm, True)
        self.range_rid, self.range_inv = T(tab.range_rid.astype(np.int64)), T(tab.range_inv_rid.astype(np.int64))
        # correlation entries: component c of entry q is component perm(c) of its representative
        self.corr = [(PERMS[p] + [3], int(r)) for p, r in zip(spin.corr_perm, tab.corr_rid)]
        self.rpa = self._rpa_matrix(tab, spin)

    def _rpa_matrix(self, tab, spin):
        """The lattice sum as a sparse map from the outer product of two slabs, [(C Nl) x (C Nl)], to the flow."""
        C, nl = self.C, self.nl
        rows, cols, vals = [], [], []
        owner = np.repeat(np.arange(nl), np.diff(tab.overlap_ptr)).astype(np.int64)
        r1, r2 = tab.overlap_rid1.astype(np.int64), tab.overlap_rid2.astype(np.int64)
        four = np.array([p + [3] for p in PERMS])
        p1, p2 = four[spin.overlap_perm1], four[spin.overlap_perm2]

        def add(c, a, b, v):
            rows.append(c * nl + owner)
            cols.append((a * nl + r1) * (C * nl) + b * nl + r2)
            vals.append(np.full(len(owner), v))

        if C == 2:
            add(0, 0, 0, 1.0), add(1, 1, 1, 4.0)
        elif C == 4:
            for c in range(4):
                add(c, p1[:, c], p2[:, c], 1.0)
        else:
            for c in range(16):
                for k in range(4):
                    a, b = c // 4, c % 4
                    add(c, 4 * p1[:, a] + p1[:, k], 4 * p2[:, k] + p2[:, b], _rpa_sign(c, k))
        idx = np.stack([np.concatenate(rows), np.concatenate(cols)])
        m = torch.sparse_coo_tensor(torch.as_tensor(idx), torch.as_tensor(np.concatenate(vals)), (C * nl, (C * nl) ** 2))
        return m.coalesce().to_sparse_csr().to(self.dev)

    # ---- reads -------------------------------------------------------------------------------
    def _interp(self, x):
        """Mesh cell of |x| and the position in it; constant beyond the mesh's ends."""
        a, n = x.abs(), self.n
        hi = torch.searchsorted(self.mesh, a.contiguous(), right=True).clamp(1, n - 1)
        lo = hi - 1
        b = (a - self.mesh[lo]) / (self.mesh[hi] - self.mesh[lo])
        return lo, hi, b.clamp(0.0, 1.0)

    def _slabs(self, s, t, u, known, local=False):
        """Interpolated slab [..., C, Nl] (or with `local` [..., C] of site 0, in both swap conventions) at (s, t, u);
        `known` = (axis, index) for a coordinate that is a mesh value.  Also the exchange and t-u flags."""
        flags = (s < 0) ^ (u < 0), (t < 0) ^ (u < 0)
        shape = torch.broadcast_shapes(s.shape, t.shape, u.shape)
        axes = []
        for k, x in enumerate((s, t, u)):
            if known is not None and known[0] == k:
                axes.append([(known[1].expand(shape), None)])
            else:
                lo, hi, b = self._interp(x.expand(shape))
                axes.append([(lo, 1.0 - b), (hi, b)])
        V = self.V.reshape(-1, self.C, self.nl)
        total = second = None
        for si, ws in axes[0]:
            for ti, wt in axes[1]:
                for ui, wu in axes[2]:
                    weight = 1.0
                    for x in (ws, wt, wu):
                        weight = x * weight if x is not None else weight
                    big, small = torch.maximum(si, ui), torch.minimum(si, ui)
                    at = ((big * (big + 1) // 2 + small) * self.n + ti)
                    swapped = (si < ui)[..., None]
                    v = V[:, :, 0][at] if local else V[at]
                    if local:
                        w1 = weight[..., None] * torch.where(swapped, self.swap_first, 1.0)
                        second = v * w1 if second is None else second + v * w1
                        v = v * (weight[..., None] * torch.where(swapped, self.swap, 1.0))
                    else:
                        v = v * (weight[..., None] * torch.where(swapped, self.swap, 1.0))[..., None]
                    total = v if total is None else total.add_(v)
        return (total, second, *flags) if local else (total, *flags)

    def bundle(self, s, t, u, known):
        v, ex, tu = self._slabs(s, t, u, known)
        f = v.reshape(*v.shape[:-2], self.C * self.nl)
        f = torch.where(ex[..., None], f[..., self.exch], f[..., self.plain]).reshape(v.shape)
        if self.C == 16:
            f = f * torch.where(tu[..., None], self.tu, 1.0)[..., None]
        return f

    def local(self, s, t, u, known=None):
        a, b, ex, tu = self._slabs(s, t, u, known, local=True)
        if self.C < 16:
            return a
        b = b.reshape(*b.shape[:-1], 4, 4).transpose(-1, -2).reshape(b.shape)
        return torch.where(ex[..., None], b, a) * torch.where(tu[..., None], self.tu, 1.0)

    def value(self, c, r12, r21, s, t, u):
        """Component c of pairs (r12, exchanged r21) at each (s, t, u), for a component that is its own exchange."""
        v, ex, _ = self._slabs(*(torch.as_tensor(x, dtype=torch.float64, device=self.dev) for x in (s, t, u)), None)
        return torch.where(ex[..., None], v[..., c, r21], v[..., c, r12])

    # ---- self-energy, propagators ------------------------------------------------------------
    def odd(self, data, x):
        x = np.asarray(x, np.float64)
        return np.sign(x) * np.interp(np.abs(x), self.w, data)

    def self_energy(self, L):
        d, p, m, z = self.C - 1, self.w + L, self.w - L, np.zeros(self.n)
        zero = torch.zeros(1, dtype=torch.int64, device=self.dev)
        onsite = {2: [(0, 0.75), (1, 1.0)], 4: [(c, 1.0) for c in range(4)], 16: [(5 * c, 1.0) for c in range(4)]}[self.C]
        val = -2.0 * (self.value(d, self.range_rid, self.range_inv, p, z, m) - self.value(d, self.range_rid, self.range_inv, m, z, p)).sum(1)
        for c, f in onsite:
            val = val + f * (self.value(c, zero, zero, p, m, z) - self.value(c, zero, zero, m, p, z))[:, 0]
        return val.cpu().numpy() / (2 * math.pi * (L + self.odd(self.v2, L)))

    def node_tables(self, L, dv2):
        rows = []
        prop = lambda a: 1.0 / (a + self.odd(self.v2, a))  # noqa: E731
        for x in self.w:
            f, c = [np.array([L])], [np.array([prop(L) * prop(L + x)])]
            if x > 2 * L:
                f.append(np.array([-L])), c.append(np.array([prop(L) * prop(L - x)]))
            p, q = _nodes(self.w, x, L)
            f.append(p), c.append(q * self.odd(dv2, p) * prop(p) ** 2 * prop(x + p))
            rows.append((np.concatenate(f), np.concatenate(c)))
        k = max(len(f) for f, _ in rows)
        wp, cf = np.zeros((self.n, k)), np.zeros((self.n, k))
        for i, (f, c) in enumerate(rows):
            wp[i, : len(f)], cf[i, : len(f)] = f, c
        return torch.as_tensor(wp, device=self.dev), torch.as_tensor(cf, device=self.dev)

    # ---- vertex flow -------------------------------------------------------------------------
    def vertex_flow(self, L, dv2):
        wp, cf = self.node_tables(L, dv2)
        n, C, nl = self.n, self.C, self.nl
        out = torch.empty(n * (n + 1) // 2 * n, C, nl, dtype=torch.float64, device=self.dev)
        su_s = torch.tensor([s for s in range(n) for _ in range(s + 1)], device=self.dev)
        su_u = torch.tensor([u for s in range(n) for u in range(s + 1)], device=self.dev)
        step = max(1, int(6e7 / (wp.shape[1] * C * nl)))
        for a in range(0, len(out), step):
            it = torch.arange(a, min(len(out), a + step), device=self.dev)
            i = [x[:, None] for x in (su_s[it // n], it % n, su_u[it // n])]
            s, t, u = (self.mesh[x] for x in i)
            w1p, w1, w2p, w2 = (0.5 * x for x in (s + t + u, s - t + u, s - t - u, s + t - u))
            q, c = wp[i[0][:, 0]], cf[i[0][:, 0]]
            k = (0, i[0])
            S = [self.bundle(s, -w1 - q, -w2 - q, k), self.bundle(s, w1p + q, -w2p - q, k),
                 self.bundle(s, w2 + q, w1 + q, k), self.bundle(s, -w2p - q, w1p + q, k)]
            total = (self._ladder(S, False) * c[..., None, None]).sum(1)
            q, c = wp[i[2][:, 0]], cf[i[2][:, 0]]
            k = (2, i[2])
            S = [self.bundle(w1 + q, q - w2p, u, k), self.bundle(w1p + q, w2 - q, u, k),
                 self.bundle(w2p - q, -w1 - q, u, k), self.bundle(w2 - q, w1p + q, u, k)]
            total -= (self._ladder(S, True) * c[..., None, None]).sum(1) * (1.0 if C == 2 else -1.0)
            q, c = wp[i[1][:, 0]], cf[i[1][:, 0]]
            k = (1, i[1])
            S = [self.bundle(w1 - q, t, w1p + q, k), self.bundle(w2p - q, t, -w2 - q, k),
                 self.bundle(w1p + q, t, w1 - q, k), self.bundle(w2 + q, t, q - w2p, k)]
            k = (2, i[1])
            loc = [self.local(w2p - q, -w2 - q, t, k), self.local(w1 - q, -w1p - q, -t, k),
                   self.local(w2 + q, q - w2p, t, k), self.local(w1p + q, q - w1, -t, k)]
            total += (self._chalice(S, loc) * c[..., None, None]).sum(1) + self._rpa_sum(S, c)
            out[it] = total / (2 * math.pi)
        return out.reshape(self.V.shape)

    def _ladder(self, S, hole):
        if self.C == 2:
            (a, h), (b, k), (c, l), (d, m) = (x.unbind(-2) for x in S)
            x = h * b + l * d + a * k + c * m + (0.5 if hole else -0.5) * (a * b + c * d)
            return torch.stack([x, 3.0 / 16.0 * (a * b + c * d) + h * k + l * m], -2)
        out = 0.0
        for A, B in ((S[0], S[1]), (S[2], S[3])):
            if self.C == 4:
                x, y, z, w = A.unbind(-2)
                p, q, r, v = B.unbind(-2)
                g = -1.0 if hole else 1.0
                out = out + torch.stack([g * (w * p + x * v) - z * q - y * r, g * (w * q + y * v) - z * p - x * r,
                                         g * (w * r + z * v) - x * q - y * p, g * (w * v + x * p + y * q + z * r)], -2)
            else:
                for a in range(16):
                    b = [a ^ c ^ 15 for c in range(16)]
                    sign = torch.tensor([float(_ladder_sign(c, a, hole)) for c in range(16)], dtype=torch.float64, device=self.dev)
                    out = out + A[..., a : a + 1, :] * B[..., b, :] * sign[:, None]
        return out

    def _chalice(self, S, loc):
        """The t channel's terms with a site-local vertex: slabs 0 and 2 on the left, 1 and 3 on the right."""
        out = 0.0
        for A, l, left in ((S[0], loc[0], True), (S[1], loc[1], False), (S[2], loc[2], True), (S[3], loc[3], False)):
            if self.C == 2:
                m = torch.stack([-l[..., 1] + 0.25 * l[..., 0], -l[..., 1] - 0.75 * l[..., 0]], -1)
                out = out + m[..., None] * A
            elif self.C == 4:
                x, y, z, d = l.unbind(-1)
                m = torch.stack([y + z - x - d, x + z - y - d, x + y - z - d, -x - y - z - d], -1)
                out = out + m[..., None] * A
            else:
                t = torch.as_tensor(_chalice_tensor(left), device=self.dev)
                out = out + torch.einsum("cal,...l->...ca", t, l) @ A
        return out

    def _rpa_sum(self, S, c):
        pairs = {2: [(2, 3, 1.0)], 4: [(0, 1, 4.0)], 16: [(0, 1, 2.0), (2, 3, 2.0)]}[self.C]
        M = 0.0
        for a, b, f in pairs:
            A = (S[a] * (f * c)[..., None, None]).flatten(-2)
            M = M + A.transpose(1, 2) @ S[b].flatten(-2)
        out = torch.empty(len(c), self.C * self.nl, dtype=torch.float64, device=self.dev)
        step = max(1, int(4e8 / M[0].numel()))
        for a in range(0, len(c), step):
            out[a : a + step] = (self.rpa @ M[a : a + step].flatten(1).t().contiguous()).t()
        return out.reshape(len(c), self.C, self.nl)

    # ---- measurement -------------------------------------------------------------------------
    def measure(self, L):
        w, C, nl = self.w, self.C, self.nl
        full = np.concatenate([-w[::-1], w])
        a = _trapezoid(np.append(full[full < -L], -L)) if L < w[-1] else (np.zeros(0), np.zeros(0))
        b = _trapezoid(np.append(L, full[full > L])) if L < w[-1] else (np.zeros(0), np.zeros(0))
        p, q = np.concatenate([a[0], b[0]]), np.concatenate([a[1], b[1]])
        g = (p + self.odd(self.v2, p)) ** -2
        T = functools.partial(torch.as_tensor, device=self.dev)
        x, y = T(p)[:, None], T(p)[None, :]
        zero = torch.zeros((), dtype=torch.float64, device=self.dev)
        f = self.bundle(x + y, zero, x - y, None)
        egg = self.local(x + y, x - y, zero)
        d = {2: [1], 4: [3], 16: [15]}[C]
        if C == 2:  # spin length 1/2
            r = f * T(np.array([-0.25, -4.0]))[:, None]
            r[..., 0, 0] += 0.5 * (-egg[..., 0] / 4 + egg[..., 1])
            r[..., 1, 0] += 0.5 * (3 * egg[..., 0] + 4 * egg[..., 1])
            on = [0.5 / (2 * math.pi), 1.0 / math.pi]
        elif C == 4:
            r = f * T(np.array([-1.0, -1.0, -1.0, -4.0]))[:, None]
            e = T(0.5 * np.array([[1, -1, -1, 1], [-1, 1, -1, 1], [-1, -1, 1, 1], [4, 4, 4, 4.0]]))
            r[..., 0] += egg @ e.t()
            on = [1 / (4 * math.pi)] * 3 + [1 / math.pi]
        else:
            r = f * T(np.where(np.arange(16) == 15, -4.0, -1.0))[:, None]
            r[..., 0] += egg @ T(_egg_matrix()).t()
            on = [1 / (4 * math.pi) if c in (0, 5, 10) else 1 / math.pi if c == 15 else 0.0 for c in range(16)]
        k = T(q * g)
        chi = (k[:, None, None, None] * k[:, None, None] * r).sum((0, 1)) / (4 * math.pi ** 2)
        chi[:, 0] += k.sum() * T(np.array(on))
        return chi.cpu().numpy()

    def correlations(self, chi):
        if self.C == 2:
            return np.array([[chi[c, r] for _, r in self.corr] for c in range(2)])
        if self.C == 4:
            return np.array([[chi[p[c], r] for p, r in self.corr] for c in range(4)])
        spin_spin = [[chi[4 * p[a] + p[b], r] for p, r in self.corr] for a in range(3) for b in range(3)]
        return np.array(spin_spin + [[chi[15, r] for _, r in self.corr]])

    def run(self, cut):
        corr, chis = [], []
        for k, c in enumerate(cut):
            L = float(c)
            chis.append(self.measure(L))
            corr.append(self.correlations(chis[-1]))
            if k + 1 < len(cut):
                dv2 = self.self_energy(L)
                dV = self.vertex_flow(L, dv2)
                step = float(cut[k + 1]) - L
                self.v2 = self.v2 + step * dv2
                self.V += step * dV
        return np.array(corr), np.array(chis)


# ---- coefficients of the 16-component flow, from Pauli products sigma_a sigma_b = i^k sigma_c (index 3: the unit) ----
def _pauli(a, b):
    """(c, k) of sigma_a sigma_b = i^k sigma_c."""
    if a == 3 or b == 3:
        return (b if a == 3 else a), 0
    if a == b:
        return 3, 0
    return 3 - a - b, 1 if (b - a) % 3 == 1 else 3


def _phase(a, b):
    """Power of i that a component with exactly one unit index carries."""
    return 3 if (a == 3) != (b == 3) else 0


def _real(k):
    return {0: 1, 2: -1}.get(k % 4, 0)


def _ladder_sign(c, a, hole):
    b = a ^ c ^ 15
    second = _pauli(b & 3, a & 3) if hole else _pauli(a & 3, b & 3)
    k = _pauli(a >> 2, b >> 2)[1] + second[1] + (2 if hole else 0)
    return _real(k + _phase(a >> 2, a & 3) + _phase(b >> 2, b & 3) - _phase(c >> 2, c & 3))


def _rpa_sign(c, k):
    return float(_real(_phase(c >> 2, k) + _phase(k, c & 3) - _phase(c >> 2, c & 3)))


@functools.lru_cache(maxsize=None)
def _chalice_tensor(left):
    """t[c, a, l]: coefficient of slab component a and site-local component l = 4 lam + rho in output c."""
    t = np.zeros((16, 16, 16))
    for c in range(16):
        for lam in range(4):
            for rho in range(4):
                kap = (c & 3 if left else c >> 2) ^ lam ^ rho
                m, k1 = _pauli(lam, kap)
                k = 2 + k1 + _pauli(m, rho)[1] + _phase(lam, rho) - _phase(c >> 2, c & 3)
                a = 4 * (c >> 2) + kap if left else 4 * kap + (c & 3)
                t[c, a, 4 * lam + rho] = _real(k + _phase(a >> 2, a & 3))
    return t


@functools.lru_cache(maxsize=None)
def _egg_matrix():
    m = np.zeros((16, 16))
    for c in range(16):
        for lam in range(4):
            rho = (c >> 2) ^ (c & 3) ^ lam
            a, k1 = _pauli(c >> 2, lam)
            b, k2 = _pauli(a, c & 3)
            e, k3 = _pauli(b, rho)
            if e == 3:
                m[c, 4 * lam + rho] = (2.0 if c == 15 else 0.5) * _real(k1 + k2 + k3 + _phase(lam, rho))
    return m


def exact(case, seed):
    core, cut, out = case["core"], _cutoffs(case), []
    # the largest stretches take longer than a check may
    if work(case)["flops"] > 4e12 and core != "tri":
        return None
    for tab, spin, mesh, v2, v4 in _inputs(case, seed):
        e = _Exact(core, tab, spin, mesh, v2, v4)
        corr, chi = e.run(cut)
        v = e.V.permute(2, 0, 1, 3).reshape(e.C, -1)
        if core == "batch":
            out.append({"zz": corr[:, 0], "dd": corr[:, 1], "v2": e.v2, "v4ss": v[0], "v4dd": v[1]})
        elif core == "f64":
            return {"zz": corr[:, 0], "dd": corr[:, 1], "v2": e.v2, "v4ss": v[0], "v4dd": v[1]}
        elif core == "su2":
            return {"zz": corr[:, 0], "dd": corr[:, 1], "chi_zz": chi[:, 0], "chi_dd": chi[:, 1], "v2": e.v2,
                    "v4ss": v[0], "v4dd": v[1]}
        elif core == "xyz":
            return {"corr": corr, "v2": e.v2, "v4": v}
        else:
            return {"corr": corr, "v2": e.v2, "v4": e.V.reshape(-1)}
    return out
