"""Performance cases of the filament step: what programs do with the library.

Every case goes through the public entry points (simcore_b200.Context, and
sc_pair_forces_noalloc for callers that own their device buffers).  The
configurations are the package's own workloads (simcore_b200/workloads.py)
at several sizes:

  kind "run"      a simulation loop: captured steps, then the positions read
                  into a pinned buffer, as a run does between two output
                  frames
  kind "host"     the two-call drop-in interface: a host program that calls
                  Interact and UpdatePositions itself, step by step, and reads
                  the bond forces and the positions
  kind "pairs"    pair forces of a configuration in the caller's own device
                  buffers
  kind "monitor"  a simulation loop with pressure records, joint-angle
                  histograms and order parameters sampled between captured runs

exact() repeats a case in 64-bit numpy: the cell list and its rebuild rule,
segment-segment distances, WCA forces with the stored forces of pairs out of
range, bending, noise from the same Philox words, both tridiagonal solves,
the midpoint update and the bond renormalisation.
"""
import ctypes
import math

import numpy as np
import torch

import simcore_b200 as sc
from simcore_b200 import workloads

DIAMETER = workloads.DIAMETER
# A rebuild every 15 or so steps and 20 steps per captured launch are the
# benchmark's own figures; the small systems run longer between two frames.


def listed():
    return [
        # One small system, the parity configuration (100 filaments of 20
        # bonds): a parameter sweep on a small box, where launches count.
        dict(name="small_fp64", kind="run", workload="A", scale=1.0, precision="fp64", steps=100),
        dict(name="small_mixed", kind="run", workload="A", scale=1.0, precision="mixed", steps=20),
        # A host program driving the two halves of the step itself.
        dict(name="drop_in_fp64", kind="host", workload="A", scale=1.0, precision="fp64", steps=4),
        # Forces of caller-owned device buffers, at an everyday size.
        dict(name="caller_buffers", kind="pairs", workload="B", scale=0.02, precision="fp64"),
        # The headline suspension (20,000 x 10 bonds) in both precisions, with
        # the integrator layouts the tuner keeps for it (block_sites), as a
        # program that tuned once sets them.
        dict(name="suspension_mixed", kind="run", workload="B", scale=1.0, precision="mixed",
             steps=20, block_sites=192),
        dict(name="suspension_fp64", kind="run", workload="B", scale=1.0, precision="fp64",
             steps=20, block_sites=128),
        # Uneven lengths (from 5 bonds up) in one nematic box, whose side is
        # longer than its longest filament.
        dict(name="uneven_mixed", kind="run", workload="C", filaments=20000, longest=200,
             precision="mixed", steps=20),
        dict(name="uneven_fp64", kind="run", workload="C", filaments=4000, longest=100,
             precision="fp64", steps=20),
        # Many independent 2D systems in one context.
        dict(name="replicas_mixed", kind="run", workload="D", replicas=64, precision="mixed",
             steps=20, block_sites=192),
        dict(name="replicas_fp64", kind="run", workload="D", replicas=16, precision="fp64",
             steps=20),
        # A crosslinked network of 50-bond filaments at the network's stable
        # time step.
        dict(name="network_mixed", kind="run", workload="E", scale=0.3, precision="mixed",
             steps=20),
        # A medium suspension watched closely: pressure every 10 steps, angle
        # histograms and order parameters at every frame.
        dict(name="monitored_fp64", kind="monitor", workload="B", scale=0.1, precision="fp64",
             steps=20),
    ]


def _between(rng, lo, hi):
    """A size between lo and hi, even over the logarithm."""
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["small", "host", "pairs", "suspension", "suspension", "uneven", "replicas",
                       "network", "monitor"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "small":
        return dict(kind="run", workload="A", scale=round(_between(rng, 0.2, 3.0), 3),
                    precision=prec, steps=rng.randrange(9, 41), n_seg=rng.randrange(7, 32))
    if kind == "host":
        return dict(kind="host", workload="A", scale=round(_between(rng, 0.3, 4.0), 3),
                    precision="fp64", steps=rng.randrange(2, 7), n_seg=rng.randrange(7, 32))
    if kind == "pairs":
        return dict(kind="pairs", workload="B", scale=round(_between(rng, 0.004, 0.02), 4),
                    precision="fp64", n_seg=rng.randrange(6, 16))
    if kind == "suspension":
        return dict(kind="run", workload="B", scale=round(_between(rng, 0.05, 0.9), 3),
                    precision=prec, steps=rng.randrange(10, 25), n_seg=rng.randrange(6, 25),
                    block_sites=rng.choice([0, 128, 192, 256]))
    if kind == "uneven":
        longest = int(_between(rng, 30, 200))
        # The fewest filaments whose box is longer than the longest of them.
        mean = (longest - 5) / math.log(longest / 5.0)
        least = (longest + 10.0) ** 3 * UNEVEN_DENSITY / mean
        return dict(kind="run", workload="C", longest=longest,
                    filaments=int(_between(rng, 1.05 * least, 20000)),
                    precision=prec, steps=rng.randrange(8, 21))
    if kind == "replicas":
        return dict(kind="run", workload="D", replicas=int(_between(rng, 3, 60)), precision=prec,
                    steps=rng.randrange(8, 21), block_sites=rng.choice([0, 128, 192, 256]))
    if kind == "network":
        return dict(kind="run", workload="E", scale=round(_between(rng, 0.06, 0.28), 4),
                    precision=prec, steps=rng.randrange(8, 21))
    return dict(kind="monitor", workload="B", scale=round(_between(rng, 0.02, 0.2), 3),
                precision="fp64", steps=2 * rng.randrange(5, 12), n_seg=rng.randrange(6, 20))


# Segments per volume of the uneven-length workload (C): 50,000 filaments of
# 5 to 200 bonds, even over the logarithm, in a cube of side 300.
UNEVEN_DENSITY = 50000 * 195 / math.log(40) / 300.0 ** 3


def _uneven_lengths(case):
    """Bonds of every filament: a property of the case, not of the seed."""
    rng = np.random.default_rng(case["filaments"])
    lo, hi = 5, case["longest"]
    return np.clip(np.round(np.exp(rng.uniform(math.log(lo), math.log(hi), case["filaments"]))),
                   lo, hi).astype(np.int32)


def _configuration(case, seed):
    """(system, filaments, sites, replicas or None) of a case.  Sizes come
    from the case alone; positions and noise keys from the seed."""
    name, seed = case["workload"], int(seed) % (1 << 20)
    if name == "C":
        n_seg = _uneven_lengths(case)
        side = (float(n_seg.sum()) / UNEVEN_DENSITY) ** (1.0 / 3.0)
        lp = np.random.default_rng(seed).uniform(10.0, 1000.0, len(n_seg))
        sites = sc.insert_filaments(3, 0.5 * side, seed, n_seg, n_seg.astype(np.float64), lp,
                                    diameter=DIAMETER, insertion="random_nematic")
        system = dict(n_dim=3, system_radius=0.5 * side, delta=5e-5, seed=seed)
        filaments = [dict(length=float(n), persistence_length=float(p), diameter=DIAMETER,
                          min_bond_length=workloads.MIN_BOND_LENGTH,
                          friction_ratio=workloads.FRICTION_RATIO) for n, p in zip(n_seg, lp)]
        return system, filaments, sites, None
    if name == "D":
        def insert(n_dim, radius, key, *args, **kw):
            return sc.insert_filaments(n_dim, radius, key + 1000 * seed, *args, **kw)
        system, filaments, sites, replicas = workloads.make_replicas(
            n_replicas=case["replicas"], insert=insert)
        replicas = [dict(r, seed=r["seed"] + 1000 * seed) for r in replicas]
        return dict(system, seed=replicas[0]["seed"]), filaments, sites, replicas
    scale = case["scale"]
    kw = {}
    if case.get("n_seg"):
        # Other filament lengths at the workload's own density of segments.
        w = workloads.WORKLOADS[name]
        kw = dict(n_seg=case["n_seg"],
                  side=w["side"] * (scale * case["n_seg"] / w["n_seg"]) ** (1.0 / 3.0))
    system, filaments, sites = workloads.make(name, scale, seed=seed, **kw)
    if name == "E":
        system = dict(system, delta=5e-5)
    return system, filaments, sites, None


def prepare(case, seed):
    system, filaments, sites, replicas = _configuration(case, seed)
    if case["kind"] == "pairs":
        offsets = np.zeros(len(filaments) + 1, dtype=np.int32)
        offsets[1:] = np.cumsum([sc.filament_n_bonds(f) + 1 for f in filaments])
        nb = int(offsets[-1]) - len(filaments)
        desc = sc.SystemDesc(n_dim=system["n_dim"], system_radius=system["system_radius"],
                             delta=system["delta"], wca_eps=1.0, wca_sig=1.0, f_cutoff=2000.0,
                             stoch_flag=1, interaction_flag=1, like_like_interactions=1,
                             seed=system["seed"], precision=0, device=0)
        return dict(case=case, desc=desc, species=sc.FilamentParams(**filaments[0]),
                    n=len(filaments), offsets=torch.from_numpy(offsets).cuda(),
                    xyz=torch.from_numpy(sites).cuda(),
                    force=torch.empty((nb, 3), dtype=torch.float64, device="cuda"),
                    torque=torch.empty((nb, 3), dtype=torch.float64, device="cuda"))
    ctx = sc.Context(system, filaments, sites, precision=case["precision"], replicas=replicas)
    links = workloads.crosslinks(case["workload"], sites, filaments,
                                 2.0 * system["system_radius"], scale=case.get("scale", 1.0),
                                 seed=int(seed) % (1 << 20))
    if links is not None:
        a, b, k, rest = links
        ctx.add_crosslinks(a, b, k_spring=k, rest_length=rest)
    if case.get("block_sites"):
        ctx.set_integrator_layout(0, case["block_sites"])
    if case["kind"] == "monitor":
        ctx.set_thermo(10)
    out = torch.empty((sites.shape[0], 3), dtype=torch.float64, pin_memory=True).numpy()
    return dict(case=case, ctx=ctx, out=out)


def run(state):
    case = state["case"]
    if case["kind"] == "pairs":
        rc = sc.lib.sc_pair_forces_noalloc(
            ctypes.byref(state["desc"]), ctypes.byref(state["species"]),
            ctypes.c_int(state["n"]), ctypes.c_void_p(state["offsets"].data_ptr()),
            ctypes.c_void_p(state["xyz"].data_ptr()), ctypes.c_void_p(state["force"].data_ptr()),
            ctypes.c_void_p(state["torque"].data_ptr()),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != sc.SC_OK:
            raise RuntimeError(sc.STATUS_NAMES.get(rc, rc))
        return {"force": state["force"], "torque": state["torque"]}
    ctx, out = state["ctx"], state["out"]
    if case["kind"] == "host":
        for _ in range(case["steps"]):
            ctx.interact()
            ctx.update_positions()
        force, torque = ctx.bond_forces()
        return {"sites": ctx.sites(out=out), "force": force, "torque": torque}
    ctx.step_graph(case["steps"])
    if case["kind"] == "monitor":
        ctx.analysis_sample(50)
        polar, nematic = ctx.global_order()
        _, _, _, hist = ctx.analysis_results(50)
        _, tensor, pressure, _ = ctx.thermo_records(64)
        return {"sites": ctx.sites(out=out), "polar": polar, "nematic": nematic,
                "angles": hist, "tensor": tensor, "pressure": pressure,
                "energy": ctx.potential_energy()}
    return {"sites": ctx.sites(out=out)}


def _sizes(case):
    """(filaments, bonds, candidate pairs) a case has on average."""
    name = case["workload"]
    if name == "D":
        w = workloads.REPLICAS["D"]
        nf = case["replicas"] * 0.5 * sum(w["n_fil"])
        per, dens, nd = w["n_seg"], w["area_fraction"] * w["n_seg"] / (w["n_seg"] + math.pi / 4), 2
    else:
        nd = 3
        if name == "C":
            nf = case["filaments"]
            per, dens = (case["longest"] - 5) / math.log(case["longest"] / 5.0), UNEVEN_DENSITY
        else:
            w = workloads.WORKLOADS[name]
            nf = max(2, round(w["n_fil"] * case["scale"]))
            per, dens = case.get("n_seg") or w["n_seg"], w["n_fil"] * w["n_seg"] / w["side"] ** 3
    cell = 2.0 ** (1.0 / 6.0)
    return nf, nf * per, nf * per * 0.5 * 3 ** nd * cell ** nd * dens


def work(case):
    """Bytes and operations one pass cannot do without.

    Per step every site is read and written with its previous position and
    projected noise (96 B), every bond's geometry is written and read and its
    force and torque accumulated (112 B, 208 B in FP64), every candidate pair
    is read (8 B); about 400 operations a site and 150 a pair.  The positions
    read at the end add 24 B a site."""
    nf, nb, pairs = _sizes(case)
    ns = nf + nb
    if case["kind"] == "pairs":
        return {"bytes": 24 * ns + 48 * nb + 4 * nf, "flops": 60 * nb + 150 * pairs}
    steps = case["steps"]
    step = 96 * ns + (208 if case["precision"] == "fp64" else 112) * nb + 8 * pairs
    return {"bytes": steps * step + 24 * ns, "flops": steps * (400 * ns + 150 * pairs)}


# ---------------------------------------------------------------------------
# 64-bit numpy restatement.

_NORMAL = 2.0 ** -32


def _philox(c, key):
    """Philox4x32-10 over arrays of counters (4) and keys (2)."""
    c = [np.asarray(v, dtype=np.uint64) for v in c]
    k = [np.asarray(v, dtype=np.uint64) for v in key]
    low = np.uint64(0xFFFFFFFF)
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ k[0], p1 & low,
             (p0 >> np.uint64(32)) ^ c[3] ^ k[1], p0 & low]
        k = [(k[0] + np.uint64(0x9E3779B9)) & low, (k[1] + np.uint64(0xBB67AE85)) & low]
    return c


def _nearest(x):
    """The reference's NINT: truncation of x + 1/2 away from zero."""
    return np.trunc(np.where(x < 0, x - 0.5, x + 0.5))


def _dot(a, b):
    return np.einsum("...i,...i->...", a, b)


class _Exact:
    """One periodic system in 64 bits: filaments padded to the longest."""

    def __init__(self, system, filaments, sites, radius, seed):
        self.nd, self.delta = system["n_dim"], system["delta"]
        self.side, self.seed = 2.0 * radius, seed
        nb = np.array([sc.filament_n_bonds(f) for f in filaments])
        length = np.array([f["length"] for f in filaments])
        self.n = n = nb + 1
        nf, m = len(n), int(n.max())
        self.j = np.arange(m)[None, :]
        self.site = self.j < n[:, None]
        self.bond = self.j < (n - 1)[:, None]
        self.r = np.zeros((nf, m, 3))
        self.r[self.site] = sites
        self.l = (length / nb)[:, None]
        self.kappa = np.array([f["persistence_length"] for f in filaments])[:, None]
        gperp = 4.0 * length / (3.0 * n * np.log(length / DIAMETER))
        gpar = gperp / workloads.FRICTION_RATIO
        self.igperp, self.dgam = (1.0 / gperp)[:, None], (1.0 / gpar - 1.0 / gperp)[:, None]
        self.sperp = np.sqrt(24.0 * gperp / self.delta)[:, None, None]
        self.spar = np.sqrt(24.0 * gpar / self.delta)[:, None, None]
        self.switch = np.ones(nf, dtype=bool)
        self.rcut2 = 2.0 ** (1.0 / 3.0)
        cell = max(math.sqrt(self.rcut2), DIAMETER, 1.5 * workloads.MIN_BOND_LENGTH)
        self.n1d = max(3, int(math.floor(self.side / cell)))
        self.limit = 0.25 * (self.side / self.n1d) ** 2
        # Global bond numbers: filament by filament.
        self.fil = np.repeat(np.arange(nf), nb)
        self.steps = self.mid = 0
        self.rp, self.noise = self.r.copy(), np.zeros_like(self.r)
        self.rebuild()

    def geometry(self):
        d = np.zeros_like(self.r)
        d[:, :-1] = self.r[:, 1:] - self.r[:, :-1]
        d[~self.bond] = 0.0
        length = np.sqrt(_dot(d, d))
        u = d / np.where(self.bond, length, 1.0)[..., None]
        return u, length, self.r + 0.5 * d

    def rebuild(self):
        _, _, pos = self.geometry()
        s = pos[self.bond][:, :self.nd] / self.side
        s = s - _nearest(s)
        c = np.minimum(np.floor(self.n1d * (s + 0.5)).astype(np.int64), self.n1d - 1)
        n1 = self.n1d
        def index(v):
            k = np.zeros(len(v), dtype=np.int64)
            for i in range(self.nd):
                k = k * n1 + v[:, i] % n1
            return k
        key = index(c)
        order = np.argsort(key, kind="stable")
        ks = key[order]
        first, second = [], []
        half = [o for o in np.ndindex(*([3] * self.nd)) if o > (1,) * self.nd]
        for off in [(1,) * self.nd] + half:
            own = off == (1,) * self.nd
            k = index(c + (np.array(off) - 1))
            lo, hi = np.searchsorted(ks, k, "left"), np.searchsorted(ks, k, "right")
            cnt = hi - lo
            a = np.repeat(np.arange(len(key)), cnt)
            b = order[np.repeat(lo - np.cumsum(cnt) + cnt, cnt) + np.arange(cnt.sum())]
            keep = a < b if own else np.ones(len(a), dtype=bool)
            first.append(a[keep])
            second.append(b[keep])
        a, b = np.concatenate(first), np.concatenate(second)
        keep = ~((np.abs(a - b) == 1) & (self.fil[a] == self.fil[b]))
        self.a, self.b = a[keep], b[keep]
        self.stored = np.zeros((len(self.a), 3))
        self.origin, self.moved = self.r.copy(), np.zeros(self.r.shape[:2])

    def interact(self):
        self.steps += 1
        if self.steps > 1 and not self.mid and self.moved.max() > self.limit:
            self.rebuild()
        u, length, pos = self.geometry()
        U, H, X = u[self.bond], 0.5 * length[self.bond], pos[self.bond]
        a, b = self.a, self.b
        dr = X[b] - X[a]
        dr -= self.side * np.round(dr / self.side)
        ua, ub, ha, hb = U[a], U[b], H[a], H[b]
        d1, d2, c = _dot(dr, ua), _dot(dr, ub), _dot(ua, ub)
        den = 1.0 - c * c
        par = den < 1e-12
        den = np.where(par, 1.0, den)
        lam = np.where(par, 0.5 * d1, (d1 - c * d2) / den)
        mu = np.where(par, -0.5 * d2, (-d2 + c * d1) / den)
        def clip(x, h):
            return np.where(np.abs(x) > h, np.where(x >= 0, h, -h), x)
        def apart(x, y):
            v = dr - x[:, None] * ua + y[:, None] * ub
            return v, _dot(v, v)
        out1, out2 = np.abs(lam) > ha, np.abs(mu) > hb
        la = clip(lam, ha)
        ma = clip(la * c - d2, hb)
        mb = clip(mu, hb)
        lb = clip(mb * c + d1, ha)
        near_a = (apart(la, ma)[1] < apart(lb, mb)[1]) | ~out2
        la, ma = np.where(out1, la, lam), np.where(out1, ma, mu)
        both = out1 & out2
        use_b = (both & ~near_a) | (out2 & ~out1)
        lam, mu = np.where(use_b, lb, la), np.where(use_b, mb, ma)
        v, r2 = apart(lam, mu)
        c1, c2 = lam[:, None] * ua, mu[:, None] * ub
        hit = r2 <= self.rcut2
        near = hit & (r2 < 1e-12)
        far = hit & ~near
        rinv = 1.0 / np.sqrt(np.where(far, r2, 1.0))
        r6 = rinv ** 6
        fac = np.clip(-(48.0 * r6 - 24.0) * r6 * rinv, -2000.0, 2000.0)
        self.stored[far] = ((fac * rinv)[:, None] * v)[far]
        if near.any():
            w = np.where(np.any(c1 != 0, axis=1)[:, None], c1 - c2, v)[near]
            m = np.sqrt(_dot(w, w))
            ok = m >= 1e-12
            rows = np.nonzero(near)[0][ok]
            self.stored[rows] = 2000.0 * w[ok] / m[ok, None]
        f = self.stored
        force, torque = np.zeros((len(U), 3)), np.zeros((len(U), 3))
        t1, t2 = np.cross(c1, f), np.cross(c2, f)
        for i in range(3):
            force[:, i] = (np.bincount(a, f[:, i], len(U)) - np.bincount(b, f[:, i], len(U)))
            torque[:, i] = (np.bincount(a, t1[:, i], len(U)) - np.bincount(b, t2[:, i], len(U)))
        self.force, self.torque = force, torque

    def solve(self, diag, off, rhs):
        """Every filament's symmetric tridiagonal system (rows = bonds)."""
        m = diag.shape[1]
        diag, off, rhs = diag.T.copy(), off.T.copy(), rhs.T.copy()
        live = self.bond.T
        diag[~live], rhs[~live] = 1.0, 0.0
        off[~live] = 0.0  # off[j] couples rows j - 1 and j
        cp, dp = np.zeros_like(diag), np.zeros_like(rhs)
        for i in range(m):
            den = diag[i] - (off[i] * cp[i - 1] if i else 0.0)
            cp[i] = (off[i + 1] if i + 1 < m else 0.0) / den
            dp[i] = (rhs[i] - (off[i] * dp[i - 1] if i else 0.0)) / den
        for i in range(m - 2, -1, -1):
            dp[i] -= cp[i] * dp[i + 1]
        return dp.T

    def tension_force(self, u, t):
        t = np.where(self.bond, t, 0.0)[..., None]
        f = t * u
        f[:, 1:] -= (t * u)[:, :-1]
        return f

    def update(self):
        nd, mid = self.nd, not self.mid
        u, _, _ = self.geometry()
        um = np.zeros_like(u)
        um[:, 1:] = u[:, :-1]
        bF, bT = np.zeros_like(self.r), np.zeros_like(self.r)
        bF[self.bond], bT[self.bond] = self.force, self.torque
        arm = np.cross(u, bT) / self.l[..., None]
        F = 0.5 * bF + arm
        F[:, 1:] += (0.5 * bF - arm)[:, :-1]
        tn = u + um
        norm = np.sqrt(_dot(tn, tn))
        tn = np.where(self.site[..., None], tn / np.where(self.site, norm, 1.0)[..., None], 0.0)
        cos = np.zeros(self.r.shape[:2])  # cos[j]: bonds j and j + 1
        cos[:, :-1] = _dot(u[:, 1:], u[:, :-1])
        cm = np.zeros_like(cos)  # cos of bonds j - 1 and j
        cm[:, 1:] = cos[:, :-1]
        if mid:
            self.rp = self.r.copy()
            draws = self.steps // 2
            fil = np.broadcast_to(np.arange(len(self.n))[:, None], cos.shape)
            w = _philox([np.broadcast_to(self.j, cos.shape), np.full(cos.shape, draws),
                         np.zeros(cos.shape), np.zeros(cos.shape)],
                        [np.full(cos.shape, self.seed), fil])
            xi = np.zeros_like(self.r)
            for i in range(nd):
                xi[..., i] = (w[i].astype(np.float64) + 0.5) * _NORMAL - 0.5
            fr = self.sperp * xi + (self.spar - self.sperp) * _dot(tn, xi)[..., None] * tn
            fr[~self.site] = 0.0
            df = np.zeros_like(fr)
            df[:, :-1] = fr[:, 1:] - fr[:, :-1]
            t = self.solve(np.full(cos.shape, 2.0), -cm, _dot(df, u))
            self.noise = fr + self.tension_force(u, t)
        F = F + self.noise
        # Metric determinants, joint by joint.
        nf, m = cos.shape
        n = self.n[:, None]
        dt = np.ones((nf, m + 1))
        dt[:, 1] = 2.0
        for i in range(2, m):
            dt[:, i] = 2 * dt[:, i - 1] - cos[:, i - 2] ** 2 * dt[:, i - 2]
        db = np.ones((nf, m + 3))
        for k in range(m - 1, 0, -1):
            inner = 2 * db[:, k + 1] - cos[:, k - 1] ** 2 * db[:, k + 2]
            db[:, k] = np.where(k == self.n - 1, 2.0, np.where(k >= self.n, 1.0, inner))
        total = np.take_along_axis(dt, n - 1, 1)
        joint = self.j < n - 2
        ke = np.where(joint, (self.kappa + self.l * cos * dt[:, :m] * db[:, 3:m + 3] / total)
                      / self.l ** 2, 0.0)
        u1 = np.zeros_like(u)
        u1[:, :-1] = u[:, 1:]
        along = ke[..., None] * (u1 - cos[..., None] * u)
        back = ke[..., None] * (u - cos[..., None] * u1)
        fs = -along
        fs[:, 1:] += (along - back)[:, :-1]
        fs[:, 2:] += back[:, :-2]
        F = F + fs
        def mobile(v):
            return self.igperp[..., None] * v + self.dgam[..., None] * _dot(tn, v)[..., None] * tn
        g = mobile(F)
        dg = np.zeros_like(g)
        dg[:, :-1] = g[:, 1:] - g[:, :-1]
        t1 = np.zeros_like(tn)
        t1[:, :-1] = tn[:, 1:]
        diag = 2.0 * self.igperp + self.dgam * (_dot(tn, u) ** 2 + _dot(t1, u) ** 2)
        off = -self.igperp * cm - self.dgam * _dot(tn, um) * _dot(tn, u)
        F = F + self.tension_force(u, self.solve(diag, off, _dot(u, dg)))
        r = self.rp + (0.5 * self.delta if mid else self.delta) * mobile(F)
        r[~self.site] = 0.0
        self.r = r
        u, length, _ = self.geometry()
        bad = np.any(self.bond & (np.abs(self.l - length) / self.l > 1e-3), axis=1)
        before = self.switch.copy()
        self.switch ^= bad
        for f in np.nonzero(bad)[0]:
            k, step = self.n[f], self.l[f, 0] * u[f, :self.n[f] - 1]
            if before[f]:
                self.r[f, :k - 1] = self.r[f, k - 1] - np.cumsum(step[::-1], axis=0)[::-1]
            else:
                self.r[f, 1:k] = self.r[f, 0] + np.cumsum(step, axis=0)
        if not mid:
            d = self.r - self.origin
            self.moved += 2.0 * _dot(d, d)
        self.mid = not self.mid if mid else False

    def step(self):
        self.interact()
        self.update()


def exact(case, seed):
    nf, nb, _ = _sizes(case)
    if case["workload"] == "E":
        return None  # tethers, whose anchors move along their filaments, are not restated
    rows = case["longest"] * nf if case["workload"] == "C" else nb  # padded to the longest
    if case.get("steps", 1) * rows > 8e6:
        return None  # beyond some 10 seconds
    system, filaments, sites, replicas = _configuration(case, seed)
    parts = [(system, filaments, sites)]
    if replicas is not None:
        parts = workloads.split_replicas(system, filaments, sites, replicas)
    out = []
    for system, filaments, sites in parts:
        e = _Exact(system, filaments, sites, system["system_radius"], system["seed"])
        if case["kind"] == "pairs":
            e.interact()
            return {"force": e.force, "torque": e.torque}
        for _ in range(case["steps"]):
            e.step()
        out.append(e.r[e.site])
    got = {"sites": np.concatenate(out)}
    if case["kind"] == "host":
        got.update(force=e.force, torque=e.torque)
    if case["kind"] == "monitor":
        got.update(polar=None, nematic=None, angles=None, tensor=None, pressure=None, energy=None)
    return got
