"""Measured cases: parallel-tempering chunks, energies and caches as a program that uses this package runs them.

A case is a dict of plain values.  ``prepare`` builds what a program holds before the call (the model of the cell, the
replicas' occupancies, the temperature ladder, the device state), ``run`` is one call of a driver's inner loop, ``exact``
the same result in float64 from the definition of the model.

Kinds:
  ce         one chunk of cluster-expansion parallel tempering with its chunk-end exchange (``pt.run_chunk``)
  ce_batch   one CUDA-graph replay of many such jobs in float32 with the exact re-anchor (``batch.CEBatch``)
  ce_energy  cluster-vector sums and energies of many configurations (start of a run, re-anchor)
  nce        one chunk of NeuralCE parallel tempering with its exchange (``nce.NCEState.run_chunk``)
  nce_cache  full NeuralCE caches of all replicas (start of a run, re-anchor)
Cells are L0 x L1 x L2 conventional fcc cells (4 L0 L1 L2 sites) of the synthetic Ni/Pt workload.
"""
import functools
import math
import os

import numpy as np
import torch

from neuralce_gb300.batch import CEBatch
from neuralce_gb300.ce import GPUClusterExpansion
from neuralce_gb300.ce_tables import synthetic_eci
from neuralce_gb300.io import Z_OF, fcc_conventional
from neuralce_gb300.nce import NCEModel, NCEState, synthetic_model
from neuralce_gb300.pt import PTState, run_chunk
from neuralce_gb300.workloads import A_FCC, cluster_space, ladder, shipped_nce_config

GOLDEN = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tests", "golden",
                      "nipt_v3_nomax_sel.json")


def _ce(name, L, R, steps, sample, warps=0, cluster=1, x=0.5):
    return dict(name=name, kind="ce", l0=L[0], l1=L[1], l2=L[2], replicas=R, steps=steps, sample=sample, warps=warps,
                cluster=cluster, x=x)


def _nce(name, L, R, steps, model, width, mma, cluster, kind="nce"):
    return dict(name=name, kind=kind, l0=L[0], l1=L[1], l2=L[2], replicas=R, steps=steps, model=model, width=width, mma=mma,
                cluster=cluster)


def listed():
    return [
        # the published CE configuration: 2,048 sites, 32 temperatures 300-1400 K, at the launch shape its tuner picks
        _ce("ce 2048x32", (8, 8, 8), 32, 1000, 100, 16, 4),
        # the driver's default exchange interval of 10 steps on a small cell: a call that is mostly latency
        _ce("ce 256x16 short", (4, 4, 4), 16, 10, 10),
        # a ragged orthorhombic cell with a Pt-poor composition, driver defaults
        _ce("ce 840x25 ragged", (5, 6, 7), 25, 500, 50, x=0.3),
        # published larger cells: many replicas, occupancies beyond on-chip memory
        _ce("ce 131072x256", (32, 32, 32), 256, 300, 100),
        _ce("ce 1048576x64", (64, 64, 64), 64, 500, 100, 16, 1),
        # the batching form: 24 independent cells of 256 to 32,000 sites, float32 with exact re-anchor, one graph replay
        dict(name="ce batch 24 fp32", kind="ce_batch", jobs=24, lmin=4, lmax=20, steps=250, chunks=2, warps=8, cluster=1),
        # energies of all replicas of a large cell (set-up of a run, check of carried energies)
        dict(name="ce energy 1048576x64", kind="ce_energy", l0=64, l1=64, l2=64, replicas=64),
        # NeuralCE: depth-3 width-64 network in float32, the tuner's 4 CTAs per replica
        _nce("nce 2048x32 fp32", (8, 8, 8), 32, 25, "synthetic", 64, 0, 4),
        # the reference's shipped model (one gated layer of width 16, three shells)
        _nce("nce 2048x32 shipped", (8, 8, 8), 32, 40, "shipped", 16, 0, 4),
        # width 128 in split bf16 (the precision form of the large configuration)
        _nce("nce 55296x16 split", (24, 24, 24), 16, 12, "synthetic", 128, 4, 8),
        # re-anchor of all replicas: the small float32 configuration and a larger split one
        _nce("nce cache 2048x32 fp32", (8, 8, 8), 32, 0, "synthetic", 64, 0, 1, "nce_cache"),
        _nce("nce cache 131072x8 split", (32, 32, 32), 8, 0, "synthetic", 128, 4, 1, "nce_cache"),
    ]


def draw(rng):
    kind = rng.choice(["ce", "ce", "ce", "ce_batch", "ce_energy", "nce", "nce", "nce_cache"])
    lu = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    if kind == "ce_batch":
        a = rng.randint(4, 8)
        return dict(kind=kind, jobs=rng.randint(4, 24), lmin=a, lmax=a + rng.randint(2, 10), steps=lu(20, 250), chunks=rng.randint(1, 2),
                    warps=rng.choice([4, 8, 16]), cluster=1)
    if kind in ("ce", "ce_energy"):
        m = math.exp(rng.uniform(math.log(4), math.log(48)))
        L = [max(4, int(round(m * rng.uniform(0.8, 1.25)))) for _ in range(3)]
        N = 4 * L[0] * L[1] * L[2]
        if kind == "ce_energy":
            R = max(1, min(lu(4, 256), (1 << 26) // N))
            return dict(kind=kind, l0=L[0], l1=L[1], l2=L[2], replicas=R)
        R = max(4, min(lu(4, 256), (1 << 26) // N))
        steps = max(10, min(lu(10, 2000), 80_000 // R))
        wc = rng.choice([(0, 1), (0, 1), (16, 1), (16, 4), (8, 2)])
        return dict(_ce("", L, R, steps, rng.choice([1, 10, 100]), wc[0], wc[1], round(rng.uniform(0.1, 0.9), 3)))
    m = math.exp(rng.uniform(math.log(5), math.log(20)))
    L = [max(5, int(round(m * rng.uniform(0.85, 1.2)))) for _ in range(3)]
    N = 4 * L[0] * L[1] * L[2]
    if rng.random() < 0.3:
        model, width, mma = "shipped", 16, 0
    else:
        model, width = "synthetic", rng.choice([32, 64, 64, 128])
        mma = rng.choice([0, 4, 4]) if width < 128 else 4
    R = max(2, min(lu(4, 64), 800_000 // N))
    if kind == "nce_cache":
        return dict(_nce("", L, R, 0, model, width, mma, 1, kind))
    return dict(_nce("", L, R, rng.randint(4, max(4, min(20, 600 // R))), model, width, mma, rng.choice([1, 2, 4])))


# ── models (kept per cell, as a program keeps them) ───────────────────────────────────────────────

def _cell(L):
    s = fcc_conventional(A_FCC, tuple(L))
    s.numbers = np.full(len(s), Z_OF["Ni"], np.int64)
    return s


@functools.lru_cache(maxsize=64)
def _ce_model(l0, l1, l2):
    cs, s = cluster_space(), _cell((l0, l1, l2))
    return GPUClusterExpansion((cs, synthetic_eci(cs, 0)), s, energy_scale=len(s)), s


@functools.lru_cache(maxsize=16)
def _nce_model(l0, l1, l2, model, width, mma):
    s = _cell((l0, l1, l2))
    if model == "shipped":
        m, _ = shipped_nce_config(GOLDEN, 2)
        return NCEModel(m.cs, s, m.params, m.mu, m.sd, shell_edges=_shell_edges(model), act="tanh", pool="mean", ys=m.ys,
                        ym=m.ym, mma=mma), s
    cs = cluster_space()
    P = synthetic_model(len(cs.orbits) + 1, 3, width, 1, 0)
    return NCEModel(cs, s, P, shell_edges=(0.0, 3.3), act="silu", pool="sum", mma=mma), s


def _shell_edges(model):
    if model != "shipped":
        return (0.0, 3.3)
    import json
    with open(GOLDEN) as f:
        return tuple(json.load(f)["shell_edges"])


def _occupancies(N, R, x, seed):
    """(R, N) int8 on the GPU: every replica an independent arrangement of round(x N) Pt."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 11)
    n_pt = int(round(x * N))
    out = torch.zeros((R, N), dtype=torch.int8, device="cuda")
    for r in range(R):
        out[r, torch.randperm(N, generator=g, device="cuda")[:n_pt]] = 1
    return out


def _batch_jobs(case, seed):
    rng = np.random.default_rng(int(seed))
    jobs = []
    geo = np.random.default_rng(5)                       # the cells are the case's, the arrangements the seed's
    for k in range(case["jobs"]):
        L = int(geo.integers(case["lmin"], case["lmax"] + 1))
        R, x = int(geo.choice([16, 32, 64])), float(geo.uniform(0.1, 0.9))
        gce, s = _ce_model(L, L, L)
        sig = _occupancies(len(s), R, x, int(rng.integers(1 << 30))).cpu().numpy()
        jobs.append(dict(gce=gce, sigma=sig, beta=ladder(R)[1], R=R, N=len(s)))
    return jobs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ce_batch":
        b = CEBatch(_batch_jobs(case, seed), precision=32, warps=case["warps"], cluster=case["cluster"])
        b.capture(case["steps"], chunks=case["chunks"], reanchor=True)
        return dict(case=case, batch=b)
    R = case["replicas"]
    N = 4 * case["l0"] * case["l1"] * case["l2"]
    if kind == "ce_energy":
        gce, _ = _ce_model(case["l0"], case["l1"], case["l2"])
        gce.handle
        return dict(case=case, gce=gce, sigma=_occupancies(N, R, 0.5, seed))
    beta = ladder(R)[1]
    if kind == "ce":
        gce, _ = _ce_model(case["l0"], case["l1"], case["l2"])
        sig = _occupancies(N, R, case["x"], seed)
        E0 = gce.batched_energy(sig).cpu().numpy()
        st = PTState(sig.cpu().numpy(), E0, beta, np.zeros(R, np.int32))
        n = case["steps"] // case["sample"]
        Es = torch.zeros((max(n, 1), R), dtype=torch.float64, device="cuda")
        return dict(case=case, gce=gce, st=st, Es=Es, step=0)
    m, _ = _nce_model(case["l0"], case["l1"], case["l2"], case["model"], case["width"], case["mma"])
    st = NCEState(m, _occupancies(N, R, 0.5, seed).cpu().numpy(), beta)
    if kind == "nce":
        st.full_cache()
    Es = torch.zeros((max(case["steps"], 1), R), dtype=torch.float64, device="cuda")
    return dict(case=case, st=st, Es=Es, step=0)


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "ce_batch":
        b = state["batch"]
        b.replay()
        # every job's state after the replay, the jobs one behind another
        cat = lambda f: [getattr(s, f) for s in b.states]
        return dict(sigma0=b.states[0].sigma, sigma1=b.states[1].sigma, E=torch.cat(cat("E")), n_acc=torch.cat(cat("n_acc")),
                    rep_of_slot=torch.cat(cat("rep_of_slot")), cv=torch.cat(cat("cv")))
    if kind == "ce_energy":
        cv = state["gce"].cluster_counts(state["sigma"])
        return dict(cv=cv, E=state["gce"].energy_from_counts(cv))
    st = state["st"]
    if kind == "ce":
        run_chunk(state["gce"], st, c["steps"], state["step"], 42, 64, c["warps"], None, c["sample"], state["Es"], True,
                  cluster=c["cluster"])
        state["step"] += c["steps"]
        return dict(sigma=st.sigma, E=st.E, E_min=st.E_min_rep, n_acc=st.n_acc, n_near=st.n_near, n_ex=st.n_ex,
                    rep_of_slot=st.rep_of_slot, slot_of_rep=st.slot_of_rep, samples=state["Es"])
    if kind == "nce_cache":
        st.full_cache()
        return dict(h0=st.h0, hmid=st.hmid, e=st.e, E=st.E)
    st.run_chunk(c["steps"], state["step"], seed=99, sample_interval=1, E_samples=state["Es"], exchange_rounds=1,
                 cluster=c["cluster"])
    state["step"] += c["steps"]
    return dict(sigma=st.sigma, E=st.E, n_acc=st.n_acc, n_ex=st.n_ex, rep_of_slot=st.rep_of_slot, samples=state["Es"], h0=st.h0,
                hmid=st.hmid, e=st.e)


# ── what a pass cannot do without ─────────────────────────────────────────────────────────────────
# CE step: half of the swaps (2 x (1 - x) of them) are of different species; each reads the 2 x 141 sites of its
# neighbourhoods and adds 2 x 2,103 signed row products (one XOR-and-count each).  State read and written once.

def work(case):
    kind = case["kind"]
    if kind == "ce_batch":
        geo = np.random.default_rng(5)
        tot = dict(bytes=0.0, flops=0.0)
        for _ in range(case["jobs"]):
            L = int(geo.integers(case["lmin"], case["lmax"] + 1))
            R, x = int(geo.choice([16, 32, 64])), float(geo.uniform(0.1, 0.9))
            w = work(dict(kind="ce", l0=L, l1=L, l2=L, replicas=R, steps=case["steps"] * case["chunks"], sample=1 << 30, x=x))
            tot = {k: tot[k] + w[k] for k in tot}
        return tot
    N, R = 4 * case["l0"] * case["l1"] * case["l2"], case["replicas"]
    if kind == "ce_energy":
        return dict(bytes=float(R * N + R * 38 * 8), flops=float(R) * N * 614)
    if kind == "ce":
        ev = 2.0 * case["x"] * (1.0 - case["x"]) * case["steps"] * R
        b = min(ev * 2 * 141, 2.0 * R * N) + ev * 2 + R * 64 + case["steps"] // case["sample"] * R * 8
        return dict(bytes=float(b), flops=ev * 2 * 2103)
    if case["model"] == "shipped":
        chans, balls, D, P, J = [18], [87, 393], 16, 3, 527
    else:
        D, P, J = case["width"], 1, 2103
        chans, balls = [38, D, D], [141, 321, 603, 1007]
    per_site = sum(2.0 * (1 + P) * c * D for c in chans) + (2.0 * P * chans[0] * D if case["model"] == "shipped" else 0.0)
    state = 4.0 * (chans[0] + D * (len(chans) - 1) + 1)
    if kind == "nce_cache":
        return dict(bytes=R * N * (1.0 + state), flops=R * N * (per_site + J))
    ev = 0.5 * case["steps"] * R
    fl = sum(2.0 * (1 + P) * c * D * min(2 * n, N) for c, n in zip(chans, balls[1:]))
    if case["model"] == "shipped":
        fl += 2.0 * P * chans[0] * D * min(2 * balls[1], N)
    rd = 4.0 * sum(c * min(2 * n, N) for c, n in zip(chans, balls[1:]))
    return dict(bytes=ev * rd, flops=ev * (fl + 2 * J))


# ── float64 from the definitions ──────────────────────────────────────────────────────────────────
# Sites as integer points of the fcc lattice (units of a / 2); E = sum over the orbits and their cluster instances of
# eci / (instances per cell x cells) x product of the members' signs (Ni -1, Pt +1).

class _Lattice:
    def __init__(self, s, perm, prim_cell, L):
        dev = "cuda"
        a = np.linalg.norm(np.asarray(s.cell)[0]) / L[0]
        self.box = torch.tensor([2 * v for v in L], device=dev)
        xyz = np.rint(np.asarray(s.positions)[perm] * 2.0 / a).astype(np.int64) % np.array([2 * v for v in L])
        self.xyz = torch.as_tensor(xyz, device=dev)
        grid = torch.full(tuple(2 * v for v in L), -1, dtype=torch.int64, device=dev)
        grid[tuple(self.xyz.T)] = torch.arange(len(xyz), device=dev)
        self.grid = grid
        ap = np.abs(np.asarray(prim_cell)).max() * 2.0
        self.prim2 = np.rint(np.asarray(prim_cell) * 2.0 / ap).astype(np.int64)
        self.N = len(xyz)

    def at(self, sites, off):
        """sites (...,) and integer offsets (m, 3) -> sites (..., m)"""
        p = (self.xyz[sites][..., None, :] + off) % self.box
        return self.grid[p[..., 0], p[..., 1], p[..., 2]]


class _Clusters:
    """Cluster instances of an orbit list: per order, the other members' offsets of every instance containing a site."""

    def __init__(self, cs, lat):
        keys = {}
        rows, tmpl = [], []
        for c, o in enumerate(cs.orbits):
            for inst in o.clusters:
                pts = [np.asarray(n, np.int64) @ lat.prim2 for (_, n) in inst]
                tmpl.append((c, [p - pts[0] for p in pts[1:]]))
                for m in range(len(pts)):
                    rows.append((c, [p - pts[m] for q, p in enumerate(pts) if q != m]))
        ix = lambda p: keys.setdefault(tuple(int(v) for v in p), len(keys))
        ix((0, 0, 0))
        mo = max(len(r[1]) for r in rows)
        self.cols = torch.tensor([r[0] for r in rows], device="cuda")
        self.mem = torch.tensor([[ix(p) + 1 for p in r[1]] + [0] * (mo - len(r[1])) for r in rows], device="cuda")
        self.tmpl = [(c, [ix(p) for p in q]) for c, q in tmpl]
        self.off = torch.tensor(list(keys), device="cuda")
        self.n = torch.tensor([len(o.clusters) for o in cs.orbits], dtype=torch.float64, device="cuda")
        self.order = torch.tensor([len(o.clusters[0]) for o in cs.orbits], dtype=torch.float64, device="cuda")
        self.K = len(cs.orbits)

    def site_sums(self, lat, spin, sites):
        """spin (R, N), sites (R, m) -> (R, m, K): per orbit the sum over the instances containing the site."""
        nb = lat.at(sites, self.off)
        v = torch.gather(spin[:, None, :].expand(-1, nb.shape[1], -1), 2, nb)
        v = torch.cat([torch.ones_like(v[..., :1]), v], -1)
        pr = v[..., 1:2] * v[..., self.mem].prod(-1)
        out = torch.zeros(pr.shape[:2] + (self.K,), dtype=torch.float64, device=spin.device)
        return out.index_add_(2, self.cols, pr.double())


def _sums(lat, cl, sig):
    """(R, K) sums over the cell's instances of each orbit."""
    spin = (2 * sig - 1).to(torch.int8)
    sites = torch.arange(lat.N, device=sig.device)
    out = torch.zeros((len(sig), cl.K), dtype=torch.int64, device=sig.device)
    per = max(1, (1 << 24) // lat.N)
    for r0 in range(0, len(sig), per):
        sp = spin[r0:r0 + per]
        nb = {}
        for c, q in cl.tmpl:
            v = sp
            for p in q:
                if p not in nb:
                    nb[p] = sp[:, lat.at(sites, cl.off[p:p + 1])[:, 0]]
                v = v * nb[p]
            out[r0:r0 + per, c] += v.sum(1, dtype=torch.int64)
    return out


def _philox(c0, c1, c2, c3, seed):
    """Philox4x32-10 (Salmon et al., 2011) on uint64 arrays of 32-bit words."""
    M = np.uint64(0xFFFFFFFF)
    c0, c1, c2, c3 = np.broadcast_arrays(*(np.asarray(v, np.uint64) for v in (c0, c1, c2, c3)))
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    S = np.uint64(32)
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c0, np.uint64(0xCD9E8D57) * c2
        c0, c1, c2, c3 = (p1 >> S) ^ c1 ^ np.uint64(k0), p1 & M, (p0 >> S) ^ c3 ^ np.uint64(k1), p0 & M
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c0, c1, c2, c3


def _uniform(hi, lo):
    return (((hi << np.uint64(21)) | (lo >> np.uint64(11))) + np.uint64(1)).astype(np.float64) * 2.0 ** -53


def _proposals(seed, T, R, cells):
    x = _philox(np.arange(T)[:, None], 0, np.arange(R)[None], 0, seed)
    return (((x[0] * np.uint64(cells)) >> np.uint64(32)).astype(np.int64), ((x[1] * np.uint64(cells)) >> np.uint64(32)).astype(np.int64),
            _uniform(x[2], x[3]))


def _exchange(E, beta, ros, seed, g):
    top = 0xFFFFFFFF
    par = int(_philox(g, 0, top, 0, seed)[0]) & 1
    ros, n = ros.copy(), 0
    for k in range((len(ros)) // 2):
        a = 2 * k + par
        if a + 1 >= len(ros) or 2 * k >= len(ros) - 1:
            continue
        w = _philox(g, 0, top - 1, k, seed)
        u = float(_uniform(w[0], w[1]))
        if math.log(u) < (float(beta[a + 1]) - float(beta[a])) * (E[ros[a + 1]] - E[ros[a]]):
            ros[[a, a + 1]] = ros[[a + 1, a]]
            n += 1
    return ros, n


def _slots(ros):
    s = np.empty(len(ros), np.int32)
    s[ros] = np.arange(len(ros))
    return s


def _chain_ce(lat, cl, eci, sig, E, beta, T, seed, sample):
    """T steps of every replica on float64 energies; eci: per orbit, per instance."""
    R = len(sig)
    ia, ib, u = (torch.as_tensor(v, device="cuda") for v in _proposals(seed, T, R, lat.N))
    lu, b64 = torch.log(u), torch.as_tensor(beta.astype(np.float64), device="cuda")
    spin = (2 * sig - 1).to(torch.int8)
    ar = torch.arange(R, device="cuda")
    E, Emin = E.clone(), E.clone()                       # the running minimum of a chunk starts at its first energy
    nacc, nnear = torch.zeros(R, dtype=torch.int64, device="cuda"), torch.zeros(R, dtype=torch.int64, device="cuda")
    Es = torch.zeros((max(T // sample, 1), R), dtype=torch.float64, device="cuda")
    for t in range(T):
        a, b = ia[t], ib[t]
        sa, sb = spin[ar, a], spin[ar, b]
        ok = sa != sb
        # flip b, then a in the changed arrangement: each flip negates the instances that contain the site
        d = -2.0 * (cl.site_sums(lat, spin, b[:, None])[:, 0] @ eci)
        spin[ar, b] = torch.where(ok, sa, sb)
        d += -2.0 * (cl.site_sums(lat, spin, a[:, None])[:, 0] @ eci)
        acc = ok & (lu[t] < -b64 * d)
        nnear += ok & ((d + lu[t] / b64).abs() < 1e-9)
        spin[ar, b] = torch.where(acc, sa, sb)
        spin[ar, a] = torch.where(acc, sb, sa)
        E = torch.where(acc, E + d, E)
        Emin = torch.minimum(Emin, E)
        nacc += acc
        if (t + 1) % sample == 0:
            Es[(t + 1) // sample - 1] = E
    ros, n = _exchange(E.cpu().numpy(), beta, np.arange(R), seed, T)
    if T % sample == 0:
        Es[T // sample - 1] = E[torch.as_tensor(ros, device="cuda")]
    return dict(sigma=((spin + 1) // 2).to(torch.int8), E=E, E_min=Emin, n_acc=nacc, n_near=nnear,
                n_ex=torch.tensor([n], device="cuda"), rep_of_slot=torch.as_tensor(ros.astype(np.int32)),
                slot_of_rep=torch.as_tensor(_slots(ros)), samples=Es)


def _lat_of(case, perm, cs):
    L = (case["l0"], case["l1"], case["l2"])
    return _Lattice(_cell(L), perm, cs.primitive.cell, L)


def _exact_ce(case, seed):
    cs = cluster_space()
    gce, s = _ce_model(case["l0"], case["l1"], case["l2"])
    lat = _lat_of(case, gce.perm, cs)
    cl = _Clusters(cs, lat)
    sig = _occupancies(lat.N, case["replicas"], case.get("x", 0.5), seed)
    cv = _sums(lat, cl, sig)
    eci = torch.as_tensor(np.asarray(gce.parameters)[1:] * len(s), device="cuda") / (cl.n * lat.N)
    E = cv.double() @ eci
    if case["kind"] == "ce_energy":
        return dict(cv=torch.cat([cv, torch.zeros_like(cv[:, :1])], 1), E=E)
    if case["steps"] * case["replicas"] > 150_000:
        return None
    return _chain_ce(lat, cl, eci, sig, E, ladder(case["replicas"])[1], case["steps"], 42, case["sample"])


class _Net:
    """The NeuralCE network in float64: layer 0 from the cluster sums of a site, layers on shell means, site energies."""

    def __init__(self, case):
        m, s = _nce_model(case["l0"], case["l1"], case["l2"], case["model"], case["width"], case["mma"])
        d = lambda v: torch.as_tensor(np.asarray(v, np.float64), device="cuda")
        self.lat = _lat_of(case, m.perm, m.cs)
        self.cl = _Clusters(m.cs, self.lat)
        self.tanh, self.mean = case["model"] == "shipped", case["model"] == "shipped"
        self.mu, self.sd = d(m.mu), d(m.sd)
        self.lin, self.hw, self.hb = d(m.params["lin"]), d(m.params["head"]["w"]), float(m.params["head"]["b"])
        self.layers = [{k: d(v) for k, v in Ly.items()} for Ly in m.params["layers"]]
        self.norm = float(self.lat.N) if self.mean else 1.0
        self.scale = float(m.ys) * self.lat.N if self.mean else 1.0
        edges = _shell_edges(case["model"])
        ap = np.abs(np.asarray(m.cs.primitive.cell)).max() * 2.0
        g = np.array([(x, y, z) for x in range(-6, 7) for y in range(-6, 7) for z in range(-6, 7) if (x + y + z) % 2 == 0])
        r = np.linalg.norm(g, axis=1) * ap / 2.0
        self.shells = []
        for p in range(len(edges) - 1):
            lo = edges[p] if p else 1e-6
            hi = edges[p + 1] + (1e-6 if p == len(edges) - 2 else 0.0)
            self.shells.append(torch.as_tensor(g[(r > lo) & (r <= hi)], device="cuda"))
        balls = [set(tuple(v) for v in self.cl.off.cpu().numpy().tolist())]
        part = [tuple(v) for sh in self.shells for v in sh.cpu().numpy().tolist()]
        for _ in self.layers:
            balls.append(balls[-1] | {(a[0] + b[0], a[1] + b[1], a[2] + b[2]) for a in balls[-1] for b in part})
        self.balls = [torch.tensor(sorted(b), device="cuda") for b in balls]

    def layer0(self, spin, sites):
        z = self.cl.site_sums(self.lat, spin, sites) / (self.cl.order * self.cl.n * self.sd[1:]) - self.mu[1:] / self.sd[1:]
        one = torch.full_like(z[..., :1], float((1.0 - self.mu[0]) / self.sd[0]))
        return torch.cat([one, z], -1)

    def layer(self, l, h, sites):
        """layer l on the sites (R, m) from level-l values h (R, N, C)"""
        Ly = self.layers[l]
        take = lambda ix: torch.gather(h, 1, ix[..., None].expand(-1, -1, h.shape[-1]))
        o, g = take(sites) @ Ly["self"] + Ly["b"], 0.0
        for p, sh in enumerate(self.shells):
            mean = 0.0
            for q in range(len(sh)):
                mean = mean + take(self.lat.at(sites, sh[q:q + 1])[..., 0])
            mean = mean / len(sh)
            o = o + mean @ Ly["shell"][p]
            if "gate" in Ly:
                g = g + mean @ Ly["gate"][p]
        o = torch.tanh(o) if self.tanh else o * torch.sigmoid(o)
        return o * torch.sigmoid(g + Ly["gb"]) if "gate" in Ly else o

    def caches(self, sig):
        spin = (2 * sig - 1).to(torch.int8)
        R, N = sig.shape
        hs = [torch.empty((R, N, len(self.mu)), dtype=torch.float64, device="cuda")]
        per = max(1, 40_000_000 // (R * len(self.cl.cols)))
        for a in range(0, N, per):
            s = torch.arange(a, min(N, a + per), device="cuda").expand(R, -1)
            hs[0][:, a:a + per] = self.layer0(spin, s)
        every = torch.arange(N, device="cuda").expand(R, -1)
        for l in range(len(self.layers)):
            hs.append(self.layer(l, hs[l], every))
        e = hs[-1] @ self.hw + hs[0] @ self.lin
        return hs, e, e.sum(1) / self.norm + self.hb

    def chain(self, sig, beta, T, seed):
        R = len(sig)
        hs, e, E = self.caches(sig)
        hs = hs[:-1]
        ia, ib, u = _proposals(seed, T, R, self.lat.N)
        spin = (2 * sig - 1).to(torch.int8)
        ar = torch.arange(R, device="cuda")
        nacc = torch.zeros(R, dtype=torch.int64, device="cuda")
        Es = torch.zeros((T, R), dtype=torch.float64, device="cuda")
        uu = torch.as_tensor(u, device="cuda")
        b64 = torch.as_tensor(beta.astype(np.float64), device="cuda")
        for t in range(T):
            a, b = torch.as_tensor(ia[t], device="cuda"), torch.as_tensor(ib[t], device="cuda")
            sa, sb = spin[ar, a], spin[ar, b]
            ok = sa != sb
            sp2 = spin.clone()
            sp2[ar, a], sp2[ar, b] = sb, sa
            ctr = torch.stack([a, b], 1)
            old, h = [], None
            for l in range(len(self.layers) + 1):
                s = self.lat.at(ctr, self.balls[l]).reshape(R, -1)
                ix = s[..., None]
                v = self.layer0(sp2, s) if l == 0 else self.layer(l - 1, hs[l - 1], s)
                if l < len(self.layers):
                    old.append((ix, torch.gather(hs[l], 1, ix.expand(-1, -1, v.shape[-1]))))
                    hs[l].scatter_(1, ix.expand(-1, -1, v.shape[-1]), v)
                else:
                    n0 = torch.gather(hs[0], 1, ix.expand(-1, -1, hs[0].shape[-1]))
                    en = v @ self.hw + n0 @ self.lin
                    e2 = e.scatter(1, s, en)
            dE = torch.where(ok, (e2 - e).sum(1) / self.norm, torch.zeros_like(E))
            dv = dE * self.scale
            acc = (dv <= 0.0) | (uu[t] < torch.exp(-b64 * dv))
            no = ~(acc & ok)
            for l, (ix, v) in enumerate(old):              # rejected: the old rows back
                k = torch.nonzero(no)[:, 0]
                hs[l][k] = hs[l][k].scatter(1, ix[k].expand(-1, -1, v.shape[-1]), v[k])
            e = torch.where(no[:, None], e, e2)
            spin = torch.where(no[:, None], spin, sp2)
            E = E + torch.where(no, torch.zeros_like(dE), dE)
            nacc += acc
            Es[t] = E
        ros, n = _exchange(E.cpu().numpy() * self.scale, beta, np.arange(R), seed, T)
        return dict(sigma=((spin + 1) // 2).to(torch.int8), E=E, n_acc=nacc, n_ex=torch.tensor([n]),
                    rep_of_slot=torch.as_tensor(ros.astype(np.int32)), samples=Es, h0=hs[0],
                    hmid=torch.stack(hs[1:]) if len(hs) > 1 else None, e=e)


def exact(case, seed):
    """Float64 results of ``run`` on the same inputs; None for the longest chains (over about 20 seconds here)."""
    if case["kind"] == "ce_batch":
        return None                    # thousands of float32 chains: a few take another turn than float64's
    if case["kind"] in ("ce", "ce_energy"):
        return _exact_ce(case, seed)
    net = _Net(case)
    sig = _occupancies(net.lat.N, case["replicas"], 0.5, seed)
    if case["kind"] == "nce_cache":
        hs, e, E = net.caches(sig)
        return dict(h0=hs[0], hmid=torch.stack(hs[1:-1]) if len(hs) > 2 else None, e=e, E=E)
    return net.chain(sig, ladder(case["replicas"])[1], case["steps"], 99)
