"""The work that the framework's performance is measured on.

A case is a molecular-dynamics run, a rebuild-heavy run, a run on
host-resident state, or the surrogate's training or inference, each through
the public calls of ``cac_code_gb300.cacg``.  ``listed()`` holds the fixed
cases, ``draw()`` more of the same ranges.

Kinds:

``md``       a caller that owns the state pushes it (put_atoms, put_nodes), runs
             velocity-Verlet steps and reads positions, velocities and forces
             back.  ``rebuild`` 1 re-bins and re-lists at every step
             (neigh_modify every 1 check no), 0 keeps the lists of set-up
             (neigh_modify every 10 check yes, as the configurations have it).
``host``     the same with the state in host memory, one run_host call.
``train``    the surrogate ensemble trained from given weights.
``predict``  the ensemble's mean and spread on held-out samples.

Models are the framework's slabs: an FCC atom block of ``cx`` x ``ky``*nae x
``kz``*nae cells between ``layers`` planes of elements (``nae`` sites per
edge) on each side, periodic in y and z, less ``holes`` atoms (vacancies),
with seeded displacements and thermal velocities.  Mixed precision evaluates
pair terms in FP32, so what depends on its forces at first order (velocities,
forces) is handed on as float32; FP64 modes hand on float64.
"""
import math

import numpy as np
import torch

from cac_code_gb300 import cacg
from cac_code_gb300 import lattice as L
from cac_code_gb300 import workloads as W

MODES = {"exact": cacg.FP64_EXACT, "fp64": cacg.FP64, "mixed": cacg.MIXED}

# Lennard-Jones in reduced units; EAM Cu: density exp(-6 (r/2.556 - 1)), Morse
# pair, embedding -1.2 sqrt(rho), cutoff 5.5, 2,000 knots each
LJ_CUT, LJ_SKIN, LJ_DT, LJ_A, LJ_T = 2.5, 2.8, 0.005, W.A_LJ, 0.1
EAM_CUT, EAM_SKIN, EAM_DT, EAM_A, EAM_T = 5.5, 7.5, 0.001, W.A_CU, 300.0
EAM_MASS, EAM_N, EAM_RHO_MAX = 63.546, 2000, 40.0
JITTER = {"lj": 0.03, "eam": 0.05}
KB = {"lj": 1.0, "eam": 8.617343e-5}
MVV2E = {"lj": 1.0, "eam": 1.0364269e-4}


def _md(name, pair, mode, cx, ky, kz, layers, nae, steps, rebuild=0, holes=0, kind="md"):
    return {"name": name, "kind": kind, "pair": pair, "mode": mode, "cx": cx, "ky": ky, "kz": kz,
            "layers": layers, "nae": nae, "steps": steps, "rebuild": rebuild, "holes": holes}


def listed():
    return [
        # the smallest systems: a parity-sized LJ slab in the default bit-exact mode
        # (1,024 atoms, 32 elements)
        _md("lj_tiny_exact", "lj", "exact", 4, 2, 2, 2, 4, 20),
        # the LJ configuration C1 (16,384 atoms, 64 elements) as a drop-in caller
        # runs it, and in mixed precision
        _md("lj_c1_exact", "lj", "exact", 16, 2, 2, 4, 8, 20),
        _md("lj_c1_mixed", "lj", "mixed", 16, 2, 2, 4, 8, 50),
        # a small EAM slab (9,680 atoms less 3 vacancies, 160 elements): launches count
        _md("eam_small_mixed", "eam", "mixed", 5, 2, 2, 10, 11, 50, holes=3),
        # ordinary EAM slabs: mostly atoms (266,200 atoms, 7,200 elements) in the
        # default mode and in mixed precision, mostly elements (247,808 atoms,
        # 64,000 elements) in FP64
        _md("eam_atoms_exact", "eam", "exact", 22, 5, 5, 72, 11, 4),
        _md("eam_atoms_mixed", "eam", "mixed", 22, 5, 5, 72, 11, 20),
        _md("eam_elems_fp64", "eam", "fp64", 8, 8, 8, 250, 11, 4),
        # lists rebuilt at every step, default mode (fast dynamics, set-up, an odd
        # number of atoms: 72,600 less 1, 1,024 elements)
        _md("eam_rebuild_exact", "eam", "exact", 6, 5, 5, 16, 11, 2, rebuild=1, holes=1),
        # host-resident stepping: a caller that takes its state back every ten steps
        _md("eam_host_mixed", "eam", "mixed", 8, 8, 8, 250, 11, 10, kind="host"),
        # the largest run: the C5 configuration in mixed precision (1,982,464 atoms,
        # 499,712 elements)
        _md("eam_c5_mixed", "eam", "mixed", 16, 16, 16, 488, 11, 10),
        # the surrogate: an epoch of training (4 members, batches of 2,048) and the
        # held-out evaluation
        {"name": "mlp_train", "kind": "train", "n": 65536, "members": 4, "batch": 2048, "epochs": 1},
        {"name": "mlp_predict", "kind": "predict", "n": 65536, "members": 4},
    ]


def _sites(c):
    atoms = 4 * c["cx"] * c["ky"] * c["kz"] * c["nae"] ** 2 - c["holes"]
    return atoms, 4 * c["ky"] * c["kz"] * c["layers"]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["md", "md", "md", "md", "md", "host", "rebuild", "train", "predict"])
    if kind == "train":
        batch = 128 * rng.randint(2, 24)
        return {"kind": "train", "n": batch * rng.randint(4, 24) + rng.randint(0, batch - 1),
                "members": rng.randint(1, 4), "batch": batch, "epochs": 1}
    if kind == "predict":
        return {"kind": "predict", "n": _log(rng, 100, 200000), "members": rng.randint(1, 4)}
    # weights of a site-step by mode, relative to mixed: no case above the largest
    cost = {"mixed": 1.0, "fp64": 25.0, "exact": 40.0}
    while True:
        pair = "eam" if kind == "host" else rng.choice(["lj", "eam", "eam"])
        mode = "mixed" if kind == "host" else rng.choice(["exact", "fp64", "mixed", "mixed"])
        if pair == "lj":
            c = _md("", pair, mode, _log(rng, 3, 40), rng.randint(2, 5), rng.randint(2, 5),
                    _log(rng, 1, 40), rng.randint(6, 9), rng.randint(10, 40))
        else:
            c = _md("", pair, mode, _log(rng, 3, 24), _log(rng, 2, 14), _log(rng, 2, 14),
                    _log(rng, 2, 400), rng.choice([11, 11, 12]), rng.randint(4, 30))
        c["holes"] = rng.randint(0, 9)
        if kind == "host":
            c["kind"] = "host"
        if kind == "rebuild":
            c["rebuild"], c["steps"] = 1, rng.randint(1, 3)
        atoms, elems = _sites(c)
        work = (atoms + 8 * elems) * c["steps"] * cost[mode]
        if kind == "rebuild":
            work += 150.0 * (atoms + 30 * elems) * c["steps"]
        if 2e5 < work < 4e7 and atoms < 1600000 and elems < 400000:
            del c["name"]
            return c


# ---------------------------------------------------------------- potential tables

def _spline(f, delta):
    """Knots f[0..n-1] as the reference's 7 coefficients per knot, 1-based rows
    (derivative 3, value 4), from five-point slopes."""
    n = len(f)
    s = np.zeros((n + 1, 7))
    v = np.zeros(n + 1)
    v[1:] = f
    s[1:, 6] = f
    d = np.zeros(n + 1)
    d[1], d[n] = v[2] - v[1], v[n] - v[n - 1]
    d[2], d[n - 1] = 0.5 * (v[3] - v[1]), 0.5 * (v[n] - v[n - 2])
    m = np.arange(3, n - 1)
    d[m] = ((v[m - 2] - v[m + 2]) + 8.0 * (v[m + 1] - v[m - 1])) / 12.0
    s[:, 5] = d
    m = np.arange(1, n)
    s[m, 4] = 3.0 * (v[m + 1] - v[m]) - 2.0 * d[m] - d[m + 1]
    s[m, 3] = d[m] + d[m + 1] - 2.0 * (v[m + 1] - v[m])
    s[1:, 2] = s[1:, 5] / delta
    s[1:, 1] = 2.0 * s[1:, 4] / delta
    s[1:, 0] = 3.0 * s[1:, 3] / delta
    return s


def _eam_tables():
    dr, drho = EAM_CUT / (EAM_N - 1), EAM_RHO_MAX / (EAM_N - 1)
    r = np.arange(EAM_N) * dr
    e = np.exp(-1.3588 * (r - 2.866))
    return {"nr": EAM_N, "dr": dr, "nrho": EAM_N, "drho": drho,
            "frho": _spline(-1.2 * np.sqrt(np.arange(EAM_N) * drho), drho),
            "rhor": _spline(np.exp(-6.0 * (r / 2.556 - 1.0)), dr),
            "z2r": _spline(r * 0.3429 * (e * e - 2.0 * e), dr)}


# ---------------------------------------------------------------- inputs

def _pinned(shape):
    t = torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    return t, t.numpy()


_BASE = {}  # the ideal slab of the last geometry: displacements differ by seed


def _model(c, seed):
    key = (c["pair"], c["cx"], c["ky"], c["kz"], c["layers"], c["nae"])
    if key not in _BASE:
        _BASE.clear()
        lj = c["pair"] == "lj"
        nae = c["nae"]
        _BASE[key] = L.make_slab_model(
            LJ_A if lj else EAM_A, 1.0 if lj else EAM_MASS, (c["cx"], c["ky"] * nae, c["kz"] * nae),
            nae, c["layers"], L.gauss_intp(nae, not lj))
    b = _BASE[key]
    rng = np.random.default_rng(seed)
    jit = JITTER[c["pair"]]
    keep = np.ones(b.natoms, dtype=bool)
    keep[rng.choice(b.natoms, size=c["holes"], replace=False)] = False
    m = L.Model(**{k: getattr(b, k) for k in b.__dataclass_fields__})
    m.atom_x = b.atom_x[keep] + rng.normal(0.0, jit, (int(keep.sum()), 3))
    m.nodex = b.nodex + rng.normal(0.0, jit, b.nodex.shape)
    L.thermalize(m, LJ_T if c["pair"] == "lj" else EAM_T, KB[c["pair"]], MVV2E[c["pair"]], seed + 1)
    L.remap_into_box(m)
    return m


def _prepare_md(c, seed):
    m = _model(c, seed)
    lj = c["pair"] == "lj"
    s = cacg.System(0)
    s.command("units lj" if lj else "units metal")
    s.command("boundary f p p")
    s.load_model(m)
    if lj:
        s.command(f"pair_style lj/cut {LJ_CUT!r}")
        s.command("pair_coeff 1 1 1.0 1.0")
    else:
        t = _eam_tables()
        s.command("pair_style eam")
        s.set_eam(t["nr"], t["dr"], t["nrho"], t["drho"], t["frho"], t["rhor"], t["z2r"],
                  EAM_CUT * EAM_CUT, EAM_MASS)
    s.command(f"neighbor {LJ_SKIN if lj else EAM_SKIN!r} bin")
    s.command("neigh_modify every 1 delay 0 check no" if c["rebuild"] else
              "neigh_modify every 10 delay 0 check yes")
    s.command(f"timestep {LJ_DT if lj else EAM_DT!r}")
    s.command("fix 1 all nve")
    s.set_precision(MODES[c["mode"]])
    s.init()
    s.setup()
    s.neighbor_build()
    s.neighbor_ebuild()
    s.neighbor_nbuild()
    s.pair_compute()
    s.pair_ecompute()
    st = {"case": c, "sys": s}
    for k, a in (("x", m.atom_x), ("v", m.atom_v), ("nodex", m.nodex), ("nodev", m.nodev)):
        st[k + "0"] = _pinned(a.shape)
        st[k + "0"][1][...] = a
        st[k] = _pinned(a.shape)
    st["f"], st["nodef"] = _pinned(m.atom_x.shape), _pinned(m.nodex.shape)
    return st


def _run_md(st):
    c, s = st["case"], st["sys"]
    if c["kind"] == "host":
        for k in ("x", "v", "nodex", "nodev"):
            st[k][0].copy_(st[k + "0"][0])
        s.run_host(c["steps"], *(st[k][1] for k in ("x", "v", "nodex", "nodev")))
        return {"x": st["x"][0], "v": _out(c, st["v"]), "nodex": st["nodex"][0],
                "nodev": _out(c, st["nodev"])}
    s.put_atoms(st["x0"][1], st["v0"][1])
    s.put_nodes(st["nodex0"][1], st["nodev0"][1])
    s.run(c["steps"])
    s.get_state_into(st["x"][1], st["v"][1], st["f"][1])
    s.get_nodes_into(st["nodex"][1], st["nodev"][1])
    return {"x": st["x"][0], "v": _out(c, st["v"]), "f": _out(c, st["f"]),
            "nodex": st["nodex"][0], "nodev": _out(c, st["nodev"])}


def _out(c, buf):
    return buf[0].to(torch.float32) if c["mode"] == "mixed" else buf[0]


def _samples(n, seed):
    """Surrogate samples as the generator makes them look: 24 displacements and 8
    nodal densities in, 24 smooth forces with a few per cent of noise out."""
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n, 32)).astype(np.float32) * np.float32(0.15)
    x[:, 24:] = x[:, 24:] * np.float32(4.0) + np.float32(3.0)
    a = np.random.default_rng(99).normal(size=(32, 24)).astype(np.float32)
    t = np.tanh(x @ a) * np.float32(20.0) + rng.normal(size=(n, 24)).astype(np.float32)
    return x, t.astype(np.float32)


def _weights(members, seed):
    """Weights of `members` networks 32 -> 256 -> 256 -> 256 -> 24, flattened as
    Mlp.set_params takes them."""
    rng = np.random.default_rng(seed + 7)
    out = []
    for _ in range(members):
        p = []
        for rows, cols in ((256, 32), (256, 256), (256, 256), (24, 256)):
            p += [rng.uniform(-1, 1, rows * cols) * math.sqrt(3.0 / cols), rng.normal(0, 0.05, rows)]
        out.append(np.concatenate(p).astype(np.float32))
    return out


def prepare(case, seed):
    c = case
    if c["kind"] in ("md", "host"):
        return _prepare_md(c, seed)
    x, t = _samples(c["n"], seed)
    if c["kind"] == "train":
        return {"case": c, "x": x, "t": t, "weights": _weights(c["members"], seed)}
    net = cacg.Mlp(0, members=c["members"], seed=1)
    net.fit_normalization(x, t)
    for k, w in enumerate(_weights(c["members"], seed)):
        net.set_params(k, w)
    return {"case": c, "x": x, "net": net}


def run(state):
    c = state["case"]
    if c["kind"] in ("md", "host"):
        return _run_md(state)
    if c["kind"] == "predict":
        mean, spread = state["net"].predict(state["x"])
        return {"mean": mean, "spread": spread}
    # what surrogate.train does, from given weights
    net = cacg.Mlp(0, members=c["members"], seed=5)
    for k, w in enumerate(state["weights"]):
        net.set_params(k, w)
    net.fit_normalization(state["x"], state["t"])
    loss = net.train(state["x"], state["t"], epochs=c["epochs"], batch=c["batch"], lr=2e-3, seed=6)
    out = {"loss": loss, "params": [net.params(k) for k in range(c["members"])]}
    net.close()
    return out


def work(case):
    c = case
    if c["kind"] in ("train", "predict"):
        params = 256 * 32 + 2 * 256 * 256 + 24 * 256 + 3 * 256 + 24
        io = c["n"] * 4 * (32 + (24 if c["kind"] == "train" else 25)) + 4 * params * c["members"]
        passes = 6 * c["epochs"] if c["kind"] == "train" else 2
        return {"bytes": io, "flops": float(passes) * c["n"] * params * c["members"]}
    atoms, elems = _sites(c)
    lj = c["pair"] == "lj"
    # neighbours within the cutoff on the perfect lattice, of an atom and of an
    # integration point; operations per pair of the pair functions
    nb, per = (54, 25) if lj else (54, 60)
    rows = 8 * nb + (0 if lj else 8 * 10)
    # per step x, v, f of atoms and nodes read and x, v, f written; the state in and out
    state = 24 * atoms + 192 * elems
    return {"bytes": float(state * (6 * c["steps"] + 9)),
            "flops": float(c["steps"]) * per * (atoms * nb + elems * rows)}


# ---------------------------------------------------------------- in 64 bits

def exact(case, seed):
    c = case
    if c["kind"] == "train":
        return None  # the order of the shuffled samples is the trainer's own
    if c["kind"] == "predict":
        return _exact_predict(c, seed)
    return _exact_md(c, seed)


def _exact_predict(c, seed):
    x, t = _samples(c["n"], seed)
    mean_x, sd_x = x.mean(axis=0).astype(np.float64), x.std(axis=0).astype(np.float64)
    mean_t, sd_t = t.mean(axis=0).astype(np.float64), t.std(axis=0).astype(np.float64)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    xs = torch.from_numpy((x.astype(np.float64) - mean_x) / sd_x).to(dev)
    ys = []
    for p in _weights(c["members"], seed):
        p = torch.from_numpy(p.astype(np.float64)).to(dev)
        h, o = xs, 0
        for k, (rows, cols) in enumerate(((256, 32), (256, 256), (256, 256), (24, 256))):
            w = p[o:o + rows * cols].reshape(rows, cols)
            b = p[o + rows * cols:o + rows * cols + rows]
            o += rows * cols + rows
            h = h @ w.T + b
            if k < 3:
                h = h * torch.sigmoid(h)
        ys.append(h)
    y = torch.stack(ys)
    sd = torch.from_numpy(sd_t).to(dev)
    mean = y.mean(dim=0) * sd + torch.from_numpy(mean_t).to(dev)
    spread = (y.var(dim=0, unbiased=False).sqrt() * sd).max(dim=1).values
    return {"mean": mean.cpu(), "spread": spread.cpu()}


def _cell_pairs(x, length, reach):
    """Ordered pairs (i, j) of points closer than `reach`, periodic in y and z
    (lengths `length`), as int32 tensors sorted by i."""
    n, dev = x.shape[0], x.device
    p = x.clone()
    p[:, 1:] -= torch.floor(p[:, 1:] / length) * length
    lo = p[:, 0].min()
    ext = torch.tensor([float(p[:, 0].max() - lo) + 1e-9, float(length[0]), float(length[1])])
    m = [max(1, int(e // reach)) for e in ext]
    if min(m[1:]) < 3:  # too few cells for a shell of neighbours: all pairs
        d = p[:, None, :] - p[None, :, :]
        d[..., 1:] -= torch.round(d[..., 1:] / length) * length
        ok = (d * d).sum(-1) < reach * reach
        ok.fill_diagonal_(False)
        i, j = torch.nonzero(ok, as_tuple=True)
        return i.int(), j.int()
    q = torch.stack([((p[:, 0] - lo) / ext[0] * m[0]), p[:, 1] / length[0] * m[1],
                     p[:, 2] / length[1] * m[2]], 1).long()
    for d in range(3):
        q[:, d].clamp_(0, m[d] - 1)
    cell = (q[:, 0] * m[1] + q[:, 1]) * m[2] + q[:, 2]
    order = torch.argsort(cell)
    cnt = torch.bincount(cell, minlength=m[0] * m[1] * m[2])
    start = torch.cumsum(cnt, 0) - cnt
    out_i, out_j = [], []
    for c0 in range(0, n, 1 << 17):
        ids = torch.arange(c0, min(n, c0 + (1 << 17)), device=dev)
        for ox in (-1, 0, 1):
            for oy in (-1, 0, 1):
                for oz in (-1, 0, 1):
                    cx = q[ids, 0] + ox
                    inside = (cx >= 0) & (cx < m[0])
                    ii = ids[inside]
                    nc = (cx[inside] * m[1] + (q[ii, 1] + oy) % m[1]) * m[2] + (q[ii, 2] + oz) % m[2]
                    k = cnt[nc]
                    i = torch.repeat_interleave(ii, k)
                    first = torch.cumsum(k, 0) - k
                    j = order[torch.repeat_interleave(start[nc] - first, k)
                              + torch.arange(i.numel(), device=dev)]
                    d = p[i] - p[j]
                    d[:, 1:] -= torch.round(d[:, 1:] / length) * length
                    ok = ((d * d).sum(1) < reach * reach) & (i != j)
                    out_i.append(i[ok].int())
                    out_j.append(j[ok].int())
    return torch.cat(out_i), torch.cat(out_j)


class _Field:
    """Forces of the pair style in 64 bits from given ordered pairs."""

    def __init__(self, c, dev):
        self.lj = c["pair"] == "lj"
        self.cut2 = (LJ_CUT if self.lj else EAM_CUT) ** 2
        if not self.lj:
            t = _eam_tables()
            self.nr, self.nrho, self.dr, self.drho = t["nr"], t["nrho"], t["dr"], t["drho"]
            for k in ("frho", "rhor", "z2r"):
                setattr(self, k, torch.from_numpy(t[k]).to(dev))

    @staticmethod
    def _at(p, n, low):
        m = torch.clamp(torch.clamp(p.long(), max=n - 1), min=low)
        return m, torch.clamp(p - m, max=1.0)

    def density(self, r2):
        """rho(r) within the cutoff, 0 beyond"""
        m, p = self._at(torch.sqrt(r2) / self.dr + 1.0, self.nr, 1)
        s = self.rhor[m]
        return torch.where(r2 < self.cut2, ((s[:, 3] * p + s[:, 4]) * p + s[:, 5]) * p + s[:, 6], 0.0)

    def embed_slope(self, rho):
        m, p = self._at(rho / self.drho + 1.0, self.nrho, 1)
        s = self.frho[m]
        return (s[..., 0] * p + s[..., 1]) * p + s[..., 2]

    def pair(self, r2, fsum):
        """force on i per unit of (x_i - x_j); fsum = F'_i + F'_j (EAM)"""
        if self.lj:
            i2 = 1.0 / r2
            i6 = i2 * i2 * i2
            f = i6 * (48.0 * i6 - 24.0) * i2
        else:
            r = torch.sqrt(r2)
            m, p = self._at(r / self.dr + 1.0, self.nr, 1)
            s, z = self.rhor[m], self.z2r[m]
            drho = (s[:, 0] * p + s[:, 1]) * p + s[:, 2]
            zp = (z[:, 0] * p + z[:, 1]) * p + z[:, 2]
            phi = (((z[:, 3] * p + z[:, 4]) * p + z[:, 5]) * p + z[:, 6]) / r
            f = -(fsum * drho + zp / r - phi / r) / r
        return torch.where(r2 < self.cut2, f, 0.0)


class _Atoms:
    def __init__(self, c, x, length):
        self.field, self.length = _Field(c, x.device), length
        self.margin = 0.4 if c["pair"] == "lj" else 1.0
        self.reach = math.sqrt(self.field.cut2) + self.margin
        self.ref = None

    def force(self, x):
        if self.ref is None or float((x - self.ref).norm(dim=1).max()) > 0.45 * self.margin:
            self.i, self.j = _cell_pairs(x, self.length, self.reach)
            self.ref = x.clone()
        fld, n = self.field, x.shape[0]
        step = 1 << 25
        fp = None
        if not fld.lj:
            rho = torch.zeros(n, dtype=x.dtype, device=x.device)
            for a in range(0, self.i.numel(), step):
                i, j = self.i[a:a + step].long(), self.j[a:a + step].long()
                rho.index_add_(0, i, fld.density(self._d(x, i, j).square().sum(1)))
            fp = fld.embed_slope(rho)
        f = torch.zeros_like(x)
        for a in range(0, self.i.numel(), step):
            i, j = self.i[a:a + step].long(), self.j[a:a + step].long()
            d = self._d(x, i, j)
            g = fld.pair(d.square().sum(1), None if fld.lj else fp[i] + fp[j])
            f.index_add_(0, i, d * g[:, None])
        return f

    def _d(self, x, i, j):
        d = x[i] - x[j]
        d[:, 1:] -= torch.round(d[:, 1:] / self.length) * self.length
        return d


class _Elements:
    """Integration-point forces over each element's own sites, gathered to its
    nodes with weight times shape function."""

    def __init__(self, c, x, dev):
        n = c["nae"]
        lj = c["pair"] == "lj"
        ip, w = L.gauss_intp(n, not lj)
        grid = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3)
        corner = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                           [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], dtype=np.float64)

        def shape(idx):
            xi = -1.0 + 2.0 * idx / (n - 1)
            return np.prod(1.0 + xi[:, None, :] * corner[None], axis=2) / 8.0
        rows, sites = shape(ip), shape(grid)
        self.field = _Field(c, dev)
        # candidates: pairs within the cutoff plus a margin on the ideal lattice
        a = (LJ_A if lj else EAM_A) * 0.5 * np.array([[0, 1, 1], [1, 0, 1], [1, 1, 0]], dtype=np.float64)
        d = np.linalg.norm((ip[:, None, :] - grid[None]) @ a, axis=2)
        r, s = np.nonzero((d < math.sqrt(self.field.cut2) + 1.2) & (d > 0.1))
        put = lambda v: torch.from_numpy(v).to(dev)  # noqa: E731
        self.r, self.rows, self.w = put(r), put(rows), put(w.astype(np.float64))
        self.diff, self.srows = put(rows[r] - sites[s]), put(sites[s])
        self.nodes = None if lj else put(np.array([int(np.where((ip == (corner[q] + 1) / 2 * (n - 1)).all(1))[0][0])
                                                   for q in range(8)]))

    def force(self, x):
        fld, out = self.field, torch.zeros_like(x)
        chunk = max(1, (1 << 25) // self.r.numel())
        for e in range(0, x.shape[0], chunk):
            nx = x[e:e + chunk]
            k = nx.shape[0]
            d = torch.einsum("pq,eqc->epc", self.diff, nx)
            r2 = d.square().sum(2).reshape(-1)
            fsum = None
            if not fld.lj:
                rho = torch.zeros(k, self.rows.shape[0], dtype=x.dtype, device=x.device)
                rho.index_add_(1, self.r, fld.density(r2).reshape(k, -1))
                erho = rho[:, self.nodes]
                fi = fld.embed_slope(erho @ self.rows.T)
                fj = fld.embed_slope(erho @ self.srows.T)
                fsum = (fi[:, self.r] + fj).reshape(-1)
            g = fld.pair(r2, fsum).reshape(k, -1, 1)
            fip = torch.zeros(k, self.rows.shape[0], 3, dtype=x.dtype, device=x.device)
            fip.index_add_(1, self.r, d * g)
            out[e:e + chunk] = torch.einsum("p,pq,epc->eqc", self.w, self.rows, fip)
        return out


def _exact_md(c, seed):
    """Velocity-Verlet of atoms and nodes on forces in 64 bits.  LJ elements are
    left out: whether an element sees its neighbours depends on the bins."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    m = _model(c, seed)
    lj = c["pair"] == "lj"
    put = lambda v: torch.from_numpy(np.ascontiguousarray(v)).to(dev)  # noqa: E731
    length = put((m.boxhi - m.boxlo)[1:])
    dt, mass = (LJ_DT, 1.0) if lj else (EAM_DT, EAM_MASS)
    half = 0.5 * dt / (mass * MVV2E[c["pair"]])
    x, v = put(m.atom_x), put(m.atom_v)
    atoms = _Atoms(c, x, length)
    f = atoms.force(x)
    for _ in range(c["steps"]):
        v = v + half * f
        x = x + dt * v
        f = atoms.force(x)
        v = v + half * f
    wrapped = c["rebuild"]
    if wrapped:  # a rebuild leaves the positions in the box, the last step's as built
        lo = put(m.boxlo[1:])
        x[:, 1:] -= torch.floor((x[:, 1:] - lo) / length) * length
    out = {"x": x.cpu(), "v": v.cpu(), "f": f.cpu(), "nodex": None, "nodev": None}
    if not lj:
        nx, nv = put(m.nodex), put(m.nodev)
        el = _Elements(c, nx, dev)
        half_n = half / (c["nae"] ** 3 / 8.0)
        g = el.force(nx)
        for _ in range(c["steps"]):
            nv = nv + half_n * g
            nx = nx + dt * nv
            g = el.force(nx)
            nv = nv + half_n * g
        if wrapped:
            lo = put(m.boxlo[1:])
            k = torch.floor((nx.mean(dim=1)[:, 1:] - lo) / length)
            nx[:, :, 1:] -= (k * length)[:, None, :]
        out["nodex"], out["nodev"] = nx.cpu(), nv.cpu()
    if c["kind"] == "host":
        del out["f"]
    return out
