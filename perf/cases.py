"""The work a user of this package has it do, as cases of one pass each.

A case is a plain dict; ``prepare`` makes what a program holds before the call
(input files read into a context, trial sites, a recorded random stream),
``run`` is one pass through the public entry points, ``exact`` the same result
from plain torch in 64 bits. Kinds:

propose   the drop-in's host loop: energy differences of a chain move (taken,
          then taken back) and of an ion move (refused)
run       a single system's device step loop (all five move kinds)
batch     independent replicas advanced together in the precision form, with
          the learned first stage where ``net`` is set
total     a stored frame: from-scratch energy and structure factor
grow      configurational-bias growth of one chain: the trial energies of
          every growth step
pressure  one wall-force pressure evaluation of a slit
train     one epoch of the surrogate's training

The precision form adds its pair and reciprocal sums in 32 bits, so its
energies are returned as 32-bit numbers.
"""
import math
import os
import tempfile

import numpy as np
import torch

import plum_gb300 as pg
from plum_gb300 import surrogate, systems

PI = 3.14159265359  # the reference's constant (utilities/constants.h)


# ------------------------------------------------------------------ the cases
def listed():
    bulk1 = dict(n_chain=10, chain_len=50, n_ion=500, box=40.0, alpha_l=5.0)
    bulk20 = dict(n_chain=100, chain_len=100, n_ion=10000, box=80.0, alpha_l=5.6, kmax=12)
    salt = dict(n_chain=40, chain_len=30, n_salt=2000, box=50.0, alpha_l=5.0, trials=32)
    return [
        # the reference's own call surface, one move at a time: latency
        dict(name="propose_1000_fp64", kind="propose", form=0, kmax=7, **bulk1),
        # the plain bulk run with a recorded stream and its per-step log
        dict(name="run_1000_fp64", kind="run", form=0, steps=256, log=True, kmax=7, **bulk1),
        # the same system with the reference's own Ewald rule (image cells)
        dict(name="run_1000_auto_fp64", kind="run", form=0, steps=128, log=False, kmax=0, **bulk1),
        # the benchmark system, plain and precision form
        dict(name="run_20000_fp64", kind="run", form=0, steps=64, log=False, **bulk20),
        dict(name="run_20000_fp32", kind="run", form=1, steps=256, log=False, **bulk20),
        # the benchmark's form: replicas with the learned first stage
        dict(name="batch_20000_net", kind="batch", replicas=32, points=1, steps=512, net=True,
             **bulk20),
        # confined brushes of uneven size, several seeds of each state point
        dict(name="batch_brush", kind="batch", replicas=32, points=8, steps=256, net=False,
             brush=20261203),
        # post-processing a stored frame of the benchmark system
        dict(name="total_20000", kind="total", form=0, **bulk20),
        # grand-canonical growth: neutral chains (precision form), charged (plain)
        dict(name="grow_neutral_fp32", kind="grow", form=1, charge=0, **salt),
        dict(name="grow_charged_fp64", kind="grow", form=0, charge=-1, **salt),
        # the pressure sample of a confined brush with charged wall sites
        dict(name="pressure_brush", kind="pressure", n_graft=40, chain_len=50, height=45.0,
             frac=0.55, n_sites=64),
        # training the surrogate: 16 Adam steps of the usual batch
        dict(name="train_65536", kind="train", rows=65536, batch=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _bulk(rng, most):
    n = _log(rng, 300, most)
    ln = _log(rng, 8, min(150, n // 3))
    n_chain = max(1, int(n * rng.uniform(0.3, 0.6)) // ln)
    n_ion = n_chain * ln  # neutral
    box = ((n_chain * ln + n_ion) / math.exp(rng.uniform(math.log(0.015), math.log(0.04)))) ** (1 / 3)
    return dict(n_chain=n_chain, chain_len=ln, n_ion=n_ion, box=round(box, 3),
                alpha_l=round(rng.uniform(5.0, 5.6), 2), kmax=rng.randint(6, 12))


def draw(rng):
    kind = rng.choice(["propose", "run", "run", "run", "batch", "total", "grow", "pressure",
                       "train"])
    if kind == "propose":
        return dict(kind=kind, form=0, **_bulk(rng, 20000))
    if kind == "run":
        if rng.random() < 0.25:  # the reference's Ewald rule, small systems
            c = _bulk(rng, 1500)
            return dict(c, kind=kind, form=rng.randint(0, 1), steps=rng.randint(40, 130),
                        log=rng.random() < 0.5, kmax=0, box=max(c["box"], 20.0))
        return dict(kind=kind, form=rng.randint(0, 1), steps=rng.randint(40, 260),
                    log=rng.random() < 0.5, **_bulk(rng, 20000))
    if kind == "batch":
        r = _log(rng, 3, 32)
        if rng.random() < 0.5:
            return dict(kind=kind, replicas=r, points=min(r, rng.randint(1, 5)),
                        steps=rng.randint(40, 256), net=False, brush=rng.randint(1, 10**6))
        return dict(kind=kind, replicas=r, points=1, steps=rng.randint(40, 256),
                    net=rng.random() < 0.5, **_bulk(rng, 12000))
    if kind == "total":
        return dict(kind=kind, form=rng.randint(0, 1), **_bulk(rng, 20000))
    if kind == "grow":
        return dict(kind=kind, form=rng.randint(0, 1), charge=rng.choice([0, -1]),
                    n_chain=rng.randint(5, 45), chain_len=rng.randint(5, 33),
                    n_salt=_log(rng, 60, 2000), box=50.0, alpha_l=5.0, trials=rng.randint(5, 40))
    if kind == "pressure":
        return dict(kind=kind, n_graft=rng.randint(16, 64), chain_len=rng.randint(20, 79),
                    height=round(rng.uniform(30, 60), 2), frac=round(rng.uniform(0.1, 1), 2),
                    n_sites=rng.choice([33, 48, 64]))
    return dict(kind=kind, rows=_log(rng, 5000, 65000), batch=rng.choice([1000, 2048, 4096]))


# --------------------------------------------------------------- configurations
class _Place:
    """Overlap-free placement, all chains at once (distances by torch)."""

    def __init__(self, rng, box, periodic, sep=0.8):
        self.rng, self.sep2 = rng, sep * sep
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.box = torch.tensor(box, dtype=torch.float64, device=self.dev)
        self.per = torch.tensor(periodic, dtype=torch.float64, device=self.dev)
        self.zlim = None if periodic[2] else (sep, box[2] - sep)
        self.got = torch.zeros((0, 3), dtype=torch.float64, device=self.dev)

    def near(self, a, b):
        hit = torch.zeros((len(a), len(b)), dtype=torch.bool, device=self.dev)
        if len(a) and len(b):
            d2 = 0
            for k in range(3):
                d = a[:, None, k] - b[None, :, k]
                d2 = d2 + (d - self.per[k] * self.box[k] * torch.round(d / self.box[k])) ** 2
            hit = d2 < self.sep2
        return hit

    def pick(self, cand, own=None):
        """cand [n, t, 3]: per row the first site clear of everything placed
        and of the rows before it; own [n, m, 3]: more beads of that row."""
        n, t, _ = cand.shape
        c = torch.as_tensor(cand, device=self.dev)
        bad = self.near(c.reshape(-1, 3), self.got).any(1).reshape(n, t)
        if self.zlim:
            bad |= (c[..., 2] <= self.zlim[0]) | (c[..., 2] >= self.zlim[1])
        first = torch.argmin(bad.int(), 1)
        ok = ~bad.gather(1, first[:, None])[:, 0]
        site = c[torch.arange(n, device=self.dev), first]
        clash = torch.tril(self.near(site, site), -1) & ok[None, :]
        return site, ok & ~clash.any(1)

    def points(self, n, span):
        out = torch.zeros((n, 3), dtype=torch.float64, device=self.dev)
        left = np.arange(n)
        while len(left):
            site, ok = self.pick(span(len(left)).reshape(len(left), 1, 3))
            sel = torch.as_tensor(left, device=self.dev)[ok]
            out[sel] = site[ok]
            self.got = torch.cat([self.got, site[ok]])
            left = left[~ok.cpu().numpy()]
        return out

    def chains(self, n, length, start):
        """n chains of unit bonds, a bead each per round; a chain that finds
        no room gives up its last ten beads."""
        base = self.got
        at = torch.arange(length, device=self.dev)
        xyz = torch.zeros((n, length, 3), dtype=torch.float64, device=self.dev)
        xyz[:, 0] = self.points(n, start)
        cnt, fails = np.ones(n, np.int64), np.zeros(n, np.int64)
        while (cnt < length).any():
            left = np.flatnonzero(cnt < length)
            sel = torch.as_tensor(left, device=self.dev)
            have = torch.as_tensor(cnt, device=self.dev)
            self.got = torch.cat([base, xyz[at[None, :] < have[:, None]]])
            v = self.rng.normal(size=(len(left), 16, 3))
            v /= np.linalg.norm(v, axis=2, keepdims=True)
            prev = xyz[sel, have[sel] - 1]
            site, ok = self.pick(prev[:, None, :] + torch.as_tensor(v, device=self.dev))
            xyz[sel[ok], have[sel[ok]]] = site[ok]
            ok = ok.cpu().numpy()
            cnt[left[ok]] += 1
            fails[left] = np.where(ok, 0, fails[left] + 1)
            back = fails >= 20
            cnt[back] = np.maximum(1, cnt[back] - 10)
            fails[back] = 0
        self.got = torch.cat([base, xyz.reshape(-1, 3)])
        return xyz


def _system(c, seed):
    """(molecule sizes, symbols, charges, xyz) of a case's bulk or GC box."""
    rng = np.random.default_rng(seed)
    L = c["box"]
    p = _Place(rng, (L, L, L), (1.0, 1.0, 1.0))
    any_ = lambda n: rng.uniform(0, L, (n, 3))  # noqa: E731
    if c["kind"] == "grow":
        nc, ln, q = c["n_chain"], c["chain_len"], float(c["charge"])
        salt = p.points(2 * c["n_salt"], any_)
        ch = p.chains(nc, ln, any_)
        sizes, sym, qs, xyz = [1] * (2 * c["n_salt"]), ["C", "A"] * c["n_salt"], \
            [1.0, -1.0] * c["n_salt"], [salt]
        ci = p.points(nc * ln if q else 0, any_).reshape(nc, -1, 3)
        for k in range(nc):
            sizes.append(ln)
            sym += ["P"] * ln
            qs += [q] * ln
            xyz.append(ch[k])
            if q:
                sizes += [1] * ln
                sym += ["P"] * ln
                qs += [-q] * ln
                xyz.append(ci[k])
        return sizes, sym, np.array(qs), torch.cat(xyz).cpu().numpy()
    nc, ln, ni = c["n_chain"], c["chain_len"], c["n_ion"]
    ch = p.chains(nc, ln, any_)
    io = p.points(ni, any_)
    return ([ln] * nc + [1] * ni, ["P"] * (nc * ln) + ["C"] * ni,
            np.array([-1.0] * (nc * ln) + [1.0] * ni),
            torch.cat([ch.reshape(-1, 3), io]).cpu().numpy())


def _write(d, sizes, sym, q, xyz, box, text):
    mol = np.repeat(np.arange(len(sizes)), sizes)
    systems.write_crd(os.path.join(d, "input_crd.dat"), mol, sym, xyz, q)
    systems.write_top(os.path.join(d, "input_top.dat"), len(mol), len(sizes), box)
    with open(os.path.join(d, "run.in"), "w") as f:
        f.write(text)


def _alpha(c):
    return (c["alpha_l"] / c["box"]) ** 2


def _write_bulk(d, c, seed):
    sizes, sym, q, xyz = _system(c, seed)
    pin = dict(real_cutoff=c["box"] / 2, kmax=c["kmax"], kcut2=-1.0) if c["kmax"] else {}
    _write(d, sizes, sym, q, xyz, (c["box"],) * 3, systems.runin_text(alpha=_alpha(c), **pin))
    return sizes, q, xyz


def _brush(d, spec, seed, charge):
    """One confined brush (systems.BrushSpec) written to d."""
    rng = np.random.default_rng(seed)
    L, H, ns = spec.lxy, spec.height, spec.n_sites
    p = _Place(rng, (L, L, H), (1.0, 1.0, 0.0))
    at = lambda n, z: np.stack([rng.uniform(0, L, n), rng.uniform(0, L, n), z], 1)  # noqa: E731
    walls = np.concatenate([at(ns, np.full(ns, z)) for z in (0.0, H)])
    ch = p.chains(spec.n_graft, spec.chain_len, lambda n: at(n, np.full(n, spec.graft_z)))
    nb = spec.n_graft * spec.chain_len
    ni = int(round(spec.charge_frac * nb))
    cq = -(rng.permutation(nb) < ni).astype(float)
    io = p.points(ni, lambda n: at(n, rng.uniform(0, H, n)))
    sizes = [1] * (2 * ns) + [spec.chain_len] * spec.n_graft + [1] * ni
    sym = ["S"] * (2 * ns) + (["L"] + ["P"] * (spec.chain_len - 1)) * spec.n_graft + ["C"] * ni
    wq = charge * np.tile(1.0 - 2.0 * (np.arange(ns) % 2), 2)
    q = np.concatenate([wq, cq, np.ones(ni)])
    xyz = np.concatenate([walls, ch.reshape(-1, 3).cpu().numpy(), io.cpu().numpy()])
    lj = tuple((s, 1.0, 1.0) for s in "PLCS")
    wall = (("P", 1.0, 1.0), ("L", 1.0, 1.0), ("C", 1.0, 1.0), ("S", 1.0, 0.0))
    _write(d, sizes, sym, q, xyz, (L, L, H), systems.runin_text(
        npbc=2, phantom=2 * ns, grafted=spec.n_graft, grafted_counterion=ni, lj_table=lj,
        alpha=(spec.alpha_times_L / L) ** 2, dipole=True, use_ext=True, wall_table=wall))
    return sizes, q, xyz


def _pressure_spec(c):
    return systems.BrushSpec(n_graft=c["n_graft"], chain_len=c["chain_len"], height=c["height"],
                             charge_frac=c["frac"], n_sites=c["n_sites"])


def _words(seed, n):
    """The first n words of std::mt19937(seed)."""
    key = np.zeros(624, np.uint32)
    x = seed & 0xFFFFFFFF
    key[0] = x
    for i in range(1, 624):
        x = (1812433253 * (x ^ (x >> 30)) + i) & 0xFFFFFFFF
        key[i] = x
    g = np.random.MT19937()
    g.state = {"bit_generator": "MT19937", "state": {"key": key, "pos": 624}}
    return g.random_raw(n).astype(np.uint32)


def _run_words(c, seed):
    return _words(seed + 77, c["steps"] * (30 + 8 * c["chain_len"]))


def _proposals(c, seed, sizes, xyz):
    """(molecule, trial positions) of a chain turned about its first bead and
    of an ion moved as BeadTranslate moves one."""
    rng = np.random.default_rng(seed + 5)
    start = np.concatenate([[0], np.cumsum(sizes)])
    m, i = int(rng.integers(c["n_chain"])), c["n_chain"] + int(rng.integers(c["n_ion"]))
    x = xyz[start[m]:start[m + 1]]
    ax = rng.normal(size=3)
    ax /= np.linalg.norm(ax)
    an = rng.uniform(0.02, 0.05)
    K = np.array([[0, -ax[2], ax[1]], [ax[2], 0, -ax[0]], [-ax[1], ax[0], 0]])
    R = np.eye(3) + np.sin(an) * K + (1 - np.cos(an)) * K @ K
    v = rng.normal(size=3)
    return (m, x[0] + (x - x[0]) @ R.T), (i, xyz[start[i]:start[i] + 1] + v / np.linalg.norm(v))


def _growth(c, seed):
    """Per growth step the trial sites, trial counterions and grown beads."""
    rng = np.random.default_rng(seed + 9)
    n, T, L = c["chain_len"], c["trials"], c["box"]
    unit = rng.normal(size=(n, T, 3))
    unit /= np.linalg.norm(unit, axis=2, keepdims=True)
    chain, ci, steps = np.zeros((0, 3)), np.zeros((0, 3)), []
    for k in range(n):
        b1 = rng.uniform(0, L, (T, 3)) if k == 0 else chain[-1] + unit[k]
        b2 = rng.uniform(0, L, (T, 3)) if c["charge"] else None
        steps.append((b1, b2, chain, ci if c["charge"] else None))
        chain = np.concatenate([chain, b1[:1]])
        if c["charge"]:
            ci = np.concatenate([ci, b2[:1]])
    return steps


def _training(c, seed):
    """Descriptors and clipped energy changes with the shipped data's spread."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = torch.Generator(device="cpu").manual_seed(int(seed))
    x = torch.rand((c["rows"], 96), generator=g).pow(2) * 20
    w = torch.randn(96, generator=g) / 12
    t = (x @ w + 2 * torch.randn(c["rows"], generator=g)).clamp(-20, 20)
    return x.to(dev), t.to(dev)


# ---------------------------------------------------------------- prepare, run
def prepare(case, seed):
    c = dict(case)
    s = {"case": c}
    with tempfile.TemporaryDirectory() as d:
        if c["kind"] == "train":
            x, t = _training(c, seed)
            mu, isd = surrogate.normalisation(x)
            s["net"] = pg.Surrogate(seed=1 + seed % 1000)
            s["net"].set_norm(mu, isd, float(t.std()))
            s["x"], s["t"] = x, t
            return s
        if c["kind"] == "batch":
            if "brush" in c:
                specs = systems.brush_ensemble(c["points"], c["brush"])
                dirs = [os.path.join(d, str(k)) for k in range(c["points"])]
                for k, spec in enumerate(specs):
                    os.makedirs(dirs[k])
                    _brush(dirs[k], spec, seed + k, 0.0)
            else:
                dirs = [d]
                _write_bulk(d, c, seed)
            s["b"] = pg.Batch([dirs[r % len(dirs)] for r in range(c["replicas"])])
            s["b"].seed(np.arange(c["replicas"], dtype=np.uint32) + np.uint32(seed % 2**31))
            s["b"].set_tune(32768 if not c.get("brush") else 4096, 1024, 608, 3)
            s["b"].set_groups(2 if c["replicas"] > 1 else 1)
            if c["net"]:
                s["net"] = surrogate.load(os.path.join(os.path.dirname(pg.__file__), "data",
                                                       "surrogate_bulk_20000_pinned.npz"))
                s["net"].set_margin(12.0)
                s["b"].set_surrogate(s["net"])
            s["reps"] = [s["b"].replica(r) for r in range(c["replicas"])]
            return s
        if c["kind"] == "pressure":
            _brush(d, _pressure_spec(c), seed, 0.5)
            s["s"] = pg.System(d)
            return s
        if c["kind"] == "grow":
            sizes, sym, q, xyz = _system(c, seed)
            gc = dict(chem_pot=0.0, deBroglie=1, gc_freq=2, chain_len=c["chain_len"],
                      bead_charge=c["charge"], bead_symbol="P", cbmc_trials=c["trials"])
            _write(d, sizes, sym, q, xyz, (c["box"],) * 3, systems.runin_text(
                lj_table=tuple((t, 1.0, 1.0) for t in "PCA"), alpha=_alpha(c), use_gc=True, gc=gc,
                coion=2 * c["n_salt"], move_prob=(0.5, 0.1, 0.2, 0.0, 0.2)))
            s["s"] = pg.System(d, form=c["form"])
            s["steps"] = _growth(c, seed)
            return s
        sizes, q, xyz = _write_bulk(d, c, seed)
        s["s"] = pg.System(d, form=c["form"])
        if c["kind"] == "propose":
            (m, t), (i, ti) = _proposals(c, seed, sizes, xyz)
            b0 = sum(sizes[:m])
            s["moves"] = [(m, t, True), (m, xyz[b0:b0 + sizes[m]], True), (i, ti, False)]
            s["flags"] = {k: np.ones(sizes[k], np.int32) for k in (m, i)}
        elif c["kind"] == "total":
            s["xyz"] = xyz + np.random.default_rng(seed + 3).uniform(-0.05, 0.05, xyz.shape)
        elif c["log"]:
            s["words"] = _run_words(c, seed)
        else:
            s["s"].seed(seed + 77)
    return s


def _values(c, v):
    return v.astype(np.float32) if c.get("form", 1) else v


def run(state):
    c = state["case"]
    if c["kind"] == "propose":
        de = []
        for m, trial, accept in state["moves"]:
            de.append(state["s"].energy_difference(m, trial, state["flags"][m]))
            state["s"].finalize(accept)
        return {"de": np.stack(de), "energies": state["s"].energies()}
    if c["kind"] == "run":
        if c["log"]:
            used, mt, ac, et = state["s"].run_moves(state["words"], c["steps"])
            return {"used": used, "types": mt, "accepted": ac, "etot": _values(c, et),
                    "xyz": state["s"].positions()}
        acc = state["s"].run(c["steps"])
        return {"accepted": acc, "energies": _values(c, state["s"].energies()),
                "xyz": state["s"].positions()}
    if c["kind"] == "batch":
        acc = state["b"].run(c["steps"])
        return {"accepted": acc, "energies": _values(c, state["b"].energies()),
                "xyz": np.concatenate([r.positions() for r in state["reps"]])}
    if c["kind"] == "total":
        state["s"].set_positions(state["xyz"])
        return {"energies": state["s"].energies(), "sk": state["s"].structure_factor()[0]}
    if c["kind"] == "grow":
        return _values(c, np.stack([state["s"].cbmc_trials(*step) for step in state["steps"]]))
    if c["kind"] == "pressure":
        return state["s"].pressure_slit()
    losses = state["net"].train(state["x"], state["t"], batch=c["batch"], epochs=1, lr=1e-3, seed=3)
    return {"params": state["net"].params(), "loss": losses.astype(np.float32)}


# ------------------------------------------------------------------------ work
def _rule(lB, alpha, edge):
    """The reference's automatic real-space cut-off and k^2 cut-off."""
    rc = 1.0
    while 0.5 * lB * math.erfc(math.sqrt(alpha) * rc) / rc > 1e-7:
        rc += 1
    kc2 = alpha
    while lB / (2 * PI * edge ** 3) * 4 * PI * PI * math.exp(-kc2 / (4 * alpha)) / kc2 > 1e-7:
        kc2 += alpha
    return rc, kc2


def _ewald(c):
    """(r_c, k vectors [n, 3] of the half space, weights, Ewald box, alpha)."""
    if "height" in c:
        L, H = 32.0, c["height"]
        box, alpha = (L, L, 3 * H if 3 * H > 150 else H + 150), (5.0 / L) ** 2
    else:
        box, alpha = (c["box"],) * 3, _alpha(c)
    if c.get("kmax"):
        rc, kc2, n = c["box"] / 2, math.inf, (c["kmax"],) * 3
    else:
        rc, kc2 = _rule(3.0, alpha, box[0])
        n = [math.ceil(math.sqrt(kc2) * b / (2 * PI)) for b in box]
    g = np.stack(np.meshgrid(*[np.arange(-m, m + 1) for m in n], indexing="ij"), -1).reshape(-1, 3)
    half = (g[:, 0] > 0) | ((g[:, 0] == 0) & ((g[:, 1] > 0) | ((g[:, 1] == 0) & (g[:, 2] > 0))))
    k = g * 2 * PI / np.array(box)
    k2 = (k ** 2).sum(1)
    keep = half & (k2 > 0) & (k2 <= kc2)
    return rc, k[keep], np.exp(-k2[keep] / (4 * alpha)) / k2[keep], box, alpha


def work(case):
    c = case
    if c["kind"] == "train":
        return {"bytes": c["rows"] * 97 * 4.0 + 8 * 29000, "flops": c["rows"] * 6.0 * 28800}
    if c["kind"] == "batch" and "brush" in c:
        spec = systems.brush_ensemble(c["points"], c["brush"])
        n = sum(s.n_graft * s.chain_len * (1 + s.charge_frac) + 128 for s in spec) / len(spec)
        m = sum(s.chain_len for s in spec) / len(spec)
        nk, share = 1500.0, 0.9
        moves = c["steps"] * c["replicas"]
        reps = c["replicas"]
    elif c["kind"] == "pressure":
        n = c["n_graft"] * c["chain_len"] * (1 + c["frac"]) + 2 * c["n_sites"]
        nk = len(_ewald(c)[1])
        return {"bytes": n * 32.0 + nk * 16 + 48,
                "flops": 2 * c["n_sites"] * n * 57.0 + 16.0 * n * nk}
    else:
        rc, k, _, box, _ = _ewald(c)
        nk = len(k)
        share = 4.19 * (rc / box[0]) ** 3  # evaluations inside the cut-off per pair
        if c["kind"] == "grow":
            n = 2 * c["n_salt"] + c["n_chain"] * c["chain_len"] * (2 if c["charge"] else 1)
            two = 2 if c["charge"] else 1
            t = c["chain_len"] * c["trials"] * two
            return {"bytes": c["chain_len"] * (n * 32.0 + (nk * 16 if c["charge"] else 0))
                    + 40.0 * t,
                    "flops": t * (20.0 * n + (25 * share * n + 26 * nk if c["charge"] else 0))}
        n = c["n_chain"] * c["chain_len"] + c["n_ion"]
        if c["kind"] == "total":
            return {"bytes": n * 48.0 + nk * 32, "flops": n * n / 2 * (20 + 25 * share)
                    + 16.0 * n * nk}
        m = c["chain_len"] * 0.6
        moves = (c.get("steps") or 3) * c.get("replicas", 1)
        reps = c.get("replicas", 1)
    return {"bytes": reps * (n * 56.0 + nk * 32),
            "flops": moves * (m * n * (20 + 2 * 25 * share) + 16.0 * m * nk + 10 * nk)}


# ----------------------------------------------------------------------- exact
class _Model:
    """LJ + Ewald + bonds of a case in 64 bits (plain torch)."""

    def __init__(self, c, q):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.rc, k, w, self.ebox, self.alpha = _ewald(c)
        self.t = lambda v: torch.as_tensor(v, dtype=torch.float64, device=self.dev)
        self.k, self.w, self.q = self.t(k), self.t(w), self.t(q)
        self.lB, self.box = 3.0, self.ebox[0]
        self.pref = self.lB / (PI * self.box ** 3) * 4 * PI * PI
        self.ref = 4 * (2.5 ** -12 - 2.5 ** -6)

    def pair(self, a, qa, b, qb, mask=None, same=False):
        """(LJ [n, m], real space [n, m]) of beads a with beads b; mask drops
        pairs, same leaves out each bead's own zero-distance image."""
        d = [a[:, None, k] - b[None, :, k] for k in range(3)]
        d = [x - self.box * torch.round(x / self.box) for x in d]
        r2 = sum(x * x for x in d)
        s6 = (1 / r2.clamp_min(1e-300)) ** 3
        lj = torch.where(r2 < 6.25, 4 * (s6 * s6 - s6) - self.ref, torch.zeros_like(r2))
        lj = torch.where(r2 <= 0, torch.full_like(r2, 1e8), lj)
        n = math.ceil(self.rc / self.box) if self.rc > self.box / 2 else 0
        re, sa = torch.zeros_like(r2), math.sqrt(self.alpha)
        for i in range(-n, n + 1):
            for j in range(-n, n + 1):
                for k in range(-n, n + 1):
                    r = sum((x + o * self.box) ** 2 for x, o in zip(d, (i, j, k))).sqrt()
                    ok = (r > 0) & (r <= self.rc)
                    re += torch.where(ok, torch.erfc(sa * r) / r.clamp_min(1e-300),
                                      torch.zeros_like(r))
        re = re * self.lB * qa[:, None] * qb[None, :]
        if mask is not None:
            lj, re = lj * mask, re * mask
        return lj, re

    def sk(self, x, q):
        out = torch.zeros(len(self.k), dtype=torch.complex128, device=self.dev)
        w = x - self.t(self.ebox) * torch.floor(x / self.t(self.ebox))
        for i in range(0, len(x), 2000):
            ph = w[i:i + 2000] @ self.k.T
            out += (q[i:i + 2000, None] * torch.complex(torch.cos(ph), torch.sin(ph))).sum(0)
        return out

    def recip(self, s):
        return float(self.pref * (self.w * (s.real ** 2 + s.imag ** 2)).sum())

    def total(self, x, sizes):
        lj = re = 0.0
        for i in range(0, len(x), 1000):
            up = torch.ones((len(x[i:i + 1000]), len(x)), dtype=torch.float64,
                            device=self.dev).triu(i + 1)
            a, b = self.pair(x[i:i + 1000], self.q[i:i + 1000], x, self.q, up)
            lj, re = lj + float(a.sum()), re + float(b.sum())
        s = self.sk(x, self.q)
        o = torch.zeros((1, 3), dtype=torch.float64, device=self.dev)
        one = torch.ones(1, dtype=torch.float64, device=self.dev)
        img = float(self.pair(o, one, o, one)[1])  # a bead's own images
        q2 = float((self.q ** 2).sum())
        ew = re + self.recip(s) - self.lB * math.sqrt(self.alpha / PI) * q2 + 0.5 * img * q2
        bond, b0 = 0.0, 0
        for n in sizes:
            if n == 1:
                break  # the chains come first
            bond += self.bond(x[b0:b0 + n])
            b0 += n
        return [lj, ew, bond, 0.0], s

    @staticmethod
    def bond(x):
        r = (x[1:] - x[:-1]).norm(dim=1)
        return float((200.0 * (r - 1.0) ** 2).sum())

    def change(self, x, lo, hi, trial, s):
        """(pair, ewald, new S(k)) of moving beads [lo, hi) to trial."""
        rest = torch.ones(len(x), dtype=torch.bool, device=self.dev)
        rest[lo:hi] = False
        up = torch.ones((hi - lo, hi - lo), dtype=torch.float64, device=self.dev).triu(1)
        lj, re = [], []
        for p in (trial, x[lo:hi]):
            a, b = self.pair(p, self.q[lo:hi], x[rest], self.q[rest])
            c, d = self.pair(p, self.q[lo:hi], p, self.q[lo:hi], up)
            lj.append(float(a.sum() + c.sum()))
            re.append(float(b.sum() + d.sum()))
        s2 = s + self.sk(trial, self.q[lo:hi]) - self.sk(x[lo:hi], self.q[lo:hi])
        return lj[0] - lj[1], re[0] - re[1] + self.recip(s2) - self.recip(s), s2


class _Chain:
    """The Monte Carlo chain itself (Simulation::Run's draws and moves)."""

    M = 4294967295.0

    def __init__(self, c, words):
        self.c, self.g, self.p = c, words, 0

    def word(self):
        self.p += 1
        return int(self.g[self.p - 1])

    def u(self):
        return self.word() / self.M

    def sphere(self):
        while True:
            a, b = 1 - 2 * self.u(), 1 - 2 * self.u()
            if a * a + b * b <= 1:
                r = a * a + b * b
                h = 2 * math.sqrt(1 - r)
                return np.array([a * h, b * h, 1 - 2 * r])

    def propose(self, x, start):
        """(type, molecule, lo, hi, trial) of the next step."""
        c = self.c
        self.word()
        ch = min(int(math.floor(self.u() * c["n_chain"])), c["n_chain"] - 1)
        io = min(int(math.floor(self.u() * c["n_ion"])), c["n_ion"] - 1)
        u, mt, cur, prob = self.u(), 0, 0.3, (0.3, 0.1, 0.2, 0.2, 0.2)
        while cur < u and mt < 4:
            mt += 1
            cur += prob[mt]
        m = ch if mt else c["n_chain"] + io
        lo, hi = start[m], start[m + 1]
        old = x[lo:hi].cpu().numpy()
        n = hi - lo
        if mt == 0:
            v = self.sphere()
            return mt, m, lo, hi, old + 3 / math.sqrt((v * v).sum()) * v
        if mt == 1:
            v = np.array([0.5 * self.word() / self.M for _ in range(3)])
            return mt, m, lo, hi, old + np.array([-a if self.word() % 2 == 0 else a for a in v])
        if mt == 2:
            pv = min(int(math.floor(n * float(self.word()) / self.M)), n - 1)
            s = float(self.word()) / self.M
            new = old.copy()
            for rng_ in (range(pv + 1, n), range(pv - 1, -1, -1)):
                for i in rng_:
                    j = i - 1 if i > pv else i + 1
                    d = old[i] - old[j] + s * self.sphere()
                    new[i] = new[j] + (1.0 + 0.2 * (self.u() - 0.5)) / np.linalg.norm(d) * d
            return mt, m, lo, hi, new
        if mt == 3:
            first = int(math.floor((n - 2) * float(self.word()) / self.M))
            last = min(int(math.floor((n - first) * float(self.word()) / self.M)) + first, n - 1)
            ax = old[last] - old[first]
            if (ax * ax).sum() > 0:
                ax = ax / np.linalg.norm(ax)
            an = self.u() * 2 * math.pi - math.pi
            K = np.array([[0, -ax[2], ax[1]], [ax[2], 0, -ax[0]], [-ax[1], ax[0], 0]])
            R = np.cos(an) * np.eye(3) + np.sin(an) * K + (1 - np.cos(an)) * np.outer(ax, ax)
            a, b = first + 1, max(last, first + 1)
            return mt, m, lo + a, lo + b, old[first] + (old[a:b] - old[first]) @ R.T
        bl = 1.0 + 0.2 * (self.u() - 0.5)
        back = self.word() % 2 == 0
        v = self.sphere()
        v = bl * v / np.linalg.norm(v)
        new = np.concatenate([old[:1] + v, old[:-1]] if back else [old[1:], old[-1:] + v])
        return mt, m, lo, hi, new


def _replay(c, seed):
    sizes, _, q, xyz = _system(c, seed)
    M = _Model(c, q)
    x = M.t(xyz)
    start = np.concatenate([[0], np.cumsum(sizes)])
    e, s = M.total(x, sizes)
    words = _run_words(c, seed)
    chain, etot, acc = _Chain(c, words), [], 0
    for _ in range(c["steps"]):
        mt, m, lo, hi, trial = chain.propose(x, start)
        trial = M.t(trial)
        pair, ew, s2 = M.change(x, lo, hi, trial, s) if hi > lo else (0.0, 0.0, s)
        new = x[start[m]:start[m + 1]].clone()
        new[lo - start[m]:hi - start[m]] = trial
        bond = M.bond(new) - M.bond(x[start[m]:start[m + 1]]) if sizes[m] > 1 else 0.0
        de = pair if pair >= 1e8 else pair + ew + bond
        if de < 1e8 and (chain.u() < math.exp(min(0.0, -de)) or de <= 0):
            x[lo:hi] = trial
            s, acc = s2, acc + 1
            e = [e[0] + pair, e[1] + ew, e[2] + bond, 0.0]
        etot.append(sum(e))
    return {"used": None, "types": None, "accepted": None, "energies": np.array(e),
            "etot": np.array(etot), "xyz": x.cpu().numpy()}


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "train":
        return None  # 16-bit operands by design; Adam's first steps follow the sign of a gradient
    if c["kind"] == "batch":
        return None  # thousands of moves of every replica: minutes
    if c["kind"] == "run":
        o = _replay(c, seed)
        return {k: o[k] for k in (("used", "types", "accepted", "etot", "xyz") if c["log"]
                                  else ("accepted", "energies", "xyz"))}
    if c["kind"] == "pressure":
        return _pressure(c, seed)
    sizes, _, q, xyz = _system(c, seed)
    M = _Model(c, q)
    if c["kind"] == "total":
        x = xyz + np.random.default_rng(seed + 3).uniform(-0.05, 0.05, xyz.shape)
        e, s = M.total(M.t(x), sizes)
        return {"energies": np.array(e), "sk": s.cpu().numpy()}
    x = M.t(xyz)
    if c["kind"] == "propose":
        (m, t), (i, ti) = _proposals(c, seed, sizes, xyz)
        start = np.concatenate([[0], np.cumsum(sizes)])
        e, s = M.total(x, sizes)
        rows = []
        for k, trial in ((m, t), (i, ti)):
            lo, hi = start[k], start[k + 1]
            pair, ew, _ = M.change(x, lo, hi, M.t(trial), s)
            bond = M.bond(M.t(trial)) - M.bond(x[lo:hi]) if sizes[k] > 1 else 0.0
            rows.append(np.array([pair + ew + bond, pair, ew, bond, 0.0])
                        if pair < 1e8 else np.array([pair, pair, 0.0, 0.0, 0.0]))
        return {"de": np.stack([rows[0], -rows[0], rows[1]]), "energies": np.array(e)}
    # grow
    sk = M.sk(x, M.q)
    q1, out = float(c["charge"]), []
    for b1, b2, chain, ci in _growth(c, seed):
        T, cl = len(b1), len(chain)
        sites = [(M.t(b1), q1)] + ([(M.t(b2), -q1)] if q1 else [])
        grown = [(M.t(chain), q1)] + ([(M.t(ci), -q1)] if q1 else [])
        one = lambda n, v: M.t(np.full(n, v))  # noqa: E731
        pair, ew = torch.zeros(T, device=M.dev, dtype=torch.float64), 0.0
        so, e = sk, 0.0
        for g, (gx, gq) in enumerate(grown):
            if cl:
                so = so + M.sk(gx, one(cl, gq))
        for a, (sx, sq) in enumerate(sites):
            lj, re = M.pair(sx, one(T, sq), x, M.q)
            pair, ew = pair + lj.sum(1), ew + re.sum(1)
            for g, (gx, gq) in enumerate(grown):
                if cl:
                    lj, re = M.pair(sx, one(T, sq), gx, one(cl, gq))
                    if a == 0 and g == 0:
                        lj[:, -1] = 0  # bonded to the bead before it
                    pair, ew = pair + lj.sum(1), ew + re.sum(1)
            ph = (sx - M.box * torch.floor(sx / M.box)) @ M.k.T
            e = e + sq * torch.complex(torch.cos(ph), torch.sin(ph))
            img = M.pair(sx[:1], one(1, sq), sx[:1], one(1, sq))[1]
            ew = ew - M.lB * math.sqrt(M.alpha / PI) * sq * sq + 0.5 * float(img)
        if q1:
            lj, re = M.pair(sites[0][0], one(T, q1), sites[1][0], one(T, -q1))
            pair, ew = pair + lj.diagonal(), ew + re.diagonal()
            n2 = (so + e).abs() ** 2 - so.abs() ** 2
            ew = ew + M.pref * (M.w * n2).sum(1)
        out.append(torch.where(pair >= 1e8, torch.full_like(pair, 1e8), pair + ew).cpu().numpy())
    return np.stack(out)


def _pressure(c, seed):
    with tempfile.TemporaryDirectory() as d:
        sizes, q, xyz = _brush(d, _pressure_spec(c), seed, 0.5)
    rc, k, w, ebox, alpha = _ewald(c)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = lambda v: torch.as_tensor(v, dtype=torch.float64, device=dev)  # noqa: E731
    ns, L, H, lB, sa = c["n_sites"], 32.0, c["height"], 3.0, math.sqrt(alpha)
    nch = c["n_graft"] * c["chain_len"]
    wall = t(xyz[:2 * ns])
    groups = {0: slice(2 * ns + nch, None), 1: slice(2 * ns, 2 * ns + nch), 2: slice(ns, 2 * ns)}
    out = np.zeros(6)
    cells = [math.ceil(rc / b) for b in ebox]
    for kid, sl in groups.items():
        b, qb = t(xyz[sl]), t(q[sl])
        for side in (0, 1):
            if kid == 2 and side == 1:
                continue
            a, qa = wall[side * ns:(side + 1) * ns], t(q[side * ns:(side + 1) * ns])
            C = -1.0 if kid == 2 else (0.5 if side else -0.5)
            d = [a[:, None, j] - b[None, :, j] for j in range(3)]
            d[0], d[1] = (x - L * torch.round(x / L) for x in d[:2])
            r = sum(x * x for x in d).sqrt()
            x6 = (1 / r.clamp(max=2.5)) ** 6  # beyond the cut-off: its r^-6 term at r
            out[kid] += C * float((d[2] / r * 4 * (12 * x6 * x6 - 6 * x6) / r).sum())
            f = torch.zeros_like(r)
            for i in range(-cells[0], cells[0] + 1):
                for j in range(-cells[1], cells[1] + 1):
                    for l in range(-cells[2], cells[2] + 1):
                        z = d[2] + l * ebox[2]
                        s = ((d[0] + i * L) ** 2 + (d[1] + j * L) ** 2 + z * z).sqrt()
                        v = (2 * math.sqrt(alpha / PI) * torch.exp(-alpha * s * s)
                             + torch.erfc(sa * s) / s) * z / (s * s)
                        f += torch.where(s <= rc, v, torch.zeros_like(v))
            out[3 + kid] += C * float((lB * qa[:, None] * qb[None, :] * f).sum())
            kk = t(k)

            def sk(p, c_):
                wr = p.clone()
                wr[:, :2] -= L * torch.floor(wr[:, :2] / L)
                ph = wr @ kk.T
                return (c_[:, None] * torch.complex(torch.cos(ph), torch.sin(ph))).sum(0)
            im = (sk(a, qa) * sk(b, qb).conj()).imag
            pre = lB * 4 * PI / (ebox[0] * ebox[1] * ebox[2]) * 2
            out[3 + kid] += C * pre * float((kk[:, 2] * t(w) * im).sum())
        if kid != 2:  # half the 9-3 wall's force on every system bead
            z = t(xyz[sl])[:, 2]
            u = H - z
            r0, k0 = 3 * 1.25992104989, 2.59807621135
            w93 = lambda h: k0 * (6 * h ** -7 - 3 * h ** -4)  # noqa: E731
            zero = torch.zeros_like(z)
            far = torch.where(u < 1.25992104989, w93(u), zero)
            f = torch.where(z < 1.25992104989, w93(z), zero) + far
            if kid == 1:  # the first bead of each chain is tethered
                first = torch.arange(len(z), device=dev) % c["chain_len"] == 0
                f = torch.where(first, w93(z) - r0 * z / (1 - (z / r0) ** 2) + far, f)
            out[kid] += 0.5 * float(f.sum())
    return out
