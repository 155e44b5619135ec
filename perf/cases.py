"""What this framework is timed on: the calls its users make, over the sizes they make them at.

Every case is one user-level call sequence through the package's public entry points:

  embed       the allocation-free step on device arrays the caller owns (its own time loop around it)
  solve       upload an initial state, run the solve to its horizon, read the final state back;
              several parameter sets in turn on one pool, as a sequential calibration runs them
  adaptive    one interval between two adaptations of a multi-level grid: the state in, the steps, the
              wavelet details that drive refinement, the state out
  stage       one TMCMC stage: every sample's forward solve and its likelihood (optionally its final field)
  gradient    loss and gradients of one calibration sample through torch.autograd
  likelihood  the log-likelihood of a state that is on the device
  stream      host-to-host solves, each from its own pinned initial state

The anatomy is a seeded synthetic brain (white and grey matter, CSF ventricles), built on the GPU.  Parameters are in
the ranges of the calibration (Dw in cm^2/day, rho in 1/day, a 25.6 cm domain).
"""
import ctypes
import math

import numpy as np
import torch

from gliomasolver_b200 import BlockPool, _lib
from gliomasolver_b200.autograd import tumor_loss
from gliomasolver_b200.tmcmc import Batch, GliomaModel, StageSample, to_gbfk_samples

L_CM = 25.6
UC = {"t1_uc": 0.7, "t2_uc": 0.25, "slope": 2.0}


def listed():
    return [
        # the smallest call: one step of a 32^3 grid inside another code's time loop
        {"name": "embed_32_f32", "kind": "embed", "bpd": 4, "real": "f32"},
        # the parity configuration: 64^3 in FP64 to T = 150 days
        {"name": "solve_64_f64", "kind": "solve", "bpd": 8, "real": "f64", "steps": 739, "sets": 1},
        # sequential calibration samples at the usual patient resolution, FP32 storage
        {"name": "solve_128_f32", "kind": "solve", "bpd": 16, "real": "f32", "steps": 1500, "sets": 2},
        # the finest uniform grid, FP32 storage
        {"name": "solve_256_f32", "kind": "solve", "bpd": 32, "real": "f32", "steps": 2000, "sets": 1},
        # a grid cropped to the head: not a power of two blocks per direction
        {"name": "solve_120_f64", "kind": "solve", "bpd": 15, "real": "f64", "steps": 400, "sets": 1},
        # an adaptive run's interval: two levels, 190 leaves
        {"name": "adaptive_190_f32", "kind": "adaptive", "base": 4, "fine": "2x3x3", "real": "f32", "steps": 20},
        # a coarse exploratory stage whose fields are kept (posterior maps)
        {"name": "stage_64_f32", "kind": "stage", "bpd": 8, "real": "f32", "samples": 48, "days": 60.0, "fields": True},
        # a calibration stage: the population's log-likelihoods
        {"name": "stage_128_f32", "kind": "stage", "bpd": 16, "real": "f32", "samples": 32, "days": 60.0, "fields": False},
        # a gradient with respect to the initial field, full precision, few checkpoints
        {"name": "gradient_64_f64", "kind": "gradient", "bpd": 8, "real": "f64", "steps": 739, "checkpoints": 32, "wrt": "c0"},
        # a gradient calibration sample (Dw, rho, origin) at patient resolution
        {"name": "gradient_128_f32", "kind": "gradient", "bpd": 16, "real": "f32", "steps": 1500, "checkpoints": 64, "wrt": "x0"},
        # the likelihood of one 256^3 state, with a PET signal
        {"name": "likelihood_256_f32", "kind": "likelihood", "bpd": 32, "real": "f32", "pet": True},
        # short forecasts from states that live in host memory
        {"name": "stream_128_f32", "kind": "stream", "bpd": 16, "real": "f32", "steps": 50, "states": 6},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["embed", "solve", "solve", "solve", "adaptive", "stage", "stage", "gradient", "gradient", "likelihood",
                       "stream"])
    real = rng.choice(["f32", "f64"])
    if kind == "embed":
        return {"kind": kind, "bpd": rng.randint(1, 8), "real": real}
    if kind == "solve":
        bpd = _log(rng, 4, 32 if real == "f32" else 24)
        most = int(2000 * min(1.0, (16 / bpd) ** 3 * (4 if real == "f32" else 2)))
        return {"kind": kind, "bpd": bpd, "real": real, "steps": _log(rng, 30, max(most, 60)), "sets": rng.randint(1, 2)}
    if kind == "adaptive":
        base = rng.randint(3, 8)
        fine = "x".join(str(rng.randint(1, base - 1)) for _ in range(3))
        return {"kind": kind, "base": base, "fine": fine, "real": real, "steps": rng.randint(5, 40)}
    if kind == "stage":
        bpd = rng.choice([4, 6, 8, 12, 16])
        most = 60 if bpd <= 8 else 24
        return {"kind": kind, "bpd": bpd, "real": real, "samples": _log(rng, 3, most), "days": rng.uniform(10.0, 60.0),
                "fields": bpd <= 8 and rng.random() < 0.5}
    if kind == "gradient":
        bpd = rng.choice([4, 8, 16])
        return {"kind": kind, "bpd": bpd, "real": real, "steps": _log(rng, 40, 700 if bpd == 16 else 1400),
                "checkpoints": _log(rng, 4, 200), "wrt": rng.choice(["c0", "x0"])}
    if kind == "likelihood":
        return {"kind": kind, "bpd": rng.choice([4, 8, 16, 32]), "real": real, "pet": rng.random() < 0.5}
    return {"kind": kind, "bpd": rng.randint(3, 16), "real": real, "steps": rng.randint(1, 80), "states": rng.randint(2, 6)}


# ---------------------------------------------------------------- inputs
def _real(case):
    return np.float64 if case["real"] == "f64" else np.float32


def _tdt(case):
    return torch.float64 if case["real"] == "f64" else torch.float32


def _coefficients(R, Dw, rho, n):
    """The solver's schedule in its own Real: rescaled Dw and Dg, rho, and the step of an n^3 grid."""
    L = R(L_CM)
    dw = R(R(Dw) / (L * L))
    dg = R(0.1 * np.float64(dw))
    h = np.float64(R(1.0 / n))
    return float(dw), float(dg), float(R(rho)), float(R(0.99 * h * h / (6.0 * np.float64(dw))))


def _grid(n, dev, origin=(0.0, 0.0, 0.0), h=None):
    x = torch.arange(n, dtype=torch.float64, device=dev) * (1.0 / n if h is None else h)
    return (x + origin[0])[None, None, :], (x + origin[1])[None, :, None], (x + origin[2])[:, None, None]


class _Brain:
    """A seeded brain as functions of position: white / grey fractions and white-matter sites for tumour origins."""

    def __init__(self, seed):
        r = np.random.default_rng([seed, 17])
        self.axes = np.array([0.40, 0.34, 0.30]) * r.uniform(0.95, 1.05)
        self.phase = r.uniform(0, 2 * np.pi, 3)
        self.amp = r.uniform(0.03, 0.06, 3)
        self.vent = r.uniform(0.18, 0.24)
        self.r = r

    def tissue(self, X, Y, Z):
        dx, dy, dz = (X - 0.5) / self.axes[0], (Y - 0.5) / self.axes[1], (Z - 0.5) / self.axes[2]
        rb = torch.sqrt(dx * dx + dy * dy + dz * dz)
        edge = 0.62 + self.amp[0] * torch.sin(5 * dx + self.phase[0]) + self.amp[1] * torch.sin(
            4 * dy + self.phase[1]) + self.amp[2] * torch.sin(6 * dz + self.phase[2])
        wm = 0.5 * (1.0 - torch.tanh((rb - edge) / 0.06))
        csf = (((dx.abs() - self.vent) / 0.12) ** 2 + (dy / 0.28) ** 2 + (dz / 0.14) ** 2) <= 1.0
        inside = (rb <= 1.0) & ~csf
        return torch.where(inside, wm, 0.0), torch.where(inside, 1.0 - wm, 0.0)

    def origin(self):
        """A white-matter position (away from the ventricles)."""
        u = self.r.normal(size=3)
        u[0] = math.copysign(max(abs(u[0]), 0.2), u[0])
        u /= np.linalg.norm(u)
        return [float(v) for v in 0.5 + self.axes * u * self.r.uniform(0.3, 0.45)]


def _bump(X, Y, Z, x0, sigma, pw, pg):
    r2 = (X - x0[0]) ** 2 + (Y - x0[1]) ** 2 + (Z - x0[2]) ** 2
    return torch.where(pw + pg > 0, torch.exp(-r2 / (2.0 * sigma * sigma)), 0.0)


def _dense_inputs(case, seed, count=1):
    """The anatomy, `count` tumours and parameter sets, in the case's Real, on the GPU."""
    dev, n, R = "cuda", 8 * case["bpd"], _tdt(case)
    brain = _Brain(seed)
    X, Y, Z = _grid(n, dev)
    pw, pg = (a.to(R).contiguous() for a in brain.tissue(X, Y, Z))
    r = np.random.default_rng([seed, 23])
    sets = []
    for _ in range(count):
        x0 = brain.origin()
        Dw, rho = math.exp(r.uniform(math.log(0.1), math.log(0.3))), math.exp(r.uniform(math.log(0.005), math.log(0.05)))
        sets.append({"x0": x0, "Dw": Dw, "rho": rho, "c0": _bump(X, Y, Z, x0, 2.0 / n, pw, pg).to(R).contiguous()})
    return pw, pg, sets


def _blocks(v):
    """A dense volume in block-pool order."""
    b = v.shape[0] // 8
    return v.reshape(b, 8, b, 8, b, 8).permute(0, 2, 4, 1, 3, 5).contiguous().reshape(-1)


def _pool(case, pw, pg):
    pool = BlockPool(case["bpd"] ** 3, case["real"])
    pool.set_uniform(case["bpd"])
    pool.upload_dense("p_w", pw.cpu().numpy())
    pool.upload_dense("p_g", pg.cpu().numpy())
    return pool


def _masks(n, brain_x0, seed, dev="cuda"):
    """Observed T1c / FLAIR masks: two noisy balls around a site, 2 % of the labels flipped, and a PET signal."""
    X, Y, Z = _grid(n, dev)
    r2 = (X - brain_x0[0] - 0.01) ** 2 + (Y - brain_x0[1] + 0.01) ** 2 + (Z - brain_x0[2]) ** 2
    g = torch.Generator(dev).manual_seed(seed)
    out = []
    for rad in (0.06, 0.11):
        flip = torch.rand(r2.shape, generator=g, device=dev) < 0.02
        out.append(((r2 < rad * rad) ^ flip).double())
    pet = torch.clamp(1.0 - torch.sqrt(r2) / 0.12, min=0.0) * (0.9 + 0.1 * torch.rand(r2.shape, generator=g, device=dev))
    return out[0], out[1], pet.double()


def _stage_rows(case, seed):
    """Parameter rows of a stage: Dw, rho, horizon in days, origin, likelihood parameters."""
    r = np.random.default_rng([seed, 31])
    brain = _Brain(seed)
    k = case["samples"]
    Dw = np.exp(r.uniform(np.log(0.1), np.log(0.3), k))
    rho = np.exp(r.uniform(np.log(0.005), np.log(0.05), k))
    tend = r.uniform(case["days"] / 6, case["days"], k)
    x0 = np.array([brain.origin() for _ in range(k)])
    lik = np.stack([r.uniform(0.015, 0.03, k), r.uniform(0.7, 1.0, k), r.uniform(0.5, 0.8, k), r.uniform(0.1, 0.4, k),
                    r.uniform(1.0, 3.0, k)], 1)
    return Dw, rho, tend, x0, lik


# ---------------------------------------------------------------- a two-level leaf set
def _ghost_positions():
    out = []
    for code in range(27):
        if code == 13:
            continue
        c = (code % 3 - 1, (code // 3) % 3 - 1, code // 9 - 1)
        s = [(-1 if v < 0 else 0) if v < 1 else 8 for v in c]
        e = [(0 if v < 0 else 8) if v < 1 else 9 for v in c]
        out += [(x, y, z) for z in range(s[2], e[2]) for y in range(s[1], e[1]) for x in range(s[0], e[0])]
    return np.array(out)


def _two_levels(base, fine):
    """Leaves of a base^3 grid whose blocks in the box `fine` are split once, and their ghost lists: copies from the same
    level, injection from the finer level, averages of the two nearest coarse points per odd direction."""
    coarse = {}
    leaves = []
    for z in range(base):
        for y in range(base):
            for x in range(base):
                if not (x < fine[0] and y < fine[1] and z < fine[2]):
                    coarse[x, y, z] = len(leaves)
                    leaves.append((0, (x, y, z)))
    table0 = -np.ones((base,) * 3, dtype=np.int64)
    for (x, y, z), i in coarse.items():
        table0[x, y, z] = i
    table1 = -np.ones((2 * base,) * 3, dtype=np.int64)
    for z in range(2 * fine[2]):
        for y in range(2 * fine[1]):
            for x in range(2 * fine[0]):
                table1[x, y, z] = len(leaves)
                leaves.append((1, (x, y, z)))
    pos = _ghost_positions()
    n0, n1 = 8 * base, 16 * base

    def cell(table, p):
        s = table[p[..., 0] >> 3, p[..., 1] >> 3, p[..., 2] >> 3]
        return np.where(s >= 0, s * 512 + (p[..., 0] & 7) + 8 * ((p[..., 1] & 7) + 8 * (p[..., 2] & 7)), -1)

    src, w0, w1, w2, counts = [], [], [], [], []
    for level, idx in leaves:
        g = np.array(idx) * 8 + pos
        if level == 0:
            p = g % n0
            own, other = cell(table0, p), cell(table1, 2 * p % n1)
            src.append(np.where(own >= 0, own, other)[:, None])
            w = [np.ones((len(pos), 1))] * 3
            keep = np.ones((len(pos), 1), dtype=bool)
        else:
            p = g % n1
            own = cell(table1, p)
            odd = p & 1
            cs, ws, ks = [], [], []
            for dz in range(2):
                for dy in range(2):
                    for dx in range(2):
                        d = np.array([dx, dy, dz])
                        q = ((p >> 1) + d) % n0
                        c = cell(table0, q)
                        c = np.where(c >= 0, c, cell(table1, 2 * q % n1))
                        first = dx + dy + dz == 0
                        cs.append(np.where(own >= 0, own, c))
                        ks.append(np.where(own >= 0, first, np.all(d <= odd, axis=1)))
                        ws.append(np.where((own >= 0)[:, None] | (odd == 0), 1.0, 0.5))
            src.append(np.stack(cs, 1))
            keep = np.stack(ks, 1)
            w = [np.stack([v[:, d] for v in ws], 1) for d in range(3)]
        counts.append(keep.sum(1))
        src[-1] = src[-1][keep]
        for a, v in zip((w0, w1, w2), w):
            a.append(np.broadcast_to(v, keep.shape)[keep])
    row_ptr = np.concatenate([[0], np.cumsum(np.concatenate(counts))])
    csr = {"row_ptr": row_ptr.astype(np.int64), "src": np.concatenate(src).astype(np.int64), "w0": np.concatenate(w0),
           "w1": np.concatenate(w1), "w2": np.concatenate(w2)}
    blocks = [(i, level, idx, 1.0 / (n1 if level else n0)) for i, (level, idx) in enumerate(leaves)]
    return blocks, csr


def _adaptive_inputs(case, seed):
    base, fine = case["base"], [int(v) for v in case["fine"].split("x")]
    blocks, csr = _two_levels(base, fine)
    dev, brain, R = "cuda", _Brain(seed), _tdt(case)
    h = torch.tensor([b[3] for b in blocks], dtype=torch.float64, device=dev)
    o = torch.tensor([b[2] for b in blocks], dtype=torch.float64, device=dev) * (8 * h)[:, None]
    k = torch.arange(8, dtype=torch.float64, device=dev)
    X = (o[:, 0, None] + k * h[:, None])[:, None, None, :]
    Y = (o[:, 1, None] + k * h[:, None])[:, None, :, None]
    Z = (o[:, 2, None] + k * h[:, None])[:, :, None, None]
    pw, pg = (a.to(R).reshape(-1).contiguous() for a in brain.tissue(X, Y, Z))
    # a grown tumour across the refined box's corner
    x0 = [f / base for f in fine]
    c0 = (0.9 * _bump(X, Y, Z, [0.5 * (0.5 + v) for v in x0], 0.08, pw.reshape(X.shape[0], 8, 8, 8).double(),
                      pg.reshape(X.shape[0], 8, 8, 8).double())).to(R).reshape(-1).contiguous()
    coef = _coefficients(_real(case), 0.2, 0.05, 16 * base)
    return blocks, csr, pw, pg, c0, coef


# ---------------------------------------------------------------- the calls
def prepare(case, seed):
    kind, n = case["kind"], 8 * case.get("bpd", 0)
    s = {"case": case}
    if kind == "embed":
        pw, pg, sets = _dense_inputs(case, seed)
        s.update(pw=_blocks(pw), pg=_blocks(pg), phi=_blocks(sets[0]["c0"]),
                 coef=_coefficients(_real(case), sets[0]["Dw"], sets[0]["rho"], n), lib=_lib.load())
    elif kind == "solve":
        pw, pg, sets = _dense_inputs(case, seed, case["sets"])
        s["pool"] = _pool(case, pw, pg)
        s["sets"] = [(q["c0"].cpu().numpy(), _coefficients(_real(case), q["Dw"], q["rho"], n)) for q in sets]
    elif kind == "adaptive":
        blocks, csr, pw, pg, c0, s["coef"] = _adaptive_inputs(case, seed)
        pool = BlockPool(len(blocks), case["real"])
        pool.set_topology(blocks, csr)
        pool.upload("p_w", pw.cpu().numpy())
        pool.upload("p_g", pg.cpu().numpy())
        s.update(pool=pool, c0=c0.cpu().numpy())
    elif kind == "stage":
        pw, pg, _ = _dense_inputs(case, seed, 0)
        rows = _stage_rows(case, seed)
        t1, fl, pet = (a.cpu().numpy() for a in _masks(n, rows[3][0], seed))
        if case["fields"]:
            b = Batch(case["bpd"], case["samples"], case["real"])
            b.set_anatomy(0, pw.cpu().numpy(), pg.cpu().numpy())
            b.set_observations(t1, fl, pet)
            stage = [StageSample(float(d), float(r), float(t), tuple(x)) for d, r, t, x in zip(*rows[:4])]
            s.update(batch=b, samples=to_gbfk_samples(stage, case["bpd"], case["real"], L_CM)[0], lik=rows[4])
        else:
            Dw, rho, tend, x0, lik = rows
            s["model"] = GliomaModel(pw.cpu().numpy(), pg.cpu().numpy(), t1, fl, pet, L_cm=L_CM, precision=case["real"],
                                     max_samples=case["samples"])
            s["theta"] = np.log(np.column_stack([Dw, rho, tend * tend * rho, x0, np.sqrt(lik[:, 0]), lik[:, 1:]]))
    elif kind == "gradient":
        pw, pg, sets = _dense_inputs(case, seed)
        s["pool"] = _pool(case, pw, pg)
        t1, fl, _ = (a.cpu().numpy() for a in _masks(n, sets[0]["x0"], seed))
        s["pool"].set_observations(t1, fl)
        s["dt"] = _coefficients(_real(case), 0.3, sets[0]["rho"], n)[3]
        for key in ("Dw", "rho"):
            s[key] = torch.tensor(sets[0][key], dtype=torch.float64, requires_grad=True)
        if case["wrt"] == "c0":
            s["c0"] = sets[0]["c0"].cpu().requires_grad_()
        else:
            s["x0"] = torch.tensor(sets[0]["x0"], dtype=torch.float64, requires_grad=True)
    elif kind == "likelihood":
        pw, pg, sets = _dense_inputs(case, seed)
        s["pool"] = _pool(case, pw, pg)
        X, Y, Z = _grid(n, "cuda")
        u = 0.95 * _bump(X, Y, Z, sets[0]["x0"], 0.05, pw, pg)
        s["pool"].upload_dense("phi", u.to(_tdt(case)).cpu().numpy())
        t1, fl, pet = (a.cpu().numpy() for a in _masks(n, sets[0]["x0"], seed))
        s["pool"].set_observations(t1, fl, pet if case["pet"] else None)
    else:
        pw, pg, sets = _dense_inputs(case, seed, case["states"])
        s["pool"] = _pool(case, pw, pg)
        s["coef"] = _coefficients(_real(case), sets[0]["Dw"], sets[0]["rho"], n)
        s["ins"] = [q["c0"].cpu().pin_memory().numpy() for q in sets]
        s["outs"] = [torch.empty((n, n, n), dtype=_tdt(case)).pin_memory().numpy() for _ in sets]
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "embed":
        out = torch.empty_like(s["phi"])
        at = ctypes.c_void_p
        rc = s["lib"].gbfk_rd_step_static(_lib.GBFK_F64 if case["real"] == "f64" else _lib.GBFK_F32, case["bpd"],
                                          at(s["pw"].data_ptr()), at(s["pg"].data_ptr()), at(s["phi"].data_ptr()),
                                          at(out.data_ptr()), *s["coef"],
                                          at(torch.cuda.current_stream().cuda_stream), torch.cuda.current_device())
        if rc:
            raise RuntimeError("gbfk_rd_step_static returned %d" % rc)
        return out
    if kind == "solve":
        outs = []
        for c0, coef in s["sets"]:
            s["pool"].upload_dense("phi", c0)
            s["pool"].rd_step(*coef, case["steps"], check_nan=True)
            outs.append(s["pool"].download_dense("phi"))
        return outs
    if kind == "adaptive":
        pool = s["pool"]
        pool.upload("phi", s["c0"])
        pool.rd_step(*s["coef"], case["steps"])
        return pool.fwt_details(), pool.download("phi", s["c0"].size)
    if kind == "stage":
        if not case["fields"]:
            return s["model"](s["theta"])
        b = s["batch"]
        b.set_samples(s["samples"])
        b.run()
        lik = b.log_likelihood(*(s["lik"][:, j] for j in range(5)))
        return lik, [b.download(i) for i in range(case["samples"])]
    if kind == "gradient":
        c0, x0 = s.get("c0"), s.get("x0")
        leaves = [s["Dw"], s["rho"], c0 if x0 is None else x0]
        for v in leaves:
            v.grad = None
        loss = tumor_loss(s["pool"], s["Dw"], s["rho"], x0, L_CM, s["dt"], case["steps"], 2.0 / (8 * case["bpd"]),
                          case["checkpoints"], c0)
        loss.backward()
        return [loss.detach()] + [v.grad for v in leaves]
    if kind == "likelihood":
        return s["pool"].log_likelihood(**UC)
    for a, b in zip(s["ins"], s["outs"]):
        s["pool"].rd_step_host(a, b, *s["coef"], case["steps"])
    s["pool"].sync()
    return s["outs"]


# ---------------------------------------------------------------- bytes and operations a pass needs
def _stage_steps(case, seed):
    """Steps of each row of a stage, counted as the solver's time loop counts them."""
    R, n = _real(case), 8 * case["bpd"]
    Dw, rho, tend, x0, lik = _stage_rows(case, seed)
    out = []
    for i in range(case["samples"]):
        dt = R(_coefficients(R, Dw[i], rho[i], n)[3])
        # GliomaModel takes the horizon through log and exp
        T = R(tend[i] if case["fields"] else math.sqrt(math.exp(math.log(tend[i] * tend[i] * rho[i])) / math.exp(math.log(rho[i]))))
        t, k = R(0), 0
        while t <= T:
            k += 1
            t = R(t + dt)
        out.append(k)
    return out


BRAIN = 0.172  # share of the domain's cells that hold tissue


def work(case):
    """One step of a solve reads and writes the state where there is tissue, and each input field once; 33 operations a cell
    (six fluxes, the reaction, the update).  Inputs and results that live on the host cross once."""
    kind = case["kind"]
    w = 8 if case["real"] == "f64" else 4
    if kind == "adaptive":
        f = [int(v) for v in case["fine"].split("x")]
        cells = 512 * (case["base"] ** 3 + 7 * f[0] * f[1] * f[2])
        return {"bytes": cells * w * (2 * case["steps"] + 4), "flops": 33 * cells * case["steps"]}
    cells = (8 * case["bpd"]) ** 3
    if kind == "embed":
        return {"bytes": 4 * cells * w, "flops": 45 * BRAIN * cells}
    if kind == "likelihood":
        return {"bytes": cells * (w + 2 + (8 if case["pet"] else 0)), "flops": 60 * cells}
    tissue = BRAIN * cells
    if kind == "solve":
        return {"bytes": case["sets"] * w * (2 * cells + 2 * tissue * case["steps"]), "flops": 33 * tissue * case["steps"] * case["sets"]}
    if kind == "stream":
        return {"bytes": case["states"] * w * (2 * cells + 2 * tissue * case["steps"]), "flops": 33 * tissue * case["steps"] * case["states"]}
    if kind == "stage":
        steps = sum(_stage_steps(case, 1))
        return {"bytes": w * tissue * (2 * steps + case["samples"]), "flops": 33 * tissue * steps + 60 * cells * case["samples"]}
    # gradient: the forward steps once, and the adjoint steps (state in, adjoint in and out)
    return {"bytes": w * tissue * case["steps"] * 5, "flops": 110 * tissue * case["steps"]}


# ---------------------------------------------------------------- the same in 64 bits, in plain torch
_SHIFT = ((2, 1), (2, -1), (1, 1), (1, -1), (0, 1), (0, -1))  # roll(axis, by) brings neighbour x-, x+, y-, y+, z-, z+


def _roll(a, k):
    return torch.roll(a, _SHIFT[k][1], _SHIFT[k][0])


def _faces(pw, pg, Dw, Dg):
    df = pw * Dw + pg * Dg
    out = []
    for k in range(6):
        o = _roll(df, k)
        s = df + o
        out.append(torch.where(s < 1e-8, 0.0, 2.0 * df * o / torch.where(s < 1e-8, 1.0, s)))
    return out


def _step64(phi, t, H, rho, ih2, dt, keep=None):
    low = (phi + t) < 0.1
    flux, sdf = torch.zeros_like(phi), torch.zeros_like(phi)
    eff = []
    for k in range(6):
        d = torch.where(_roll(low, k ^ 1), 2.0 * H[k], H[k])  # the opposite neighbour below 0.1 doubles this face
        flux += d * _roll(phi, k)
        sdf += d
        if keep is not None:
            eff.append(d)
    flux = ih2 * (flux - sdf * phi)
    dom = (t + phi) > 0
    pre = torch.where(dom, phi + dt * (flux + rho * phi * (1.0 - phi)), phi)
    if keep is not None:
        keep.update(eff=eff, sdf=sdf, flux=flux, dom=dom, pre=pre)
    return pre.clamp(0.0, 1.0)


def _solve64(pw, pg, c0, coef, steps):
    pw, pg, phi = pw.double(), pg.double(), c0.double()
    Dw, Dg, rho, dt = coef
    ih2 = float(phi.shape[0]) ** 2
    H, t = _faces(pw, pg, Dw, Dg), pw + pg
    for _ in range(steps):
        phi = _step64(phi, t, H, rho, ih2, dt)
    return phi


def _likelihood64(u, t1, fl, pet, p):
    s2, scale, t1uc, t2uc, slope = p
    out = [0.0, 0.0, 0.0]
    if pet is not None:
        on = pet > 0
        r = (u - scale * pet)[on]
        out[0] = float(-0.5 * on.sum() * math.log(2 * math.pi * s2) - 0.5 / s2 * (r * r).sum())
    for j, (m, uc) in enumerate(((t1, t1uc), (fl, t2uc))):
        d = u - uc
        t = torch.where(d > 0, torch.ones_like(d), d * d) / slope
        near = torch.log1p(-0.5 * torch.exp(-t))
        far = math.log(0.5) - t
        la, lb = torch.where(d > 0, near, far), torch.where(d > 0, far, near)
        half = torch.full_like(d, math.log(0.5))
        la, lb = torch.where(d == 0, half, la), torch.where(d == 0, half, lb)
        out[1 + j] = float(torch.where(m > 0, la, lb).sum())
    return out + [sum(out)]


def _gradient64(case, seed):
    n, R = 8 * case["bpd"], _real(case)
    pw, pg, sets = _dense_inputs(case, seed)
    t1, fl, _ = _masks(n, sets[0]["x0"], seed)
    Dw, Dg, rho, _ = _coefficients(R, sets[0]["Dw"], sets[0]["rho"], n)
    dt = _coefficients(R, 0.3, sets[0]["rho"], n)[3]
    sigma, x0, ih2 = 2.0 / n, sets[0]["x0"], float(n) ** 2
    X, Y, Z = _grid(n, "cuda")
    c0 = sets[0]["c0"].double()
    pw, pg = pw.double(), pg.double()
    H, t = _faces(pw, pg, Dw, Dg), pw + pg
    states = [c0]
    for _ in range(case["steps"]):
        states.append(_step64(states[-1], t, H, rho, ih2, dt))
    u = states.pop()
    lik = _likelihood64(u, t1, fl, None, (1.0, 1.0, UC["t1_uc"], UC["t2_uc"], UC["slope"]))
    lam = torch.zeros_like(u)
    for m, uc in ((t1, UC["t1_uc"]), (fl, UC["t2_uc"])):
        d = u - uc
        e = torch.exp(-d * d / UC["slope"])
        g = torch.where(m > 0, -2.0 * d, e * d / (1.0 - 0.5 * e)) / UC["slope"]
        lam -= torch.where(d < 0, g, 0.0)
    gDw = grho = 0.0
    while states:
        phi, k = states.pop(), {}
        _step64(phi, t, H, rho, ih2, dt, k)
        mu = torch.where((k["pre"] > 0) & (k["pre"] <= 1), lam, 0.0)
        m = torch.where(k["dom"], mu, 0.0)
        grho = grho + (m * phi * (1.0 - phi)).sum() * dt
        gDw = gDw + (m * k["flux"]).sum() * dt / Dw
        acc = m * (-ih2 * k["sdf"] + rho * (1.0 - 2.0 * phi))
        for j in range(6):
            acc += _roll(ih2 * m * k["eff"][j], j ^ 1)
        lam = mu + dt * acc
    L = np.float64(R(L_CM) * R(L_CM))
    out = [torch.tensor(-(lik[1] + lik[2]), dtype=torch.float64), (gDw / L).cpu(), grho.cpu()]
    if case["wrt"] == "c0":
        return out + [lam.cpu()]
    w = lam * c0 / (sigma * sigma)
    return out + [torch.stack([(w * (X - x0[0])).sum(), (w * (Y - x0[1])).sum(), (w * (Z - x0[2])).sum()]).cpu()]


def _adaptive64(case, seed):
    blocks, csr, pw, pg, c0, (Dw, Dg, rho, dt) = _adaptive_inputs(case, seed)
    dev, nb = "cuda", len(blocks)
    R = _real(case)
    rows = torch.from_numpy(np.repeat(np.arange(nb * 488), np.diff(csr["row_ptr"]))).to(dev)
    src = torch.from_numpy(csr["src"]).to(dev)
    w = torch.from_numpy(csr["w0"] * csr["w1"] * csr["w2"]).to(dev)
    pos = _ghost_positions() + 1
    at = torch.from_numpy(pos[:, 0] + 10 * (pos[:, 1] + 10 * pos[:, 2])).to(dev)
    ih2 = torch.tensor([1.0 / np.float64(R(b[3])) ** 2 for b in blocks], dtype=torch.float64, device=dev).reshape(-1, 1, 1, 1)

    def lab(f):
        out = torch.zeros(nb, 1000, dtype=torch.float64, device=dev)
        out[:, at] = torch.zeros(nb * 488, dtype=torch.float64, device=dev).index_add_(0, rows, f[src] * w).reshape(nb, 488)
        out = out.reshape(nb, 10, 10, 10)
        out[:, 1:9, 1:9, 1:9] = f.reshape(nb, 8, 8, 8)
        return out

    def nbr(a, k):
        ax, by = _SHIFT[k]
        i = [slice(None)] + [slice(1, 9)] * 3
        i[ax + 1] = slice(1 - by, 9 - by)
        return a[tuple(i)]

    lw, lg = lab(pw.double()), lab(pg.double())
    ldf, lt = lw * Dw + lg * Dg, lw + lg
    mid = (slice(None),) + (slice(1, 9),) * 3
    H = []
    for k in range(6):
        a, b = ldf[mid], nbr(ldf, k)
        H.append(torch.where(a + b < 1e-8, 0.0, 2 * a * b / torch.where(a + b < 1e-8, 1.0, a + b)))
    phi = c0.double()
    for _ in range(case["steps"]):
        l = lab(phi)
        low, own = (l + lt) < 0.1, l[mid]
        flux, sdf = torch.zeros_like(own), torch.zeros_like(own)
        for k in range(6):
            d = torch.where(nbr(low, k ^ 1), 2 * H[k], H[k])
            flux += d * nbr(l, k)
            sdf += d
        new = own + dt * (ih2 * (flux - sdf * own) + rho * own * (1 - own))
        phi = torch.where(lt[mid] + own > 0, new, own).clamp(0.0, 1.0).reshape(-1)
    l = lab(phi)[:, 1:, 1:, 1:]
    best = torch.zeros(nb, dtype=torch.float64, device=dev)
    for code in range(1, 8):
        d = l
        for ax in range(3):
            even = d.narrow(ax + 1, 0, 8).unflatten(ax + 1, (4, 2)).select(ax + 2, 0)
            if code >> (2 - ax) & 1:
                odd = d.narrow(ax + 1, 0, 8).unflatten(ax + 1, (4, 2)).select(ax + 2, 1)
                nxt = d.narrow(ax + 1, 1, 8).unflatten(ax + 1, (4, 2)).select(ax + 2, 1)
                d = odd - 0.5 * (even + nxt)
            else:
                d = even
        best = torch.maximum(best, d.reshape(nb, -1).abs().max(1).values)
    return best.cpu().numpy(), phi.cpu().numpy()


def exact(case, seed):
    kind, n = case["kind"], 8 * case.get("bpd", 0)
    if kind == "adaptive":
        return _adaptive64(case, seed)
    if kind == "gradient":
        if case["steps"] * 8 * n ** 3 > 60e9:
            return None  # the states do not fit beside each other
        return _gradient64(case, seed)
    if kind == "embed":
        pw, pg, sets = _dense_inputs(case, seed)
        coef = _coefficients(_real(case), sets[0]["Dw"], sets[0]["rho"], n)
        return _blocks(_solve64(pw, pg, sets[0]["c0"], coef, 1))
    if kind == "solve":
        pw, pg, sets = _dense_inputs(case, seed, case["sets"])
        return [_solve64(pw, pg, q["c0"], _coefficients(_real(case), q["Dw"], q["rho"], n), case["steps"]).cpu().numpy()
                for q in sets]
    if kind == "stream":
        pw, pg, sets = _dense_inputs(case, seed, case["states"])
        coef = _coefficients(_real(case), sets[0]["Dw"], sets[0]["rho"], n)
        return [_solve64(pw, pg, q["c0"], coef, case["steps"]).cpu().numpy() for q in sets]
    if kind == "likelihood":
        pw, pg, sets = _dense_inputs(case, seed)
        X, Y, Z = _grid(n, "cuda")
        u = (0.95 * _bump(X, Y, Z, sets[0]["x0"], 0.05, pw, pg)).to(_tdt(case)).double()
        t1, fl, pet = _masks(n, sets[0]["x0"], seed)
        return np.array(_likelihood64(u, t1, fl, pet if case["pet"] else None,
                                      (0.000361, 0.85, UC["t1_uc"], UC["t2_uc"], UC["slope"])))
    pw, pg, _ = _dense_inputs(case, seed, 0)
    Dw, rho, tend, x0, lik = _stage_rows(case, seed)
    steps = _stage_steps(case, seed)
    if sum(steps) * max(1.0, n ** 3 / 1e6) > 50000:
        return None  # too long in plain torch
    t1, fl, pet = _masks(n, x0[0], seed)
    X, Y, Z = _grid(n, "cuda")
    out, fields = [], []
    for i in range(case["samples"]):
        v = x0[i] if case["fields"] else np.exp(np.log(x0[i]))
        c0 = _bump(X, Y, Z, v, 2.0 / n, pw, pg).to(_tdt(case))
        u = _solve64(pw, pg, c0, _coefficients(_real(case), Dw[i], rho[i], n), steps[i])
        p = list(lik[i])
        if not case["fields"]:
            p = [math.exp(math.log(math.sqrt(p[0]))) ** 2] + p[1:]
        out.append(_likelihood64(u, t1, fl, pet, p))
        fields.append(u.cpu().numpy())
    out = np.array(out)
    return (out, fields) if case["fields"] else out[:, 3]
