"""Timed cases of the update-and-measure path, driven through the package's public entry points.

Each case is one piece of work that a program using the library asks for again and again: sweeps of one lattice with a
measurement after each, a batch of replicas advanced together, a stream of requests served, a stored configuration
analysed.  Couplings are the repository's workloads' (J_xy = 1.2, J_z(z) uniform in [0.5, 1.5]) at temperatures in
[1.1, 1.5], from the state that a run has after its first sweeps from the cold start.
"""
import importlib.util
import math
import os
import random
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
J_XY = 1.2
ONE_BIN = 1 << 30  # measurements per bin: every pass of a case adds to the first bin row


def _package():
    """The package directory `slsf-rs_b200/` as module `slsf_rs_b200`."""
    if "slsf_rs_b200" not in sys.modules:
        d = os.path.join(ROOT, "slsf-rs_b200")
        spec = importlib.util.spec_from_file_location("slsf_rs_b200", os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["slsf_rs_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["slsf_rs_b200"]


_context = None


def _ctx():
    """One device context per process, as a program has."""
    global _context
    if _context is None:
        _context = _package().Context()
    return _context


# Lattices of one case: "L" (a cube), "LxMxN", or several separated by "+", repeated over the case's replicas.
def _shapes(text):
    out = []
    for part in text.split("+"):
        d = [int(v) for v in part.split("x")]
        out.append(tuple(d * 3) if len(d) == 1 else tuple(d))
    return out


def _dims(case):
    shapes = _shapes(case["lattice"])
    return [shapes[i % len(shapes)] for i in range(case.get("replicas", 1))]


def listed():
    return [
        # The smallest call: one 8^3 lattice (the reference's smallest examples), one sweep and one measurement per
        # step from the host; launches and round trips count.
        {"name": "step_l8", "kind": "steps", "lattice": "8", "sweeps": 1, "snapshot": False},
        # One 64^3 lattice driven as carlo-mc drives the model, a sweep and a measurement per step, with a snapshot
        # of the angles at the end.
        {"name": "plain_l64", "kind": "steps", "lattice": "64", "sweeps": 8, "snapshot": True},
        # The same on a large lattice whose sides are no powers of two (finite-size scaling in L_z).
        {"name": "plain_100x90x70", "kind": "steps", "lattice": "100x90x70", "sweeps": 4, "snapshot": True},
        # The two updates called one by one (re-exported lower-level functions), 128^3, and a measurement at the end.
        {"name": "updates_l128", "kind": "updates", "lattice": "128", "sweeps": 4},
        # The large lattice with observables and C_z after every sweep, in one batched call.
        {"name": "large_l256_corr_z", "kind": "large", "lattice": "256", "sweeps": 4, "r_z": 128},
        # A whole small run of one task through the host layer: thermalization, bins, estimates.
        {"name": "model_l12", "kind": "model", "lattice": "12", "sweeps": 300},
        # The headline batch: L = 32 replicas of many disorder realisations, one session step.
        {"name": "session_l32", "kind": "session", "lattice": "32", "replicas": 1184, "sweeps": 20},
        # Production job files' small lattices, L = 8 to 24 and the odd multiples of two among them.
        {"name": "batch_small", "kind": "batch", "lattice": "8+10+12+16+18+20+24+16x16x32", "replicas": 1024,
         "sweeps": 50},
        # Replicas too large for one thread block.
        {"name": "batch_l64", "kind": "batch", "lattice": "64", "replicas": 32, "sweeps": 8},
        # A stream of requests of all sizes through the server.
        {"name": "served_mixed", "kind": "served", "lattice": "8+16+24+32+48+64+36x40x44+20x20x60", "replicas": 192,
         "sweeps": 120},
        # A job that measures all correlation functions after every sweep.
        {"name": "fused_corr_l16", "kind": "fused", "lattice": "16+8", "replicas": 64, "sweeps": 50, "r_xy": 8, "r_z": 8},
        # A stored configuration analysed: observables and all correlation functions to half the side.
        {"name": "analysis_l96", "kind": "analysis", "lattice": "96", "r_xy": 48, "r_z": 48},
    ]


def _even(rng, lo, hi):
    """An even side, spread over its logarithm."""
    return max(lo, min(hi, 2 * int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 2))))


def draw(rng: random.Random):
    kind = rng.choice(["steps", "steps", "updates", "large", "model", "session", "batch", "batch", "served", "fused",
                       "analysis"])
    if kind in ("steps", "updates"):
        d = [_even(rng, 4, 160) for _ in range(3)]
        case = {"kind": kind, "lattice": "%dx%dx%d" % tuple(d), "sweeps": rng.randint(1, 8)}
        if kind == "steps":
            case["snapshot"] = rng.random() < 0.5
        return case
    if kind == "large":
        d = [_even(rng, 66, 256) for _ in range(3)]
        if rng.random() < 0.5:  # sides that are multiples of 32 are common for large lattices
            d = [32 * rng.randint(3, 8) for _ in range(3)]
        return {"kind": kind, "lattice": "%dx%dx%d" % tuple(d), "sweeps": rng.randint(2, 4), "r_z": d[2] // 2}
    if kind == "model":
        return {"kind": kind, "lattice": str(_even(rng, 4, 48)), "sweeps": rng.randint(60, 300)}
    if kind == "analysis":
        d = [_even(rng, 4, 128) for _ in range(3)]
        return {"kind": kind, "lattice": "%dx%dx%d" % tuple(d), "r_xy": min(d[0], d[1]) // 2, "r_z": d[2] // 2}
    if kind == "fused":
        d = (_even(rng, 4, 32), _even(rng, 4, 32), _even(rng, 4, 32))
        return {"kind": kind, "lattice": "%dx%dx%d" % d, "replicas": rng.randint(1, 64), "sweeps": rng.randint(5, 40),
                "r_xy": min(d[0], d[1]) // 2, "r_z": d[2] // 2}
    # batches: one to three shapes, as many replicas and sweeps as stay under the listed batches' work
    shapes = []
    for _ in range(rng.randint(1, 3)):
        side = _even(rng, 4, 64)
        shapes.append("%dx%dx%d" % (side, side, _even(rng, 4, 64)) if rng.random() < 0.5 else str(side))
    text = "+".join(shapes)
    volume = max(a * b * c for a, b, c in _shapes(text))
    sweeps = rng.randint(4, 60)
    most = max(1, min(512, int(6e7 / (volume * sweeps))))
    replicas = max(1, int(round(math.exp(rng.uniform(0, math.log(most))))))
    if kind == "session":
        text = shapes[0]
    return {"kind": kind, "lattice": text, "replicas": replicas, "sweeps": sweeps}


class _State:
    """A case's handles; closes the session before its tasks."""

    def __init__(self, case):
        self.case = case
        self.tasks, self.handles, self.session, self.server = [], None, None, None

    def __del__(self):
        for h in [self.session, self.server, *self.tasks]:
            if h is not None:
                h.close()


def _disorder(rng, lz):
    return rng.uniform(0.5, 1.5, lz)


def prepare(case, seed):
    slsf, ctx, kind = _package(), _ctx(), case["kind"]
    rng = np.random.default_rng([20260710, seed])
    s = _State(case)
    if kind == "model":
        d = _shapes(case["lattice"])[0]
        s.desc = slsf.theta_task(d, float(rng.uniform(1.1, 1.5)), sweeps=case["sweeps"], thermalization=20, binsize=10,
                                 seed=int(rng.integers(1 << 40)), j_xy_array=np.full(d[2], J_XY),
                                 j_z_array=_disorder(rng, d[2]))
        return s
    if kind == "served":
        s.server = slsf.Server(ctx, epoch_sweeps=100, keep_bins=False)
        s.requests = [dict(tag=i, dims=d, temperature=float(rng.uniform(1.0, 1.6)), seed=int(rng.integers(1 << 40)),
                           j_xy=np.full(d[2], J_XY), j_z=_disorder(rng, d[2]),
                           sweeps=int(rng.integers(case["sweeps"] // 4, case["sweeps"] + 1)) + 8, thermalization=8,
                           n_bins=4) for i, d in enumerate(_dims(case))]
        return s
    if kind == "analysis":
        d = _shapes(case["lattice"])[0]
        s.theta, j_z = _configuration(d, seed)
        s.tasks = [slsf.Task(ctx, d, np.full(d[2], J_XY), j_z, 1.3)]
        return s
    bins = 0 if kind in ("steps", "updates") else 1 if kind == "large" else 8
    for d in _dims(case):
        t = slsf.Task(ctx, d, np.full(d[2], J_XY), _disorder(rng, d[2]), float(rng.uniform(1.1, 1.5)), wolff_steps=1,
                      seed=int(rng.integers(1 << 40)), thermalization=0, binsize=ONE_BIN, n_bins=bins)
        t.init_cold()
        s.tasks.append(t)
    if kind in ("steps", "updates"):
        s.tasks[0].sweep(10)
        return s
    s.handles = ctx.handle_array(s.tasks)
    ctx.batch_run(s.tasks, 10, handles=s.handles)
    if kind in ("large", "fused"):
        for t in s.tasks:
            t.corr_setup(case.get("r_xy", 0), case["r_z"], ONE_BIN, 1)
            t.corr_fuse(1)
    if kind in ("session", "fused"):
        s.session = ctx.session(s.tasks, case["sweeps"])
    return s


def _numbers(stats):
    """Step statistics as whole numbers [tasks, 4]."""
    return np.array([[v["sweeps"], v["accepted"], v["wolff_clusters"], v["wolff_cluster_sites"]] for v in stats],
                    dtype=np.int64)


def run(s):
    case, ctx = s.case, _ctx()
    kind = case["kind"]
    if kind == "steps":
        t = s.tasks[0]
        stats, obs = [], []
        for _ in range(case["sweeps"]):
            stats.append(t.sweep(1))
            obs.append(list(t.measure().values()))
        out = {"stats": _numbers(stats), "observables": np.array(obs)}
        if case["snapshot"]:
            out["theta"] = t.theta
        return out
    if kind == "updates":
        t = s.tasks[0]
        acceptance, sizes = [], []
        for _ in range(case["sweeps"]):
            acceptance.append(t.metropolis_sweep())
            sizes.append(t.wolff_step())
        return {"acceptance": np.array(acceptance), "cluster_sizes": np.array(sizes, dtype=np.int64),
                "observables": np.array(list(t.measure().values()))}
    if kind == "model":
        e = _package().model_run(ctx, s.desc, batched=True)
        return {k: (np.array(v) if isinstance(v, tuple) else v) for k, v in e.items()}
    if kind == "served":
        for r in s.requests:
            s.server.submit(**r)
        active, pending = s.server.step()
        while active or pending:
            active, pending = s.server.step()
        done = sorted(s.server.poll(), key=lambda r: r["tag"])
        return {"counts": np.array([[r["tag"], r["status"], r["sweeps"], r["accepted"], r["cluster_sites"]] for r in done],
                                   dtype=np.int64),
                "estimates": np.array([[v for key in sorted(r["est"]) for v in np.atleast_1d(r["est"][key])] for r in done],
                                      dtype=np.float64)}
    if kind == "analysis":
        t = s.tasks[0]
        t.theta = s.theta
        out = t.measure()
        out.update(t.correlations(case["r_xy"], case["r_z"]))
        return out
    if s.session is not None:
        stats = s.session.step()
    else:
        stats = ctx.batch_run(s.tasks, case["sweeps"], handles=s.handles)
    bins, measured = ctx.batch_bins(s.tasks, s.tasks[0].n_bins, handles=s.handles)
    out = {"stats": _numbers(stats), "bins": bins, "measured": measured.astype(np.int64)}
    if kind in ("large", "fused"):
        corr = [t.corr_bins(1) for t in s.tasks]
        out["correlations"] = np.concatenate([c[0].ravel() for c in corr])
        out["correlation_measurements"] = np.array([c[1] for c in corr], dtype=np.int64)
    return out


# Operations that one site-update cannot do without: a Metropolis proposal (two trig pairs, the local field of six
# neighbours, the energy difference, one exponential, two uniforms), its share of a Wolff step (three bond tests with
# a uniform and an exponential each, one reflection) and of the measurement (three bonds, cosine and sine).
FLOPS_SITE = 60.0


def work(case):
    kind = case["kind"]
    if kind == "analysis":
        lx, ly, lz = _shapes(case["lattice"])[0]
        v = lx * ly * lz
        values = 8 + (3 + lz) * case["r_xy"] + case["r_z"]
        # three transforms of length n cost 5 n log2 n per line of n sites
        flops = v * (20 + 5 * (math.log2(lx) + math.log2(ly) + math.log2(lz)))
        return {"bytes": 4.0 * v + 8.0 * values, "flops": flops}
    if kind == "model":
        lx, ly, lz = _shapes(case["lattice"])[0]
        v, sweeps = lx * ly * lz, case["sweeps"] + 20
        return {"bytes": 8.0 * v, "flops": FLOPS_SITE * v * sweeps}
    sites = float(sum(a * b * c for a, b, c in _dims(case)))
    flops = FLOPS_SITE * sites * case["sweeps"] * (0.625 if kind == "served" else 1.0)
    tasks = len(_dims(case))
    # the state is read once and written once per pass; bins and statistics come back
    nbytes = 8.0 * sites + 32.0 * tasks
    if kind == "steps" and case["snapshot"]:
        nbytes += 4.0 * sites
    if kind in ("session", "batch", "fused", "served"):
        nbytes += 8.0 * 12 * 8 * tasks
    return {"bytes": nbytes, "flops": flops}


def _configuration(d, seed):
    """An ordered-phase configuration (a uniform direction with smooth and local fluctuations) and its couplings."""
    rng = np.random.default_rng([20260711, seed])
    lx, ly, lz = d
    z, y, x = np.meshgrid(np.arange(lz), np.arange(ly), np.arange(lx), indexing="ij", sparse=True)
    a = rng.uniform(0, 2 * np.pi) + rng.normal(0, 0.5, (lz, ly, lx))
    for _ in range(4):
        k = rng.integers(-2, 3, 3)
        a = a + rng.normal(0, 0.4) * np.cos(2 * np.pi * (k[0] * x / lx + k[1] * y / ly + k[2] * z / lz)
                                            + rng.uniform(0, 2 * np.pi))
    theta = np.mod(a, 2 * np.pi).astype(np.float32).ravel()
    return theta, _disorder(rng, lz)


def exact(case, seed):
    """The analysis of a given configuration in 64 bits.  The other cases follow a Markov chain whose decisions are
    taken in 32 bits: no 64-bit value belongs to their outputs."""
    if case["kind"] != "analysis":
        return None
    d = _shapes(case["lattice"])[0]
    lx, ly, lz = d
    theta, j_z = _configuration(d, seed)
    s = np.exp(1j * theta.astype(np.float64)).reshape(lz, ly, lx)
    v = float(s.size)
    j = {2: J_XY, 1: J_XY, 0: j_z[:, None, None]}
    bond = {ax: j[ax] * s * np.conj(np.roll(s, -1, ax)) for ax in (2, 1, 0)}
    c = {ax: float(b.real.sum()) for ax, b in bond.items()}
    out = {"energy": -(c[2] + c[1] + c[0]) / v, "magnetization_squared": float(abs(s.sum()) ** 2) / v ** 2,
           "cos_x": c[2], "cos_y": c[1], "cos_z": c[0], "sin_x": float(bond[2].imag.sum()),
           "sin_y": float(bond[1].imag.sum()), "sin_z": float(bond[0].imag.sum())}

    def lags(ax, r):
        """sum over lines of s(k) . s(k + r), for r = 1..R, by layer z (ax 2, 1) or whole (ax 0)."""
        f = np.fft.ifft(np.abs(np.fft.fft(s, axis=ax)) ** 2, axis=ax).real
        f = np.moveaxis(f, ax, -1)[..., 1:r + 1]
        return f.sum(axis=1) if ax else f.sum(axis=(0, 1))

    gx, gy, gz = lags(2, case["r_xy"]), lags(1, case["r_xy"]), lags(0, case["r_z"])
    cx, cy = gx.sum(0) / v, gy.sum(0) / v
    out.update({"corr_x": cx, "corr_y": cy, "corr_xy": (cx + cy) / 2, "corr_xy_by_z": (gx + gy) / (2.0 * lx * ly),
                "corr_z": gz / v})
    return out
