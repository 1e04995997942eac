"""What a user of this framework has it do, as measurable cases: whole model
runs from host arrays (upload, steps, read-back) in the three precisions, the
ensemble forms, the tracer-advection benchmark and the emulator's
convolutions, each through the package's public entry points.

``exact`` restates every path in 64-bit torch without this package's code.
"""
import ctypes
import math

import numpy as np
import torch

import psyclonebench_gb300 as P
from psyclonebench_gb300 import emulator, ensemble, model, workloads

LIB = P.load_library()
_DP = ctypes.POINTER(ctypes.c_double)

FP64, MIXED, FP64_EQUIVALENT = 0, 1, 2

# ---- the cases ---------------------------------------------------------------


def listed():
    return [
        # The parity namelist: the reference's own 128 x 128 run from rest,
        # checksums every 100 steps.  Launch latency and a chip that one
        # small domain cannot fill.
        {"name": "step_parity_128", "kind": "step", "nx": 128, "ny": 128, "precision": FP64,
         "steps": 1000, "sums_every": 100, "start": "rest", "land": False, "driver": "run"},
        # An odd-sized regional model with an island and a ragged coast,
        # restarted from a state in motion.
        {"name": "step_fp64_601x413", "kind": "step", "nx": 601, "ny": 413, "precision": FP64,
         "steps": 200, "sums_every": 0, "start": "waves", "land": True, "driver": "run"},
        # The largest single domain, driven as the reference's Fortran driver
        # does: one c_invoke_time_step call per step from host arrays.
        {"name": "step_fp64_4096", "kind": "step", "nx": 4096, "ny": 4096, "precision": FP64,
         "steps": 20, "sums_every": 0, "start": "waves", "land": False, "driver": "calls"},
        # Mixed precision on bathymetry, the configuration the mixed form is
        # judged on, at a quarter of its cells.
        {"name": "step_mixed_2048", "kind": "step", "nx": 2048, "ny": 2048, "precision": MIXED,
         "steps": 1000, "sums_every": 0, "start": "waves", "land": False, "driver": "run"},
        # FP64-equivalent (double-float) steps of an odd-sized coastal model.
        {"name": "step_df_1501x1103", "kind": "step", "nx": 1501, "ny": 1103,
         "precision": FP64_EQUIVALENT, "steps": 300, "sums_every": 100, "start": "waves",
         "land": True, "driver": "run"},
        # What a hybrid roll-out's judge runs for a window: 8 equal domains,
        # a state handed over on the device, 500 FP64 steps, handed back.
        {"name": "ens_fp64_8x256", "kind": "ens", "count": 8, "lo": 256, "hi": 256,
         "precision": FP64, "runs": 1, "steps": 500, "handover": True},
        # Training data for the emulator: trajectories of many equal domains
        # in mixed precision, a snapshot every 10 steps.
        {"name": "ens_mixed_96x256", "kind": "ens", "count": 96, "lo": 256, "hi": 256,
         "precision": MIXED, "runs": 20, "steps": 10, "handover": False},
        # Uneven domains (64 to 1024 cells a side) in the FP64-equivalent
        # form, from rest, read back to the host.
        {"name": "ens_df_16x64to1024", "kind": "ens", "count": 16, "lo": 64, "hi": 1024,
         "precision": FP64_EQUIVALENT, "runs": 1, "steps": 200, "handover": False},
        # The tracer-advection benchmark at the largest size of the
        # reference's sweep, on its own kind of fields.
        {"name": "tra_512x512x75", "kind": "tra", "jpi": 512, "jpj": 512, "jpk": 75, "iters": 50,
         "masks": "benchmark"},
        # A small basin with land and currents of either sign.
        {"name": "tra_93x67x31", "kind": "tra", "jpi": 93, "jpj": 67, "jpk": 31, "iters": 100,
         "masks": "sea"},
        # The emulator's hidden layer at the training batch: forward with
        # bias and ReLU, and the weight gradient of its backward pass.
        {"name": "conv_48x48_16x256", "kind": "conv", "batch": 16, "h": 256, "w": 256, "cin": 48,
         "cout": 48, "relu": True, "out": "bf16"},
        {"name": "wgrad_48x48_16x256", "kind": "wgrad", "batch": 16, "h": 256, "w": 256,
         "cin": 48, "cout": 48},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "ens", "ens", "tra", "conv", "wgrad"])
    if kind == "step":
        precision = rng.choice([FP64, FP64, MIXED, FP64_EQUIVALENT])
        nx, ny = _log_int(rng, 64, 4096), _log_int(rng, 64, 4096)
        steps = max(10, min(500, int(20 * 4096 * 4096 / (nx * ny))))
        driver = rng.choice(["run", "run", "calls"])
        return {"kind": "step", "nx": nx, "ny": ny, "precision": precision, "steps": steps,
                "sums_every": rng.choice([0, steps // 5]) if driver == "run" else 0,
                "start": rng.choice(["rest", "waves", "waves"]), "land": rng.random() < 0.5,
                "driver": driver}
    if kind == "ens":
        precision = rng.choice([FP64, MIXED, FP64_EQUIVALENT])
        equal = rng.random() < 0.5
        n = _log_int(rng, 64, 512)
        count = max(2, min(64, 3000000 // (n * n))) if equal else rng.randint(2, 12)
        return {"kind": "ens", "count": count, "lo": n if equal else 64,
                "hi": n if equal else 1024, "precision": precision,
                "runs": rng.choice([1, 4]), "steps": rng.randint(10, 50),
                "handover": equal and rng.random() < 0.5}
    if kind == "tra":
        return {"kind": "tra", "jpi": _log_int(rng, 32, 512), "jpj": _log_int(rng, 32, 512),
                "jpk": rng.randint(5, 75), "iters": rng.randint(10, 50),
                "masks": rng.choice(["benchmark", "sea"])}
    shape = {"batch": rng.randint(1, 16), "h": _log_int(rng, 40, 256),
             "w": rng.choice([128, 256]), "cin": rng.choice([16, 32, 48]),
             "cout": rng.choice([16, 32, 48, 64])}
    if kind == "conv":
        return dict(shape, kind="conv", relu=rng.random() < 0.7, out=rng.choice(["bf16", "fp32"]))
    return dict(shape, kind="wgrad")


def work(case):
    kind = case["kind"]
    if kind in ("conv", "wgrad"):
        px, ci, co = case["batch"] * case["h"] * case["w"], case["cin"], case["cout"]
        flops = 2.0 * 9 * ci * co * px
        if kind == "wgrad":
            return {"bytes": px * 2.0 * (ci + co) + 4.0 * (9 * ci * co + co), "flops": flops}
        return {"bytes": px * (2.0 * ci + (2.0 if case["out"] == "bf16" else 4.0) * co) +
                18.0 * ci * co, "flops": flops}
    if kind == "tra":
        pts = case["jpi"] * case["jpj"] * case["jpk"]
        # per point and iteration: 8 fields read, 1 written; about 40 operations
        return {"bytes": 72.0 * pts * case["iters"], "flops": 40.0 * pts * case["iters"]}
    # per cell and step: (ssh, u, v) read and written, three depths, the mask;
    # 230 adds and multiplies and 17 divides
    per_cell = {FP64: 76.0, MIXED: 48.0, FP64_EQUIVALENT: 76.0}[case["precision"]]
    if kind == "step":
        cells, steps = case["nx"] * case["ny"], case["steps"]
    else:
        cells = sum(s["nx"] * s["ny"] for s in _specs(case, 0))
        steps = case["runs"] * case["steps"]
    return {"bytes": per_cell * cells * steps, "flops": 247.0 * cells * steps}


def prepare(case, seed):
    return {"step": _StepRun, "ens": _EnsRun, "tra": _TraRun, "conv": _Conv,
            "wgrad": _WeightGrad}[case["kind"]](case, seed)


def run(state):
    return state.run()


def exact(case, seed):
    return {"step": _exact_step, "ens": _exact_ens, "tra": _exact_tra, "conv": _exact_conv,
            "wgrad": _exact_wgrad}[case["kind"]](case, seed)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(g, n, lo, hi):
    return (lo + (hi - lo) * torch.rand(n, generator=g, device="cuda",
                                        dtype=torch.float64)).tolist()


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


# ---- one domain --------------------------------------------------------------

RDT_FLAT, RDT_BATHYMETRY = 20.0, 5.0  # s


def _waves(g, xs, ys, modes, lo, hi):
    """Sum of plane waves of random direction and phase, amplitudes summing
    to at most `hi` - `lo` about their middle; xs, ys in [0, 1]."""
    acc = torch.full((ys.numel(), xs.numel()), 0.5 * (lo + hi), dtype=torch.float64,
                     device="cuda")
    for k in range(modes):
        kx, ky, ph = _uniform(g, 3, 0.0, 1.0)
        a = xs * (2 * math.pi * (1 + 5 * kx)) + 2 * math.pi * ph
        b = ys * (2 * math.pi * (6 * ky - 3))
        acc += (0.5 * (hi - lo) / modes) * (
            torch.outer(torch.cos(b), torch.cos(a)) - torch.outer(torch.sin(b), torch.sin(a)))
    return acc


def _domain(case, seed):
    """Arrays of a domain as torch float64 / int32 on the GPU: T-mask, depths
    and the starting (ssh, u, v), with the extents and the time step."""
    g = _gen(seed)
    nx, ny = case["nx"], case["ny"]
    w, h = (nx + 3 + 7) // 8 * 8, ny + 3
    xe, ye = nx, ny  # internal T cells 1..nx x 1..ny
    m = torch.zeros((h, w), dtype=torch.int32, device="cuda")
    m[1:ye + 1, 1:xe + 1] = 1
    m[0, :] = -1  # the open south side, as the reference's set-up leaves it
    if case["land"]:
        # a ragged west coast of 1-4 cells and an island in the middle
        depth = torch.randint(1, 5, (h, 1), generator=g, device="cuda")
        coast = torch.arange(w, device="cuda")[None, :] <= depth
        rows = torch.arange(h, device="cuda")[:, None]
        m[coast & (rows >= 4) & (rows <= ye)] = 0
        m[ny // 2:ny // 2 + max(2, ny // 8), nx // 2:nx // 2 + max(2, nx // 10)] = 0
    x = torch.arange(w, dtype=torch.float64, device="cuda") / w
    y = torch.arange(h, dtype=torch.float64, device="cuda") / h
    rest = case["start"] == "rest"
    if rest and not case["land"]:
        (d,) = _uniform(g, 1, 90.0, 110.0)
        ht, hu, hv = (torch.full((h, w), d, dtype=torch.float64, device="cuda")
                      for _ in range(3))
    else:
        s = int(torch.randint(0, 2 ** 31, (1,), generator=g, device="cuda"))
        ht, hu, hv = (_waves(_gen(s), x + dx, y + dy, 8, 60.0, 480.0)
                      for dx, dy in ((0.0, 0.0), (0.5 / w, 0.0), (0.0, 0.5 / h)))
    z = torch.zeros((h, w), dtype=torch.float64, device="cuda")
    sn, un, vn = z.clone(), z.clone(), z.clone()
    if not rest:
        wet = m > 0
        wet_u, wet_v = wet & (_e(m) > 0), wet & (_n(m) > 0)
        sn = torch.where(wet, _waves(g, x, y, 6, -0.2, 0.2), z)
        un = torch.where(wet_u, _waves(g, x, y, 6, -0.1, 0.1), z)
        vn = torch.where(wet_v, _waves(g, x, y, 6, -0.1, 0.1), z)
    flat = rest and not case["land"]
    return {"m": m, "ht": ht, "hu": hu, "hv": hv, "sn": sn, "un": un, "vn": vn,
            "ext": (1, xe, 1, ye), "rdt": RDT_FLAT if flat else RDT_BATHYMETRY,
            "cbfr": 1.5e-4 if flat else 1e-3, "visc": 0.1 if flat else 100.0,
            "amp": 0.2, "period_h": 12.42}


class _StepRun:
    """A program that holds one model in (pinned) host arrays, runs it and
    reads the final state."""

    def __init__(self, case, seed):
        d = _domain(case, seed)
        h, w = d["m"].shape
        xs, xe, ys, ye = d["ext"]
        m = model.Model.from_extents(w, h, xs, xe, ys, ye)
        m.rdt, m.cbfr, m.visc = d["rdt"], d["cbfr"], d["visc"]
        self._held = []

        def array(value, dtype=torch.float64):
            t = _pinned((h, w), dtype)
            if isinstance(value, torch.Tensor):
                t.copy_(value)
            else:
                t.fill_(value)
            self._held.append(t)
            return t.numpy()

        su, sv = _face_ssh(d, d["sn"])
        state = {"sshn_t": d["sn"], "ssha_t": d["sn"], "un": d["un"], "ua": d["un"],
                 "vn": d["vn"], "va": d["vn"], "sshn_u": su, "sshn_v": sv}
        for k in model.FIELDS:
            m.f[k] = array(d[k] if k in ("ht", "hu", "hv") else state.get(k, 0.0))
        for k in model.GRID:
            m.grid[k] = (array(d["m"], torch.int32) if k == "tmask" else
                         array(50.0 if k.startswith("gphi") else
                               1.0e6 if k.startswith("area") else 1000.0))
        self.m, self.case = m, case
        self.out = {k: array(0.0) for k in ("sshn_t", "un", "vn")}
        n = case["steps"] // case["sums_every"] if case["sums_every"] else 0
        self.sums = np.zeros((n, 3))

    def run(self):
        m, c = self.m, self.case
        LIB.nl2d_set_precision(c["precision"])
        if c["driver"] == "calls":
            for k in range(c["steps"]):
                LIB.c_invoke_time_step(*m.step_args(1 + k))
        else:
            model.register(LIB, m)
            P.check(LIB.nl2d_run_steps(1, c["steps"], c["sums_every"],
                                       self.sums.ctypes.data_as(_DP)), "nl2d_run_steps")
        for k, a in self.out.items():
            LIB.c_read_from_device(m.f[k].ctypes.data, a.ctypes.data, 1, 1, m.width, m.height,
                                   True)
        P.check(None, "the run")
        if c["driver"] == "calls":
            LIB.nl2d_finalize()  # the program's end: the next pass is a new run
        return dict(self.out, sums=self.sums)


def _exact_step(case, seed):
    d = _domain(case, seed)
    s = _Solver([d])
    sums = []
    for k in range(case["steps"]):
        s.step(1 + k)
        if case["sums_every"] and (k + 1) % case["sums_every"] == 0:
            sums.append(s.sums(0))
    return {"sshn_t": s.sn[0], "un": s.un[0], "vn": s.vn[0],
            "sums": torch.stack(sums) if sums else None}


# ---- ensembles ---------------------------------------------------------------


def _specs(case, seed):
    if case["lo"] == case["hi"]:
        return emulator.emulator_domain_specs(case["count"], seed, case["lo"])
    # the sizes stand for the case, the seed for bathymetry, tides and sides
    sizes = workloads.ensemble_domains(case["count"], 7, case["lo"], case["hi"])
    specs = workloads.ensemble_domains(case["count"], seed, case["lo"], case["hi"])
    for s, z in zip(specs, sizes):
        s["nx"], s["ny"] = z["nx"], z["ny"]
    return specs


def _handover_state(case, seed):
    """Interior (ssh, u, v) of every domain, FP32 [domain][ny][nx][3]."""
    n, g = case["lo"], _gen(seed)
    x = torch.arange(n, dtype=torch.float64, device="cuda") / n
    st = torch.stack([torch.stack([_waves(g, x, x, 4, -a, a) for a in (0.1, 0.05, 0.05)], dim=2)
                      for _ in range(case["count"])])
    return st.float().contiguous()


class _EnsRun:
    """A program that builds an ensemble of domains, runs it (`runs` runs of
    `steps` steps) and takes the states: snapshots on the device for equal
    domains, host arrays otherwise."""

    def __init__(self, case, seed):
        self.case = case
        self.doms = [ensemble.build_domain(s) for s in _specs(case, seed)]
        self.equal = case["lo"] == case["hi"]
        self.start = _handover_state(case, seed) if case["handover"] else None
        if self.equal:
            n = case["lo"]
            self.buf = torch.zeros(case["count"], n, n, 3, device="cuda")
            torch.cuda.synchronize()

    def run(self):
        c = self.case
        e = ensemble.Ensemble(self.doms, lib=LIB)
        if c["precision"]:
            e.set_precision(c["precision"])
        e.run(1, 0)  # builds the schedule
        if self.start is not None:
            self._ck(LIB.nl2d_ens_import_interior(ctypes.c_void_p(self.start.data_ptr())))
        sums = None
        for r in range(c["runs"]):
            _, sums = e.run(1 + r * c["steps"], c["steps"], c["steps"])
            if self.equal:
                self._ck(LIB.nl2d_ens_export_interior(ctypes.c_void_p(self.buf.data_ptr())))
        if self.equal:
            out = {"state": self.buf}
        else:
            out = {"fields": [e.read(k) for k in range(c["count"])]}
        e.close()
        return dict(out, sums=sums)

    @staticmethod
    def _ck(rc):
        P.check(rc, "ensemble hand-over")


def _exact_ens(case, seed):
    doms = []
    for s in _specs(case, seed):
        b = ensemble.build_domain(s)  # the caller's own arrays: inputs, not results
        w, h, xs, xe, ys, ye = b["dims"]
        z = torch.zeros((h, w), dtype=torch.float64, device="cuda")
        doms.append({"m": torch.tensor(b["tmask"], device="cuda"),
                     **{k: torch.tensor(b[k], device="cuda") for k in ("ht", "hu", "hv")},
                     "sn": z, "un": z, "vn": z, "ext": (xs, xe, ys, ye), "rdt": 5.0,
                     "cbfr": 1e-3, "visc": 100.0, "amp": b["tide"][0], "period_h": b["tide"][1]})
    if case["handover"]:
        for d, st in zip(doms, _handover_state(case, seed).double()):
            _hand_over(d, st)
    groups = [doms] if case["lo"] == case["hi"] else [[d] for d in doms]
    fields, sums = [], []
    for g in groups:
        s = _Solver(g)
        for k in range(case["runs"] * case["steps"]):
            s.step(1 + k)
        fields += [(s.sn[q], s.un[q], s.vn[q]) for q in range(len(g))]
        sums += [s.sums(q) for q in range(len(g))]
    sums = torch.stack(sums)[None]
    if case["lo"] != case["hi"]:
        return {"fields": fields, "sums": sums}
    xs, xe, ys, ye = doms[0]["ext"]
    state = torch.stack([torch.stack([f[ys:ye + 1, xs:xe + 1] for f in t], dim=2)
                         for t in fields])
    return {"state": state, "sums": sums}


def _hand_over(d, st):
    """Sets a domain's interior from [ny][nx][3]; the velocity on an open
    face west or south of the interior is the adjacent interior face's."""
    xs, xe, ys, ye = d["ext"]
    for q, k in enumerate(("sn", "un", "vn")):
        a = torch.zeros_like(d[k])
        a[ys:ye + 1, xs:xe + 1] = st[:, :, q]
        d[k] = a
    m = d["m"]
    west = (m[ys:ye + 1, xs - 1] < 0)
    d["un"][ys:ye + 1, xs - 1] = torch.where(west, d["un"][ys:ye + 1, xs], 0.0)
    south = (m[ys - 1, xs:xe + 1] < 0)
    d["vn"][ys - 1, xs:xe + 1] = torch.where(south, d["vn"][ys, xs:xe + 1], 0.0)


# ---- the shallow-water step in 64-bit torch ----------------------------------


def _e(a):
    return torch.roll(a, -1, -1)


def _w(a):
    return torch.roll(a, 1, -1)


def _n(a):
    return torch.roll(a, -1, -2)


def _s(a):
    return torch.roll(a, 1, -2)


def _box(like, x0, x1, y0, y1):
    b = torch.zeros(like.shape[-2:], dtype=torch.bool, device="cuda")
    b[y0:y1 + 1, x0:x1 + 1] = True
    return b


def _face_ssh(d, sn):
    """Sea-surface height on the east and north faces (zero outside the
    ranges next_ssh covers); the areas of a T cell and a face are equal."""
    m = d["m"]
    xs, xe, ys, ye = d["ext"]
    out = []
    area = torch.tensor(1.0e6, dtype=torch.float64, device="cuda")  # on the GPU: a true divide
    for sh, box in ((_e, _box(m, xs, xe - 1, ys, ye)), (_n, _box(m, xs, xe, ys, ye - 1))):
        mn, nb = sh(m), sh(sn)
        both = 0.5 * (area * sn + area * nb) / area
        v = torch.where(m * mn > 0, both, torch.where(m <= 0, nb, sn))
        out.append(torch.where(box & (m + mn > 0), v, torch.zeros_like(v)))
    return out


class _Solver:
    """NEMOLite2D steps of equal-sized domains, [domain][row][column], on a
    uniform 1 km grid at 50 degrees north."""

    def __init__(self, doms):
        for k in ("m", "ht", "hu", "hv", "sn", "un", "vn"):
            setattr(self, k, torch.stack([d[k] for d in doms]))
        d = doms[0]
        self.ext, self.rdt, self.cbfr, self.visc = d["ext"], d["rdt"], d["cbfr"], d["visc"]
        self.tide = [(q["amp"], q["period_h"]) for q in doms]
        self.cor = 2.0 * 7.292116e-05 * math.sin(50.0 * (3.1415926535897932 / 180.0))
        self.g = 9.80665
        m = self.m
        xs, xe, ys, ye = self.ext
        box = lambda *r: _box(m, *r)  # noqa: E731
        me, mn, mw, ms = _e(m), _n(m), _w(m), _s(m)
        self.inner = box(xs, xe, ys, ye)
        self.copy = box(xs - 1, xe + 1, ys - 1, ye)
        self.open_t = self.inner & (m > 0) & ((ms < 0) | (mn < 0) | (me < 0) | (mw < 0))
        self.mom_u = box(xs, xe - 1, ys, ye) & (m > 0) & (me > 0)
        self.mom_v = box(xs, xe, ys, ye - 1) & (m + me > 0) & (m > 0) & (mn > 0)
        self.dry_s, self.dry_n = (ms <= 0) | (_e(ms) <= 0), (mn <= 0) | (_e(mn) <= 0)
        self.dry_w, self.dry_e = (mw <= 0) | (_n(mw) <= 0), (me <= 0) | (_n(me) <= 0)
        whole_u, whole_v = box(xs - 1, xe, ys - 1, ye + 1), box(xs - 1, xe + 1, ys - 1, ye)
        self.solid_u, self.solid_v = whole_u & (m * me == 0), whole_v & (m * mn == 0)
        self.fl_u0 = whole_u & (m + me > -1) & (m < 0)
        self.fl_u1 = whole_u & (m + me > -1) & ~(m < 0) & (me < 0)
        self.fl_v0 = whole_v & (m + mn > -1) & (m < 0)
        self.fl_v1 = whole_v & (m + mn > -1) & ~(m < 0) & (mn < 0)
        self.z = torch.zeros_like(self.sn)

    def _momentum(self, a, b, ha, hb, sa, sb, E, W, N, S, dry_s, dry_n, cor):
        """New `a` (the velocity along E / W) before the boundary conditions,
        `b` the other velocity, ha / hb and sa / sb the depths and heights at
        their faces; N / S shift across."""
        z, sn, ht = self.z, self.sn, self.ht
        dx = 1000.0
        dep = ht + sn
        Ha, Hb = ha + sa, hb + sb
        ue, uw = 0.5 * (a + E(a)) * dx, 0.5 * (a + W(a)) * dx
        adv = (torch.where(uw < 0, a, W(a)) * uw * dep -
               torch.where(ue < 0, E(a), a) * ue * E(dep))
        bs = 0.5 * (S(b) + E(S(b)))
        bn = 0.5 * (b + E(b))
        vs, vn = bs * dx, bn * dx
        ds, dn = 0.5 * (S(Hb) + E(S(Hb))), 0.5 * (Hb + E(Hb))
        adv = (adv + torch.where(vs < 0, a, torch.where(dry_s, z, S(a))) * vs * ds -
               torch.where(vn < 0, torch.where(dry_n, z, N(a)), a) * vn * dn)
        ge, gw = (E(a) - a) / dx * E(dep), (a - W(a)) / dx * dep
        gs = torch.where(dry_s, z, (a - S(a)) / (2 * dx) * (Ha + S(Ha)))
        gn = torch.where(dry_n, z, (N(a) - a) / (2 * dx) * (Ha + N(Ha)))
        vis = self.visc * ((ge - gw) * dx + 0.5 * (gn - gs) * dx)
        c = 0.5 * cor * (bs + bn) * dx * dx * Ha
        hpg = -self.g * Ha * dx * (E(sn) - sn)
        return ((a * Ha + self.rdt * (adv + vis + c + hpg) / (dx * dx)) / ha /
                (1.0 + self.cbfr * self.rdt))

    def step(self, istep):
        sn, un, vn, hu, hv, z = self.sn, self.un, self.vn, self.hu, self.hv, self.z
        su, sv = _face_ssh({"m": self.m, "ext": self.ext}, sn)
        fu, fv = (su + hu) * un, (sv + hv) * vn
        ssh = sn + (_w(fu) - fu + _s(fv) - fv) * self.rdt / 1.0e6
        t = istep * self.rdt
        tide = torch.tensor([a * math.sin(2.0 * 3.14159 / (p * 3600.0) * t)
                             for a, p in self.tide], dtype=torch.float64, device="cuda")
        ssh = torch.where(self.open_t, tide[:, None, None], torch.where(self.inner, ssh, sn))
        ua = self._momentum(un, vn, hu, hv, su, sv, _e, _w, _n, _s, self.dry_s, self.dry_n,
                            self.cor)
        va = self._momentum(vn, un, hv, hu, sv, su, _n, _s, _e, _w, self.dry_w, self.dry_e,
                            -self.cor)
        ua = torch.where(self.solid_u, z, torch.where(self.mom_u, ua, un))
        va = torch.where(self.solid_v, z, torch.where(self.mom_v, va, vn))
        cu, cv = torch.sqrt(self.g / hu), torch.sqrt(self.g / hv)
        ua = torch.where(self.fl_u0, _e(ua) + cu * (su - _e(su)),
                         torch.where(self.fl_u1, _w(ua) + cu * (su - _w(su)), ua))
        va = torch.where(self.fl_v0, _n(va) + cv * (sv - _n(sv)),
                         torch.where(self.fl_v1, _s(va) + cv * (sv - _s(sv)), va))
        self.sn = torch.where(self.copy, ssh, sn)
        self.un = torch.where(self.copy, ua, un)
        self.vn = torch.where(self.copy, va, vn)

    def sums(self, q):
        xs, xe, ys, ye = self.ext
        return torch.stack([self.sn[q, ys:ye + 1, xs:xe + 1].abs().sum(),
                            self.un[q, ys:ye + 1, xs:xe].abs().sum(),
                            self.vn[q, ys:ye, xs:xe + 1].abs().sum()])


# ---- tracer advection --------------------------------------------------------

TRA_ARRAYS = ("ztfreez", "pun", "pvn", "pwn", "umask", "vmask", "tmask", "rnfmsk", "rnfmsk_z",
              "upsmsk", "mydomain", "tsn")


def _tra_fields(case, seed):
    """The benchmark's arrays (Fortran layout a(ji, jj, jk) -> a[jk, jj, ji])
    on the GPU: its own initial values with 10 % of noise, or a basin of 0 / 1
    masks with temperatures and Courant numbers of either sign."""
    g = _gen(seed)
    ni, nj, nk = case["jpi"], case["jpj"], case["jpk"]
    i, j, k = (torch.arange(1, n + 1, dtype=torch.float64, device="cuda") for n in (ni, nj, nk))
    rand = lambda *s: torch.rand(s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    v2 = j[:, None] * i[None, :] / (ni * nj)
    f = {}
    if case["masks"] == "benchmark":
        v3 = k[:, None, None] * j[:, None] * i / (ni * nj * nk)
        for n in ("mydomain", "tsn", "pun", "pvn", "pwn", "umask", "vmask", "tmask"):
            f[n] = v3 * (0.95 + 0.1 * rand(nk, nj, ni))
        for n in ("ztfreez", "rnfmsk", "upsmsk"):
            f[n] = v2 * (0.95 + 0.1 * rand(nj, ni))
    else:
        sea = (rand(nj, ni) > 0.1).double()
        bottom = (k[:, None, None] <= (0.3 + 0.7 * rand(nj, ni)) * nk).double()
        f["tmask"] = sea * bottom
        f["umask"], f["vmask"] = f["tmask"] * _e(f["tmask"]), f["tmask"] * _n(f["tmask"])
        f["mydomain"] = (4.0 + 20.0 * rand(nk, nj, ni)) * f["tmask"]
        f["tsn"] = f["mydomain"].clone()
        for n, mk in (("pun", "umask"), ("pvn", "vmask"), ("pwn", "tmask")):
            f[n] = (1.6 * rand(nk, nj, ni) - 0.8) * f[mk]
        f["ztfreez"] = torch.full((nj, ni), -1.8, dtype=torch.float64, device="cuda")
        f["rnfmsk"] = (rand(nj, ni) > 0.98).double()
        f["upsmsk"] = (rand(nj, ni) > 0.99).double()
    f["rnfmsk_z"] = torch.floor(k / nk)
    return f


class _TraRun:
    """The benchmark program: a first call from host arrays, the remaining
    iterations on the resident field, the field read back."""

    def __init__(self, case, seed):
        self.case = case
        self.f = {}
        for n, t in _tra_fields(case, seed).items():
            self.f[n] = _pinned(t.shape, torch.float64)
            self.f[n].copy_(t)
        self.out = _pinned(self.f["mydomain"].shape, torch.float64)

    @staticmethod
    def _p(t):
        return ctypes.cast(t.data_ptr(), _DP)

    def run(self):
        c = self.case
        LIB.tra_adv_compute(*[self._p(self.f[n]) for n in TRA_ARRAYS], c["jpi"], c["jpj"],
                            c["jpk"])
        ms = ctypes.c_double(0.0)
        rc = LIB.tra_adv_run(c["iters"] - 1, ctypes.byref(ms)) or LIB.tra_adv_read(
            self._p(self.out))
        if rc or LIB.tra_adv_last_error(None, 0):
            raise P.Nl2dError("tracer advection failed (%d)" % rc)
        LIB.tra_adv_finalize()  # the program's end: the next pass is a new run
        return self.out


def _exact_tra(case, seed):
    f = _tra_fields(case, seed)
    nk, nj, ni = f["tmask"].shape
    m = f["mydomain"].clone()
    zice = (f["tsn"] <= f["ztfreez"] + 0.1).double()
    up = torch.maximum(torch.maximum(f["rnfmsk"] * f["rnfmsk_z"][:, None, None], f["upsmsk"]),
                       zice) * f["tmask"]
    zind = 1.0 - up

    def limited(a, b):
        s = (a + b) * (0.25 + torch.copysign(torch.full_like(a, 0.25), a * b))
        lim = torch.minimum(torch.minimum(s.abs(), 2.0 * b.abs()), 2.0 * a.abs())
        return torch.copysign(torch.ones_like(s), s) * lim

    half = torch.full_like(m, 0.5)
    edge = None  # the x difference east of the last interior column
    ii, jj = slice(1, ni - 1), slice(1, nj - 1)
    for it in range(case["iters"]):
        fl = {}
        for ax, (vel, mask) in (("x", ("pun", "umask")), ("y", ("pvn", "vmask"))):
            up_, dn = (_e, _w) if ax == "x" else (_n, _s)
            dif = f[mask] * (up_(m) - m)
            if ax == "x":
                dif[:, :, ni - 1] = 0.0 if edge is None else edge
            else:
                dif[:, nj - 1, :] = 0.0
            sl = limited(dif, dn(dif))
            z0 = torch.copysign(half, f[vel])
            zu = z0 - 0.5 * f[vel]
            far = up_(m) + zind * (zu * up_(sl))
            near = m + zind * (zu * sl)
            al = 0.5 - z0
            flux = f[vel] * (al * far + (1.0 - al) * near)
            if ax == "x":
                flux[:, :, 0] = dif[:, :, 0]
            else:
                flux[:, 0, :] = dif[:, 0, :]
            fl[ax] = flux - dn(flux)
        h = m.clone()
        h[:nk - 1, jj, ii] -= (fl["x"] + fl["y"])[:nk - 1, jj, ii]
        if edge is None:
            c = m[:, :, ni - 1]
            edge = f["tmask"][:, :, ni - 1] * (torch.roll(c, 1, 0) - c)
            edge[0] = f["pwn"][0, :, ni - 1] * c[0]
        zd = f["tmask"] * (torch.roll(h, 1, 0) - h)
        zd[0] = 0.0
        zd[nk - 1] = 0.0
        zn = torch.roll(zd, -1, 0)
        sl = limited(zd, zn)
        sl[0] = 0.0
        sl[nk - 1] = 0.0
        p1 = torch.roll(f["pwn"], -1, 0)
        z0 = torch.copysign(half, p1)
        zw = z0 - 0.5 * p1
        below, here = (torch.roll(h, -1, 0) + zind * (zw * torch.roll(sl, -1, 0)),
                       h + zind * (zw * sl))
        al = 0.5 + z0
        fw1 = p1 * (al * below + (1.0 - al) * here)
        fw = torch.roll(fw1, 1, 0)
        fw[0] = f["pwn"][0] * h[0]
        m = h
        m[:nk - 1, jj, ii] = (fw1 - fw)[:nk - 1, jj, ii]
    return m


# ---- the emulator's convolutions ---------------------------------------------


def _images(case, seed):
    g = _gen(seed)
    b, h, w, ci, co = (case[k] for k in ("batch", "h", "w", "cin", "cout"))
    x = torch.randn(b * h * w, ci, generator=g, device="cuda").relu_().to(torch.bfloat16)
    wt = (torch.randn(9, co, ci, generator=g, device="cuda") * math.sqrt(2.0 / (9 * ci))).to(
        torch.bfloat16)
    bias = 0.1 * torch.randn(co, generator=g, device="cuda")
    dy = (0.01 * torch.randn(b * h * w, co, generator=g, device="cuda")).to(torch.bfloat16)
    return x, wt, bias, dy


def _vp(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


class _Conv:
    """One layer's forward pass: BF16 activations in and out (hidden layers)
    or FP32 out (the last layer, and input gradients without bias)."""

    def __init__(self, case, seed):
        self.case = case
        self.x, self.w, self.b, dy = _images(case, seed)
        n = self.x.shape[0]
        self.bf16 = case["out"] == "bf16"
        self.y = torch.zeros(n, case["cout"], device="cuda",
                             dtype=torch.bfloat16 if self.bf16 else torch.float32)
        self.err = torch.zeros(1, dtype=torch.int32, device="cuda")

    def run(self):
        c = self.case
        P.check(LIB.nl2d_emu_conv3x3(
            _vp(self.x), _vp(self.w), _vp(self.b), _vp(self.y if self.bf16 else None),
            _vp(None if self.bf16 else self.y), c["batch"], c["h"], c["w"], c["cin"], c["cout"],
            int(c["relu"]), _vp(self.err), None), "nl2d_emu_conv3x3")
        return {"y": self.y, "err": self.err}


class _WeightGrad:
    """One layer's weight and bias gradients, into zeroed buffers as a
    training step does."""

    def __init__(self, case, seed):
        self.case = case
        self.x, w, b, self.dy = _images(case, seed)
        self.dw = torch.zeros(w.shape, device="cuda")
        self.db = torch.zeros_like(b)
        self.err = torch.zeros(1, dtype=torch.int32, device="cuda")

    def run(self):
        c = self.case
        self.dw.zero_()
        self.db.zero_()
        P.check(LIB.nl2d_emu_conv_wgrad(_vp(self.x), _vp(self.dy), _vp(self.dw), _vp(self.db),
                                        c["batch"], c["h"], c["w"], c["cin"], c["cout"],
                                        _vp(self.err), None), "nl2d_emu_conv_wgrad")
        return {"dw": self.dw, "db": self.db, "err": self.err}


def _taps(x):
    """The nine shifted images, zero outside, of x [b][h][w][c]."""
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    h, w = x.shape[1:3]
    return [p[:, t // 3:t // 3 + h, t % 3:t % 3 + w].reshape(-1, x.shape[3]) for t in range(9)]


def _exact_conv(case, seed):
    x, wt, bias, _ = _images(case, seed)
    img = x.double().reshape(case["batch"], case["h"], case["w"], case["cin"])
    y = bias.double().repeat(x.shape[0], 1)
    for t, xt in enumerate(_taps(img)):
        y += xt @ wt[t].double().t()
    return {"y": y.relu_() if case["relu"] else y, "err": None}


def _exact_wgrad(case, seed):
    x, _, _, dy = _images(case, seed)
    img = x.double().reshape(case["batch"], case["h"], case["w"], case["cin"])
    d = dy.double()
    dw = torch.stack([d.t() @ xt for xt in _taps(img)])
    return {"dw": dw, "db": d.sum(dim=0), "err": None}
