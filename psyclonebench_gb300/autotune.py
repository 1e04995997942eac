"""Autotuner for the ensemble's schedule and tile shapes.

The search space is what the ensemble exposes (nl2d_ens_schedule,
nl2d_ens_tile):

* FP64 form: persistent CTAs per SM (1 or 2), tile assignment (contiguous
  cost-balanced chunks, longest processing time first, or one tile per CTA
  left to the hardware block scheduler), the cost weight given to the
  domains' ring cells (which take the general per-cell path), and the tile
  shape (32 x 16, 32 x 8, 16 x 16, 64 x 8, 32 x 32).  The reference's
  tiled OpenMP layer (psykal_omp/time_step_mod.f90:587-1182) takes its tile
  size as a run parameter; here it is searched.  The search has two stages:
  every schedule at one shape, then every other shape under the best schedule
  and under one-tile-per-CTA (the runner-up where that is the best): the
  knobs a new ensemble starts with are among them.  The strip height is
  left to the marches' own rules.
* Mixed and FP64-equivalent ("df") forms: the column march's strip height
  (the form's own rule, or 8, 16, 32 or 64 rows), under the FP64 knobs
  already applied.

Each candidate is timed on a few steps of the actual ensemble (after one
untimed step), the domains are put back at rest, and the fastest candidate
is kept.  Results are cached on disk per (domain size histogram, precision,
version of the kernels' costs), so a repeated ensemble of the same shape skips
the search.  Results do not depend on any knob: the FP64 form is bit-identical
under every one.
"""
import hashlib
import json
import os

from .ensemble import DEFAULT_KNOBS

# Raised whenever the kernels or the meaning of a knob change what a choice
# costs: entries stored under another version are not used.
COSTS_VERSION = 3

# (CTAs per SM, policy, boundary weight); policy 2 (one tile per CTA)
# ignores the CTAs per SM and the edge weight
SCHEDULES = ([(cps, pol, bw) for cps in (1, 2) for pol in (0, 1) for bw in (0.0, 4.0, 16.0)] +
             [(2, 2, 0.0)])
SHAPES = ((32, 16), (32, 8), (16, 16), (64, 8), (32, 32))
FIRST_SHAPE = SHAPES[0]  # the one every schedule is timed at
MARCH_ROWS = (DEFAULT_KNOBS["march_rows"], 8, 16, 32, 64)


def cache_path():
    base = os.environ.get("NL2D_TUNE_CACHE") or os.path.join(
        os.environ.get("XDG_CACHE_HOME", os.path.expanduser("~/.cache")), "psyclonebench_gb300")
    return os.path.join(base, "ensemble_schedule.json")


def signature(domains, precision="fp64"):
    """Histogram of interior sizes (log2 bins per axis) plus precision and the
    version of the kernels' costs."""
    hist = {}
    for d in domains:
        w, h, xs, xe, ys, ye = d["dims"]
        key = "%d:%d" % ((xe - xs + 1).bit_length(), (ye - ys + 1).bit_length())
        hist[key] = hist.get(key, 0) + 1
    blob = json.dumps([COSTS_VERSION, precision, sorted(hist.items())])
    return hashlib.sha1(blob.encode()).hexdigest()[:16]


def _load():
    try:
        with open(cache_path()) as f:
            return json.load(f)
    except Exception:
        return {}


def _store(db):
    p = cache_path()
    try:
        os.makedirs(os.path.dirname(p), exist_ok=True)
        with open(p, "w") as f:
            json.dump(db, f, indent=1)
    except OSError:
        pass


def _apply(ens, c):
    knobs = [c["ctas_per_sm"], c["policy"], c["boundary_weight"], tuple(c["tile"])]
    if c["march_rows"] != DEFAULT_KNOBS["march_rows"]:
        knobs.append(c["march_rows"])
    ens.schedule(*knobs)


def _time(ens, c, steps):
    _apply(ens, c)
    ens.run(1, 1)  # untimed: builds the schedule and graph
    ms, _ = ens.run(2, steps)
    ens.reset()
    return ms / steps


def _fp64_candidates(schedules=None):
    if schedules is None:
        return [{"ctas_per_sm": cps, "policy": pol, "boundary_weight": bw,
                 "tile": list(FIRST_SHAPE), "march_rows": DEFAULT_KNOBS["march_rows"]}
                for cps, pol, bw in SCHEDULES]
    out = []
    for shape in SHAPES[1:]:
        for cps, pol, bw in schedules:
            out.append({"ctas_per_sm": cps, "policy": pol, "boundary_weight": bw,
                        "tile": list(shape), "march_rows": DEFAULT_KNOBS["march_rows"]})
    return out


def tune(ens, steps=4, precision="fp64", use_cache=True, base=None):
    """Picks and applies the fastest knobs for `ens` in its current form
    (precision "fp64", "mixed" or "df"); returns a dict with the choice and
    the timings.  For "mixed" and "df", `base` holds the FP64 knobs to keep
    (default: those a new ensemble starts with).  Leaves the ensemble at rest."""
    sig = signature(ens.domains, precision)
    db = _load() if use_cache else {}
    if sig in db:
        c = db[sig]
        _apply(ens, c)
        return dict(c, cached=True)
    timings = []
    if precision in ("mixed", "df"):
        b = dict(base or DEFAULT_KNOBS)
        for mr in MARCH_ROWS:
            c = {"ctas_per_sm": b["ctas_per_sm"], "policy": b["policy"],
                 "boundary_weight": b["boundary_weight"], "tile": list(b["tile"]),
                 "march_rows": mr}
            timings.append((_time(ens, c, steps), c))
    else:
        for c in _fp64_candidates():
            timings.append((_time(ens, c, steps), c))
        order = [(c["ctas_per_sm"], c["policy"], c["boundary_weight"])
                 for _, c in sorted(timings, key=lambda t: t[0])]
        # the best schedule and one tile per CTA (the runner-up where that is the best)
        scheds = [order[0], order[1] if order[0][1] == 2 else (2, 2, 0.0)]
        for c in _fp64_candidates(scheds):
            timings.append((_time(ens, c, steps), c))
    ms, best = min(timings, key=lambda t: t[0])
    choice = dict(best, ms_per_step=ms,
                  timings=[dict(c, ms_per_step=t) for t, c in timings])
    _apply(ens, best)
    db[sig] = choice
    if use_cache:
        _store(db)
    return dict(choice, cached=False)
