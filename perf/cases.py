"""Timed workloads of the framework, through its public entry points.

A case is a dict of plain values.  Its `kind` says which call a user's
program makes; sizes are (nz, ny, nx) with x fastest.  Fields are normalised
Perlin fBm in [0, 1] and their decompressed copies the project's compressor
stand-ins ("sz3": plateaus of width 2 eps, "zfp": dense bounded noise), the
inputs of every workload of this repository.

  correct      one field corrected on the device (f, fhat -> corrected field)
  naive        the same through the naive-MSz strategy
  host         the whole host-buffer pipeline: pinned inputs in, packed edit
               symbols and clamp list out
  batch        many small fields of uneven shapes corrected together
  serve        a burst of jobs handed to a running correction server
  segment      steepest-direction codes and both manifold labels of a field
  verify       re-verification of a corrected field against its original
  extract      edit output (symbols and clamp list) of a corrected field
  reconstruct  the corrected field rebuilt from its edit output
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from pmsz_anonymous_gb300 import api

Q = 5
DTYPES = {"f32": torch.float32, "f64": torch.float64}


def _field(kind, name, shape, dtype, comp, eps, octaves, period, persistence=0.5):
    nz, ny, nx = shape
    return {"name": name, "kind": kind, "nz": nz, "ny": ny, "nx": nx, "dtype": dtype, "comp": comp, "eps": eps,
            "octaves": octaves, "period": period, "persistence": persistence}


def listed():
    return [
        # one block of a small simulation, or a quick look at a new data set:
        # the smallest plain call, where launches and latency count
        _field("correct", "correct_64_f32_sz3", (64, 64, 64), "f32", "sz3", 1e-3, 4, 32),
        # a cropped region with ragged axes: rows that are no multiple of 16
        # bytes, a last tile that is partly empty in every axis
        _field("correct", "correct_ragged_f32_zfp", (173, 141, 203), "f32", "zfp", 1e-4, 4, 32),
        # the per-rank block of a weak-scaling run, the headline workload
        _field("correct", "correct_512_f64_zfp", (512, 512, 512), "f64", "zfp", 1e-4, 5, 64),
        # a large single domain with quantised plateaus (cosmology-sized cuts)
        _field("correct", "correct_large_f32_sz3", (576, 768, 704), "f32", "sz3", 1e-4, 6, 128, 0.55),
        # segmentation-only correction, the reference's second program
        _field("naive", "naive_160_f64_zfp", (160, 144, 176), "f64", "zfp", 1e-4, 4, 32),
        # what the command-line program does between reading and encoding
        _field("host", "host_256_f64_zfp", (256, 320, 288), "f64", "zfp", 1e-4, 5, 64),
        # many time steps / variables of uneven shapes in one call; half sz3,
        # half zfp, error bounds over three decades
        {"name": "batch_32_f32_mixed", "kind": "batch", "fields": 32, "layout": 100, "lo": 32, "hi": 256, "f64_share": 0.0},
        # a burst of jobs at a correction service, 70 % fp32 / 30 % fp64
        {"name": "serve_24_mixed", "kind": "serve", "fields": 24, "layout": 1000, "lo": 32, "hi": 192, "f64_share": 0.3},
        # topological segmentation of a field (codes, then AS / DS labels)
        _field("segment", "segment_f32", (320, 288, 352), "f32", "zfp", 1e-4, 5, 64),
        # checking a corrected field before it is archived
        _field("verify", "verify_f64_zfp", (384, 448, 416), "f64", "zfp", 1e-4, 5, 64),
        # the encoder's input from a corrected field kept on the device
        _field("extract", "extract_f64_zfp", (512, 448, 480), "f64", "zfp", 1e-4, 5, 64),
        # reading an archive back; an odd voxel count
        _field("reconstruct", "reconstruct_f64_zfp", (511, 449, 479), "f64", "zfp", 1e-4, 5, 64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape(rng, lo, hi, cap):
    while True:
        s = tuple(_log_int(rng, lo, hi) for _ in range(3))
        if s[0] * s[1] * s[2] <= cap:
            return s


def draw(rng):
    kind = rng.choice(["correct", "correct", "correct", "naive", "host", "batch", "serve", "segment", "verify",
                       "extract", "reconstruct"])
    if kind in ("batch", "serve"):
        return {"kind": kind, "fields": rng.randint(2, 24), "layout": rng.randrange(1 << 20), "lo": 32,
                "hi": _log_int(rng, 64, 192), "f64_share": rng.choice([0.0, 0.3])}
    # the naive strategy's iteration count grows with size and error bound
    hi, cap = {"correct": (768, 130_000_000), "naive": (144, 2_000_000), "host": (384, 16_000_000)}.get(
        kind, (512, 60_000_000))
    nz, ny, nx = _shape(rng, 32, hi, cap)
    return {"kind": kind, "nz": nz, "ny": ny, "nx": nx, "dtype": rng.choice(["f32", "f64"]),
            "comp": rng.choice(["sz3", "zfp"]),
            "eps": 10.0 ** (rng.uniform(-5, -3) if kind == "naive" else rng.uniform(-5, -2)),
            "octaves": rng.randint(3, 6), "period": rng.choice([32, 64, 128]), "persistence": 0.5}


def _members(case):
    """The fields of a batch or of a burst of jobs (everything but the seed)."""
    rng = random.Random(case["layout"])
    out = []
    for k in range(case["fields"]):
        size = (lambda: rng.randint(case["lo"], case["hi"])) if case["kind"] == "batch" else \
            (lambda: _log_int(rng, case["lo"], case["hi"]))
        nz, ny, nx = size(), size(), size()
        out.append({"nz": nz, "ny": ny, "nx": nx, "dtype": "f64" if rng.random() < case["f64_share"] else "f32",
                    "comp": "sz3" if k % 2 == 0 else "zfp", "eps": 10.0 ** rng.uniform(-5, -2),
                    "octaves": 4 if case["kind"] == "batch" else rng.randint(3, 6), "period": 32, "persistence": 0.5})
    return out


def _make(c, seed):
    seed = int(seed) & 0x7FFFFFFF
    f = api.gen_perlin((c["nz"], c["ny"], c["nx"]), seed=seed, octaves=c["octaves"], base_freq=1.0 / c["period"],
                       persistence=c["persistence"], dtype=DTYPES[c["dtype"]], device="cuda")
    return f, api.standin(f, c["eps"], c["comp"], seed=seed)


def _pairs(case, seed):
    return [(*_make(c, seed * 4099 + k), c["eps"]) for k, c in enumerate(_members(case))]


def _pools(pairs):
    """One buffer per type for the corrected fields of many jobs (fields start
    on 256-byte boundaries), and each field's start in its buffer."""
    size, spans = {}, []
    for _, fh, _ in pairs:
        key = str(fh.dtype)
        spans.append(size.get(key, 0))
        size[key] = spans[-1] + (fh.numel() + 63) // 64 * 64
    return {str(fh.dtype): torch.zeros(size[str(fh.dtype)], dtype=fh.dtype, device=fh.device)
            for _, fh, _ in pairs}, spans


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        pairs = _pairs(case, seed)
        pools, spans = _pools(pairs)
        work = [pools[str(fh.dtype)][a: a + fh.numel()].view(fh.shape) for (_, fh, _), a in zip(pairs, spans)]
        state = {"kind": kind, "pairs": pairs, "pools": pools, "work": work}
        if kind == "serve":
            state["server"] = api.Server(hbm_budget_bytes=120 << 30)
        torch.cuda.synchronize()
        return state
    f, fh = _make(case, seed)
    state = {"kind": kind, "f": f, "fh": fh, "eps": case["eps"]}
    if kind in ("correct", "naive"):
        state["work"] = torch.empty_like(fh)
    elif kind == "host":
        n = f.numel()
        state["f"] = f.cpu().pin_memory()
        state["fh"] = fh.cpu().pin_memory()
        state["deltas"] = torch.empty(api.packed_len(n, Q), dtype=torch.uint8).pin_memory()
        state["clamp"] = torch.zeros(n, dtype=f.dtype).pin_memory()
    elif kind in ("verify", "extract", "reconstruct"):
        cur = fh.clone()
        api.correct(f, cur, case["eps"], q=Q)
        state["cur"] = cur
        if kind == "extract":
            state["clamp"] = torch.zeros(fh.numel(), dtype=fh.dtype, device=fh.device)
        if kind == "reconstruct":
            deltas, clamp, _ = api.extract_edits(fh, cur, f, case["eps"], q=Q)
            state["deltas"], state["clamp"] = deltas, clamp.clone()
            state["out"] = torch.empty_like(fh)
            del state["f"], state["cur"]
    torch.cuda.synchronize()
    return state


LOG_ROWS = 256


def _rows(log):
    """The sweep log in a table of LOG_ROWS rows (more only for longer logs)."""
    rows = LOG_ROWS
    while rows < len(log):
        rows *= 2
    out = np.zeros((rows, log.shape[1]), np.int64)
    out[: len(log)] = log
    return out


def _result(r):
    return {"status": r.status, "sweeps": r.sweeps, "iteration": r.iteration, "edits": r.edits, "log": _rows(r.log)}


def run(state):
    kind = state["kind"]
    if kind in ("correct", "naive"):
        # the decompressed field is kept (the edit output compares with it)
        work = state["work"]
        work.copy_(state["fh"])
        r = api.correct(state["f"], work, state["eps"], q=Q, strategy="naive" if kind == "naive" else "pmsz")
        return {"field": work, **_result(r)}
    if kind == "host":
        r, extra = api.correct_host(state["f"], state["fh"], state["eps"], q=Q, deltas=state["deltas"],
                                    clamp=state["clamp"], edits_only=True, packed_deltas=True)
        return {"packed": state["deltas"], "clamp": state["clamp"], "n_clamp": extra["n_clamp"],
                "edit_count": extra["edit_count"], **_result(r)}
    if kind == "batch":
        for w, (_, fh, _) in zip(state["work"], state["pairs"]):
            w.copy_(fh)
        rs = api.correct_batch([(f, w, eb) for w, (f, _, eb) in zip(state["work"], state["pairs"])], q=Q)
        return {"fields": state["pools"], "stats": np.array([(r.status, r.sweeps, r.iteration, r.edits) for r in rs]),
                "logs": _rows(np.concatenate([r.log for r in rs]).astype(np.int64))}
    if kind == "serve":
        for w, (_, fh, _) in zip(state["work"], state["pairs"]):
            w.copy_(fh)
        torch.cuda.current_stream().synchronize()  # submit wants the fields' producing work completed
        srv = state["server"]
        ids = [srv.submit(f, w, eb) for w, (f, _, eb) in zip(state["work"], state["pairs"])]
        infos = [srv.wait(j) for j in ids]
        return {"fields": state["pools"],
                "stats": np.array([[int(i[k]) for k in ("done", "status", "sweeps", "edits")] for i in infos])}
    if kind == "segment":
        codes = api.codes(state["f"])
        asc, desc = api.labels(codes)
        return {"codes": codes, "asc": asc, "desc": desc}
    if kind == "verify":
        return api.verify(state["f"], state["cur"], state["eps"])
    if kind == "extract":
        deltas, clamp, edits = api.extract_edits(state["fh"], state["cur"], state["f"], state["eps"], q=Q)
        state["clamp"][: clamp.numel()] = clamp
        return {"deltas": deltas, "clamp": state["clamp"], "n_clamp": clamp.numel(), "edit_count": edits}
    if kind == "reconstruct":
        return api.reconstruct(state["fh"], state["deltas"], state["clamp"], state["eps"], q=Q, out=state["out"])
    raise ValueError(kind)


def work(case):
    """Each input read once, each output written once; the comparisons of one
    15-point argmax and argmin per field count as operations.  Clamp values
    (a few per thousand voxels) are left out."""
    kind = case["kind"]
    if kind in ("batch", "serve"):
        parts = [work({**m, "kind": "correct"}) for m in _members(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n = case["nz"] * case["ny"] * case["nx"]
    s = 4 if case["dtype"] == "f32" else 8
    nbytes = {"correct": 3 * s * n, "naive": 3 * s * n,
              "host": 2 * s * n + api.packed_len(n, Q),
              "segment": n * (s + 1) + n * 16,       # codes, two int64 labels
              "verify": 2 * s * n,
              "extract": n * (3 * s + 1),
              "reconstruct": n * (2 * s + 1)}[kind]
    flops = {"segment": 28, "extract": 2, "reconstruct": 1}.get(kind, 56) * n
    return {"bytes": int(nbytes), "flops": int(flops)}


# ---- plain torch values --------------------------------------------------------------------------
# The corrected field is defined in the field's own type (its edits subtract
# delta and test the bound in that type), so the sweeps below run in that type
# and their result is widened to 64 bits.

# (dx, dy, dz) of the 15 stencil points, in the order of (dz, dy, dx)
OFFSETS = [(0, -1, -1), (1, -1, -1), (0, 0, -1), (1, 0, -1), (0, -1, 0), (1, -1, 0), (-1, 0, 0), (0, 0, 0),
           (1, 0, 0), (-1, 1, 0), (0, 1, 0), (-1, 0, 1), (0, 0, 1), (-1, 1, 1), (0, 1, 1)]
SELF = 7


def _flat_offsets(shape, device):
    _, ny, nx = shape
    return torch.tensor([dx + nx * (dy + ny * dz) for dx, dy, dz in OFFSETS], dtype=torch.int64, device=device)


def _steepest(v):
    """Ranks of the steepest ascent and descent point of every voxel (flat)."""
    def span(d, n):
        return (slice(max(0, -d), n - max(0, d)), slice(max(0, d), n - max(0, -d)))
    hi = torch.full_like(v, -math.inf)
    lo = torch.full_like(v, math.inf)
    asc = torch.full(v.shape, SELF, dtype=torch.uint8, device=v.device)
    desc = asc.clone()
    for r, (dx, dy, dz) in enumerate(OFFSETS):
        if any(abs(d) >= n for d, n in zip((dz, dy, dx), v.shape)):
            continue
        (zi, zo), (yi, yo), (xi, xo) = (span(d, n) for d, n in zip((dz, dy, dx), v.shape))
        at, nb = (zi, yi, xi), v[zo, yo, xo]
        up, down = nb >= hi[at], nb < lo[at]
        hi[at] = torch.where(up, nb, hi[at])
        lo[at] = torch.where(down, nb, lo[at])
        asc[at] = asc[at].masked_fill(up, r)
        desc[at] = desc[at].masked_fill(down, r)
    return asc.view(-1), desc.view(-1)


def _edit(f, v, cnt, req, eps, delta):
    """One edit of every requested voxel; how many changed value or count."""
    i = req.nonzero().view(-1)
    old, c, o = v[i], cnt[i], f[i]
    low = old - delta
    step = ((o - low).abs() <= eps) & (c < Q - 1)
    new, nc = torch.where(step, low, o - eps), torch.where(step, c + 1, torch.full_like(c, Q))
    v[i], cnt[i] = new, nc
    return int(((new != old) | (nc != c)).sum())


def _request(req, off, where, rank):
    i = where.nonzero().view(-1)
    req[i + off[rank[i].long()]] = True


def _extrema(oa, od, ca, cd, off, req):
    """Requests at false and missing extrema; the voxels that have them."""
    omax = oa == SELF
    omin = ~omax & (od == SELF)
    r1, r2 = (ca == SELF) != omax, (cd == SELF) != omin
    _request(req, off, r1 & omax, ca)
    req |= r1 & ~omax
    _request(req, off, r2 & ~omin, od)
    req |= r2 & omin
    return r1 | r2


def _correct(f, fh, eb, max_sweeps=10000):
    off = _flat_offsets(f.shape, f.device)
    oa, od = _steepest(f)
    ff, v = f.reshape(-1), fh.clone()
    eps, delta = torch.tensor(eb, dtype=f.dtype, device=f.device), torch.tensor(eb / Q, dtype=f.dtype, device=f.device)
    cnt = torch.zeros(ff.numel(), dtype=torch.int16, device=f.device)
    for _ in range(max_sweeps):
        ca, cd = _steepest(v)
        req = torch.zeros(ff.numel(), dtype=torch.bool, device=f.device)
        ext = _extrema(oa, od, ca, cd, off, req)
        up, down = ~ext & (ca != oa), ~ext & (cd != od)
        _request(req, off, up, ca)
        _request(req, off, down, od)
        if not bool((ext | up | down).any()) or not _edit(ff, v.view(-1), cnt, req, eps, delta):
            break
    return v


def _roots(rank, off):
    nxt = torch.arange(rank.numel(), dtype=torch.int64, device=rank.device) + off[rank.long()]
    while True:
        hop = nxt[nxt]
        if torch.equal(hop, nxt):
            return nxt
        nxt = hop


def _repair(oa, od, ca, cd, as0, ds0, as1, ds1, off, req):
    """Requests of the integral-path repair at the first divergences."""
    omax = oa == SELF
    omin = ~omax & (od == SELF)
    cur = (ds0 != ds1).nonzero().view(-1)
    while True:
        go = ~(omax[cur] | omin[cur] | (od[cur] != cd[cur]))
        if not bool(go.any()):
            break
        cur = torch.where(go, cur + off[od[cur].long()], cur)
    cur = cur[~omin[cur] & (od[cur] != cd[cur])]
    req[cur + off[od[cur].long()]] = True
    r1 = torch.where(omax, od, oa)
    cur = (as0 != as1).nonzero().view(-1)
    while True:
        go = (r1[cur] == ca[cur]) & (r1[cur] != SELF)
        if not bool(go.any()):
            break
        cur = torch.where(go, cur + off[r1[cur].long()], cur)
    cur = cur[r1[cur] != ca[cur]]
    req[cur + off[ca[cur].long()]] = True


def _correct_naive(f, fh, eb):
    off = _flat_offsets(f.shape, f.device)
    oa, od = _steepest(f)
    as0, ds0 = _roots(oa, off), _roots(od, off)
    ff, v = f.reshape(-1), fh.clone()
    eps, delta = torch.tensor(eb, dtype=f.dtype, device=f.device), torch.tensor(eb / Q, dtype=f.dtype, device=f.device)
    cnt = torch.zeros(ff.numel(), dtype=torch.int16, device=f.device)
    extrema = True
    while True:
        moved = 0
        while extrema:
            ca, cd = _steepest(v)
            req = torch.zeros(ff.numel(), dtype=torch.bool, device=f.device)
            extrema = bool(_extrema(oa, od, ca, cd, off, req).any())
            step = _edit(ff, v.view(-1), cnt, req, eps, delta)
            if extrema and not step:
                return v
            moved += step
        ca, cd = _steepest(v)
        req = torch.zeros(ff.numel(), dtype=torch.bool, device=f.device)
        _repair(oa, od, ca, cd, as0, ds0, _roots(ca, off), _roots(cd, off), off, req)
        moved += _edit(ff, v.view(-1), cnt, req, eps, delta)
        ca, cd = _steepest(v)
        req = torch.zeros(ff.numel(), dtype=torch.bool, device=f.device)
        extrema = bool(_extrema(oa, od, ca, cd, off, req).any())
        same = torch.equal(_roots(ca, off), as0) and torch.equal(_roots(cd, off), ds0)
        if (same and not extrema) or not moved:
            return v


def exact(case, seed):
    kind = case["kind"]
    none = {"status": None, "sweeps": None, "iteration": None, "edits": None, "log": None}
    if kind in ("batch", "serve"):
        pairs = _pairs(case, seed)
        pools, spans = _pools(pairs)
        pools = {k: t.double() for k, t in pools.items()}
        for (f, fh, eb), a in zip(pairs, spans):
            pools[str(fh.dtype)][a: a + fh.numel()] = _correct(f, fh, eb).double().view(-1)
        return {"fields": pools, "stats": None, **({"logs": None} if kind == "batch" else {})}
    if kind in ("segment", "verify"):  # whole numbers only
        return None
    f, fh = _make(case, seed)
    if kind == "naive":
        return {"field": _correct_naive(f, fh, case["eps"]).double(), **none}
    cur = _correct(f, fh, case["eps"])
    if kind == "correct":
        return {"field": cur.double(), **none}
    if kind == "reconstruct":
        return cur.double()
    low = f - torch.tensor(case["eps"], dtype=f.dtype, device=f.device)
    values = low[(cur != fh) & (cur == low) & (low != 0)].double()
    clamp = torch.zeros(f.numel(), dtype=torch.float64, device=f.device)
    clamp[: values.numel()] = values
    if kind == "host":
        return {"packed": None, "clamp": clamp.cpu(), "n_clamp": None, "edit_count": None, **none}
    return {"deltas": None, "clamp": clamp, "n_clamp": None, "edit_count": None}
