"""The sweeps of many fields in one launch (csrc/sweep_multi.cuh) where they can
go wrong, against the CPU oracle: tables of one type and of both, fields of one
voxel and of several chunks side by side, fields that stop at different sweeps,
plateaus next to smooth fields, more log rows than one read brings back, jobs that join a running server.  Whole numbers and bits:
equal, no tolerance."""
import numpy as np
import pytest

from oracle import oracle as O
from pmsz_anonymous_gb300 import capi
from pmsz_anonymous_gb300 import fields as F

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def api():
    from pmsz_anonymous_gb300 import api as A
    return A


def _pair(kind, shape, dtype, seed):
    rng = np.random.default_rng(seed)
    if kind == "plateaus":
        f = rng.integers(0, 5, size=shape).astype(dtype)
        return f, (f + rng.integers(-1, 2, size=shape)).astype(dtype), 1.0
    f = F.perlin_field(shape, seed, 4, 1 / 16, dtype=dtype)
    eb = {"sparse": 1e-4, "dense": 1e-2}[kind]
    return f, F.standin(f, eb, "zfp", seed), eb


# one voxel, a row, less than a chunk of 2048 voxels, one chunk and a bit,
# several chunks with ragged rows
SHAPES = [(1, 1, 1), (1, 1, 40), (5, 9, 33), (8, 8, 32), (9, 8, 32), (3, 33, 257), (40, 24, 100), (34, 37, 41)]
KINDS = ["sparse", "dense", "plateaus"]


def _set(types, count):
    out = []
    for i in range(count):
        shape, dtype = SHAPES[i % len(SHAPES)], types[i % len(types)]
        out.append(_pair(KINDS[(i // len(SHAPES) + i) % 3], shape, dtype, 30 + i))
    return out


def _to(device, a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(device)


@pytest.mark.parametrize("types,count,limit,q", [
    ([np.float32], 24, 400, 5), ([np.float64], 24, 400, 5), ([np.float32, np.float64], 48, 400, 5),
    ([np.float64, np.float32], 70, 3, 5), ([np.float32, np.float64], 40, 600, 40)])
def test_batch(cuda, types, count, limit, q):
    pairs = _set(types, count)
    work = [_to(cuda, fh) for _, fh, _ in pairs]
    items = [(_to(cuda, f), w, eb) for (f, _, eb), w in zip(pairs, work)]
    for (f, fh, eb), w, r in zip(pairs, work, api().correct_batch(items, q=q, max_sweeps=limit)):
        if np.isnan(f).any():  # the perlin field of a single voxel: refused, the others go on
            assert (r.status, r.sweeps) == (capi.PMSZ_ERR_ARG, 1)
            continue
        ref, _, st, sw, recs = O.correct(f, fh, eb, q=q, max_sweeps=limit)
        assert (r.status, r.sweeps) == (st, sw)
        np.testing.assert_array_equal(r.log[:, :5], recs)
        np.testing.assert_array_equal(w.cpu().numpy().view(np.uint8), ref.view(np.uint8))


@pytest.mark.parametrize("max_jobs", [1, 7, 256])
def test_server(cuda, max_jobs):
    pairs = _set([np.float32, np.float64], 48)
    work = [_to(cuda, fh) for _, fh, _ in pairs]
    fs = [_to(cuda, f) for f, _, _ in pairs]
    torch.cuda.synchronize()
    with api().Server(max_jobs=max_jobs) as srv:
        ids = [srv.submit(f, w, eb) for f, w, (_, _, eb) in zip(fs[:30], work, pairs)]
        first = srv.wait(ids[0])  # the others join sets that already run
        ids += [srv.submit(f, w, eb) for f, w, (_, _, eb) in zip(fs[30:], work[30:], pairs[30:])]
        infos = [first] + [srv.wait(i) for i in ids[1:]]
    for (f, fh, eb), w, info in zip(pairs, work, infos):
        if np.isnan(f).any():
            assert (info["status"], info["sweeps"]) == (capi.PMSZ_ERR_ARG, 1)
            continue
        ref, _, st, sw, recs = O.correct(f, fh, eb, max_sweeps=10000)
        assert (info["status"], info["sweeps"], info["edits"]) == (st, sw, int(recs[:, 3].sum()))
        np.testing.assert_array_equal(w.cpu().numpy().view(np.uint8), ref.view(np.uint8))
