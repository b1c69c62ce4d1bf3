"""The sweeps in one cooperative launch (csrc/sweep.cuh) where they can go
wrong, against the CPU oracle: one group of words and several, sparse and dense
sweeps, failed certificates beyond the buffer, limits on the sweeps, logs longer
than what one read brings back.  Fields and
counters are bits and whole numbers: equal, no tolerance."""
import numpy as np
import pytest

from oracle import oracle as O
from pmsz_anonymous_gb300 import fields as F

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def api():
    from pmsz_anonymous_gb300 import api as A
    return A


def _check(device, f, fh, eb, shift=0, **kw):
    ref, cnt, st, sw, recs = O.correct(f, fh, eb, **kw)
    dev = []
    for a in (f, fh):  # `shift` elements into a buffer: no tensor map, unaligned rows
        buf = torch.empty(a.size + shift, dtype=torch.from_numpy(a[:1]).dtype, device=device)
        buf[shift:] = torch.from_numpy(np.ascontiguousarray(a)).ravel().to(device)
        dev.append(buf[shift:].view(a.shape))
    r = api().correct(*dev, eb, **kw)
    assert (r.status, r.sweeps) == (st, sw)
    np.testing.assert_array_equal(r.log[:, :5], recs)
    np.testing.assert_array_equal(dev[1].cpu().numpy().view(np.uint8), ref.view(np.uint8))
    return r


def _pair(kind, shape, dtype, seed):
    rng = np.random.default_rng(seed)
    if kind == "plateaus":  # ties everywhere: every certificate of a sweep fails
        f = rng.integers(0, 5, size=shape).astype(dtype)
        return f, (f + rng.integers(-1, 2, size=shape)).astype(dtype), 1.0
    f = F.perlin_field(shape, seed, 4, 1 / 16, dtype=dtype)
    eb = {"sparse": 1e-4, "dense": 1e-2}[kind]
    return f, F.standin(f, eb, "zfp", seed), eb


# a single voxel row, less than a group of 8 words, one group, groups that end
# inside rows and planes, rows of several words with a remainder
SHAPES = [(1, 1, 40), (1, 7, 32), (2, 4, 32), (5, 9, 33), (9, 10, 70), (3, 33, 257), (40, 24, 100)]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["sparse", "dense", "plateaus"])
@pytest.mark.parametrize("shift", [0, 1])
def test_sweeps(cuda, shape, dtype, kind, shift):
    f, fh, eb = _pair(kind, shape, dtype, 11)
    _check(cuda, f, fh, eb, shift, max_sweeps=400)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("limit", [1, 2, 3, 64, 65, 300])
def test_limits(cuda, dtype, limit):
    f, fh, eb = _pair("dense", (24, 24, 40), dtype, 4)
    _check(cuda, f, fh, eb, q=40, max_sweeps=limit)


# chunks of 2, 4 and 8 groups (several rounds of them: test_gpu_rounds.py): the
# full-field sweeps are the reference here
@pytest.mark.parametrize("shape", [(120, 250, 500), (250, 256, 500), (401, 400, 410)], ids=str)
def test_chunks(cuda, shape):
    A = api()
    f = A.gen_perlin(shape, 3, 4, 1 / 32, 0.5, dtype=torch.float32)
    fh = A.standin(f, 1e-3, "sz3", 3)
    a, b = fh.clone(), fh.clone()
    ra = A.correct(f, a, 1e-3, max_sweeps=6)
    rb = A.correct(f, b, 1e-3, max_sweeps=6, full_sweeps=True)
    assert (ra.status, ra.sweeps) == (rb.status, rb.sweeps) and ra.sweeps > 3
    np.testing.assert_array_equal(ra.log[:, :5], rb.log[:, :5])
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))
