"""Direction codes and full sweeps of fields with many ties in the truncated
proxies (csrc/march.cuh), where a row of 32 voxels is decided in place or voxel
by voxel through the queue: rows with any number of tied voxels, infinities and
NaN of every sign (codes order them by their keys), ragged tiles, shallow and
deep columns, and thin fields.  Codes, fields and counters are whole numbers and bits: equal, no
tolerance."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

OFFSETS = sorted([(0, 0, 0), (0, 0, 1), (0, 0, -1), (0, 1, 0), (0, -1, 0), (1, 0, 0), (-1, 0, 0), (0, 1, -1), (0, -1, 1),
                  (1, 0, -1), (-1, 0, 1), (1, 1, 0), (-1, -1, 0), (1, 1, -1), (-1, -1, 1)])  # (dz, dy, dx) in rank order


def api():
    from pmsz_anonymous_gb300 import api as A
    return A


def _field(kind, shape, dtype):
    rng = np.random.default_rng(len(kind) + sum(shape))
    n = int(np.prod(shape))
    if kind == "ints":
        return rng.integers(0, 5, size=shape).astype(dtype)
    if kind == "ramp":
        return (np.arange(n) / (4.0 * n)).astype(dtype).reshape(shape)
    if kind == "special":
        pool = np.array([0.0, -0.0, 1.0, -1.0, np.finfo(dtype).tiny / 4, np.inf, -np.inf, np.nan, -np.nan, np.finfo(dtype).max])
        return rng.choice(pool.astype(dtype), size=shape)
    # row j of a plane: j mod 33 voxels of a plateau, then noise
    f = rng.random(shape).astype(dtype)
    x, y = np.arange(shape[2]) % 32, np.arange(shape[1]) % 33
    f[:, x[None, :] < y[:, None]] = 0.5
    return f


def _codes(f):
    """Steepest ranks on order-preserving integer keys."""
    b = f.view(np.int32 if f.dtype == np.float32 else np.int64)
    top = np.iinfo(b.dtype).max
    key = np.where(b < 0, -(b & top), b)
    lo, hi = np.iinfo(b.dtype).min, top
    asc = np.full(f.shape, 7)
    desc = np.full(f.shape, 7)
    up, down = np.full(f.shape, lo), np.full(f.shape, hi)
    nz, ny, nx = f.shape
    for r, (dz, dy, dx) in enumerate(OFFSETS):
        there = tuple(slice(max(0, -d), n - max(0, d)) for d, n in zip((dz, dy, dx), f.shape))
        from_ = tuple(slice(max(0, d), n - max(0, -d)) for d, n in zip((dz, dy, dx), f.shape))
        k = key[from_]
        asc[there] = np.where(k >= up[there], r, asc[there])
        up[there] = np.maximum(up[there], k)
        desc[there] = np.where(k < down[there], r, desc[there])
        down[there] = np.minimum(down[there], k)
    return (asc | (desc << 4)).astype(np.uint8)


SHAPES = [(1, 1, 40), (1, 2, 33), (9, 10, 34), (5, 17, 65), (12, 40, 100), (70, 40, 70)]
# thin fields, whose voxels are decided one by one, and the first that are not
THIN = [(1, 1, 1), (1, 1, 5000), (2, 1, 300), (700, 1, 33), (5, 900, 1), (3, 2, 65), (1, 4, 32), (1, 5, 32), (4, 3, 32), (1, 500, 17)]


@pytest.fixture(params=[None, 7, 64], ids=["depth-by-size", "depth-7", "depth-64"])
def depth(request):
    api().tune_clear()
    yield request.param
    api().tune_clear()


@pytest.mark.parametrize("shape", SHAPES + THIN, ids=str)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["ints", "ramp", "rows", "special"])
def test_codes(cuda, shape, dtype, kind, depth):
    f = _field(kind, shape, dtype)
    if depth:
        api().tune_set(shape, torch.from_numpy(f).dtype, depth, 1)
    got = api().codes(torch.from_numpy(f).to(cuda)).cpu().numpy()
    np.testing.assert_array_equal(got, _codes(f))


@pytest.mark.parametrize("shape", SHAPES + THIN, ids=str)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["ints", "ramp", "rows"])
def test_full_sweeps(cuda, shape, dtype, kind, depth):
    f = _field(kind, shape, dtype)
    eb = 1.0 if kind == "ints" else 1e-2
    rng = np.random.default_rng(3)
    fh = (f + rng.integers(-1, 2, size=shape) * dtype(eb)).astype(dtype)
    if depth:
        api().tune_set(shape, torch.from_numpy(f).dtype, depth, 1)
    ref, _, st, sw, recs = O.correct(f, fh, eb, max_sweeps=60)
    d = torch.from_numpy(fh).to(cuda)
    r = api().correct(torch.from_numpy(f).to(cuda), d, eb, max_sweeps=60, full_sweeps=True)
    assert (r.status, r.sweeps) == (st, sw)
    np.testing.assert_array_equal(r.log[:, :5], recs)
    assert (r.log[:, 6] == f.size).all()  # every sweep examines every voxel
    np.testing.assert_array_equal(d.cpu().numpy().view(np.uint8), ref.view(np.uint8))
