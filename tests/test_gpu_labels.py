"""Manifold labels (tile roots, exit walks, the general jumping) and the
verification counts at the sizes and chains where they can go wrong, against
the CPU oracle.  Whole numbers: equal, no tolerance."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O
from pmsz_anonymous_gb300 import capi, fields as F

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def api():
    from pmsz_anonymous_gb300 import api as A
    return A


def _dev(a, device):
    return torch.from_numpy(np.ascontiguousarray(a)).to(device)


def _snake(shape):
    """Values growing along one path that runs through every voxel of a plane
    at a time: the longest monotone chains a field can have."""
    nz, ny, nx = shape
    f = np.arange(nz * ny * nx, dtype=np.float64).reshape(shape)
    f[:, 1::2, :] = f[:, 1::2, ::-1].copy()
    return f


def _field(kind, shape):
    if kind == "perlin":
        return F.perlin_field(shape, 2, 4, 1 / 8, dtype=np.float64)
    if kind == "ramp":
        return np.arange(np.prod(shape), dtype=np.float64).reshape(shape)
    if kind == "snake":
        return _snake(shape)
    return np.random.default_rng(4).integers(0, 3, size=shape).astype(np.float64)


# one tile, one voxel more in every axis, tiles cut short, lines and planes
SHAPES = [(16, 16, 32), (17, 17, 33), (15, 31, 40), (1, 1, 5000), (3000, 1, 1), (2, 700, 3), (33, 48, 100), (1, 1, 1)]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("kind", ["perlin", "ramp", "snake", "plateaus"])
def test_labels(cuda, shape, kind):
    if kind == "perlin" and min(shape) == 1:
        pytest.skip("a constant noise field")
    f = _field(kind, shape)
    codes = api().codes(_dev(f, cuda))
    asc, desc = O.label(f)
    want = [np.asarray(O.path_compress(d)).ravel().astype(np.int64) for d in (asc, desc)]
    a, d = api().labels(codes)
    assert a.dtype == d.dtype == torch.int64
    np.testing.assert_array_equal(a.cpu().numpy().ravel(), want[0])
    np.testing.assert_array_equal(d.cpu().numpy().ravel(), want[1])
    # the 32-bit entry point, one kind at a time and both
    L, n = capi.load(), f.size
    nz, ny, nx = shape
    s = torch.cuda.current_stream().cuda_stream
    for ask in ((1, 0), (0, 1), (1, 1), (0, 0)):
        out = [torch.empty(n, dtype=torch.int32, device=cuda) for _ in range(2)]
        ptr = [o.data_ptr() if k else None for o, k in zip(out, ask)]
        capi.check(L.pmsz_labels(codes.data_ptr(), nx, ny, nz, ptr[0], ptr[1], ctypes.c_void_p(s)))
        for o, k, w in zip(out, ask, want):
            if k:
                np.testing.assert_array_equal(o.cpu().numpy().astype(np.int64), w)


def test_cycles_are_refused(cuda):
    # two voxels that name each other, inside one tile and across two: no
    # field has such codes, and no launch may wait for their end
    for x in (3, 31):
        codes = torch.full((4, 4, 64), 0x77, dtype=torch.uint8, device=cuda)
        codes[1, 1, x] = 0x78      # ascent to x + 1
        codes[1, 1, x + 1] = 0x76  # ascent to x - 1
        with pytest.raises(capi.PmszError):
            api().labels(codes)


@pytest.mark.parametrize("shape", [(17, 17, 33), (1, 1, 5000), (33, 48, 100)], ids=str)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["ramp", "plateaus", "snake"])
def test_verify(cuda, shape, dtype, kind):
    f = _field(kind, shape).astype(dtype)
    rng = np.random.default_rng(8)
    eb = 0.25
    # at the bound, one ulp inside and outside, far outside, not finite
    steps = np.array([0, eb, -eb, np.nextafter(dtype(eb), dtype(0)), np.nextafter(dtype(eb), dtype(1)), 3.0, -3.0], dtype)
    fp = (f + rng.choice(steps, size=shape)).astype(dtype)
    fp.ravel()[:: 97] = np.inf
    for bound in (eb, 0.0, -1.0):
        want = O.verify(f, fp, bound)
        want["bound_strict"] = want.pop("bound_violations")
        e = dtype(bound)
        want["bound_beyond_clamp"] = int((~((fp >= f - e) & (fp <= f + e))).sum())
        got = api().verify(_dev(f, cuda), _dev(fp, cuda), bound)
        assert got == want, (bound, got, want)


# nibbles of 15 name no neighbour: such a voxel is its own label, in the tiles as
# in the general jumping, however many of them a tile holds
@pytest.mark.parametrize("shape", [(16, 16, 32), (17, 33, 65), (40, 48, 70), (1, 1, 5000), (2, 1, 300)], ids=str)
@pytest.mark.parametrize("share", [1.0, 0.5, 0.01])
def test_nibbles_beyond_the_ranks_stay_put(cuda, shape, share):
    n = int(np.prod(shape))
    rng = np.random.default_rng(17)
    codes = api().codes(_dev(_field("ramp", shape), cuda)).cpu().numpy().ravel()
    off = api().rank_offsets()
    nx, ny = shape[2], shape[1]
    flat = off[:, 0] + nx * (off[:, 1] + ny * off[:, 2])
    nibbles = [codes & 15, codes >> 4]
    want = []
    for k in range(2):
        hit = rng.random(n) < share
        nibbles[k] = np.where(hit, 15, nibbles[k]).astype(np.uint8)
        p = np.arange(n) + np.where(hit, 0, flat[np.minimum(nibbles[k], 14)])
        while not np.array_equal(p, p[p]):
            p = p[p]
        want.append(p)
    both = _dev((nibbles[0] | (nibbles[1] << 4)).astype(np.uint8).reshape(shape), cuda)
    a, d = api().labels(both)
    np.testing.assert_array_equal(a.cpu().numpy().ravel(), want[0])
    np.testing.assert_array_equal(d.cpu().numpy().ravel(), want[1])


def _ridge(shape, sign):
    """A line of voxels that rises (falls) along x for longer than the exit walks
    go, in a field whose other chains are short: long chains of one kind only."""
    rng = np.random.default_rng(21)
    f = rng.random(shape)
    f[shape[0] // 2, shape[1] // 2, :] = 10 + np.arange(shape[2]) * 0.01
    return sign * f


@pytest.mark.parametrize("shape", [(8, 9, 3000), (20, 33, 1500), (2, 3, 4000)], ids=str)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["up", "down", "ramp", "noise"])
def test_verify_of_long_chains(cuda, shape, dtype, kind):
    f = {"up": lambda: _ridge(shape, 1), "down": lambda: _ridge(shape, -1), "ramp": lambda: _field("ramp", shape),
         "noise": lambda: np.random.default_rng(5).random(shape)}[kind]().astype(dtype)
    rng = np.random.default_rng(9)
    for change in ("some", "ridge"):
        fp = f.copy()
        if change == "some":
            fp += (rng.random(shape) < 0.01) * dtype(0.5)
        else:  # only the line itself: every chain that follows it is cut
            fp[shape[0] // 2, shape[1] // 2, shape[2] // 3] += dtype(3 if kind != "down" else -3)
        want = O.verify(f, fp, 0.25)
        want["bound_strict"] = want.pop("bound_violations")
        want["bound_beyond_clamp"] = int((~((fp >= f - dtype(0.25)) & (fp <= f + dtype(0.25)))).sum())
        assert api().verify(_dev(f, cuda), _dev(fp, cuda), 0.25) == want
