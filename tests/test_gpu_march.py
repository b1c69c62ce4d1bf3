"""The full-field passes (csrc/march.cuh) at the sizes and values where they can
go wrong, against the CPU oracle: tile and column edges, both plane sources
(tensor copies and element copies), queues that overflow, ties, signed zeros,
denormals, infinities and values above the sentinel.  Codes, fields and
per-sweep counters are whole numbers or bits: equal, no tolerance."""
import numpy as np
import pytest

from oracle import oracle as O
from pmsz_anonymous_gb300 import fields as F

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def api():
    from pmsz_anonymous_gb300 import api as A
    return A


def _dev(a, device, shift=0):
    """A device copy that starts `shift` elements into its buffer (a shifted
    or ragged field has no tensor map and takes the element copies)."""
    flat = torch.from_numpy(np.ascontiguousarray(a)).ravel()
    buf = torch.empty(flat.numel() + shift, dtype=flat.dtype, device=device)
    buf[shift:] = flat.to(device)
    return buf[shift:].view(a.shape)


def _field(kind, shape, dtype, seed):
    rng = np.random.default_rng(seed)
    if kind == "perlin":
        return F.perlin_field(shape, seed, 4, 1 / 16, dtype=dtype)
    if kind == "plateaus":  # nearly every voxel ties: the exact queue overflows
        return rng.integers(0, 4, size=shape).astype(dtype)
    tiny = np.finfo(dtype).tiny
    pool = np.array([0.0, -0.0, tiny / 8, -tiny / 8, tiny, -tiny, 1.0, -1.0, np.inf, -np.inf,
                     2e30, -2e30, 1 + np.finfo(dtype).eps, np.finfo(dtype).max], dtype)
    return rng.choice(pool, size=shape)


def _targets(codes, shape, high):
    nz, ny, nx = shape
    off = api().rank_offsets()
    r = ((codes >> 4) if high else (codes & 15)).astype(np.int64).ravel()
    return np.arange(r.size) + off[r, 0] + nx * (off[r, 1] + ny * off[r, 2])


# one tile with its halo inside (34 x 10 x 6), one short of it, several tiles
# and columns, faces only, single rows / planes / columns
SHAPES = [(34, 10, 34), (6, 10, 36), (5, 9, 33), (3, 1, 65), (1, 17, 32), (70, 2, 1), (37, 25, 100)]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["perlin", "plateaus", "special"])
@pytest.mark.parametrize("shift", [0, 1])
def test_codes(cuda, shape, dtype, kind, shift):
    f = _field(kind, shape, dtype, 3)
    c = api().codes(_dev(f, cuda, shift)).cpu().numpy()
    asc, desc = O.label(f)
    np.testing.assert_array_equal(_targets(c, shape, 0), asc)
    np.testing.assert_array_equal(_targets(c, shape, 1), desc)


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("comp,eb", [("zfp", 1e-3), ("sz3", 3e-2), ("mixed", 0.5)])
@pytest.mark.parametrize("shift,full", [(0, False), (1, False), (0, True)])
def test_first_sweeps(cuda, shape, dtype, comp, eb, shift, full):
    f = _field("plateaus" if comp == "mixed" else "perlin", shape, dtype, 5)
    # integers against noise: every direction of fhat is wrong (the rule queue overflows)
    fh = F.standin(f, eb, "zfp" if comp == "mixed" else comp, 5)
    ref, _, st, sw, recs = O.correct(f, fh, eb, max_sweeps=3)
    df, dfh = _dev(f, cuda, shift), _dev(fh, cuda, shift)
    r = api().correct(df, dfh, eb, max_sweeps=3, full_sweeps=full)
    assert (r.status, r.sweeps) == (st, sw)
    np.testing.assert_array_equal(r.log[:, :5], recs)
    np.testing.assert_array_equal(dfh.cpu().numpy().view(np.uint8), ref.view(np.uint8))


@pytest.mark.parametrize("depth", [1, 3, 128, 200])
def test_column_depths(cuda, depth):
    shape, dtype, eb = (131, 12, 40), np.float32, 2e-3
    f = _field("perlin", shape, dtype, 7)
    fh = F.standin(f, eb, "sz3", 7)
    ref, _, st, sw, recs = O.correct(f, fh, eb)
    api().tune_set(shape, torch.float32, depth, 1)
    try:
        dfh = _dev(fh, cuda)
        r = api().correct(_dev(f, cuda), dfh, eb)
    finally:
        api().tune_clear()
    assert (r.status, r.sweeps) == (st, sw)
    np.testing.assert_array_equal(r.log[:, :5], recs)
    np.testing.assert_array_equal(dfh.cpu().numpy().view(np.uint8), ref.view(np.uint8))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("where", [(0, 0, 0), (19, 8, 31), (39, 16, 47)])
def test_bad_values_are_refused(cuda, dtype, where):
    from pmsz_anonymous_gb300 import capi
    f = _field("perlin", (40, 17, 48), dtype, 9)
    for bad in (np.nan, -np.nan) + ((1e30,) if dtype is np.float64 else ()):
        for target in (0, 1):
            pair = [f.copy(), f.copy()]
            pair[target][where] = bad
            with pytest.raises(capi.PmszError):
                api().correct(_dev(pair[0], cuda), _dev(pair[1], cuda), 1e-3)
