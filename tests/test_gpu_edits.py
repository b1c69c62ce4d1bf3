"""Edit extraction without counters and the symbol pass of the reconstruction
(csrc/edits.cu) at tile edges, tails and unaligned symbol arrays, and the
verification of fields whose directions agree in one kind only, against the
CPU oracle.  Whole numbers and bits: equal, no tolerance."""
import numpy as np
import pytest

from oracle import oracle as O
from pmsz_anonymous_gb300 import capi

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def api():
    from pmsz_anonymous_gb300 import api as A
    return A


def _dev(a, device):
    return torch.from_numpy(np.ascontiguousarray(a)).to(device)


def _triple(n, dtype, share, seed):
    """prev, cur, f with about `share` of the voxels edited: steps, clamps, zeros."""
    rng = np.random.default_rng(seed)
    eb, q = 0.125, 5
    f = rng.integers(-8, 9, size=n).astype(dtype) / dtype(8)  # f - eb is exact, and 0 for some
    prev = (f + rng.integers(-1, 2, size=n).astype(dtype) * dtype(eb / 2)).astype(dtype)
    kind = np.where(rng.random(n) < share, rng.integers(1, 6, size=n), 0)
    step = dtype(eb / q)
    cur = prev.copy()
    for k in range(1, 5):
        cur = np.where(kind == k, (prev - dtype(k) * step).astype(dtype), cur)
    cur = np.where(kind == 5, (f - dtype(eb)).astype(dtype), cur).astype(dtype)
    return prev, cur, f, eb, q


@pytest.mark.parametrize("n", [1, 31, 255, 256, 2047, 2048, 2049, 4096 + 33, 3 * 2048 - 7, 70001])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("share", [0.0, 0.02, 1.0])
def test_extract_and_rebuild(cuda, n, dtype, share):
    prev, cur, f, eb, q = _triple(n, dtype, share, n)
    d, cl, edits = O.extract_edits(prev, cur, f, eb, q)
    A = api()
    gd, gc, ge = A.extract_edits(_dev(prev, cuda), _dev(cur, cuda), _dev(f, cuda), eb, q=q)
    np.testing.assert_array_equal(gd.cpu().numpy(), d)
    np.testing.assert_array_equal(gc.cpu().numpy().view(np.uint8), cl.view(np.uint8))
    assert ge == edits
    if not np.count_nonzero(d == q) == cl.size:  # a clamp value of 0 leaves the list: not to be rebuilt
        with pytest.raises(capi.PmszError):
            A.reconstruct(_dev(prev, cuda), gd, gc, eb, q=q)
        return
    want = O.reconstruct(prev, d, cl, eb, q)
    for shift in (0, 1, 8):  # symbols off a 16-byte boundary
        buf = torch.empty(n + shift, dtype=torch.uint8, device=cuda)
        buf[shift:] = gd
        out = A.reconstruct(_dev(prev, cuda), buf[shift:], gc, eb, q=q)
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint8), want.view(np.uint8))


@pytest.mark.parametrize("q", [1, 5, 127, 255])
def test_symbols_above_q(cuda, q):
    n = 2 * 2048 + 77
    rng = np.random.default_rng(q)
    prev = rng.standard_normal(n)
    d = rng.integers(0, q + 1, size=n).astype(np.uint8)
    cl = rng.standard_normal(np.count_nonzero(d == q))
    A = api()
    got = A.reconstruct(_dev(prev, cuda), _dev(d, cuda), _dev(cl, cuda), 0.5, q=q)
    np.testing.assert_array_equal(got.cpu().numpy(), O.reconstruct(prev, d, cl, 0.5, q))
    for at in (0, 2047, 2048, n - 1) if q < 255 else ():
        e = d.copy()
        e[at] = q + 1
        with pytest.raises(capi.PmszError):
            A.reconstruct(_dev(prev, cuda), _dev(e, cuda), _dev(cl, cuda), 0.5, q=q)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("change", ["none", "ascent", "descent", "both"])
def test_verify_one_kind(cuda, dtype, change):
    # a ramp along x; raising or lowering the end of a row moves one kind of
    # chain end to the voxel before it, and every label of that row with it
    f = np.broadcast_to(np.arange(40, dtype=dtype), (3, 5, 40)).copy()
    f += (np.arange(5, dtype=dtype) * dtype(100))[None, :, None] + (np.arange(3, dtype=dtype) * dtype(1000))[:, None, None]
    fp = f.copy()
    if change in ("ascent", "both"):
        fp[2, 4, 39] = fp[2, 4, 38] - dtype(0.5)
    if change in ("descent", "both"):
        fp[0, 0, 0] = fp[0, 0, 1] + dtype(0.5)
    want = O.verify(f, fp, 4.0)
    assert (want["as_mismatch"] > 0) == (change in ("ascent", "both"))
    assert (want["ds_mismatch"] > 0) == (change in ("descent", "both"))
    got = api().verify(_dev(f, cuda), _dev(fp, cuda), 4.0)
    for k in ("dir_mismatch", "ext_mismatch", "as_mismatch", "ds_mismatch"):
        assert got[k] == want[k], k
