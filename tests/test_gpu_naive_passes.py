"""The passes of the naive strategy (csrc/naive.cu) where they can go wrong,
against the CPU oracle: limits that cut the passes enqueued together, more
changed voxels than a pass lists, fields of a voxel and of several spans, chains
of directions longer than the label walks.  Bits and whole numbers: equal, no
tolerance."""
import numpy as np
import pytest

from oracle import oracle as O
from pmsz_anonymous_gb300 import fields as F

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def api():
    from pmsz_anonymous_gb300 import api as A
    return A


def _check(device, f, fh, eb, **kw):
    ref, _, st, sw, recs = O.correct_naive(f, fh, eb, **kw)
    d = torch.from_numpy(np.ascontiguousarray(fh)).to(device)
    r = api().correct(torch.from_numpy(np.ascontiguousarray(f)).to(device), d, eb, strategy="naive", **kw)
    assert (r.status, r.sweeps) == (st, sw)
    np.testing.assert_array_equal(r.log[:, :5], recs)
    np.testing.assert_array_equal(d.cpu().numpy().view(np.uint8), ref.view(np.uint8))
    return r


@pytest.mark.parametrize("limit", [1, 2, 3, 4, 5, 6, 7, 9, 12, 300])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_limits(cuda, limit, dtype):
    f = F.perlin_field((20, 24, 40), 6, 4, 1 / 16, dtype=dtype)
    _check(cuda, f, F.standin(f, 2e-3, "zfp", 6), 2e-3, max_sweeps=limit)


# 16 voxels a thread and 4096 a block: one, less than a step, tails, several spans
@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 1, 13), (1, 3, 17), (2, 64, 33), (9, 31, 47), (40, 36, 44)], ids=str)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("noise", [0.0, 0.05, 1.0])
def test_changed_lists(cuda, shape, dtype, noise):
    # integers with noise in a share of the voxels: at 1.0 nearly every voxel is
    # a false extremum, far more than a 32nd of the field
    rng = np.random.default_rng(5)
    f = rng.integers(0, 9, size=shape).astype(dtype)
    step = (rng.integers(-3, 4, size=shape) * (rng.random(shape) < noise)).astype(dtype) / dtype(4)
    _check(cuda, f, (f + step).astype(dtype), 1.0, max_sweeps=60)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_long_chains(cuda, dtype):
    f = np.arange(6000, dtype=dtype).reshape(1, 1, -1)
    fh = f.copy()
    fh[0, 0, 100:5900:700] += dtype(1.25)  # false extrema, and labels that end in the wrong place
    fh[0, 0, 333:5900:900] -= dtype(0.75)
    _check(cuda, f, fh, 2.0, max_sweeps=400)
