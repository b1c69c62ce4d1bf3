"""Fields a few rows or planes thick: labels by tiles and by the general jumping
(csrc/verify.cu takes lines and fields of fewer than four rows a tile to the
latter), corrections and verification of them, against the CPU oracle; steps out
of the domain, which no field's codes hold, stay inside the arrays.  Whole
numbers and bits: equal."""
import numpy as np
import pytest

from oracle import oracle as O
from pmsz_anonymous_gb300 import fields as F

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SHAPES = [(1, 1, 3000), (1, 3, 900), (3, 1, 700), (1, 4, 500), (2, 2, 333), (1, 90, 77), (2, 40, 65), (200, 1, 40),
          (300, 1, 1), (1, 500, 1)]


def _dev(a, device):
    return torch.from_numpy(np.ascontiguousarray(a)).to(device)


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("kind", ["perlin", "ramp"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_thin(cuda, shape, kind, dtype):
    from pmsz_anonymous_gb300 import api as A
    f = F.perlin_field(shape, 4, 4, 1 / 16, dtype=dtype) if kind == "perlin" else np.arange(
        np.prod(shape), dtype=dtype).reshape(shape) / dtype(64)
    eb = 1e-2
    fh = F.standin(f, eb, "zfp", 4)
    asc, desc = O.label(f)
    a, d = A.labels(A.codes(_dev(f, cuda)))
    np.testing.assert_array_equal(a.cpu().numpy().ravel(), O.path_compress(asc))
    np.testing.assert_array_equal(d.cpu().numpy().ravel(), O.path_compress(desc))
    got, want = A.verify(_dev(f, cuda), _dev(fh, cuda), eb), O.verify(f, fh, eb)
    for k in ("dir_mismatch", "ext_mismatch", "as_mismatch", "ds_mismatch"):
        assert got[k] == want[k], k
    ref, _, st, sw, recs = O.correct(f, fh, eb, max_sweeps=300)
    w = _dev(fh, cuda)
    r = A.correct(_dev(f, cuda), w, eb, max_sweeps=300)
    assert (r.status, r.sweeps) == (st, sw)
    np.testing.assert_array_equal(r.log[:, :5], recs)
    np.testing.assert_array_equal(w.cpu().numpy().view(np.uint8), ref.view(np.uint8))


@pytest.mark.parametrize("shape", [(1, 1, 64), (1, 4, 64)], ids=str)
def test_steps_out_of_the_domain_stay_put(cuda, shape):
    from pmsz_anonymous_gb300 import api as A
    codes = torch.full(shape, 0x77, dtype=torch.uint8, device=cuda)
    codes[0, 0, 0] = 0x70   # ascent to (x - 1, y - 1, z - 1)
    codes[0, 0, 63] = 0xE7  # descent to (x + 1, y + 1, z + 1)
    a, d = A.labels(codes)
    n = codes.numel()
    assert torch.equal(a.ravel().cpu(), torch.arange(n)) and torch.equal(d.ravel().cpu(), torch.arange(n))
