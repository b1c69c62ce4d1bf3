"""Corrections of fields of special values (csrc/march.cuh, csrc/sweep.cuh): signed
zeros, denormals, infinities and the largest numbers, where comparing values
and comparing keys could part, against the CPU oracle.  Bits and whole numbers:
equal, no tolerance."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def api():
    from pmsz_anonymous_gb300 import api as A
    return A


def _pool(kind, dtype):
    tiny, big = np.finfo(dtype).tiny, np.finfo(dtype).max
    return {"zeros": [0.0, -0.0, tiny / 8, -tiny / 8],
            "small": [0.0, -0.0, tiny / 8, -tiny / 8, tiny / 4, tiny, -tiny],
            "large": [0.0, -0.0, 1.0, big, -big, np.inf, -np.inf, 1e29]}[kind]


@pytest.mark.parametrize("shape", [(34, 10, 34), (5, 9, 33), (1, 17, 32), (37, 25, 100)], ids=str)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["zeros", "small", "large"])
def test_special(cuda, shape, dtype, kind):
    rng = np.random.default_rng(len(kind) + shape[0])
    pool = np.array(_pool(kind, dtype), dtype)
    f = rng.choice(pool, size=shape)
    fh = np.where(rng.random(shape) < 0.3, rng.choice(pool, size=shape), f).astype(dtype)
    eb = float(np.finfo(dtype).tiny) if kind != "large" else 0.5
    ref, _, st, sw, recs = O.correct(f, fh, eb, max_sweeps=40)
    for full in (False, True):
        d = torch.from_numpy(fh).to(cuda)
        r = api().correct(torch.from_numpy(f).to(cuda), d, eb, max_sweeps=40, full_sweeps=full)
        assert (r.status, r.sweeps) == (st, sw)
        np.testing.assert_array_equal(r.log[:, :5], recs)
        np.testing.assert_array_equal(d.cpu().numpy().view(np.uint8), ref.view(np.uint8))
