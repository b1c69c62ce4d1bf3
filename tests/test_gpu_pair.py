"""The two-field pass of the verification (csrc/march.cuh) by tensor copies and by
element copies, with ties, infinities and NaN, against the direction codes and
labels of each field by itself and the bound on the CPU.  Whole numbers: equal."""
import numpy as np
import pytest

from pmsz_anonymous_gb300 import fields as F

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _dev(a, device, shift):
    flat = torch.from_numpy(np.ascontiguousarray(a)).ravel()
    buf = torch.empty(flat.numel() + shift, dtype=flat.dtype, device=device)
    buf[shift:] = flat.to(device)
    return buf[shift:].view(a.shape)


@pytest.mark.parametrize("shape", [(70, 26, 100), (37, 25, 101), (3, 1, 65), (1, 17, 32)], ids=str)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["perlin", "plateaus", "special"])
@pytest.mark.parametrize("shift", [0, 1])
def test_pair(cuda, shape, dtype, kind, shift):
    from pmsz_anonymous_gb300 import api as A
    rng = np.random.default_rng(12)
    if kind == "perlin":
        f = F.perlin_field(shape, 2, 4, 1 / 16, dtype=dtype)
        fp = F.standin(f, 1e-3, "zfp", 2)
        eb = 5e-4
    else:
        f = rng.integers(0, 4, size=shape).astype(dtype)
        fp = np.where(rng.random(shape) < 0.2, f + rng.integers(-1, 2, size=shape), f).astype(dtype)
        eb = 0.5
        if kind == "special":
            for v in (np.inf, -np.inf, np.nan, -0.0, np.finfo(dtype).max):
                f = np.where(rng.random(shape) < 0.02, dtype(v), f)
                fp = np.where(rng.random(shape) < 0.02, dtype(v), fp)
    df, dp = _dev(f, cuda, shift), _dev(fp, cuda, shift)
    c0, c1 = A.codes(df), A.codes(dp)
    k0, k1 = c0.cpu().numpy(), c1.cpu().numpy()
    self_, e = 7, dtype(eb)
    with np.errstate(all="ignore"):
        want = {"dir_mismatch": int((k0 != k1).sum()),
                "ext_mismatch": int(((((k0 & 15) == self_) != ((k1 & 15) == self_)) |
                                     (((k0 >> 4) == self_) != ((k1 >> 4) == self_))).sum()),
                "bound_strict": int((~(np.abs(fp - f) <= e)).sum()),
                "bound_beyond_clamp": int((~((fp >= f - e) & (fp <= f + e))).sum())}
    l0, l1 = A.labels(c0), A.labels(c1)
    want["as_mismatch"] = int((l0[0] != l1[0]).sum())
    want["ds_mismatch"] = int((l0[1] != l1[1]).sum())
    assert A.verify(df, dp, eb) == want
