"""The sweeps behind the host copy (k_sweep_wave in csrc/sweep.cuh): fields of
several copy slabs whose planes begin inside a group of bitmap words, sparse and
dense, with ties, and limits on the sweeps below and above the wavefront's, against the correction of the same field on the device.  Bits and
whole numbers: equal, no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _pair(A, kind, shape, dtype, device):
    if kind == "plateaus":
        gen = torch.Generator(device=device).manual_seed(3)
        f = torch.randint(0, 5, shape, generator=gen, device=device).to(dtype)
        return f, f + torch.randint(-1, 2, shape, generator=gen, device=device).to(dtype), 1.0
    eb = {"sparse": 1e-4, "dense": 1e-2}[kind]
    f = A.gen_perlin(shape, 9, 4, 1 / 32, 0.5, dtype=dtype, device=device)
    return f, A.standin(f, eb, "zfp", 9), eb


@pytest.mark.parametrize("shape,dtype", [((131, 173, 211), torch.float64), ((262, 150, 237), torch.float32),
                                         ((700, 33, 257), torch.float64), ((2, 1500, 2100), torch.float64)], ids=str)
@pytest.mark.parametrize("kind", ["sparse", "dense", "plateaus"])
@pytest.mark.parametrize("limit", [1, 2, 5, 8, 400])
def test_waves(cuda, shape, dtype, kind, limit):
    from pmsz_anonymous_gb300 import api as A
    f, fh, eb = _pair(A, kind, shape, dtype, cuda)
    want = fh.clone()
    ref = A.correct(f, want, eb, max_sweeps=limit)
    hf, hfh = f.cpu().pin_memory(), fh.cpu().pin_memory()
    got, _ = A.correct_host(hf, hfh, eb, max_sweeps=limit)
    assert (got.status, got.sweeps) == (ref.status, ref.sweeps)
    np.testing.assert_array_equal(got.log, ref.log)
    bits = torch.int64 if dtype == torch.float64 else torch.int32
    assert torch.equal(hfh.view(bits), want.cpu().view(bits))
