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


# NaNs of every kind of payload: quiet and signalling, either sign, the payload
# in the high or (fp64) the low word only, where the high word is an infinity's
NAN_BITS = {np.float64: [0x7FF8000000000000, 0xFFF8000000000000, 0x7FF0000000000001, 0xFFF0000000000001,
                         0x7FF00000FFFFFFFF, 0xFFF00000FFFFFFFF, 0xFFFFFFFFFFFFFFFF],
            np.float32: [0x7FC00000, 0xFFC00000, 0x7F800001, 0xFF800001, 0xFFFFFFFF]}


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("target", [0, 1], ids=["f", "fhat"])
@pytest.mark.parametrize("shape,where", [((40, 17, 48), (20, 8, 23)), ((40, 17, 48), (0, 0, 0)),
                                         ((19, 21, 37), (18, 20, 36))], ids=str)
def test_nans_of_every_payload_are_refused(cuda, shape, where, target, dtype):
    from pmsz_anonymous_gb300 import capi
    A = api()
    base = np.random.default_rng(6).random(shape).astype(dtype)
    for bits in NAN_BITS[dtype]:
        pair = [base.copy(), base.copy()]
        pair[target].view(np.uint32 if dtype is np.float32 else np.uint64)[where] = bits
        assert np.isnan(pair[target][where])
        dev = [torch.from_numpy(a).to(cuda) for a in pair]
        for full in (False, True):
            with pytest.raises(capi.PmszError):
                A.correct(dev[0], dev[1].clone(), 1e-3, max_sweeps=40, full_sweeps=full)
        with pytest.raises(capi.PmszError):
            A.correct_host(*[torch.from_numpy(a).pin_memory() for a in pair], 1e-3, max_sweeps=40)
        good = torch.from_numpy(base).to(cuda)
        got = A.correct_batch([(dev[0], dev[1].clone(), 1e-3), (good, good.clone(), 1e-3)], max_sweeps=40)
        assert [r.status for r in got] == [capi.PMSZ_ERR_ARG, capi.PMSZ_OK], hex(bits)
        work = dev[1].clone()
        torch.cuda.synchronize()
        with A.Server(max_sweeps=40) as srv:
            assert srv.wait(srv.submit(dev[0], work, 1e-3))["status"] == capi.PMSZ_ERR_ARG, hex(bits)


# beyond the sentinel (1e30) and down to the lowest values nothing is special: such
# fields take the ordinary path, and a NaN or a sentinel among them is found
@pytest.mark.parametrize("shape", [(34, 10, 34), (5, 9, 33), (37, 25, 100)], ids=str)
@pytest.mark.parametrize("dtype,scale", [(np.float64, s) for s in (1e30, 1e35, -1e35, 1e308, -1e308)] +
                         [(np.float32, s) for s in (1e35, -1e35, 3e38, -3e38)], ids=str)
def test_huge_values(cuda, shape, dtype, scale):
    from pmsz_anonymous_gb300 import capi
    rng = np.random.default_rng(shape[0])
    f = (rng.random(shape) * 0.5 + 0.25) * scale  # (|scale| itself does not occur)
    eb = abs(scale) * 1e-2 if abs(scale) < 1e300 else 9e299
    f = f.astype(dtype)
    fh = (f + rng.uniform(-1, 1, shape) * eb * 0.9).astype(dtype)
    ref, _, st, sw, recs = O.correct(f, fh, eb, max_sweeps=40)
    for full in (False, True):
        d = torch.from_numpy(fh).to(cuda)
        r = api().correct(torch.from_numpy(f).to(cuda), d, eb, max_sweeps=40, full_sweeps=full)
        assert (r.status, r.sweeps) == (st, sw)
        np.testing.assert_array_equal(r.log[:, :5], recs)
        np.testing.assert_array_equal(d.cpu().numpy().view(np.uint8), ref.view(np.uint8))
    at = tuple(s // 2 for s in shape)
    for bad in [np.nan, -np.nan] + ([1e30] if dtype is np.float64 else []):
        for k in range(2):
            pair = [f.copy(), fh.copy()]
            pair[k][at] = bad
            with pytest.raises(capi.PmszError):
                api().correct(*[torch.from_numpy(a).to(cuda) for a in pair], eb, max_sweeps=40)
