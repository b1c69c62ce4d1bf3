"""The server's worker where a CUDA call fails (csrc/server.cu over a fake of the
runtime, no GPU): the running jobs end with that error, once nothing of theirs is
in flight, their budget and scratch are given back, and the jobs behind them run;
a worker that cannot start refuses jobs instead of leaving them waiting."""
import os
import subprocess

import pytest

from pmsz_anonymous_gb300 import _build, capi

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    _build.build()
    out = str(tmp_path_factory.mktemp("native") / "server_failures")
    native = os.path.join(HERE, "native")
    r = subprocess.run([_build.nvcc(), *_build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-cudart", "none",
                        f"-I{_build.INCLUDE}", os.path.join(native, "server_failures.cu"),
                        os.path.join(native, "fake_runtime.cpp"), os.path.join(_build.BUILD, "server.cu.o"), "-o", out],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


def _run(program, scenario):
    r = subprocess.run([program, scenario], capture_output=True, text=True, timeout=60)
    lines = [line.split() for line in r.stdout.splitlines()]
    jobs = [dict(zip(w[2::2], map(int, w[3::2]))) for w in lines if w[0] == "job"]
    left = [int(w[1]) for w in lines if w[0] == "left"]
    return r.returncode, jobs, left


OK = {"submit": 0, "done": 1, "status": capi.PMSZ_OK, "in_flight": 0}


@pytest.mark.parametrize("scenario,status", [("none", capi.PMSZ_OK), ("sweeps", capi.PMSZ_ERR_CUDA),
                                             ("buffers", capi.PMSZ_ERR_CUDA), ("scratch", capi.PMSZ_ERR_OOM)])
def test_a_failed_generation(program, scenario, status):
    rc, jobs, left = _run(program, scenario)
    assert jobs == [dict(OK, status=status), OK, OK]
    assert rc == 0 and left == [0]


def test_a_worker_that_cannot_start(program):
    rc, jobs, left = _run(program, "setup")
    assert rc == 0 and left == [0] and len(jobs) == 3
    for j in jobs:  # refused, or (submitted before the worker gave up) failed
        assert (j["submit"], j["done"], j["status"]) in [(capi.PMSZ_ERR_CUDA, 0, -1), (0, 1, capi.PMSZ_ERR_CUDA)]
    assert jobs[2]["submit"] == capi.PMSZ_ERR_CUDA
