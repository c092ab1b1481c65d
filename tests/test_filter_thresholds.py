"""The filter kernels' threshold arithmetic at the ends of its range: compiled
for the CPU from the header the kernels use, and on the GPU an infinite weight
beside minima far below the bytes' range."""
import os
import shutil
import subprocess

import numpy as np
import pytest
import scipy.sparse as sp

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.mark.skipif(shutil.which("g++") is None or
                    not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")),
                    reason="needs g++ and the CUDA headers")
def test_threshold_arithmetic(tmp_path):
    exe = tmp_path / "check"
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "minhashcuda_b200", "csrc"),
                           "-I", CUDA_INCLUDE, os.path.join(ROOT, "tests", "filter_threshold_check.cc"),
                           "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("low", ["ln_c", "r"])
def test_infinite_weight_below_the_range(low, monkeypatch):
    """The row's first half has values near -500 for every sample, evaluated
    before the infinite weights of its second half are scanned; bytes there are
    the generator's, a part of them 240 and more.  The first infinite weight
    wins for every sample, as in the dense kernel."""
    import oracle as O
    from wmh_testlib import device_logf, engine_gen, gamma_params

    monkeypatch.setenv("MHCUDA_B200_FILTER", "1")
    monkeypatch.setenv("MHCUDA_B200_CHUNK", "4096")  # the rows whole: a piece starts its search anew
    rng = np.random.default_rng(3)
    dim, samples, rows = 700, 128, 4
    rs, lc, b = gamma_params(rng, dim, samples)
    if low == "ln_c":
        lc[:, :350] = -500.0
    else:
        rs[:, :350], b[:, :350] = 500.0, 0.0
    lc[:, 350:] += 2.0  # more bytes of 240 and above
    data = rng.lognormal(0.0, 1.0, (rows, dim)).astype(np.float32)
    data[:, 500::40] = np.inf
    m = sp.csr_matrix((data.ravel(), np.tile(np.arange(dim, dtype=np.int32), rows),
                       np.arange(rows + 1) * dim), shape=(rows, dim))
    with engine_gen(dim, samples, deferred=True) as eng:
        eng.assign(rs, lc, b)
        out = eng.calc_csr(m)
    want = O.COracle(rs, lc, b).hash_csr(m, lnw=device_logf(m.data))
    assert (want[..., 0] == 500).all()
    np.testing.assert_array_equal(out, want)
