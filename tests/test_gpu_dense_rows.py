"""The dense hash kernels' ends of rows against the oracle, bit for bit: t kept
with the minimum (short rows, tiny launches) or recomputed, rows that cross
chunks, and the shortest chunks."""
import numpy as np
import pytest

import oracle as O
from wmh_testlib import device_logf, engine_gen, gamma_params, random_csr

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def no_filter(monkeypatch):
    monkeypatch.setenv("MHCUDA_B200_FILTER", "0")


def check(m, samples, params):
    with engine_gen(m.shape[1], samples, deferred=True) as eng:
        eng.assign(*params)
        out = eng.calc_csr(m)
    want = O.COracle(*params).hash_csr(m, lnw=device_logf(m.data))
    np.testing.assert_array_equal(out, want)


@pytest.mark.parametrize("samples", [16, 80, 64, 100, 128, 256])
@pytest.mark.parametrize("mean", [5, 40, 700])
def test_short_and_long_rows(samples, mean):
    """Both sides of the rule that keeps t, one, two and four samples a lane."""
    rng = np.random.default_rng(samples + mean)
    dim = 3000
    m = random_csr(rng, 700_000 // (mean + 20), dim, mean, empty_frac=0.02, zero_frac=0.05)
    check(m, samples, gamma_params(rng, dim, samples))


@pytest.mark.parametrize("rows,mean", [(1, 1), (1, 7), (1, 8), (1, 9), (1, 300), (3, 65), (40, 60)])
def test_tiny_launches(rows, mean):
    """Chunks of 8 entries and rows over many of them."""
    rng = np.random.default_rng(rows * 1000 + mean)
    dim = 900
    m = random_csr(rng, rows, dim, 0, long_rows=[(r, mean + r) for r in range(rows)])
    check(m, 128, gamma_params(rng, dim, 128))


def test_packed_columns(monkeypatch):
    """The copy pipeline's packed columns with t kept."""
    rng = np.random.default_rng(1)
    dim = 5000
    monkeypatch.setenv("MHCUDA_B200_PIPELINE_MIN_NNZ", "1")
    monkeypatch.setenv("MHCUDA_B200_BLOCK_NNZ", "3000")
    m = random_csr(rng, 900, dim, 23, long_rows=[(100, 2500)])
    check(m, 128, gamma_params(rng, dim, 128))
