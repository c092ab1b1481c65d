"""The bound-filtered hash kernels against the oracle, bit for bit.

The filter is forced on (MHCUDA_B200_FILTER=1) so that small matrices reach
it; hashes must equal the oracle's on every form the dense kernels take: tile
edges of the sample count, rows around window and batch sizes, weights of
every class, and parameter tables the bounds were not made for.
"""
import numpy as np
import pytest
import scipy.sparse as sp

import oracle as O
from wmh_testlib import device_logf, engine_gen, gamma_params, random_csr

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def force_filter(monkeypatch):
    monkeypatch.setenv("MHCUDA_B200_FILTER", "1")


def check(m, samples, params):
    with engine_gen(m.shape[1], samples, deferred=True) as eng:
        eng.assign(*params)
        out = eng.calc_csr(m)
    want = O.COracle(*params).hash_csr(m, lnw=device_logf(m.data))
    np.testing.assert_array_equal(out, want)


def edge_rows(rng, dim, scale=1):
    """Rows of 0, 1 and of lengths around 32, 64, 128 and 256 entries, shuffled
    between runs of empty rows."""
    lens = [0, 0, 1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 900, 0] * scale
    lens = rng.permutation(lens)
    return random_csr(rng, len(lens), dim, 0, long_rows=list(enumerate(lens)))


@pytest.mark.parametrize("samples", [32, 33, 48, 63, 64, 65, 100, 127, 128, 129, 200, 255, 256, 300])
def test_sample_tiles_and_row_edges(samples):
    rng = np.random.default_rng(samples)
    dim = 3000
    check(edge_rows(rng, dim, 3), samples, gamma_params(rng, dim, samples))


@pytest.mark.parametrize("values", ["classes", "tiny", "huge", "wide"])
def test_weight_classes(values):
    rng = np.random.default_rng(len(values))
    dim, samples = 2000, 128
    m = edge_rows(rng, dim, 4)
    d = m.data.copy()
    if values == "classes":
        for v, p in ((-1.0, 0.1), (0.0, 0.1), (np.nan, 0.05), (np.inf, 0.02), (1e-42, 0.1)):
            d[rng.random(d.size) < p] = v
    elif values == "tiny":
        d[:] = np.float32(1e-38) * rng.random(d.size).astype(np.float32)
    elif values == "huge":
        d[:] = np.float32(3e38) * rng.random(d.size).astype(np.float32)  # sums overflow
    else:  # 60 orders of magnitude inside a row
        d[:] = (10.0 ** rng.uniform(-37, 37, d.size)).astype(np.float32)
    check(sp.csr_matrix((d, m.indices, m.indptr), shape=m.shape), samples,
          gamma_params(rng, dim, samples))


@pytest.mark.parametrize("table", ["shift_up", "shift_down", "odd", "equal", "large"])
def test_assigned_tables(table):
    """shift_up: every minimum lies above the guess (rescans); shift_down and
    odd: bytes at the ends of their range; equal: ties everywhere; large: all
    parameters outside the range the bounds cover."""
    rng = np.random.default_rng(len(table))
    dim, samples = 1500, 128
    rs, lc, b = gamma_params(rng, dim, samples)
    if table == "shift_up":
        lc += 6
    elif table == "shift_down":
        lc -= 11
    elif table == "odd":
        pick = rng.random(rs.shape)
        rs[pick < 0.02] = 0.0
        rs[(pick >= 0.02) & (pick < 0.04)] = -1.5
        rs[(pick >= 0.04) & (pick < 0.05)] = np.nan
        rs[(pick >= 0.05) & (pick < 0.06)] = 1e-30
        lc[(pick >= 0.06) & (pick < 0.07)] = 90.0
        b[(pick >= 0.07) & (pick < 0.08)] = -40.0
    elif table == "equal":
        rs[:], lc[:], b[:] = 1.25, 0.5, 0.375
    else:
        rs *= 100
    check(edge_rows(rng, dim, 3), samples, (rs, lc, b))


@pytest.mark.parametrize("samples", [64, 128])
def test_rows_over_many_chunks(samples, monkeypatch):
    """Rows cut into pieces, chunks that begin at rows and chunks that cannot."""
    rng = np.random.default_rng(3)
    dim = 30000
    m = random_csr(rng, 60, dim, 20, long_rows=[(0, 20000), (9, 700), (10, 650), (59, 9000)])
    params = gamma_params(rng, dim, samples)
    for chunk in ("64", "512", "4096"):
        monkeypatch.setenv("MHCUDA_B200_CHUNK", chunk)
        check(m, samples, params)


@pytest.mark.parametrize("dim", [900, 1 << 21])
def test_packed_columns_and_batches(dim, monkeypatch):
    """The copy pipeline's packed columns (4 and 8 high bits), and batches."""
    rng = np.random.default_rng(7)
    samples = 128
    params = gamma_params(rng, min(dim, 900), samples)
    m = edge_rows(rng, 900, 2)
    with engine_gen(dim, samples, seed=5) as eng:
        want = eng.calc_csr(m)
        monkeypatch.setenv("MHCUDA_B200_PIPELINE_MIN_NNZ", "1")
        monkeypatch.setenv("MHCUDA_B200_BLOCK_NNZ", "1000")
        np.testing.assert_array_equal(eng.calc_csr(m), want)
        monkeypatch.setenv("MHCUDA_B200_FILTER", "0")
        np.testing.assert_array_equal(eng.calc_csr(m), want)
    if dim == 900:
        check(m, samples, params)


@pytest.mark.parametrize("samples", [100, 128, 200])
def test_full_width_tiles(samples):
    """Enough entries per warp for the widest tiles (smaller inputs get
    narrower ones), long rows kept whole and cut."""
    rng = np.random.default_rng(samples)
    dim = 9000
    m = random_csr(rng, 4400, dim, 1100, long_rows=[(3, 9000), (1700, 8000), (4399, 9000)])
    check(m, samples, gamma_params(rng, dim, samples))
