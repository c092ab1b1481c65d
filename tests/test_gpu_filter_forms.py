"""Forms of the bound-filtered kernels against the oracle, bit for bit: device
batches at every tile width, packed columns whose high bits are set, and single
launches at the widest tiles."""
import re

import numpy as np
import pytest

import oracle as O
from test_gpu_batch_device import DeviceBatch, _check, _gen, _ragged
from wmh_testlib import device_logf, engine_gen, gamma_params, random_csr

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def force_filter(monkeypatch):
    monkeypatch.setenv("MHCUDA_B200_FILTER", "1")


@pytest.mark.parametrize("samples", [32, 64, 100, 128, 200, 256])
@pytest.mark.parametrize("skew", [0, 3])
def test_filtered_batches(samples, skew):
    """Ragged batches with matrices without rows and without entries, entered off
    the 16-byte grid too; the first call launches, the second captures, the third
    replays."""
    import minhashcuda_b200
    lib = minhashcuda_b200.capi()
    rng = np.random.default_rng(1000 + samples + skew)
    dim = 3000
    params = gamma_params(rng, dim, samples)
    co = O.COracle(*params)
    g = _gen(lib, dim, samples, params)
    try:
        mats = _ragged(rng, dim, 80)
        mats.append(random_csr(rng, 30, dim, 0))  # rows without entries
        mats.append(random_csr(rng, 3, dim, 2900))
        batch = DeviceBatch(mats, samples, skew=skew)
        for _ in range(3):
            assert batch.run(lib, g) == 0
            _check(co, mats, batch.results())
    finally:
        lib.mhcuda_fini(g)


@pytest.mark.parametrize("dim,samples", [(1 << 18, 100), ((1 << 20) + 12345, 32)])
@pytest.mark.parametrize("shift", [0, 6])
def test_packed_columns_over_the_whole_range(dim, samples, shift, monkeypatch):
    """4 and 8 high bits of packed columns that use all of them: in the windows,
    in the pieces' merge (rows over several chunks) and, with ln_c shifted above
    every guess, in the second scan of a row."""
    monkeypatch.setenv("MHCUDA_B200_PIPELINE_MIN_NNZ", "1")
    monkeypatch.setenv("MHCUDA_B200_BLOCK_NNZ", "20000")
    monkeypatch.setenv("MHCUDA_B200_CHUNK", "512")
    rng = np.random.default_rng(samples)
    m = random_csr(rng, 120, dim, 200, long_rows=[(0, 3000), (50, 700), (119, 9000)])
    assert m.indices.max() >> 16 == (dim - 1) >> 16 and len(np.unique(m.indices >> 16)) > 3
    with engine_gen(dim, samples, seed=5) as eng:
        table = eng.retrieve()
        if shift:
            table[1][...] += shift
            eng.assign(*table)
        out = eng.calc_csr(m)
    np.testing.assert_array_equal(out, O.COracle(*table).hash_csr(m, lnw=device_logf(m.data)))


@pytest.mark.parametrize("samples,rows", [(100, 5200), (128, 5200), (200, 2700), (256, 2700)])
def test_single_launches_at_the_widest_tiles(samples, rows, capfd, monkeypatch):
    """Enough entries per warp that tiles are not narrowed: s_pad compiled in (128,
    256) and not, one tile and two, long rows kept whole and cut."""
    rng = np.random.default_rng(samples)
    dim = 9000
    m = random_csr(rng, rows, dim, 1100, long_rows=[(3, 9000), (1700, 8000), (rows - 1, 9000)])
    params = gamma_params(rng, dim, samples)
    with engine_gen(dim, samples, deferred=True, verbosity=2) as eng:
        eng.assign(*params)
        capfd.readouterr()
        out = eng.calc_csr(m)
        assert re.search(r"plan: .* filter=(\d)", capfd.readouterr().out).group(1) == "8"
    np.testing.assert_array_equal(out, O.COracle(*params).hash_csr(m, lnw=device_logf(m.data)))
