"""Which parameter tables take the bound-filtered kernel by themselves: those of
a generator's distribution, whatever their size; assigned tables of others go to
the dense kernel, which is many times faster on them."""
import re

import numpy as np
import pytest

from wmh_testlib import engine_gen, gamma_params

pytestmark = pytest.mark.gpu


def planned_filter(eng, capfd):
    """Lanes of the filtered kernel in the plan of a call that is large and
    whose rows are long enough for it; 0 for the dense kernel."""
    rng = np.random.default_rng(1)
    rows, length = 1200, 400
    n = rows * length
    capfd.readouterr()
    eng.calc(rng.lognormal(0.0, 1.0, n), rng.integers(0, eng.dim, n),
             np.arange(rows + 1, dtype=np.uint64) * length)
    return int(re.search(r"plan: .*filter=(\d+)", capfd.readouterr().out).group(1))


@pytest.mark.parametrize("dim,samples", [(8, 100), (130, 128), (2001, 65), (5000, 128)])
def test_tables_of_a_generator(dim, samples, capfd):
    with engine_gen(dim, samples, seed=dim, verbosity=2) as eng:
        assert planned_filter(eng, capfd) > 0
        table = eng.retrieve()
        eng.assign(*table)  # a saved table
        assert planned_filter(eng, capfd) > 0
        eng.assign(*gamma_params(np.random.default_rng(dim), dim, samples))
        assert planned_filter(eng, capfd) > 0


def others(rs, lc, b):
    rng = np.random.default_rng(5)
    yield "below the bytes' range", rs, lc - 500, b
    yield "above it", rs, lc + 20, b
    yield "shifted up", rs, lc + 1, b
    yield "shifted down", rs, lc - 2, b
    yield "wide r", rs * 100, lc, b
    yield "narrow r", rs * np.float32(0.3), lc, b
    yield "beta outside", rs, lc, b + 5
    yield "all equal", rs * 0 + 1.25, lc * 0 + 0.5, b
    yield "zeros", rs * 0, lc * 0, b * 0
    yield "normal", np.abs(rng.normal(size=rs.shape)), rng.normal(size=rs.shape), b
    yield "not a number", rs * np.nan, lc, b
    odd = lc.copy()
    odd[:, ::2] -= 500
    yield "half of the columns", rs, odd, b
    odd = lc.copy()
    odd[7] += 3
    yield "one sample", rs, odd, b


@pytest.mark.parametrize("dim,samples", [(130, 128), (5000, 100)])
def test_tables_of_other_distributions(dim, samples, capfd):
    table = gamma_params(np.random.default_rng(2), dim, samples)
    with engine_gen(dim, samples, deferred=True, verbosity=2) as eng:
        for name, *other in others(*table):
            if dim == 130 and name == "one sample":
                continue  # six standard deviations of 130 columns hide it
            eng.assign(*other)
            assert planned_filter(eng, capfd) == 0, name
        eng.assign(*table)
        assert planned_filter(eng, capfd) > 0
