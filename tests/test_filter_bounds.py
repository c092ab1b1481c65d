"""The filter's skip rule on the CPU: an entry whose value would replace a
sample's minimum is never ruled out.

The byte and threshold arithmetic of the filtered kernels is restated in
float32 numpy; for every entry the threshold is set to the value the entry
itself evaluates to, the lowest at which it may still be skipped as a tie or a
worse one, and the entry has to pass.
"""
import numpy as np
import pytest

F = np.float32


def bound_byte(r, c, b):
    known = (r >= F(2.0**-60)) & (r <= 64) & (np.abs(c) <= 64) & (np.abs(b) <= 2)
    with np.errstate(invalid="ignore"):
        x = np.floor((c - r - F(2.0**-9) + F(12.0)) * F(20.0))
    return np.where(known, np.clip(x, 0, 255), 0).astype(np.int64)


def quant_up(x):
    y = np.ceil(x.astype(np.float64) * 20.0 + 0.01).astype(F)  # one rounding, as the fma
    return np.clip(np.nan_to_num(y, nan=0.0, posinf=8191, neginf=-8192), -8192, 8191).astype(np.int64)


def ln_a(w, r, c, b):
    """kernel.cu:101-105 with the fused multiply-add; float64 holds the exact
    product, so the sum is rounded to float32 all but once."""
    with np.errstate(all="ignore"):
        t = np.floor((w / r).astype(F) + b)
        tb = (t - b).astype(F)
        fused = (c.astype(np.float64) - tb.astype(np.float64) * r.astype(np.float64)).astype(F)
        return fused - r


def tables(rng, n, kind):
    r = rng.gamma(2.0, 1.0, n).astype(F)
    c = np.log(rng.gamma(2.0, 1.0, n)).astype(F)
    b = rng.uniform(0.0, 1.0, n).astype(F)
    if kind == "extreme":
        r = np.exp(rng.uniform(np.log(1e-18), np.log(64.0), n)).astype(F)
        c = rng.uniform(-64.0, 64.0, n).astype(F)
        b = rng.uniform(-2.0, 2.0, n).astype(F)
    elif kind == "outside":
        r = (r * rng.choice([0.0, -1.0, 1.0, 1e3, 1e-30], n)).astype(F)
        c = (c * rng.choice([1.0, 100.0], n)).astype(F)
        b = (b * rng.choice([1.0, 50.0], n)).astype(F)
    return r, c, b


@pytest.mark.parametrize("kind", ["gamma", "extreme", "outside"])
@pytest.mark.parametrize("weights", ["lognormal", "whole range"])
def test_an_entry_that_could_win_is_never_skipped(kind, weights):
    rng = np.random.default_rng(len(kind) * 10 + len(weights))
    n = 400_000
    r, c, b = tables(rng, n, kind)
    x = rng.lognormal(0.0, 1.0, n) if weights == "lognormal" else 10.0 ** rng.uniform(-44, 38, n)
    with np.errstate(divide="ignore"):
        w = np.log(x.astype(F))
    v = ln_a(w, r, c, b)
    could = v < np.finfo(F).max  # NaN and infinite values never replace a minimum
    passes = bound_byte(r, c, b) <= np.maximum(quant_up(v) + quant_up(w) + 240, 0)
    assert could.sum() > n // 4
    assert passes[could].all()
