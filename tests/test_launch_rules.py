"""The planner's size rules on the CPU, against which kernel was measured faster
(or as fast) on columns whose parameters come from L2, where the filtered kernel
gains least: a launch that the dense kernel hashes faster stays with it."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

pytestmark = pytest.mark.skipif(
    shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")),
    reason="needs g++ and the CUDA headers")


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    exe = tmp_path_factory.mktemp("rules") / "check"
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "minhashcuda_b200", "csrc"),
                           "-I", CUDA_INCLUDE, os.path.join(ROOT, "tests", "launch_rules_check.cc"),
                           "-o", str(exe)])
    return lambda *args: subprocess.run([str(exe), *map(str, args)], check=True, capture_output=True,
                                        text=True).stdout


M = 1_000_000


# Zipf(1.1) columns over 2^20 dimensions: (samples, evaluations, entries per row),
# how much faster the filtered kernel is.
@pytest.mark.parametrize("samples,evals,row,gain", [
    (64, 512 * M, 104, 0.77), (64, 512 * M, 150, 0.99), (64, 597 * M, 233, 0.89), (64, 686 * M, 268, 0.93),
    (128, 512 * M, 104, 0.74), (128, 512 * M, 150, 0.94), (256, 512 * M, 130, 0.81),
    (100, 400 * M, 104, 0.84), (200, 512 * M, 130, 0.95), (384, 512 * M, 150, 0.93),
    (96, 542 * M, 142, 0.88), (112, 512 * M, 130, 0.92), (48, 9 * M, 106, 0.76),
    (128, 70 * M, 300, 0.82), (128, 100 * M, 1400, 0.81), (256, 100 * M, 600, 0.79),
    (64, 70 * M, 1400, 0.86), (64, 40 * M, 300, 0.85), (100, 100 * M, 1400, 0.93),
    (128, 9 * M, 104, 0.87), (128, 18 * M, 300, 0.85), (32, 18 * M, 300, 0.88),
    (128, 100 * M, 6000, 0.87),
    (32, 128 * M, 200, 1.52), (32, 26 * M, 300, 1.06), (64, 512 * M, 300, 1.32),
    (100, 600 * M, 300, 1.5), (128, 512 * M, 210, 1.10), (128, 220 * M, 300, 1.31),
    (128, 220 * M, 1400, 1.18), (128, 50 * M, 300, 1.13), (256, 512 * M, 240, 1.14),
    (200, 512 * M, 170, 1.12), (160, 512 * M, 150, 1.22), (128, 70 * M, 12288, 1.05),
    (128, 20 * M, 20000, 1.45),
])
def test_launches(rule, samples, evals, row, gain):
    nnz = evals // samples
    s_pad = (samples + 3) // 4 * 4
    assert rule("filter", s_pad, samples, nnz, max(1, nnz // row)) == str(int(gain > 1))


@pytest.mark.parametrize("samples,evals,row,gain", [
    (128, 13 * M, 104, 0.58), (128, 101 * M, 600, 0.79), (128, 201 * M, 300, 0.91),
    (128, 401 * M, 1400, 0.91), (256, 403 * M, 600, 0.90), (64, 200 * M, 300, 0.98),
    (100, 52 * M, 300, 0.84), (32, 18 * M, 300, 0.86),
    (128, 801 * M, 300, 1.35), (256, 803 * M, 1400, 1.13), (64, 801 * M, 600, 1.50),
    (100, 202 * M, 300, 1.21), (32, 50 * M, 300, 1.20),
    (256, 6000 * M, 195, 1.0001),  # uniform columns, ragged: 2.15
])
def test_device_batches(rule, samples, evals, row, gain):
    nnz = evals // samples
    assert rule("batch", (samples + 3) // 4 * 4, nnz, max(1, nnz // row)) == str(int(gain > 1))


# How much faster a dense launch is with t kept, on Zipf columns and on uniform
# ones: kept where the loss on the one side is below 2%, or nothing is lost.
@pytest.mark.parametrize("s_pad,spl,row,zipf,uniform", [
    (64, 2, 20, 1.04, 1.11), (64, 2, 50, 0.996, 1.11), (64, 2, 100, 0.966, 1.07),
    (64, 2, 300, 0.94, 1.01), (128, 4, 20, 1.08, 1.18), (128, 4, 70, 1.004, 1.08),
    (128, 4, 140, 0.976, 1.03), (128, 4, 500, 0.956, 1.0), (256, 4, 70, 1.006, 1.08),
    (256, 4, 180, 0.968, 1.02), (200, 4, 100, 1.005, 1.05), (200, 4, 300, 1.0, 1.004),
    (512, 4, 140, 0.997, 1.03), (32, 1, 20, 0.85, 0.85),
])
def test_t_kept(rule, s_pad, spl, row, zipf, uniform):
    assert rule("keep", s_pad, spl, 0, row) == str(int(min(zipf, uniform) > 0.98))


def test_t_kept_in_tiny_launches(rule):
    assert rule("keep", 128, 1, 1, 300) == "1"


@pytest.mark.parametrize("mean_row", [130, 1400, 60_000])
@pytest.mark.parametrize("share", [2000, 40_000, 300_000])
def test_filtered_items_follow_min_items(rule, share, mean_row):
    """Up to eight items per warp asked for, chunks are what they are without; more
    make them shorter, also beyond the 32 waves aimed at."""
    split = lambda items: list(map(int, rule("split", share * 3552, 3552, 32, mean_row, items).split()))  # noqa: E731
    chunk = max(share // 32, min(share // 8, mean_row))
    chunk = max(128, (chunk + 31) // 32 * 32)
    assert split(2) == split(8) == [chunk, max(chunk, min(share // 4, 8192))]
    for items in (16, 64):
        got = split(items)
        assert got[0] <= max(128, share // items + 31)
        assert got[0] + got[1] <= max(256, 3 * share // items + 31)


@pytest.mark.parametrize("s_pad,rows,both", [
    (128, 600, 0), (128, 1200, 1), (64, 2000, 0), (64, 2400, 1), (256, 600, 1), (32, 500, 0), (32, 520, 1)])
def test_batches_that_launch_both_kernels(rule, s_pad, rows, both):
    """A batch that could only be filtered with rows of over 4096 entries is spared
    the second launch."""
    assert rule("both", s_pad, rows) == str(both)


# The rule's lines fall as launches grow: (samples, evaluations, mean row), how much
# faster the filtered kernel is on Zipf columns and on uniform ones (geometric means
# over even and ragged rows).
@pytest.mark.parametrize("samples,evals,row,zipf,uniform", [
    (128, 900 * M, 140, 1.01, 1.30), (128, 2000 * M, 125, 1.14, 1.32), (128, 4000 * M, 106, 0.98, 1.22),
    (128, 150 * M, 260, 1.08, 1.33), (128, 150 * M, 160, 0.81, 1.16), (128, 300 * M, 125, 0.79, 1.03),
    (128, 450 * M, 200, 1.00, 1.27), (128, 50 * M, 125, 1.01, 1.23), (128, 30 * M, 125, 0.86, 0.96),
    (128, 20 * M, 330, 1.09, 1.29), (128, 20 * M, 200, 0.95, 1.11), (128, 12 * M, 420, 1.06, 1.34),
    (64, 1000 * M, 240, 1.09, 1.52), (64, 2000 * M, 185, 1.12, 1.32), (64, 4000 * M, 155, 1.02, 1.21),
    (64, 2000 * M, 110, 0.88, 1.00), (64, 30 * M, 160, 1.06, 1.34), (64, 150 * M, 310, 1.13, 1.40),
    (100, 1000 * M, 116, 1.07, 1.07), (200, 140 * M, 220, 1.20, 1.26), (100, 300 * M, 130, 0.89, 1.00),
    (100, 140 * M, 130, 0.78, 1.01), (160, 90 * M, 230, 1.17, 1.31), (48, 50 * M, 420, 1.08, 1.21),
    (48, 50 * M, 130, 0.77, 0.92), (160, 500 * M, 122, 1.09, 1.11), (32, 140 * M, 106, 1.03, 1.20),
    (32, 30 * M, 130, 0.96, 1.11), (256, 2000 * M, 110, 1.00, 1.18),
])
def test_lines_fall_with_the_launch(rule, samples, evals, row, zipf, uniform):
    nnz = evals // samples
    assert rule("filter", (samples + 3) // 4 * 4, samples, nnz, max(1, nnz // row)) == str(
        int(zipf >= 0.98 and uniform > 1.05))


@pytest.mark.parametrize("row", [1, 104, 120, 168, 288])
def test_batch_lines(rule, row):
    """A batch's line is that of half its evaluations; a forced one takes any row."""
    got = [int(rule("row", row, evals // 2)) for evals in (200 * M, 1000 * M, 2000 * M, 4000 * M, 8000 * M)]
    assert got == sorted(got, reverse=True)
    assert got[0] <= max(row, 288) and got[-1] >= min(row, 104)
    if row <= 104:
        assert got == [row] * 5


def test_the_benchmarks_copy_of_the_rule(rule, monkeypatch):
    """bench.py names the kernel of its launches by the same lines."""
    import importlib.util
    spec = importlib.util.spec_from_file_location("bench_module", os.path.join(ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    monkeypatch.delenv("MHCUDA_B200_FILTER", raising=False)
    for evals in (140 * M, 200 * M, 900 * M, 2000 * M, 9000 * M):
        for row in (100, 110, 130, 150, 180, 220, 1400):
            nnz = evals // 128
            assert str(int(bench.filtered(nnz, nnz // row, 128))) == rule("filter", 128, 128, nnz, nnz // row)
