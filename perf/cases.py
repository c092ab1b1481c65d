"""Performance cases of the weighted-MinHash engine.

Each case is a plain dict; `prepare` makes what a user's program holds before
the call (the generator, the matrices, output buffers), `run` is one pass
through the public entry points, `work` the traffic and arithmetic the pass
cannot do without.  Inputs come from the package's seeded workload generators
(minhashcuda_b200.synth), so a case and a seed name one input.

Kinds of case:

  device        mhcuda_calc_device on a matrix in device memory
  batch_device  mhcuda_calc_batch_device on many matrices in device memory
  host          mhcuda_calc on pageable float32/uint32 host arrays
  host_wide     mhcuda_calc_typed on float64/int64 host arrays (scipy's types)
  serve         a burst of requests through the continuous-batching server
  lsh           band keys and Jaccard estimates on hashes in device memory
"""
import ctypes
import math

import numpy as np
import torch

import minhashcuda_b200 as mh
from minhashcuda_b200 import synth
from minhashcuda_b200.server import Server

# Row-length laws: "poisson" (mean), "lognormal" (median, sigma; clipped to
# [1, 50000]) and "tail" (mean of the shortest rows; P(longer than k times it)
# ~ 1/k, clipped to [1, 50000]).
LAWS = {"poisson": synth.NNZ_POISSON, "lognormal": synth.NNZ_LOGNORMAL, "tail": synth.NNZ_ZIPF}
ZIPF_S = 1.1
MOST_EVALS = 4e10  # of a drawn device case; the largest listed one has 9.4e10


def listed():
    return [
        # One document against a resident generator: an online query, where
        # launches and latency are everything.
        dict(name="query", kind="device", rows=1, law="poisson", nnz=300, sigma=0.0, dim=1 << 20,
             samples=128, cols="uniform", tuned=False),
        # The 6400 x 130 integer matrix of the reference's tests as one plain
        # host call: small data, a sparse matrix of few columns.
        dict(name="small_matrix", kind="host", rows=6400, law="small", nnz=26, sigma=0.0, dim=130,
             samples=128, cols="uniform"),
        # Short texts (titles, messages): many rows of about 20 entries.
        dict(name="short_rows", kind="device", rows=400_000, law="poisson", nnz=20, sigma=0.0,
             dim=1 << 20, samples=128, cols="uniform", tuned=False),
        # A mid-size corpus with a sample count that is no power of two.
        dict(name="documents", kind="device", rows=20_011, law="poisson", nnz=300, sigma=0.0,
             dim=1_000_000, samples=100, cols="zipf", tuned=False),
        # The benchmark's large configuration (1M-word vocabulary, Zipf columns,
        # 1400 entries per row), one 524,288-row block of it, tuned once as a
        # production caller would.
        dict(name="corpus", kind="device", rows=524_288, law="poisson", nnz=1400, sigma=0.0,
             dim=1_000_000, samples=128, cols="zipf", tuned=True),
        # The streamed configuration: uniform columns over 12M dimensions and
        # ragged rows, where no column is hot.
        dict(name="wide_vocabulary", kind="device", rows=131_072, law="lognormal", nnz=200,
             sigma=1.354, dim=12_000_000, samples=128, cols="uniform", tuned=False),
        # Heavy-tailed row lengths (up to 50,000 entries) at 256 samples, the
        # large resident generator of the serving configuration's kind.
        dict(name="heavy_tail", kind="device", rows=30_000, law="tail", nnz=50, sigma=2.0,
             dim=1 << 22, samples=256, cols="uniform", tuned=False),
        # Many uneven matrices in device memory hashed as one batch (the
        # batched configuration, a sixteenth of its 4096 matrices).
        dict(name="batch", kind="batch_device", matrices=256, max_rows=4096, law="lognormal",
             nnz=64, sigma=1.5, dim=1 << 20, samples=256, cols="uniform"),
        # A matrix held by numpy hashed through the drop-in call, pageable
        # memory in and out: the way most programs use the library.
        dict(name="host_corpus", kind="host", rows=40_000, law="poisson", nnz=1400, sigma=0.0,
             dim=1_000_000, samples=128, cols="zipf"),
        # The same in the types scipy gives (float64 values, int64 indices).
        dict(name="host_wide_types", kind="host_wide", rows=12_000, law="poisson", nnz=1400,
             sigma=0.0, dim=1_000_000, samples=128, cols="zipf"),
        # A burst of requests of very different sizes through the server.
        dict(name="serve_burst", kind="serve", requests=48, max_rows=4000, law="tail", nnz=50,
             sigma=2.0, dim=1 << 20, samples=128, cols="uniform"),
        # Near-duplicate search on finished hashes: LSH bands of 4 samples and
        # Jaccard estimates of candidate pairs.
        dict(name="near_duplicates", kind="lsh", rows=400_000, samples=128, band=4,
             pairs=500_000),
    ]


def _log_between(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["device"] * 6 + ["batch_device", "batch_device", "host", "host",
                                        "host_wide", "lsh"])
    samples = rng.choice([32, 64, 100, 128, 128, 128, 200, 256])
    if kind == "lsh":
        return dict(kind=kind, rows=int(_log_between(rng, 5_000, 400_000)), samples=samples,
                    band=rng.randint(2, 8), pairs=int(_log_between(rng, 10_000, 500_000)))
    law = rng.choice(["poisson", "lognormal", "tail"])
    cols = rng.choice(["zipf", "uniform"]) if law == "poisson" else "uniform"
    dim = int(_log_between(rng, 1 << 16, 1 << 22))
    c = dict(kind=kind, law=law, dim=dim, samples=samples, cols=cols)
    if law == "poisson":
        c.update(nnz=int(_log_between(rng, 8, 1500)), sigma=0.0)
    elif law == "lognormal":
        c.update(nnz=int(_log_between(rng, 8, 400)), sigma=round(rng.uniform(0.5, 1.5), 3))
    else:
        c.update(nnz=int(_log_between(rng, 8, 100)), sigma=2.0)
    if kind == "batch_device":
        c.update(matrices=int(_log_between(rng, 4, 200)), max_rows=int(_log_between(rng, 16, 3000)))
        return c
    most = {"device": MOST_EVALS / samples, "host": 4e7, "host_wide": 1.2e7}[kind]
    nnz = _log_between(rng, 2e3, most)
    c["rows"] = max(1, min(1 << 20, int(nnz / _mean_nnz(c))))
    if kind == "device":
        c["tuned"] = False
    return c


# ---- inputs ---------------------------------------------------------------


class Generator:
    """A generator handle, released with its state."""

    def __init__(self, dim, samples, seed):
        status = ctypes.c_int(-1)
        self.handle = mh.capi().mhcuda_init(dim, samples, seed, 0, 0, 0, ctypes.byref(status))
        if not self.handle:
            raise mh.MHCUDAError("mhcuda_init", status.value)

    def __del__(self):
        if getattr(self, "handle", None):
            mh.capi().mhcuda_fini(self.handle)
            self.handle = None


def _workload(case, seed):
    return synth.Workload("case", rows=case.get("rows", 0), dim=case["dim"],
                          samples=case["samples"], seed=seed, nnz_kind=LAWS[case["law"]],
                          nnz_p1=float(case["nnz"]), nnz_p2=case["sigma"],
                          nnz_lo=0 if case["law"] == "poisson" else 1,
                          nnz_hi=2048 if case["cols"] == "zipf" else 50_000, cols=case["cols"],
                          zipf_s=ZIPF_S)


def _small(seed):
    """The reference tests' matrix with values and zeros drawn from `seed`."""
    return synth.small_csr(seed % (1 << 31))


def _batch_rows(case):
    """Row counts of a batch's matrices or a burst's requests, log-uniform; a
    property of the case, as its other sizes are."""
    top = case.get("matrices", case.get("requests"))
    rng = np.random.default_rng(top * 8192 + case["max_rows"])
    r = np.floor(np.exp(rng.uniform(0.0, math.log(case["max_rows"]), top))).astype(np.int64)
    return np.clip(r, 1, case["max_rows"])


def prepare(case, seed):
    if case["kind"] == "lsh":
        return _prepare_lsh(case, seed)
    st = dict(case=case, lib=mh.capi(), gen=Generator(case["dim"], case["samples"], seed & 0x7FFFFFFF))
    samples = case["samples"]
    if case["kind"] == "device":
        w = _workload(case, seed)
        indptr, cols, weights, nnz = synth.device_csr(w, 0, case["rows"])
        out = torch.zeros((case["rows"], samples, 2), dtype=torch.int32, device="cuda")
        st.update(indptr=indptr, cols=cols, weights=weights, nnz=nnz, out=out,
                  stream=torch.cuda.Stream())
        torch.cuda.synchronize()
        if case["tuned"]:
            mh.check("mhcuda_autotune", st["lib"].mhcuda_autotune(
                st["gen"].handle, weights.data_ptr(), cols.data_ptr(), indptr.data_ptr(),
                case["rows"], nnz, out.data_ptr(), st["stream"].cuda_stream, None, None))
    elif case["kind"] == "batch_device":
        # Every matrix has arrays of its own; the hashes go to one buffer.
        w, mats, row0 = _workload(case, seed), [], 0
        lengths = _batch_rows(case)
        out = torch.zeros((int(lengths.sum()), samples, 2), dtype=torch.int32, device="cuda")
        for r in lengths:
            indptr, cols, weights, _ = synth.device_csr(w, row0, int(r))
            mats.append((weights, cols, indptr, out[row0:row0 + int(r)]))
            row0 += int(r)
        n = len(mats)
        arr = lambda i: (ctypes.c_void_p * n)(*[m[i].data_ptr() for m in mats])  # noqa: E731
        st.update(mats=mats, out=out, count=n, weights=arr(0), cols=arr(1), indptr=arr(2), outs=arr(3),
                  lengths=(ctypes.c_uint32 * n)(*[m[3].shape[0] for m in mats]),
                  stream=torch.cuda.Stream())
    elif case["kind"] in ("host", "host_wide"):
        if case["law"] == "small":
            indptr, cols, weights = _small(seed)
        else:
            indptr, cols, weights = synth.host_csr(_workload(case, seed), 0, case["rows"])
        if case["kind"] == "host_wide":
            weights = weights.astype(np.float64)
            cols, indptr = cols.astype(np.int64), indptr.astype(np.int64)
        st.update(indptr=indptr, cols=cols, weights=weights,
                  out=np.zeros((case["rows"], samples, 2), np.uint32))
    else:
        w, reqs, row0 = _workload(case, seed), [], 0
        for r in _batch_rows(case):
            indptr, cols, weights = synth.host_csr(w, row0, int(r))
            reqs.append((weights, cols, indptr, np.zeros((int(r), samples, 2), np.uint32)))
            row0 += int(r)
        st.update(reqs=reqs, server=Server(hbm_budget=2 << 30, lanes=4))
    torch.cuda.synchronize()
    return st


def _prepare_lsh(case, seed):
    """Hashes of rows that come in groups of near-duplicates: every row keeps
    the (k, t) of its group's first row at a random share of the samples."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    rows, samples, pairs = case["rows"], case["samples"], case["pairs"]
    kw = dict(generator=g, device="cuda")
    hashes = torch.randint(0, 1 << 20, (rows, samples, 2), dtype=torch.int32, **kw)
    first = torch.arange(rows, device="cuda") // 4 * 4
    share = torch.rand((rows, 1, 1), **kw)
    keep = torch.rand((rows, samples, 1), **kw) < share
    hashes = torch.where(keep, hashes[first], hashes).contiguous()
    a = torch.randint(0, rows, (pairs,), **kw)
    b = torch.where(torch.rand(pairs, **kw) < 0.5, (a // 4 * 4 + 1).clamp(max=rows - 1),
                    torch.randint(0, rows, (pairs,), **kw))
    st = dict(case=case, lib=mh.capi(), gen=Generator(16, samples, seed & 0x7FFFFFFF),
              hashes=hashes, pairs=torch.stack([a, b], 1).to(torch.int32).contiguous(),
              keys=torch.zeros((rows, samples // case["band"]), dtype=torch.int64, device="cuda"),
              estimates=torch.zeros(pairs, device="cuda"), stream=torch.cuda.Stream())
    torch.cuda.synchronize()
    return st


# ---- one pass -------------------------------------------------------------


def run(st):
    kind, lib = st["case"]["kind"], st["lib"]
    gen = st["gen"].handle
    if kind == "device":
        mh.check("mhcuda_calc_device", lib.mhcuda_calc_device(
            gen, st["weights"].data_ptr(), st["cols"].data_ptr(), st["indptr"].data_ptr(),
            st["case"]["rows"], st["nnz"], st["out"].data_ptr(), st["stream"].cuda_stream))
        return st["out"]
    if kind == "batch_device":
        mh.check("mhcuda_calc_batch_device", lib.mhcuda_calc_batch_device(
            gen, st["count"], st["weights"], st["cols"], st["indptr"], st["lengths"], st["outs"],
            st["stream"].cuda_stream))
        return st["out"]
    if kind == "host":
        mh.check("mhcuda_calc", lib.mhcuda_calc(
            gen, st["weights"].ctypes.data, st["cols"].ctypes.data, st["indptr"].ctypes.data,
            st["case"]["rows"], st["out"].ctypes.data))
        return st["out"]
    if kind == "host_wide":
        mh.check("mhcuda_calc_typed", lib.mhcuda_calc_typed(
            gen, st["weights"].ctypes.data, mh.FLOAT64, st["cols"].ctypes.data, mh.INT64,
            st["indptr"].ctypes.data, mh.INT64, st["case"]["rows"], st["out"].ctypes.data))
        return st["out"]
    if kind == "serve":
        srv = st["server"]
        tickets = [srv.submit_raw(gen, w, c, p, len(p) - 1, out) for w, c, p, out in st["reqs"]]
        return [srv.wait(t) for t in tickets]
    case = st["case"]
    mh.check("mhcuda_lsh_bands", lib.mhcuda_lsh_bands(
        gen, st["hashes"].data_ptr(), case["rows"], case["band"], st["keys"].data_ptr(),
        st["stream"].cuda_stream))
    mh.check("mhcuda_jaccard", lib.mhcuda_jaccard(
        gen, st["hashes"].data_ptr(), case["rows"], st["pairs"].data_ptr(), case["pairs"],
        st["estimates"].data_ptr(), st["stream"].cuda_stream))
    return {"keys": st["keys"], "estimates": st["estimates"]}


# ---- what a pass cannot do without ----------------------------------------


def _mean_nnz(case):
    n = float(case["nnz"])
    if case["law"] == "lognormal":
        n *= math.exp(case["sigma"] ** 2 / 2)
    elif case["law"] == "tail":
        n *= 1.0 + math.log(50_000 / n) + 0.577
    return n


def _distinct(case, entries):
    """Expected distinct columns among `entries` draws: each one's parameters
    are read at least once."""
    dim = case["dim"]
    if case["cols"] == "zipf":
        p = np.arange(1, dim + 1, dtype=np.float64) ** -ZIPF_S
        return float(-np.expm1(-entries * (p / p.sum())).sum())
    return dim * -math.expm1(-entries / dim)


def work(case):
    """CSR and offsets in, hashes out, and the 12 bytes of parameters of every
    (distinct column, sample) once; eight float32 operations per (entry,
    sample)."""
    samples = case["samples"]
    if case["kind"] == "lsh":
        read = 8.0 * samples * case["rows"] + 8.0 * case["pairs"]
        return {"bytes": read + 8.0 * (samples // case["band"]) * case["rows"] + 4.0 * case["pairs"],
                "flops": 0.0}
    if case["kind"] in ("batch_device", "serve"):
        rows = int(_batch_rows(case).sum())
    else:
        rows = case["rows"]
    entries = rows * _mean_nnz(case)
    per_entry = 16.0 if case["kind"] == "host_wide" else 8.0
    per_row = 8.0 if case["kind"] == "host_wide" else 4.0
    return {"bytes": per_entry * entries + per_row * rows + 8.0 * samples * rows
            + 12.0 * samples * _distinct(case, entries),
            "flops": 8.0 * entries * samples}


# ---- exact values ---------------------------------------------------------


def exact(case, seed):
    """The Jaccard estimates in 64 bits.  Hashes and band keys are whole
    numbers: they are compared as such."""
    if case["kind"] != "lsh":
        return None
    st = _prepare_lsh(case, seed)
    h, pairs = st["hashes"], st["pairs"].long()
    est = torch.empty(case["pairs"], dtype=torch.float64, device="cuda")
    for i in range(0, case["pairs"], 65_536):
        p = pairs[i:i + 65_536]
        est[i:i + 65_536] = (h[p[:, 0]] == h[p[:, 1]]).all(2).double().mean(1)
    return {"keys": None, "estimates": est}
