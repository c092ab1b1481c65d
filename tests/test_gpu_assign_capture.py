"""Assigning a table under a caller's CUDA graph of an earlier call."""
import ctypes

import numpy as np
import pytest

import oracle as O
from wmh_testlib import device_logf, engine_gen, gamma_params, random_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scarce", [False, True])
def test_captured_filtered_call_follows_assign(scarce, monkeypatch):
    """A captured call of the bound-filtered kernel hashes with the table assigned
    after the capture, also when device memory is too scarce for assign to rewrite
    the bounds (it needs three blocks of the table for that, one without)."""
    import torch
    monkeypatch.setenv("MHCUDA_B200_FILTER", "1")
    dim, samples = 1 << 20, 64
    rng = np.random.default_rng(3)
    first = gamma_params(rng, dim, samples)
    second = gamma_params(rng, dim, samples)
    m = random_csr(rng, 50, dim, 300)
    block = dim * samples * 4
    with engine_gen(dim, samples, deferred=True) as eng:
        eng.assign(*first)
        dev = [torch.from_numpy(x).cuda() for x in (
            m.data, m.indices.astype(np.uint32).view(np.int32), m.indptr.astype(np.uint32).view(np.int32))]
        out = torch.zeros((m.shape[0], samples, 2), dtype=torch.int32, device="cuda")

        def call(stream):
            return eng.lib.mhcuda_calc_device(eng.h, *[x.data_ptr() for x in dev], m.shape[0], m.nnz,
                                              out.data_ptr(), ctypes.c_void_p(stream.cuda_stream))

        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        assert call(stream) == 0  # the workspace, before the capture
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            assert call(torch.cuda.current_stream()) == 0
        graph.replay()
        torch.cuda.synchronize()
        lnw = device_logf(m.data)
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32),
                                      O.COracle(*first).hash_csr(m, lnw=lnw))
        hold = None
        if scarce:
            torch.cuda.empty_cache()
            free = torch.cuda.mem_get_info()[0]
            hold = torch.empty(free - 2 * block, dtype=torch.uint8, device="cuda")
            assert block < torch.cuda.mem_get_info()[0] < 3 * block
        try:
            eng.assign(*second)
        finally:
            del hold
            torch.cuda.empty_cache()  # back to the device: the engine allocates beside torch
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32),
                                      O.COracle(*second).hash_csr(m, lnw=lnw))
