"""Plans after the autotuner chose the filtered kernel."""
import re

import numpy as np
import pytest

from wmh_testlib import engine_gen

pytestmark = pytest.mark.gpu


def test_a_dense_launch_is_not_tuned_by_a_filtered_winner(capfd, monkeypatch):
    """At 32 samples the autotuner's filtered choice reports 4 samples per lane, a
    dense tile three quarters empty; a dense launch of that shape is planned as
    without a choice."""
    import torch
    dim, samples, rows, length = 1 << 16, 32, 7000, 300
    rng = np.random.default_rng(0)
    w = rng.lognormal(0.0, 1.0, rows * length).astype(np.float32)
    c = rng.integers(0, dim, rows * length).astype(np.uint32)
    p = (np.arange(rows + 1) * length).astype(np.uint32)

    def plan(eng):
        capfd.readouterr()
        eng.calc(w, c, p)
        return re.search(r"plan: .*", capfd.readouterr().out).group(0)

    with engine_gen(dim, samples, seed=1, verbosity=2) as eng:
        monkeypatch.setenv("MHCUDA_B200_FILTER", "0")
        untuned = plan(eng)
        monkeypatch.delenv("MHCUDA_B200_FILTER")
        dev = [torch.from_numpy(x.view(np.int32) if x.dtype != np.float32 else x).cuda() for x in (w, c, p)]
        out = torch.zeros((rows, samples, 2), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        rc = eng.lib.mhcuda_autotune(eng.h, *[x.data_ptr() for x in dev], rows, rows * length,
                                     out.data_ptr(), None, None, None)
        assert rc == 0
        if " filter=0 " in plan(eng):
            pytest.skip("the dense kernel won")
        monkeypatch.setenv("MHCUDA_B200_FILTER", "0")
        assert plan(eng) == untuned
