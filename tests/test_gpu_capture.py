"""A graph captured by the caller keeps working when the context would give up
the optional tensor-core forms for a later allocation, and follows a new key."""
import numpy as np
import pytest

import luthe_b200 as L
import oracle
from conftest import from_dev, to_dev

pytestmark = pytest.mark.gpu
N, STEPS = 2048, 24


@pytest.mark.parametrize("count", [7, 160])
def test_captured_launches_survive_a_full_budget_and_a_new_key(count):
    import torch
    p = L.default_params(lwe_dim=STEPS)
    keys, keys2 = L.keygen(p, 23), L.keygen(p, 24)
    luts = L.lut_build(p, np.arange(16, dtype=np.uint32)[::-1].copy())[None]
    with L.Engine(p) as probe:
        probe.upload_keys(keys)
        full = probe.device_bytes
    with L.Engine(p, hbm_budget=full + (8 << 20)) as eng:
        eng.upload_keys(keys)
        eng.upload_luts(luts)
        ids = np.zeros(count, np.uint32)
        msgs = np.arange(count, dtype=np.uint32) % 16
        ct = L.encrypt(p, keys["glwe_key"], msgs, 3)
        d_in, d_ids, d_out = to_dev(ct), to_dev(ids), to_dev(np.zeros((count, N + 1), np.uint64))
        eng.ks_pbs_noalloc(d_in, d_ids, d_out, count)
        torch.cuda.synchronize()
        want = oracle.OracleBsk(keys["bsk"], STEPS, N).ks_pbs(keys["ksk"], ct, luts, ids)
        assert np.array_equal(from_dev(d_out, np.uint64), want)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            eng.ks_pbs_noalloc(d_in, d_ids, d_out, count, torch.cuda.current_stream())
        eng.reserve(1 << 20)  # does not fit beside the optional forms
        d_out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(from_dev(d_out, np.uint64), want)
        eng.upload_keys(keys2)
        ct2 = L.encrypt(p, keys2["glwe_key"], msgs, 4)
        d_in.copy_(to_dev(ct2))
        g.replay()
        torch.cuda.synchronize()
        want2 = oracle.OracleBsk(keys2["bsk"], STEPS, N).ks_pbs(keys2["ksk"], ct2, luts, ids)
        assert np.array_equal(from_dev(d_out, np.uint64), want2)
        eng.check_device_error()
        del g
