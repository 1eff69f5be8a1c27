"""The tensor-core blind rotation at the smallest numbers of steps: its phases,
rings and counters start and end within one to three steps."""
import numpy as np
import pytest

import luthe_b200 as L
import oracle
from conftest import from_dev, to_dev

pytestmark = pytest.mark.gpu
N = 2048


@pytest.mark.parametrize("steps", [1, 2, 3])
def test_few_steps(steps):
    import torch
    count = torch.cuda.get_device_properties(0).multi_processor_count + 1
    p = L.default_params(lwe_dim=steps)
    keys = L.keygen(p, 83)
    ob = oracle.OracleBsk(keys["bsk"], steps, N)
    rng = np.random.default_rng(steps)
    luts = rng.integers(0, 2**64, (1, 2 * N), dtype=np.uint64)
    with L.Engine(p) as eng:
        eng.upload_keys(keys)
        eng.upload_luts(luts)
        for m in (count, 400, 592):
            lwe = rng.integers(0, 2 * N, (m, steps + 1), dtype=np.uint32)
            ids = np.zeros(m, np.uint32)
            d_out = to_dev(np.zeros((m, N + 1), np.uint64))
            eng.blind_rotate(to_dev(lwe), to_dev(ids), d_out, m)
            eng.check_device_error()
            assert np.array_equal(from_dev(d_out, np.uint64), ob.blind_rotate(lwe, luts, ids)), m
