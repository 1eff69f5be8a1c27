"""The hand-off between CTAs of the tensor-core blind rotation: products and
evaluations of every tile of a launch (five of 128 ciphertexts, the last one
partly filled) are read by other CTAs than wrote them, in every step.  Launch
after launch on fresh inputs, every output word equal to the oracle's."""
import numpy as np
import pytest

import luthe_b200 as L
import oracle
from conftest import from_dev, to_dev

pytestmark = pytest.mark.gpu
N, STEPS = 2048, 8


@pytest.mark.parametrize("count", [300, 513, 592])
def test_every_tile_of_consecutive_launches(count):
    p = L.default_params(lwe_dim=STEPS)
    keys = L.keygen(p, 29)
    ob = oracle.OracleBsk(keys["bsk"], STEPS, N)
    rng = np.random.default_rng(count)
    luts = rng.integers(0, 2**64, (2, 2 * N), dtype=np.uint64)
    with L.Engine(p) as eng:
        eng.upload_keys(keys)
        eng.upload_luts(luts)
        runs = []
        for _ in range(4):
            lwe = rng.integers(0, 2 * N, (count, STEPS + 1), dtype=np.uint32)
            ids = rng.integers(0, 2, count).astype(np.uint32)
            d_out = to_dev(np.zeros((count, N + 1), np.uint64))
            eng.blind_rotate(to_dev(lwe), to_dev(ids), d_out, count)
            runs.append((lwe, ids, d_out))
        eng.check_device_error()
        for lwe, ids, d_out in runs:
            got, want = from_dev(d_out, np.uint64), ob.blind_rotate(lwe, luts, ids)
            assert np.array_equal(got, want), np.nonzero((got != want).any(1))[0]
