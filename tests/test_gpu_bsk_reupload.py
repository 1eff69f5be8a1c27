"""A key uploaded over another one, in the evaluation domain and back in the
standard domain, reaches every form of the blind rotation: batches of more than
one ciphertext per SM (the expanded key) and of a few (the slab)."""
import numpy as np
import pytest

import luthe_b200 as L
import oracle
from conftest import from_dev, to_dev

pytestmark = pytest.mark.gpu
N, STEPS = 2048, 12


def test_both_forms_follow_the_key():
    import torch
    p = L.default_params(lwe_dim=STEPS)
    count = torch.cuda.get_device_properties(0).multi_processor_count + 4
    rng = np.random.default_rng(6)
    lwe = rng.integers(0, 2 * N, (count, STEPS + 1), dtype=np.uint32)
    luts = rng.integers(0, 2**64, (1, 2 * N), dtype=np.uint64)
    ids = np.zeros(count, np.uint32)
    first, second = L.keygen(p, 61), L.keygen(p, 62)
    with L.Engine(p) as eng:
        eng.upload_keys(first)
        eng.upload_luts(luts)
        for form, keys in (("std", first), ("eval", second), ("std", first)):
            if form == "std":
                eng.upload_bsk(keys["bsk"])
            else:
                eng.upload_bsk_eval(np.stack([oracle.ntt_eval(x) for x in keys["bsk"].reshape(-1, N)]).reshape(-1))
            want = oracle.OracleBsk(keys["bsk"], STEPS, N).blind_rotate(lwe, luts, ids)
            for m in (count, 5):
                d_out = to_dev(np.zeros((m, N + 1), np.uint64))
                eng.blind_rotate(to_dev(lwe[:m]), to_dev(ids[:m]), d_out, m)
                eng.check_device_error()
                assert np.array_equal(from_dev(d_out, np.uint64), want[:m]), (form, m)
