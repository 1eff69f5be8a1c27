"""Calls on a stream of a green context (16 of the SMs): batches on both sides of
one ciphertext per SM, and the smallest ones, give the oracle's outputs, and the
context's other streams keep their forms."""
import numpy as np
import pytest

import luthe_b200 as L
import oracle
from conftest import from_dev, to_dev

pytestmark = pytest.mark.gpu
N, STEPS = 2048, 12


def _ok(r):
    assert int(r[0]) == 0, r
    return r[1] if len(r) == 2 else r[1:]


def test_a_stream_with_some_of_the_SMs():
    import torch
    drv = pytest.importorskip("cuda.bindings.driver")
    torch.zeros(1, device="cuda")
    dev = _ok(drv.cuDeviceGet(0))
    sms = _ok(drv.cuDeviceGetDevResource(dev, drv.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups = _ok(drv.cuDevSmResourceSplitByCount(1, sms, 0, 16))[0]
    desc = _ok(drv.cuDevResourceGenerateDesc([groups[0]], 1))
    green = _ok(drv.cuGreenCtxCreate(desc, dev, drv.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream = _ok(drv.cuGreenCtxStreamCreate(green, drv.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    p = L.default_params(lwe_dim=STEPS)
    keys = L.keygen(p, 71)
    ob = oracle.OracleBsk(keys["bsk"], STEPS, N)
    rng = np.random.default_rng(71)
    luts = rng.integers(0, 2**64, (2, 2 * N), dtype=np.uint64)
    with L.Engine(p) as eng:
        eng.upload_keys(keys)
        eng.upload_luts(luts)
        for count in (1, 20, 60, nsm, nsm + 1, 2 * nsm + 30):
            lwe = rng.integers(0, 2 * N, (count, STEPS + 1), dtype=np.uint32)
            ids = rng.integers(0, 2, count).astype(np.uint32)
            want = ob.blind_rotate(lwe, luts, ids)
            for s in (int(stream), None):
                d_lwe, d_ids, d_out = to_dev(lwe), to_dev(ids), to_dev(np.zeros((count, N + 1), np.uint64))
                torch.cuda.synchronize()
                eng.blind_rotate(d_lwe, d_ids, d_out, count, s)
                if s:
                    _ok(drv.cuStreamSynchronize(stream) + (None,))
                torch.cuda.synchronize()
                eng.check_device_error()
                assert np.array_equal(from_dev(d_out, np.uint64), want), (count, s)
    _ok(drv.cuStreamDestroy(stream) + (None,))
    _ok(drv.cuGreenCtxDestroy(green) + (None,))
