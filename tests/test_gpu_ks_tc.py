"""The tensor-core key switch (batches above 32 ciphertexts): every output word
of every parameter set, in both tie rules, equal to the dp4a form's (a context
without room for the tensor-core form) and on edge rows to the oracle's, at the
edges of its row tiles (128, 256), of the split over K (1024 and less) and of
its passes (3584)."""
import numpy as np
import pytest

import luthe_b200 as L
import oracle
from conftest import from_dev, to_dev

pytestmark = pytest.mark.gpu
N = 2048


@pytest.fixture(scope="module", params=sorted(L.PARAM_SETS))
def setup(request):
    p = L.param_set(request.param)
    rng = np.random.default_rng(p.lwe_dim)
    ksk = rng.integers(0, 1 << 21, (p.lwe_dim + 1) * N * p.ks_level, dtype=np.uint32)
    ksk[: 4 * N] = (1 << 21) - 1
    tc, plain = L.Engine(p), L.Engine(p, hbm_budget=60 << 20)
    tc.upload_ksk(ksk)
    plain.upload_ksk(ksk)
    assert plain.device_bytes < 60 << 20 < tc.device_bytes  # no room beside the dp4a form's key
    yield p, ksk, tc, plain
    tc.close()
    plain.close()


def _switch(eng, d_in, count, n, rule):
    d21 = to_dev(np.zeros((count, n + 1), np.uint32))
    d2n = to_dev(np.zeros((count, n + 1), np.uint32))
    eng.set_tie_rule(rule)
    try:
        eng.keyswitch(d_in, d21, d2n, count)
        eng.check_device_error()
    finally:
        eng.set_tie_rule(L.TIE_RTL)
    return from_dev(d21, np.uint32), from_dev(d2n, np.uint32)


@pytest.mark.parametrize("count", [33, 128, 129, 257, 1024, 1025, 3585])
def test_every_output(setup, count):
    p, ksk, tc, plain = setup
    n = p.lwe_dim
    rng = np.random.default_rng(count)
    x = rng.integers(0, 2**64, (count, N + 1), dtype=np.uint64)
    tot = p.ks_base_log * p.ks_level
    edge = [0, 1, 2**64 - 1, 1 << 63, (1 << 63) - 1, 1 << (64 - tot), 1 << (63 - tot), 2**64 - (1 << (63 - tot)),
            0x5555555555555555, 0xAAAAAAAAAAAAAAAA, 0x8888888888888888, 0x4444444444444444]
    x[0] = 2**64 - 1
    x[1] = rng.choice(np.array(edge, np.uint64), N + 1)
    x[-1] = rng.choice(np.array(edge, np.uint64), N + 1)
    x[2] = 1 << 63
    rule = L.TIE_GENERATOR if count % 2 else L.TIE_RTL
    d_in = to_dev(x)
    got21, got2n = _switch(tc, d_in, count, n, rule)
    again21, _ = _switch(tc, d_in, count, n, rule)  # the partial sums were left clear
    want21, want2n = _switch(plain, d_in, count, n, rule)
    assert np.array_equal(got21, want21) and np.array_equal(got2n, want2n)
    assert np.array_equal(again21, got21)
    for c in (0, 1, 2, 32, count - 1):
        o21, o2n = oracle.keyswitch(x[c], ksk, n, N, ks_bl=p.ks_base_log, ks_lc=p.ks_level,
                                    gtv_top_tie=rule == L.TIE_GENERATOR)
        assert np.array_equal(got21[c], o21) and np.array_equal(got2n[c], o2n), c
