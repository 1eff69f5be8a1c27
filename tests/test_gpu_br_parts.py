"""The blind rotation of the smallest batches, one ciphertext on a cluster of
eight or four SMs: every output word equal to the oracle's at the smallest
batch, around the sizes at which the launch changes form on 148 SMs, in both tie
rules, both PBS bases, with an odd and an even number of steps (the exchange
buffers alternate) and with many-LUT outputs."""
import numpy as np
import pytest

import luthe_b200 as L
import oracle
from conftest import from_dev, to_dev

pytestmark = pytest.mark.gpu
N = 2048


@pytest.fixture(scope="module", params=[(23, 24), (22, 24), (23, 1), (22, 3)])
def setup(request):
    bw, steps = request.param
    p = L.default_params(lwe_dim=steps, pbs_base_log=bw)
    keys = L.keygen(p, 19)
    eng = L.Engine(p)
    eng.upload_keys(keys)
    yield p, keys, eng, oracle.OracleBsk(keys["bsk"], steps, N)
    eng.close()


def _run(eng, p, ob, lwe, luts, ids, generator):
    eng.upload_luts(luts)
    eng.set_tie_rule(L.TIE_GENERATOR if generator else L.TIE_RTL)
    oracle.set_tie_rule(generator)
    try:
        d_out = to_dev(np.zeros((len(ids), N + 1), np.uint64))
        eng.blind_rotate(to_dev(lwe), to_dev(ids), d_out, len(ids))
        eng.check_device_error()
        got, want = from_dev(d_out, np.uint64), ob.blind_rotate(lwe, luts, ids, pbs_bl=p.pbs_base_log)
    finally:
        eng.set_tie_rule(L.TIE_RTL)
        oracle.set_tie_rule(False)
    assert np.array_equal(got, want), np.nonzero((got != want).any(1))[0]


@pytest.mark.parametrize("count", [1, 2, 14, 15, 16, 17, 18, 19, 32, 34, 35, 36, 37, 38])
def test_every_output_equals_the_oracle(setup, count):
    p, keys, eng, ob = setup
    rng = np.random.default_rng(count)
    lwe = rng.integers(0, 2 * N, (count, p.lwe_dim + 1), dtype=np.uint32)
    lwe[0] = 2 * N - 1
    luts = rng.integers(0, 2**64, (3, 2 * N), dtype=np.uint64)
    _run(eng, p, ob, lwe, luts, rng.integers(0, 3, count).astype(np.uint32), generator=count % 2 == 0)


@pytest.mark.parametrize("generator", [False, True])
@pytest.mark.parametrize("count", [12, 24])
def test_ties_and_extreme_words(setup, generator, count):
    p, keys, eng, ob = setup
    bw = p.pbs_base_log
    rng = np.random.default_rng(7)
    half = 1 << (63 - bw)  # the rounding bit
    words = [0, 1, 1 << 63, (1 << 63) - 1, (1 << 63) - half, (1 << 63) - half - 1, (1 << 63) + half, half, half - 1,
             2**64 - 1, 2**64 - half, 1 << 62, 3 << 62, 0xFFFFFFFF00000000, 0xFFFFFFFF]
    luts = np.stack([np.full(2 * N, w, np.uint64) for w in words[:9]] +
                    [rng.choice(np.array(words, np.uint64), 2 * N) for _ in range(3)])
    lwe = rng.choice(np.array([0, 1, N - 1, N, N + 1, 2 * N - 1], np.uint32), (count, p.lwe_dim + 1))
    _run(eng, p, ob, lwe, luts, (np.arange(count) % len(luts)).astype(np.uint32), generator)


@pytest.mark.parametrize("mlk", [2, 4, 8])
@pytest.mark.parametrize("count", [3, 21])
def test_many_lut_outputs(setup, mlk, count):
    p, keys, eng, ob = setup
    rng = np.random.default_rng(mlk)
    luts = np.stack([L.lut_build(p, rng.integers(0, 16, 16).astype(np.uint32)) for _ in range(3)])
    ids = rng.integers(0, 3, count).astype(np.uint32)
    ct = L.encrypt(p, keys["glwe_key"], rng.integers(0, 16 // mlk, count).astype(np.uint32), 5)
    eng.upload_luts(luts)
    d_out = to_dev(np.zeros((count * mlk, N + 1), np.uint64))
    eng.ks_pbs_ml(to_dev(ct), to_dev(ids), d_out, count, mlk)
    eng.check_device_error()
    assert np.array_equal(from_dev(d_out, np.uint64), ob.ks_pbs(keys["ksk"], ct, luts, ids, pbs_bl=p.pbs_base_log, mlk=mlk))


@pytest.mark.parametrize("count", [1, 20])
def test_lut_id_out_of_range_is_reported(setup, count):
    p, keys, eng, ob = setup
    ids = np.zeros(count, np.uint32)
    ids[-1] = 5
    eng.upload_luts(L.lut_build(p, np.arange(16, dtype=np.uint32))[None])
    d_out = to_dev(np.zeros((count, N + 1), np.uint64))
    eng.blind_rotate(to_dev(np.zeros((count, p.lwe_dim + 1), np.uint32)), to_dev(ids), d_out, count)
    with pytest.raises(L.LutheError) as ei:
        eng.check_device_error()
    assert ei.value.code == L.E_PARAM
