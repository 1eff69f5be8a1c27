"""The tensor-core blind rotation (batches above one ciphertext per SM): every
output word equal to the oracle's, at the edges of its tiles (128 ciphertexts),
its couples of ciphertexts, its launches (592) and of the rule that hands
remainders to the butterfly kernels, in both tie rules, both PBS bases and with
many-LUT outputs.  A short LWE key (24 steps) keeps the oracle quick: the
kernel's step loop does not depend on n."""
import numpy as np
import pytest

import luthe_b200 as L
import oracle
from conftest import from_dev, to_dev

pytestmark = pytest.mark.gpu
N, STEPS = 2048, 24


@pytest.fixture(scope="module", params=[23, 22])
def setup(request):
    p = L.default_params(lwe_dim=STEPS, pbs_base_log=request.param)
    keys = L.keygen(p, 17)
    eng = L.Engine(p)
    eng.upload_keys(keys)
    yield p, keys, eng, oracle.OracleBsk(keys["bsk"], STEPS, N)
    eng.close()


def _nsm():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


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


# one more than the SM count (odd: a half-empty couple), around the tiles, one
# and two couples per CTA, the largest launch, a launch and remainders of one
# ciphertext and of one launch more
@pytest.mark.parametrize("count", ["nsm+1", 255, 256, 257, 297, 385, 592, 593, 592 + 300])
def test_every_output_equals_the_oracle(setup, count):
    p, keys, eng, ob = setup
    count = _nsm() + 1 if count == "nsm+1" else count
    rng = np.random.default_rng(count)
    lwe = rng.integers(0, 2 * N, (count, STEPS + 1), dtype=np.uint32)
    lwe[0] = 0
    lwe[-1] = 2 * N - 1
    luts = rng.integers(0, 2**64, (3, 2 * N), dtype=np.uint64)
    _run(eng, p, ob, lwe, luts, rng.integers(0, 3, count).astype(np.uint32), generator=count % 2 == 0)


@pytest.mark.parametrize("generator", [False, True])
def test_ties_and_extreme_words(setup, generator):
    """LUT words whose differences meet the decomposition's ties (a top digit of
    B/2 with and without the rounding bit), its rounding points and the ends of
    the torus, under rotations by 0, N and both ends."""
    p, keys, eng, ob = setup
    bw, count = p.pbs_base_log, _nsm() + 12
    rng = np.random.default_rng(7)
    half = 1 << (63 - bw)  # the rounding bit
    words = [0, 1, 1 << 63, (1 << 63) - 1, (1 << 63) - half, (1 << 63) - half - 1, (1 << 63) + half, half, half - 1,
             2**64 - 1, 2**64 - half, 1 << 62, 3 << 62, 0xFFFFFFFF00000000, 0xFFFFFFFF]
    luts = np.stack([np.full(2 * N, w, np.uint64) for w in words] +
                    [rng.choice(np.array(words, np.uint64), 2 * N) for _ in range(5)])
    lwe = rng.choice(np.array([0, 1, N - 1, N, N + 1, 2 * N - 1], np.uint32), (count, STEPS + 1))
    _run(eng, p, ob, lwe, luts, (np.arange(count) % len(luts)).astype(np.uint32), generator)


@pytest.mark.parametrize("mlk", [2, 8])
def test_many_lut_outputs(setup, mlk):
    p, keys, eng, ob = setup
    count = _nsm() + 5
    rng = np.random.default_rng(mlk)
    luts = np.stack([L.lut_build(p, rng.integers(0, 16, 16).astype(np.uint32)) for _ in range(3)])
    ids = rng.integers(0, 3, count).astype(np.uint32)
    ct = L.encrypt(p, keys["glwe_key"], rng.integers(0, 16 // mlk, count).astype(np.uint32), 5)
    eng.upload_luts(luts)
    d_out = to_dev(np.zeros((count * mlk, N + 1), np.uint64))
    eng.ks_pbs_ml(to_dev(ct), to_dev(ids), d_out, count, mlk)
    eng.check_device_error()
    assert np.array_equal(from_dev(d_out, np.uint64), ob.ks_pbs(keys["ksk"], ct, luts, ids, pbs_bl=p.pbs_base_log, mlk=mlk))


def test_lut_id_out_of_range_is_reported(setup):
    p, keys, eng, ob = setup
    count = _nsm() + 2
    ids = np.zeros(count, np.uint32)
    ids[-1] = 5
    eng.upload_luts(L.lut_build(p, np.arange(16, dtype=np.uint32))[None])
    d_out = to_dev(np.zeros((count, N + 1), np.uint64))
    eng.blind_rotate(to_dev(np.zeros((count, STEPS + 1), np.uint32)), to_dev(ids), d_out, count)
    with pytest.raises(L.LutheError) as ei:
        eng.check_device_error()
    assert ei.value.code == L.E_PARAM


def test_budget_without_room_for_the_expanded_key(setup):
    """The expanded key and its workspace are optional: a context without room
    for them, and one that gives them up for a later allocation, compute the
    same outputs on the butterfly kernels."""
    p, keys, eng, ob = setup
    count = _nsm() + 3
    rng = np.random.default_rng(3)
    lwe = rng.integers(0, 2 * N, (count, STEPS + 1), dtype=np.uint32)
    luts = rng.integers(0, 2**64, (1, 2 * N), dtype=np.uint64)
    ids = np.zeros(count, np.uint32)
    full = eng.device_bytes
    with L.Engine(p, hbm_budget=64 << 20) as small:
        small.upload_keys(keys)
        assert small.device_bytes < 64 << 20
        _run(small, p, ob, lwe, luts, ids, False)
    with L.Engine(p, hbm_budget=full + (8 << 20)) as tight:
        tight.upload_keys(keys)
        had = tight.device_bytes
        _run(tight, p, ob, lwe, luts, ids, False)
        tight.reserve(1 << 20)  # does not fit beside them
        assert tight.device_bytes < had + (1 << 20) * (STEPS + 1) * 4
        _run(tight, p, ob, lwe, luts, ids, False)
