"""The launch forms that batches take where the context has no room for the
tensor-core forms: one and two ciphertexts per CTA in whole waves and with a
tail, the autotuned shape, the dp4a key switch in one pass and split over K; and
every form's bounded wait made to run out.  A budget of 20 MB holds a key of 90
steps (two column tiles of the key switch) and nothing optional."""
import os
import subprocess
import sys
import textwrap

import numpy as np
import pytest

import luthe_b200 as L
import oracle
from conftest import from_dev, to_dev

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
N, STEPS, BUDGET = 2048, 90, 20 << 20


@pytest.fixture(scope="module")
def setup():
    p = L.default_params(lwe_dim=STEPS)
    keys = L.keygen(p, 37)
    luts = np.random.default_rng(37).integers(0, 2**64, (3, 2 * N), dtype=np.uint64)
    with L.Engine(p, hbm_budget=BUDGET) as eng:
        eng.upload_keys(keys)
        eng.upload_luts(luts)
        assert eng.device_bytes < 12 << 20  # no optional form
        yield eng, keys, luts, oracle.OracleBsk(keys["bsk"], STEPS, N)


def _rotate(setup, count):
    eng, keys, luts, ob = setup
    rng = np.random.default_rng(count)
    lwe = rng.integers(0, 2 * N, (count, STEPS + 1), dtype=np.uint32)
    ids = rng.integers(0, 3, count).astype(np.uint32)
    d_out = to_dev(np.zeros((count, N + 1), np.uint64))
    eng.blind_rotate(to_dev(lwe), to_dev(ids), d_out, count)
    eng.check_device_error()
    got, want = from_dev(d_out, np.uint64), ob.blind_rotate(lwe, luts, ids)
    assert np.array_equal(got, want), np.nonzero((got != want).any(1))[0]


# on 148 SMs: half an SM each, a wave and a small tail (one SM each, pairs, clusters), two waves, and a larger tail
@pytest.mark.parametrize("cts_per_cta", [1, 2])
@pytest.mark.parametrize("count", [149, 296, 301, 330, 360, 444, 450, 593])
def test_waves_and_tails(setup, cts_per_cta, count):
    eng = setup[0]
    eng.set_br_config(cts_per_cta, 1)
    try:
        _rotate(setup, count)
    finally:
        eng.set_br_config(2, 1)


def test_autotuned_shape(setup):
    eng = setup[0]
    assert eng.autotune(518)["chosen"]["cts_per_cta"] in (1, 2)
    try:
        for count in (30, 100, 148, 220, 356, 518):
            _rotate(setup, count)
    finally:
        eng.set_br_config(2, 1)


@pytest.mark.parametrize("count", [1, 5, 32, 33, 70])
def test_dp4a_key_switch(setup, count):
    eng, keys = setup[:2]
    x = np.random.default_rng(count).integers(0, 2**64, (count, N + 1), dtype=np.uint64)
    want = [oracle.keyswitch(row, keys["ksk"], STEPS, N) for row in x]
    for _ in range(2):  # the partial sums are left clear
        d21, d2n = (to_dev(np.zeros((count, STEPS + 1), np.uint32)) for _ in range(2))
        eng.keyswitch(to_dev(x), d21, d2n, count)
        assert np.array_equal(from_dev(d21, np.uint32), np.stack([w[0] for w in want]))
        assert np.array_equal(from_dev(d2n, np.uint32), np.stack([w[1] for w in want]))


CHILD = textwrap.dedent("""
    import sys
    sys.path.insert(0, ROOT)
    import numpy as np
    import torch
    import luthe_b200 as L

    p = L.default_params(lwe_dim=STEPS)
    keys = L.keygen(p, 5)
    # clusters of eight, of four, pairs, one per SM, tensor cores; then two per CTA alone, with a tail, one per CTA
    for budget, g, counts in ((0, 2, (4, 20, 60, 120, 300)), (BUDGET, 2, (296, 301, 420)), (BUDGET, 1, (200,))):
        eng = L.Engine(p, hbm_budget=budget)
        eng.upload_keys(keys)
        eng.upload_luts(L.lut_build(p, np.arange(16, dtype=np.uint32))[None])
        eng.set_br_config(g, 1)
        for count in counts:
            d_in = torch.zeros((count, STEPS + 1), dtype=torch.int32, device="cuda")
            d_ids = torch.zeros(count, dtype=torch.int32, device="cuda")
            d_out = torch.zeros((count, p.poly_size + 1), dtype=torch.int64, device="cuda")
            eng.blind_rotate(d_in, d_ids, d_out, count)
            torch.cuda.synchronize()
            try:
                eng.check_device_error()
            except L.LutheError as e:
                assert e.code == L.E_TIMEOUT and "unsafe" not in str(e), e
            else:
                raise SystemExit(f"no timeout reported for {count} ciphertexts")
            eng.check_device_error()  # the flag was cleared
        eng.close()
    print("ok")
""").replace("ROOT", repr(ROOT)).replace("STEPS", str(STEPS)).replace("BUDGET", str(BUDGET))


def test_every_form_reports_a_wait_that_ran_out():
    env = dict(os.environ, LUTHE_SLAB_WAIT_POLLS="0")
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout[-2000:] + r.stderr[-2000:]
