"""Calls of one context on streams that nothing orders: large blind rotations and
key switches take turns at the buffers of the tensor-core forms, and a replayed
capture of either runs beside them on buffers of its own."""
import numpy as np
import pytest

import luthe_b200 as L
import oracle
from conftest import from_dev, to_dev

pytestmark = pytest.mark.gpu
N, STEPS, COUNT = 2048, 24, 300


@pytest.fixture(scope="module")
def setup():
    p = L.default_params(lwe_dim=STEPS)
    keys = L.keygen(p, 31)
    luts = np.random.default_rng(31).integers(0, 2**64, (2, 2 * N), dtype=np.uint64)
    with L.Engine(p) as eng:
        eng.upload_keys(keys)
        eng.upload_luts(luts)
        yield eng, keys, luts, oracle.OracleBsk(keys["bsk"], STEPS, N)


class Job:
    """One call's inputs, outputs and expected outputs."""

    def __init__(self, setup, kind, seed):
        self.eng, keys, luts, ob = setup
        self.kind, rng = kind, np.random.default_rng(seed)
        if kind == "blind_rotate":
            lwe = rng.integers(0, 2 * N, (COUNT, STEPS + 1), dtype=np.uint32)
            ids = rng.integers(0, 2, COUNT).astype(np.uint32)
            self.args = to_dev(lwe), to_dev(ids), to_dev(np.zeros((COUNT, N + 1), np.uint64))
            self.out, self.want = self.args[2], ob.blind_rotate(lwe, luts, ids)
        else:
            x = rng.integers(0, 2**64, (COUNT, N + 1), dtype=np.uint64)
            self.args = to_dev(x), None, to_dev(np.zeros((COUNT, STEPS + 1), np.uint32))
            self.out = self.args[2]
            self.want = np.stack([oracle.keyswitch(row, keys["ksk"], STEPS, N)[1] for row in x])

    def run(self, stream):
        getattr(self.eng, self.kind)(*self.args, COUNT, stream)

    def check(self):
        assert np.array_equal(from_dev(self.out, self.want.dtype), self.want)


@pytest.mark.parametrize("kind", ["blind_rotate", "keyswitch"])
def test_unordered_streams(setup, kind):
    import torch
    streams = [torch.cuda.Stream() for _ in range(3)]
    jobs = [Job(setup, kind, k) for k in range(6)]
    torch.cuda.synchronize()
    for k, job in enumerate(jobs):
        job.run(streams[k % 3])
    torch.cuda.synchronize()
    setup[0].check_device_error()
    for job in jobs:
        job.check()


@pytest.mark.parametrize("kind", ["blind_rotate", "keyswitch"])
def test_replays_beside_calls(setup, kind):
    import torch
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    captured, direct = Job(setup, kind, 11), Job(setup, kind, 12)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=a):
        captured.run(a)
    for _ in range(4):
        with torch.cuda.stream(a):
            captured.out.zero_()
            g.replay()
        direct.run(b)
    torch.cuda.synchronize()
    setup[0].check_device_error()
    captured.check()
    direct.check()
    del g


def test_two_contexts(setup):
    """Large batches of two contexts on two streams: each launch needs every SM
    at once, and neither waits for the other's CTAs."""
    import torch
    keys, luts, ob = setup[1:]
    with L.Engine(L.default_params(lwe_dim=STEPS)) as second:
        second.upload_keys(keys)
        second.upload_luts(luts)
        streams = [torch.cuda.Stream() for _ in range(2)]
        jobs = [Job((eng, keys, luts, ob), "blind_rotate", 20 + k) for k, eng in enumerate([setup[0], second] * 4)]
        torch.cuda.synchronize()
        for k, job in enumerate(jobs):
            job.run(streams[k % 2])
        torch.cuda.synchronize()
        for eng in (setup[0], second):
            eng.check_device_error()
        for job in jobs:
            job.check()


@pytest.mark.parametrize("kind", ["blind_rotate", "keyswitch"])
def test_branches_of_one_capture(setup, kind):
    import torch
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    jobs = [Job(setup, kind, 40 + k) for k in range(4)]
    torch.cuda.synchronize()
    for _ in range(2):  # two captures
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=a):
            b.wait_stream(a)
            for k, job in enumerate(jobs):
                job.run((a, b)[k % 2])
            a.wait_stream(b)
        for job in jobs:
            job.out.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        setup[0].check_device_error()
        for job in jobs:
            job.check()
        del g
