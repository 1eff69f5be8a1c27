"""Linear DOps on buffers that lie alike to 16 bytes (on the boundary and 8 bytes
off it), on buffers that lie differently (word by word), in place, and at
counts around a CTA's share (1024 pairs of words, 2049 words a BLWE)."""
import numpy as np
import pytest

import luthe_b200 as L

pytestmark = pytest.mark.gpu
W = 2049
OPS = {"add": lambda a, b, m, c: a + b, "sub": lambda a, b, m, c: a - b, "mac": lambda a, b, m, c: a * m + b,
       "adds": lambda a, b, m, c: a + c, "subs": lambda a, b, m, c: a - c, "ssub": lambda a, b, m, c: c - a,
       "muls": lambda a, b, m, c: a * m}


@pytest.fixture(scope="module")
def engine():
    with L.Engine() as e:
        yield e


@pytest.mark.parametrize("op", sorted(OPS))
@pytest.mark.parametrize("offsets", [(0, 0, 0), (1, 1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1)])
@pytest.mark.parametrize("count", [1, 2, 3, 8, 301])
def test_alignments_and_ends(engine, op, offsets, count):
    import torch
    rng = np.random.default_rng(count)
    a, b = (rng.integers(0, 2**64, (count, W), dtype=np.uint64) for _ in range(2))
    imm = np.uint64(11)
    const = np.zeros((count, W), np.uint64)
    const[:, -1] = imm << np.uint64(59)
    want = OPS[op](a, b, imm, const)
    mem = [torch.full((count * W + 3,), 7, dtype=torch.int64, device="cuda") for _ in range(3)]
    view = [m[o: o + count * W] for m, o in zip(mem, offsets)]
    view[0].copy_(torch.from_numpy(a.view(np.int64)).reshape(-1))
    view[1].copy_(torch.from_numpy(b.view(np.int64)).reshape(-1))
    code = getattr(L, "OP_" + op.upper())
    engine.lwe_op(code, view[0], view[1] if op in ("add", "sub", "mac") else None, view[2], int(imm), count)
    assert np.array_equal(view[2].cpu().numpy().view(np.uint64).reshape(count, W), want)
    ends = torch.cat([mem[2][: offsets[2]], mem[2][offsets[2] + count * W:]])
    assert torch.all(ends == 7)  # nothing beyond the output
    engine.lwe_op(code, view[0], view[1] if op in ("add", "sub", "mac") else None, view[0], int(imm), count)  # in place
    assert np.array_equal(view[0].cpu().numpy().view(np.uint64).reshape(count, W), want)
