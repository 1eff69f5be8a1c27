"""Host logic of the context on the CPU: luthe_b200/csrc/api.cu compiled against
a fake CUDA runtime (tests/ctx_harness) that knows which operations are ordered
before which.  Kernels do nothing; the GPU tests cover them."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import luthe_b200 as L

HERE = os.path.dirname(os.path.abspath(__file__))
N, STEPS = 2048, 2
vp, sz = ctypes.c_void_p, ctypes.c_size_t


@pytest.fixture(scope="module")
def lib():
    subprocess.run([os.path.join(HERE, "ctx_harness", "build.sh")], check=True)
    h = ctypes.CDLL(os.path.join(HERE, "ctx_harness", "libctx_harness.so"))
    h.harness_stream.restype = h.harness_end_capture.restype = vp
    h.harness_begin_capture.argtypes = h.harness_end_capture.argtypes = [vp]
    h.harness_replay.argtypes = [vp, vp]
    h.harness_limit.argtypes = [vp]
    h.harness_fork.argtypes = [vp, vp]
    h.harness_fail_brx.argtypes = [ctypes.c_int]
    h.harness_fail_malloc.argtypes = [ctypes.c_int, ctypes.c_int]
    h.harness_fail_optional.argtypes = [ctypes.c_int, ctypes.c_int]
    h.harness_bsk_words.argtypes = [vp, vp, vp]
    h.luthe_ctx_create.argtypes = [vp, ctypes.c_int, ctypes.c_uint64, ctypes.POINTER(vp)]
    h.luthe_ctx_destroy.argtypes = [vp]
    h.luthe_device_bytes.argtypes = [vp]
    h.luthe_device_bytes.restype = ctypes.c_uint64
    for name in ("bsk", "bsk_eval", "ksk"):
        getattr(h, f"luthe_upload_{name}").argtypes = [vp, vp]
    h.luthe_upload_luts.argtypes = [vp, vp, ctypes.c_uint32]
    for name in ("ks_pbs", "ks_pbs_graph", "ks_pbs_noalloc"):
        getattr(h, f"luthe_{name}").argtypes = [vp, vp, vp, vp, sz, vp]
    h.luthe_keyswitch.argtypes = [vp, vp, vp, vp, sz, vp]
    h.luthe_blind_rotate.argtypes = [vp, vp, vp, vp, sz, vp]
    return h


class Ctx:
    """A context with keys; calls pass pointers that the fake kernels never read."""

    def __init__(self, lib, keys=True, budget=0):
        self.lib, self.params = lib, L.default_params(lwe_dim=STEPS)
        lib.harness_reset()
        self.h = vp()
        assert lib.luthe_ctx_create(ctypes.byref(self.params), 0, budget, ctypes.byref(self.h)) == 0
        self.ksk = np.zeros((STEPS + 1) * N * self.params.ks_level, np.uint32)
        if keys:
            assert self.upload_bsk(1) == 0 and self.upload_ksk() == 0 and self.upload_luts() == 0

    def upload_bsk(self, word, form="bsk"):
        key = np.full(STEPS * 4 * N, word, np.uint64)
        return getattr(self.lib, f"luthe_upload_{form}")(self.h, key.ctypes.data)

    def upload_ksk(self):
        return self.lib.luthe_upload_ksk(self.h, self.ksk.ctypes.data)

    def upload_luts(self):
        lut = np.zeros(2 * N, np.uint64)
        return self.lib.luthe_upload_luts(self.h, lut.ctypes.data, 1)

    def call(self, name, count, stream):
        p = vp(64)
        return getattr(self.lib, f"luthe_{name}")(self.h, p, p, p, count, stream)

    def log(self):
        buf = ctypes.create_string_buffer(1 << 16)
        self.lib.harness_log(buf, len(buf))
        return buf.value.decode().rstrip(";").split(";")

    def close(self):
        self.lib.luthe_ctx_destroy(self.h)


@pytest.fixture
def ctx(lib):
    c = Ctx(lib)
    yield c
    c.close()


@pytest.mark.parametrize("name,count", [("keyswitch", 1), ("keyswitch", 4000), ("blind_rotate", 149),
                                        ("blind_rotate", 1200), ("ks_pbs_noalloc", 300), ("ks_pbs_graph", 300)])
def test_calls_on_several_streams_take_turns_at_the_buffers(ctx, name, count):
    """Calls on streams that the caller left unordered, the context's own graphs
    among them: no two uses of a buffer of the tensor-core forms may overlap."""
    streams = [ctx.lib.harness_stream() for _ in range(3)] + ([] if name == "ks_pbs_graph" else [None])
    for _ in range(3):
        for s in streams:
            assert ctx.call(name, count, s) == 0
            assert ctx.call("keyswitch", 40, s) == 0
    forms = {f.split()[0] for f in ctx.log()}
    assert "ks_tc" in forms and ("brx" in forms) == (name != "keyswitch")  # the forms in question ran
    assert ctx.lib.harness_races() == 0


@pytest.mark.parametrize("name", ["keyswitch", "blind_rotate", "ks_pbs", "ks_pbs_noalloc"])
def test_captured_launches_have_buffers_of_their_own(ctx, name):
    """A launch that the caller captured may be replayed while the context's
    other calls run: it waits for no event of theirs (a capture refuses that)
    and shares no buffer with them."""
    a, b = ctx.lib.harness_stream(), ctx.lib.harness_stream()
    assert ctx.call(name, 300, b) == 0
    ctx.lib.harness_begin_capture(a)
    assert ctx.call(name, 300, a) == 0
    g = ctx.lib.harness_end_capture(a)
    for _ in range(2):
        ctx.lib.harness_replay(g, a)
        assert ctx.call(name, 300, b) == 0
        assert ctx.call("ks_pbs_graph", 300, b) == 0
    assert ctx.lib.harness_races() == 0


def _bsk_words(ctx):
    w = np.zeros(2, np.uint64)
    ctx.lib.harness_bsk_words(ctx.h, w.ctypes.data, w.ctypes.data + 8)
    return w.tolist()


def test_a_failed_key_upload_leaves_one_key(ctx):
    """The two device forms of the BSK come from one key.  While captured
    launches hold the expanded form, an evaluation-domain upload that finds no
    memory for its copy must leave the key that was there in both."""
    a = ctx.lib.harness_stream()
    ctx.lib.harness_begin_capture(a)
    assert ctx.call("ks_pbs", 300, a) == 0
    ctx.lib.harness_end_capture(a)
    before = _bsk_words(ctx)
    ctx.lib.harness_fail_malloc(0, 2)
    assert ctx.upload_bsk(2, "bsk_eval") == L.E_CUDA
    assert _bsk_words(ctx) == before
    assert ctx.upload_bsk(2, "bsk_eval") == 0
    slab, expanded = _bsk_words(ctx)
    assert slab != before[0] and expanded == 2


def test_a_form_that_cannot_be_set_up_is_done_without(lib):
    """The tensor-core forms are optional: where one cannot be set up, uploads
    succeed, hold nothing for it, and calls run the other form."""
    c = Ctx(lib, keys=False)
    assert c.upload_luts() == 0
    lib.harness_fail_optional(801, 801)
    for _ in range(2):
        assert c.upload_bsk(1) == 0 and c.upload_bsk(1, "bsk_eval") == 0 and c.upload_ksk() == 0
    assert lib.luthe_device_bytes(c.h) < 16 << 20
    assert c.call("ks_pbs", 300, None) == 0
    assert c.log() == ["ks_dp4a 300", "br 300"]
    lib.harness_fail_optional(0, 0)
    assert c.upload_bsk(1) == 0 and c.upload_ksk() == 0
    assert c.call("ks_pbs", 300, None) == 0
    assert c.log() == ["ks_tc 300", "brx 300"]
    c.close()


@pytest.mark.parametrize("name", ["blind_rotate", "ks_pbs", "ks_pbs_graph"])
@pytest.mark.parametrize("count", [1, 20, 149, 1200])
def test_streams_with_some_of_the_SMs(ctx, name, count):
    """On a stream that has some of the SMs only, the tensor-core blind rotation
    (CTAs on every SM that wait for one another) and the clusters of eight and
    four SMs (counted on the whole device) are not launched."""
    s = ctx.lib.harness_stream()
    ctx.lib.harness_limit(s)
    assert ctx.call(name, count, s) == 0
    assert [f for f in ctx.log() if f.startswith("br")] == [f"br {count}"]


def test_a_refused_cooperative_launch_runs_the_other_form(ctx):
    ctx.lib.harness_fail_brx(720)
    assert ctx.call("blind_rotate", 700, ctx.lib.harness_stream()) == 0
    assert ctx.log() == ["br 592", "br 108"]
    ctx.lib.harness_fail_brx(1)  # any other error is reported
    assert ctx.call("blind_rotate", 700, ctx.lib.harness_stream()) == L.E_CUDA


@pytest.mark.parametrize("name,first,direct,captured", [("blind_rotate", "ksk", "brx 300", "br 300"),
                                                        ("keyswitch", "bsk", "ks_tc 300", "ks_dp4a 300")])
def test_a_budget_for_one_set_of_buffers(lib, name, first, direct, captured):
    """A budget that holds a tensor-core form with one set of buffers, not two:
    the context's calls use it, and captured launches take the other form."""
    def uploads(c):
        for key in (first, "ksk" if first == "bsk" else "bsk"):
            assert (c.upload_ksk() if key == "ksk" else c.upload_bsk(1)) == 0
        assert c.upload_luts() == 0
        return c
    probe = uploads(Ctx(lib, keys=False))
    full = lib.luthe_device_bytes(probe.h)
    probe.close()
    c = uploads(Ctx(lib, keys=False, budget=full - (16 << 20)))
    s = lib.harness_stream()
    for _ in range(2):
        assert c.call(name, 300, None) == 0
        assert c.log() == [direct]
        lib.harness_begin_capture(s)
        assert c.call(name, 300, s) == 0
        lib.harness_end_capture(s)
        assert c.log() == [captured]
    assert lib.luthe_device_bytes(c.h) <= full - (16 << 20)
    c.close()


@pytest.mark.parametrize("name", ["keyswitch", "blind_rotate", "ks_pbs_noalloc"])
def test_branches_of_one_capture_take_turns(ctx, name):
    """Calls on the branches of one capture share the set of captured launches:
    no two uses may overlap.  A later capture starts without the earlier one's."""
    for _ in range(2):
        a, b = ctx.lib.harness_stream(), ctx.lib.harness_stream()
        ctx.lib.harness_begin_capture(a)
        ctx.lib.harness_fork(a, b)
        for s in (a, b, b, a):
            assert ctx.call(name, 300, s) == 0
        ctx.lib.harness_end_capture(b)
        ctx.lib.harness_end_capture(a)
    assert ctx.lib.harness_races() == 0
