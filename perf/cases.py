"""The workloads the engine's speed is measured on: calls that a program makes
through the public entry points of luthe_b200, over the sizes such programs use.

A case is a dict of plain values.  Kinds:

  pbs     Engine.ks_pbs / ks_pbs_ml on device buffers: the batched PBS DOp
  host    Engine.ks_pbs_host: the same from and to host buffers
  ks      Engine.keyswitch on its own
  ntt     Engine.ntt_fwd and Engine.ntt_inv (one of each)
  nttmul  Engine.ntt_mul: negacyclic products of polynomial pairs
  lwe     Engine.lwe_op: a linear DOp on a batch of BLWEs
  serve   Server.run: 16-bit integer operations as DOp programs
"""
import numpy as np
import torch

import luthe_b200 as L
from luthe_b200 import iops

N = 2048
P = 0xFFFFFFFF00000001
PSI = 0x984EC5194D005735  # the 4096-th root of unity of luthe_ntt_fwd
SETS = ["default", "msg2_carry2_pfail64_132b_gaussian_1f72dba", "msg2_carry2_pfail64_132b_tuniform_7e47d8c",
        "msg2_carry2_gaussian", "msg2_carry2_tuniform"]
OPS = {"add": L.OP_ADD, "sub": L.OP_SUB, "mac": L.OP_MAC, "adds": L.OP_ADDS, "subs": L.OP_SUBS,
       "ssub": L.OP_SSUB, "muls": L.OP_MULS}
TWO_INPUTS = ("add", "sub", "mac")


def listed():
    return [
        # one bootstrap alone: the latency of a single PBS DOp
        {"name": "pbs_1", "kind": "pbs", "count": 1, "set": "default", "mlk": 1, "tie": "rtl"},
        # a small odd batch with two functions per rotation (PBS_ML2), the
        # carry + message extraction of the radix programs
        {"name": "pbs_17_ml2", "kind": "pbs", "count": 17, "set": "default", "mlk": 2, "tie": "rtl"},
        # a middling batch on the reference's largest parameter set (n = 887,
        # PBS 2^22, KS 3x5), in the tie rule of the reference's generator
        {"name": "pbs_256_tuniform", "kind": "pbs", "count": 256, "set": "msg2_carry2_tuniform", "mlk": 1,
         "tie": "generator"},
        # the larger batches of the benchmark's uneven mix, where throughput counts
        {"name": "pbs_1000", "kind": "pbs", "count": 1000, "set": "default", "mlk": 1, "tie": "rtl"},
        {"name": "pbs_4096", "kind": "pbs", "count": 4096, "set": "default", "mlk": 1, "tie": "rtl"},
        # ciphertexts that live in host memory, copied in and out in the call
        {"name": "host_601", "kind": "host", "count": 601, "set": "default"},
        # key switches on their own: one request's worth, and the largest
        # batch of the benchmark's configurations
        {"name": "ks_65_2x7", "kind": "ks", "count": 65, "set": "msg2_carry2_pfail64_132b_tuniform_7e47d8c",
         "tie": "rtl"},
        {"name": "ks_16384", "kind": "ks", "count": 16384, "set": "default", "tie": "rtl"},
        # both transforms on an odd number of polynomials (key preparation,
        # plaintext products kept in the evaluation domain)
        {"name": "ntt_333", "kind": "ntt", "count": 333},
        # the benchmark's polynomial products
        {"name": "nttmul_4096", "kind": "nttmul", "count": 4096},
        # linear DOps: a multiply-accumulate over a large batch
        {"name": "lwe_mac_4096", "kind": "lwe", "op": "mac", "count": 4096, "imm": 4},
        # a handful of concurrent requests through the serving loop
        {"name": "serve_6", "kind": "serve", "count": 6},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choice(["pbs", "pbs", "pbs", "host", "ks", "ks", "ntt", "nttmul", "lwe", "serve"])
    if kind == "pbs":
        return {"kind": kind, "count": _log(rng, 1, 3500), "set": rng.choice(SETS), "mlk": rng.choice([1, 1, 2, 4, 8]),
                "tie": rng.choice(["rtl", "generator"])}
    if kind == "host":
        return {"kind": kind, "count": _log(rng, 1, 1500), "set": rng.choice(SETS)}
    if kind == "ks":
        return {"kind": kind, "count": _log(rng, 1, 16384), "set": rng.choice(SETS),
                "tie": rng.choice(["rtl", "generator"])}
    if kind in ("ntt", "nttmul"):
        return {"kind": kind, "count": _log(rng, 1, 4096)}
    if kind == "lwe":
        return {"kind": kind, "op": rng.choice(sorted(OPS)), "count": _log(rng, 1, 8192), "imm": rng.randrange(1, 16)}
    return {"kind": kind, "count": rng.randrange(1, 13)}


# ------------------------------------------------------------------ inputs

def _tie(case):
    return L.TIE_GENERATOR if case.get("tie") == "generator" else L.TIE_RTL


def _words(seed, shape):
    """Uniform 64-bit words (BLWE words are uniform on the torus)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(-2**63, 2**63 - 1, shape, dtype=torch.int64, device="cuda", generator=g)


def _residues(seed, shape):
    """Uniform residues mod p as 64-bit words."""
    w = _words(seed, shape)
    return torch.where(_ge_p(w), w - (P - 2**64), w)


def _ksk(params, seed):
    """Key-switch key words: uniform mod 2^21 but for the bodies, which hide among them."""
    rng = np.random.default_rng(seed)
    k = rng.integers(0, 1 << 21, (params.lwe_dim + 1) * N * params.ks_level, dtype=np.uint32)
    return k


def _messages(case, params, keys, seed):
    """Encrypted messages, LUT ids and four random LUTs (mlk functions packed in each)."""
    rng = np.random.default_rng(seed)
    mlk, count = case.get("mlk", 1), case["count"]
    luts = np.stack([L.lut_build(params, rng.integers(0, 16, 16).astype(np.uint32)) for _ in range(4)])
    msgs = rng.integers(0, 16 // mlk, count).astype(np.uint32)
    ids = rng.integers(0, 4, count).astype(np.uint32)
    return L.encrypt(params, keys["glwe_key"], msgs, seed + 1), ids, luts


def prepare(case, seed):
    kind, count = case["kind"], case["count"]
    st = {"case": case}
    if kind in ("pbs", "host", "serve"):
        params = L.param_set(case.get("set", "default"))
        keys = L.keygen(params, seed)
        eng = L.Engine(params)
        eng.upload_keys(keys)
        st["eng"] = eng
        if kind == "serve":
            eng.upload_luts(np.stack([L.lut_build(params, t) for t in iops.lut_tables()]))
            st["server"] = L.Server(eng, pool_bytes=1 << 28, max_pbs=512)
            st["requests"] = _requests(params, keys, count, seed)
            return st
        eng.set_tie_rule(_tie(case))
        ct, ids, luts = _messages(case, params, keys, seed)
        eng.upload_luts(luts)
        eng.reserve(count)
        if kind == "host":
            st["in"] = torch.from_numpy(ct.view(np.int64)).pin_memory()
            st["out"] = torch.empty_like(st["in"]).pin_memory()
            st["args"] = (st["in"].numpy().view(np.uint64), ids, st["out"].numpy().view(np.uint64))
            return st
        st["in"] = torch.from_numpy(ct.view(np.int64)).cuda()
        st["ids"] = torch.from_numpy(ids.view(np.int32)).cuda()
        st["out"] = torch.empty((count * case["mlk"], N + 1), dtype=torch.int64, device="cuda")
        return st
    params = L.param_set(case.get("set", "default"))
    eng = st["eng"] = L.Engine(params)
    if kind == "ks":
        eng.upload_ksk(_ksk(params, seed))
        eng.set_tie_rule(_tie(case))
        st["in"] = _words(seed, (count, N + 1))
        st["out21"] = torch.empty((count, params.lwe_dim + 1), dtype=torch.int32, device="cuda")
        st["out2n"] = torch.empty_like(st["out21"])
    elif kind == "lwe":
        st["a"] = _words(seed, (count, N + 1))
        st["b"] = _words(seed + 1, (count, N + 1)) if case["op"] in TWO_INPUTS else None
        st["out"] = torch.empty_like(st["a"])
    else:
        st["a"] = _residues(seed, (count, N))
        st["b"] = _residues(seed + 1, (count, N))
        st["out"] = torch.empty_like(st["a"])
        st["out2"] = torch.empty_like(st["a"])
    return st


def _requests(params, keys, count, seed):
    """16-bit operations as the serving loop gets them: adds, compares with a
    constant and multiplies in turn, on random operands."""
    rng = np.random.default_rng(seed)
    reqs = []
    for r in range(count):
        a, b = (int(v) for v in rng.integers(0, 65536, 2))
        blocks = iops.to_blocks(a) + iops.to_blocks(b)
        if r % 3 == 0:
            prog, n_dst = iops.prog_add(), 8
        elif r % 3 == 1:
            prog, n_dst, blocks = iops.prog_cmp_gt(b), 1, iops.to_blocks(a)
        else:
            prog, n_dst = iops.prog_mul(), 8
        src = L.encrypt(params, keys["glwe_key"], np.array(blocks, np.uint32), seed + 10 + r)
        reqs.append((prog, src, n_dst))
    return reqs


# --------------------------------------------------------------------- run

def run(st):
    case, eng = st["case"], st.get("eng")
    kind, count, s = case["kind"], case["count"], torch.cuda.current_stream()
    if kind == "pbs":
        if case["mlk"] == 1:
            eng.ks_pbs(st["in"], st["ids"], st["out"], count, s)
        else:
            eng.ks_pbs_ml(st["in"], st["ids"], st["out"], count, case["mlk"], s)
        return st["out"]
    if kind == "host":
        eng.ks_pbs_host(*st["args"])
        return st["out"]
    if kind == "serve":
        return [torch.from_numpy(o.view(np.int64)) for o in st["server"].run(st["requests"])]
    if kind == "ks":
        eng.keyswitch(st["in"], st["out21"], st["out2n"], count, s)
        return [st["out21"], st["out2n"]]
    if kind == "ntt":
        eng.ntt_fwd(st["a"], st["out"], count, s)
        eng.ntt_inv(st["b"], st["out2"], count, s)
        return [st["out"], st["out2"]]
    if kind == "nttmul":
        eng.ntt_mul(st["a"], st["b"], st["out"], count, s)
        return st["out"]
    eng.lwe_op(OPS[case["op"]], st["a"], st["b"], st["out"], case["imm"], count, s)
    return st["out"]


# -------------------------------------------------------------------- work

# multiplies mod p of one transform (N/2 log2 N) and of one blind-rotation
# step (four transforms and the 2 x 2 products), two operations each
_NTT = N // 2 * 11
_STEP = 4 * _NTT + 4 * N
_PBS_OF = {0: 8, 1: 15, 2: 101}  # PBS of an add, a compare and a multiply


def work(case):
    kind, count = case["kind"], case["count"]
    p = L.PARAM_SETS[case.get("set", "default")]
    n, ks_l = p["lwe_dim"], p["ks_level"]
    row = (N + 1) * 8
    ksk = (n + 1) * N * ks_l * 21 // 8
    ks_flops = 2 * N * ks_l * (n + 1)
    if kind in ("pbs", "host"):
        outs = count * case.get("mlk", 1)
        return {"bytes": count * (row + 4) + outs * row + ksk + n * 4 * N * 8,
                "flops": count * (ks_flops + 2 * n * _STEP)}
    if kind == "serve":
        pbs = sum(_PBS_OF[r % 3] for r in range(count))
        return {"bytes": pbs * 2 * row + ksk + n * 4 * N * 8, "flops": pbs * (ks_flops + 2 * n * _STEP)}
    if kind == "ks":
        return {"bytes": count * (row + 8 * (n + 1)) + ksk, "flops": count * ks_flops}
    if kind == "ntt":
        return {"bytes": 4 * count * N * 8, "flops": 2 * count * 2 * _NTT}
    if kind == "nttmul":
        return {"bytes": 3 * count * N * 8, "flops": count * 2 * (3 * _NTT + N)}
    return {"bytes": count * row * (3 if case["op"] in TWO_INPUTS else 2), "flops": 2 * count * (N + 1)}


# ------------------------------------------------------------------- exact
#
# Plain 64-bit torch.  Words are unsigned 64-bit values carried in int64.

_LOW = 0xFFFFFFFF
_SIGN = -2**63


def _srl(x, k):
    return (x >> k) & ((1 << (64 - k)) - 1)


def _lt(a, b):
    """a < b as unsigned words"""
    return (a ^ _SIGN) < (b ^ _SIGN)


def _ge_p(a):
    return ~_lt(a, torch.full_like(a, P - 2**64))


def _canon(a):
    return torch.where(_ge_p(a), a - (P - 2**64), a)


def _addp(a, b):
    s = a + b
    return torch.where(_lt(s, a), s + _LOW, _canon(s))  # 2^64 = 2^32 - 1 mod p; a, b < p


def _subp(a, b):
    return torch.where(_lt(a, b), a - b + (P - 2**64), a - b)


def _mulp(a, b):
    a0, a1, b0, b1 = a & _LOW, _srl(a, 32), b & _LOW, _srl(b, 32)
    p00, p01, p10, p11 = a0 * b0, a0 * b1, a1 * b0, a1 * b1
    mid = _srl(p00, 32) + (p01 & _LOW) + (p10 & _LOW)
    lo = (p00 & _LOW) | (mid << 32)
    hi = p11 + _srl(p01, 32) + _srl(p10, 32) + _srl(mid, 32)
    h0, h1 = hi & _LOW, _srl(hi, 32)
    return _addp(_subp(_canon(lo), h1), _canon(h0 * _LOW))  # 2^96 = -1


def _i64(v):
    return v - 2**64 if v >= 2**63 else v


def _ntt_cyclic(a, w):
    """sum_j a_j w^(jk) over the last axis (length a power of two), w a root of that order."""
    n = a.shape[-1]
    if n == 1:
        return a
    even, odd = _ntt_cyclic(a[..., 0::2].contiguous(), w * w % P), _ntt_cyclic(a[..., 1::2].contiguous(), w * w % P)
    t = torch.tensor([_i64(pow(w, k, P)) for k in range(n // 2)], dtype=torch.int64, device=a.device)
    m = _mulp(odd, t)
    return torch.cat([_addp(even, m), _subp(even, m)], -1)


def _powers(w, device):
    return torch.tensor([_i64(pow(w, j, P)) for j in range(N)], dtype=torch.int64, device=device)


def _forward(a):
    return _ntt_cyclic(_mulp(a, _powers(PSI, a.device)), PSI * PSI % P)


def _inverse(a):
    inv = pow(PSI, P - 2, P)
    y = _mulp(_ntt_cyclic(a, inv * inv % P), _powers(inv, a.device))
    return _mulp(y, torch.full_like(y[:1, :1], _i64(pow(N, P - 2, P))))


def _ks_digits(v, bl, lv, generator):
    """Balanced base-2^bl digits of the top bl*lv bits, least significant first."""
    tot = bl * lv
    half, base = 1 << (bl - 1), 1 << bl
    rb = _srl(v, 63 - tot) & 1
    c = _srl(v, 64 - tot) + rb
    msb, low = (c >> (tot - 1)) & 1, c & ((1 << (tot - 1)) - 1)
    top = torch.zeros_like(c) if generator else msb & ((low > 0).long() | rb)
    carry, digits = torch.zeros_like(c), []
    for i in range(lv):
        raw = (c >> (bl * i)) & (base - 1)
        nxt = (c >> (bl * (i + 1))) & (base - 1) if i + 1 < lv else top * (base - 1)
        t = raw + carry
        # above B/2: negative; at B/2: the sign of the digit above decides
        neg = (t > half) | ((t == half) & ((nxt & half) > 0))
        digits.append(torch.where(neg, t - base, t))
        carry = neg.long()
    return torch.stack(digits, -1)


def _exact_ks(case, seed):
    params = L.param_set(case["set"])
    n, lv = params.lwe_dim, params.ks_level
    x = _words(seed, (case["count"], N + 1))
    key = torch.from_numpy(_ksk(params, seed).view(np.int32)).cuda().view(n + 1, N * lv).t().double()
    out21 = []
    for rows in x.split(2048):
        d = _ks_digits(rows[:, :N], params.ks_base_log, lv, case["tie"] == "generator").reshape(len(rows), -1)
        s = -(d.double() @ key).long()  # below 2^38: exact in 64 bits
        s[:, n] += _srl(rows[:, N], 43) + (_srl(rows[:, N], 42) & 1)
        out21.append(s & ((1 << 21) - 1))
    o = torch.cat(out21)
    return [o.int(), (((o >> 9) + ((o >> 8) & 1)) & 4095).int()]


def exact(case, seed):
    kind, count = case["kind"], case["count"]
    if kind in ("pbs", "host", "serve"):
        return None  # hundreds of chained transforms: minutes in plain torch
    if kind == "ks":
        return _exact_ks(case, seed)
    if kind == "lwe":
        a = _words(seed, (count, N + 1))
        b = _words(seed + 1, (count, N + 1)) if case["op"] in TWO_INPUTS else None
        cst = torch.zeros_like(a[:1])
        cst[:, N] = _i64((case["imm"] << 59) % 2**64)
        return {"add": lambda: a + b, "sub": lambda: a - b, "mac": lambda: a * case["imm"] + b,
                "adds": lambda: a + cst, "subs": lambda: a - cst, "ssub": lambda: cst - a,
                "muls": lambda: a * case["imm"]}[case["op"]]()
    a, b = _residues(seed, (count, N)), _residues(seed + 1, (count, N))
    if kind == "ntt":
        return [_forward(a), _inverse(b)]
    return _inverse(_mulp(_forward(a), _forward(b)))
