"""The work that programs built on this framework have it do, as cases that can be timed.

Each case is one call, or the few calls in a row, that a homomorphic-encryption program makes
through ``cupoly_b200.engine.Engine`` or ``cupoly_b200.batch``, with every operand resident on the
GPU.  Ring degrees are powers of two by nature (nphi 2048 .. 32768); the RNS width k, the number
of polynomials and the order of sizes in a mixed batch are what is ragged in use.

Kinds:
  polymul    negacyclic products mod each prime, coefficients in and out (one, or a batch)
  bfv        one BFV homomorphic multiplication per call, the plain drop-in form
  bfv_batch  the batched BFV multiplication of many ciphertext pairs in one call
  mixed      independent products of mixed ring degrees and widths, one CUDA graph
  dgt        forward or inverse transforms of a batch, in place
  relin      relinearization: the xi decomposition of c2 and its dot products with two key halves
  ckks       CKKS multiply, rescale and modulus raising of a batch
  sample     fresh encryption noise: ternary secrets, Gaussian errors, uniform masks, transformed
  io         big-integer coefficients to residues and back (encode and decode)
"""
import numpy as np
import torch

from cupoly_b200.batch import MixedPolymul, random_specs
from cupoly_b200.engine import FORWARD, GAUSSIAN, INVERSE, TERNARY, UNIFORM, BBase, Engine, QBase, QBBase

SIZES = (2048, 4096, 8192, 16384, 32768)


def listed():
    return [
        # A single product per call, as an interactive program or a test makes it: launches and
        # latency are all there is to it.
        {"name": "polymul 4096 k2 x1", "kind": "polymul", "nphi": 4096, "k": 2, "batch": 1},
        # One homomorphic multiplication per call: what a program ported from a per-call library does.
        {"name": "bfv 8192 k5 x1", "kind": "bfv", "nphi": 8192, "k": 5, "t": 256},
        # Batched multiplications at the three parameter sets that the framework is quoted on; the
        # middle one with a ragged batch, the last one the largest that a program keeps resident.
        {"name": "bfv_batch 8192 k5 x128", "kind": "bfv_batch", "nphi": 8192, "k": 5, "t": 256, "batch": 128},
        {"name": "bfv_batch 16384 k10 x37", "kind": "bfv_batch", "nphi": 16384, "k": 10, "t": 256, "batch": 37},
        {"name": "bfv_batch 32768 k16 x64", "kind": "bfv_batch", "nphi": 32768, "k": 16, "t": 65537, "batch": 64},
        # A server's mix of products: 1024 instances, nphi 2048 .. 16384, k 1 .. 8.
        {"name": "mixed 1024", "kind": "mixed", "count": 1024, "kmax": 8, "specs_seed": 12648430},
        # Transforms alone, as key and plaintext preparation calls them: an odd batch of small
        # rings forward, a few wide polynomials of the largest ring back.
        {"name": "dgt forward 4096 k3 x301", "kind": "dgt", "nphi": 4096, "k": 3, "batch": 301, "inverse": False},
        {"name": "dgt inverse 32768 k9 x27", "kind": "dgt", "nphi": 32768, "k": 9, "batch": 27, "inverse": True},
        # Key switching after a batch of multiplications.
        {"name": "relin 8192 k5 x64", "kind": "relin", "nphi": 8192, "k": 5, "batch": 64},
        # CKKS evaluation of a batch of ciphertext polynomials.
        {"name": "ckks 16384 k8 x16", "kind": "ckks", "nphi": 16384, "k": 8, "prec": 55, "batch": 16},
        # Randomness of a batch of fresh encryptions at the largest parameter set.
        {"name": "sample 32768 k16 x16", "kind": "sample", "nphi": 32768, "k": 16, "batch": 16},
        # Encoding and decoding of a batch of messages.
        {"name": "io 8192 k5 x128", "kind": "io", "nphi": 8192, "k": 5, "batch": 128},
    ]


def _log_int(rng, lo, hi):
    """An integer spread evenly over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(("polymul", "bfv", "bfv_batch", "bfv_batch", "mixed", "dgt", "dgt", "relin", "ckks", "sample", "io"))
    if kind == "mixed":
        return {"kind": kind, "count": _log_int(rng, 64, 1024), "kmax": rng.randint(1, 8),
                "specs_seed": rng.randrange(1 << 30)}
    nphi = rng.choice(SIZES)
    k = rng.randint(1, 16)
    # the batch's Q residues take at most `room` bytes: far below the largest listed case's
    room = {"polymul": 1 << 27, "dgt": 1 << 28, "bfv_batch": 1 << 27, "relin": 1 << 26, "ckks": 1 << 26,
            "sample": 1 << 27, "io": 1 << 27, "bfv": 1 << 27}[kind]
    if kind == "ckks":
        k = rng.randint(2, 12)
    if kind == "io":
        k = rng.randint(1, 12)
    most = max(1, room // (8 * nphi * k * (k if kind == "relin" else 1)))
    case = {"kind": kind, "nphi": nphi, "k": k}
    if kind != "bfv":
        case["batch"] = _log_int(rng, 1, min(most, 1024))
    if kind in ("bfv", "bfv_batch"):
        case["t"] = rng.choice((256, 65537))
    if kind == "dgt":
        case["inverse"] = rng.random() < 0.5
    if kind == "ckks":
        case["prec"] = rng.choice((45, 48, 52, 55))
    return case


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)
    return g


def _uniform(out, primes, g):
    """Residue r of every polynomial of out (..., nres, N, 2) uniform in [0, primes[r])."""
    for r, p in enumerate(primes):
        x = out[..., r, :, :]
        x.copy_(torch.randint(0, p, x.shape, generator=g, device="cuda", dtype=torch.int64))
    return out


def prepare(case, seed):
    """Inputs uniform in their range, made from the seed on the GPU; the engine, its outputs and its
    workspace, which a program makes once and keeps."""
    g = _generator(seed)
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "mixed":
        m = MixedPolymul(random_specs(case["count"], case["specs_seed"], kmax=case["kmax"]), kmax=case["kmax"])
        for grp in m.groups.values():
            primes = torch.tensor(grp["engine"].Q, dtype=torch.int64, device="cuda")
            lim = primes[grp["rid"].long()].view(-1, 1, 1)
            for x in (grp["a"], grp["b"]):  # uniform below 2^62, then folded below the row's prime
                x.copy_(torch.randint(0, 1 << 62, x.shape, generator=g, device="cuda", dtype=torch.int64))
                x.mul_(2).add_(torch.randint(0, 2, x.shape, generator=g, device="cuda", dtype=torch.int64))
                x.remainder_(lim)
        m.capture()
        st["mixed"] = m
        return st
    nphi, k = case["nphi"], case["k"]
    P = case.get("batch", 1)
    if kind == "ckks":
        e = Engine.ckks(k, 0, nphi, case["prec"])
        st["a"] = _uniform(e.empty(QBase, P), e.Q, g)
        st["b"] = _uniform(e.empty(QBase, P), e.Q, g)
        st["c"] = e.empty(QBase, P)
        st["raised"] = e.zeros(QBBase, P)
        st["ws"] = e.ckks_batch_workspace(P)
    elif kind == "polymul":
        e = Engine(k, 0, nphi, 256)
        st["a"] = _uniform(e.empty(QBase, P), e.Q, g)
        st["b"] = _uniform(e.empty(QBase, P), e.Q, g)
        st["c"] = e.empty(QBase, P)
        st["ws"] = e.polymul_workspace(QBase, P)
    elif kind in ("bfv", "bfv_batch"):
        e = Engine(k, 0, nphi, case["t"])
        st["ins"] = [_uniform(e.empty(QBase, P), e.Q, g) for _ in range(4)]
        if kind == "bfv":
            st["outs"] = [e.empty(QBase) for _ in range(3)]
            e.workspace()
        else:
            st["c"] = e.empty(QBase, 3 * P)
            st["ws"] = e.bfv_mul_batch_workspace(P)
    elif kind == "dgt":
        e = Engine(k, 0, nphi, 256)
        st["x"] = _uniform(e.empty(QBase, P), e.Q, g)
    elif kind == "relin":
        e = Engine(k, 0, nphi, 256)
        st["c2"] = _uniform(e.empty(QBase, P), e.Q, g)
        st["dec"] = e.empty(QBase, P * k)
        st["keys"] = [_uniform(e.empty(QBase, k), e.Q, g) for _ in range(2)]
        st["outs"] = [e.empty(QBase, P) for _ in range(2)]
    elif kind == "sample":
        e = Engine(k, 0, nphi, 65537)
        st["seed"] = int(seed)
        st["outs"] = [e.empty(QBase, P) for _ in range(3)]
    elif kind == "io":
        e = Engine(k, 0, nphi, 256)
        # k limbs of 64 bits below the product of k 63-bit primes: the top limb has 63 - k bits
        c = torch.randint(-(1 << 62), 1 << 62, (P, nphi, k), generator=g, device="cuda", dtype=torch.int64).mul_(2)
        c.add_(torch.randint(0, 2, c.shape, generator=g, device="cuda", dtype=torch.int64))
        c[..., k - 1] = torch.randint(0, 1 << (63 - k), (P, nphi), generator=g, device="cuda", dtype=torch.int64)
        st["coefs"] = c
        st["x"] = e.empty(QBase, P)
        st["back"] = torch.empty_like(c)
    else:
        raise ValueError("unknown kind %r" % kind)
    st["e"] = e
    return st


def run(st):
    kind = st["kind"]
    if kind == "mixed":
        st["mixed"].replay()
        return [g["c"] for g in st["mixed"].groups.values()]
    e, case = st["e"], st["case"]
    P = case.get("batch", 1)
    if kind == "polymul":
        e.polymul(st["c"], st["a"], st["b"], QBase, st["ws"], P)
        return st["c"]
    if kind == "bfv":
        e.bfv_mul(*st["outs"], *st["ins"])
        return st["outs"]
    if kind == "bfv_batch":
        e.bfv_mul_batch(st["c"], *st["ins"], P, st["ws"])
        return st["c"]
    if kind == "dgt":
        return e.dgt(st["x"], QBase, INVERSE if case["inverse"] else FORWARD, P)
    if kind == "relin":
        e.xi_batch(st["dec"], st["c2"], P)
        for out, key in zip(st["outs"], st["keys"]):
            e.dot_batch(out, st["dec"], key, case["k"], P, QBase, b_shared=True)
        return st["outs"]
    if kind == "ckks":
        level = case["k"] - 1
        e.mul_batch(st["c"], st["a"], st["b"], QBase, P)
        e.ckks_rescale_batch(st["c"], level, P)
        e.ckks_modulus_raising_batch(st["raised"], st["c"], level - 1, st["ws"], P)
        return [st["c"], st["raised"]]
    if kind == "sample":
        for i, (out, dist) in enumerate(zip(st["outs"], (TERNARY, GAUSSIAN, UNIFORM))):
            e.sample(out, QBase, dist, st["seed"], i * P, P, to_dgt=True)
        return st["outs"]
    e.crt(st["x"], st["coefs"], QBase)
    e.icrt(st["back"], st["x"], QBase)
    return [st["x"], st["back"]]


def work(case):
    """Bytes of every input and output once.  All of the arithmetic is on integers: no floating
    operations are counted."""
    kind = case["kind"]
    if kind == "mixed":
        return {"bytes": sum(24 * n * k for n, k in random_specs(case["count"], case["specs_seed"], kmax=case["kmax"])),
                "flops": 0}
    nphi, k, P = case["nphi"], case["k"], case.get("batch", 1)
    poly = 8 * nphi * k  # one polynomial over Q
    bytes_ = {
        "polymul": 3 * P * poly,
        "bfv": 7 * poly,
        "bfv_batch": 7 * P * poly,
        "dgt": 2 * P * poly,
        "relin": (3 * P + 2 * k) * poly,  # c2 in, two sums out, the keys
        "ckks": 3 * P * poly + P * 8 * nphi * (2 * k + 1),  # a, b, rescaled c; the raised polynomials over Q and B
        "sample": 3 * P * poly,
        "io": 3 * P * poly,
    }[kind]
    return {"bytes": bytes_, "flops": 0}


def exact(case, seed):
    """The products of a small polymul case, by big-integer multiplication (one slot of 144 bits per
    coefficient); nothing for the other kinds, whose outputs are whole numbers as well."""
    if case["kind"] != "polymul" or case["nphi"] * case["k"] * case["batch"] > 32768:
        return None
    st = prepare(case, seed)
    N, n = case["nphi"] // 2, case["nphi"]
    a, b = (st[v].cpu().numpy() for v in ("a", "b"))
    out = np.zeros_like(a)

    def packed(x):  # (N, 2) folded residues -> sum_c x_c 2^(144 c)
        slots = np.zeros((n, 18), dtype=np.uint8)
        slots[:, :8] = np.ascontiguousarray(np.concatenate([x[:, 0], x[:, 1]])).view(np.uint8).reshape(n, 8)
        return int.from_bytes(slots.tobytes(), "little")

    for q in range(a.shape[0]):
        for r, p in enumerate(st["e"].Q):
            raw = (packed(a[q, r]) * packed(b[q, r])).to_bytes(2 * n * 18, "little")
            c = [int.from_bytes(raw[18 * i:18 * i + 18], "little") for i in range(2 * n)]
            m = np.array([(c[i] - c[i + n]) % p for i in range(n)], dtype=np.int64)
            out[q, r] = np.stack([m[:N], m[N:]], axis=-1)
    return torch.from_numpy(out)
