"""Workloads of the encrypted-aggregation path, taken through the public entry points.

A case is a plain dict; ``kind`` names the call a program makes, the rest its sizes and options:

  chain      the primitive chain of one value vector on the pyCAHEL interface: encode, encrypt, multiply, relinearize,
             rescale, rotate, decrypt, decode (one ciphertext at a time: launch latency and host work count)
  pair       the distance of one pair of clients as the driver of ``lancelot-main-GPU/utils/byzantine_fl.py`` issues it:
             encode and encrypt both clients' chunks, sub / square / add per chunk, relinearize, rescale, hoisting,
             rotate-and-sum, decrypt, decode
  keys       session set-up of a server: context, secret, public, relinearization and Galois keys
  encrypt    a client's upload: one flattened update encoded and encrypted
  round      a whole distance round of the batched driver: encrypt all clients, all pair distances, decrypt, sort
  aggregate  mask multiplication over the encrypted clients, size-3 decryption and decoding of the average
  hmult      multiply + relinearize + rescale of a batch of ciphertext pairs with ``limbs`` primes left
  ntt        the negacyclic transform of a batch of polynomials, in place

``api`` selects the two forms of the interface: "module" is the compiled ``pyCAHEL`` module (host arrays and lists),
"mirror" the Python classes over torch memory.  Integer results are exact; decoded values are double precision.
"""
import math

import numpy as np
import torch

from lancelot_b200 import cabi, krum
from lancelot_b200 import pycahel as mirror
from lancelot_b200.pybind import pyCAHEL as module

KRUM_BITS = [60, 40, 40, 60]           # three data primes and one special prime: the Krum chain
WIDE_BITS = [60] + [50] * 23 + [60] * 8  # 24 data and 8 special primes (dnum = 3): the deep chain
SCALE = 2.0 ** 40


def listed():
    return [
        # the smallest call sequence: one 4096-slot product at N = 2^13
        {"name": "chain_n13", "kind": "chain", "api": "module", "log_n": 13, "values": 4096},
        # one pair of clients on the one-call-per-operation driver; four chunks of 32768 slots
        {"name": "pair_n16_c4", "kind": "pair", "api": "mirror", "log_n": 16, "dim": 4 * 32768 - 1000},
        # what every new session pays: 26 Galois keys and the rest at N = 2^16
        {"name": "keys_n16", "kind": "keys", "log_n": 16, "rotations": 26},
        # one client's upload of an odd-length update from pinned host memory: 51 chunks, the last one ragged
        {"name": "encrypt_n16_c51", "kind": "encrypt", "log_n": 16, "dim": 1663370, "host": True, "dtype": "float32"},
        # a small federation with a small model
        {"name": "round_4x50k_n14", "kind": "round", "clients": 4, "dim": 50890, "log_n": 14, "host": False, "dtype": "float64"},
        # the 10-client round (102 chunks each at N = 2^15), updates arriving in pinned host memory
        {"name": "round_10x1.6m_n15", "kind": "round", "clients": 10, "dim": 1663370, "log_n": 15, "host": True, "dtype": "float32"},
        # the 20-client round (342 chunks each at N = 2^16), the largest workload there is
        {"name": "round_20x11m_n16", "kind": "round", "clients": 20, "dim": 11173962, "log_n": 16, "host": False, "dtype": "float32"},
        # the aggregation phase of the same federation: three of twenty clients averaged
        {"name": "aggregate_20x11m", "kind": "aggregate", "clients": 20, "dim": 11173962, "log_n": 16, "selected": 3},
        # deep chain, one ciphertext pair: latency of a single product
        {"name": "hmult_wide_b1", "kind": "hmult", "chain": "wide", "limbs": 24, "log_n": 16, "batch": 1},
        # deep chain, a batch of eight pairs
        {"name": "hmult_wide_b8", "kind": "hmult", "chain": "wide", "limbs": 24, "log_n": 16, "batch": 8},
        # bulk forward transforms of 24 fifty-bit limbs
        {"name": "ntt_fwd_24x50_b32", "kind": "ntt", "direction": "forward", "primes": "50", "limbs": 24, "log_n": 16, "batch": 32},
        # a few inverse transforms over the Krum chain's mixed primes
        {"name": "ntt_inv_krum_b5", "kind": "ntt", "direction": "inverse", "primes": "krum", "limbs": 4, "log_n": 15, "batch": 5},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["chain", "pair", "keys", "encrypt", "round", "round", "aggregate", "hmult", "ntt", "ntt"])
    if kind == "chain":
        log_n = rng.randint(12, 16)
        return {"kind": kind, "api": rng.choice(["module", "mirror"]), "log_n": log_n, "values": _log_uniform(rng, 64, 1 << (log_n - 1))}
    if kind == "pair":
        log_n = rng.randint(13, 16)
        return {"kind": kind, "api": rng.choice(["module", "mirror"]), "log_n": log_n, "dim": _log_uniform(rng, 1000, 12 << (log_n - 1))}
    if kind == "keys":
        log_n = rng.randint(12, 16)
        return {"kind": kind, "log_n": log_n, "rotations": rng.randint(1, log_n + 10)}
    host, dtype = rng.choice([True, False]), rng.choice(["float32", "float32", "float64"])
    if kind == "encrypt":
        return {"kind": kind, "log_n": rng.randint(13, 16), "dim": _log_uniform(rng, 5000, 11173962), "host": host, "dtype": dtype}
    if kind == "round":
        return {"kind": kind, "clients": rng.randint(3, 20), "dim": _log_uniform(rng, 20000, 11173962), "log_n": rng.randint(14, 16), "host": host, "dtype": dtype}
    if kind == "aggregate":
        clients = rng.randint(3, 20)
        return {"kind": kind, "clients": clients, "dim": _log_uniform(rng, 20000, 11173962), "log_n": rng.randint(14, 16), "selected": rng.randint(1, clients // 2)}
    if kind == "hmult":
        chain = rng.choice(["wide", "krum"])
        wide = chain == "wide"
        return {"kind": kind, "chain": chain, "limbs": rng.randint(4, 24) if wide else rng.randint(2, 3), "log_n": 16 if wide else rng.randint(13, 16),
                "batch": _log_uniform(rng, 1, 16 if wide else 128)}
    primes = rng.choice(["50", "krum", "60"])
    return {"kind": kind, "direction": rng.choice(["forward", "inverse"]), "primes": primes, "limbs": 4 if primes == "krum" else rng.randint(1, 24),
            "log_n": rng.randint(12, 16), "batch": _log_uniform(rng, 1, 128)}


# ---- inputs ------------------------------------------------------------------------------------------


class _Seeds:
    """Fixed key and encryption seeds in place of the operating system's, handed out in order: 64 bytes per seed."""

    def __init__(self, rng, count):
        self.blob, self.at = rng.bytes(64 * count), 0

    def __call__(self, count):
        lo = self.at
        self.at = lo + 64 * count
        return self.blob[lo:self.at]


def _rotation_steps(log_slots):
    slots = 1 << log_slots
    return [s for s in range(1, 16) if s < slots], [1 << k for k in range(4, log_slots)]


def _session(m, log_n, rotations, seeds):
    """context, keys and encoder of one party on either form of the interface"""
    n = 1 << log_n
    p = m.params(m.scheme_type.ckks)
    p.set_poly_modulus_degree(n)
    p.set_coeff_modulus(m.coeff_modulus_create(n, KRUM_BITS))
    p.set_special_modulus_size(1)
    p.set_galois_elts(m.get_elts_from_steps(rotations, n))
    m.set_seed_source(seeds)
    ctx = m.context(p, True, m.sec_level_type.tc128 if n >= 8192 else m.sec_level_type.none)
    sk, pk, rlk, glk = m.secret_key(p), m.public_key(ctx), m.relin_key(ctx), m.galois_key(ctx)
    sk.gen_secretkey(ctx)
    sk.gen_publickey(ctx, pk)
    sk.gen_relinkey(ctx, rlk)
    sk.create_galois_keys(ctx, glk)
    m.set_seed_source(None)
    return {"m": m, "params": p, "ctx": ctx, "sk": sk, "pk": pk, "rlk": rlk, "glk": glk, "encoder": m.ckks_encoder(ctx)}


def _updates(case, rng_seed, clients):
    """flattened client updates: small weights, a fifth of the clients far away (the Byzantine ones)"""
    g = torch.Generator(device="cuda")
    g.manual_seed(rng_seed)
    x = torch.randn(clients, case["dim"], generator=g, device="cuda", dtype=torch.float32) * 1e-2
    bad = clients // 5
    x[:bad] += torch.rand(bad, case["dim"], generator=g, device="cuda", dtype=torch.float32) * 10 - 5
    x = x.to(getattr(torch, case.get("dtype", "float32")))
    if case.get("host"):
        h = torch.empty(x.shape, dtype=x.dtype, pin_memory=True)
        h.copy_(x)
        return h
    return x


def _moduli(case):
    n = 1 << case["log_n"]
    if case["kind"] == "hmult":
        return cabi.coeff_modulus_create(n, WIDE_BITS if case["chain"] == "wide" else KRUM_BITS), 8 if case["chain"] == "wide" else 1
    bits = KRUM_BITS if case["primes"] == "krum" else [int(case["primes"])] * case["limbs"]
    return cabi.coeff_modulus_create(n, bits), 0


def _residues(shape, moduli, seed):
    """uniform residues [..., limb, N], one prime per limb"""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.empty(shape, dtype=torch.int64, device="cuda")
    for i, q in enumerate(moduli[: shape[-2]]):
        x[..., i, :] = torch.randint(0, q, x[..., i, :].shape, dtype=torch.int64, device="cuda", generator=g)
    return x


def prepare(case, seed):
    kind, rng = case["kind"], np.random.RandomState(seed % (1 << 31))
    s = {"kind": kind, "case": case}
    s["first"], s["power"] = _rotation_steps(case["log_n"] - 1)
    if kind in ("chain", "pair"):
        s.update(_session(module if case["api"] == "module" else mirror, case["log_n"], s["first"] + s["power"], _Seeds(rng, 256)))
    if kind == "chain":
        s["x"], s["y"] = rng.uniform(-1, 1, case["values"]), rng.uniform(-1, 1, case["values"])
        s["seeds"] = _Seeds(rng, 4)
    elif kind == "pair":
        slots = 1 << (case["log_n"] - 1)
        chunks = -(-case["dim"] // slots)
        v = [np.pad(rng.normal(0, 1e-2, case["dim"]).astype(np.float32), (0, chunks * slots - case["dim"])) for _ in range(2)]
        s["a"], s["b"] = (np.array_split(x, chunks) for x in v)
        s["zeros"] = np.zeros(slots)
        s["seeds"] = _Seeds(rng, 2 + 4 * chunks)
    elif kind == "keys":
        s["seeds"] = _Seeds(rng, 256)
    elif kind in ("encrypt", "round", "aggregate"):
        clients = 1 if kind == "encrypt" else case["clients"]
        s["server"] = krum.EncryptedKrum(log_slots=case["log_n"] - 1, seed=seed)
        u = _updates(case, seed, clients)
        if kind == "encrypt":
            s["update"] = u[0]
        elif kind == "round":
            s["updates"] = u
        else:
            s["cts"] = s["server"].encrypt_slices(u, 0, s["server"].n_chunks(case["dim"]))
            s["selected"] = [int(c) for c in rng.permutation(clients)[: case["selected"]]]
            s["seeds"] = _Seeds(rng, 4)
    elif kind == "hmult":
        moduli, special = _moduli(case)
        ctx = s["ctx"] = cabi.Context(case["log_n"], moduli, special)
        sk = ctx.gen_secret_key(np.frombuffer(rng.bytes(64), dtype=np.uint8))
        s["rlk"] = ctx.gen_switch_key(sk, ctx.multiply_poly_qp(sk, sk), np.frombuffer(rng.bytes(128 * (ctx.size_Q // special)), dtype=np.uint8))
        s["a"], s["b"] = (_residues((case["batch"], 2, case["limbs"], ctx.N), moduli, seed + k) for k in (0, 1 << 32))
    elif kind == "ntt":
        moduli, _ = _moduli(case)
        ctx = s["ctx"] = cabi.Context(case["log_n"], moduli, 0)
        s["data"] = _residues((case["batch"], len(moduli), ctx.N), moduli, seed)
    return s


# ---- one pass ----------------------------------------------------------------------------------------


def _chain(s):
    m, ctx, enc = s["m"], s["ctx"], s["encoder"]
    ct1 = s["pk"].encrypt_asymmetric(ctx, enc.encode(ctx, s["x"], SCALE))
    ct2 = s["pk"].encrypt_asymmetric(ctx, enc.encode(ctx, s["y"], SCALE))
    m.multiply_inplace(ctx, ct1, ct2)
    m.relinearize_inplace(ctx, ct1, s["rlk"])
    m.rescale_to_next_inplace(ctx, ct1)
    rotated = m.ciphertext(ctx)
    m.rotate_vector(ctx, ct1, 1, s["glk"], rotated)
    return enc.decode(ctx, s["sk"].decrypt(ctx, rotated))


def _pair(s):
    m, ctx, enc, pk = s["m"], s["ctx"], s["encoder"], s["pk"]
    acc = pk.encrypt_asymmetric(ctx, enc.encode(ctx, s["zeros"], SCALE))
    m.square_inplace(ctx, acc)
    tmp = m.ciphertext(ctx)
    for x1, x2 in zip(s["a"], s["b"]):
        ct1 = pk.encrypt_asymmetric(ctx, enc.encode(ctx, x1, SCALE))
        ct2 = pk.encrypt_asymmetric(ctx, enc.encode(ctx, x2, SCALE))
        m.sub(ctx, ct2, ct1, tmp)
        m.square_inplace(ctx, tmp)
        m.add_inplace(ctx, acc, tmp)
    m.relinearize_inplace(ctx, acc, s["rlk"])
    m.rescale_to_next_inplace(ctx, acc)
    acc.set_scale(SCALE)
    rot = m.hoisting(ctx, acc, s["glk"], s["first"])
    m.add_inplace(ctx, acc, rot)
    tmp_rot = m.ciphertext(ctx)
    for step in s["power"]:
        m.rotate_vector(ctx, acc, step, s["glk"], tmp_rot)
        m.add_inplace(ctx, acc, tmp_rot)
    return enc.decode(ctx, s["sk"].decrypt(ctx, acc))


def run(s):
    kind, case = s["kind"], s["case"]
    if "seeds" in s:
        s["seeds"].at = 0
    if kind in ("chain", "pair"):
        s["m"].set_seed_source(s["seeds"])
        return np.array(_chain(s) if kind == "chain" else _pair(s))
    if kind == "keys":
        k = _session(mirror, case["log_n"], (s["first"] + s["power"])[: case["rotations"]], s["seeds"])
        return {"secret": k["sk"].data, "public": k["pk"].data, "relin": k["rlk"].data, "galois": k["glk"].keys}
    if kind == "encrypt":
        return s["server"].encrypt_client(s["update"])
    if kind == "round":
        distances, order = s["server"].round(s["updates"])
        return {"distances": np.array(distances), "order": order}
    if kind == "aggregate":
        mirror.set_seed_source(s["seeds"])
        return s["server"].aggregate(s["cts"], s["selected"], case["dim"])
    ctx = s["ctx"]
    if kind == "hmult":
        L, batch = case["limbs"], case["batch"]
        ct3 = ctx.multiply(L, s["a"], s["b"], batch=batch)
        ctx.relinearize_batch(L, ct3, s["rlk"])
        return ctx.rescale_strided(L, ct3, batch, 2, 3 * L * ctx.N)
    transform = ctx.ntt_forward if case["direction"] == "forward" else ctx.ntt_inverse
    transform(s["data"], case["batch"], s["data"].shape[1], 0)
    return s["data"]


# ---- what a pass cannot do without ---------------------------------------------------------------------
# Bytes: inputs and keys read once, results written once; in a round also the ciphertexts of all clients, written once
# by the encryption and read once by the pair distances (they fit no cache and every pair needs them).
# Operations: modular products and sums, of which a transform of one limb takes 3/2 N log2 N.


def _switch_transforms(L, P, alpha):
    """limb transforms of one key switch: input, digits without their own limbs, special limbs, results"""
    beta = -(-L // alpha)
    return L + beta * (L + P) - L + 2 * P + 2 * L


def work(case):
    kind, log_n = case["kind"], case["log_n"]
    n = 1 << log_n
    limb, transform, slots = 8 * n, 1.5 * n * log_n, n // 2
    first, power = (len(x) for x in _rotation_steps(log_n - 1))
    public, relin, rotation = 8 * limb, 24 * limb, 12 * limb  # key limbs read: 2 x 4, 3 x 2 x 4, and 2 x 2 x 3 at level 2
    encode, encrypt = 3 * transform, 12 * transform
    switch3, switch2 = _switch_transforms(3, 1, 1) * transform, _switch_transforms(2, 1, 1) * transform
    rescale = (2 + 4) * transform
    chunks = -(-case["dim"] // slots) if "dim" in case else 0
    item = 8 if case.get("dtype") == "float64" else 4
    if kind == "chain":
        out = 1 << max(1, (case["values"] - 1).bit_length())
        return {"bytes": 16 * case["values"] + public + relin + rotation + 8 * out,
                "flops": 2 * (encode + encrypt) + switch3 + rescale + switch2 + 2 * transform}
    if kind == "pair":
        return {"bytes": 8 * case["dim"] + public + relin + (first + power) * rotation + 8 * slots,
                "flops": (2 * chunks + 1) * (encode + encrypt) + switch3 + rescale + (1 + power) * switch2 + 2 * transform}
    if kind == "keys":
        keys = case["rotations"]
        return {"bytes": (4 + 8 + 24 + 24 * keys) * limb, "flops": 4 * (2 + 3 + 3 * keys) * transform}
    if kind == "encrypt":
        return {"bytes": case["dim"] * item + public + 6 * limb * chunks, "flops": chunks * (encode + encrypt)}
    if kind == "round":
        k, pairs = case["clients"], case["clients"] * (case["clients"] - 1) // 2
        return {"bytes": k * case["dim"] * item + public + relin + (first + power) * rotation + 2 * 6 * limb * k * chunks,
                "flops": k * chunks * (encode + encrypt) + pairs * chunks * 3 * n * 8 + pairs * (switch3 + rescale + (1 + power) * switch2)}
    if kind == "aggregate":
        k = case["clients"]
        return {"bytes": 6 * limb * k * chunks + public + 3 * limb + 8 * case["dim"], "flops": chunks * (k * 3 * n * 8 + 3 * transform)}
    if kind == "hmult":
        L, b, P = case["limbs"], case["batch"], 8 if case["chain"] == "wide" else 1
        transforms = _switch_transforms(L, P, P) + 2 + 2 * (L - 1)
        return {"bytes": b * (4 * L + 2 * (L - 1)) * limb + -(-L // P) * 2 * (L + P) * limb, "flops": b * (transforms * transform + 4 * L * n)}
    rows = case["batch"] * case["limbs"]
    return {"bytes": 2 * rows * limb, "flops": rows * transform}


def tolerance(case):
    # ciphertexts, keys and residues are exact integers; decoded slots come out of a double-precision transform of up to
    # 2^15 points, whose rounding stays below 1e-12 of the result (the encryption noise is fixed by the seeds)
    if case["kind"] in ("chain", "pair", "round", "aggregate"):
        return {"rel": 1e-11}
    return "exact"
