"""The work that users of this library run on a GPU, as timed cases.

A homomorphic-encryption program encodes and encrypts on the client side, multiplies,
relinearizes, rescales and rotates ciphertexts (or multiplies them by plaintext
matrices) on the server side, and decrypts and decodes the results. Each case is one of
these through the C ABI (``include/troy_b200.h``, bound by ``tb_capi``) or the batched
step built on it (``ckks_step``), over device buffers that the program keeps:

* ``chain``: ciphertext pairs through multiply -> relinearize -> (CKKS: rescale, BGV:
  modulus switch) -> one rotation each;
* ``poly_mul``: raw negacyclic products (forward NTT, dyadic product, inverse NTT);
* ``encrypt``: encode slot values and encrypt them;
* ``decrypt``: decrypt ciphertexts and decode the slots;
* ``matmul``: encrypted vectors times plaintext matrices (coefficient encoding).

Ciphertexts and keys of the evaluation cases are uniform residues, which is what
encrypted data and key-switching keys look like; the decryption cases take real
encryptions of the values they return.
"""
from __future__ import annotations

import ctypes
import functools
import math
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "seal-cuda_b200", "python"))

import tb_capi  # noqa: E402
from ckks_step import BatchedCkksStep  # noqa: E402

_SCHEMES = {"bfv": tb_capi.SCHEME_BFV, "ckks": tb_capi.SCHEME_CKKS, "bgv": tb_capi.SCHEME_BGV,
            "raw": tb_capi.SCHEME_RAW}
_PLAIN_BITS = 20      # batching plain modulus of the BFV / BGV parameter sets
_MAX_STEPS = 13       # rotation steps (Galois keys) of a batch: 1, 2, 4, ..., 4096


def listed():
    return [
        # the benchmark's workload: a server's large batch, 13 rotation keys
        {"name": "ckks_chain_n16384_64", "kind": "chain", "scheme": "ckks", "n": 16384,
         "bits": "60 40 40 40 40 40 40 40 60", "batch": 64},
        # one pair per call, as callers of a single-ciphertext evaluator drive it: latency
        {"name": "ckks_chain_n8192_1", "kind": "chain", "scheme": "ckks", "n": 8192, "bits": "60 40 60", "batch": 1},
        # a deep circuit's large ring, a small and odd batch
        {"name": "ckks_chain_n32768_5", "kind": "chain", "scheme": "ckks", "n": 32768,
         "bits": "60 40 40 40 40 40 40 40 40 40 40 60", "batch": 5},
        # exact integer arithmetic in batches (the largest ring of the uneven batches)
        {"name": "bfv_chain_n16384_48", "kind": "chain", "scheme": "bfv", "n": 16384,
         "bits": "48 48 48 48 48 48 48 48 48", "batch": 48},
        # the smallest BFV parameters, one pair: latency and launches
        {"name": "bfv_chain_n4096_1", "kind": "chain", "scheme": "bfv", "n": 4096, "bits": "36 36 37", "batch": 1},
        # BGV with modulus switching, an odd batch in the middle of the range
        {"name": "bgv_chain_n8192_33", "kind": "chain", "scheme": "bgv", "n": 8192, "bits": "43 43 44 44 44",
         "batch": 33},
        # polynomial products without a scheme (the transform sweep's shape), odd count
        {"name": "poly_mul_n16384_255", "kind": "poly_mul", "scheme": "raw", "n": 16384,
         "bits": "50 50 50 50 50 50 50 50", "batch": 255},
        # a client (or a server-side test harness) encrypting a batch of vectors
        {"name": "ckks_encrypt_n16384_16", "kind": "encrypt", "scheme": "ckks", "n": 16384,
         "bits": "60 40 40 40 40 40 40 40 60", "batch": 16, "level": 8, "symmetric": False},
        # reading back the results of a chain: one level below the top
        {"name": "ckks_decrypt_n16384_16", "kind": "decrypt", "scheme": "ckks", "n": 16384,
         "bits": "60 40 40 40 40 40 40 40 60", "batch": 16, "level": 7},
        # one small integer vector: latency
        {"name": "bfv_encrypt_n4096_1", "kind": "encrypt", "scheme": "bfv", "n": 4096, "bits": "36 36 37", "batch": 1,
         "level": 2, "symmetric": False},
        {"name": "bfv_decrypt_n8192_7", "kind": "decrypt", "scheme": "bfv", "n": 8192, "bits": "43 43 44 44 44",
         "batch": 7, "level": 4},
        # the serving loop's wave: requests of an encrypted vector times a plaintext matrix
        {"name": "bfv_matmul_n8192_12", "kind": "matmul", "scheme": "bfv", "n": 8192, "bits": "43 43 44 44 44",
         "batch": 12, "inputs": 1000, "outputs": 200},
    ]


def draw(rng: random.Random):
    kind = rng.choice(["chain", "chain", "chain", "poly_mul", "encrypt", "decrypt", "matmul"])
    n = 1 << rng.choice([12, 13, 13, 14, 14, 15])
    most = {4096: 4, 8192: 6, 16384: 9, 32768: 12}[n]     # data primes
    L = rng.randint(2, most)

    def count(limit):
        return max(1, int(math.exp(rng.uniform(0, math.log(max(2, limit))))))

    if kind == "poly_mul":
        bits = rng.choice([40, 50, 55, 58])
        return {"kind": kind, "scheme": "raw", "n": n, "bits": " ".join([str(bits)] * L),
                "batch": count(33000000 // (n * L))}
    scheme = "bfv" if kind == "matmul" else rng.choice(["ckks", "ckks", "bfv", "bgv"])
    if scheme == "ckks":
        small = rng.choice([36, 40, 45])
        bits = [60] + [small] * (L - 1) + [60]
    else:
        b = rng.choice([40, 44, 48, 55])
        bits = [b] * (L + 1)
    case = {"kind": kind, "scheme": scheme, "n": n, "bits": " ".join(map(str, bits))}
    if kind == "chain":
        # at most the benchmark step's transforms: n L (L + 1) words per pair and key switch
        limit = 64 * 16384 * 8 * 9 // (n * L * (L + 1))
        return dict(case, batch=count(limit if scheme == "ckks" else limit // 2))
    if kind == "matmul":
        inputs, outputs = rng.randint(64, 1024), rng.randint(16, 256)
        blocks = max(1, inputs * outputs // n) + 2
        return dict(case, batch=count(min(48, 20000000 // (n * L * blocks))), inputs=inputs, outputs=outputs)
    limit = 5000000 // (n * L)
    case = dict(case, batch=count(limit), level=rng.randint(2 if scheme == "ckks" else 1, L))
    if kind == "encrypt":
        case["symmetric"] = rng.random() < 0.25
    return case


# ------------------------------------------------------------------ preparation


def _bits(case):
    return [int(b) for b in case["bits"].split()]


@functools.lru_cache(maxsize=None)
def _context(scheme, n, bits):
    """The parameter context a program creates once and keeps."""
    lib = tb_capi.lib()
    b = [int(x) for x in bits.split()]
    out = (ctypes.c_uint64 * len(b))()
    tb_capi.check(lib.tb_coeff_modulus_create(ctypes.c_uint64(n), (ctypes.c_int * len(b))(*b), len(b), out))
    t = ctypes.c_uint64(0)
    if scheme in ("bfv", "bgv"):
        tb_capi.check(lib.tb_plain_modulus_batching(ctypes.c_uint64(n), _PLAIN_BITS, ctypes.byref(t)))
    return tb_capi.Context(_SCHEMES[scheme], n, [int(m) for m in out], t.value)


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _residues(lead, moduli, n, gen):
    """Uniform residues [lead...][limb][n]."""
    out = torch.empty(tuple(lead) + (len(moduli), n), dtype=torch.int64, device="cuda")
    for i, q in enumerate(moduli):
        out[..., i, :] = torch.randint(0, q, tuple(lead) + (n,), generator=gen, device="cuda")
    return out


def _empty(*shape):
    return torch.empty(shape, dtype=torch.int64, device="cuda")


def _seed_words(seed):
    r = random.Random(seed)
    return (ctypes.c_uint64 * 8)(*[r.getrandbits(64) for _ in range(8)])


def _steps(case):
    """Galois steps of a chain's batch: powers of two, at most one per pair."""
    half = case["n"] // 2
    return [1 << i for i in range(_MAX_STEPS) if (1 << i) < half][: max(1, min(_MAX_STEPS, case["batch"]))]


def _elements(ctx, steps):
    out = []
    for k in steps:
        e = ctypes.c_uint32()
        ctx("galois_elt_from_step", k, ctypes.byref(e))
        out.append(e.value)
    return out


def _scale(case):
    """CKKS scale: the size of the chain's middle primes."""
    return 2.0 ** _bits(case)[1]


def prepare(case, seed):
    ctx = _context(case["scheme"], case["n"], case["bits"])
    gen = _generator(seed)
    return _PREPARE[case["kind"]](case, ctx, gen, seed)


def _prepare_chain(case, ctx, gen, seed):
    n, batch, moduli = case["n"], case["batch"], ctx.moduli
    K, L = len(moduli), len(moduli) - 1
    s = {"case": case, "ctx": ctx,
         "a": _residues((batch, 2), moduli[:L], n, gen), "b": _residues((batch, 2), moduli[:L], n, gen),
         "rlk": _residues((K - 1, 2), moduli, n, gen)}
    if case["scheme"] == "ckks":
        steps = _steps(case)
        gks = [_residues((K - 1, 2), moduli, n, gen) for _ in steps]
        # two concurrent sub-batches (an odd batch runs as one)
        s["step"] = BatchedCkksStep(torch, ctx, L, n, batch, s["rlk"], _elements(ctx, steps), gks, 2)
        s["out"] = _empty(batch, 2, L - 1, n)
        return s
    s["elt"] = _elements(ctx, [1])[0]
    s["gk"] = _residues((K - 1, 2), moduli, n, gen)
    s["product"] = _empty(batch, 3, L, n)
    if case["scheme"] == "bgv":
        s["switched"] = _empty(batch, 2, L - 1, n)
    s["out"] = _empty(batch, 2, L - (case["scheme"] == "bgv"), n)
    return s


def _prepare_poly_mul(case, ctx, gen, seed):
    n, batch, moduli = case["n"], case["batch"], ctx.moduli
    return {"case": case, "ctx": ctx, "x": _residues((batch,), moduli, n, gen), "w": _residues((batch,), moduli, n, gen),
            "xf": _empty(batch, len(moduli), n), "out": _empty(batch, len(moduli), n)}


def _slot_values(case, ctx, gen):
    """Slot values of a batch: complex numbers in the unit square (CKKS) or residues mod t."""
    n, batch = case["n"], case["batch"]
    if case["scheme"] == "ckks":
        return torch.rand((batch, n // 2, 2), generator=gen, device="cuda", dtype=torch.float64) * 2 - 1
    return torch.randint(0, ctx.t, (batch, n), generator=gen, device="cuda")


def _keys(case, ctx, seed):
    n, K = case["n"], len(ctx.moduli)
    sk, pk = _empty(K, n), _empty(2, K, n)
    stream = torch.cuda.current_stream()
    words = _seed_words(seed)
    ctx("keygen_secret", words, sk, stream)
    ctx("keygen_public", words, sk, pk, stream)
    return sk, pk


def _prepare_encrypt(case, ctx, gen, seed):
    n, batch, L = case["n"], case["batch"], case["level"]
    sk, pk = _keys(case, ctx, seed)
    plain = _empty(batch, L, n) if case["scheme"] == "ckks" else _empty(batch, n)
    return {"case": case, "ctx": ctx, "sk": sk, "pk": pk, "seed": _seed_words(seed + 1),
            "values": _slot_values(case, ctx, gen), "plain": plain, "out": _empty(batch, 2, L, n)}


def _prepare_decrypt(case, ctx, gen, seed):
    s = _prepare_encrypt(dict(case, symmetric=False), ctx, gen, seed)
    ct = _run_encrypt(s)["ct"]
    n, batch, L = case["n"], case["batch"], case["level"]
    s.update(case=case, ct=ct, out=torch.empty((batch, n // 2, 2), dtype=torch.float64, device="cuda")
             if case["scheme"] == "ckks" else _empty(batch, n))
    return s


def _blocks(case):
    """(input block, output block) of the coefficient encoding of one vector times an
    inputs x outputs matrix: the fewest polynomials to send and receive."""
    n, inputs, outputs = case["n"], case["inputs"], case["outputs"]
    best = None
    for i in range(1, min(inputs, n - 1) + 1):
        o = min(n // i, outputs)
        c = -(-inputs // i) + -(-outputs // o)
        if best is None or c < best[0]:
            best = (c, i, o)
    return best[1], best[2]


def _prepare_matmul(case, ctx, gen, seed):
    n, batch, L = case["n"], case["batch"], len(ctx.moduli) - 1
    inputs, outputs = case["inputs"], case["outputs"]
    ib, ob = _blocks(case)
    nin, nout = -(-inputs // ib), -(-outputs // ob)
    records, off, ia, iw = [], [0], [], []
    for r in range(batch):
        base = r * inputs * outputs
        for li in range(nin):
            for lj in range(nout):
                records += [base & 0xffffffff, base >> 32, inputs, outputs, ib, ob, li * ib, lj * ob]
        for lj in range(nout):
            for li in range(nin):
                ia.append(r * nin + li)
                iw.append((r * nin + li) * nout + lj)
            off.append(len(ia))
    words = lambda v: torch.from_numpy(np.array(v, np.uint32).view(np.int32)).cuda()  # noqa: E731
    nw = batch * nin * nout
    return {"case": case, "ctx": ctx, "L": L, "ct": _residues((batch * nin, 2), ctx.moduli[:L], n, gen),
            "weights": torch.randint(0, ctx.t, (batch, inputs, outputs), generator=gen, device="cuda"),
            "records": words(records), "off": words(off), "ia": words(ia), "iw": words(iw),
            "ctn": _empty(batch * nin, 2, L, n), "plain": _empty(nw, n), "plain_ntt": _empty(nw, L, n),
            "out": _empty(batch * nout, 2, L, n), "nw": nw, "nout": batch * nout, "nin": batch * nin}


_PREPARE = {"chain": _prepare_chain, "poly_mul": _prepare_poly_mul, "encrypt": _prepare_encrypt,
            "decrypt": _prepare_decrypt, "matmul": _prepare_matmul}


# ------------------------------------------------------------------ one pass


def run(state):
    return _RUN[state["case"]["kind"]](state)


def _run_chain(s):
    case, ctx = s["case"], s["ctx"]
    n, batch, L = case["n"], case["batch"], len(ctx.moduli) - 1
    stream = torch.cuda.current_stream()
    if case["scheme"] == "ckks":
        s["step"](s["a"], s["b"], s["out"], stream)
        return {"ct": s["out"]}
    t3 = s["product"]
    ctx("multiply", L, s["a"], 0, s["b"], 0, t3, 0, batch, stream)
    ctx("relinearize", L, t3, 0, s["rlk"], batch, stream)
    if case["scheme"] == "bgv":
        ctx("rescale_to_next", L, t3, 3 * L * n, s["switched"], 0, 2, batch, stream)
        ctx("apply_galois", L - 1, s["elt"], s["switched"], 0, s["out"], 0, s["gk"], batch, stream)
    else:
        ctx("apply_galois", L, s["elt"], t3, 3 * L * n, s["out"], 0, s["gk"], batch, stream)
    return {"ct": s["out"]}


def _run_poly_mul(s):
    case, ctx = s["case"], s["ctx"]
    batch, limbs, stream = case["batch"], len(ctx.moduli), torch.cuda.current_stream()
    ctx("ntt_forward", s["x"], s["xf"], batch, 0, limbs, 0, stream)
    ctx("dyadic_product", s["xf"], s["w"], s["out"], batch, 0, limbs, stream)
    ctx("ntt_inverse", s["out"], s["out"], batch, 0, limbs, 0, stream)
    return {"transform": s["xf"], "product": s["out"]}


def _run_encrypt(s):
    case, ctx = s["case"], s["ctx"]
    n, batch, L, stream = case["n"], case["batch"], case["level"], torch.cuda.current_stream()
    if case["scheme"] == "ckks":
        ctx("ckks_encode", L, s["values"], 0, n // 2, _scale(case), s["plain"], batch, stream)
        stride, count = L * n, 0
    else:
        ctx("batch_encode", s["values"], 0, n, s["plain"], batch, stream)
        stride, count = n, n
    name, key = ("encrypt_symmetric", s["sk"]) if case["symmetric"] else ("encrypt", s["pk"])
    ct = s["out"]
    ctx(name, s["seed"], key, L, s["plain"], stride, count, ct, 0, batch, stream)
    return {"plain": s["plain"], "ct": ct}


def _run_decrypt(s):
    case, ctx = s["case"], s["ctx"]
    batch, L, stream = case["batch"], case["level"], torch.cuda.current_stream()
    ctx("decrypt", s["sk"], L, 2, s["ct"], 0, s["plain"], 0, 1, batch, stream)
    if case["scheme"] == "ckks":
        ctx("ckks_decode", L, s["plain"], _scale(case), s["out"], 0, batch, stream)
    else:
        ctx("batch_decode", s["plain"], s["out"], 0, batch, stream)
    return {"plain": s["plain"], "values": s["out"]}


def _run_matmul(s):
    ctx, L, n = s["ctx"], s["L"], s["case"]["n"]
    stream = torch.cuda.current_stream()
    ctx("ntt_forward", s["ct"], s["ctn"], 2 * s["nin"], 0, L, 0, stream)
    ctx("matmul_encode_weights", s["weights"], s["records"], s["nw"], s["plain"], stream)
    ctx("plain_to_ntt", L, s["plain"], n, n, s["plain_ntt"], s["nw"], stream)
    ctx("dyadic_accumulate", L, 2, s["ctn"], 0, s["plain_ntt"], 0, s["out"], 0, s["off"], s["ia"], s["iw"], s["nout"],
        stream)
    ctx("ntt_inverse", s["out"], s["out"], 2 * s["nout"], 0, L, 0, stream)
    return {"ct": s["out"]}


_RUN = {"chain": _run_chain, "poly_mul": _run_poly_mul, "encrypt": _run_encrypt, "decrypt": _run_decrypt,
        "matmul": _run_matmul}


# ------------------------------------------------------------------ work and correctness


def work(case):
    """Bytes: each input and key read once, each output written once. The arithmetic is
    64-bit modular integers (no floating point) except the CKKS encoder's transform."""
    n, batch, bits = case["n"], case["batch"], _bits(case)
    L = len(bits) - 1
    flops = 0
    if case["kind"] == "chain":
        lo = L if case["scheme"] == "bfv" else L - 1          # level of the rotation
        steps = len(_steps(case)) if case["scheme"] == "ckks" else 1
        words = batch * (4 * L + 2 * lo) + 2 * L * (L + 1) + steps * 2 * lo * (lo + 1)
    elif case["kind"] == "poly_mul":
        words = 4 * batch * len(bits)
    elif case["kind"] == "matmul":
        ib, ob = _blocks(case)
        words = batch * 2 * L * (-(-case["inputs"] // ib) + -(-case["outputs"] // ob))
        words += batch * case["inputs"] * case["outputs"] / n
    else:
        lv, ckks = case["level"], case["scheme"] == "ckks"
        plain = lv if ckks else 1                            # written (encode, decrypt) once
        key = lv if case["kind"] == "decrypt" or case["symmetric"] else 2 * (lv + 1)
        words = batch * (2 * lv + plain + 1) + key
        if ckks:
            flops = 5 * batch * n * math.log2(n)
    return {"bytes": 8.0 * n * words, "flops": flops}


def tolerance(case):
    """Ciphertext, plaintext and slot words are exact. CKKS decoding runs in FP64: log2 n
    butterflies of rounded products, measured 4e-16 off the exact values."""
    if case["kind"] == "decrypt" and case["scheme"] == "ckks":
        return {"rel": 2e-15}
    return "exact"


def _mul_mod(a, b, q):
    """a * b mod q of uint64 arrays (residues below q < 2^61): the quotient from the 64-bit
    mantissa of a long double, the remainder corrected by one q."""
    qt = (a.astype(np.longdouble) * b / q).astype(np.uint64)
    r = (a * b - qt * np.uint64(q)).astype(np.int64)
    r = np.where(r < 0, r + q, r)
    return np.where(r >= q, r - q, r).astype(np.uint64)


def _bit_reverse(v, bits):
    r = 0
    for _ in range(bits):
        r, v = (r << 1) | (v & 1), v >> 1
    return r


def _minimal_root(q, m):
    """The smallest primitive m-th root of unity mod q (m a power of two)."""
    g = next(r for r in (pow(x, (q - 1) // m, q) for x in range(2, q)) if pow(r, m // 2, q) == q - 1)
    best = cur = g
    sq = g * g % q
    for _ in range(m // 2 - 1):
        cur = cur * sq % q
        best = min(best, cur)
    return best


def _inverse_transform(x, q, n):
    """Coefficients of the polynomial whose value at psi^(2 bitrev(j) + 1) is x[..., j]."""
    logn = n.bit_length() - 1
    inv_psi = pow(_minimal_root(q, 2 * n), -1, q)
    power = [1] * n
    for i in range(1, n):
        power[i] = power[i - 1] * inv_psi % q
    x = x.copy()
    t, m = 1, n
    while m > 1:
        h = m // 2
        w = np.array([power[_bit_reverse(h + i, logn)] for i in range(h)], np.uint64)
        v = x.reshape(x.shape[:-1] + (h, 2, t))
        lo, hi = v[..., 0, :].copy(), v[..., 1, :].copy()
        s = lo + hi
        v[..., 0, :] = np.where(s >= q, s - np.uint64(q), s)
        d = np.where(lo >= hi, lo - hi, lo + np.uint64(q) - hi)
        v[..., 1, :] = _mul_mod(d, np.broadcast_to(w[:, None], d.shape), q)
        t, m = 2 * t, h
    return _mul_mod(x, np.full_like(x, pow(n, -1, q)), q)


def exact(case, seed):
    """The CKKS decoder's values in plain numpy: the phase c0 + c1 s of the ciphertexts, its
    integer coefficients by the Chinese remainder theorem, and their values at the slots."""
    if case["kind"] != "decrypt" or case["scheme"] != "ckks":
        return None
    n, batch, L = case["n"], case["batch"], case["level"]
    if n * batch * L > 2500000:
        return None
    s = prepare(case, seed)
    torch.cuda.synchronize()
    words = lambda t: t.cpu().numpy().view(np.uint64)  # noqa: E731
    ct, sk, moduli = words(s["ct"]), words(s["sk"]), s["ctx"].moduli[:L]
    Q = math.prod(moduli)
    x = np.zeros((batch, n), object)
    for i, q in enumerate(moduli):
        phase = _mul_mod(ct[:, 1, i], np.broadcast_to(sk[i], (batch, n)), q) + ct[:, 0, i]
        phase = np.where(phase >= q, phase - np.uint64(q), phase)
        m = _inverse_transform(phase, q, n)
        x += m.astype(object) * (Q // q * pow(Q // q, -1, q))
    x %= Q
    x = np.where(x > Q // 2, x - Q, x)
    coeff = (x.astype(np.longdouble) / np.longdouble(_scale(case)))
    zeta = np.exp(1j * np.pi * np.arange(n) / n)
    at = np.fft.ifft(coeff.astype(np.float64) * zeta, axis=-1) * n   # value at zeta^(2 k + 1)
    power, index = 1, []
    for _ in range(n // 2):
        index.append((power - 1) // 2)
        power = power * 3 % (2 * n)
    slots = at[:, index]
    return {"plain": None, "values": np.stack([slots.real, slots.imag], -1)}
