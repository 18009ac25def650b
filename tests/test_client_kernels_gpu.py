"""The fused client-side kernels (stream generation, encryption, decryption, encoders) and
the sums behind the matrix helpers and the BFV lift, at the sizes where their rules
change, against the oracle."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import tb_capi  # noqa: E402
from session import CkksCodec, OracleSession  # noqa: E402

BFV, CKKS, BGV = 1, 2, 3
SEED = np.arange(101, 109, dtype=np.uint64)
SEEDP = (ctypes.c_uint64 * 8)(*[int(x) for x in SEED])


def _dev(a):
    return torch.from_numpy(np.array(a, np.uint64, order="C").view(np.int64)).cuda()


def _host(t):
    return t.cpu().numpy().view(np.uint64)


def _empty(*shape):
    return torch.empty(shape, dtype=torch.int64, device="cuda")


def _residues(rng, lead, moduli, n):
    return np.stack([rng.integers(0, q, tuple(lead) + (n,), dtype=np.uint64) for q in moduli], -2)


def _with_plain(O, scheme, ct, plain):
    """ct, an encryption of zero from the oracle, plus the plaintext (as Encryptor does)."""
    ct = ct.copy()
    data = O.moduli[:ct.shape[1]]
    if scheme == BFV:
        ct[0] = O._multiply_add_plain_scaling_variant(data, ct[0], plain)
    else:
        ct[0] = np.stack([((ct[0, l].astype(object) + (plain[l] if scheme == CKKS else plain).astype(object)) % q)
                          for l, q in enumerate(data)]).astype(np.uint64)
    return ct


def _client(orc, scheme, seedp):
    """Context of three primes (two data primes), secret and public key."""
    n = 4096
    moduli = orc.coeff_modulus_create(n, [36, 36, 40])
    t = orc.plain_modulus_batching(n, 20) if scheme != CKKS else 0
    ctx = tb_capi.Context(scheme, n, moduli, t)
    sk, pk = _empty(3, n), _empty(2, 3, n)
    ctx("keygen_secret", seedp, sk, None)
    ctx("keygen_public", seedp, sk, pk, None)
    return n, moduli, t, ctx, sk, pk


def _plains(rng, scheme, count, moduli, t, n):
    return _residues(rng, (count,), moduli, n) if scheme == CKKS else rng.integers(0, t, (count, n), dtype=np.uint64)


@pytest.mark.parametrize("scheme", [BFV, BGV, CKKS])
@pytest.mark.parametrize("count", [1, 3, 40])   # 40: several refills of the stream per CTA
def test_batched_encryption_words(orc, scheme, count):
    """Every encryption of a seeded batch has the oracle's words for its own plaintext (each
    starts the seed's stream anew), asymmetric and symmetric, with padded strides too, and
    decrypts to its plaintext."""
    n, moduli, t, ctx, sk, pk = _client(orc, scheme, SEEDP)
    O = OracleSession(scheme, n, moduli, t, SEED)
    L, ckks = 2, scheme == CKKS
    plain = _plains(np.random.default_rng(5), scheme, count, moduli[:L], t, n)
    zero = np.zeros((L, n) if ckks else n, np.uint64)
    zeros = {"encrypt": (np.asarray(O.encrypt_plain(zero)).reshape(2, L, n), pk),
             "encrypt_symmetric": (O.encrypt_zero_symmetric(moduli[:L], ckks), sk)}
    for name, (z, key) in zeros.items():
        for pad in (0, 2):
            padded = np.zeros((count, zero.size + pad), np.uint64)
            padded[:, :zero.size] = plain.reshape(count, -1)
            out = _empty(count, 2 * L * n + pad)
            ctx(name, SEEDP, key, L, _dev(padded), zero.size + pad, n, out, 2 * L * n + pad, count, None)
            got = np.ascontiguousarray(_host(out)[:, :2 * L * n]).reshape(count, 2, L, n)
            for i in range(count):
                assert np.array_equal(got[i], _with_plain(O, scheme, z, plain[i])), (name, pad, i)
        if not ckks:
            dec = _empty(count, n)
            ctx("decrypt", sk, L, 2, _dev(got), 0, dec, 0, 1, count, None)
            assert np.array_equal(_host(dec), plain), name
    if not ckks and count == 1:   # the oracle's own encryption of a plaintext
        assert np.array_equal(_with_plain(O, scheme, zeros["encrypt"][0], plain[0]),
                              np.asarray(O.encrypt_plain(plain[0])).reshape(2, L, n))


@pytest.mark.parametrize("scheme", [BFV, BGV, CKKS])
def test_every_encryption_of_a_batch_has_samples_of_its_own(orc, scheme):
    """Without a seed each ciphertext draws its own u, e_0 and e_1. The public key (1000, 0)
    and no dropped prime make them readable: c_0 = 1000 u + e_0 (t e_0 for BGV), c_1 = e_1."""
    n, moduli, t, ctx, sk, _ = _client(orc, scheme, None)
    K, count = 3, 6
    factor = t if scheme == BGV else 1
    scale = 1000 * factor   # above 2 x 21 factor, the binomial samples' range
    pk = np.zeros((2, K, n), np.uint64)
    pk[0] = scale
    out = _empty(count, 2, K, n)
    ctx("encrypt", None, _dev(pk), K, None, 0, 0, out, 0, count, None)
    seen = {"u": set(), "e0": set(), "e1": set()}
    for ct in _host(out):
        if scheme == CKKS:
            ct = np.stack([orc.ntt_inverse_rns(12, moduli, p) for p in ct])
        q = np.array(moduli, np.int64)[None, :, None]
        c = ct.astype(np.int64)
        c = np.where(c > q // 2, c - q, c)
        assert (c == c[:, :1]).all()   # the same integers modulo every prime
        u = np.rint(c[0, 0] / scale).astype(np.int64)
        e0, e1 = c[0, 0] - scale * u, c[1, 0]
        assert not (e0 % factor).any() and not (e1 % factor).any()
        for name, v, top in (("u", u, 1), ("e0", e0 // factor, 21), ("e1", e1 // factor, 21)):
            assert abs(v).max() <= top and len(set(v.tolist())) > 2, name
            seen[name].add(v.tobytes())
    assert all(len(v) == count for v in seen.values())


@pytest.mark.parametrize("scheme", [BFV, BGV, CKKS])
def test_unseeded_batches_decrypt(orc, scheme):
    """Batches without a seed: no two ciphertexts share c_1, and each decrypts to its own
    plaintext (CKKS: up to the dropped prime's rounding, (n + 1) / 2 and the noise)."""
    n, moduli, t, ctx, sk, pk = _client(orc, scheme, None)
    L, count = 2, 5
    plain = _plains(np.random.default_rng(7), scheme, count, moduli[:L], t, n)
    for name, key in (("encrypt", pk), ("encrypt_symmetric", sk)):
        out = _empty(count, 2, L, n)
        ctx(name, None, key, L, _dev(plain), plain[0].size, n, out, 0, count, None)
        assert len({c.tobytes() for c in _host(out)[:, 1]}) == count, name
        dec = _empty(count, L, n) if scheme == CKKS else _empty(count, n)
        ctx("decrypt", sk, L, 2, out, 0, dec, 0, 1, count, None)
        got = _host(dec)
        if scheme != CKKS:
            assert np.array_equal(got, plain), name
            continue
        for b in range(count):
            for l, q in enumerate(moduli[:L]):
                noise = orc.ntt_inverse(12, q, (got[b, l] + np.uint64(q) - plain[b, l]) % np.uint64(q)).astype(np.int64)
                assert abs(np.where(noise > q // 2, noise - q, noise)).max() < n, (name, b, l)


@pytest.mark.parametrize("logn", [6, 12, 13, 14, 15, 16])
def test_ckks_codec_words(orc, logn):
    """Block transforms of the special FFT: one block, 1 - 3 joining stages, and degrees with
    stages in between; encoded words equal the oracle's, decoded values its values."""
    n = 1 << logn
    moduli = orc.coeff_modulus_create(n, [50, 40, 50])
    L, B = 2, 2
    ctx = tb_capi.Context(CKKS, n, moduli)
    codec = CkksCodec(n, moduli)
    rng = np.random.default_rng(logn)
    for count in (n // 2, n // 2 - 1):
        v = rng.uniform(-1, 1, (B, count)) + 1j * rng.uniform(-1, 1, (B, count))
        vals = torch.from_numpy(np.ascontiguousarray(np.stack([v.real, v.imag], -1))).cuda()
        plain = _empty(B, L, n)
        ctx("ckks_encode", L, vals, 0, count, 2.0 ** 40, plain, B, None)
        got = _host(plain)
        for b in range(B):
            exp = np.asarray(codec.encode(v[b], 2.0 ** 40, L)).reshape(L, n)
            if logn < 16:
                assert np.array_equal(got[b], exp), b
            else:   # the oracle's and the library's root tables differ in last places there
                g, x = (orc.ntt_inverse_rns(logn, moduli[:L], w).astype(object) for w in (got[b], exp))
                for l in range(L):
                    assert np.isin((g[l] - x[l]) % moduli[l], (0, 1, moduli[l] - 1)).all(), (b, l)
        out = torch.empty((B, n // 2, 2), dtype=torch.float64, device="cuda")
        ctx("ckks_decode", L, plain, 2.0 ** 40, out, 0, B, None)
        dec = out.cpu().numpy()
        dec = dec[..., 0] + 1j * dec[..., 1]
        for b in range(B):
            # 2 log2 n roundings of values below 2 sqrt(n) in FP64
            assert np.abs(dec[b] - codec.decode(got[b], 2.0 ** 40)).max() < 2.0 ** -40, b


@pytest.mark.parametrize("limbs", [1, 5, 12, 13])
def test_ckks_decode_limb_counts(orc, limbs):
    """CRT composition with the words in registers (up to 12 limbs) and in memory."""
    n = 4096
    moduli = orc.coeff_modulus_create(n, [45] * (limbs + 1))
    ctx = tb_capi.Context(CKKS, n, moduli)
    rng = np.random.default_rng(limbs)
    plain = _residues(rng, (1,), moduli[:limbs], n)
    scale = float(np.prod([float(q) for q in moduli[:limbs]])) / 2.0 ** 10
    out = torch.empty((1, n // 2, 2), dtype=torch.float64, device="cuda")
    ctx("ckks_decode", limbs, _dev(plain), scale, out, 0, 1, None)
    got = out.cpu().numpy()[0]
    exp = CkksCodec(n, moduli).decode(plain[0], scale)
    # coefficients below 2^9, log2 n roundings of sums of them
    assert np.abs(got[:, 0] + 1j * got[:, 1] - exp).max() < 2.0 ** -25


def test_ckks_decode_of_an_unaligned_plaintext(orc):
    """A plaintext that starts in the middle of a 16-byte pair decodes like an aligned one."""
    n, L, B = 4096, 2, 3
    moduli = orc.coeff_modulus_create(n, [40, 40, 41])
    ctx = tb_capi.Context(CKKS, n, moduli)
    plain = _dev(_residues(np.random.default_rng(3), (B,), moduli[:L], n))
    buf = _empty(B * L * n + 1)
    buf[1:] = plain.view(-1)
    assert buf[1:].data_ptr() % 16 == 8
    for name in ("ckks_decode", "ckks_decode_polynomial"):
        a, b = (torch.empty((B, n), dtype=torch.float64, device="cuda") for _ in range(2))
        ctx(name, L, plain, 2.0 ** 40, a, 0, B, None)
        ctx(name, L, buf[1:], 2.0 ** 40, b, 0, B, None)
        assert torch.equal(a, b), name


@pytest.mark.parametrize("scheme", [BFV, BGV, CKKS])
def test_phase_of_larger_ciphertexts(orc, scheme):
    """Decryption of sizes 2 .. 4 with strides: c_0 + c_1 s + c_2 s^2 + ..."""
    n, logn, L, B = 4096, 12, 2, 2
    moduli = orc.coeff_modulus_create(n, [40, 40, 41])
    t = orc.plain_modulus_batching(n, 20) if scheme != CKKS else 0
    ctx = tb_capi.Context(scheme, n, moduli, t)
    data = moduli[:L]
    rng = np.random.default_rng(scheme)
    sk = _empty(3, n)
    ctx("keygen_secret", SEEDP, sk, None)
    s = _host(sk)[:L]
    for size in (2, 3, 4):
        stride = size * L * n + 6
        ct = _residues(rng, (B, size), data, n)
        buf = np.zeros((B, stride), np.uint64)
        buf[:, :size * L * n] = ct.reshape(B, -1)
        ph = np.empty((B, L, n), np.uint64)
        for b in range(B):
            x = ct[b] if scheme == CKKS else orc.ntt_forward_rns(logn, data, ct[b])
            acc = x[size - 1]
            for k in range(size - 2, -1, -1):
                acc = orc.dyadic_rns(data, acc, s) + x[k]
                acc = np.stack([acc[l] % np.uint64(data[l]) for l in range(L)])
            ph[b] = acc if scheme == CKKS else orc.ntt_inverse_rns(logn, data, acc)
        if scheme == CKKS:
            out = _empty(B, L, n)
            ctx("decrypt", sk, L, size, _dev(buf), stride, out, 0, 1, B, None)
            assert np.array_equal(_host(out), ph), size
        else:   # the same plaintext as the size-2 ciphertext (phase, 0)
            two = np.stack([ph, np.zeros_like(ph)], 1)
            a, b2 = _empty(B, n), _empty(B, n)
            ctx("decrypt", sk, L, size, _dev(buf), stride, a, 0, 1, B, None)
            ctx("decrypt", sk, L, 2, _dev(two), 0, b2, 0, 1, B, None)
            assert torch.equal(a, b2), size


@pytest.mark.parametrize("n", [64, 4096])
def test_batch_codec_counts(orc, n):
    """Slots beyond `count` are zero, and decoding may write over its plaintexts."""
    t = orc.plain_modulus_batching(n, 20)
    ctx = tb_capi.Context(BFV, n, orc.coeff_modulus_create(n, [40, 40]), t)
    rng = np.random.default_rng(n)
    for count in (n, n - 1, 1):
        v = rng.integers(0, t, (3, count), dtype=np.uint64)
        plain = _empty(3, n)
        ctx("batch_encode", _dev(v), 0, count, plain, 3, None)
        ctx("batch_decode", plain, plain, 0, 3, None)
        got = _host(plain)
        assert np.array_equal(got[:, :count], v) and not got[:, count:].any()


@pytest.mark.parametrize("shift,stride", [(0, 4098), (0, 8192), (4096, 4096), (-4096, 4096), (5, 4097)])
def test_batch_decode_over_its_plaintexts(orc, shift, stride):
    """Slots that overlap other plaintexts than their own: several waves of transforms."""
    n, batch = 4096, 800
    t = orc.plain_modulus_batching(n, 20)
    ctx = tb_capi.Context(BFV, n, orc.coeff_modulus_create(n, [40, 40]), t)
    v = np.random.default_rng(stride).integers(0, t, (batch, n), dtype=np.uint64)
    plain = _empty(batch, n)
    ctx("batch_encode", _dev(v), 0, n, plain, batch, None)
    buf = _empty((batch + 2) * max(n, stride) + abs(shift))
    base = max(0, -shift)
    buf[base:base + batch * n] = plain.view(-1)
    ctx("batch_decode", buf[base:], buf[base + shift:], stride, batch, None)
    got = _host(buf[base + shift:base + shift + batch * stride]).reshape(batch, stride)[:, :n]
    assert np.array_equal(got, v)


@pytest.mark.parametrize("size,pad", [(2, 0), (2, 1), (3, 0), (1, 3)])   # odd strides: 8-byte accesses
def test_dyadic_accumulate_strides(orc, size, pad):
    n, L = 256, 2
    moduli = orc.coeff_modulus_create(n, [58, 40, 40])
    ctx = tb_capi.Context(BFV, n, moduli, 65537)
    rng = np.random.default_rng(size)
    na, nw, terms = 4, 5, [1, 70, 3]   # 70: more than one reduction of the sums
    a, w = _residues(rng, (na, size), moduli[:L], n), _residues(rng, (nw,), moduli[:L], n)
    sa, sw = size * L * n + pad, L * n + pad
    pa, pw = np.zeros((na, sa), np.uint64), np.zeros((nw, sw), np.uint64)
    pa[:, :size * L * n], pw[:, :L * n] = a.reshape(na, -1), w.reshape(nw, -1)
    off = np.concatenate([[0], np.cumsum(terms)]).astype(np.int32)
    ia, iw = rng.integers(0, na, off[-1], dtype=np.int32), rng.integers(0, nw, off[-1], dtype=np.int32)
    out = _empty(len(terms), sa)
    cu = lambda x: torch.from_numpy(x).cuda()  # noqa: E731
    ctx("dyadic_accumulate", L, size, _dev(pa), sa, _dev(pw), sw, out, sa, cu(off), cu(ia), cu(iw), len(terms), None)
    got = _host(out)[:, :size * L * n].reshape(len(terms), size, L, n)
    for o in range(len(terms)):
        exp = sum(a[ia[k]].astype(object) * w[iw[k]].astype(object)[None] for k in range(off[o], off[o + 1]))
        for l in range(L):
            assert np.array_equal(got[o, :, l], (exp[:, l] % moduli[l]).astype(np.uint64)), (o, l)


@pytest.mark.parametrize("bits,limbs", [(57, 1), (57, 6), (57, 7), (57, 8), (57, 14), (57, 16), (58, 8), (60, 7)])
def test_bfv_lift_sums(orc, bits, limbs):
    """The lift's split sums (moduli below 2^58, up to 16 limbs; folded every seven terms) and
    the general ones, with the largest residues among the inputs."""
    n = 256
    moduli = orc.coeff_modulus_create(n, [bits] * (limbs + 1))
    t = orc.plain_modulus_batching(n, 20)
    ctx = tb_capi.Context(BFV, n, moduli, t)
    data = moduli[:limbs]
    rng = np.random.default_rng(limbs)
    a, b = _residues(rng, (1, 2), data, n), _residues(rng, (1, 2), data, n)
    for l, q in enumerate(data):
        a[0, 0, l] = q - 1
        b[0, 1, l, ::2] = q - 1
    out = _empty(1, 3, limbs, n)
    ctx("multiply", limbs, _dev(a), 0, _dev(b), 0, out, 0, 1, None)
    assert np.array_equal(_host(out)[0], orc.bfv_multiply(n, data, t, a[0], b[0]))
