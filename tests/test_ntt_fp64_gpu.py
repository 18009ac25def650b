"""Transforms in exact FP64 arithmetic (moduli below 2^50, N = 4096 .. 32768) against the
oracle, word for word: primes at the edges of the form (the largest below 2^48, which run
without reductions, the largest below 2^49 and 2^50, which reduce at every pass, the first
one above 2^50, in integer form, and small ones), extreme inputs (all q - 1, alternating,
up to 4 q - 1 where the transforms take lazy words), and launches on both sides of every
size rule, which count limbs against the device's SMs: up to a quarter of them clusters of
eight CTAs, up to half CTA pairs, then one CTA a limb (2^15: CTA pairs), and from three
(2^13) or six (2^12) limbs an SM on half the threads."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import tb_capi  # noqa: E402
from test_ntt_gpu import _dev, _host, _is_prime, _ntt_prime  # noqa: E402


def _prime_above(bits, m):
    q = (1 << bits) // m * m + 1
    while q < (1 << bits) or not _is_prime(q):
        q += m
    return q


def _rows(n, q, top, seed):
    """Input polynomials with words below `top` (q, or 4 q for lazy words)."""
    rng = np.random.default_rng(seed)
    rows = np.stack([np.full(n, top - 1, np.uint64), np.zeros(n, np.uint64),
                     rng.integers(0, top, n, dtype=np.uint64), rng.integers(0, 2, n, dtype=np.uint64) * np.uint64(top - 1)])
    rows[1, ::2] = top - 1
    return rows


def _counts(logn):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    many = {12: 6 * sms, 13: 3 * sms}.get(logn)
    return sorted({1, 4, sms // 4, sms // 4 + 1, sms // 2, sms // 2 + 1, sms + 12,
                   *((many - 1, many, many + 12) if many else (460,))})


@pytest.mark.parametrize("logn", [12, 13, 14, 15])
@pytest.mark.parametrize("kind", ["20", "40", "48", "49", "50", "above50"])
def test_fp64_transforms(orc, logn, kind):
    n = 1 << logn
    q = _prime_above(50, 2 * n) if kind == "above50" else _ntt_prime(int(kind), 2 * n)
    ctx = tb_capi.Context(tb_capi.SCHEME_RAW, n, [q])
    for top in (q, 4 * q):
        rows = _rows(n, q, top, logn)
        fwd = np.stack([orc.ntt_forward(logn, q, r) for r in rows])
        lazy = rows % np.uint64(2 * q)   # the inverse takes words below 2 q
        inv = np.stack([orc.ntt_inverse(logn, q, r) for r in lazy])
        for polys in _counts(logn):
            x = _dev(np.ascontiguousarray(np.resize(rows, (polys, n))))
            out = torch.empty_like(x)
            ctx("ntt_forward", x, out, polys, 0, 1, 0, None)
            assert np.array_equal(_host(out), np.resize(fwd, (polys, n))), ("forward", polys, top // q)
            y = _dev(np.ascontiguousarray(np.resize(lazy, (polys, n))))
            ctx("ntt_inverse", y, out, polys, 0, 1, 0, None)
            assert np.array_equal(_host(out), np.resize(inv, (polys, n))), ("inverse", polys, top // q)
            ctx("ntt_forward", x, x, polys, 0, 1, 0, None)   # in place
            assert np.array_equal(_host(x), np.resize(fwd, (polys, n))), ("in place", polys, top // q)
    ctx.close()
