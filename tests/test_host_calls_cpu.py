"""What the library's host code asks of the device, on a machine without a GPU: the
library is loaded over a stand-in for the CUDA runtime (fake_cudart.cpp) that records
allocations, copies and launches and runs no kernel. Each test runs in a process of its
own, so that the stand-in stays out of this one."""
import os
import subprocess
import sys
import textwrap

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
LIB = os.path.join(ROOT, "seal-cuda_b200", "lib", "libtroy_b200.so")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PRELUDE = """
import ctypes, sys
fake = ctypes.CDLL({fake!r}, mode=ctypes.RTLD_GLOBAL)
fake.fake_record.restype = ctypes.c_char_p
sys.path.insert(0, {python!r})
import tb_capi
from tb_capi import SCHEME_BFV, SCHEME_CKKS, SCHEME_BGV, SCHEME_RAW
lib = tb_capi.lib()
STREAM = 0x5000   # a stream that is not ordered after the legacy stream


def primes(n, *bits):
    out = (ctypes.c_uint64 * len(bits))()
    tb_capi.check(lib.tb_coeff_modulus_create(ctypes.c_uint64(n), (ctypes.c_int * len(bits))(*bits), len(bits), out))
    return [int(q) for q in out]


def context(scheme, n, *bits):
    t = ctypes.c_uint64(0)
    if scheme in (SCHEME_BFV, SCHEME_BGV):
        tb_capi.check(lib.tb_plain_modulus_batching(ctypes.c_uint64(n), 20, ctypes.byref(t)))
    return tb_capi.Context(scheme, n, primes(n, *bits), t.value)


def words(n):
    # a device buffer (the stand-in's device memory is host memory), 256-byte aligned
    raw = (ctypes.c_uint64 * (n + 32))()
    words.keep.append(raw)
    return (ctypes.addressof(raw) + 255) // 256 * 256


words.keep = []


def calls(f):
    # the records of f(): tuples (kind, numbers..., [kernel name])
    fake.fake_reset()
    f()
    out = []
    for line in fake.fake_record().decode().splitlines():
        out.append(tuple(int(x) if x.isdigit() else x for x in line.split()))
    return out


def kinds(records, kind):
    return [r[1:] for r in records if r[0] == kind]
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    """Runs a program over the stand-in runtime in a fresh process; fails with its output."""
    if not os.path.exists(LIB):
        pytest.skip("library not built")
    so = str(tmp_path_factory.mktemp("fake") / "libcudart.so.12")
    script = so + ".map"
    with open(script, "w") as f:
        f.write("libcudart.so.12 { global: *; };\n")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(CUDA, "include"),
                    os.path.join(HERE, "fake_cudart.cpp"), "-o", so, "-Wl,-soname,libcudart.so.12",
                    "-Wl,--version-script=" + script], check=True)
    prelude = PRELUDE.format(fake=so, python=os.path.join(ROOT, "seal-cuda_b200", "python"))

    def run(program):
        r = subprocess.run([sys.executable, "-c", prelude + textwrap.dedent(program)], capture_output=True, text=True,
                           timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
        return r.stdout

    return run


@pytest.mark.parametrize("context,first_use", [
    ("SCHEME_CKKS, 4096, 40, 40, 41", "'ckks_decode', 2, words(8192), 2.0 ** 30, words(4096), 0, 1, STREAM"),
    ("SCHEME_CKKS, 4096, 40, 40, 41", "'ckks_encode', 2, words(4096), 0, 2048, 2.0 ** 30, words(8192), 1, STREAM"),
    ("SCHEME_BFV, 4096, 36, 36, 37", "'batch_encode', words(4096), 0, 4096, words(4096), 1, STREAM"),
    ("SCHEME_CKKS, 4096, 40, 40, 41",
     "'apply_galois', 2, 3, words(16384), 0, words(16384), 0, words(49152), 1, STREAM"),
], ids=["crt_constants", "fft_roots", "slot_map", "galois_table"])
def test_tables_of_a_first_call_are_on_the_device_before_its_kernels(host, context, first_use):
    host(f"""
        c = context({context})
        fake.cudaStreamSynchronize(None)   # the context's own tables: the test below
        records = calls(lambda: c({first_use}))
        assert kinds(records, "launch")
        assert not kinds(records, "race"), kinds(records, "race")
        """)


@pytest.mark.parametrize("context,call", [
    ("SCHEME_RAW, 4096, 40, 41", "'ntt_forward', words(8192), words(8192), 1, 0, 2, 0, STREAM"),
    ("SCHEME_RAW, 2048, 36, 37", "'ntt_forward', words(4096), words(4096), 1, 0, 2, 0, STREAM"),
    ("SCHEME_BGV, 4096, 36, 36, 37",
     "'multiply', 2, words(16384), 0, words(16384), 0, words(24576), 0, 1, STREAM"),
    ("SCHEME_BFV, 2048, 27, 27",
     "'multiply', 1, words(4096), 0, words(4096), 0, words(6144), 0, 1, STREAM"),
], ids=["fp64_tables", "twiddles", "bgv", "bfv"])
def test_tables_of_a_context_are_on_the_device_when_it_is_returned(host, context, call):
    host(f"""
        c = context({context})
        records = calls(lambda: c({call}))
        assert kinds(records, "launch")
        assert not kinds(records, "race"), kinds(records, "race")
        """)


@pytest.mark.parametrize("batch,shift,stride", [(3, 0, 4098), (3, 0, 8192), (2, 4096, 4096), (3, -4096, 4096),
                                                (5, 8, 4096), (3, 0, 4096), (3, 0, 0), (3, 3 * 4096, 4100)])
def test_batch_decode_reads_no_plaintext_that_it_may_have_written(host, batch, shift, stride):
    """Slots over the plaintexts: the transforms of one launch run in any order, so unless
    every plaintext is replaced by its own slots, they read a copy."""
    host(f"""
        n, batch, shift, stride = 4096, {batch}, {shift}, {stride}
        c = context(SCHEME_BFV, n, 36, 36, 37)
        base = words((2 * batch + 4) * 8192) + 8 * n
        plain, slots = base, base + 8 * shift
        records = calls(lambda: c("batch_decode", plain, slots, stride, batch, STREAM))
        (stream, blocks, threads, src, dst, name), = [r for r in kinds(records, "launch") if "BatchDecodeOp" in r[5]]
        s = stride or n
        assert dst == slots
        reads, writes = (src, src + 8 * batch * n), (dst, dst + 8 * ((batch - 1) * s + n))
        disjoint = reads[1] <= writes[0] or writes[1] <= reads[0]
        assert disjoint or (src == dst and s == n), (reads, writes)
        copies = kinds(records, "copy")
        assert src == plain or copies == [(STREAM, src, plain, 8 * batch * n)]
        """)


@pytest.mark.parametrize("call", ["ckks_decode", "ckks_decode_polynomial"])
@pytest.mark.parametrize("offset", [0, 8])
def test_ckks_decode_transforms_aligned_words(host, call, offset):
    """The transforms load pairs of words at once; a plaintext that starts in the middle of
    a pair is copied first."""
    host(f"""
        c = context(SCHEME_CKKS, 4096, 40, 40, 41)
        plain = words(3 * 4096) + {offset}
        records = calls(lambda: c("{call}", 2, plain, 2.0 ** 30, words(4096), 0, 1, STREAM))
        (stream, blocks, threads, src, dst, name), = [r for r in kinds(records, "launch") if "PlainNttOp" in r[5]]
        assert src % 16 == 0 and dst % 16 == 0, (src, dst)
        copies = kinds(records, "copy")
        assert src == plain or copies == [(STREAM, src, plain, 8 * 2 * 4096)]
        assert (src == plain) == ({offset} == 0)
        """)


@pytest.mark.parametrize("n,tables", [(8192, 4), (16384, 4), (32768, 2), (65536, 2)])
def test_twiddle_memory(host, n, tables):
    """Twiddles in natural order, forward and inverse, and again in the order of the radix-8
    passes where one CTA transforms a whole limb (up to 2^14 coefficients) and reads that."""
    host(f"""
        moduli = primes({n}, 60, 60, 60)
        records = calls(lambda: tb_capi.Context(SCHEME_RAW, {n}, moduli, 0))
        assert max(b for _, b in kinds(records, "malloc")) == 16 * {n} * {tables} * len(moduli)
        """)


@pytest.mark.parametrize("logn,limbs", [(12, 37), (12, 6 * 148), (13, 37), (13, 3 * 148), (14, 74)])
@pytest.mark.parametrize("forward", [0, 1])
def test_size_rules_are_off_with_the_switch(host, logn, limbs, forward):
    """Launches of few and of many limbs take the set variant with the small-launch rules
    off, and forms of their own with them on."""
    host(f"""
        logn, limbs, forward = {logn}, {limbs}, {forward}
        n = 1 << logn
        c = context(SCHEME_RAW, n, 40)
        x = words(limbs * n)

        def shape():
            records = calls(lambda: c("ntt_forward" if forward else "ntt_inverse", x, x, limbs, 0, 1, 0, STREAM))
            (stream, blocks, threads, src, dst, name), = kinds(records, "launch")
            return blocks, threads

        own = shape()
        lib.tb_ntt_set_small_launch_pairs(0)
        for v in (0, 1, 2):
            tb_capi.check(lib.tb_ntt_set_variant(forward, logn, v))
            assert shape() == (limbs, min(1024, n // 8) >> v), v
        tb_capi.check(lib.tb_ntt_set_variant(forward, logn, 0))
        assert own != shape()
        lib.tb_ntt_set_small_launch_pairs(1)
        assert own == shape()
        """)
