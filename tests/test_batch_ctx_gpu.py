"""The reference's BatchModCtx surface (batch_mod_ctx.cuh:132-179) on the GPU.

Compiles tests/cpp/batch_ctx_check.cpp -- a restatement of the reference's
own GMP-checked suite (correctness_tests.cuh:96-639) -- against
include/batch_mod_ctx.cuh, libpfb200.so and GMP (the declaration-only
oracle/include/gmp.h over the image's libgmp.so.10), and runs it: residue
round trips, raw squares and products against mpz_mul, modsq and modmul,
16 chained squarings, x^0xDEADBEEF against mpz_powm_ui, (N-1)^2 = 1 and
check_passed, for 512- to 332 000-bit moduli (five lengths, the longest, of
100 000 digits, on the integer engine).  Every check must pass on every
modulus.
"""
import ctypes as C
import os
import random
import subprocess

import numpy as np
import pytest

import pfb200

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GMP = next((p for p in ("/usr/lib/x86_64-linux-gnu/libgmp.so.10", "/usr/lib64/libgmp.so.10")
            if os.path.exists(p)), None)


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    if GMP is None:
        pytest.skip("no libgmp runtime")
    out = str(tmp_path_factory.mktemp("cpp") / "batch_ctx_check")
    libdir = os.path.dirname(pfb200.LIB_PATH)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "oracle", "include"), "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "batch_ctx_check.cpp"), "-o", out,
                    "-L", libdir, "-lpfb200", "-Wl,-rpath," + libdir, GMP,
                    "-L", "/usr/local/cuda/lib64", "-lcudart"], check=True)
    return out


def test_batch_mod_ctx_against_gmp(check):
    r = subprocess.run([check], capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stderr[-2000:]
    rows = [l.split() for l in r.stdout.strip().split("\n")]
    names = {row[0] for row in rows}
    assert names == {"roundtrip", "raw_sq", "raw_mul", "modsq", "modmul", "chain16", "powm", "nm1_sq",
                     "check_passed"}
    assert {int(row[1]) for row in rows} == {512, 2048, 20000, 166000, 332000}
    for name, bits, vals, ok, bad in rows:
        assert int(bad) == 0 and int(ok) > 0, (name, bits, vals)


def test_more_moduli_than_resident_blocks():
    """160 moduli of 50 000 digits (one block of the length class fits an SM):
    a square and a product of each, read back, against Python."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = random.Random(12)
    n, bits = 160, 166_000
    n16 = (bits + 15) // 16
    Ns = [rng.getrandbits(bits) | (1 << (bits - 1)) | 1 for _ in range(n)]
    ab = [[rng.randrange(N) for N in Ns] for _ in range(2)]

    def rows(xs):
        return np.frombuffer(b"".join(x.to_bytes(2 * n16, "little") for x in xs), dtype=np.uint16).astype(np.uint64)

    def ptr(x):
        return x.ctypes.data_as(C.POINTER(C.c_uint64))

    L, vp = C.CDLL(pfb200.LIB_PATH), C.c_void_p
    L.pfb_mr_ctx_modsq.argtypes = [vp, vp, vp, vp]
    L.pfb_mr_ctx_modmul.argtypes = [vp, vp, vp, vp, vp]
    L.pfb_mr_ctx_from_residue.argtypes = [vp, vp, C.POINTER(C.c_uint64)]
    L.pfb_mr_ctx_destroy.argtypes = [vp]
    eng, ctx = pfb200.MillerRabin(0), vp()
    assert L.pfb_mr_ctx_create(eng._h, ptr(rows(Ns)), n16, n, C.byref(ctx)) == 0
    a, b = (torch.from_numpy(rows(xs).astype(np.int64)).cuda() for xs in ab)
    t = torch.empty_like(a)
    out = np.zeros(n * n16, dtype=np.uint64)
    torch.cuda.synchronize()
    assert L.pfb_mr_ctx_modsq(ctx, a.data_ptr(), t.data_ptr(), None) == 0
    assert L.pfb_mr_ctx_modmul(ctx, t.data_ptr(), b.data_ptr(), t.data_ptr(), None) == 0
    assert L.pfb_mr_ctx_from_residue(ctx, t.data_ptr(), ptr(out)) == 0
    L.pfb_mr_ctx_destroy(ctx)
    eng.close()
    got = out.astype(np.uint16).reshape(n, n16)
    R = (1 << (22 * 8192)) + 1
    for i in range(n):
        x = int.from_bytes(got[i].tobytes(), "little")
        assert x < Ns[i] and (x * R % Ns[i] * R % Ns[i] * R - ab[0][i] ** 2 * ab[1][i]) % Ns[i] == 0, i
