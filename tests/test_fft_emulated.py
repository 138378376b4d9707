"""The floating-point Montgomery engine (csrc/fft_device.cuh,
csrc/fft_kernels.cuh), unchanged, on the CPU through the stand-in CUDA
runtime of tests/cpp/emul/.

One squaring per length class at the widest limbs the class may use, on limb
patterns of the largest size a limb can have, must equal the integer result
exactly (x^2 / R' mod N, R' = 2^(n b) + 1); whole tests and modular powers
must equal Python's and the oracle's.
"""
import os
import random
import subprocess

import pytest

import lucas
import oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# complex points and widest limb of every class
CLASSES = [(64, 19), (96, 18), (128, 18), (192, 18), (256, 17), (384, 17), (512, 17), (768, 16), (1024, 16),
           (1536, 16), (2048, 16), (3072, 15), (4096, 15), (6144, 15), (8192, 15), (12288, 14)]


def _build(exe, *flags):
    subprocess.run(["g++", *flags, "-std=c++20", "-Wno-unknown-pragmas",
                    "-I", os.path.join(ROOT, "tests", "cpp", "emul"),
                    "-I", os.path.join(ROOT, "prime-finder_b200", "csrc"),
                    "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cpp", "fft_job_emul.cpp"), "-o", exe], check=True)


@pytest.fixture(scope="module")
def emul(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fft") / "fft_job_emul")
    _build(exe, "-O2")

    def run(lines):
        out = subprocess.run([exe], input="\n".join(lines) + "\n", capture_output=True, text=True, check=True,
                             timeout=900).stdout.strip().split("\n")
        assert len(out) == len(lines)
        return [line.split() for line in out]
    return run


@pytest.mark.parametrize("cls", range(len(CLASSES)))
def test_one_squaring_with_the_largest_limbs(emul, cls):
    rng = random.Random(100 + cls)
    n, top = 2 * CLASSES[cls][0], CLASSES[cls][1]
    cases = []
    for b in {top, 11}:
        for kind in range(5):
            for dbl in (0, 1):
                N = rng.getrandbits(n * b - 7) | 1 | (1 << (n * b - 8))
                if kind == 3:  # every balanced digit of N at its largest
                    N = sum((1 << (b - 1)) << (b * i) for i in range(n - 1)) | 1
                cases.append((b, dbl, kind, N))
    out = emul(["step %d %d %d %d %x" % (cls, b, dbl, kind, N) for b, dbl, kind, N in cases])
    for (b, dbl, kind, N), o in zip(cases, out):
        if o == ["none"]:  # N shares a factor with R': the host takes another radix
            continue
        x, y, limb = int(o[0], 16), int(o[1], 16), int(o[2])
        R = (1 << (n * b)) + 1
        assert (y * R - (x * x << dbl)) % N == 0, (cls, b, dbl, kind)
        assert abs(y) < (N * 7 // 10 << dbl) and limb <= (1 << (b - 1)) + 40, (cls, b, dbl, kind)


def test_strong_tests(emul):
    rng = random.Random(11)
    ns = [3, 5, 7, 9, 15, 17, 257, 561, 1105, 2047, 3277, 65537, 1000001, (1 << 61) - 1, (1 << 521) - 1, 2 ** 64 + 13]
    ns += [rng.getrandbits(b) | 1 | (1 << (b - 1)) for b in (24, 33, 100, 1000, 2426, 2427, 4600)]
    cases = [(2, n) for n in ns] + [(3, 1000003), (7, 3215031751), (65535, 1000033), (3, 561), (65535, 65537)]
    for (a, n), o in zip(cases, emul(["job 1 %d %x" % c for c in cases])):
        res = oracle.strong_residue(n, a)[1]
        assert (int(o[2]), int(o[3], 16)) == (oracle.strong_test(n, a), res), (a, n)


def test_modular_powers_of_every_class(emul):
    """Short exponents at both ends of every class."""
    rng = random.Random(13)
    cases = []
    for (C, top), lower in zip(CLASSES, [(0, 0)] + CLASSES):
        for bits in (2 * lower[0] * lower[1] - 5, 2 * C * top - 6):
            if bits > 0:
                N = rng.getrandbits(bits) | 1 | (1 << (bits - 1))
                cases.append((rng.choice([2, 2, 3]), N, rng.getrandbits(10) | 512))
    out = emul(["job 0 %d %x %x" % c for c in cases])
    for (a, N, E), o in zip(cases, out):
        assert int(o[3], 16) == pow(a, E, N), (a, N.bit_length(), o[:2])
    assert {int(o[0]) for o in out} == set(range(len(CLASSES)))


@pytest.mark.parametrize("bits", [2 * C * b - 9 for C, b in CLASSES[12:]])
def test_overlapping_launches_of_one_class(emul, bits):
    """Two launches on candidates of one class (advances of a resident batch on
    two streams), the second running between the passes of the first one's
    steps: neither touches what the other keeps in global memory."""
    rng = random.Random(bits)
    case = []
    for _ in range(2):
        case += [rng.getrandbits(bits) | 1 | (1 << (bits - 1)), rng.getrandbits(7) | 64]
    o = emul(["overlap 2 %x %x %x %x" % tuple(case)])[0]
    assert [int(x, 16) for x in o[1:]] == [pow(2, case[1], case[0]), pow(2, case[3], case[2])]


def test_strong_lucas_tests(emul):
    rng = random.Random(12)
    ns = [5459, 5777, 10877, 16109, 18971, 3, 5, 7, 11, 13, 25, 49, 1000003, 1000001, (1 << 61) - 1, (1 << 127) - 1]
    ns += [rng.getrandbits(b) | 1 | (1 << (b - 1)) for b in (30, 50, 70)]
    for D in (5, -7, -11, 13, -15, 17, -19, -23):  # one composite and one prime per Q
        for want_prime in (False, True):
            while True:
                n = rng.getrandbits(100) | (1 << 99) | 1
                n = oracle.nextprime(n) if want_prime else n
                if lucas.selfridge_d(n) == D:
                    break
            ns.append(n)
    assert [int(o[2]) for o in emul(["job 2 2 %x" % n for n in ns])] == [lucas.strong_lucas(n) for n in ns]


@pytest.mark.parametrize("cls", [c for c, (C, _) in enumerate(CLASSES) if C >= 128 and C & (C - 1) == 0])
def test_context_operations(emul, cls):
    """Fully reduced results in the integer engine's radix, 2^(22 C) + 1, with
    operands up to N - 1 and moduli that fill the length or are short."""
    rng = random.Random(40 + cls)
    C = CLASSES[cls][0]
    ri = None
    lines, want = [], []
    for bits in (22 * C - 6, 22 * C - 37, max(20, 11 * C - 3)):
        N = rng.getrandbits(bits) | 1 | (1 << (bits - 1))
        try:
            ri = pow((1 << (22 * C)) + 1, -1, N)
        except ValueError:
            continue
        for a, b in ((rng.randrange(N), rng.randrange(N)), (N - 1, N - 1), (0, 1), (1, N - 2)):
            for op, r in ((0, a * a * ri % N), (1, a * b * ri % N), (4, a * ri % N)):
                lines.append("ctx %d %d %x %x %x" % (cls, op, N, a, b))
                want.append(r)
    out = emul(lines)
    for line, o, r in zip(lines, out, want):
        assert int(o[0], 16) == r, line[:20]


def test_in_bounds_under_address_sanitizer(tmp_path):
    exe = str(tmp_path / "fft_job_asan")
    _build(exe, "-O1", "-g", "-fsanitize=address")
    rng = random.Random(3)
    lines = ["job 1 2 %x" % n for n in (3, 561, (1 << 89) - 1)] + ["job 1 7 %x" % 1000003]
    lines += ["job 2 2 %x" % n for n in (5459, (1 << 61) - 1)] + ["ctx 14 1 %x 5 7" % ((1 << 900) - 1)]
    for cls, (C, b) in enumerate(CLASSES):
        lines.append("step %d %d 1 4 %x" % (cls, b, rng.getrandbits(2 * C * b - 7) | 1 | (1 << (2 * C * b - 8))))
    r = subprocess.run([exe], input="\n".join(lines) + "\n", capture_output=True, text=True, timeout=900,
                       env=dict(os.environ, ASAN_OPTIONS="detect_leaks=0"))
    assert r.returncode == 0, r.stderr[-2000:]
    assert len(r.stdout.strip().split("\n")) == len(lines)
