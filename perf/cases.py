"""Timed work of the two hot paths: the Phase-1 sieve and the Miller-Rabin engine.

Every case goes through a public entry point of ``pfb200`` (or of the C ABI
behind it where the package has no wrapper) with inputs made from a seed:

  dropin    trial_div_gpu: host prime list, 100 x 100 grid, one triple
  sieve     Sieve.run on a resident prime list into a device mask, then
            Sieve.survivors per triple: what Phase 1 of a search does
  masks     Sieve.run of many triples with the masks returned to the host
  test      MillerRabin.test: strong base-2 tests, verdicts and residues
  powm      MillerRabin.powm: modular powers with the exponents given
  lucas     MillerRabin.lucas: strong Lucas tests
  ctx       pfb_mr_ctx_modsq / modmul chains (BatchModCtx's operations) on a
            context of many moduli, read back with from_residue
  pipeline  pipeline_run: sieve, then decide every survivor

The numbers are the search's candidates N = 10^a - k 10^b - j 10^c - 1 and
rev(N), the triples follow ``pfb200.workloads.uneven_tuples`` (c small, b
anywhere below a) scaled to the digit count.
"""
import ctypes as C
import functools
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "prime-finder_b200"))

import pfb200  # noqa: E402


def listed():
    return [
        # the reference's own call: every odd prime below 1e8, one triple, 100 x 100 grid
        {"name": "dropin_1e8", "kind": "dropin", "limit": 100_000_000, "digits": 50_000},
        # the same call with a short list: the smallest sieve, launch latency counts
        {"name": "dropin_1e5", "kind": "dropin", "limit": 100_000, "digits": 3_000},
        # one wide grid of a production search with the full prime list
        {"name": "sieve_9999", "kind": "sieve", "limit": 100_000_000, "K": 9999, "n": 1, "digits": 50_000},
        # a few ragged medium grids, shorter list
        {"name": "sieve_1237", "kind": "sieve", "limit": 20_000_000, "K": 1237, "n": 3, "digits": 70_000},
        # many triples of the reference's grid in one call, masks to the host
        {"name": "masks_100", "kind": "masks", "limit": 10_000_000, "K": 100, "n": 64, "digits": 50_000},
        # a handful of short numbers: the latency of one call
        {"name": "test_few", "kind": "test", "n": 5, "lo": 200, "hi": 600},
        # an ordinary batch, two candidates per SM, uneven lengths
        {"name": "test_batch", "kind": "test", "n": 296, "lo": 1_000, "hi": 3_000},
        # longer numbers, fewer than SMs
        {"name": "test_long", "kind": "test", "n": 61, "lo": 5_000, "hi": 10_000},
        # strong Lucas tests: general products beside squarings
        {"name": "lucas", "kind": "lucas", "n": 40, "lo": 400, "hi": 900},
        # the squaring chain of the 50 000-digit batch, four squarings to a product
        {"name": "ctx_50k", "kind": "ctx", "n": 128, "digits": 50_000, "ops": 24},
        # 100 000-digit modular powers, the longest numbers the engine takes
        {"name": "powm_100k", "kind": "powm", "n": 16, "lo": 99_000, "hi": 100_000, "ebits": 3_000},
        # a whole small search: sieve, strong tests, remaining rounds
        {"name": "pipeline", "kind": "pipeline", "limit": 1_000_000, "K": 60, "n": 3, "lo": 300, "hi": 500},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dropin", "sieve", "masks", "test", "powm", "lucas", "ctx", "pipeline"])
    if kind == "dropin":
        return {"kind": kind, "limit": _log(rng, 50_000, 100_000_000), "digits": _log(rng, 1_000, 100_000)}
    if kind == "sieve":
        K = _log(rng, 40, 9_999)
        return {"kind": kind, "limit": _log(rng, 1_000_000, 100_000_000), "K": K,
                "n": 1 if K > 3_000 else rng.randint(1, 4), "digits": _log(rng, 3_000, 100_000)}
    if kind == "masks":
        return {"kind": kind, "limit": _log(rng, 100_000, 10_000_000), "K": rng.randint(50, 150),
                "n": rng.randint(3, 64), "digits": _log(rng, 3_000, 100_000)}
    if kind in ("test", "lucas"):
        lo = _log(rng, 120, 4_000 if kind == "test" else 700)
        n = max(1, min(_log(rng, 1, 300), int(148 * max(1.0, (2_500.0 / lo) ** 2))))
        return {"kind": kind, "n": n if kind == "test" else max(8, min(n, 60)), "lo": lo,
                "hi": int(lo * rng.uniform(1.0, 2.5))}
    if kind == "powm":
        lo = _log(rng, 3_000, 100_000)
        return {"kind": kind, "n": rng.randint(1, 16), "lo": lo, "hi": min(100_000, int(lo * rng.uniform(1.0, 1.5))),
                "ebits": rng.randint(300, 3_000)}
    if kind == "ctx":
        d = _log(rng, 300, 100_000)
        return {"kind": kind, "n": rng.randint(1, 128 if d <= 55_000 else 48), "digits": d, "ops": rng.randint(4, 24)}
    lo = rng.randint(120, 400)
    return {"kind": kind, "limit": _log(rng, 100_000, 1_000_000), "K": rng.randint(20, 60), "n": rng.randint(1, 3),
            "lo": lo, "hi": lo + rng.randint(0, 100)}


# ------------------------------------------------------------------ inputs ---

@functools.lru_cache(maxsize=8)
def _primes(limit):
    """Odd primes below limit (Eratosthenes over the odd numbers)."""
    s = np.ones(limit // 2, dtype=bool)
    s[0] = False
    for i in range(3, math.isqrt(limit) + 1, 2):
        if s[i // 2]:
            s[i * i // 2::i] = False
    return (2 * np.nonzero(s)[0] + 1).astype(np.uint32)


@functools.lru_cache(maxsize=None)
def _engine():
    return pfb200.MillerRabin(0)


@functools.lru_cache(maxsize=None)
def _ctx_lib():
    L = pfb200.lib()
    vp, u64 = C.c_void_p, C.POINTER(C.c_uint64)
    L.pfb_mr_ctx_create.argtypes = [vp, u64, C.c_int, C.c_int, C.POINTER(vp)]
    L.pfb_mr_ctx_modsq.argtypes = [vp, vp, vp, vp]
    L.pfb_mr_ctx_modmul.argtypes = [vp, vp, vp, vp, vp]
    L.pfb_mr_ctx_from_residue.argtypes = [vp, vp, u64]
    L.pfb_mr_ctx_destroy.argtypes = [vp]
    L.pfb_mr_ctx_destroy.restype = None
    return L


def _triple(rng, digits):
    """(a, b, c): a within 2 % of digits, c from a/500 to a/50, b anywhere between c and a."""
    while True:
        a = rng.randint(digits - digits // 50, digits)
        c = rng.randint(a // 500 + 1, a // 50 + 2)
        b = rng.randint(c + 1, a - 1)
        if a - b >= 6 and b - c >= 5:
            return a, b, c


_SMALL = [p for p in range(3, 200, 2) if all(p % q for q in range(3, 15, 2) if q < p)]


def _candidates(rng, n, lo, hi):
    """n candidates of lo..hi digits with no prime factor below 200, N and rev(N) alike."""
    out = []
    while len(out) < n:
        a, b, c = _triple(rng, rng.randint(lo, hi))
        for _ in range(200):
            k, j, rev = rng.randint(1, 9999), rng.randint(1, 9999), bool(rng.getrandbits(1))
            x = pfb200.build_candidate(a, b, c, k, j, rev)
            r = x % math.prod(_SMALL)
            if all(r % p for p in _SMALL):
                out.append(x)
                break
    return out


def _short_prime(rng):
    """A prime of 100 to 200 bits (Fermat to four bases)."""
    while True:
        x = rng.getrandbits(rng.randint(100, 200)) | 1
        if x > 1 << 90 and all(x % p for p in _SMALL) and all(pow(b, x - 1, x) == 1 for b in (2, 3, 5, 7)):
            return x


def _room(K):
    """Survivors a list has room for (a sieved grid keeps a few per cent)."""
    return K * K // 8 + 64


class _Ctx:
    """A context of moduli with its device operands."""

    def __init__(self, moduli, n16, a, b):
        L = _ctx_lib()
        arr = np.zeros((len(moduli), n16), dtype=np.uint64)
        for i, x in enumerate(moduli):
            l = pfb200.int_to_limbs16(x)
            arr[i, :len(l)] = l
        h = C.c_void_p()
        rc = L.pfb_mr_ctx_create(_engine()._h, arr.ctypes.data_as(C.POINTER(C.c_uint64)), n16, len(moduli), C.byref(h))
        if rc:
            raise pfb200.PfbError(rc, "pfb_mr_ctx_create")
        self.h = h
        self.a = torch.from_numpy(a.astype(np.int64)).cuda()
        self.b = torch.from_numpy(b.astype(np.int64)).cuda()
        self.t = [torch.empty_like(self.a) for _ in range(2)]
        self.out = np.zeros((len(moduli), n16), dtype=np.uint64)

    def __del__(self):
        if getattr(self, "h", None):
            _ctx_lib().pfb_mr_ctx_destroy(self.h)
            self.h = None


def _ctx_inputs(case, seed):
    rng = random.Random(seed)
    moduli = _candidates(rng, case["n"], case["digits"], case["digits"])
    n16 = max(len(pfb200.int_to_limbs16(x)) for x in moduli)
    # working forms below each modulus: its top limb left zero
    ab = np.random.default_rng(seed).integers(0, 1 << 16, size=(2, case["n"], n16), dtype=np.int64)
    for i, x in enumerate(moduli):
        ab[:, i, len(pfb200.int_to_limbs16(x)) - 1:] = 0
    return moduli, n16, ab[0], ab[1]


def prepare(case, seed):
    kind, rng = case["kind"], random.Random(seed)
    if kind == "dropin":
        return {"case": case, "primes": _primes(case["limit"]), "abc": _triple(rng, case["digits"])}
    if kind in ("sieve", "masks"):
        abc = [_triple(rng, case["digits"]) for _ in range(case["n"])]
        st = {"case": case, "abc": abc, "sieve": pfb200.Sieve(_primes(case["limit"]))}
        if kind == "sieve":
            K = case["K"]
            st["mask"] = torch.zeros((case["n"], pfb200.mask_bytes(K)), dtype=torch.uint8, device="cuda")
            st["list"] = torch.zeros((case["n"], _room(K)), dtype=torch.int32, device="cuda")
        return st
    if kind in ("test", "lucas", "powm"):
        xs = _candidates(rng, case["n"], case["lo"], case["hi"])
        if kind == "lucas":  # one number in four is a prime, as among base-2 probable primes
            xs = [_short_prime(rng) if rng.random() < 0.25 else x for x in xs]
        st = {"case": case, "numbers": [pfb200.int_to_limbs16(x) for x in xs]}
        if kind == "powm":
            st["exps"] = [pfb200.int_to_limbs16(rng.getrandbits(case["ebits"]) | (1 << (case["ebits"] - 1)))
                          for _ in xs]
        _engine()
        return st
    if kind == "ctx":
        return {"case": case, "ctx": _Ctx(*_ctx_inputs(case, seed))}
    abc = [_triple(rng, rng.randint(case["lo"], case["hi"])) for _ in range(case["n"])]
    return {"case": case, "abc": abc, "sieve": pfb200.Sieve(_primes(case["limit"])), "engine": _engine()}


# ------------------------------------------------------------------- calls ---

def _limbs(xs, case):
    """Residues as rows of 16-bit limbs, wide enough for the longest number of the case."""
    out = np.zeros((len(xs), int(case["hi"] * math.log2(10) / 16) + 2), dtype=np.int32)
    for i, x in enumerate(xs):
        l = pfb200.int_to_limbs16(x)
        out[i, :len(l)] = l
    return out


def _records(recs, case):
    """Records as rows (a, b, c, k, j, result), zero rows up to the size of the grid."""
    out = np.zeros((case["n"] * case["K"] ** 2, 6), dtype=np.int64)
    out[:len(recs)] = np.array(recs, dtype=np.int64).reshape(-1, 6)
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "dropin":
        return pfb200.trial_div_gpu(state["primes"], *state["abc"]).view(np.int32)
    if kind == "masks":
        return state["sieve"].run(state["abc"], case["K"])
    if kind == "sieve":
        sv, K = state["sieve"], case["K"]
        sv.run(state["abc"], K, mask=state["mask"])
        counts = [sv.survivors(state["mask"][t], K, state["list"][t], _room(K)) for t in range(case["n"])]
        return [state["mask"], state["list"], np.array(counts, dtype=np.int64)]
    if kind == "test":
        ver, res = _engine().test(state["numbers"])
        return {"verdicts": np.array(ver, dtype=np.int32), "residues": _limbs(res, case)}
    if kind == "lucas":
        return np.array(_engine().lucas(state["numbers"]), dtype=np.int32)
    if kind == "powm":
        return _limbs(_engine().powm(state["numbers"], state["exps"]), case)
    if kind == "ctx":
        L, c = _ctx_lib(), state["ctx"]
        st = torch.cuda.current_stream().cuda_stream or None
        x = c.a
        for i in range(case["ops"]):
            y = c.t[i & 1]
            if i % 5 == 4:
                rc = L.pfb_mr_ctx_modmul(c.h, x.data_ptr(), c.b.data_ptr(), y.data_ptr(), st)
            else:
                rc = L.pfb_mr_ctx_modsq(c.h, x.data_ptr(), y.data_ptr(), st)
            if rc:
                raise pfb200.PfbError(rc, "pfb_mr_ctx")
            x = y
        rc = L.pfb_mr_ctx_from_residue(c.h, x.data_ptr(), c.out.ctypes.data_as(C.POINTER(C.c_uint64)))
        if rc:
            raise pfb200.PfbError(rc, "pfb_mr_ctx_from_residue")
        return {"working": x, "plain": c.out.astype(np.int32)}
    recs, _ = pfb200.pipeline_run(state["sieve"], state["engine"], state["abc"], case["K"])
    return _records(recs, case)


# -------------------------------------------------------------------- work ---

def _pi(x):
    return x / (math.log(x) - 1.08) if x > 10 else 4.0


def _square_ops(bits):
    """Operations of one modular squaring of `bits` bits: a full product and
    two half products (quotient and remainder) of n = bits/16 digits through
    real transforms of 2.5 n log2 n operations; six transforms of length 2n
    and n each way come to about eight of length n."""
    n = bits / 16.0
    return 8 * 2.5 * n * math.log2(max(2.0, n))


def _sieve_work(limit, K, n, digits):
    primes = _pi(limit)
    # two powers of ten per prime (the slope and the offset), one division
    # chain, and a mark per hit: 2 K^2 sum(1/p) of them
    ops = n * (primes * (2 * 2 * math.log2(digits) + 2 * math.log2(limit)) +
               2.0 * K * K * (math.log(math.log(limit)) + 0.26 - 0.5))
    return {"bytes": 4.0 * primes + n * K * K / 8.0, "flops": ops}


def work(case):
    kind = case["kind"]
    if kind == "dropin":
        return _sieve_work(case["limit"], 100, 1, case["digits"])
    if kind in ("sieve", "masks"):
        return _sieve_work(case["limit"], case["K"], case["n"], case["digits"])
    if kind == "ctx":
        bits = case["digits"] * math.log2(10)
        return {"bytes": case["n"] * (4 * bits / 16 * 8), "flops": case["n"] * case["ops"] * _square_ops(bits)}
    if kind == "pipeline":
        bits = (case["lo"] + case["hi"]) / 2 * math.log2(10)
        w = _sieve_work(case["limit"], case["K"], case["n"], case["lo"])
        # survivors: about 1 / (1.78 ln limit / 2)^2 of the grid (both forms free of small factors)
        surv = case["n"] * case["K"] ** 2 * min(1.0, (2 / (1.78 * math.log(case["limit"]))) ** 2)
        return {"bytes": w["bytes"] + surv * bits / 8, "flops": w["flops"] + surv * bits * _square_ops(bits)}
    bits = (case["lo"] + case["hi"]) / 2 * math.log2(10)
    steps = case["ebits"] if kind == "powm" else bits * (2.5 if kind == "lucas" else 1.0)
    return {"bytes": 2 * case["n"] * bits / 8, "flops": case["n"] * steps * _square_ops(bits)}


def tolerance(case):
    return "exact"  # bit masks, verdicts, residues and records


# ------------------------------------------------------------------- exact ---

def _powmod(base, e, p):
    """base^e mod p over arrays of p < 2^32 (uint64 arithmetic)."""
    r, x = np.ones_like(p), base % p
    while e:
        if e & 1:
            r = r * x % p
        x = x * x % p
        e >>= 1
    return r


def _rev(x):
    return int(str(x)[::-1])


def _grid(primes, a, b, c, K):
    """mask[k-1, j-1]: some odd prime p != 5 of the list divides N or rev(N)."""
    mask = np.zeros((K, K), dtype=bool)
    p = primes[(primes != 5) & (primes > 2)].astype(np.uint64)
    small = p[p < 4 * K]
    for q in (int(v) for v in small):  # every cell's residue
        k, j = np.arange(1, K + 1), np.arange(1, K + 1)
        n = (pow(10, a, q) - (k * pow(10, b, q))[:, None] - (j * pow(10, c, q))[None, :] - 1) % q
        rk = np.array([_rev(v) * pow(10, a - b - len(str(v)), q) % q for v in range(1, K + 1)])
        rj = np.array([_rev(v) * pow(10, a - c - len(str(v)), q) % q for v in range(1, K + 1)])
        r = (pow(10, a, q) - rk[:, None] - rj[None, :] - 1) % q
        mask |= (n == 0) | (r == 0)
    p = p[p >= 4 * K]
    one, ten = np.uint64(1), np.uint64(10)
    t = np.array([0, 9, 0, 3, 0, 0, 0, 7, 0, 1], dtype=np.uint64)[(p % ten).astype(np.int64)]
    inv = (p * t + one) // ten
    am1 = (_powmod(np.full_like(p, 10), a, p) + p - one) % p
    off, slope = am1 * _powmod(inv, c, p) % p, _powmod(np.full_like(p, 10), b - c, p)
    roff = am1 * _powmod(inv, a - c, p) % p  # rev(j) 10^-lj == roff - rev(k) 10^-lk rslope
    rslope = _powmod(inv, b - c, p)
    for k in range(1, K + 1):
        j = (off + p - np.uint64(k) * slope % p) % p
        j = j[(j >= 1) & (j <= K)].astype(np.int64)
        mask[k - 1, j - 1] = True
        y = (roff + p - np.uint64(_rev(k)) * _powmod(inv, len(str(k)), p) % p * rslope % p) % p
        for lj in range(1, len(str(K)) + 1):
            y = y * ten % p
            for v in np.unique(y[(y >= 1) & (y < np.uint64(10) ** np.uint64(lj)) & ((y % ten != 0) | (lj == 1))]):
                j = int(str(int(v)).zfill(lj)[::-1])
                if j <= K and len(str(j)) == lj:
                    mask[k - 1, j - 1] = True
    return mask


def _packed(mask):
    K = mask.shape[0]
    bits = np.packbits(mask.reshape(-1), bitorder="little")
    return np.concatenate([bits, np.zeros(_bytes(K) - len(bits), dtype=np.uint8)])


def _bytes(K):
    """Bytes of a packed K x K mask: whole 32-bit words."""
    return 4 * ((K * K + 31) // 32)


def exact(case, seed):
    kind, rng = case["kind"], random.Random(seed)
    if kind in ("dropin", "sieve", "masks"):
        K, n = (100, 1) if kind == "dropin" else (case["K"], case["n"])
        if n * (_pi(case["limit"]) * K * 1e-7 + K * K * 4 * K * 5e-8) > 15:
            return None
        primes = _primes(case["limit"])
        grids = [_grid(primes, *_triple(rng, case["digits"]), K) for _ in range(n)]
        packed = [_packed(g) for g in grids]
        if kind == "dropin":
            return packed[0].view(np.int32)
        if kind == "masks":
            return np.concatenate(packed)
        lists = np.zeros((n, _room(K)), dtype=np.int32)
        counts = np.zeros(n, dtype=np.int64)
        for t, g in enumerate(grids):
            k, j = np.nonzero(~g)
            lists[t, :len(k)] = ((k + 1) << 16) | (j + 1)
            counts[t] = len(k)
        return [np.stack(packed), lists, counts]
    if kind in ("test", "powm"):
        bits = (case["lo"] + case["hi"]) / 2 * 3.33
        if case["n"] * (bits if kind == "test" else case["ebits"]) * (bits / 30) ** 2 * 2.5e-9 > 15:
            return None
        xs = _candidates(rng, case["n"], case["lo"], case["hi"])
        if kind == "powm":
            return _limbs([pow(2, rng.getrandbits(case["ebits"]) | (1 << (case["ebits"] - 1)), x) for x in xs], case)
        ver, res = [], []
        for x in xs:
            s = ((x - 1) & (1 - x)).bit_length() - 1
            r = y = pow(2, (x - 1) >> s, x)
            ok = y in (1, x - 1)
            for _ in range(s - 1):
                y = y * y % x
                ok = ok or y == x - 1
            ver.append(int(ok))
            res.append(r)
        return {"verdicts": np.array(ver, dtype=np.int32), "residues": _limbs(res, case)}
    if kind == "ctx":
        if case["n"] * case["ops"] * (case["digits"] * 3.33 / 30) ** 2 * 4e-9 > 15:
            return None
        moduli, n16, a, b = _ctx_inputs(case, seed)
        plain = np.zeros((case["n"], n16), dtype=np.int32)
        working = np.zeros((case["n"], n16), dtype=np.int64)
        for i, N in enumerate(moduli):
            bits, H = N.bit_length(), 128
            while 22 * H < bits + 6 or math.gcd((1 << (22 * H)) + 1, N) > 1:
                H *= 2
            ri = pow((1 << (22 * H)) + 1, -1, N)
            x, y = pfb200.limbs16_to_int(a[i]), pfb200.limbs16_to_int(b[i])
            for o in range(case["ops"]):
                x = x * (y if o % 5 == 4 else x) * ri % N
            l = pfb200.int_to_limbs16(x)
            working[i, :len(l)] = l
            l = pfb200.int_to_limbs16(x * ri % N)
            plain[i, :len(l)] = l
        return {"working": working, "plain": plain}
    return None
