"""Performance cases of the library's public entry points.

Every case is a call a program makes through ``cumodp_b200``: products mod a
Fourier prime on device and host arrays, natural-order transforms (single and
list, both directions), batches of uneven degree, the bivariate product, a
subproduct-tree level and the exact integer products.  Device entry points get
a caller stream, as a program that pipelines its calls passes one; transforms
and the bivariate product work in place, so their pass starts with the copy a
program makes when it keeps its coefficients.  All results are whole numbers:
every correct implementation gives the same ones.
"""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

import cumodp_b200 as cm

P = 469762049  # 7 * 2^26 + 1, the prime of the benchmark configurations
# Fourier primes of the configurations and tests, with their 2-adic orders
PRIMES = {469762049: 26, 754974721: 24, 962592769: 21, 998244353: 23}

_STREAM = None


def _stream():
    """The one stream this program issues its device work on."""
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


def listed():
    return [
        # the smallest call: one short product on device arrays (a leaf of a recursive algorithm); latency
        {"name": "product_255", "kind": "product", "la": 256, "lb": 256, "p": P},
        # the single-product configuration: two degree-4095 polynomials, transform 2^13; latency
        {"name": "product_4095", "kind": "product", "la": 4096, "lb": 4096, "p": P},
        # an ordinary product of unequal, odd lengths (transform 2^16) mod another prime
        {"name": "product_30011x18008", "kind": "product", "la": 30011, "lb": 18008, "p": 962592769},
        # the headline configuration: two degree-(2^23 - 1) polynomials, transform 2^24
        {"name": "product_2^24", "kind": "product", "la": 1 << 23, "lb": 1 << 23, "p": P},
        # the drop-in call of a C program: host arrays in and out, ragged lengths
        {"name": "host_product_20011x13001", "kind": "host_product", "la": 20011, "lb": 13001, "p": P},
        # the batched configuration: 4096 pairs, degrees log-uniform in [32, 65536], one call
        {"name": "batch_4096", "kind": "batch", "count": 4096, "lo": 32, "hi": 65536, "shape": 3, "p": P},
        # the large single transform configuration
        {"name": "fft_2^24", "kind": "fft", "k": 24, "p": P, "inverse": False},
        # a list of middle-sized transforms, the inverse direction, an odd number of rows
        {"name": "list_ifft_3001x2^12", "kind": "list", "m": 3001, "k": 12, "p": 754974721, "inverse": True},
        # bivariate product, operands zero-padded to a 2^12 x 2^12 grid
        {"name": "bivariate_2^12x2^12", "kind": "bivariate", "em": 12, "en": 12, "p": P},
        # one level of a subproduct tree over 2^20 points: 2^11 products of monic degree-512 polynomials
        {"name": "subproduct_512x2048", "kind": "subproduct", "l": 512, "pairs": 2048, "p": P},
        # exact product of signed int64 polynomials, the configuration's degree 8191 and |c| <= 10^10
        {"name": "exact_8191", "kind": "exact", "la": 8192, "lb": 8192, "bound": 10 ** 10},
        # exact product of big signed coefficients: 1024 terms of 1024 bits
        {"name": "big_1024x1024", "kind": "big", "n": 1024, "words": 16},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    """One more case of the listed kinds; sizes log-uniform over each kind's range, odd ones among them."""
    kind = rng.choice(["product", "product", "product", "host_product", "batch", "fft", "list", "list", "bivariate",
                       "subproduct", "exact", "big"])
    p = rng.choice(sorted(PRIMES))
    order = PRIMES[p]
    if kind == "product":
        # degrees drawn independently; the sum stays within the prime's transform and 2^24
        top = 1 << (min(order, 24) - 1)
        return {"kind": kind, "la": _log_uniform(rng, 17, top), "lb": _log_uniform(rng, 17, top), "p": p}
    if kind == "host_product":
        return {"kind": kind, "la": _log_uniform(rng, 100, 1 << 18), "lb": _log_uniform(rng, 100, 1 << 18), "p": p}
    if kind == "batch":
        count = _log_uniform(rng, 16, 4096)
        hi = 65536 if count >= 1024 else _log_uniform(rng, 512, 65536)
        return {"kind": kind, "count": count, "lo": 32, "hi": hi, "shape": rng.randrange(1 << 20), "p": p}
    if kind == "fft":
        return {"kind": kind, "k": rng.randint(6, min(order, 24)), "p": p, "inverse": rng.random() < 0.5}
    if kind == "list":
        k = rng.randint(6, 16)
        return {"kind": kind, "m": _log_uniform(rng, 3, (1 << 24) >> k), "k": k, "p": p, "inverse": rng.random() < 0.5}
    if kind == "bivariate":
        em = rng.randint(5, 12)
        return {"kind": kind, "em": em, "en": rng.randint(6, min(14, 23 - em)), "p": p}
    if kind == "subproduct":
        l = _log_uniform(rng, 16, 16384)
        return {"kind": kind, "l": l, "pairs": _log_uniform(rng, 2, max(2, (1 << 20) // l)), "p": p}
    if kind == "exact":
        return {"kind": kind, "la": _log_uniform(rng, 64, 1 << 18), "lb": _log_uniform(rng, 64, 1 << 18),
                "bound": rng.choice([10 ** 6, 10 ** 10, 10 ** 12])}
    return {"kind": kind, "n": _log_uniform(rng, 32, 1024), "words": rng.randint(1, 16)}


# ------------------------------------------------------------------ inputs ----
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed & 0x7FFFFFFF)
    return g


def _residues(g, n, p):
    return torch.randint(0, p, (n,), generator=g, device="cuda", dtype=torch.int32)


def _root(k, p):
    a = 2
    while pow(a, (p - 1) // 2, p) == 1:
        a += 1
    return pow(a, (p - 1) >> k, p)


def _batch_shape(case):
    r = np.random.RandomState(case["shape"])

    def degrees():
        return np.floor(np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]), case["count"]))).astype(np.int32)
    df, dg = degrees(), degrees()

    def offsets(lens):
        off = np.zeros(len(lens), np.int64)
        off[1:] = np.cumsum(lens.astype(np.int64))[:-1]
        return off
    return df, dg, offsets(df + 1), offsets(dg + 1), offsets(df + dg + 1)


def prepare(case, seed):
    g, kind, p = _gen(seed), case["kind"], case.get("p")
    s = {"case": case, "p": p}
    if kind in ("product", "host_product"):
        la, lb = case["la"], case["lb"]
        f, h = _residues(g, la, p), _residues(g, lb, p)
        if kind == "host_product":
            s.update(f=f.cpu().numpy(), g=h.cpu().numpy())
        else:
            s.update(f=f, g=h, h=torch.empty(la + lb - 1, dtype=torch.int32, device="cuda"))
    elif kind == "batch":
        df, dg, fo, go, ho = _batch_shape(case)
        nf, ng = int((df + 1).sum()), int((dg + 1).sum())
        s.update(df=df, dg=dg, fo=fo, go=go, ho=ho, f=_residues(g, nf, p), g=_residues(g, ng, p),
                 h=torch.empty(nf + ng - len(df), dtype=torch.int32, device="cuda"))
    elif kind in ("fft", "list"):
        n = case.get("m", 1) << case["k"]
        s.update(x=_residues(g, n, p), y=torch.empty(n, dtype=torch.int32, device="cuda"), w=_root(case["k"], p))
    elif kind == "bivariate":
        m, n = 1 << case["em"], 1 << case["en"]
        for name in ("f", "g"):
            grid = torch.zeros((m, n), dtype=torch.int32, device="cuda")
            grid[:m // 2, :n // 2] = _residues(g, (m // 2) * (n // 2), p).view(m // 2, n // 2)
            s[name] = grid
        s.update(tf=torch.empty_like(s["f"]), tg=torch.empty_like(s["g"]))
    elif kind == "subproduct":
        n = 2 * case["pairs"] * case["l"]
        s.update(x=_residues(g, n, p), y=torch.empty(n, dtype=torch.int32, device="cuda"))
    elif kind == "exact":
        b = case["bound"]
        for name in ("la", "lb"):
            s[name] = torch.randint(-b, b + 1, (case[name],), generator=g, device="cuda", dtype=torch.int64)
        s.update(c=torch.empty(2 * (case["la"] + case["lb"] - 1), dtype=torch.int64, device="cuda"),
                 bits=int(b).bit_length())
    else:
        n, words = case["n"], case["words"]
        for name in ("a", "b"):
            v = torch.randint(-(1 << 63), (1 << 63) - 1, (n, words + 1), generator=g, device="cuda", dtype=torch.int64)
            v[:, words] >>= 63  # the sign word
            s[name] = v
        bits = 64 * words
        s.update(bits=bits, out_words=int(cm.lib().cumodp_twoconv_big_out_words(n, n, bits)))
        s["c"] = torch.empty((2 * n - 1) * s["out_words"], dtype=torch.int64, device="cuda")
    return s


# -------------------------------------------------------------------- runs ----
def run(s):
    case, p, kind = s["case"], s["p"], s["case"]["kind"]
    if kind == "host_product":
        return cm.fftmul_uni(s["f"], s["g"], p).view(np.int32)
    st = _stream()
    sp = st.cuda_stream
    if kind == "product":
        cm.fftmul_uni_dev(s["h"].data_ptr(), case["la"] + case["lb"] - 1, s["f"].data_ptr(), case["la"] - 1,
                          s["g"].data_ptr(), case["lb"] - 1, p, sp)
        return s["h"]
    if kind == "batch":
        cm.fftmul_batch_dev(s["df"], s["fo"], s["f"].data_ptr(), s["dg"], s["go"], s["g"].data_ptr(), s["ho"],
                            s["h"].data_ptr(), p, sp)
        return s["h"]
    if kind in ("fft", "list"):
        with torch.cuda.stream(st):
            s["y"].copy_(s["x"])
        if kind == "fft":
            cm.fft_uni_dev(s["y"].data_ptr(), case["k"], s["w"], p, case["inverse"], sp)
        else:
            cm.list_fft_dev(s["y"].data_ptr(), case["m"], case["k"], s["w"], p, case["inverse"], sp)
        return s["y"]
    if kind == "bivariate":
        with torch.cuda.stream(st):
            s["tf"].copy_(s["f"])
            s["tg"].copy_(s["g"])
        cm.bivariate_mul_dev(case["em"], case["en"], s["tf"].data_ptr(), s["tg"].data_ptr(), p, sp)
        return s["tf"]
    if kind == "subproduct":
        cm.subproduct_level_dev(case["l"], case["pairs"], s["x"].data_ptr(), s["y"].data_ptr(), p, sp)
        return s["y"]
    if kind == "exact":
        rc = cm.lib().cumodp_twoconv_mul_i64_dev(case["la"], s["la"].data_ptr(), case["lb"], s["lb"].data_ptr(),
                                                 s["c"].data_ptr(), s["bits"], 0, ctypes.c_void_p(sp))
    else:
        rc = cm.lib().cumodp_twoconv_mul_big_dev(case["n"], s["a"].data_ptr(), case["n"], s["b"].data_ptr(),
                                                 case["words"] + 1, s["c"].data_ptr(), s["out_words"], s["bits"],
                                                 ctypes.c_void_p(sp))
    if rc:
        raise cm.CumodpError(rc, kind)
    return s["c"]


# -------------------------------------------------------------------- work ----
def _transform(n):
    """Modular products of one radix-2 transform, each counted as two operations."""
    lg = max(1, math.ceil(math.log2(max(2, n))))
    return lg * (1 << lg)


def work(case):
    kind = case["kind"]
    if kind in ("product", "host_product"):
        lc = case["la"] + case["lb"] - 1
        return {"bytes": 4 * (case["la"] + case["lb"] + lc), "flops": 3 * _transform(lc)}
    if kind == "batch":
        df, dg = (d.astype(np.int64) for d in _batch_shape(case)[:2])
        return {"bytes": int(4 * (2 * df + 2 * dg + 3).sum()),
                "flops": sum(3 * _transform(int(n)) for n in df + dg + 1)}
    if kind in ("fft", "list"):
        m, n = case.get("m", 1), 1 << case["k"]
        return {"bytes": 8 * m * n, "flops": m * _transform(n)}
    if kind == "bivariate":
        m, n = 1 << case["em"], 1 << case["en"]
        return {"bytes": 12 * m * n, "flops": 3 * (m * _transform(n) + n * _transform(m))}
    if kind == "subproduct":
        return {"bytes": 16 * case["pairs"] * case["l"], "flops": 3 * case["pairs"] * _transform(2 * case["l"])}
    if kind == "exact":
        lc = case["la"] + case["lb"] - 1
        return {"bytes": 8 * (case["la"] + case["lb"]) + 16 * lc, "flops": 9 * _transform(lc)}
    n, words = case["n"], case["words"]
    # a product of two integers of n slots, cut into 36-bit limbs, over three primes
    limbs = n * 2 * math.ceil(64 * words / 36)
    return {"bytes": 8 * (2 * n * (words + 1) + (2 * n - 1) * (2 * words + 1)), "flops": 9 * _transform(2 * limbs)}


def tolerance(case):
    return "exact"  # residues, and exact integers


# ------------------------------------------------------------------- exact ----
def _powers(w, n, p):
    t = torch.ones(1, dtype=torch.int64, device="cuda")
    while t.numel() < n:
        t = torch.cat([t, t * pow(w, t.numel(), p) % p])
    return t[:n]


def _ntt(x, w, p):
    """Natural-order DFT with root w along the last axis (Stockham, radix 2, 64-bit integers)."""
    shape, n = x.shape, x.shape[-1]
    y = x.reshape(-1, n).to(torch.int64) % p
    l, m = n // 2, 1
    while l >= 1:
        y = y.view(-1, 2, l, m)
        u, v = y[:, 0], y[:, 1]
        t = _powers(w, l, p).view(1, l, 1)
        y = torch.stack([(u + v) % p, (u - v) % p * t % p], dim=2)
        l, m, w = l // 2, 2 * m, w * w % p
    return y.reshape(shape)


def _intt(x, w, p):
    return _ntt(x, pow(w, p - 2, p), p) * pow(x.shape[-1], p - 2, p) % p


def _padded(x, n, p):
    y = torch.zeros(x.shape[:-1] + (n,), dtype=torch.int64, device="cuda")
    y[..., :x.shape[-1]] = x.to(torch.int64) % p
    return y


def _product(a, b, p):
    """a * b mod p along the last axis."""
    lc = a.shape[-1] + b.shape[-1] - 1
    k = max(1, (lc - 1).bit_length())
    w, n = _root(k, p), 1 << k
    return _intt(_ntt(_padded(a, n, p), w, p) * _ntt(_padded(b, n, p), w, p) % p, w, p)[..., :lc]


def _i32(x):
    return x.to(torch.int32)


def _exact_i64(a, b):
    """The signed 128-bit coefficients (lo, hi words) of the product: three primes, Garner's lift."""
    p0, p1, p2 = 469762049, 998244353, 754974721
    r = [_product(a, b, q).cpu().numpy().astype(object) for q in (p0, p1, p2)]
    v1 = (r[1] - r[0]) * pow(p0, p1 - 2, p1) % p1
    x = r[0] + v1 * p0
    v2 = (r[2] - x) * pow(p0 * p1, p2 - 2, p2) % p2
    x = x + v2 * (p0 * p1)
    full = p0 * p1 * p2
    x = np.where(x > full // 2, x - full, x) % (1 << 128)
    words = np.empty((len(x), 2), dtype=np.uint64)
    words[:, 0], words[:, 1] = x % (1 << 64), x >> 64
    return torch.from_numpy(words.view(np.int64).reshape(-1))


def _exact_big(a, b, out_words):
    """Big signed coefficients by one product of two Python integers (Kronecker substitution)."""
    def ints(v):
        m, w = v.shape
        raw = v.cpu().numpy().tobytes()
        return [int.from_bytes(raw[8 * w * i:8 * w * (i + 1)], "little", signed=True) for i in range(m)]

    fa, fb = ints(a), ints(b)
    slot = 8 * (2 * a.shape[1] + 2)  # bytes a coefficient takes, sign included
    bias = 1 << (8 * slot - 1)

    def packed(f):  # sum of f_i 2^(8 slot i): the biased digits minus the bias in each
        digits = b"".join((c + bias).to_bytes(slot, "little") for c in f)
        return int.from_bytes(digits, "little") - bias * (((1 << (8 * slot * len(f))) - 1) // ((1 << (8 * slot)) - 1))

    n = len(fa) + len(fb) - 1
    c = packed(fa) * packed(fb) + bias * (((1 << (8 * slot * n)) - 1) // ((1 << (8 * slot)) - 1))
    raw = c.to_bytes(slot * n, "little")
    top = 1 << (64 * out_words)
    out = b"".join(((int.from_bytes(raw[slot * i:slot * (i + 1)], "little") - bias) % top).to_bytes(8 * out_words,
                                                                                                  "little")
                   for i in range(n))
    return torch.from_numpy(np.frombuffer(out, dtype=np.int64).copy())


def exact(case, seed):
    s, kind, p = prepare(case, seed), case["kind"], case.get("p")
    if kind == "product":
        return _i32(_product(s["f"], s["g"], p))
    if kind == "host_product":
        f, g = (torch.from_numpy(s[k]).cuda() for k in "fg")
        return _i32(_product(f, g, p)).cpu().numpy()
    if kind == "batch":
        h = torch.empty_like(s["h"])
        lens = (s["df"].astype(np.int64) + s["dg"] + 1)
        for lg in range(1, 18):  # one padded transform per size, over all of its products
            of = [i for i in range(len(lens)) if max(1, (int(lens[i]) - 1).bit_length()) == lg]
            for at in range(0, len(of), 64):
                some = of[at:at + 64]
                n = 1 << lg
                fa = torch.zeros((len(some), n), dtype=torch.int64, device="cuda")
                ga = torch.zeros_like(fa)
                for j, i in enumerate(some):
                    la, lb = int(s["df"][i]) + 1, int(s["dg"][i]) + 1
                    fa[j, :la] = s["f"][int(s["fo"][i]):int(s["fo"][i]) + la]
                    ga[j, :lb] = s["g"][int(s["go"][i]):int(s["go"][i]) + lb]
                w = _root(lg, p)
                c = _intt(_ntt(fa, w, p) * _ntt(ga, w, p) % p, w, p)
                for j, i in enumerate(some):
                    h[int(s["ho"][i]):int(s["ho"][i]) + int(lens[i])] = _i32(c[j, :int(lens[i])])
        return h
    if kind in ("fft", "list"):
        x = s["x"].view(-1, 1 << case["k"])
        return _i32((_intt if case["inverse"] else _ntt)(x, s["w"], p)).reshape(-1)
    if kind == "bivariate":
        wm, wn = _root(case["em"], p), _root(case["en"], p)

        def both(x, f):
            return f(f(x, wn, p).T.contiguous(), wm, p).T.contiguous()
        return _i32(both(both(s["f"], _ntt) * both(s["g"], _ntt) % p, _intt))
    if kind == "subproduct":
        l, pairs = case["l"], case["pairs"]
        x = s["x"].view(pairs, 2, l)
        one = torch.ones((pairs, 1), dtype=torch.int32, device="cuda")
        a, b = (torch.cat([x[:, i], one], dim=1) for i in (0, 1))
        return _i32(_product(a, b, p)[:, :2 * l]).reshape(-1)
    if kind == "exact":
        return _exact_i64(s["la"], s["lb"])
    return _exact_big(s["a"], s["b"], s["out_words"])
