"""One-launch products at the edges of their lengths (transforms 2^5 .. 2^16), and the kernels
around them: exact 64-bit products over several primes in one launch, the signed lift, and the
warp-per-coefficient sum of big coefficients.  Bit-exact against the oracle."""
import ctypes

import numpy as np
import pytest

from cumodp_b200.workloads import SplitMix64

pytestmark = pytest.mark.gpu


def _dev(x, off=0):
    import torch
    t = torch.zeros(len(x) + off, dtype=torch.int64 if x.dtype == np.int64 else torch.int32, device="cuda")
    t[off:] = torch.from_numpy(x.view(np.int64 if x.dtype == np.int64 else np.int32)).cuda()
    return t


@pytest.mark.parametrize("p", [469762049, 962592769, 1053818881])
@pytest.mark.parametrize("k", range(5, 17))
def test_lengths_of_every_form(cm, oracle_mod, p, k):
    """The shortest and longest product of each transform length, unbalanced and balanced,
    truncated and zero-extended, and in place."""
    import torch
    n = 1 << k
    r = SplitMix64(p + k)
    for la, lb in [(n // 2 + 1, 1), (n // 4 + 1, n // 4 + 1), (n, 1), (1, n), (n // 2, n // 2 + 1), (n - 6, 7)]:
        a, b = r.residues(la, p), r.residues(lb, p)
        want = oracle_mod.polymul(a, b, p)
        lc = la + lb - 1
        for lh in (lc, lc - lc // 3, lc + 37):
            ta, tb = _dev(a, 1), _dev(b, 3)
            th = torch.full((lh + 2,), -1, dtype=torch.int32, device="cuda")
            cm.fftmul_uni_dev(th.data_ptr() + 4, lh, ta.data_ptr() + 4, la - 1, tb.data_ptr() + 12, lb - 1, p)
            got = th.cpu().numpy()
            assert got[0] == -1 and got[-1] == -1
            full = np.zeros(lh, np.uint32)
            full[:min(lh, lc)] = want[:lh]
            assert np.array_equal(got[1:-1].view(np.uint32), full)
        th = _dev(np.concatenate([a, np.zeros(lb - 1, np.uint32)]))  # H over F
        cm.fftmul_uni_dev(th.data_ptr(), lc, th.data_ptr(), la - 1, tb.data_ptr() + 12, lb - 1, p)
        assert np.array_equal(th.cpu().numpy().view(np.uint32), want)


@pytest.mark.parametrize("k", [5, 9, 11, 12, 14, 16, 17])
def test_words_past_p_and_full_length_cyclic(cm, oracle_mod, k):
    """Operands of n words (the cyclic convolution) and any 32-bit word as input."""
    import torch
    p, n = 754974721, 1 << k
    r = SplitMix64(k)
    a = (r.next_u64(n) & np.uint64(0xFFFFFFFF)).astype(np.uint32)
    b = r.residues(n, p)
    w = oracle_mod.polymul(a % np.uint32(p), b, p).astype(np.uint64)
    want = w[:n].copy()
    want[:n - 1] += w[n:]
    ta, tb = _dev(a), _dev(b)
    rc = cm.lib().cumodp_cyclic_mul_dev(k, ctypes.c_void_p(ta.data_ptr()), ctypes.c_void_p(tb.data_ptr()), p, None)
    assert rc == 0
    assert np.array_equal(ta.cpu().numpy().view(np.uint32), (want % p).astype(np.uint32))
    assert torch.equal(tb, _dev(b))


@pytest.mark.parametrize("bits", [2, 30, 34, 40])
@pytest.mark.parametrize("n,m", [(1, 1), (20, 13), (32768, 32769), (32769, 32769)])
def test_exact_products_around_the_one_launch_limit(cm, oracle_mod, bits, n, m):
    """int64 products on both sides of 2^16 points, extreme values included; the result pointer 8
    bytes off a 16-byte boundary."""
    import torch
    r = SplitMix64(bits + n)
    bound = (1 << bits) - 1
    a, b = r.int64_in(n, bound), r.int64_in(m, bound)
    a[0], b[-1], a[n // 2] = bound, -bound, -bound
    if n > 100:  # long runs of the extreme value: the lift's largest magnitudes
        a[:n // 2], b[:n // 2] = -bound, bound
    want = oracle_mod.polymul_i128(a, b)
    ta, tb = _dev(a, 1), _dev(b)
    tc = torch.zeros(2 * (n + m - 1) + 1, dtype=torch.int64, device="cuda")
    rc = cm.lib().cumodp_twoconv_mul_i64_dev(n, ta.data_ptr() + 8, m, tb.data_ptr(), tc.data_ptr() + 8, bits, 0, None)
    assert rc == 0
    assert cm.int128_words_to_ints(tc[1:].cpu().numpy()) == want


@pytest.mark.parametrize("bits,na,nb,words,out_words", [
    (170, 40, 33, 3, 7), (170, 40, 33, 3, 2), (600, 5, 3, 12, 200), (4095, 3, 5, 64, 160), (4096, 2, 2, 65, 136),
    (181, 3000, 2900, 3, 6), (36, 700, 800, 1, 2), (100, 900, 1000, 2, 4)])
def test_big_sums(cm, oracle_mod, bits, na, nb, words, out_words):
    """Carries and signs through every word: all-ones and zero-word coefficients beside random ones, the
    output narrower and far wider than the product."""
    if words > 64:
        words = 64  # 4096-bit magnitudes do not fit 64 signed words: the most negative one does
    r = SplitMix64(bits + na)
    top = (1 << min(bits, 64 * words - 1)) - 1

    def coefficients(n):
        raw = r.next_u64(n * 64).reshape(n, 64)
        out = []
        for i, row in enumerate(raw):
            v = 0
            for w in row:
                v = (v << 64) | int(w)
            v &= top
            out.append([v, -v, top, -top, -(1 << 64) if bits > 64 else -1, 0][int(row[0]) % 6])
        return out
    a, b = coefficients(na), coefficients(nb)
    want = oracle_mod.bigint_polymul(a, b)
    got = cm.twoconv_mul_big(a, b, in_words=words, out_words=out_words)
    half = 1 << (64 * out_words - 1)
    assert got == [((v + half) % (2 * half)) - half for v in want]
