"""Natural-order row transforms at every row length of the list kernel: one row, a partly filled CTA, odd
row counts, both directions, words past p, off the buffer's start, and as the rows of 2-D transforms."""
import numpy as np
import pytest

from cumodp_b200.workloads import SplitMix64

pytestmark = pytest.mark.gpu


def _root(k, p):
    a = 2
    while pow(a, (p - 1) // 2, p) == 1:
        a += 1
    return pow(a, (p - 1) >> k, p)


@pytest.mark.parametrize("p", [65537, 469762049, 1053818881])
@pytest.mark.parametrize("k", range(6, 15))
def test_rows(cm, oracle_mod, p, k):
    import torch
    n, w = 1 << k, _root(k, p)
    r = SplitMix64(p + k)
    for m in (1, 2, 17, 301):
        x = (r.next_u64(m * n) & np.uint64(0xFFFFFFFF)).astype(np.uint32)
        x[:n] = 0xFFFFFFFF
        d = torch.full((m * n + 8,), -1, dtype=torch.int32, device="cuda")
        d[4:-4] = torch.from_numpy(x.view(np.int32)).cuda()
        cm.list_fft_dev(d.data_ptr() + 16, m, k, w, p, False)
        got = d.cpu().numpy()
        assert (got[:4] == -1).all() and (got[-4:] == -1).all()
        y = got[4:-4].view(np.uint32).reshape(m, n)
        for i in sorted({0, m // 2, m - 1}):
            assert np.array_equal(y[i], oracle_mod.ntt(x[i * n:(i + 1) * n] % np.uint32(p), w, p))
        cm.list_fft_dev(d.data_ptr() + 16, m, k, w, p, True)
        assert np.array_equal(d[4:-4].cpu().numpy().view(np.uint32), x % np.uint32(p))


@pytest.mark.parametrize("em,en", [(0, 6), (1, 6), (5, 7), (4, 13), (11, 6)])
def test_rows_of_2d_transforms(cm, oracle_mod, em, en):
    import torch
    p = 469762049
    m, n, wm, wn = 1 << em, 1 << en, _root(em, p) if em else 1, _root(en, p)
    x = SplitMix64(em * 16 + en).residues(m * n, p)
    d = torch.from_numpy(x.view(np.int32)).cuda()
    cm.fft_bivariate_dev(d.data_ptr(), em, wm, en, wn, p)
    got = d.cpu().numpy().view(np.uint32).reshape(m, n)
    rows = np.stack([oracle_mod.ntt(v, wn, p) for v in x.reshape(m, n)])
    for c in (0, 1, n // 2, n - 1):
        want = oracle_mod.ntt(np.ascontiguousarray(rows[:, c]), wm, p) if em else rows[:, c]
        assert np.array_equal(got[:, c], want)
    cm.fft_bivariate_dev(d.data_ptr(), em, wm, en, wn, p, True)
    assert np.array_equal(d.cpu().numpy().view(np.uint32), x)
