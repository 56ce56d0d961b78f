"""Bivariate products on the three-pass kernels: every split of the rows of a grid between the column
and the row passes, at the smallest and largest row lengths of each, against 2-D transforms in exact
64-bit arithmetic."""
import numpy as np
import pytest

from cumodp_b200.workloads import SplitMix64

pytestmark = pytest.mark.gpu


def _cyclic_at(f, g, ys, xs, p):
    """Coefficients (y, x) of the 2-D cyclic convolution, straight from the definition."""
    m, n = f.shape
    out = []
    for y, x in zip(ys, xs):
        h = g[(y - np.arange(m)) % m][:, (x - np.arange(n)) % n]
        out.append(sum(int(v) for v in (f.astype(np.uint64) * h % p).sum(axis=1)) % p)
    return out


@pytest.mark.parametrize("p,em,en", [
    (469762049, 1, 10), (469762049, 5, 6), (754974721, 6, 6), (962592769, 9, 7), (469762049, 9, 14),
    (469762049, 10, 6), (998244353, 10, 14), (469762049, 11, 6), (962592769, 11, 13), (469762049, 11, 14),
    (469762049, 12, 6), (1053818881, 12, 12), (469762049, 12, 13), (469762049, 13, 7), (469762049, 13, 12),
    (469762049, 3, 13)])
def test_cyclic_convolution_of_full_grids(cm, p, em, en):
    import torch
    m, n = 1 << em, 1 << en
    r = SplitMix64(p + 64 * em + en)
    f, g = r.residues(m * n, p).reshape(m, n), r.residues(m * n, p).reshape(m, n)
    F, G = (torch.from_numpy(v.view(np.int32)).cuda() for v in (f, g))
    cm.bivariate_mul_dev(em, en, F.data_ptr(), G.data_ptr(), p)
    got = F.cpu().numpy().view(np.uint32)
    assert got.max() < p
    few = 3 if m * n > 1 << 22 else 12
    ys, xs = r.next_u64(few) % np.uint64(m), r.next_u64(few) % np.uint64(n)
    ys, xs = [0, m - 1] + [int(v) for v in ys], [0, n - 1] + [int(v) for v in xs]
    assert [int(got[y, x]) for y, x in zip(ys, xs)] == _cyclic_at(f, g, ys, xs, p)
    # the sums over each row and column are cyclic convolutions too: every coefficient takes part
    x = torch.from_numpy(got.astype(np.int64)).sum() % p
    assert int(x) == int(f.astype(np.uint64).sum() % p) * int(g.astype(np.uint64).sum() % p) % p
    sign = lambda v: int((v[::2].astype(np.int64).sum() - v[1::2].astype(np.int64).sum()) % p)
    assert sign(got) == sign(f) * sign(g) % p
    assert sign(got.T) == sign(f.T) * sign(g.T) % p


_NO_ROOM = """
import sys, numpy as np, torch
import cumodp_b200 as cm
from cumodp_b200.workloads import SplitMix64
p, em, en = 469762049, int(sys.argv[1]), int(sys.argv[2])
r = SplitMix64(64 * em + en)
def product(em, en, fail):
    f, g = (r.residues(1 << (em + en), p) for _ in range(2))
    out = []
    for n in fail:
        F, G = (torch.from_numpy(v.view(np.int32).copy()).cuda() for v in (f, g))
        cm.inject_alloc_failures(n)
        cm.bivariate_mul_dev(em, en, F.data_ptr(), G.data_ptr(), p)
        cm.inject_alloc_failures(0)
        out.append(F.cpu().numpy())
    return out
product(1, 10, [0])
a, b = product(em, en, [1, 0])  # the first allocation of the larger grid is its workspace
assert np.array_equal(a, b)
print("same")
"""


@pytest.mark.parametrize("em,en", [(5, 8), (12, 6)])
def test_grid_without_room_for_its_workspace(em, en):
    """The workspace of two grids cannot be had: the paths with less workspace give the same product (in a
    process of its own, where no earlier call has left a larger workspace)."""
    import pathlib
    import subprocess
    import sys
    root = pathlib.Path(__file__).resolve().parents[1]
    r = subprocess.run([sys.executable, "-c", _NO_ROOM, str(em), str(en)], cwd=root, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("same"), r.stdout + r.stderr
