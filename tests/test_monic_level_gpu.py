"""Subproduct-tree levels in one launch, at the edges of their transform lengths, with more pairs than
CTAs and words past p."""
import numpy as np
import pytest

from cumodp_b200.workloads import SplitMix64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [469762049, 1053818881])
@pytest.mark.parametrize("l,npairs", [(1, 5000), (15, 40), (16, 20000), (17, 3), (31, 7), (32, 900), (33, 5), (64, 64),
                                      (255, 3), (256, 1), (257, 9), (512, 2500), (1023, 2), (1024, 700), (1025, 3),
                                      (2047, 5), (2048, 301), (2049, 3)])
def test_levels_in_one_launch(cm, oracle_mod, p, l, npairs):
    import torch
    r = SplitMix64(l * 7 + npairs)
    x = (r.next_u64(2 * npairs * l) & np.uint64(0xFFFFFFFF)).astype(np.uint32)
    x[:2 * l] = p - 1
    d = torch.from_numpy(x.view(np.int32)).cuda()
    out = torch.full((2 * npairs * l + 1,), -1, dtype=torch.int32, device="cuda")
    cm.subproduct_level_dev(l, npairs, d.data_ptr(), out.data_ptr(), p)
    got = out.cpu().numpy()
    assert got[-1] == -1
    idx = sorted({0, npairs // 2, npairs - 1})
    M = np.concatenate([x[2 * j * l:2 * (j + 1) * l] for j in idx]) % np.uint32(p)
    want = oracle_mod.subproduct_level(M, l, p)
    assert np.array_equal(np.concatenate([got[2 * j * l:2 * (j + 1) * l] for j in idx]).view(np.uint32), want)
