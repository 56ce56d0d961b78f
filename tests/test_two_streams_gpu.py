"""Calls on two streams share the library's scratch and job tables: interleaved without any synchronisation by the
caller, each must give what it gives alone."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

P = 469762049


def _root(k):
    return pow(3, (P - 1) >> k, P)


def _words(g, n, p=P):
    return torch.randint(0, p, (n,), generator=g, device="cuda", dtype=torch.int32)


def _make(cm, kind, seed):
    """(run(stream), result tensor): each pass computes the result from inputs it does not change."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    if kind == "product":
        n = (1 << 19) + 77 * seed
        a, b, h = _words(g, n), _words(g, n), torch.empty(2 * n - 1, dtype=torch.int32, device="cuda")
        return lambda s: cm.fftmul_uni_dev(h.data_ptr(), 2 * n - 1, a.data_ptr(), n - 1, b.data_ptr(), n - 1, P, s), h
    if kind in ("fft", "list"):
        k, m = (20, 1) if kind == "fft" else (16, 20)
        x, y = _words(g, m << k), torch.empty(m << k, dtype=torch.int32, device="cuda")

        def run(s):
            with torch.cuda.stream(torch.cuda.ExternalStream(s)):
                y.copy_(x)
            if kind == "fft":
                cm.fft_uni_dev(y.data_ptr(), k, _root(k), P, False, s)
            else:
                cm.list_fft_dev(y.data_ptr(), m, k, _root(k), P, True, s)
        return run, y
    if kind == "bivariate":
        f, h = _words(g, 1 << 20), _words(g, 1 << 20)
        y, z = torch.empty_like(f), torch.empty_like(h)

        def run(s):
            with torch.cuda.stream(torch.cuda.ExternalStream(s)):
                y.copy_(f)
                z.copy_(h)
            cm.bivariate_mul_dev(10, 10, y.data_ptr(), z.data_ptr(), P, s)
        return run, y
    if kind in ("exact", "exact_long"):
        n = 30000 if kind == "exact" else 150000
        a, b = (torch.randint(-10 ** 9, 10 ** 9, (n,), generator=g, device="cuda") for _ in range(2))
        c = torch.empty(4 * n - 2, dtype=torch.int64, device="cuda")

        def run(s):
            assert cm.lib().cumodp_twoconv_mul_i64_dev(n, a.data_ptr(), n, b.data_ptr(), c.data_ptr(), 30, 0,
                                                       ctypes.c_void_p(s)) == 0
        return run, c
    if kind == "big":
        n, words = 500, 8
        a, b = (torch.randint(-2 ** 62, 2 ** 62, (n, words), generator=g, device="cuda") for _ in range(2))
        ow = cm.lib().cumodp_twoconv_big_out_words(n, n, 64 * words)
        c = torch.empty((2 * n - 1) * ow, dtype=torch.int64, device="cuda")

        def run(s):
            assert cm.lib().cumodp_twoconv_mul_big_dev(n, a.data_ptr(), n, b.data_ptr(), words, c.data_ptr(), ow,
                                                       64 * words, ctypes.c_void_p(s)) == 0
        return run, c
    # batch: one shape, so one cached plan and job table for both streams' operands
    lens = np.array([70000, 3000, 150000, 500, 9000], np.int32)
    off = np.concatenate([[0], np.cumsum(lens.astype(np.int64))[:-1]])
    a, b = _words(g, int(lens.sum())), _words(g, int(lens.sum()))
    h = torch.empty(2 * int(lens.sum()), dtype=torch.int32, device="cuda")
    h.zero_()
    return lambda s: cm.fftmul_batch_dev(lens - 1, off, a.data_ptr(), lens - 1, off, b.data_ptr(), 2 * off,
                                         h.data_ptr(), P, s), h


@pytest.mark.parametrize("kinds", [(k, k) for k in ("product", "fft", "list", "bivariate", "exact", "exact_long", "big",
                                                    "batch")] + [("fft", "bivariate"), ("exact", "big"), ("list", "fft")])
def test_interleaved_calls_on_two_streams(cm, kinds):
    streams = [torch.cuda.Stream() for _ in kinds]
    jobs = [_make(cm, k, i + 1) for i, k in enumerate(kinds)]
    want = []
    torch.cuda.synchronize()
    for (run, out), s in zip(jobs, streams):
        run(s.cuda_stream)
        torch.cuda.synchronize()
        want.append(out.clone())
        out.fill_(-1) if kinds[0] != "batch" else out.zero_()
    torch.cuda.synchronize()
    for _ in range(20):
        for (run, _), s in zip(jobs, streams):
            run(s.cuda_stream)
    torch.cuda.synchronize()
    for (_, out), w in zip(jobs, want):
        assert torch.equal(out, w)


@pytest.mark.parametrize("kind", ["product", "fft", "bivariate", "exact"])
def test_captured_calls_replay(cm, kind):
    """After a first call the others can be captured into a graph, scratch and all; replays give the same result."""
    s = torch.cuda.Stream()
    run, out = _make(cm, kind, 3)
    run(s.cuda_stream)
    torch.cuda.synchronize()
    want = out.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        run(s.cuda_stream)
        run(s.cuda_stream)
    out.fill_(-1)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
