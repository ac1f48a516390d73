"""The decode attention over short contexts (one CTA of eight or sixteen warps walks them) and one key tile beyond, against plain attention in float64:
contexts at the edges of key tiles, rounds and of the form itself, whatever number of splits was asked for, windows, fresh keys, and tokens
without a list of their sequences (token i is sequence i's)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [1, 2])
@pytest.mark.parametrize("width", [512, 576])                   # tokens a row of the block table stands for: 8 key tiles, and 9
@pytest.mark.parametrize("heads", [(14, 2, 64), (12, 2, 128), (4, 4, 32), (16, 1, 64)])
@pytest.mark.parametrize("window", [0, 100])
def test_short_contexts(heads, width, splits, window):
    """P and the result are rounded to bfloat16, each by up to 2^-8 of a value: 2^-7 of the norm, as the other tests of this kernel."""
    import torch

    from easy_gpt.cpp_b200 import kernels

    NH, G, HD = heads
    contexts = [1, 16, 63, 64, 65, 128, 255, 256, 257, 449, 511, 512]
    T, page, rng = len(contexts), 16, np.random.default_rng([NH, HD, width])
    pages = width // page
    bf = lambda *s: torch.from_numpy(rng.standard_normal(s).astype(np.float32)).bfloat16().cuda()  # noqa: E731
    cache = bf(T * pages + 1, 2, G, page, HD)
    table = torch.from_numpy(rng.permutation(T * pages).reshape(T, pages).astype(np.int32)).cuda()
    q, out = bf(T, NH * HD), torch.full((T, NH * HD), float("nan"), device="cuda", dtype=torch.bfloat16)
    positions = torch.tensor([c - 1 for c in contexts], dtype=torch.int32, device="cuda")
    fresh = torch.tensor([c - 1 for c in contexts], dtype=torch.int32, device="cuda")
    acc, ml = torch.empty(T * NH * splits * HD, device="cuda"), torch.empty(T * NH * splits * 2, device="cuda")
    counters, status = torch.zeros(T * G, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    scale = HD ** -0.5
    k, v = cache[:, 0], cache[:, 1]
    rc = kernels.library().eg_attention_paged(torch.cuda.current_stream().cuda_stream, q.data_ptr(), NH * HD, k.data_ptr(), v.data_ptr(), table.data_ptr(), pages, None,
                                              positions.data_ptr(), fresh.data_ptr(), out.data_ptr(), NH * HD, acc.data_ptr(), ml.data_ptr(), T, NH, G, HD, page,
                                              k.stride(0), k.stride(1), cache.shape[0], window, scale, splits, status.data_ptr(), None, 0, counters.data_ptr(), 2, None, None)
    torch.cuda.synchronize()
    assert rc == 0 and int(status[0]) == 0 and int(counters.abs().sum()) == 0
    for t, c in enumerate(contexts):
        rows = cache[table[t].long()].double()                   # [pages, 2, G, page, HD]
        kk, vv = (rows[:, i].permute(1, 0, 2, 3).reshape(G, -1, HD)[:, :c] for i in (0, 1))
        first = max(0, c - window) if window else 0
        s = torch.einsum("ghd,gkd->ghk", q[t].double().view(G, NH // G, HD), kk) * scale
        s[..., :first] = -math.inf
        want = torch.einsum("ghk,gkd->ghd", s.softmax(-1), vv).reshape(-1)
        assert float((out[t].double() - want).norm() / want.norm()) < 2.0 ** -7, (t, c)


def launch(q, cache, table, contexts, heads, page=16, window=0, splits=1):
    """eg_attention_paged over `contexts`; cache [pages, 2, G, page, HD], table [T, pages of a row]"""
    import torch

    from easy_gpt.cpp_b200 import kernels

    (NH, G, HD), T = heads, len(contexts)
    out = torch.full((T, NH * HD), float("nan"), device="cuda", dtype=torch.bfloat16)
    positions = torch.tensor([c - 1 for c in contexts], dtype=torch.int32, device="cuda")
    acc, ml = torch.empty(T * NH * splits * HD, device="cuda"), torch.empty(T * NH * splits * 2, device="cuda")
    counters, status = torch.zeros(T * G, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    k, v = cache[:, 0], cache[:, 1]
    rc = kernels.library().eg_attention_paged(torch.cuda.current_stream().cuda_stream, q.data_ptr(), NH * HD, k.data_ptr(), v.data_ptr(), table.data_ptr(), table.shape[1], None,
                                              positions.data_ptr(), positions.data_ptr(), out.data_ptr(), NH * HD, acc.data_ptr(), ml.data_ptr(), T, NH, G, HD, page,
                                              k.stride(0), k.stride(1), cache.shape[0], window, HD ** -0.5, splits, status.data_ptr(), None, 0, counters.data_ptr(), 2, None, None)
    torch.cuda.synchronize()
    assert rc == 0 and int(status[0]) == 0 and int(counters.abs().sum()) == 0
    return out


def plain(q, cache, table, contexts, heads):
    import torch

    (NH, G, HD), out = heads, []
    for t, c in enumerate(contexts):
        rows = cache[table[t].long()].double()                   # [pages, 2, G, page, HD]
        kk, vv = (rows[:, i].permute(1, 0, 2, 3).reshape(G, -1, HD)[:, :c] for i in (0, 1))
        s = torch.einsum("ghd,gkd->ghk", q[t].double().view(G, NH // G, HD), kk) * HD ** -0.5
        out.append(torch.einsum("ghk,gkd->ghd", s.softmax(-1), vv).reshape(-1))
    return torch.stack(out)


@pytest.mark.parametrize("tiles", range(1, 9))
@pytest.mark.parametrize("tokens, heads", [(12, (14, 2, 64)), (37, (2, 2, 64)), (38, (2, 2, 64)), (74, (2, 2, 64)), (75, (2, 2, 64)), (12, (8, 8, 32)), (9, (8, 8, 32)), (7, (12, 2, 128)),
                                           (8, (12, 2, 128)), (38, (12, 2, 128))])
def test_forms_of_short_contexts(tokens, heads, tiles):
    """Every size of the block table that the form covers, on both sides of the numbers of CTAs where it changes (16, 74 and 148 of them)."""
    import torch

    (NH, G, HD), rng = heads, np.random.default_rng([tokens, tiles])
    contexts = [int(c) for c in rng.integers(1, 64 * tiles + 1, tokens)]
    contexts[0], contexts[-1] = 64 * tiles, 64 * tiles - 15
    pages = 4 * tiles
    bf = lambda *s: torch.from_numpy(rng.standard_normal(s).astype(np.float32)).bfloat16().cuda()  # noqa: E731
    cache, q = bf(tokens * pages, 2, G, 16, HD), bf(tokens, NH * HD)
    table = torch.from_numpy(rng.permutation(tokens * pages).reshape(tokens, pages).astype(np.int32)).cuda()
    got, want = launch(q, cache, table, contexts, heads), plain(q, cache, table, contexts, heads)
    assert float(((got.double() - want).norm(dim=1) / want.norm(dim=1)).max()) < 2.0 ** -7


@pytest.mark.parametrize("tokens", [8, 48])
@pytest.mark.parametrize("context", [64, 128, 256])
@pytest.mark.parametrize("heads", [(14, 2, 64), (16, 2, 32)])
def test_the_largest_key_of_sixteen_has_an_exact_weight(heads, context, tokens):
    """One key of every sixteen counts.  Where a warp has sixteen keys its weight is 1, so that nothing is rounded before the result is:
    as many values as a float32 sum moves over a tie differ from the rounded result in 64 bits, where weights rounded to bfloat16 move half."""
    import torch

    if tokens == 48 and heads[2] == 64 and context > 64:
        pytest.skip("four warps walk these, a tile at a time")
    if context == 256 and (tokens == 48 or heads[2] == 32):
        tokens = 8                                               # (sixteen warps: small launches)
    (NH, G, HD), rng = heads, np.random.default_rng([context, tokens])
    pages = context // 16
    f = lambda *s: torch.from_numpy(rng.standard_normal(s).astype(np.float32)).cuda()  # noqa: E731
    direction = f(tokens, G, HD)
    q = direction[:, :, None].expand(tokens, G, NH // G, HD).reshape(tokens, NH * HD).bfloat16()
    unit = direction / direction.square().sum(-1, keepdim=True) * HD ** 0.5
    cache = f(tokens * pages, 2, G, 16, HD)
    score = f(tokens, pages, 16) - 60.0
    score[:, :, 7] = f(tokens, pages)
    cache[:, 0] = (score[:, :, None, :, None] * unit[:, None, :, None, :]).reshape(tokens * pages, G, 16, HD)
    cache = cache.bfloat16()
    table = torch.arange(tokens * pages, dtype=torch.int32, device="cuda").view(tokens, pages)
    contexts = [context] * tokens
    got, want = launch(q, cache, table, contexts, heads), plain(q, cache, table, contexts, heads)
    assert float((got != want.bfloat16()).float().mean()) < 0.02
