"""The decode attention over short contexts (one CTA of eight warps walks them) and one key tile beyond, against plain attention in float64:
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
    """P and the result are rounded to bfloat16: 2^-8 of the values' norm, as the other tests of this kernel."""
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
