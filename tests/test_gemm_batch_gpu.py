"""The decode chain's products for 17 to 64 tokens (csrc/gemm_batch.cu) by themselves, against the same in float64 from the bfloat16
values: numbers of tokens at the edges of both token tiles, K of a stage or few a CTA and of more than the ring, clusters of every size,
and which sizes are taken (host arithmetic)."""
import ctypes

import numpy as np
import pytest

P, L, I, F = ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int, ctypes.c_float
SWIGLU, QKV, RESID = 2, 3, 4


def library():
    from easy_gpt.cpp_b200 import kernels

    lib = kernels.library()
    lib.eg_gemm_batch.argtypes = [P, I, I, P, L, P, I, I, I, P, L, F, P, I, P, L, I, I, I, P, P, P, P, I, L, L, L, P, P, P, P, P, L, P]
    return lib


def test_which_sizes_are_taken():
    takes = library().eg_gemm_batch_takes
    assert takes(RESID, 896, 896, 0) == 56 and takes(RESID, 896, 4864, 0) == 112 and takes(SWIGLU, 9728, 896, 0) == 1 and takes(QKV, 1152, 896, 64) == 1
    for n, k in ((896, 100), (100, 896), (896, 128), (9728 * 4, 896)):      # K and N off the tiles, fewer stages than CTAs, more CTAs than are on the GPU at once
        assert takes(RESID, n, k, 0) == 0
    assert takes(QKV, 1152, 896, 32) == 0 and takes(QKV, 1152, 896, 96) == 0 and takes(1, 896, 896, 0) == 0 and takes(SWIGLU, 64 * 297, 896, 0) == 0
    for n in range(64, 20000, 64):                                          # partial sums of squares are read four at a time
        assert takes(RESID, n, 1024, 0) % 4 == 0


def bf16(rng, *shape):
    import torch

    return torch.from_numpy(rng.standard_normal(shape).astype(np.float32)).bfloat16()


def off(got, want):
    return float((got.double() - want).norm() / want.norm())


def run(epilogue, M, N, K, rng, heads, with_bias, scale=1.0, pad=0, prefetch=0):
    """(what the kernel gave, the same in float64); scale: of the partial sums of squares; pad: what a row of x is longer than K; prefetch: bytes
    that the L2 is asked for"""
    import torch

    lib = library()
    f32 = lambda *s: torch.from_numpy(rng.standard_normal(s).astype(np.float32)).cuda()  # noqa: E731
    W, x = bf16(rng, N, K).cuda(), bf16(rng, M, K + pad).cuda()[:, :K]
    bias = f32(N) if with_bias else None
    soon = torch.empty(max(prefetch, 1), device="cuda", dtype=torch.uint8) if prefetch else None
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    y = x.double() @ W.double().T
    empty = lambda *s, t=torch.bfloat16: torch.full(s, float("nan"), device="cuda", dtype=t)  # noqa: E731
    a = dict(out=None, ldo=0, rot=None, slots=None, k=None, v=None, ps=1, pst=0, hst=0, pool=0, resid=None, gain=None, xn=None, ss=None, ssi=None)
    if epilogue == RESID:
        parts = lib.eg_gemm_batch_takes(RESID, N, K, 0)
        resid, gain = f32(M, N) * 30, f32(N)
        a.update(resid=resid.clone(), gain=gain, xn=empty(M, N), ss=empty(M, parts, t=torch.float32))
    else:
        ss = f32(M, 24).square() * scale
        a["ssi"] = ss
        y *= 1.0 / torch.sqrt(ss.double().sum(1, keepdim=True) / K + 1e-6)
    if with_bias:
        y += bias.double()
    if epilogue == SWIGLU:
        a.update(out=empty(M, N // 2), ldo=N // 2)
    if epilogue == QKV:
        H, G, hd = heads
        rot = f32(M, hd // 2, 2)
        slots = torch.from_numpy(rng.permutation(80)[:M].astype(np.int32))
        slots[M // 2] = -1                                       # a token that is not kept
        cache = torch.full((5, 2, G, 16, hd), 7.0, device="cuda", dtype=torch.bfloat16)
        a.update(out=empty(M, H * hd), ldo=H * hd, rot=rot, slots=slots.cuda(), ps=16, pst=2 * G * 16 * hd, hst=16 * hd, pool=80, k=cache, v=cache[:, 1])
    ptr = lambda t: None if t is None else t.data_ptr()  # noqa: E731
    rc = lib.eg_gemm_batch(torch.cuda.current_stream().cuda_stream, epilogue, 2, ptr(W), K, ptr(bias), M, N, K, ptr(x), K + pad, 1e-6, ptr(a["ssi"]), 24 if a["ssi"] is not None else 0,
                           ptr(a["out"]), a["ldo"], *heads, ptr(a["rot"]), ptr(a["slots"]), ptr(a["k"]), ptr(a["v"]), a["ps"], a["pst"], a["hst"], a["pool"], ptr(a["resid"]),
                           ptr(a["gain"]), ptr(a["xn"]), ptr(a["ss"]), ptr(soon), prefetch, ptr(status))
    torch.cuda.synchronize()
    assert rc == 0 and int(status[0]) == 0
    if epilogue == SWIGLU:
        g, u = y[:, 0::2], y[:, 1::2]
        return [a["out"]], [u * g / (1 + torch.exp(-g))]
    if epilogue == RESID:
        new = resid.double() + y
        return [a["resid"] - resid, a["xn"], a["ss"]], [y, new * gain.double(), a["resid"].double().view(M, parts, -1).square().sum(-1)]
    t = y.view(M, H + 2 * G, hd)
    c, s = (rot[..., i].double()[:, None] for i in (0, 1))
    lo, hi = t[..., :hd // 2], t[..., hd // 2:]
    turned = torch.cat([lo * c - hi * s, lo * s + hi * c], -1)
    want = torch.full((5, 2, G, 16, hd), 7.0, device="cuda", dtype=torch.float64)
    for m in range(M):
        slot = int(slots[m])
        if slot >= 0:
            want[slot // 16, 0, :, slot % 16] = turned[m, H:H + G]
            want[slot // 16, 1, :, slot % 16] = t[m, H + G:]
    return [a["out"], cache], [turned[:, :H].reshape(M, -1), want]


CASES = [(RESID, 896, 896, (0, 0, 0)), (RESID, 896, 4864, (0, 0, 0)), (RESID, 64, 256, (0, 0, 0)), (RESID, 1536, 8960, (0, 0, 0)), (SWIGLU, 9728, 896, (0, 0, 0)),
         (SWIGLU, 64, 64, (0, 0, 0)), (SWIGLU, 1024, 1536, (0, 0, 0)), (QKV, 1152, 896, (14, 2, 64)), (QKV, 192, 1088, (1, 1, 64)), (QKV, 2048, 1536, (12, 2, 128))]


@pytest.mark.gpu
@pytest.mark.parametrize("M", [17, 31, 32, 33, 50, 64])
@pytest.mark.parametrize("epilogue,N,K,heads", CASES)
def test_products(epilogue, N, K, heads, M):
    """Results that are rounded to bfloat16 once: at most 2^-9 of each value, so of the norm (2^-8 where the residual's term was rounded
    before and xn is rounded behind); partial sums of squares are float32."""
    got, want = run(epilogue, M, N, K, np.random.default_rng([epilogue, M, N]), heads, with_bias=(M % 2 == 1))
    for g, w, bound in zip(got, want, (2.0 ** -8, 2.0 ** -8, 1e-6)):
        assert off(g, w) < bound, off(g, w)


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(32, 64, 256), (64, 896, 896), (17, 2048, 256)])
def test_a_chain_of_products_whatever_the_dependents_wait_for(M, N, K):
    """Products one behind the other, started when the one in front is done (0), when it has begun (1) and when it has passed its own
    wait (2): the same sums, bit for bit."""
    import torch

    lib, rng = library(), np.random.default_rng([M, N, K])
    f32 = lambda *s: torch.from_numpy(rng.standard_normal(s).astype(np.float32)).cuda()  # noqa: E731
    W, x, resid, gain = bf16(rng, N, K).cuda(), bf16(rng, M, K).cuda(), f32(M, N) * 30, f32(N)
    parts = lib.eg_gemm_batch_takes(RESID, N, K, 0)
    got = []
    for mode in (0, 1, 2):
        r, xn, ss = resid.clone(), torch.empty(M, N, device="cuda", dtype=torch.bfloat16), torch.empty(M, parts, device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        for _ in range(24):
            assert lib.eg_gemm_batch(torch.cuda.current_stream().cuda_stream, RESID, mode, W.data_ptr(), K, None, M, N, K, x.data_ptr(), K, 1e-6, None, 0, None, 0, 0, 0, 0,
                                     None, None, None, None, 1, 0, 0, 0, r.data_ptr(), gain.data_ptr(), xn.data_ptr(), ss.data_ptr(), None, 0, status.data_ptr()) == 0
        torch.cuda.synchronize()
        assert int(status[0]) == 0
        got.append((r, xn, ss))
    step = (x.double() @ W.double().T).float().bfloat16().float()           # (a step's rounding may go the other way where its sum is off by a little)
    assert off(got[0][0] - resid, 24 * step.double()) < 2.0 ** -8
    for other in got[1:]:
        assert all(bool((a == b).all()) for a, b in zip(got[0], other))


@pytest.mark.gpu
@pytest.mark.parametrize("M", [17, 32, 33, 64])
@pytest.mark.parametrize("epilogue,N,K,heads", [(QKV, 512, 512, (2, 1, 128)), (QKV, 1152, 896, (14, 2, 64)), (QKV, 2048, 1536, (12, 2, 128)), (SWIGLU, 9728, 896, (0, 0, 0)),
                                                (SWIGLU, 128, 64, (0, 0, 0)), (RESID, 896, 4864, (0, 0, 0)), (RESID, 256, 320, (0, 0, 0))])
def test_products_value_by_value(epilogue, N, K, heads, M):
    """Products of order one, so that gates are neither open nor shut, every value by itself: one rounding to bfloat16 (eight bits: at most 2^-8 of
    it; two of them for xn, its own and its term's, which the gain multiplies), and what float32 sums of K products lose, 2^-24 sqrt(K) of the largest, at most 1e-4 of the usual value.  Heads
    of 128 in clusters of four and of eight; rows of x longer than K, and with weights asked for ahead, where the epilogue takes them."""
    plain_rows = epilogue == RESID
    got, want = run(epilogue, M, N, K, np.random.default_rng([epilogue, M, N, 5]), heads, M % 2 == 0, scale=K * K / 24, pad=64 if plain_rows else 0,
                    prefetch=100_000 if plain_rows else 0)
    for i, (g, w) in enumerate(zip(got, want)):
        slack = 2.0 ** -8 * w.abs() + 1e-4 * float(w.square().mean().sqrt())
        if plain_rows and i == 1:                                # xn: the gain is normal, 4.5 at most
            slack = slack + 2.0 ** -8 * 4.5 * want[0].abs()
        if plain_rows and i == 2:
            slack = 1e-5 * w
        assert bool(((g.double() - w).abs() <= slack).all()), (i, float(((g.double() - w).abs() - slack).max()))
