"""Host-side choices of the kernel bindings (no GPU needed): which sizes go to which kernel."""
import torch

from easy_gpt.cpp_b200 import kernels


def test_fused_norm_limit_follows_the_width():
    assert kernels.fused_norm_max_tokens(896) == kernels.FUSED_NORM_MAX_TOKENS
    assert kernels.fused_norm_max_tokens(3584) == kernels.FUSED_NORM_MAX_TOKENS
    # 16 rows of 8192 bfloat16 values do not fit 200 KB of shared memory, 8 rows do
    assert kernels.fused_norm_max_tokens(8192) == min(8, kernels.FUSED_NORM_MAX_TOKENS)
    assert kernels.fused_norm_max_tokens(20000) == 0
    assert kernels.fused_norm_max_tokens(120) == 0            # rows of 240 bytes: the decode product wants multiples of 32


def test_decode_product_policy():
    assert kernels.gemm_skinny_takes(torch.bfloat16, 1, 896)
    assert kernels.gemm_skinny_takes(torch.bfloat16, kernels.SKINNY_MAX_TOKENS, 4864)
    assert not kernels.gemm_skinny_takes(torch.bfloat16, kernels.SKINNY_MAX_TOKENS + 1, 896)
    assert not kernels.gemm_skinny_takes(torch.bfloat16, 4, 900)            # K % 16
    assert not kernels.gemm_skinny_takes(torch.float32, 4, 896)
    assert [kernels.skinny_padded_tokens(m) for m in (1, 8, 9, 16, 17, 33, 64)] == [8, 8, 16, 16, 32, 64, 64]


def test_decode_product_plans_cover_the_matrix():
    for rows, width, head in ((1152, 896, 64), (896, 896, 0), (9728, 896, 0), (896, 4864, 0), (151936, 896, 0),
                              (4608, 3584, 128), (3584, 18944, 0), (48, 48, 0), (391, 80, 0)):
        rb, ks, split = kernels.skinny_plan(rows, width, head)
        assert rb >= 1 and ks >= 1 and split >= 1
        assert rb * ks <= 32                                        # warps of a CTA
        if head:
            assert rb * 16 == head and 1 <= split <= 8
            # only heads that are much for one SM are cut, and only where the heads leave most SMs idle
            assert (split == 1) == (head * width * 2 < (192 << 10) or (rows // head) * 8 > kernels.sm_count())


def test_the_native_engine_plans_like_the_pytorch_face():
    """The launch rules exist twice, in ``csrc/engine/plans.hpp`` for the native engine and in ``kernels.py`` for the
    PyTorch face: over the sizes of the family's models and some odd ones they must give the same plans."""
    from easy_gpt.cpp_b200 import native

    assert native.plan(4)[0] == kernels.sm_count()
    shapes = [(1152, 896, 64), (896, 896, 0), (9728, 896, 0), (896, 4864, 0), (151936, 896, 0), (2048, 1536, 128),
              (1536, 1536, 0), (17920, 1536, 0), (1536, 8960, 0), (151936, 1536, 0), (4608, 3584, 128), (3584, 3584, 0),
              (37888, 3584, 0), (3584, 18944, 0), (152064, 3584, 0), (48, 48, 0), (391, 80, 0), (160, 112, 16), (96, 2048, 32),
              (256, 4096, 0), (640, 640, 0), (5120, 5120, 128), (8192, 8192, 0), (1024, 28672, 0)]
    for rows, width, head in shapes:
        assert native.plan(0, rows, width, head)[:3] == tuple(kernels.skinny_plan(rows, width, head)), (rows, width, head)
    for tokens in (1, 2, 4, 8, 9, 16, 17, 24, 32, 48, 64, 128):
        for heads, kv, head in ((14, 2, 64), (12, 2, 128), (28, 4, 128), (4, 4, 32), (16, 1, 256), (3, 1, 64)):
            for context in (1, 63, 64, 500, 4096, 8192, 32768, 131072):
                assert native.plan(1, tokens, heads, kv, context, head)[0] == \
                    kernels.attention_paged_splits(tokens, heads, kv, context, head), (tokens, heads, kv, context, head)
    for width in (48, 120, 896, 1536, 3584, 5000, 8192, 20000):
        assert native.plan(2, width)[0] == kernels.fused_norm_max_tokens(width), width
    # the prompt attention's rule, for contexts short enough that the native engine's extra rule for long ranges is silent
    for tiles in (1, 2, 3, 4, 8, 16, 40, 200):
        for heads, head in ((14, 64), (12, 128), (28, 128), (4, 64)):
            assert native.plan(3, tiles, heads, head, 2048)[:2] == tuple(kernels.attention_prefill_parts(tiles, heads, head)), (tiles, heads, head)


def test_the_streaming_product_is_planned_alike_for_1_to_16_tokens():
    """Which products the streaming kernel takes, and the order of their sums, hang off the epilogue, N and K alone; what a token tile
    decides (the ring, CTAs an SM) has to fit: sizes of real models among them where a tile of 16 tokens fits and one of 8 does not, or
    the other way round."""
    sizes = [(n, k) for n in (8, 900, 896, 1536, 2048, 2560, 3072, 3584, 4096, 5120, 6416, 9728, 37888, 151936)
             for k in (16, 208, 896, 1536, 2064, 4864, 8192, 8960, 11008, 13824, 14336, 18944)]
    taken = 0
    for epilogue in range(5):
        for n, k in sizes:
            if epilogue == kernels.EPI_QKV_ROPE and n % 32:
                continue
            plans = [kernels.gemm_stream_plan(epilogue, n, k, m) for m in range(1, 17)]
            assert len({p[:3] if p else None for p in plans}) == 1, (epilogue, n, k, plans[0], plans[-1])
            for m, p in enumerate(plans, 1):
                if p is None:
                    continue
                taken += 1
                rb_log, split, k_len, per_sm, stages, grid, share = p
                tile, rows = 8 if m <= 8 else 16, 16 << rb_log
                assert split in (1, 2, 3, 4, 5, 6, 7, 8) and (split - 1) * k_len < k <= split * k_len and k_len % 64 == 0
                assert (grid * share if share else grid * (rows >> 4)) * 16 >= n - grid * 16
                shared = 2048 + stages * 16384 + tile * (k_len * 2 + 16) + 8 * tile * 80 + (split - 1) * rows * tile * 4
                assert 1 <= stages <= 16 and shared * per_sm <= 227 * 1024, (epilogue, n, k, m, p)
                if split > 1:
                    assert grid * split <= 148 * per_sm and not share
    assert taken > 2000
    assert kernels.gemm_stream_plan(kernels.EPI_F32, 2048, 11008, 16) and not kernels.gemm_stream_plan(kernels.EPI_F32, 5120, 13824, 1)


def test_no_more_is_asked_ahead_of_the_l2_than_it_can_hold():
    from easy_gpt.cpp_b200 import native

    for bytes_, want in ((0, 0), (17 << 20, 17 << 20), (32 << 20, 32 << 20), (55 << 20, 32 << 20), (126 << 20, 32 << 20), (37888 * 3584 * 2, 0), (1 << 40, 0)):
        assert native.plan(5, bytes_)[0] == want, bytes_


def test_general_delta_steps_in_chunks():
    """Entries of 32 tokens on average, one of which has 48 where there are more than two (heads of 64): shorter ones are faster in blocks.  The
    scratch memory that a caller makes from tokens and heads alone holds every such step's chunks: tokens / 16 of each entry, rounded up, of 7,232
    values each."""
    from easy_gpt.cpp_b200 import kernels

    lib = kernels.library()
    takes, record = lib.eg_general_delta_in_chunks, lib.eg_general_delta_record
    for counts, want in (([31], 0), ([32], 1), ([2047], 1), ([63], 1), ([40, 20], 0), ([33] * 2, 1), ([33] * 3, 0), ([33] * 8, 0), ([33] * 31, 0), ([40] * 4, 0), ([48] * 4, 1),
                         ([48] * 31, 1), ([500] + [1] * 14, 1), ([1000] + [1] * 30, 1), ([1000] + [1] * 40, 0), ([90, 31, 20, 1], 1)):
        assert takes(sum(counts), len(counts), max(counts), 64) == want, counts
    assert not any(takes(4096, 1, 4096, dim) for dim in (16, 32, 63, 65, 128)) and takes(0, 0, 0, 64) == 0
    for entries in range(1, 80):
        for tokens in range(entries, 40 * entries + 400):
            if takes(tokens, entries, tokens - entries + 1, 64):
                assert (tokens + 15 * entries) // 16 * 7232 <= tokens * record(64)
    assert record(64) >= 6 * 64 + 8 and record(32) == 6 * 32 + 8
