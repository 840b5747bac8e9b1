"""Launch rules that depend on the head size and on the 32-bit product's sizes (host side only)."""
from rocmforge_b200.kernels import basic


def test_small_heads_share_long_contexts_further():
    assert [basic.decode_splits(64, 2, n, None, 64) for n in (512, 1024, 4096)] == [1, 4, 4]
    assert basic.decode_splits(64, 2, 4096, None, 128) == 1 and basic.decode_splits(64, 2, 4096) == 1
    assert basic.decode_splits(64, 2, 4096, 512, 64) == 1                   # a window of 512: nine pages at most
    for B in (1, 2, 7, 33, 64, 300):
        for nkv in (1, 2, 14):
            for longest in (1, 64, 1000, 1024, 5000):
                s = basic.decode_splits(B, nkv, longest, None, 64)
                assert s in (1, 2, 4, 8, 16) and s <= max(1, basic.decode_pages(longest, None)) and s >= basic.decode_splits(B, nkv, longest)


def test_splits_of_the_32_bit_product_are_never_empty():
    for N in (1, 128, 129, 896, 1152, 9728, 151936):
        for K in (4, 32, 100, 896, 4864, 18944):
            s = basic.split_k_for_f32_tc(N, K, 148)
            kb = (K + 31) // 32
            assert 1 <= s and (s - 1) * ((kb + s - 1) // s) < kb and (s == 1 or s * ((N + 127) // 128) <= 148)


def test_channel_decays_chunk_by_each_sequences_own_length():
    """A sequence's chunks, and with them the order of its sums, must not depend on what the others of its step bring."""
    import numpy as np
    from rocmforge_b200.engine.batch import StepBatch, StepRequest
    from rocmforge_b200.parts.delta import GatedDeltaRule
    part = GatedDeltaRule(256, 2, 2, 128, 128, 4, 8, 8, 1e-6)
    few = GatedDeltaRule(256, 2, 2, 64, 128, 4, 8, 8, 1e-6)
    assert part.step_table_names() == ("channel_chunks",) and few.step_table_names() == ()
    tables = {"channel_chunks": lambda b: part.step_table("channel_chunks", b)}
    n = [20, 512, 511, 1, 700]
    t = StepBatch([StepRequest(i, [1] * k) for i, k in enumerate(n)], [0] * 5, 10, tables).tables["channel_chunks"]
    first, pairs = t[:6].tolist(), t[6:].reshape(-1, 2).tolist()
    assert first == [0, 0, 8, 8, 8, 19]
    assert pairs == [[1, 64 * i] for i in range(8)] + [[4, 64 * i] for i in range(11)]
    for alone in ([20], [511, 400], [1, 1]):
        assert StepBatch([StepRequest(i, [1] * k) for i, k in enumerate(alone)], [0] * len(alone), 10, tables).tables["channel_chunks"].size == 0
    # chunks of all sequences of a step whose longest is long enough: the table of the other recurrences
    t = StepBatch([StepRequest(i, [1] * k) for i, k in enumerate([20, 65])], [0, 0], 10,
                  {"x": lambda b: part.step_table("retention_chunks", b)}).tables["x"]
    assert np.array_equal(t, [0, 1, 3, 0, 0, 1, 0, 1, 64])


def test_attention_in_32_bits_goes_by_each_sequences_own_tokens():
    """Which kernel a sequence takes must not depend on what the others of its step bring."""
    import torch
    from rocmforge_b200.engine.batch import StepBatch, StepRequest
    from rocmforge_b200.kernels import F32_PROMPT_FROM as many
    from rocmforge_b200.parts import MIXERS, POSITIONS
    part = MIXERS.build("gqa_attention", hidden=32, n_heads=2, n_kv_heads=1, head_dim=64, qkv_bias=False,
                        position=POSITIONS.build("rope_neox", head_dim=64, theta=1e4))
    part.bind({n: torch.zeros(*sp.shape) for n, sp in part.param_specs().items()}, torch.float32)
    assert part.step_table_names() == ("f32_prompt_tiles", "f32_token_rows")

    def tables(n, starts=None):
        t = StepBatch([StepRequest(i, [1] * k) for i, k in enumerate(n)], starts or [0] * len(n), 10,
                      {name: (lambda b, name=name: part.step_table(name, b)) for name in part.step_table_names()}).tables
        return t["f32_prompt_tiles"].reshape(-1, 2).tolist(), t["f32_token_rows"].tolist()
    assert tables([1, many, 2, 130]) == ([[1, 0], [3, 0], [3, 128]], [0, many + 1, many + 2])
    assert tables([130, many], [0, 500]) == ([[0, 0], [0, 128], [1, 0]], [])
    assert tables([many - 1, 5]) == ([], []) and tables([1, 1, 1]) == ([], [])


def test_forms_of_products_of_few_tokens():
    """1: tiles of 64 weight rows, 2: eight epilogue warps, 0: the general form (one function for all products of a step, whose
    instructions stay at hand).  A form of its own slows a step down where its product gains less than its instructions cost."""
    from rocmforge_b200.csrc import build
    from rocmforge_b200.kernels import tensor_core as tc
    form = build.load("gemm_tcgen05").rf_gemm_tc_skinny_form
    of = lambda M, N, K, mode, splits=1, normed=0: form(M, N, K, K, mode, splits, normed, 148)
    for mode in (tc.STORE, tc.SWIGLU, tc.REGLU, tc.GEGLU, tc.CLAMPGLU):
        assert [of(M, 9728, 2048, mode) for M in (1, 16, 33, 64, 65, 128)] == [1] * 6
        assert [of(M, 148 * 128 + 2, 2048, mode) for M in (1, 16, 17, 32, 33, 64, 65, 128)] == [0, 0, 0, 0, 2, 2, 2, 2]
        assert of(8, 9728, 2048, mode, normed=1) == 0
    assert [of(M, 17920, 1536, tc.SWIGLU) for M in (17, 24, 32)] == [0, 0, 0]          # was up to 8 % of a step slower in half tiles
    assert [of(M, 2304, 2048, tc.STORE) for M in (17, 32)] == [1, 1]
    assert [of(M, N, K, tc.F32) for M, N, K in ((1, 16, 1024), (16, 64, 2048), (16, 64, 1016), (17, 64, 2048), (64, 64, 2048), (8, 32000, 2048))
            ] == [1, 1, 0, 0, 0, 0]
    for mode in (tc.RESIDUAL, tc.PARTIAL, tc.RESNORM):
        assert all(of(M, 9728, 2048, mode) == 0 for M in (1, 17, 64, 128))
    assert of(64, 4608, 3584, tc.PARTIAL, splits=8) == 0
    # activations of less than 128 KB in a tile that reaches beyond 128 KB
    assert [of(M, 9728, 896, tc.SWIGLU) for M in (64, 65, 73, 74, 128)] == [1, 0, 0, 1, 1]
    assert [of(M, 17920, 1536, tc.SWIGLU) for M in (33, 42, 43, 64)] == [0, 0, 1, 1]
    assert [of(M, 40000, 896, tc.STORE) for M in (65, 74)] == [0, 2]


def test_when_decode_attention_forms_its_own_queries():
    """Heads of 64 always; heads of 128 where the attention's CTAs find room beside the q|k|v product's."""
    def takes(B, heads, kv, width, longest=512, span=None, hd=128):
        N = (heads + 2 * kv) * hd
        product = (N + 127) // 128 * tc.split_k_for(N, width, 148, tokens=B)
        return basic.decode_forms_queries(B, kv, hd, longest, span, product, 148)
    from rocmforge_b200.kernels import tensor_core as tc
    assert all(takes(B, 14, 2, 896, n, hd=64) for B in (1, 8, 64, 128) for n in (512, 1024, 16384))
    assert [B for B in range(1, 17) if takes(B, 28, 4, 3584)] == [1, 2, 3, 4, 5]          # 7B; at 6 and 8 the writer's step is shorter
    assert [B for B in range(1, 17) if takes(B, 28, 4, 3584, 1024)] == [1, 2]
    assert [B for B in range(1, 9) if takes(B, 40, 8, 5120)] == [1, 2, 3]                 # 14B
    assert [B for B in range(1, 9) if takes(B, 48, 8, 6144)] == [1, 2]
    assert [B for B in range(1, 33) if takes(B, 16, 2, 2048)] == list(range(1, 17))
    assert not any(takes(B, 28, 4, 3584, 8192) for B in (1, 2, 8, 64)) and takes(1, 28, 4, 3584, 8192, 128)
    assert not takes(1, 16, 2, 4096, hd=256)


def test_k_splits_of_a_short_k():
    from rocmforge_b200.kernels import tensor_core as tc
    for tokens in (1, 16, 17, 32):
        assert [tc.split_k_for(1024, 64 * kb, 148, tokens) for kb in range(7, 18)] == [1, 4, 3, 5, 4, 6, 5, 7, 5, 8, 4]
    for tokens in (33, 64, 128, None):                    # at most six stacks
        assert [tc.split_k_for(1024, 64 * kb, 148, tokens) for kb in range(7, 18)] == [1, 4, 3, 5, 4, 6, 5, 5, 5, 6, 4]
    for N in (896, 1152, 1536, 2304, 3112, 4608, 6144, 9728, 18944, 40000):
        for K in (512, 520, 576, 640, 704, 768, 832, 896, 960, 1000, 1024):
            for tokens in (8, 32, 64):
                s, kb, tiles = tc.split_k_for(N, K, 148, tokens), (K + 63) // 64, (N + 127) // 128
                per = -(-kb // s)
                assert (s - 1) * per < kb, "no split is empty"
                assert s == 1 or (tiles * s <= 2 * 148 and per >= 2)
                assert tiles * s <= 148 or s <= kb // 4, "more than a CTA per SM: at least four blocks a split"
    # the product that finishes the residual update: splits of four blocks and more, as many as form a cluster
    assert [tc.resnorm_splits(n, n) for n in (512, 768, 896, 1024, 2048, 3584)] == [2, 2, 2, 4, 8, 8]
