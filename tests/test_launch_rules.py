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
