"""The decode attention that forms its own queries, keys and values, against the writer and the attention it stands for: the same
additions and rotations in the same order, so the same bits in the cache and, with tiles of as many keys, in its results."""
import pytest
import torch

from rocmforge_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("nh,nkv,hd,lengths,parts,splits,warps,span,bias", [
    (14, 2, 64, [1, 32, 33, 64, 65, 500], 3, 2, 8, {}, torch.bfloat16),
    (14, 2, 64, [1, 63, 64, 200, 1025], 1, 1, 4, {}, None),                       # one sum; a CTA of four warps with all pages
    (28, 4, 128, [512, 1, 97, 64], 15, 4, 8, {}, torch.float32),                  # more sums than are asked for at once
    (8, 1, 128, [700, 128, 129], 8, 1, 4, {}, torch.bfloat16),                    # eight heads a group: more items than threads
    (16, 2, 128, [33, 300], 9, 2, 8, {}, torch.bfloat16),
    (8, 1, 64, [70], 2, 16, 4, {}, None),                                         # more CTAs than pages
    (4, 4, 64, [5, 200, 640], 4, 2, 4, {"window": 100}, None),
    (6, 2, 64, [64, 65, 130], 5, 2, 8, {"chunk": 64}, torch.float32),
])
def test_against_writer_and_attention(nh, nkv, hd, lengths, parts, splits, warps, span, bias):
    g = torch.Generator(DEV).manual_seed(nh * hd + len(lengths))
    B, width = len(lengths), (nh + 2 * nkv) * hd
    per = [(n + 63) // 64 for n in lengths]
    pages = torch.randperm(sum(per), generator=torch.Generator().manual_seed(3)).tolist()
    table = torch.zeros((B, max(per)), dtype=torch.int32)
    for i, n in enumerate(per):
        table[i, :n] = torch.tensor(pages[sum(per[:i]):sum(per[:i + 1])])
    table = table.to(DEV)
    kp, vp = (torch.randn((sum(per), nkv, 64, hd), generator=g, device=DEV).bfloat16() for _ in range(2))
    for i, n in enumerate(lengths):                       # what lies behind a sequence's end, its newest place included, is never used
        for cache in (kp, vp):
            cache[table[i, per[i] - 1].long(), :, (n - 1) % 64:] = float("nan")
    sums = torch.randn((parts, B, width), generator=g, device=DEV)
    b = None if bias is None else torch.randn((width,), generator=g, device=DEV).to(bias)
    freq = 1e4 ** (-torch.arange(hd // 2, device=DEV, dtype=torch.float32) / (hd // 2))
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    seq, pos = i32(list(range(B))), i32([n - 1 for n in lengths])
    slot = i32(list(range(B)))
    k1, v1, k2, v2 = kp.clone(), vp.clone(), kp.clone(), vp.clone()
    q = kernels.rope_kv_write(sums, nh, nkv, hd, freq, seq, pos, slot, table, k1, v1, bias=b, compute_dtype=torch.bfloat16)
    scale, window, chunk = hd ** -0.5, span.get("window"), span.get("chunk")
    want = kernels.attention_decode_warps(q, nh, nkv, hd, k1, v1, seq, pos, slot, table, scale, window, splits=splits, warps=warps, chunk=chunk)
    got = kernels.attention_decode_formed(sums, nh, nkv, hd, freq, k2, v2, seq, pos, slot, table, scale, window, splits=splits, warps=warps,
                                          bias=b, chunk=chunk)
    bits = lambda t: t.view(torch.int16)
    assert want.isfinite().all()
    assert torch.equal(bits(k1), bits(k2)) and torch.equal(bits(v1), bits(v2))
    if hd == 64:
        assert torch.equal(bits(got), bits(want))
    else:
        # tiles of 16 keys: a weight is rounded by 2^-9 of itself, by either kernel against its own tile's maximum, and so is a result
        torch.testing.assert_close(got.float(), want.float(), atol=2.0 ** -8 * float(v1.nan_to_num().abs().max()), rtol=2.0 ** -8)
    kernels.tensor_core.check_status(torch.device(DEV))
