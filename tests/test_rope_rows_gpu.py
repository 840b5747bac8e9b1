"""The rotation and cache write of prompt steps (64 tokens and more, whole heads turned as split pairs, rows of one tensor)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DTS = [torch.float32, torch.bfloat16]


@pytest.mark.parametrize("dt", DTS)
@pytest.mark.parametrize("nh,nkv,hd", [(4, 2, 16), (3, 1, 72), (14, 2, 64), (5, 5, 128), (2, 1, 104), (1, 1, 2048)])
@pytest.mark.parametrize("T", [64, 300, 2367, 2371, 4741])
@pytest.mark.parametrize("writes", [True, False])
def test_prompt_rows(dt, nh, nkv, hd, T, writes):
    """Against the rotation in 64 bits by the kernel's own 32-bit angles; one token a block up to 2,367 tokens, then 2, 4 or 8.  Sequences begin and end inside a block, the last block is
    not full, pages start as NaN so that a stray write shows.  A rotated number carries two roundings of 32 bits for each product and
    one for the sum, 2 ulp of sine and cosine, and the rounding to the compute dtype."""
    from rocmforge_b200 import kernels
    g = torch.Generator().manual_seed(T + hd)
    cuts = sorted({0, T, *torch.randint(1, T, (9,), generator=g).tolist()})
    lens = [b - a for a, b in zip(cuts, cuts[1:])]
    start = [int(x) for x in torch.randint(0, 150, (len(lens),), generator=g)]
    seq = torch.cat([torch.full((n,), i) for i, n in enumerate(lens)])
    pos = torch.cat([torch.arange(s, s + n) for s, n in zip(start, lens)])
    need = [(s + n + 63) // 64 for s, n in zip(start, lens)]
    order = torch.randperm(sum(need), generator=g).tolist()
    table = torch.zeros(len(lens), max(need), dtype=torch.int32)
    for i, n in enumerate(need):
        for j in range(n):
            table[i, j] = order.pop()
    slots = torch.arange(len(lens)).flip(0)
    x = torch.randn(T, (nh + 2 * nkv) * hd, generator=g).to(dt)
    inv = (1e4 ** (-torch.arange(hd // 2, dtype=torch.float64) * 2 / hd)).float()
    pages = [torch.full((sum(need), nkv, 64, hd), float("nan"), dtype=dt, device=DEV) for _ in range(2)]
    by_slot = torch.zeros_like(table)
    by_slot[slots] = table
    i32 = lambda t: t.to(torch.int32).to(DEV)
    got = x.to(DEV)
    q = kernels.rope_kv_write(got, nh, nkv, hd, inv.to(DEV), i32(seq), i32(pos), i32(slots), i32(by_slot), *pages, write_kv=writes)
    assert torch.equal(got[:, nh * hd:].cpu(), x[:, nh * hd:])
    ang = (pos.float()[:, None] * inv).double()[:, None]
    c, s = ang.cos(), ang.sin()
    v = x.double().view(T, nh + 2 * nkv, hd)
    a, b = v[:, :nh + nkv, :hd // 2], v[:, :nh + nkv, hd // 2:]
    ref = torch.cat([a * c - b * s, a * s + b * c], -1)
    size = (torch.cat([a, a], -1).abs() + torch.cat([b, b], -1).abs())
    bound = size * 2.0 ** -21 + (ref.abs() * 2.0 ** -8 if dt == torch.bfloat16 else 0)
    out = q[:, :nh * hd].double().cpu().view(T, nh, hd)
    assert ((out - ref[:, :nh]).abs() <= bound[:, :nh]).all()
    if not writes:
        assert all(p.isnan().all() for p in pages)
        return
    where = table.long()[seq, pos // 64]
    kp, vp = (p.cpu() for p in pages)
    assert ((kp[where, :, pos % 64].double() - ref[:, nh:]).abs() <= bound[:, nh:]).all()
    assert torch.equal(vp[where, :, pos % 64], x.view(T, -1, hd)[:, nh + nkv:])
    for p in (kp, vp):
        p[where, :, pos % 64] = float("nan")
        assert p.isnan().all()


def test_heads_of_four_element_groups_run_at_the_speed_of_their_bytes():
    """Heads of 104 in bfloat16 (whole accesses of 8 bytes, not of 16) and of 96: the time per byte is within a factor of two, so they do
    not fall to the form with a pair a thread."""
    from rocmforge_b200 import kernels

    def time(hd, nh=32, nkv=8, T=8192):
        x = torch.randn(T, (nh + 2 * nkv) * hd, device=DEV).bfloat16()
        pages = [torch.zeros(T // 64, nkv, 64, hd, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
        i32 = lambda t: t.to(torch.int32).to(DEV)
        args = (nh, nkv, hd, torch.rand(hd // 2, device=DEV), i32(torch.zeros(T)), i32(torch.arange(T)), i32(torch.zeros(1)),
                i32(torch.arange(T // 64))[None], *pages)
        best = 1e9
        for _ in range(6):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            for _ in range(10):
                kernels.rope_kv_write(x, *args)
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]))
        return best / hd
    assert time(104) < 2 * time(96)
