"""Normed heads of a prompt step: a token or two a block and two heads a warp in flight.  Sizes at the edges of both: the last block with
one token, fewer heads than warps, heads that do not fill the last pair."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("T", [256, 2047, 2048, 2049])
@pytest.mark.parametrize("nh,nkv,hd", [(1, 1, 64), (5, 1, 128), (16, 4, 128), (7, 1, 256)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32], ids=str)
def test_the_bits_of_a_few_rows(T, nh, nkv, hd, dt):
    """The form for few rows sums a head's squares in the same order, so every bit is the same."""
    from rocmforge_b200 import kernels
    torch.manual_seed(T + nh)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    pages = -(-T // 64)
    table, seq, pos, slot = i32(list(range(pages))).view(1, -1), i32([0] * T), i32(list(range(T))), i32([0])
    src = torch.randn(T, (nh + 2 * nkv) * hd, device=DEV).to(dt)
    inv = 1e4 ** (-torch.arange(hd // 2, device=DEV).float() / (hd // 2))
    w = torch.rand(2, hd, device=DEV) + 0.5

    def run(rows):
        kp, vp = (torch.zeros(pages, nkv, 64, hd, device=DEV, dtype=dt) for _ in range(2))
        x, q = src.clone(), []
        for a in range(0, T, rows):
            b = min(T, a + rows)
            q.append(kernels.head_norm_kv_write(x[a:b], nh, nkv, hd, hd, inv, seq[a:b], pos[a:b], slot, table, kp, vp, True, compute_dtype=dt,
                                                rot_dim=hd, unit_norm_eps=1e-6, q_norm_weight=w[0], k_norm_weight=w[1])[:, :nh * hd].clone())
        return torch.cat(q), kp, vp
    for a, b in zip(run(T), run(255)):
        assert torch.equal(a, b)
