"""The delta rule with a decay per key channel in chunks of 64 tokens (csrc/delta.cu), against the recurrence in 64 bits and the scan."""
import pytest
import torch
from plain import ludusun_plain as P

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def i32(*v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("H,G,dim,vdim", [(4, 2, 24, 12), (3, 3, 64, 40), (1, 1, 256, 8), (2, 1, 128, 128), (2, 2, 1, 5), (1, 1, 130, 70),
                                          (2, 1, 30, 33), (1, 1, 200, 20), (2, 2, 68, 36)])
def test_chunks_with_a_decay_per_channel(H, G, dim, vdim):
    """Sequences of a whole number of chunks, of one token more, of a few tokens, side by side and cut in two steps; a continued
    state; decays of exactly 0 and 1 and tiny ones, for whole tokens and single channels; keys that repeat."""
    from rocmforge_b200 import kernels
    torch.manual_seed(dim + H)
    lens, slots = [129, 64, 3, 200], [1, 4, 0, 3]
    T = sum(lens)
    q = torch.randn(T, G * dim, device=DEV) * dim ** -0.5
    k = torch.nn.functional.normalize(torch.randn(T, G, dim, device=DEV), dim=-1)
    k[20:60], k[150:158] = k[20:21].clone(), k[150:151].clone()
    k = k.reshape(T, G * dim).contiguous()
    v = torch.randn(T, 3 + H * vdim, device=DEV)[:, 3:]
    beta, decay = torch.rand(T, H, device=DEV), torch.rand(T, H * dim, device=DEV) ** 0.2
    for t, g in ((0, 0.0), (5, 1.0), (63, 0.0), (64, 1e-30), (65, 1e-30), (128, 1.0), (193, 0.0), (260, 1.0)):
        decay[t] = g
    decay[300:340] = 1.0
    decay[100, ::3], decay[101, 1::2], decay[350:, -1] = 0.0, 1.0, 1e-38
    starts = [sum(lens[:i]) for i in range(4)]
    state = torch.zeros(6, H, dim, vdim, device=DEV)
    begin = torch.randn(H, dim, vdim, device=DEV)
    state[4] = begin
    scan_state = state.clone()

    def run(ends, cut, f, state):
        live = [i for i in range(4) if ends[i] > cut[i]]
        rows = torch.cat([torch.arange(starts[i] + cut[i], starts[i] + ends[i]) for i in live]).to(DEV)
        ns = [ends[i] - cut[i] for i in live]
        counts = [(n + 63) // 64 for n in ns]
        table = [sum(counts[:j]) for j in range(len(live) + 1)] + [x for j, n in enumerate(ns) for r in range(0, n, 64) for x in (j, r)]
        cu = [sum(ns[:j]) for j in range(len(ns) + 1)]
        at = i32(*[slots[i] for i in live])
        if f == "scan":
            kq = (q.view(T, G, dim) * k.view(T, G, dim)).sum(-1)
            o = kernels.delta_scan(q[rows], k[rows], kq[rows], decay[rows], beta[rows], v[rows], state, i32(*cu), at, H, G, dim, vdim)
        else:
            o = kernels.delta_chunked(q[rows], k[rows], decay[rows], beta[rows], v[rows], state, i32(*table), i32(*cu), at, H, G, dim, vdim)
        return {i: o[cu[j]:cu[j + 1]] for j, i in enumerate(live)}
    first, second = run([70, 64, 3, 100], [0] * 4, "chunks", state), run([129, 64, 3, 200], [70, 64, 3, 100], "chunks", state)
    scan = run(lens, [0] * 4, "scan", scan_state)
    for i in range(4):
        a, b = starts[i], starts[i] + lens[i]
        got = torch.cat([first[i], second[i]]) if i in second else first[i]
        for h in range(H):
            g = slice(h // (H // G) * dim, (h // (H // G) + 1) * dim)
            want, end = P.delta_recurrence(*(x[a:b].double().cpu() for x in (q[:, g], k[:, g], v[:, h * vdim:(h + 1) * vdim], beta[:, h],
                                             decay[:, h * dim:(h + 1) * dim])), S=begin[h].double().cpu() if slots[i] == 4 else None)
            # 32-bit sums over some hundred tokens and channels: 2e-5 of the result's size, as for the chunks with one decay per head
            for y, z, x in ((got, scan[i], want), (state[slots[i], h], scan_state[slots[i], h], end)):
                if y.dim() == 2 and y.shape[0] == b - a and y is got:
                    y, z = y[:, h * vdim:(h + 1) * vdim], z[:, h * vdim:(h + 1) * vdim]
                size = x.norm() + 1e-6
                assert (y.double().cpu() - x).norm() < 2e-5 * size and (z.double().cpu() - x).norm() < 2e-5 * size, (i, h)
    assert not state[2].any() and not state[5].any()
