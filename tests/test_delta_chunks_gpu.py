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


def ragged(lens, H, G, dim, vdim, per_head, seed):
    torch.manual_seed(seed)
    T = sum(lens)
    q, k = (torch.nn.functional.normalize(torch.randn(T, G, dim, device=DEV), dim=-1).reshape(T, G * dim).contiguous() for _ in range(2))
    v, beta = torch.randn(T, H * vdim, device=DEV), torch.rand(T, H, device=DEV)
    decay = torch.rand(T, H if per_head else H * dim, device=DEV) ** 0.1
    return q, k, (q.view(T, G, dim) * k.view(T, G, dim)).sum(-1), decay, beta, v


def chunk_table(lens):
    counts = [(n + 63) // 64 for n in lens]
    return i32(*([sum(counts[:j]) for j in range(len(lens) + 1)] + [x for j, n in enumerate(lens) for r in range(0, n, 64) for x in (j, r)]))


@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("H,G,dim,vdim", [(4, 2, 24, 12), (2, 1, 128, 40), (1, 1, 200, 20)])
def test_passes_over_the_chunks_change_no_bit(per_head, H, G, dim, vdim):
    """Chunks are taken in passes of bounded scratch memory: passes of 1, 3 and 7 chunks, which cut sequences anywhere, against one pass."""
    from rocmforge_b200 import kernels
    lens, slots = [300, 64, 1, 130, 449], [3, 0, 5, 1, 2]
    q, k, kq, decay, beta, v = ragged(lens, H, G, dim, vdim, per_head, dim)
    cu = i32(*[sum(lens[:j]) for j in range(6)])
    begin = torch.randn(6, H, dim, vdim, device=DEV)
    got = []
    for most in (0, 1, 3, 7):
        state = begin.clone()
        got.append((kernels.delta_chunked(q, k, decay, beta, v, state, chunk_table(lens), cu, i32(*slots), H, G, dim, vdim, chunks_per_pass=most), state))
    for o, state in got[1:]:
        assert torch.equal(o, got[0][0]) and torch.equal(state, got[0][1])


@pytest.mark.parametrize("per_head", [False, True])
def test_the_chunks_scratch_memory_is_bounded(per_head):
    """30,000 tokens of 16 heads of 128 x 128: beyond its result the call holds 512 MB and a little, not a size that grows with the prompt."""
    from rocmforge_b200 import kernels
    lens, H, dim = [17000, 13000], 16, 128
    q, k, kq, decay, beta, v = ragged(lens, H, H, dim, dim, per_head, 1)
    state, table, cu = torch.zeros(2, H, dim, dim, device=DEV), chunk_table(lens), i32(0, 17000, 30000)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    o = kernels.delta_chunked(q, k, decay, beta, v, state, table, cu, i32(0, 1), H, H, dim, dim)
    assert torch.cuda.max_memory_allocated() - before < o.numel() * 4 + (520 << 20)


def test_a_sequences_sums_do_not_depend_on_the_others():
    """Sequences of 20, 511, 512, 700 and 1 tokens in one step and alone in theirs: the same outputs and states, bit for bit, through
    the mixer's own choice of kernels."""
    from types import SimpleNamespace
    from rocmforge_b200.engine.batch import StepBatch, StepRequest
    from rocmforge_b200.parts.delta import GatedDeltaRule
    H, G, dim, vdim = 2, 1, 128, 40
    part = GatedDeltaRule(256, H, G, dim, vdim, 4, 8, 8, 1e-6)
    lens, slots = [20, 511, 512, 700, 1], [2, 0, 4, 1, 3]
    data = ragged(lens, H, G, dim, vdim, False, 5)
    begin = torch.randn(5, H, dim, vdim, device=DEV)

    def run(which):
        batch = StepBatch([StepRequest(slots[i], [1] * lens[i]) for i in which], [0] * len(which), 10,
                          {n: (lambda b, n=n: part.step_table(n, b)) for n in part.step_table_names()})
        rows = torch.cat([torch.arange(sum(lens[:i]), sum(lens[:i + 1])) for i in which]).to(DEV)
        ctx = SimpleNamespace(cu_q=i32(*batch.cu_q.tolist()), seq_slot=i32(*batch.slots), max_new=batch.max_new, is_decode=False, host=batch,
                              tables={n: torch.from_numpy(t).to(DEV) for n, t in batch.tables.items()})
        state = begin.clone()
        return part.recurrence(ctx, *(x[rows] for x in data), state), state, rows
    whole, state, _ = run(range(5))
    for i in range(5):
        o, alone, rows = run([i])
        assert torch.equal(o, whole[rows]) and torch.equal(alone[slots[i]], state[slots[i]]), lens[i]
