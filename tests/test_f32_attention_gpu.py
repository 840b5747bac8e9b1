"""The 32-bit attention kernels for prompts and for single tokens (csrc/attention_f32.cuh) at the edges of their tiles, against 64 bits
and against the generic kernel."""
import random

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def batch(starts, news, nh, nkv, hd, seed=0):
    """Sequences with ``starts`` cached and ``news`` new tokens over shuffled pages; what no sequence holds is NaN."""
    g, r = torch.Generator().manual_seed(seed), random.Random(seed)
    ends = [a + b for a, b in zip(starts, news)]
    n_pages = sum((n + 63) // 64 for n in ends) + 2
    order = list(range(n_pages))
    r.shuffle(order)
    kp = torch.full((n_pages, nkv, 64, hd), float("nan"))
    vp, table, ks, vs = kp.clone(), torch.zeros(len(ends), max((n + 63) // 64 for n in ends), dtype=torch.int32), [], []
    for i, n in enumerate(ends):
        k, v = torch.randn(n, nkv, hd, generator=g), torch.randn(n, nkv, hd, generator=g)
        for p in range((n + 63) // 64):
            table[i, p], m = order.pop(), min(64, n - p * 64)
            kp[table[i, p], :, :m] = k[p * 64:p * 64 + m].transpose(0, 1)
            vp[table[i, p], :, :m] = v[p * 64:p * 64 + m].transpose(0, 1)
        ks.append(k), vs.append(v)
    q = torch.randn(sum(news), nh * hd + 8, generator=g).to(DEV)[:, :nh * hd]            # rows with a stride
    tiles = sorted(((i, a) for i, n in enumerate(news) for a in range(0, n, 128)), key=lambda t: starts[t[0]] + t[1])
    cu = [0]
    for n in news:
        cu.append(cu[-1] + n)
    return dict(q=q, kp=kp.to(DEV), vp=vp.to(DEV), table=table.to(DEV), ks=ks, vs=vs, starts=starts, news=news, nh=nh, nkv=nkv, hd=hd,
                seq=i32([i for i, n in enumerate(news) for _ in range(n)]), pos=i32([s + j for s, n in zip(starts, news) for j in range(n)]),
                slot=i32(list(range(len(ends)))), cu=i32(cu), start=i32(starts), new=i32(news), tiles=i32([x for t in tiles for x in t]))


def run(b, kind, scale=None, window=None, chunk=None, **kw):
    from rocmforge_b200 import kernels
    scale = scale or b["hd"] ** -0.5
    head = (b["q"], b["nh"], b["nkv"], b["hd"], b["kp"], b["vp"])
    if kind == "prompt":
        return kernels.attention_f32_prompt(*head, b["tiles"], b["slot"], b["start"], b["new"], b["cu"], b["table"], scale, window, chunk=chunk)
    f = kernels.attention_generic if kind == "generic" else kernels.attention_f32_token
    return f(*head, b["seq"], b["pos"], b["slot"], b["table"], scale, window, chunk=chunk, **kw)


def exact(b, window=None, chunk=None):
    out, c, G = [], 0, b["nh"] // b["nkv"]
    for k, v, s, n in zip(b["ks"], b["vs"], b["starts"], b["news"]):
        q = b["q"][c:c + n].cpu().double().view(n, b["nh"], b["hd"])
        c += n
        sc = torch.einsum("qhd,khd->hqk", q, k.double().repeat_interleave(G, 1)) * b["hd"] ** -0.5
        i, j = torch.arange(s, s + n)[:, None], torch.arange(s + n)[None]
        low = (i - window + 1).clamp(min=0) if window else (i // chunk * chunk if chunk else i * 0)
        p = sc.masked_fill((j > i) | (j < low), float("-inf")).softmax(-1)
        out.append(torch.einsum("hqk,khd->qhd", p, v.double().repeat_interleave(G, 1)).reshape(n, -1))
    return torch.cat(out).to(DEV)


def close(y, want):
    """Scores of a few units have errors of some 2^-22, and so have the weights they make: 2^-19 of a row's largest value is ample."""
    assert (y.double() - want).abs().max() <= 2.0 ** -19 * want.abs().max()


SHAPES = [dict(), dict(window=65), dict(window=1), dict(chunk=48), dict(window=500)]


@pytest.mark.parametrize("span", SHAPES, ids=str)
@pytest.mark.parametrize("nh,nkv,hd", [(4, 2, 64), (7, 1, 64), (5, 1, 128), (6, 6, 128)])
def test_prompts(nh, nkv, hd, span):
    b = batch([0, 3, 64, 130, 63, 0], [1, 129, 128, 257, 2, 64], nh, nkv, hd, seed=nh)
    y = run(b, "prompt", **span)
    close(y, exact(b, **span))
    close(y, run(b, "generic", **span).double())


@pytest.mark.parametrize("span", SHAPES, ids=str)
@pytest.mark.parametrize("nh,nkv,hd", [(3, 3, 32), (6, 2, 32), (7, 1, 64), (8, 2, 64), (9, 1, 64), (10, 2, 128), (17, 1, 32), (2, 1, 128)])
def test_single_tokens(nh, nkv, hd, span):
    b = batch([0, 1, 7, 63, 64, 65, 1000, 31], [1, 1, 1, 1, 1, 1, 1, 3], nh, nkv, hd, seed=hd)
    want = exact(b, **span)
    for splits in (1, 2, 4, 8):
        close(run(b, "token", splits=splits, **span), want)


@pytest.mark.parametrize("span", [dict(), dict(window=65), dict(chunk=300)], ids=str)
@pytest.mark.parametrize("nh,nkv,hd", [(6, 2, 32), (7, 1, 64), (9, 1, 64), (10, 2, 128)])
def test_a_tokens_sums_do_not_depend_on_the_number_of_ctas(nh, nkv, hd, span):
    """How many CTAs share a token follows the step's size; its sums must not, so every number gives the same bits.  Contexts at the
    edges of the shares: 31 to 1,025 keys."""
    b = batch([0, 30, 31, 63, 64, 127, 128, 255, 256, 511, 700, 1000, 1024], [1] * 13, nh, nkv, hd, seed=hd)
    want = run(b, "token", splits=8, **span)
    for splits in (1, 2, 4):
        assert torch.equal(run(b, "token", splits=splits, **span), want)


@pytest.mark.parametrize("hd", [64, 128, 32])
def test_a_sequences_kernel_does_not_depend_on_the_others(hd):
    """Sequences that bring 1 to 200 tokens in one step and each alone in its own: the same bits, through the mixer's own choice; and
    some tokens of a step by their indices, the others' rows left as they were."""
    from test_parts_gpu import context
    from rocmforge_b200 import kernels
    from rocmforge_b200.cache import SequenceCache
    from rocmforge_b200.parts import MIXERS, POSITIONS
    nh, nkv, lens, starts = 4, 2, [200, 1, 64, 63, 17], [0, 300, 70, 5, 0]
    mixer = MIXERS.build("gqa_attention", hidden=32, n_heads=nh, n_kv_heads=nkv, head_dim=hd, qkv_bias=False,
                         position=POSITIONS.build("rope_neox", head_dim=hd, theta=1e4))
    g = torch.Generator().manual_seed(hd)
    mixer.bind({n: torch.randn(*sp.shape, generator=g).to(DEV) for n, sp in mixer.param_specs().items()}, torch.float32)
    cache = SequenceCache({0: mixer.cache_request()}, max_tokens=2048, dtype=torch.float32, device=DEV)
    slots = [cache.alloc_slot() for _ in lens]
    cache.prepare(slots, [a + b for a, b in zip(starts, lens)])
    view = cache.view(0)
    for pages in (view.k_pages, view.v_pages):
        pages.copy_(torch.randn(pages.shape, generator=g))
    q = torch.randn(sum(lens), nh * hd, generator=g).to(DEV)

    def attend(which):
        ctx = context(torch.float32, [(slots[i], [0] * lens[i], []) for i in which], [starts[i] for i in which], parts=[mixer])
        rows = torch.cat([torch.arange(sum(lens[:i]), sum(lens[:i + 1])) for i in which])
        return mixer.attend(ctx, q[rows.to(DEV)].contiguous(), view), rows
    whole, _ = attend(range(len(lens)))
    assert whole.isfinite().all()
    for i in range(len(lens)):
        o, rows = attend([i])
        assert torch.equal(o, whole[rows.to(DEV)]), lens[i]
    b = batch([0, 9, 100], [3, 1, 2], nh, nkv, hd)
    want, out = run(b, "token"), torch.full((6, nh * hd), 7.0, device=DEV)
    assert run(b, "token", rows=i32([5, 0, 3]), out=out) is out
    assert torch.equal(out[[5, 0, 3]], want[[5, 0, 3]]) and (out[[1, 2, 4]] == 7).all()


def test_no_larger_error_than_the_generic_kernel():
    for kind, b in (("prompt", batch([0, 700], [900, 400], 4, 2, 64)), ("token", batch([900] * 4, [1] * 4, 14, 2, 64)),
                    ("prompt", batch([0], [700], 4, 1, 128)), ("token", batch([500] * 4, [1] * 4, 10, 2, 128))):
        want = exact(b)
        err = [float((run(b, k).double() - want).norm()) for k in (kind, "generic")]
        assert err[0] <= err[1], (kind, err)


def test_large_scores_and_what_is_not_finite():
    """Scores far apart, a value or a key that is infinite or not a number: as the generic kernel."""
    b = batch([0, 40], [200, 100], 4, 2, 64, seed=5)
    b["q"].mul_(30.0)
    for kind in ("prompt", "token"):
        y, want = run(b, kind), run(b, "generic")
        assert (y - want).abs().max() <= 2.0 ** -12 * want.abs().max()          # scores of hundreds: errors of 2^-14 in the exponent
    b = batch([0, 40], [200, 100], 4, 2, 64, seed=6)      # (scores of a few units: no weight is zero, by which an infinite value is NaN)
    page = int(b["table"][1, 1])
    b["vp"][page, 0, 5, 3], b["vp"][page, 1, 6, 0], b["kp"][page, 1, 9, 1] = float("inf"), float("nan"), float("nan")
    b["kp"][int(b["table"][0, 0]), 0, 2, 0] = float("-inf")
    for kind in ("prompt", "token"):
        y, want = run(b, kind), run(b, "generic")
        fine = want.isfinite()
        assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.isinf(), want.isinf())
        assert (y - want).abs()[fine].max() <= 2.0 ** -19 * want.abs()[fine].max()


@pytest.mark.parametrize("kind", ["prompt", "token"])
def test_large_scores_against_64_bits(kind):
    """A score of some hundreds carries an error of 2^-22 of the sum of its 64 products' sizes, of up to a thousand: 2^-12 in the
    exponent, and so in a weight."""
    b = batch([0, 40], [200, 100], 4, 2, 64, seed=5)
    b["q"].mul_(30.0)
    want = exact(b)
    assert (run(b, kind).double() - want).abs().max() <= 2.0 ** -12 * want.abs().max()


def test_whatever_is_not_finite_costs_a_bounded_time():
    """1,999 tokens with a value, or a key, that is infinite or not a number at the first position, so that every row of its kv head
    meets it: the generic kernel's kinds of results in at most eight times its time.  (A warp forms four rows at once and the generic
    kernel a token's seven heads: 4.1 times its time with every row formed again, where one thread a row took 140 times.)"""
    def us(f):
        f()
        a, e = torch.cuda.Event(True), torch.cuda.Event(True)
        a.record()
        for _ in range(3):
            f()
        e.record()
        torch.cuda.synchronize()
        return a.elapsed_time(e) / 3 * 1e3
    for hd, nh, nkv in ((64, 14, 2), (128, 4, 4)):
        for what, value in (("vp", float("inf")), ("vp", float("nan")), ("kp", float("nan")), ("kp", float("inf"))):
            b = batch([0], [1999], nh, nkv, hd, seed=9)
            b["q"].mul_(0.1)
            b[what][int(b["table"][0, 0]), :, 0, 7] = value
            y, want = run(b, "prompt"), run(b, "generic")
            assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.isinf(), want.isinf())
            fine = want.isfinite()
            assert (y - want).abs()[fine].max() <= 2.0 ** -19 * want.abs()[fine].max()
            assert us(lambda: run(b, "prompt")) < 8 * us(lambda: run(b, "generic")), (hd, what, value)


def test_rules():
    from rocmforge_b200 import kernels
    assert kernels.f32_token_splits(1, 1) == 8 and kernels.f32_token_splits(1, 1, longest=100) == 2
    assert kernels.f32_token_splits(300, 2) == 1 and kernels.f32_token_splits(1, 1, 5000, 64) == 2
    for nh, nkv, hd in [(4, 2, 48), (4, 2, 16), (4, 2, 256)]:
        assert not kernels.attention_f32_prompt_supported(nh, nkv, hd) and not kernels.attention_f32_token_supported(nh, nkv, hd)
    b = batch([0], [3], 4, 2, 16)
    for kind in ("prompt", "token"):
        with pytest.raises(kernels.KernelError):
            run(b, kind)
