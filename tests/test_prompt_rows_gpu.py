"""The forms that prompt steps take of the per-head writer, the weighted update, the convolution and the delta rule's inputs: the
same rows in one large step and in small ones, which run the general forms."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DTS = [torch.float32, torch.bfloat16]


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def near(a, b, dt):
    ulp = 2.0 ** -21 if dt == torch.float32 else 2.0 ** -7
    assert torch.equal(a.isnan(), b.isnan())
    # a pair's rotation, or a sum with the stream, may leave little of what it started from: 2^-20 of the largest value beside an ulp
    left = (a.double() - b.double()).abs() - ulp * b.double().abs()
    assert float(left.nan_to_num(0).max()) <= 2.0 ** -20 * float(b.double().abs().nan_to_num(0).max())


@pytest.mark.parametrize("dt", DTS)
@pytest.mark.parametrize("nh,nkv,hd,opts", [
    (6, 2, 64, dict(rot_dim=64, norm_after_rotation=True, unit_norm_eps=1e-6, magnitude=1.2)),
    (5, 1, 128, dict(rot_dim=128, unit_norm_eps=1e-5, weights=True)),
    (3, 3, 256, dict(rot_dim=0, bias=True, q_temperature=(0.1, 64.0), values_are_keys=True)),
    (3, 1, 256, dict(rot_dim=256, unit_norm_eps=1e-6, weights=True)), (2, 1, 256, dict(rot_dim=256, unit_norm_eps=1e-6, norm_after_rotation=True)),
    (2, 2, 128, dict(rot_dim=128, unit_norm_eps=1e-6, norm_after_rotation=True, bias=True)),
    (4, 2, 128, dict(rot_dim=0)), (4, 2, 64, dict(rot_dim=32, unit_norm_eps=1e-6)), (4, 4, 128, dict(rot_dim=128, writes=False))])
def test_head_rows(dt, nh, nkv, hd, opts):
    from rocmforge_b200 import kernels
    torch.manual_seed(hd + nh)
    opts = dict(opts)
    T, vk, writes = 1300, opts.get("values_are_keys", False), opts.pop("writes", True)
    width = (nh + (0 if not writes else (1 if vk else 2) * nkv)) * hd
    src = torch.randn(T, width + 16, device=DEV).to(dt)
    rot = opts["rot_dim"]
    inv = (1e4 ** (-torch.arange(rot // 2, device=DEV).float() / max(rot // 2, 1))) if rot else None
    if opts.pop("weights", False):
        opts.update(q_norm_weight=torch.rand(hd, device=DEV) + 0.5, k_norm_weight=torch.rand(hd, device=DEV) + 0.5)
    if opts.pop("bias", False):
        opts["bias"] = torch.randn(width, device=DEV)
    seq = i32([0] * 700 + [1] * 600)
    pos = i32(list(range(3, 703)) + list(range(600)))
    table = i32(list(range(24))).view(2, 12)

    def run(cuts):
        kp, vp = (torch.full((24, nkv, 64, hd), float("nan"), device=DEV).to(dt) for _ in range(2))
        vp = kp if vk else vp
        q = []
        for a, b in zip(cuts, cuts[1:]):
            q.append(kernels.head_norm_kv_write(src[a:b, :width], nh, nkv, hd, hd, inv, seq[a:b], pos[a:b], i32([0, 1]), table, kp, vp, writes,
                                                compute_dtype=dt, **opts)[:, :nh * hd].clone())
        return torch.cat(q), kp, vp
    keep = src.clone()
    big = run([0, 1300])
    src.copy_(keep)
    small = run(list(range(0, 1300, 100)) + [1300])
    src.copy_(keep)
    middle = run([0, 256, 1300])
    for a, b, c in zip(big, small, middle):
        near(a, b, dt), near(c, b, dt)
        # a head's sums are added in the same order whatever the form, so not a bit differs
        for p, q in ((a, b), (c, b)):
            assert torch.equal(p.isnan(), q.isnan()) and torch.equal(p.nan_to_num(0), q.nan_to_num(0))


@pytest.mark.parametrize("dt", DTS)
@pytest.mark.parametrize("H", [4, 1000, 1024, 2048, 4096, 5000, 8192])
@pytest.mark.parametrize("two", [False, True])
def test_weighted_update(dt, H, two):
    from rocmforge_b200 import kernels
    torch.manual_seed(H)
    T = 601
    h, a, b = (torch.randn(T, H, device=DEV) for _ in range(3))
    w = torch.rand(H, device=DEV) + 0.5
    want = h.double() + 0.7 * a.double() + (0.3 * b.double() if two else 0)
    for nxt in (None, (w, 1e-6), (w.bfloat16(), 1e-6)):
        got = h.clone()
        y = kernels.weighted_add(got, [(a, 0.7)] + ([(b, 0.3)] if two else []), dt, next_norm=nxt)
        near(got, want, torch.float32)
        if nxt is not None:
            ref = want / torch.sqrt((want * want).mean(-1, keepdim=True) + 1e-6) * nxt[0].double()
            near(y, ref, dt)


@pytest.mark.parametrize("dt", DTS)
@pytest.mark.parametrize("H", [4, 252, 1000, 1028, 2048, 2052, 4096, 4100, 8192])
@pytest.mark.parametrize("two", [False, True])
def test_the_weighted_update_of_many_rows_has_the_bits_of_fewer(dt, H, two):
    """The same rows in a step of 512 and more and in one of fewer (297 to 511, which run the form of 256 threads a row); 517 rows
    leave the last block with one."""
    from rocmforge_b200 import kernels
    torch.manual_seed(H)
    T = 517
    h, a, b = (torch.randn(T, H, device=DEV) for _ in range(3))
    h[7] *= 1e4
    w = torch.rand(H, device=DEV) + 0.5
    for nxt in (None, (w, 1e-6), (w.bfloat16(), 1e-6)):
        def run(rows):
            got = h[rows].clone()
            return got, kernels.weighted_add(got, [(a[rows].clone(), 0.7)] + ([(b[rows].clone(), 0.3)] if two else []), dt, next_norm=nxt)
        big, fewer, rest = run(slice(0, T)), run(slice(0, 300)), run(slice(T - 299, T))
        for x, y, z in zip(big, fewer, rest):
            assert x is None or (torch.equal(x[:300], y) and torch.equal(x[T - 299:], z))


@pytest.mark.parametrize("dt", DTS)
@pytest.mark.parametrize("C,taps", [(260, 4), (64, 2), (1028, 3), (8, 1)])
def test_convolution(dt, C, taps):
    from rocmforge_b200 import kernels
    torch.manual_seed(C)
    lens = [1, 700, 2, 3, 9, 500]
    T = sum(lens)
    src = torch.randn(T, C + 12, device=DEV).to(dt)
    w, bias = torch.randn(C, taps, device=DEV), torch.randn(C, device=DEV)
    state = torch.randn(8, taps - 1, C, device=DEV)
    starts = [sum(lens[:i]) for i in range(len(lens))]

    def run(steps, st):
        at, out = list(starts), torch.empty(T, C, device=DEV)
        for ns in steps:
            live = [i for i, n in enumerate(ns) if n]
            rows = torch.cat([torch.arange(at[i], at[i] + ns[i]) for i in live]).to(DEV)
            cu = [0]
            for i in live:
                cu.append(cu[-1] + ns[i])
            x = torch.empty(cu[-1], C + 12, device=DEV, dtype=dt).copy_(src[rows])
            out[rows] = kernels.conv_silu(x, 4, C, st, w, bias, i32([j for j, i in enumerate(live) for _ in range(ns[i])]), i32(cu), i32([i + 1 for i in live]))
            for i in live:
                at[i] += ns[i]
        return out
    s1, s2 = state.clone(), state.clone()
    small = [[min(10, max(0, n - k)) for n in lens] for k in range(0, max(lens), 10)]
    a, b = run([lens], s1), run([s for s in small if any(s)], s2)
    assert torch.equal(a, b) and torch.equal(s1, s2)          # the taps are added in the same order


@pytest.mark.parametrize("dt", DTS)
@pytest.mark.parametrize("H,G,D,per_head", [(4, 2, 128, False), (3, 3, 36, False), (2, 1, 64, True), (1, 1, 4, False), (2, 2, 32, False), (2, 1, 100, True)])
def test_delta_inputs(dt, H, G, D, per_head):
    from rocmforge_b200 import kernels
    torch.manual_seed(D)
    T, nd = 650, H if per_head else H * D
    qkv, a = torch.randn(T, 2 * G * D + 8, device=DEV), torch.randn(T, nd + (4 - nd % 4) % 4, device=DEV) * 3
    bsrc, dtb, al = torch.randn(T, H, device=DEV).to(dt), torch.randn(nd, device=DEV), torch.randn(H, device=DEV)
    f = lambda r: kernels.delta_prepare(qkv[r], a[r][:, :nd], dtb, al, bsrc[r], H, G, D, 0.3, 1e-6)
    big, small = f(slice(0, T)), [f(slice(k, min(k + 100, T))) for k in range(0, T, 100)]
    for i, x in enumerate(big):
        assert torch.equal(x, torch.cat([s[i] for s in small]))       # the same sums in the same order
