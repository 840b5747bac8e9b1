"""The true 32-bit product on the tensor cores (csrc/gemm_f32_tc.cuh) at the edges of its tiles, against 64 bits and against the
CUDA-core kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def operands(M, N, K, seed=0, pad=0):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(M, K + pad, generator=g).to(DEV)[:, :K]
    return x, (torch.randn(N, K, generator=g) * 0.1).to(DEV)


def bound(x, w, splits=1):
    """Rounding of the parts that are left out (2^-22 of each product), of a stage's sums in the tensor cores (12 of them, an ulp
    each at most) and of one addition per stage of 32 and per split, all relative to the sum of the products' sizes.  Beside it what
    the number formats cannot hold: a part ends at 2^-133, bfloat16's smallest number, so each operand may miss 2^-133 (numbers below
    2^-110 lose their last bits); a product or sum may lose what lies below 2^-126 where the tensor cores take such results for zero,
    twelve times a stage."""
    K = w.shape[1]
    X, W = x.abs().double(), w.abs().double()
    tiny = 2.0 ** -133 * (X.sum(1)[:, None] + W.sum(1)[None]) + 12 * ((K + 31) // 32) * 2.0 ** -126
    return (X @ W.t()) * (2.0 ** -22 + (12 + (K + 31) // 32 + splits) * 2.0 ** -24) + tiny


@pytest.mark.parametrize("M", [1, 16, 17, 33, 64, 65, 128, 129, 300])
@pytest.mark.parametrize("N,K", [(1, 4), (127, 32), (130, 36), (256, 896), (384, 100), (896, 260)])
def test_store_add_partial_swiglu(M, N, K):
    from rocmforge_b200 import kernels
    from rocmforge_b200.kernels import basic
    x, w = operands(M, N, K, pad=8)
    ref, most = x.double() @ w.double().t(), bound(x, w)
    assert kernels.f32_tc_takes(x, w) == (K >= 20)
    y = kernels.gemm_f32_tc(x, w)
    assert ((y.double() - ref).abs() <= most).all()
    bias = torch.randn(N, device=DEV)
    assert ((kernels.gemm_f32_tc(x, w, bias).double() - ref - bias.double()).abs() <= most + 2.0 ** -23 * (ref.abs() + bias.abs())).all()
    acc = torch.randn(M, N + 3, device=DEV)
    before = acc.clone()
    kernels.gemm_f32_tc(x, w, bias.bfloat16(), mode=basic.F32_ADD, out=acc[:, :N])
    want = before[:, :N].double() + ref + bias.bfloat16().double()
    assert ((acc[:, :N].double() - want).abs() <= most + 2.0 ** -22 * (ref.abs() + bias.abs() + before[:, :N].abs())).all()
    assert torch.equal(acc[:, N:], before[:, N:])
    for splits in {1, 2, (K + 31) // 32}:
        kb = (K + 31) // 32
        if (splits - 1) * ((kb + splits - 1) // splits) >= kb:
            continue
        parts = kernels.gemm_f32_tc(x, w, mode=basic.F32_PARTIAL, splits=splits)
        assert ((parts.double().sum(0) - ref).abs() <= bound(x, w, splits)).all()
    if N % 2 == 0:
        a = kernels.gemm_f32_tc(x, w, mode=basic.F32_SWIGLU)
        assert torch.allclose(a, kernels.swiglu(y), rtol=1e-6, atol=1e-6 * float(y.abs().max()))
    # the same bits whatever tile the row lies in and whatever rows are beside it
    for bn in (16, 32, 64, 128):
        assert torch.equal(kernels.gemm_f32_tc(x, w, tile_tokens=bn), y), bn
    assert torch.equal(kernels.gemm_f32_tc(x[M - 1:], w)[0], y[M - 1])
    assert torch.equal(kernels.gemm_plain(x, w), y if K >= 20 else kernels.gemm_simt(x, w))


@pytest.mark.parametrize("K", [4, 8, 12, 16, 20, 24, 32, 36, 64, 100, 896, 3584, 4864])
def test_no_larger_error_than_the_cuda_cores(K):
    """Of whatever kernel the route takes, over a few thousand results of each of three draws."""
    from rocmforge_b200 import kernels
    for M, N, seed in [(64, 896, 1), (40, 1152, 2), (200, 640, 3)]:
        x, w = operands(M, N, K, seed=seed)
        ref = x.double() @ w.double().t()
        err = [float((k(x, w).double() - ref).norm() / ref.norm()) for k in (kernels.gemm_plain, kernels.gemm_simt)]
        assert err[0] <= err[1], (M, N, K, err)


def test_extreme_and_infinite_numbers():
    """The largest and smallest numbers, infinities and NaN give what the CUDA-core kernel gives for them."""
    from rocmforge_b200 import kernels
    from rocmforge_b200.kernels import basic
    x, w = operands(70, 200, 96, seed=3)
    big = 3.4028234e38
    x[0], w[0] = 0.0, 0.0
    x[0, 5], w[0, 5] = big, 1.0                  # the largest number, by one
    x[1, 7], x[2, 8], x[3, 9], x[69, 95] = float("inf"), float("-inf"), float("nan"), float("inf")
    w[5, 0], w[199, 95], w[7, 7] = float("inf"), float("-inf"), 0.0
    x[4] = 1e-38                                 # products below the smallest normal number
    x[6] = torch.randn(96, device=DEV) * 2.0 ** -100
    a, b = kernels.gemm_f32_tc(x, w), kernels.gemm_simt(x, w)
    assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf())
    assert torch.equal(a[a.isinf()], b[b.isinf()]) and float(a[0, 0]) == float(b[0, 0])
    fine = a.isfinite()
    fine[0] = False
    x64, w64 = (torch.nan_to_num(t, 0, 0, 0).double() for t in (x, w))
    assert ((a.double() - x64 @ w64.t()).abs()[fine] <= bound(x64, w64)[fine]).all()
    acc = torch.ones(70, 200, device=DEV)
    kernels.gemm_f32_tc(x, w, mode=basic.F32_ADD, out=acc)
    assert torch.equal(acc.isnan(), b.isnan()) and torch.equal(acc.isinf(), b.isinf())
    p = kernels.gemm_f32_tc(x, w, mode=basic.F32_PARTIAL, splits=3).sum(0)
    assert torch.equal(p.isfinite(), b.isfinite())
    s, t = kernels.gemm_f32_tc(x, w, mode=basic.F32_SWIGLU), kernels.swiglu(b)
    assert torch.equal(s.isnan(), t.isnan()) and torch.equal(s.isinf(), t.isinf())


def test_what_the_route_leaves_to_the_cuda_cores():
    from rocmforge_b200 import kernels
    for M, N, K, pad in [(5, 7, 6, 0), (5, 7, 9, 3), (5, 9, 8, 2)]:
        x, w = operands(M, N, K, pad=pad)
        assert not kernels.f32_tc_takes(x, w)
        assert torch.equal(kernels.gemm_plain(x, w), kernels.gemm_simt(x, w))
    x, w = operands(5, 9, 8)
    shifted = torch.zeros(41, device=DEV)[1:].view(5, 8)
    assert not kernels.f32_tc_takes(shifted, w) and not kernels.f32_tc_takes(x.bfloat16(), w.bfloat16())
    assert kernels.gemm_plain(x[:0], w).shape == (0, 9)
    for bad in [dict(x=x, w=w[:, :4]), dict(x=x.double(), w=w.double()), dict(x=x.cpu(), w=w)]:
        with pytest.raises(kernels.KernelError):
            kernels.gemm_plain(bad["x"], bad["w"])


def us(f, n=5):
    f()
    a, b = torch.cuda.Event(True), torch.cuda.Event(True)
    a.record()
    for _ in range(n):
        f()
    b.record()
    torch.cuda.synchronize()
    return a.elapsed_time(b) / n * 1e3


@pytest.mark.parametrize("M,N,K,mode", [(1999, 896, 4864, "store"), (300, 512, 896, "swiglu"), (64, 512, 896, "partial"), (140, 130, 132, "add")])
def test_whatever_is_not_finite_costs_a_bounded_time(M, N, K, mode):
    """A NaN, an infinity or a sum that overflows in one token and in every token: the CUDA-core kernel's kinds of results, the other
    tokens' bits as they were, no status, and no more than sixteen times the CUDA-core kernel's time (it reads both operands once
    for 128 x 128 results; here a result reads its two rows, 128 numbers at a time)."""
    from rocmforge_b200 import kernels
    from rocmforge_b200.kernels import basic, tensor_core
    kw = dict(store={}, swiglu=dict(mode=basic.F32_SWIGLU), partial=dict(mode=basic.F32_PARTIAL, splits=4), add=dict(mode=basic.F32_ADD))[mode]

    def call(x, w):
        if mode != "add":
            return kernels.gemm_f32_tc(x, w, **kw)
        return kernels.gemm_f32_tc(x, w, out=torch.ones(M, N, device=DEV), **kw)

    def plain(x, w):
        y = kernels.gemm_simt(x, w)
        return kernels.swiglu(y) if mode == "swiglu" else y
    x, w = operands(M, N, K, seed=1)
    fine = call(x, w)
    limit = 16 * us(lambda: plain(x, w)) + 200
    for kind, value in (("nan", float("nan")), ("inf", float("inf")), ("overflow", 3e38)):
        for rows in ([M // 2], range(M)):
            y = x.clone()
            rows = torch.tensor(list(rows), device=DEV)
            y[rows, (rows * 7) % K] = value
            if kind == "overflow":
                y[rows] = y[rows].sign() * value
            got, want = call(y, w), plain(y, w)
            flat = got.sum(0) if mode == "partial" else got
            if kind != "overflow":                  # (where a sum overflows follows its order)
                assert torch.equal(flat.isnan(), want.isnan()) and torch.equal(flat.isinf(), want.isinf()) and not want[rows].isfinite().any()
                assert torch.equal(flat[flat.isinf()], want[want.isinf()])
            if len(rows) == 1:
                keep = [i for i in range(M) if i != M // 2]
                assert torch.equal(got[..., keep, :], fine[..., keep, :])
            assert us(lambda: call(y, w)) < limit, (kind, len(rows))
    assert int(tensor_core.status_word(torch.device(DEV))[0]) == 0
