"""Products of few tokens whose weight has fewer tiles of 128 rows than the GPU has SMs go in tiles of 64 rows, gated and bfloat16 ones
with eight epilogue warps: the same sums as in tiles of 128, bit for bit, and right against 64 bits."""
import pytest
import torch

from rocmforge_b200 import kernels
from rocmforge_b200.kernels._ffi import sm_count

pytestmark = pytest.mark.gpu
DEV = "cuda"
tc = kernels.tensor_core

UNITS = {tc.SWIGLU: lambda g, u: torch.nn.functional.silu(g) * u, tc.REGLU: lambda g, u: g.relu() * u,
         tc.GEGLU: lambda g, u: torch.nn.functional.gelu(g, approximate="tanh") * u,
         tc.CLAMPGLU: lambda g, u: g.clamp(max=1.5) * torch.sigmoid(1.702 * g.clamp(max=1.5)) * (u.clamp(-1.5, 1.5) + 1)}


@pytest.mark.parametrize("mode", [tc.STORE, tc.F32, tc.SWIGLU, tc.REGLU, tc.GEGLU, tc.CLAMPGLU])
@pytest.mark.parametrize("M,N,K", [
    (1, 64, 64), (16, 130, 72), (16, 2048, 1536),                                  # the ring once, and more often than once, around
    (17, 62, 896), (32, 320, 1000), (33, 9728, 896), (64, 1000, 64), (65, 66, 128), (128, 2112, 520),
    (8, 148 * 128, 64), (8, 148 * 128 + 2, 64), (128, 148 * 128, 72)])             # the last tiles of 64, the first of 128
def test_tiles_of_64_rows(M, N, K, mode):
    g = torch.Generator(DEV).manual_seed(M + N + K + mode)
    x = torch.randn((M, K), generator=g, device=DEV).bfloat16()
    w = (torch.randn((N, K), generator=g, device=DEV) * K ** -0.5).bfloat16()
    extra = dict(limit=1.5, alpha=1.702) if mode == tc.CLAMPGLU else {}
    got = tc.gemm_tc_skinny(x, w, mode=mode, **extra)
    many = torch.zeros((sm_count() * 128 + 256 + N, K), dtype=torch.bfloat16, device=DEV)
    many[:N] = w                                                                   # the same rows in a weight of many tiles
    cols = N // 2 if mode in tc.GATED else N
    want = tc.gemm_tc_skinny(x, many, mode=mode, **extra)[:, :cols].contiguous()
    assert torch.equal(got.view(torch.int32 if mode == tc.F32 else torch.int16), want.view(torch.int32 if mode == tc.F32 else torch.int16))
    ref = x.double() @ w.double().T
    if mode in UNITS:
        ref = UNITS[mode](ref[:, ::2], ref[:, 1::2])
    # sums of K products of numbers of size 1 and K^-1/2 in 32 bits: K 2^-24 of them at most; bfloat16 results are rounded by 2^-9
    torch.testing.assert_close(got.double(), ref, atol=2e-5 + K * 2.0 ** -24, rtol=2e-5 if mode == tc.F32 else 2.0 ** -8)


@pytest.mark.parametrize("mode", [tc.STORE, tc.SWIGLU, tc.GEGLU])
@pytest.mark.parametrize("M,N,K", [
    (64, 320, 1024), (65, 320, 896), (73, 320, 896), (74, 320, 896),               # around the last rows that end below 128 KB
    (17, 320, 896), (32, 148 * 128 + 130, 128), (33, 148 * 128 + 2, 136), (65, 148 * 128 + 2, 136)])
def test_form_for_one_kind_of_output(M, N, K, mode):
    g = torch.Generator(DEV).manual_seed(M + N + K + mode)
    x = torch.randn((M, K), generator=g, device=DEV).bfloat16()
    w = (torch.randn((N, K), generator=g, device=DEV) * K ** -0.5).bfloat16()
    got = tc.gemm_tc_skinny(x, w, mode=mode)
    sums = tc.gemm_tc_skinny(x, w, mode=tc.F32)                                    # the general form
    if mode == tc.STORE:
        assert torch.equal(got.view(torch.int16), sums.bfloat16().view(torch.int16))
    else:
        # the same sums: only the unit's own arithmetic (a few 2^-24) lies between, so at most bfloat16's rounding (2^-9) differs
        want = UNITS[mode](sums[:, ::2].double(), sums[:, 1::2].double())
        torch.testing.assert_close(got.double(), want, atol=1e-6, rtol=2.0 ** -8)


@pytest.mark.parametrize("M", [8, 32, 64, 100])
def test_bias_and_numbers_that_are_not_finite(M):
    g = torch.Generator(DEV).manual_seed(M)
    x, w = torch.randn((M, 256), generator=g, device=DEV).bfloat16(), torch.randn((200, 256), generator=g, device=DEV).bfloat16()
    b = torch.randn((200,), generator=g, device=DEV)
    x[M // 2, 3], x[0, 7] = float("inf"), float("nan")
    got = tc.gemm_tc_skinny(x, w, b, mode=tc.STORE)
    assert got[0].isnan().all() and not got[M // 2].isfinite().any()
    rows = [i for i in range(M) if i not in (0, M // 2)]
    ref = x[rows].double() @ w.double().T + b.double()
    torch.testing.assert_close(got[rows].double(), ref, atol=1e-3, rtol=2.0 ** -8)
