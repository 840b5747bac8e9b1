"""Clustered products whose activations go in several bands of row groups (beyond a quarter of L2): every tile once, the same bits as
the same rows in products of one band."""
import pytest
import torch

from rocmforge_b200 import kernels

pytestmark = pytest.mark.gpu
tc = kernels.tensor_core


@pytest.mark.parametrize("M,N,K,mode,parts", [
    (8200, 384, 4096, tc.STORE, 0), (16640, 300, 2048, tc.F32, 0), (9000, 512, 4096, tc.SWIGLU, 0), (8321, 896, 4864, tc.RESIDUAL, 1),
    (8321, 896, 9728, tc.RESIDUAL, 2),                     # two K parts of several bands each
    (70000, 256, 520, tc.STORE, 0)])
@pytest.mark.parametrize("cluster,pair", [(2, True), (2, False), (4, True)])
def test_bands(M, N, K, mode, parts, cluster, pair):
    g = torch.Generator("cuda").manual_seed(M + N + K)
    x = torch.randn((M, K), generator=g, device="cuda").bfloat16()
    w = (torch.randn((N, K), generator=g, device="cuda") * K ** -0.5).bfloat16()
    assert M * K // max(parts, 1) * 2 > torch.cuda.get_device_properties(0).L2_cache_size // 4
    h = torch.randn((M, N), generator=g, device="cuda") if mode == tc.RESIDUAL else None
    was = tc.cluster_pair()
    tc.set_cluster_pair(pair)
    try:
        run = lambda a, out: tc.gemm_tc(a, w, mode=mode, cluster=cluster, parts=parts, **({} if out is None else dict(out=out)))
        want = torch.cat([run(x[i:i + 2048], None if h is None else h[i:i + 2048].clone()) for i in range(0, M, 2048)])
        got = run(x, None if h is None else h.clone())
    finally:
        tc.set_cluster_pair(was)
    bits = lambda t: t.view(torch.int32 if t.dtype == torch.float32 else torch.int16)
    assert torch.equal(bits(got), bits(want))
    tc.check_status(torch.device("cuda:0"))
