"""Residual products with the dynamic tanh behind them in their epilogue: the bits of the product and of the tanh's own kernel."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# shared tiles with few and many CTAs, tiles of a CTA's own (gate-sized N, one block of K), edges of 128 features, rows that take no
# accesses of four values
@pytest.mark.parametrize("N, K, pitch", [(2048, 2048, 2048), (2048, 8192, 2052), (256, 64, 256), (20000, 128, 20000), (130, 512, 130), (1030, 1024, 1031)])
@pytest.mark.parametrize("T", [1, 4, 16, 17, 33, 64, 65, 128])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_tanh_in_the_residual_epilogue(N, K, pitch, T, dtype):
    from gguf_rs_cli_b200 import kernels as k
    g = torch.Generator(device=DEV).manual_seed(N + K + T)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)
    x, w, bias = r(T, K).bfloat16(), (r(N, K) / math.sqrt(K)).bfloat16(), r(N)
    weight, shift, start = (1 + 0.1 * r(N)).to(dtype), r(N).to(dtype), r(T, N)
    padded = lambda t, d: torch.full((T, pitch), 7.0, device=DEV, dtype=d)[:, :N].copy_(t)
    for scale, b in ((1.0, None), (0.5, bias)):
        plain, xb, ssq = padded(start, torch.float32), padded(start, torch.bfloat16), torch.empty((N + 127) // 128, T, device=DEV)
        k.gemm_tc(x, w, b, None, resid_x=plain, resid_xb=xb, ssq_out=ssq, resid_scale=scale)
        want = torch.empty(T, N, device=DEV, dtype=torch.bfloat16)
        k.add_dyt(plain.contiguous(), None, weight, shift, 0.7, want)
        got, rows = padded(start, torch.float32), padded(start, torch.bfloat16)
        k.gemm_tc_dyt(x, w, b, got, rows, weight, shift, 0.7, resid_scale=scale)
        assert torch.equal(got, plain), float((got - plain).abs().max())
        assert torch.equal(rows, want), (rows != want).nonzero()[:4].tolist()
        assert (got._base[:, N:] == 7.0).all() and (rows._base[:, N:] == 7.0).all()
    torch.cuda.synchronize()
    k.check_tc_status()
