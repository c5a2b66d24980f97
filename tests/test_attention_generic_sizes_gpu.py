"""The general attention kernel in 32 bits: the instances for key rows that start on 16 bytes and for few CTAs, and the others."""
import math

import pytest
import torch

from tests.test_kernels_gpu import DEV, F32, attention_case, rel_err

pytestmark = pytest.mark.gpu


# the smallest and largest heads of every instance, with rows of whole 16 bytes and without
@pytest.mark.parametrize("hd", [1, 4, 62, 63, 64, 65, 68, 127, 128, 129, 132, 255, 256, 257, 260, 639, 640, 641, 644, 1151, 1152])
@pytest.mark.parametrize("qlens", [[10, 1, 1, 1], [130, 1, 65, 30]])       # 52 CTAs, which fit the device at two an SM, and 904
def test_heads_of_every_instance(hd, qlens):
    from gguf_rs_cli_b200 import kernels
    nh, nkv = 4, 2
    lens = [130, 1, 65, 300]
    q, seq_of, pos, table, kc, vc, want = attention_case(nh, nkv, hd, lens, qlens, F32, seed=hd)
    out = torch.empty(q.shape[0], nh * hd, device=DEV)
    kernels.attention_generic(q, out, nh, nkv, hd, seq_of, pos, table, 1 << 20, kc, vc, 0, 1 / math.sqrt(hd))
    # scores of deviation 1 whose sums of hd terms err by at most hd 2^-24 of their terms' sizes: the bound of the other sizes
    assert rel_err(out, want) < 2e-5


@pytest.mark.parametrize("hd", [64, 100, 192, 320])
@pytest.mark.parametrize("qlens", [[10, 1, 1, 1], [130, 1, 65, 30]])
def test_keys_that_start_on_4_bytes_give_the_same_bits(hd, qlens):
    """A cache that starts between two 16-byte boundaries takes the other instance for many CTAs, and the same one's other loads for few: same
    sums, same order."""
    from gguf_rs_cli_b200 import kernels
    nh, nkv = 4, 2
    q, seq_of, pos, table, kc, vc, _ = attention_case(nh, nkv, hd, [130, 1, 65, 300], qlens, F32, seed=hd)
    flat = torch.empty(kc.numel() + 4, device=DEV)
    outs = []
    for off in (0, 1):
        k = flat[off:off + kc.numel()].view_as(kc)
        k.copy_(kc)
        outs.append(torch.empty(q.shape[0], nh * hd, device=DEV))
        kernels.attention_generic(q, outs[-1], nh, nkv, hd, seq_of, pos, table, 1 << 20, k, vc, 0, 1 / math.sqrt(hd))
    assert torch.equal(*outs)
