"""The tensor-core decode kernels in every shape of a CTA that the library takes by itself, with sequences of unequal
lengths, so that some are shared by several CTAs and others are not."""
import math

import pytest
import torch


def test_sharing_is_fixed_within_a_graph_class():
    """Like the number of splits: a captured graph of a class of lengths holds the grid, so the rule may look at the class only."""
    from gguf_rs_cli_b200 import kernels
    sms = 148
    for heads, kv, hd in ((32, 8, 128), (40, 40, 128), (32, 8, 64), (32, 1, 128)):
        for T in (1, 4, 8, 16, 32, 64, 200):
            seen = {}
            for max_kv in list(range(1, 3000, 7)) + list(range(3000, 140000, 997)):
                got = kernels.decode_sharing(T, heads, kv, hd, max_kv, sms)
                assert seen.setdefault(kernels.decode_split_class(max_kv), got) == got
                assert got[0] >= 1 and got[1] >= 1
                assert T * kv * (1 + (heads // kv > 16)) > sms or got == (kernels.decode_splits(T, heads, kv, max_kv, sms, True), 1)


# (heads, KV heads, head size, sequences, padding tokens): up to one CTA an SM, two, three, four, more; short sequences and long ones
SHAPES = [(40, 40, 128, 3, 0), (40, 40, 128, 6, 1), (40, 40, 128, 6, 4), (24, 8, 128, 57, 3), (40, 40, 128, 15, 1),
          (32, 8, 64, 20, 2), (40, 40, 64, 9, 0)]


@pytest.mark.gpu
@pytest.mark.parametrize("nh,nkv,hd,n,pad", SHAPES)
@pytest.mark.parametrize("longest", [449, 2050])
@pytest.mark.parametrize("window", [0, 700])
def test_attention_decode_shapes(nh, nkv, hd, n, pad, longest, window):
    from gguf_rs_cli_b200 import kernels as k
    from tests.test_kernels_gpu import BF, DEV, attention_case, rel_err
    lens = [longest] + [(1, 63, 64, 65, 310, longest - 1, 16, longest // 2)[i % 8] for i in range(n - 1)]
    q, seq_of, pos, table, kc, vc, want = attention_case(nh, nkv, hd, lens, [1] * n, BF, nh + hd + n, window=window or None)
    T = n + pad
    rows = list(range(n // 2)) + list(range(n // 2 + pad, T))            # padding tokens between the others
    qp = torch.randn(T, nh * hd, device=DEV).to(BF)
    sp = torch.full((T,), -1, dtype=torch.int32, device=DEV)
    pp = torch.full((T,), 9000, dtype=torch.int32, device=DEV)           # what a padding token's position says is not looked at
    qp[rows], sp[rows], pp[rows] = q, seq_of, pos
    got = []
    for _ in range(2):
        out = torch.full((T, nh * hd), float("nan"), dtype=BF, device=DEV)
        k.attention_decode(qp, out, nh, nkv, hd, sp, pp, table, 1 << 20, kc, vc, window, 1 / math.sqrt(hd), mma=True, max_kv=longest)
        got.append(out)
    # weights rounded to 8 bits before the product with the values, the result to 8 bits: 2^-9 each, per entry
    assert rel_err(got[0][rows], want) < 1e-2
    assert torch.equal(got[0], got[1])                                    # counters are back at zero, the order of the merge is fixed
    assert pad == 0 or not got[0][n // 2:n // 2 + pad].any()
