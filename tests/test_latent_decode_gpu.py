"""Latent attention of single tokens, the two kernels and their merge, against 64-bit sums."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
# heads, kv_rank, rot_dim: tensor cores (32, 16, 8 and 32 lanes a row), then CUDA cores
SIZES = [(16, 512, 64), (5, 64, 16), (2, 64, 0), (8, 128, 32), (3, 40, 24)]


def _step(lens, H, C, R, seed=0):
    """A step of one token per sequence: queries, cache pages in any order, and what the kernels read of a context."""
    from gguf_rs_cli_b200.parts.base import Workspace
    g = torch.Generator(device=DEV).manual_seed(seed)
    T, width = len(lens), (max(lens) + 63) // 64
    q = torch.randn(T, H * (C + R), generator=g, device=DEV).bfloat16()
    cache = torch.randn(T * width, 1, 64, C + R, generator=g, device=DEV).bfloat16()
    table = torch.randperm(T * width, generator=g, device=DEV).int().view(T, width)
    ctx = SimpleNamespace(max_kv=max(lens), ws=Workspace(DEV), seq_of=torch.arange(T, device=DEV, dtype=torch.int32),
                          pos=torch.tensor([n - 1 for n in lens], device=DEV, dtype=torch.int32))
    return q, cache, table, ctx


def _plain(q, cache, table, lens, H, C, R, scale, window=0):
    out = []
    for t, n in enumerate(lens):
        rows = cache[table[t].long()].reshape(-1, C + R)[:n].double()
        s = q[t].double().view(H, C + R) @ rows.T * scale
        if window:
            s[:, :max(0, n - window)] = -torch.inf
        out.append((torch.softmax(s, -1) @ rows[:, :C]).flatten())
    return torch.stack(out)


def _check(got, want):
    """Half a unit in the last place of bfloat16 is 2^-9 of a value; sums of a few thousand 32-bit terms are far below the other half."""
    assert ((got.double() - want).abs() <= 2 ** -8 * want.abs().amax(1, keepdim=True)).all()


@pytest.mark.parametrize("H, C, R", SIZES)
@pytest.mark.parametrize("lens", [[1], [1, 1000, 33, 64, 740], [32, 65, 2], [736] * 4, [300] * 40])
def test_unequal_lengths_in_one_step(H, C, R, lens):
    """Splits follow the longest sequence: a short one leaves most of its splits without keys."""
    from gguf_rs_cli_b200 import kernels
    q, cache, table, ctx = _step(lens, H, C, R)
    scale = (C + R) ** -0.5
    for window in (0, 45):
        out = torch.full((len(lens), H * C), 7.0, device=DEV, dtype=torch.bfloat16)
        kernels.latent_decode(q, out, H, C, R, ctx, table, table.shape[1], cache, scale, window=window)
        _check(out, _plain(q, cache, table, lens, H, C, R, scale, window))


@pytest.mark.parametrize("H, C, R", SIZES)
@pytest.mark.parametrize("splits", [1, 2, 7, 8, 9, 63, 64, 65, 128, 129, 300])
def test_any_number_of_splits(H, C, R, splits):
    """The merge holds 64 splits' factors at a time, up to 8 in registers; the entry takes as many as a grid has rows."""
    from gguf_rs_cli_b200 import native
    from gguf_rs_cli_b200.native import call, ptr, stream_ptr
    lens = [4500, 70, 1]
    q, cache, table, ctx = _step(lens, H, C, R, seed=splits)
    g = torch.Generator(device=DEV).manual_seed(splits)
    sink, gate = torch.randn(H, generator=g, device=DEV), torch.randn(3, H, generator=g, device=DEV).bfloat16()
    scale = (C + R) ** -0.5
    scratch = torch.full((native.library().gb_latent_decode_scratch_floats(3, H, C, splits),), torch.nan, device=DEV)
    out = torch.full((3, H * C), 7.0, device=DEV, dtype=torch.bfloat16)
    call("gb_latent_decode", ptr(q), q.stride(0), ptr(out), out.stride(0), 3, H, C, R, ptr(ctx.seq_of), ptr(ctx.pos), ptr(table),
         table.shape[1], table.shape[1], ptr(cache), float(scale), splits, ptr(scratch), 0, ptr(sink), ptr(gate), gate.stride(0), stream_ptr())
    want = []
    for t, n in enumerate(lens):
        rows = cache[table[t].long()].reshape(-1, C + R)[:n].double()
        s = torch.cat([q[t].double().view(H, C + R) @ rows.T * scale, sink.double()[:, None]], 1)
        want.append(((torch.softmax(s, -1)[:, :-1] @ rows[:, :C]) * torch.sigmoid(gate[t].double())[:, None]).flatten())
    _check(out, torch.stack(want))


@pytest.mark.parametrize("H, C, R", SIZES)
def test_a_nan_is_not_lost_behind_larger_scores(H, C, R):
    """The first 32 keys' scores are 200 below the others', so that their split's factor e^-200 is 0 in 32 bits; a NaN in one of
    those rows has to reach the result as it does in one pass over all keys."""
    from gguf_rs_cli_b200 import kernels
    lens = [256, 256]                                 # eight blocks of keys, eight splits
    q, cache, table, ctx = _step(lens, H, C, R)
    q[:], cache[:] = 1.0, 0.0
    for t in range(2):
        cache[table[t, 0].long(), 0, :32, 0] = -200.0
    cache[table[1, 0].long(), 0, 7, 1] = torch.nan
    out = torch.full((2, H * C), 7.0, device=DEV, dtype=torch.bfloat16)
    kernels.latent_decode(q, out, H, C, R, ctx, table, table.shape[1], cache, 1.0)
    assert (out[0] == 0).all() and out[1].isnan().all()
