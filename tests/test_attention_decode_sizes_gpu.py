"""The CUDA-core kernel of single tokens where its sizes choose what runs: groups of up to 4 with heads of up to 64 either side of
three CTAs an SM, and every way of adding up splits, against 64-bit sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _step(T, L, nkv, G, hd, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    width = (L + 63) // 64
    k, v = (torch.randn(T * width, nkv, 64, hd, generator=g, device=DEV).bfloat16() for _ in range(2))
    q = torch.randn(T, nkv * G * hd, generator=g, device=DEV).bfloat16()
    table = torch.randperm(T * width, generator=g, device=DEV).int().view(T, width)
    pos = (L - 1 - torch.arange(T, device=DEV) % min(L, 50)).int()
    return q, k, v, table, pos


def _run(q, k, v, table, pos, nkv, G, hd, splits, rows=slice(None)):
    from gguf_rs_cli_b200 import kernels
    T = pos[rows].numel()
    out = torch.full((T, nkv * G * hd), 7.0, device=DEV, dtype=torch.bfloat16)
    return kernels.attention_decode(q[rows], out, nkv * G, nkv, hd, torch.arange(T, device=DEV, dtype=torch.int32), pos[rows],
                                    table[rows], table.shape[1], k, v, 0, hd ** -0.5, splits=splits, mma=False)


def _plain(q, k, v, table, pos, nkv, G, hd):
    out = []
    for t, n in enumerate((pos + 1).tolist()):
        pages = table[t].long()
        kk, vv = (c[pages].transpose(0, 1).reshape(nkv, -1, hd)[:, :n].double() for c in (k, v))
        s = torch.softmax(q[t].double().view(nkv, G, hd) @ kk.transpose(1, 2) * hd ** -0.5, -1)
        out.append((s @ vv).flatten())
    return torch.stack(out)


def _check(got, want):
    """Half a unit in the last place of bfloat16 is 2^-9 of a value; sums of a few hundred 32-bit terms are far below the other half."""
    assert ((got.double() - want).abs() <= 2 ** -8 * want.abs().amax(1, keepdim=True)).all()


@pytest.mark.parametrize("G, hd", [(3, 64), (4, 48), (4, 64)])
@pytest.mark.parametrize("more", [-1, 0, 1])
def test_a_token_does_not_depend_on_how_many_there_are(G, hd, more):
    """More CTAs than three an SM run in another instance of the kernel: the same sums, bit for bit."""
    nkv = 4
    T = 3 * torch.cuda.get_device_properties(0).multi_processor_count // nkv + more
    step = _step(T, 130, nkv, G, hd)
    many = _run(*step, nkv, G, hd, 1)
    for a in range(0, T, 40):
        assert torch.equal(many[a:a + 40], _run(*step, nkv, G, hd, 1, slice(a, a + 40)))
    _check(many, _plain(*step, nkv, G, hd))


@pytest.mark.parametrize("G, hd", [(1, 128), (4, 64), (4, 128), (4, 192), (8, 64), (8, 128), (11, 192), (8, 256)])
@pytest.mark.parametrize("splits", [1, 2, 3, 4, 6, 7, 8, 12, 15, 16])
def test_every_number_of_splits(G, hd, splits):
    step = _step(3, 900, 2, G, hd, seed=splits)
    _check(_run(*step, 2, G, hd, splits), _plain(*step, 2, G, hd))
