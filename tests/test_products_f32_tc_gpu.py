"""32-bit products on the tensor cores: every tile width, its edges, shared tiles, operands that are not finite, and the
distance from 64 bits beside the one-thread sums of the CUDA-core kernel."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _operands(T, N, K, seed, positive=False):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x, w = torch.randn(T, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV) / math.sqrt(K)
    return (x.abs(), w.abs()) if positive else (x, w)


# widths of 32, 64, 96, 128, 160 and 192 tokens, several of them, K that ends inside a block, one block, shared tiles and whole ones
@pytest.mark.parametrize("T", [1, 16, 17, 32, 33, 64, 96, 97, 128, 160, 187, 192, 193, 400])
@pytest.mark.parametrize("N, K", [(128, 512), (130, 2048), (3000, 516), (257, 4), (20000, 548), (2048, 4096)])
@pytest.mark.parametrize("positive", [False, True])
def test_closer_to_64_bits_than_one_thread(T, N, K, positive):
    from gguf_rs_cli_b200 import kernels as k
    x, w = _operands(T, N, K, T + N + K, positive)
    bias = torch.randn(N, device=DEV) if K == 516 else None
    want = x.double() @ w.double().T
    if bias is not None:
        want += bias.double()
    got, plain = torch.full((T, N + 4), 7.0, device=DEV)[:, :N], torch.empty(T, N, device=DEV)
    k.gemm_f32_tc(x, w, bias, got)
    k.gemm_f32(x, w, bias, plain)
    torch.cuda.synchronize()
    k.check_tc_status()
    e, e_plain = [float((a.double() - want).norm() / want.norm()) for a in (got, plain)]
    # a result is rounded once (2^-25 in the mean of a binade's ends) and the sums of 32 that it adds are; the product left out is 2^-34
    assert e <= max(1.1 * e_plain, 1.5e-7) and e < 4e-7, (e, e_plain)
    assert (got._base[:, N:] == 7.0).all()
    again, low = torch.empty_like(plain), torch.empty(T, N, dtype=torch.bfloat16, device=DEV)
    k.gemm_f32_tc(x, w, bias, again)
    k.gemm_f32_tc(x, w, bias, low)
    assert torch.equal(again, got) and torch.equal(low, got.bfloat16())          # the order of the sums is fixed; counters are back at zero


@pytest.mark.parametrize("n", [1, 2, 3, 4, 6, 8, 12, 16])
@pytest.mark.parametrize("apart", [False, True])
@pytest.mark.parametrize("positive", [False, True])
def test_rows_of_few_terms(n, apart, positive):
    """Rows of X with n entries, in one or two blocks of 32 of K or all over it: as close to 64 bits as one 32-bit FMA behind another."""
    from gguf_rs_cli_b200 import kernels as k
    T, N, K = 64, 1024, 2048
    full, w = _operands(T, N, K, 10 * n + apart, positive)
    x = torch.zeros_like(full)
    for t in range(T):
        at = torch.randperm(K, device=DEV)[:n] if apart else (torch.arange(n, device=DEV) + 37 * t) % K
        x[t, at] = full[t, at]
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    got, plain = torch.empty(T, N, device=DEV), torch.empty(T, N, device=DEV)
    k.gemm_f32_tc(x, w, None, got)
    k.gemm_f32(x, w, None, plain)
    e, e_plain = [float((a.double() - want).norm() / want.norm()) for a in (got, plain)]
    # Terms far apart are rounded when their piece of K is complete and again when the pieces are added, an FMA once: 1.15 to 1.19 measured for two to four.
    assert e <= (1.01 if n == 1 else 1.25 if apart else 1.0) * e_plain, (e, e_plain)
    # one product: its large part is exact, the small ones are cut at 2^-23 of themselves, 2^-8 of it, and the sum is rounded once; n: n sums of either kind
    # and of pieces, each rounded once
    assert ((got.double() - want).abs() <= (1 if n == 1 else 3 * n) * (1 + 2.0 ** -6) * 2.0 ** -24 * size).all()


def test_rows_of_larger_matrices_and_the_dispatch():
    from gguf_rs_cli_b200 import kernels as k
    x, w = _operands(40, 1030, 1032, 3)
    for K, tc in ((1024, True), (1020, False)):
        xs, ws = x[:, 4:4 + K], w[:, 8:8 + K]
        got, direct = torch.empty(40, 1030, device=DEV), torch.empty(40, 1030, device=DEV)
        k.gemm(xs, ws, None, got)
        (k.gemm_f32_tc if tc else k.gemm_generic)(xs, ws, None, direct)
        want = xs.double() @ ws.double().T
        assert torch.equal(direct, got) and float((got.double() - want).norm() / want.norm()) < (4e-7 if tc else 2e-6)


@pytest.mark.parametrize("N, K", [(1024, 1024), (2048, 8192), (3072, 2048), (20000, 2048), (40000, 1024), (1030, 1100)])
def test_a_rows_result_does_not_depend_on_the_rows_beside_it(N, K):
    """One, two, four CTAs' share of K, or sixteen, tiles of every width: the same bits for a token, alone or among others."""
    from gguf_rs_cli_b200 import kernels as k
    x, w = _operands(450, N, K, N + K)
    want = torch.empty(450, N, device=DEV)
    k.gemm(x, w, None, want)
    for lo, hi in ((0, 1), (3, 5), (0, 16), (1, 18), (0, 33), (7, 80), (0, 100), (10, 140), (0, 192), (50, 243), (100, 450)):
        got = torch.empty(hi - lo, N, device=DEV)
        k.gemm(x[lo:hi], w, None, got)
        assert torch.equal(got, want[lo:hi]), (lo, hi)
    torch.cuda.synchronize()
    k.check_tc_status()


@pytest.mark.parametrize("T", [1, 16, 30, 64, 90, 187, 700])
@pytest.mark.parametrize("N, K", [(300, 1024), (20000, 1028), (2048, 8192)])
def test_tiny_operands_beside_large_ones(T, N, K):
    """Rows of X, of W, and single entries too small for three bfloat16 terms, beside operands that make a result of them that counts: what one 32-bit FMA
    behind another gives.  Beside operands of ordinary size they change nothing, and neither do zeros."""
    from gguf_rs_cli_b200 import kernels as k

    def run(x, w, bias=None, dtype=torch.float32):
        got, plain = torch.empty(T, N, device=DEV, dtype=dtype), torch.empty(T, N, device=DEV, dtype=dtype)
        k.gemm_f32_tc(x, w, bias, got)
        k.gemm_f32(x, w, bias, plain)
        return got, plain
    x0, w0 = _operands(T, N, K, T + K)
    for tiny, large in ((1e-34, 1e30), (1e-36, 1e12), (1e-38, 1e30), (1e-42, 1e30)):
        for a, b in ((tiny, large), (large, tiny)):
            got, plain = run(x0 * a, w0 * b)
            assert torch.equal(got, plain), (a, b)                              # all of them are summed again
    bias = torch.randn(N, device=DEV) * 1e-12
    for dtype in (torch.float32, torch.bfloat16):
        got, plain = run(x0 * 1e-42, w0 * 1e30, bias, dtype)
        assert torch.equal(got, plain)
    ordinary, _ = run(x0, w0)
    x, w = x0.clone(), w0.clone()
    x[:, 5::7], w[::3, 11] = 1e-39, -1e-37                                       # what is lost is below 2^-134 times K times 5
    got, plain = run(x, w)
    want = x.double() @ w.double().T
    assert float((got.double() - want).norm()) <= 1.01 * float((plain.double() - want).norm())
    assert not torch.equal(got, plain) and not torch.equal(got, ordinary)
    x[T // 2], w[:, 3] = 0.0, 1e33
    x[T // 2, 3] = 1.23456789e-39                                                # the only term of a row, 1e-6
    got, plain = run(x, w)
    assert torch.equal(got[T // 2], plain[T // 2]) and (got[T // 2] != 0).all()
    k.check_tc_status()


def test_operands_that_are_not_finite_and_large_ones():
    """Infinities, NaN (with a payload in its last bits only), numbers next to the largest, and subnormal ones: what one thread's sum gives."""
    from gguf_rs_cli_b200 import kernels as k
    x, w = _operands(50, 200, 640, 5)
    x[3, 100], x[7, 5], x[9, 639] = math.inf, -math.inf, math.nan
    x[11, 50] = torch.tensor(0x7F800001, dtype=torch.int32).view(torch.float32)
    x[20, :] = 0.0
    x[20, 3], w[17, 3] = 3.4e38, 1.0
    x[21, 4], w[18, 4] = 3.4e38, 4.0
    x[22] *= 1e-39
    w[30, 9] = math.inf
    x[23, 9] = 0.0
    got, want = torch.empty(50, 200, device=DEV), torch.empty(50, 200, device=DEV)
    k.gemm_f32_tc(x, w, None, got)
    k.gemm_generic(x, w, None, want)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    inf = want.isinf()
    assert torch.equal(got[inf], want[inf]) and inf.any() and want.isnan().any()
    # a row's error is measured against its own size; row 22 holds sums of subnormal numbers, taken one product behind another like
    # gemm_generic's unless nothing is left of them at all (below 2^-126)
    fin = want.isfinite()
    a, b = torch.where(fin, got, 0.0).double(), torch.where(fin, want, 0.0).double()
    assert ((a - b).norm(dim=1) <= 2e-6 * b.norm(dim=1) + 2.0 ** -126).all()
    assert torch.equal(got[22][got[22] != 0], want[22][got[22] != 0]) and (got[22] != 0).sum() > 100


def test_streams_have_counters_of_their_own():
    from gguf_rs_cli_b200 import kernels as k
    x, w = _operands(100, 2048, 2048, 9)
    want = torch.empty(100, 2048, device=DEV)
    k.gemm_f32_tc(x, w, None, want)
    torch.cuda.synchronize()
    streams, outs = [torch.cuda.Stream() for _ in range(2)], []
    for _ in range(20):
        for s in streams:
            with torch.cuda.stream(s):
                outs.append(torch.empty(100, 2048, device=DEV))
                k.gemm_f32_tc(x, w, None, outs[-1])
    torch.cuda.synchronize()
    k.check_tc_status()
    assert all(torch.equal(o, want) for o in outs)


@pytest.mark.parametrize("T, N, K", [(2048, 2048, 2048), (2048, 2048, 8192), (1500, 1100, 14336), (5000, 2048, 1024), (187, 16384, 2048), (1, 40000, 1024)])
def test_scratch_memory_is_bounded(T, N, K):
    """However many tokens and pieces of K: sums wait in registers, in the result, or in memory of a fixed size; a row's bits stay what they are alone."""
    from gguf_rs_cli_b200 import kernels as k, native
    x, w = _operands(T, N, K, N + K)
    most = native.library().gb_gemm_f32_tc_scratch_max()
    assert most <= 8 << 20
    for code in (0, 1):
        assert native.library().gb_gemm_f32_tc_scratch_floats(T, N, K, code, 148) <= most
    got, low = torch.empty(T, N, device=DEV), torch.empty(T, N, device=DEV, dtype=torch.bfloat16)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    k.gemm_f32_tc(x, w, None, got)
    k.gemm_f32_tc(x, w, None, low)
    torch.cuda.synchronize()
    k.check_tc_status()
    assert torch.cuda.max_memory_allocated() - before <= 4 * most + (1 << 20)
    assert torch.equal(low, got.bfloat16())
    for lo, hi in ((0, 1), (T // 2, T // 2 + 40), (T - 1, T)):
        hi = min(hi, T)
        part = torch.empty(hi - lo, N, device=DEV)
        k.gemm_f32_tc(x[lo:hi], w, None, part)
        assert torch.equal(part, got[lo:hi])
    want = x.double() @ w.double().T
    assert float((got.double() - want).norm() / want.norm()) < 4e-7


def test_products_on_two_streams_wait_for_nobody():
    """Launches that share the device with one another, of every width, shared tiles among them: nothing waits for CTAs that have not started."""
    from gguf_rs_cli_b200 import kernels as k
    cases = [(_operands(T, N, K, T + K), T, N) for T, N, K in ((1, 2048, 8192), (30, 4096, 4096), (100, 2048, 8192), (187, 2048, 2048), (60, 3072, 2048))]
    want = []
    for (x, w), T, N in cases:
        want.append(torch.empty(T, N, device=DEV))
        k.gemm_f32_tc(x, w, None, want[-1])
    torch.cuda.synchronize()
    streams, outs = [torch.cuda.Stream() for _ in range(4)], []
    for i in range(40):
        for j, s in enumerate(streams):
            (x, w), T, N = cases[(i + j) % len(cases)]
            with torch.cuda.stream(s):
                outs.append(((i + j) % len(cases), torch.empty(T, N, device=DEV)))
                k.gemm_f32_tc(x, w, None, outs[-1][1])
    torch.cuda.synchronize()
    k.check_tc_status()
    assert all(torch.equal(o, want[i]) for i, o in outs)


@pytest.mark.parametrize("N, K", [(19072, 1024), (28672, 1100), (30000, 1060), (37000, 1024), (37888, 1024)])
def test_two_unequal_pieces_of_k(N, K):
    """More tiles of features than SMs: few tokens have a tile's first piece of K or several tiles' second ones, prompts whole tiles: the same bits."""
    from gguf_rs_cli_b200 import kernels as k
    x, w = _operands(200, N, K, N + K)
    bias, want = torch.randn(N, device=DEV), torch.empty(200, N, device=DEV)
    k.gemm_f32_tc(x, w, bias, want)
    exact = x.double() @ w.double().T + bias.double()
    assert float((want.double() - exact).norm() / exact.norm()) < 2e-7
    for T in (1, 15, 16, 17, 32, 33, 96, 97, 128):
        for dtype in (torch.float32, torch.bfloat16):
            got = torch.full((T, N + 4), 7.0, device=DEV, dtype=dtype)
            k.gemm_f32_tc(x[:T], w, bias, got[:, :N])
            assert torch.equal(got[:, :N], want[:T].to(dtype)) and (got[:, N:] == 7.0).all(), (T, dtype)
    k.check_tc_status()


def test_heads_of_more_features_than_a_round_holds_stay_on_cuda_cores():
    from gguf_rs_cli_b200 import kernels as k
    x, w = _operands(3, 37889, 1024, 4)
    for N, kernel in ((37888, k.gemm_f32_tc), (37889, k.gemm_f32)):
        got, direct = torch.empty(3, N, device=DEV), torch.empty(3, N, device=DEV)
        k.gemm(x, w[:N], None, got)
        kernel(x, w[:N], None, direct)
        assert torch.equal(got, direct)
