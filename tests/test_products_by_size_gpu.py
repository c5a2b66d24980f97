"""The products that a size chooses, at the sizes where each can go wrong: 32-bit rows that start on 16 bytes (bit for bit the
general kernel's sums), and the token tiles of the kernel that pairs two SMs."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def K():
    from gguf_rs_cli_b200 import kernels
    return kernels


def _operands(T, N, Kd, seed, dtype=torch.bfloat16):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randn(T, Kd, generator=g, device=DEV).to(dtype)
    w = (torch.randn(N, Kd, generator=g, device=DEV) / math.sqrt(Kd)).to(dtype)
    return x, w, torch.randn(N, generator=g, device=DEV), g


def _sum_bound(x, w):
    """A 32-bit sum of K exact products in any order is off by at most K 2^-24 times the sum of their magnitudes; its bound is
    never reached, a sixteenth of it still is a hundred times what random signs give."""
    return x.shape[1] * 2.0 ** -28 * (x.double().abs() @ w.double().abs().T) + 1e-6


@pytest.mark.parametrize("T", [1, 2, 4, 5, 8, 9, 16, 17, 31, 48, 49, 144, 200])
def test_32_bit_products_are_the_general_kernels_bit_for_bit(T):
    k = K()
    # the last two: few tokens take several tiles a CTA with several pieces of K each
    for N, Kd in ((64, 64), (130, 176), (1, 4), (257, 132), (3072, 260), (20000, 96), (20000, 260), (40000, 516)):
        x, w, b, _ = _operands(T, N, Kd, N + Kd, torch.float32)
        for bias in (None, b):
            want, got = torch.empty(T, N, device=DEV), torch.full((T, N + 5), 7.0, device=DEV)[:, :N]
            k.gemm_generic(x, w, bias, want)
            assert k.gemm_f32_supported(x, w)
            k.gemm_f32(x, w, bias, got)
            assert torch.equal(got, want), (N, Kd)
    wide = torch.randn(T, 520, device=DEV)
    w = torch.randn(96, 520, device=DEV)
    assert not k.gemm_f32_supported(wide[:, 1:513], w[:, :512]) and not k.gemm_f32_supported(wide[:, :510], w[:, :510])
    want, got = torch.empty(T, 96, device=DEV), torch.empty(T, 96, device=DEV)
    k.gemm_generic(wide[:, 4:516], w[:, 8:520], None, want)
    k.gemm_f32(wide[:, 4:516], w[:, 8:520], None, got)
    assert torch.equal(got, want)


@pytest.mark.parametrize("tile", [96, 112, 176, 192, 208, 224, 240, 256, 0])
def test_token_tiles_of_two_sms(tile):
    """Every width gives the widest tile's results bit for bit (each is one ascending sum), whatever the number of tokens."""
    from gguf_rs_cli_b200 import native
    k = K()
    try:
        native.call("gb_gemm_tc_set_tile", 256)
        for T, N, Kd in ((1000, 512, 256), (769, 640, 136), (2049, 300, 64), (300, 30000, 64)):
            x, w, b, _ = _operands(T, N, Kd, T)
            w2 = k.interleave_gate_up(w[:N // 2], w[N // 2:N // 2 * 2])
            got = []
            for t in (256, tile):
                native.call("gb_gemm_tc_set_pair_tile", t)
                outs = [torch.full((T, N), 9.0, device=DEV, dtype=d) for d in (torch.bfloat16, torch.float32)]
                gated = torch.full((T, N // 2), 9.0, device=DEV, dtype=torch.bfloat16)
                for o in outs:
                    k.gemm_tc(x, w, b, o)
                k.gemm_tc(x, w2, None, gated, swiglu_features=N // 2)
                # a norm's factor per token, and a sum into the residual stream with its copy and the new sums of squares
                scaled, resid = torch.full((T, N), 9.0, device=DEV), torch.ones(T, N, device=DEV)
                copy, ssq = torch.empty(T, N, device=DEV, dtype=torch.bfloat16), torch.empty((N + 127) // 128, T, device=DEV)
                parts = x.float().pow(2).view(T, 2, Kd // 2).sum(2).t().contiguous()
                k.gemm_tc(x, w, None, scaled, row_ssq=parts, ssq_parts=2, norm_size=Kd, eps=1e-5)
                k.gemm_tc(x, w, b, None, resid_x=resid, resid_xb=copy, ssq_out=ssq)
                got.append(outs + [gated, scaled, resid, copy, ssq])
            assert all(torch.equal(a, c) for a, c in zip(*got)), (T, N, Kd)
            plain = x.double() @ w.double().T
            outs, scaled, resid, copy, ssq = got[1][:2], *got[1][3:]
            assert ((outs[1].double() - plain - b.double()).abs() <= _sum_bound(x, w)).all()
            rstd = (x.double().pow(2).mean(1, keepdim=True) + 1e-5).rsqrt()
            # the factor itself is a 32-bit reciprocal root of a 32-bit mean: 2^-20 of the result covers both
            assert ((scaled.double() - plain * rstd).abs() <= _sum_bound(x, w) * rstd + 2.0 ** -20 * (plain * rstd).abs()).all()
            assert ((resid.double() - 1 - plain - b.double()).abs() <= _sum_bound(x, w) + 2.0 ** -22 * resid.double().abs()).all()
            assert torch.equal(copy, resid.bfloat16())
            sums = torch.nn.functional.pad(resid.double().pow(2), (0, -N % 128)).view(T, -1, 128).sum(2).t()
            assert ((ssq.double() - sums).abs() <= 2.0 ** -17 * sums).all()      # 128 squares, each addition off by at most 2^-24 of the sum
    finally:
        native.call("gb_gemm_tc_set_pair_tile", 0)
        native.call("gb_gemm_tc_set_tile", 0)
    torch.cuda.synchronize()
    k.check_tc_status()


@pytest.mark.parametrize("T", [129, 300, 769, 2049])
@pytest.mark.parametrize("N", [64, 128, 200, 300, 640])
def test_residual_sums_stay_inside_their_rows(T, N):
    """A pair's second CTA has no features where the last tile's end in its first half: it writes no sums of squares, which would
    lie behind the ceil(N/128) rows that the caller gave."""
    k = K()
    x, w, b, _ = _operands(T, N, 64, T + N)
    tiles = (N + 127) // 128
    resid, copy = torch.ones(T, N, device=DEV), torch.empty(T, N, device=DEV, dtype=torch.bfloat16)
    ssq = torch.full((tiles + 2, T), 7.0, device=DEV)
    k.gemm_tc(x, w, b, None, resid_x=resid, resid_xb=copy, ssq_out=ssq)
    assert (ssq[tiles:] == 7.0).all() and torch.equal(copy, resid.bfloat16())
    sums = torch.nn.functional.pad(resid.double().pow(2), (0, -N % 128)).view(T, -1, 128).sum(2).t()
    assert ((ssq[:tiles].double() - sums).abs() <= 2.0 ** -17 * sums).all()      # 128 squares, an addition off by 2^-24 of the sum at most


def test_pairs_of_sms_are_counted_before_the_first_product():
    """The width of a tile goes by how many pairs the device holds, asked before the kernel's first launch in a process."""
    import subprocess
    import sys
    code = """if True:
        import torch
        from gguf_rs_cli_b200 import kernels, native
        x = torch.zeros(1024, 256, device="cuda", dtype=torch.bfloat16)
        first = native.library().gb_gemm_tc_pair_slots()
        kernels.gemm_tc(x, x, None, torch.empty(1024, 1024, device="cuda"))
        torch.cuda.synchronize()
        assert 0 < first == native.library().gb_gemm_tc_pair_slots() <= torch.cuda.get_device_properties(0).multi_processor_count // 2
    """
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr


@pytest.mark.parametrize("T", [129, 191, 300, 512, 769])
def test_a_few_hundred_tokens(T):
    """Either side of every border of the rule: K at 1,024, tiles of 64 tokens per K, more of them than SMs, and for gated products
    than twice as many.  A bfloat16 result is the 32-bit one, rounded, whichever kernel a size takes."""
    k = K()
    for N, Kd in ((256, 8192), (4096, 8192), (640, 2040), (640, 2048), (1300, 2048), (6144, 64), (130, 8200), (256, 1016), (256, 1024),
                  (1500, 1024), (3000, 3072), (4096, 4096)):
        x, w, b, _ = _operands(T, N, Kd, T + N)
        out = torch.empty(T, N, device=DEV)
        k.gemm_tc(x, w, b, out)
        assert ((out.double() - x.double() @ w.double().T - b.double()).abs() <= _sum_bound(x, w)).all(), (N, Kd)
        low = torch.empty(T, N, device=DEV, dtype=torch.bfloat16)
        k.gemm_tc(x, w, b, low)
        assert torch.equal(low, out.bfloat16()), (N, Kd)
    for F, Kd in ((100, 1024), (520, 1024), (1024, 512), (3000, 256), (4736, 136)):
        x, w, _, _ = _operands(T, 2 * F, Kd, T + F)
        gate, up = (x.double() @ w[i * F:(i + 1) * F].double().T for i in (0, 1))
        want = torch.nn.functional.silu(gate) * up
        got = torch.empty(T, F, device=DEV)
        k.gemm_tc(x, k.interleave_gate_up(w[:F], w[F:]), None, got, swiglu_features=F)
        assert (got.double() - want).norm() <= 1e-5 * want.norm(), (F, Kd)           # 32-bit sums of up to 1,024 terms
        low = torch.empty(T, F, device=DEV, dtype=torch.bfloat16)
        k.gemm_tc(x, k.interleave_gate_up(w[:F], w[F:]), None, low, swiglu_features=F)
        assert torch.equal(low, got.bfloat16()), (F, Kd)
    torch.cuda.synchronize()
    k.check_tc_status()


@pytest.mark.parametrize("N, K", [(1000, 16), (1001, 16), (1001, 20), (4096, 4)])
@pytest.mark.parametrize("T", [1, 17])
def test_products_of_one_block_of_k_are_the_same_bits_on_either_kernel(T, N, K):
    from gguf_rs_cli_b200 import kernels as k
    g = torch.Generator(device="cuda").manual_seed(N + K)
    x, w = torch.randn(T, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    outs = [f(x, w, None, torch.empty(T, N, device="cuda")) for f in (k.gemm, k.gemm_f32, k.gemm_generic)]
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


@pytest.mark.parametrize("T", [1, 4, 16, 17, 64, 127])
@pytest.mark.parametrize("N", [6672, 2624, 132, 1030, 2047])
def test_shared_tiles_at_a_matrixs_edge(N, T):
    """The last tile's features, where several CTAs share a tile: the bits of the same matrix with rows of zeros up to a whole tile, for
    rows that take accesses of four values and rows that do not; nothing is written beside them."""
    k = K()
    x, w, b, g = _operands(T, N, 2048, N + T)
    P = (N + 127) // 128 * 128
    wp, bp = torch.zeros(P, 2048, device=DEV, dtype=w.dtype), torch.zeros(P, device=DEV)
    wp[:N], bp[:N] = w, b
    for pitch in (N, (N + 7) // 4 * 4, N + 3):
        for dtype in (torch.float32, torch.bfloat16):
            want, got = torch.empty(T, P, device=DEV, dtype=dtype), torch.full((T, pitch), 9.0, device=DEV, dtype=dtype)
            k.gemm_tc(x, wp, bp, want)
            k.gemm_tc(x, w, b, got[:, :N])
            assert torch.equal(got[:, :N], want[:, :N]) and (got[:, N:] == 9.0).all(), (pitch, dtype)
        start, parts = torch.randn(T, P, generator=g, device=DEV), P // 128
        full, fullb, ssq_full = start.clone(), torch.empty(T, P, device=DEV, dtype=torch.bfloat16), torch.empty(parts, T, device=DEV)
        k.gemm_tc(x, wp, bp, None, resid_x=full, resid_xb=fullb, ssq_out=ssq_full, resid_scale=0.5)
        res, resb = torch.full((T, pitch), 9.0, device=DEV), torch.full((T, pitch), 9.0, device=DEV, dtype=torch.bfloat16)
        res[:, :N], ssq = start[:, :N], torch.full((parts, T), 9.0, device=DEV)
        k.gemm_tc(x, w, b, None, resid_x=res[:, :N], resid_xb=resb[:, :N], ssq_out=ssq, resid_scale=0.5)
        assert torch.equal(res[:, :N], full[:, :N]) and torch.equal(resb[:, :N], fullb[:, :N])
        assert (res[:, N:] == 9.0).all() and (resb[:, N:] == 9.0).all()
        want = torch.nn.functional.pad(full[:, :N].double() ** 2, (0, P - N)).view(T, parts, 128).sum(2).T
        # 128 squares, each rounded once, and their sum in any order: 128 roundings at most
        assert ((ssq.double() - want).abs() <= 129 * 2.0 ** -24 * want).all()
