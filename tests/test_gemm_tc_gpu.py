"""tcgen05 / TMA GEMM against a PyTorch fp32 reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from layerstorm_b200.ops import _native as nat


def run(M, N, K, out_bf16=False, bias=False, splitk=True, ldx=None, seed=0):
    g = torch.Generator().manual_seed(seed)
    ldx = ldx or K
    x = (torch.randn(M, ldx, generator=g)).to(torch.bfloat16).cuda()
    w = (torch.randn(N, K, generator=g) * 0.05).to(torch.bfloat16).cuda()
    b = torch.randn(N, generator=g).cuda() if bias else None
    out = torch.zeros(M, N, device="cuda", dtype=torch.bfloat16 if out_bf16 else torch.float32)
    part = torch.zeros(16 * M * N, device="cuda") if splitk else None
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    nat.call("lsb_gemm_bf16_tc", out, x, w, b, M, N, K, ldx, K, N, int(out_bf16), part, 16 * M * N if splitk else 0, err, None)
    torch.cuda.synchronize()
    assert int(err[0]) == 0, f"kernel reported wait timeout code {int(err[0])}"
    ref = x[:, :K].float() @ w.float().T
    if bias:
        ref = ref + b
    tol = 2e-2 if out_bf16 else 2e-3
    e = (out.float() - ref).abs().max() / ref.abs().max()
    assert float(e) < tol, (M, N, K, float(e))


def test_gemm_tc_smallest():
    run(16, 128, 64, splitk=False)


@pytest.mark.parametrize("M,N,K", [(16, 128, 256), (32, 256, 512), (64, 384, 1024), (128, 512, 512), (256, 256, 2048),
                                   (300, 200, 264), (17, 130, 72), (2048, 1024, 512)])
def test_gemm_tc_shapes(M, N, K):
    run(M, N, K, splitk=False)


def test_gemm_tc_splitk_bias_bf16():
    run(32, 256, 4096, splitk=True, bias=True)
    run(48, 512, 2048, splitk=True, out_bf16=True, bias=True)
    run(64, 128, 1024, ldx=1032, splitk=True)


@pytest.mark.parametrize("M,B,N,K", [(64, 4, 128, 64), (300, 8, 512, 256), (2048, 3, 256, 128)])
def test_gemm_tc_batched_strided(M, B, N, K):
    """Per-head products as one launch: x[m, b, :K] (heads interleaved in a row), w[b], out[m, b, :N]."""
    g = torch.Generator().manual_seed(3)
    pad = 64                                            # a rope tail sits between the heads' K columns
    x = torch.randn(M, B, K + pad, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(B, N, K, generator=g) * 0.05).to(torch.bfloat16).cuda()
    out = torch.zeros(M, B, N + 8, device="cuda", dtype=torch.bfloat16)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    nat.call("lsb_gemm_bf16_tc_batched", out, x, w, M, N, K, B, B * (K + pad), K + pad, K, N * K, B * (N + 8), N + 8, 1, err)
    torch.cuda.synchronize()
    assert int(err[0]) == 0
    ref = torch.einsum("mbk,bnk->mbn", x[:, :, :K].float(), w.float())
    e = (out[:, :, :N].float() - ref).abs().max() / ref.abs().max()
    assert float(e) < 2e-2, float(e)
    assert float(out[:, :, N:].abs().max()) == 0.0      # nothing written past N


@pytest.mark.parametrize("fmt", ["fp8_e4m3", "nvfp4"])
@pytest.mark.parametrize("M,N,K", [(16, 128, 128), (100, 256, 512), (300, 384, 1024)])
def test_quantised_linear_tensor_core_path(fmt, M, N, K):
    """QLinear with many rows (de-quantisation fused into the tcgen05 pipeline) == the same weights through fp32 matmul
    == the row-streaming GEMV path."""
    from layerstorm_b200.models.device_model import QLinear
    g = torch.Generator().manual_seed(11)
    wf = torch.randn(N, K, generator=g) * 0.05
    lin = QLinear.from_float(wf.cuda(), fmt, "cuda")
    x = torch.randn(M, K, generator=g).to(torch.bfloat16).cuda()
    ref = x.float() @ lin.dequant().float().T
    for dt, tol in ((torch.float32, 3e-3), (torch.bfloat16, 2e-2)):
        out = torch.zeros(M, N + 16, device="cuda", dtype=dt)
        lin(out, x, M, ldo=N + 16)
        torch.cuda.synchronize()
        e = (out[:, :N].float() - ref).abs().max() / ref.abs().max()
        assert float(e) < tol, (fmt, dt, float(e))
    few = torch.zeros(4, N, device="cuda")
    lin(few, x, 4)                                       # GEMV path on the first rows
    torch.cuda.synchronize()
    assert float((few - ref[:4]).abs().max() / ref.abs().max()) < 3e-3


@pytest.mark.parametrize("M,N,K", [(129, 8, 2048), (257, 200, 2056), (513, 384, 2112), (300, 1000, 2048), (700, 30000, 2048), (300, 2000, 2056), (1100, 576, 4096),
                                   (300, 19000, 8200), (513, 12600, 8192)])
@pytest.mark.parametrize("ob", [0, 1])
def test_two_weight_tiles_per_cta(M, N, K, ob):
    """Reductions from 2048 on over more than 128 rows, in every form that they run in (one weight tile per CTA: one wave, just above it, three waves of a long
    reduction; two tiles): a last weight tile that is empty or not full, token tiles and stages that are not full, with and without split reductions, a bias,
    nothing written beyond the matrix."""
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = (torch.randn(n, K, generator=g, device="cuda").bfloat16() for n in (M, N))
    bias = torch.randn(N, generator=g, device="cuda")
    out = torch.zeros(M + 1, N + 8, device="cuda", dtype=torch.bfloat16 if ob else torch.float32)
    part, err = torch.zeros(1 << 24, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    nat.call("lsb_gemm_bf16_tc", out, x, w, bias, M, N, K, K, K, N + 8, ob, part, part.numel(), err, None)
    want = x.double() @ w.double().T + bias.double()
    assert int(err) == 0 and float(out[M:].abs().sum()) == 0.0 and float(out[:M, N:].abs().sum()) == 0.0
    # fp32 sums (2^-24 sqrt(K) = 3e-6), rounded to bf16 (2^-9) where asked
    assert float((out[:M, :N].double() - want).norm() / want.norm()) < (3e-3 if ob else 1e-5)


@pytest.mark.parametrize("N", [72, 144, 1000])
@pytest.mark.parametrize("M", [5, 12, 40, 100, 142, 398])
def test_matrices_that_end_inside_a_warps_rows(M, N):
    """Lanes with and without a row of the matrix side by side in every token tile, split reduction, bias and both output types; and as a batch."""
    K = 4096
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, w = (torch.randn(n, K, generator=g, device="cuda").bfloat16() for n in (M, N))
    bias, part, err = torch.randn(N, generator=g, device="cuda"), torch.zeros(1 << 24, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    want = x.double() @ w.double().T
    # fp32 sums (2^-24 sqrt(K) = 4e-6), rounded to bf16 (2^-9) where asked
    for split in (False, True):
        for dt, tol in ((torch.float32, 1e-5), (torch.bfloat16, 3e-3)):
            out = torch.zeros(M + 1, N + 8, device="cuda", dtype=dt)
            nat.call("lsb_gemm_bf16_tc", out, x, w, bias, M, N, K, K, K, N + 8, int(dt == torch.bfloat16), part if split else None, part.numel() if split else 0, err, None)
            assert int(err) == 0 and float(out[M:].abs().sum()) == 0.0 and float(out[:M, N:].abs().sum()) == 0.0
            assert float((out[:M, :N].double() - want - bias.double()).norm() / want.norm()) < tol
    B, out = 4, torch.zeros(4, M, N, device="cuda")
    nat.call("lsb_gemm_bf16_tc_batched", out, x, w, M, N, K // B, B, K, K // B, K, K // B, N, M * N, 0, err)
    parts = torch.stack([x[:, b * K // B: (b + 1) * K // B].double() @ w[:, b * K // B: (b + 1) * K // B].double().T for b in range(B)])
    assert int(err) == 0 and float((out.double() - parts).norm() / parts.norm()) < 1e-5


@pytest.mark.parametrize("M", [5, 16, 17, 33, 64, 65, 127, 200, 256, 257, 321])
@pytest.mark.parametrize("N", [8, 12, 56, 64, 72, 100, 136, 264])
def test_bf16_rows_by_tma_and_by_stores_are_the_same(M, N):
    """Rows of 16-byte pitch at a 16-byte address leave by TMA, others by stores: the same bits, nothing outside the matrix; and as a batch in [row, head] order."""
    K = 128
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, w = (torch.randn(n, K, generator=g, device="cuda").bfloat16() for n in (M, N))
    bias, err = torch.randn(N, generator=g, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    want = x.double() @ w.double().T + bias.double()
    got, even = [], (N + 15) // 8 * 8
    for ld, at in ((even, 0), (N + 3, 0), (even, 1)):
        buf = torch.zeros((M + 1) * ld + 8, device="cuda", dtype=torch.bfloat16)
        nat.call("lsb_gemm_bf16_tc", buf[at:], x, w, bias, M, N, K, K, K, ld, 1, None, 0, err, None)
        out = buf[at: at + (M + 1) * ld].view(M + 1, ld)
        assert int(err) == 0 and float(out[M:].abs().sum()) == 0.0 and float(out[:M, N:].abs().sum()) == 0.0 and float(buf[:at].abs().sum()) == 0.0
        got.append(out[:M, :N].clone())
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    assert float((got[0].double() - want).norm() / want.norm()) < 3e-3          # 2^-9, rounding to bf16
    B, out = 2, torch.zeros(M + 1, 2, even, device="cuda", dtype=torch.bfloat16)
    nat.call("lsb_gemm_bf16_tc_batched", out, x, w, M, N, K // B, B, K, K // B, K, K // B, B * even, even, 1, err)
    parts = torch.stack([x[:, b * K // B: (b + 1) * K // B].double() @ w[:, b * K // B: (b + 1) * K // B].double().T for b in range(B)], 1)
    assert int(err) == 0 and float(out[M:].abs().sum()) == 0.0 and float(out[:, :, N:].abs().sum()) == 0.0
    assert float((out[:M, :, :N].double() - parts).norm() / parts.norm()) < 3e-3


@pytest.mark.parametrize("M", [4, 5, 6, 7, 8])
@pytest.mark.parametrize("N,K", [(8, 64), (72, 136), (1024, 4096), (1040, 4096)])
def test_bf16_linear_of_few_rows(M, N, K, monkeypatch):
    """Both sides of the lines between the weight-streaming kernel and the tensor-core GEMM: five rows, seven for small matrices."""
    from layerstorm_b200.models.device_model import QLinear
    called, call = [], nat.call
    monkeypatch.setattr(nat, "call", lambda name, *a: (called.append(name), call(name, *a))[1])
    g = torch.Generator().manual_seed(N + M)
    lin = QLinear.from_float(torch.randn(N, K, generator=g), "bf16", "cuda")
    x = torch.randn(M, K, generator=g).to(torch.bfloat16).cuda()
    for dt in (torch.float32, torch.bfloat16):
        out = torch.zeros(M, N, device="cuda", dtype=dt)
        lin(out, x, M)
        want = x.double() @ lin.w.double().T
        assert float((out.double() - want).norm() / want.norm()) < (1e-5 if dt == torch.float32 else 3e-3)
    assert called == ["lsb_gemm_bf16_tc" if M >= (5 if N == 1040 else 7) else "lsb_gemv_bf16"] * 2


@pytest.mark.parametrize("M", [1, 2, 4, 5, 16, 17, 31, 33])
@pytest.mark.parametrize("B,N,K,dr", [(5, 512, 128, 64), (3, 72, 512, 0), (16, 128, 8, 8), (2, 40, 264, 0)])
def test_products_per_head_of_any_number_of_rows(M, B, N, K, dr):
    """Per-head products of few and many rows with and without rotated tails; rows and heads of other tensors between them stay as they are."""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, w = torch.randn(M, B, K + dr, generator=g, device="cuda").bfloat16(), torch.randn(B, N, K, generator=g, device="cuda").bfloat16()
    inv, pos = torch.rand(max(dr // 2, 1), generator=g, device="cuda"), torch.randint(0, 5000, (M,), generator=g, device="cuda", dtype=torch.int32)
    out = torch.full((M + 1, B, N + dr + 8), 3.0, device="cuda", dtype=torch.bfloat16)
    nat.call("lsb_batched_gemv_bf16", out, x, w, M, B, N, K, B * (K + dr), K + dr, B * (N + dr + 8), N + dr + 8, dr, inv if dr else None, pos)
    want = torch.einsum("mbk,bnk->mbn", x[..., :K].double(), w.double())
    assert float((out[:M, :, :N].double() - want).norm() / want.norm()) < 3e-3          # fp32 sums rounded to bf16 (2^-9)
    assert bool((out[M:] == 3.0).all()) and bool((out[:, :, N + dr:] == 3.0).all())
    if dr:
        a = pos.double()[:, None, None] * inv.double()
        e, o = x[..., K::2].double(), x[..., K + 1::2].double()
        tail = torch.stack((e * a.cos() - o * a.sin(), e * a.sin() + o * a.cos()), -1).flatten(-2)
        # angles of up to 5000 in fp32 (5000 x 2^-24 = 3e-4) and rounding to bf16 (2^-9)
        assert float((out[:M, :, N: N + dr].double() - tail).norm() / tail.norm()) < 3e-3


@pytest.mark.parametrize("M", [1, 5, 8, 9, 11, 12, 14, 16, 17])
@pytest.mark.parametrize("N,K", [(16, 64), (144, 448), (2320, 1536), (1040, 512), (576, 4096), (4752, 7168), (8192, 4096), (130, 512)])
def test_few_rows_of_bf16_weights(M, N, K):
    """Few-row form and, behind its limits, the tiles: both against 64 bits; rows with padding between them, bias, weights asked for early or late.

    A sum of K products in fp32, each rounded once, is off at most K 2^-24 times the sum of the absolute products; the bf16 output by half a unit more.
    """
    g = torch.Generator().manual_seed(M * 1000 + N)
    x = torch.randn(M, K + 8, generator=g).bfloat16().cuda()
    w = torch.randn(N, K + 16, generator=g).bfloat16().cuda()
    bias = torch.randn(N, generator=g).cuda()
    err, part = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(16 * M * N, device="cuda")
    xd, wd = x[:, :K].double(), w[:, :K].double()
    want, size = xd @ wd.T + bias.double(), xd.abs() @ wd.abs().T + bias.double().abs()
    for flag, dt in [(0, torch.float32), (2, torch.float32), (1, torch.bfloat16), (3, torch.bfloat16)]:
        out = torch.full((M, N + 24), 7.0, device="cuda", dtype=dt)
        nat.call("lsb_gemm_bf16_tc", out, x, w, bias, M, N, K, K + 8, K + 16, N + 24, flag, part, part.numel(), err, None)
        bound = (K + 2) * 2.0 ** -24 * size + (want.abs() * 2.0 ** -8 if dt == torch.bfloat16 else 0)
        assert bool(((out[:, :N].double() - want).abs() <= bound).all())
        assert bool((out[:, N:] == 7).all())
        out.fill_(7.0)
        nat.call("lsb_gemv_bf16", out, x, w, bias, M, N, K, K + 8, K + 16, N + 24, 1.0, flag & 1, None)
        assert bool(((out[:, :N].double() - want).abs() <= bound).all())
        assert bool((out[:, N:] == 7).all())
    assert int(err) == 0


@pytest.mark.parametrize("M", [1, 2, 5, 33])
def test_products_per_head_of_rows_and_heads_that_share_memory(M):
    """One row for all heads, one head's input for all rows: strides of zero, as the kernel that streams them took at any number of rows."""
    B, N, K = 4, 72, 128
    g = torch.Generator(device="cuda").manual_seed(M)
    w = torch.randn(B, N, K, generator=g, device="cuda").bfloat16()
    for xs_m, xs_b in ((K, 0), (0, K), (0, 0)):
        x = torch.randn(max(M, B), K, generator=g, device="cuda").bfloat16()
        rows = torch.as_strided(x, (M, B, K), (xs_m, xs_b, 1))
        out, err = torch.full((M + 1, B, N), 3.0, device="cuda", dtype=torch.bfloat16), torch.zeros(1, dtype=torch.int32, device="cuda")
        nat.call("lsb_head_products_bf16", out, x, w, M, B, N, K, xs_m, xs_b, B * N, N, 0, None, None, err)
        want = torch.einsum("mbk,bnk->mbn", rows.double(), w.double())
        assert int(err) == 0 and bool((out[M] == 3.0).all())
        assert float((out[:M].double() - want).norm() / want.norm()) < 3e-3          # fp32 sums rounded to bf16 (2^-9)


def test_products_per_head_of_rows_far_apart():
    """Rows 2^32 + 8 elements apart: a stride that 32 bits cut down to 8."""
    B, N, K, far = 2, 72, 128, 2 ** 32 + 8
    g = torch.Generator(device="cuda").manual_seed(5)
    big = torch.empty(far + B * K, dtype=torch.bfloat16, device="cuda")
    big[: B * K + 8] = torch.randn(B * K + 8, generator=g, device="cuda").bfloat16()
    big[far:] = torch.randn(B * K, generator=g, device="cuda").bfloat16()
    w, err = torch.randn(B, N, K, generator=g, device="cuda").bfloat16(), torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.zeros(2, B, N, device="cuda", dtype=torch.bfloat16)
    nat.call("lsb_head_products_bf16", out, big, w, 2, B, N, K, far, K, B * N, N, 0, None, None, err)
    want = torch.einsum("mbk,bnk->mbn", torch.stack([big[: B * K], big[far:]]).view(2, B, K).double(), w.double())
    assert int(err) == 0 and float((out.double() - want).norm() / want.norm()) < 3e-3


@pytest.mark.parametrize("B,N,K,dr", [(16, 512, 192, 64), (8, 256, 512, 0)])
def test_products_per_head_of_a_row_do_not_depend_on_its_company(B, N, K, dr):
    """The same bits for a row alone and beside any number of others: every number of rows sums in one order."""
    g = torch.Generator(device="cuda").manual_seed(N)
    x, w = torch.randn(300, B, K + dr, generator=g, device="cuda").bfloat16(), torch.randn(B, N, K, generator=g, device="cuda").bfloat16()
    inv, pos = torch.rand(max(dr // 2, 1), generator=g, device="cuda"), torch.randint(0, 5000, (300,), generator=g, device="cuda", dtype=torch.int32)
    err, first = torch.zeros(1, dtype=torch.int32, device="cuda"), None
    for M in (1, 2, 3, 4, 5, 8, 16, 17, 31, 32, 33, 65, 129, 300):
        out = torch.zeros(M, B, N + dr, device="cuda", dtype=torch.bfloat16)
        nat.call("lsb_head_products_bf16", out, x, w, M, B, N, K, B * (K + dr), K + dr, B * (N + dr), N + dr, dr, inv if dr else None, pos, err)
        first = out if first is None else first
        assert int(err) == 0 and torch.equal(out[0], first[0]), M
