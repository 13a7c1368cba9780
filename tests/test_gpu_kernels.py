"""Each CUDA kernel alone against its plain statement (tests/plain_ops.py), at sizes other
than the engine's, in 32-bit and in bfloat16."""
import math
from types import SimpleNamespace

import pytest
import torch

import plain_ops

pytestmark = pytest.mark.gpu

DEV = "cuda"
DTYPES = [torch.float32, torch.bfloat16]


def k():
    import fastmlx_b200.kernels as kern
    return kern


def status():
    return torch.zeros(4, dtype=torch.int32, device=DEV)


def close(got, ref, dtype, what="", scale=None, extra=0.0):
    """32-bit: a few units of float32 rounding of the result's scale.  bfloat16: the same
    value may round to the neighbouring bfloat16 (one unit in the last place = 2^-7
    relative at worst) when 32-bit and 64-bit arithmetic land on different sides."""
    got, ref = got.detach().double().cpu(), ref.detach().double().cpu()
    s = ref.abs().max().item() if scale is None else scale
    s = max(s, 1e-30)
    if dtype == torch.float32:
        tol = 2e-6 * s
        bad = (got - ref).abs() > tol + 2e-6 * ref.abs()
    else:
        bad = (got - ref).abs() > 2.0 ** -7 * ref.abs() + 1e-3 * s + extra
    assert not bad.any(), f"{what} (extra {extra:.2e}): {int(bad.sum())} of {bad.numel()} off, worst {(got - ref).abs().max().item():.3e} (scale {s:.3e})"


def rnd(*shape, dtype=torch.float32, seed=0, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(dtype)


# ----------------------------------------------------------------------------- rows
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("V,d,n", [(131, 80, 7), (320, 2048, 33), (50, 100, 5), (17, 3, 4)])
def test_embedding(dtype, V, d, n):
    table = rnd(V, d, dtype=dtype)
    ids = torch.randint(0, V, (n,), dtype=torch.int32)
    st = status()
    out = k().embedding(ids.to(DEV), table.to(DEV), st)
    assert torch.equal(out.cpu(), table[ids.long()])
    assert st.tolist()[0] == 0


def test_embedding_bad_id_leaves_code_not_fault():
    table = rnd(10, 16).to(DEV)
    st = status()
    out = k().embedding(torch.tensor([1, 10, 2], dtype=torch.int32, device=DEV), table, st)
    assert st.tolist()[0] == k().BAD_TOKEN and st.tolist()[1] == 10
    assert torch.equal(out[0].cpu(), table[1].cpu()) and float(out[1].abs().sum()) == 0.0


# ----------------------------------------------------------------------------- norm
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("rows,d,eps", [(1, 64, 1e-5), (5, 192, 1e-6), (33, 80, 1e-3), (4, 2048, 1e-5), (3, 1000, 1e-5), (2, 5, 0.0)])
@pytest.mark.parametrize("with_residual", [False, True])
def test_add_rmsnorm(dtype, rows, d, eps, with_residual):
    x = rnd(rows, d, dtype=dtype, seed=1, scale=3.0)
    res = rnd(rows, d, dtype=dtype, seed=2, scale=5.0) if with_residual else None
    w = 1 + rnd(d, seed=3, scale=0.1)
    ref_out, ref_res = plain_ops.add_rmsnorm(x.clone(), res.clone() if with_residual else None, w, eps)
    xd = x.to(DEV)
    rd = res.to(DEV) if with_residual else None
    out, res_out = k().add_rmsnorm(xd, rd, w.to(DEV), eps)
    close(out, ref_out, dtype, "norm")
    if with_residual:
        assert res_out.data_ptr() == rd.data_ptr()
        close(res_out, ref_res, dtype, "residual")
    else:
        assert res_out.data_ptr() == xd.data_ptr()


@pytest.mark.parametrize("rows,d,eps", [(1, 64, 1e-5), (5, 192, 1e-6), (33, 80, 1e-3), (4, 2048, 1e-5), (3, 1000, 1e-5), (2, 5, 0.0),
                                        (8, 8192, 1e-5), (3, 8200, 1e-5)])
def test_add_rmsnorm_with_a_32_bit_stream(rows, d, eps):
    """bfloat16 activations beside a stream kept in 32-bit: the first call makes the stream from
    x, later calls add to it without rounding it, and the stream alone can be normalised."""
    x = rnd(rows, d, dtype=torch.bfloat16, seed=1, scale=3.0)
    y = rnd(rows, d, dtype=torch.bfloat16, seed=2, scale=0.01)          # small against the stream, as a layer's output is
    w = 1 + rnd(d, seed=3, scale=0.1)
    wd = w.to(DEV)
    ref0, ref_stream = plain_ops.add_rmsnorm(x.clone(), None, w, eps, stream_dtype=torch.float32)
    out0, stream = k().add_rmsnorm(x.to(DEV), None, wd, eps, stream_dtype=torch.float32)
    assert stream.dtype == torch.float32 and out0.dtype == torch.bfloat16
    assert torch.equal(stream.cpu(), x.float())
    close(out0, ref0, torch.bfloat16, "norm of the first value")
    for i in range(3):
        ref1, ref_stream = plain_ops.add_rmsnorm(y.clone(), ref_stream, w, eps)
        out1, stream2 = k().add_rmsnorm(y.to(DEV), stream, wd, eps)
        assert stream2.data_ptr() == stream.data_ptr()
        close(stream, ref_stream, torch.float32, "32-bit stream")
        close(out1, ref1, torch.bfloat16, "norm over a 32-bit stream")
    # three additions of a value that bfloat16 would have lost against the stream
    assert (stream.cpu() - x.float() - 3 * y.float()).abs().max() < 1e-5 * x.float().abs().max()
    ref2, _ = plain_ops.add_rmsnorm(None, ref_stream.clone(), w, eps, out_dtype=torch.bfloat16)
    out2, _ = k().add_rmsnorm(None, stream, wd, eps, out_dtype=torch.bfloat16)
    close(out2, ref2, torch.bfloat16, "norm of the stream alone")


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("rows,I", [(1, 176), (7, 512), (3, 200), (65, 8192), (2, 1)])
def test_silu_mul(dtype, rows, I):
    gu = rnd(rows, 2 * I, dtype=dtype, seed=4, scale=4.0)
    close(k().silu_mul(gu.to(DEV)), plain_ops.silu_mul(gu), dtype, "silu_mul")


# ----------------------------------------------------------------------------- matrix products
@pytest.mark.parametrize("M,N,K", [(1, 64, 64), (7, 131, 80), (65, 192, 500), (130, 70, 33), (3, 320, 192), (64, 64, 16)])
@pytest.mark.parametrize("bias", [False, True])
def test_gemm_f32_fixed_order(M, N, K, bias):
    x, w = rnd(M, K, seed=5), rnd(N, K, seed=6)
    b = rnd(N, seed=7) if bias else None
    ref = plain_ops.linear(x, w, b, torch.float64)
    got = k().linear(x.to(DEV), w.to(DEV), b.to(DEV) if bias else None, torch.float32)
    bound = (x.abs().double() @ w.abs().double().t()) * 1.2e-7 * 4 + 1e-30   # a few roundings of the running sum
    assert ((got.cpu().double() - ref).abs() <= bound * (K ** 0.5 + 2)).all()


def test_gemm_f32_result_does_not_depend_on_the_batch():
    """A row's product is bit-identical whether it runs alone or among 100 others."""
    x, w = rnd(101, 300, seed=8).to(DEV), rnd(77, 300, seed=9).to(DEV)
    full = k().linear(x, w, None, torch.float32)
    for r in (0, 50, 100):
        alone = k().linear(x[r:r + 1].contiguous(), w, None, torch.float32)
        assert torch.equal(alone[0], full[r])
    part = k().linear(x[37:90], w, None, torch.float32)       # a strided view of rows
    assert torch.equal(part, full[37:90])


@pytest.mark.parametrize("M,N,K", [(1, 64, 64), (9, 136, 80), (70, 192, 512), (2048, 320, 192)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("bias", [False, True])
def test_linear_bf16(M, N, K, out_dtype, bias):
    x, w = rnd(M, K, dtype=torch.bfloat16, seed=5), rnd(N, K, dtype=torch.bfloat16, seed=6)
    b = rnd(N, seed=7).bfloat16().float() if bias else None
    ref = plain_ops.linear(x, w, b, torch.float64)
    got = k().linear(x.to(DEV), w.to(DEV), b.to(DEV) if bias else None, out_dtype)
    assert got.dtype == out_dtype
    close(got, ref, out_dtype if out_dtype == torch.bfloat16 else torch.float32, "linear", scale=ref.abs().max().item() * 8)


@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (128, 256, 64), (256, 256, 512), (2048, 3072, 2048), (300, 200, 136),
                                   (1, 320, 192), (100, 8, 8), (129, 385, 72), (640, 2048, 8192)])
@pytest.mark.parametrize("bn", [128, 192, 256])
def test_gemm_tcgen05(M, N, K, bn):
    """The tensor-memory product against the plain one: tiles cut by every edge (rows, columns
    and k that are no multiples of 128 / bn / 64), all three tile widths."""
    x, w = rnd(M, K, dtype=torch.bfloat16, seed=21), rnd(N, K, dtype=torch.bfloat16, seed=22, scale=0.05)
    st = status()
    got = k().gemm_tcgen05(x.to(DEV), w.to(DEV), st, bn=bn)
    assert st.tolist()[0] == 0
    close(got, plain_ops.linear(x, w, None, torch.float64), torch.bfloat16, f"tcgen05 product, tile width {bn}")


@pytest.mark.parametrize("M,I,K", [(128, 128, 64), (300, 384, 136), (2048, 1024, 512), (5, 256, 64)])
def test_gemm_tcgen05_epilogues(M, I, K):
    x = rnd(M, K, dtype=torch.bfloat16, seed=31)
    wg, wu = rnd(I, K, dtype=torch.bfloat16, seed=32, scale=0.1), rnd(I, K, dtype=torch.bfloat16, seed=33, scale=0.1)
    blk = k().GATE_UP_BLOCK
    w = torch.stack([wg.view(-1, blk, K), wu.view(-1, blk, K)], dim=1).reshape(2 * I, K).contiguous()
    st = status()
    got = k().gemm_tcgen05(x.to(DEV), w.to(DEV), st, epilogue=k().EPI_SILU_MUL)
    # as the unfused path: both products rounded to bfloat16, then silu(gate) * up
    g = plain_ops.linear(x, wg, None, torch.bfloat16)
    u = plain_ops.linear(x, wu, None, torch.bfloat16)
    ref = plain_ops.silu_mul(torch.cat([g, u], dim=1))
    assert got.shape == (M, I) and st.tolist()[0] == 0
    close(got, ref, torch.bfloat16, "fused SiLU-mul epilogue", extra=2.0 ** -8 * ref.abs().max().item())
    # the same weight through the unfused kernels
    gu = k().linear(x.to(DEV), w.to(DEV), None, torch.bfloat16)
    close(k().silu_mul(gu, blk), ref, torch.bfloat16, "blocked SiLU-mul", extra=2.0 ** -8 * ref.abs().max().item())
    res = rnd(M, 2 * I, dtype=torch.bfloat16, seed=34)
    got = k().gemm_tcgen05(x.to(DEV), w.to(DEV), st, epilogue=k().EPI_RESIDUAL, residual=res.to(DEV))
    ref = (plain_ops.linear(x, w, None, torch.bfloat16).double() + res.double())
    close(got, ref, torch.bfloat16, "residual epilogue", extra=2.0 ** -8 * ref.abs().max().item())


@pytest.mark.parametrize("M", [1, 31, 33, 128, 200, 257])
@pytest.mark.parametrize("epilogue,bn,N", [("EPI_PLAIN", 128, 136), ("EPI_PLAIN", 192, 400), ("EPI_PLAIN", 256, 520), ("EPI_SILU_MUL", 256, 512),
                                           ("EPI_SILU_MUL", 128, 256), ("EPI_GELU_MUL", 256, 256), ("EPI_RELU2", 256, 300), ("EPI_RESIDUAL", 256, 281)])
def test_tcgen05_epilogues_store_the_same_wherever_the_output_lies(M, epilogue, bn, N):
    """Tiles whose rows end inside a warp's, outputs that start on 32, 16 and 2 bytes, a residual that lies likewise or is the output itself:
    the same bits, and nothing beside them is written."""
    x, w = rnd(M, 136, dtype=torch.bfloat16, seed=41).to(DEV), rnd(N, 136, dtype=torch.bfloat16, seed=42, scale=0.1).to(DEV)
    e, n_out, st = getattr(k(), epilogue), N // 2 if epilogue.endswith("_MUL") else N, status()
    res = rnd(M, N, dtype=torch.bfloat16, seed=43).to(DEV) if epilogue == "EPI_RESIDUAL" else None
    base = torch.zeros(M, -(-n_out // 16) * 16, dtype=torch.bfloat16, device=DEV)[:, :n_out]
    k().gemm_tcgen05(x, w, st, epilogue=e, residual=res, bn=bn, out=base)
    product = x.double() @ w.double().t()
    if res is not None:
        close(base, product + res.double(), torch.bfloat16, epilogue, extra=2.0 ** -8 * product.abs().max().item())
    elif epilogue == "EPI_PLAIN":
        close(base, product, torch.bfloat16, epilogue)
    for off, pad in ((0, 16), (8, 8), (1, 3), (16, 16)):
        wide = torch.full((M + 2, off + n_out + pad), 7.0, dtype=torch.bfloat16, device=DEV)
        out = wide[1:M + 1, off:off + n_out]
        if res is not None:
            out.copy_(res)
        k().gemm_tcgen05(x, w, st, epilogue=e, residual=out if res is not None else None, bn=bn, out=out)
        assert torch.equal(out, base), (off, pad)
        assert (wide[0] == 7).all() and (wide[-1] == 7).all() and (wide[:, :off] == 7).all() and (wide[:, off + n_out:] == 7).all()
    assert st.tolist() == [0] * 4


@pytest.mark.parametrize("N", [16, 200, 264])
@pytest.mark.parametrize("used", [1, 130, 300, 384])
def test_grouped_tcgen05_writes_rows_in_use_alone(N, used):
    """32-bit outputs of the grouped product, rows of 16 bytes and not: padding rows between the pairs and rows behind those in use stay as
    they were, columns end inside a group of 16."""
    from fastmlx_b200.kernels import call
    K, experts = 136, 3
    x, w = rnd(384, K, dtype=torch.bfloat16, seed=51).to(DEV), rnd(experts * N, K, dtype=torch.bfloat16, seed=52).to(DEV)
    tile_expert = torch.tensor([2, 0, 1], dtype=torch.int32, device=DEV)
    token = torch.arange(384, dtype=torch.int32, device=DEV)
    token[torch.randperm(384, generator=torch.Generator().manual_seed(used))[:90].to(DEV)] = -1
    n_used, st = torch.tensor([used], dtype=torch.int32, device=DEV), status()
    want = torch.cat([x[128 * t:128 * t + 128].double() @ w[N * e:N * e + N].double().t() for t, e in enumerate((2, 0, 1))])
    rows = (token >= 0) & (torch.arange(384, device=DEV) < used)
    for ldc in (-(-N // 4) * 4, N + 1, N + 12):
        c = torch.full((384, ldc), 7.0, device=DEV)
        call("tc", "fmx_grouped_tcgen05", x.data_ptr(), x.stride(0), w.data_ptr(), w.stride(0), c.data_ptr(), ldc, 384, N, K, experts, n_used.data_ptr(),
             tile_expert.data_ptr(), token.data_ptr(), None, 0.0, 0, 0, st.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert (c[~rows] == 7).all() and (c[:, N:] == 7).all()
        close(c[rows][:, :N], want[rows], torch.float32, "grouped product", scale=8 * want.abs().max().item())
    assert st.tolist() == [0] * 4


@pytest.mark.parametrize("M", [1, 2, 7, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(16, 32), (64, 64), (131, 80), (3072, 2048), (2048, 8192), (50, 8), (320, 192), (17, 1000)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemv(M, N, K, out_dtype):
    """The product with the whole of K in one block: every row count up to 16, widths that are
    no multiple of the 32-wide k block or of the 8-feature tile, bias, residual in place, both
    tile widths."""
    x, w = rnd(M, K, dtype=torch.bfloat16, seed=11), rnd(N, K, dtype=torch.bfloat16, seed=12, scale=0.05)
    b = rnd(N, seed=13) if N % 2 else None
    ref = plain_ops.linear(x, w, b, torch.float64)
    scale = ref.abs().max().item() * 8 if out_dtype == torch.float32 else None
    xd, wd, bd = x.to(DEV), w.to(DEV), b.to(DEV) if b is not None else None
    for wide, warps in ((8, 8), (16, 8), (32, 8), (8, 16), (16, 16)):
        got = k().gemv(xd, wd, bd, out_dtype, wide=wide, warps=warps)
        close(got, ref, out_dtype, "gemv", scale=scale)
        alone = k().gemv(xd[M - 1:].contiguous(), wd, bd, out_dtype, wide=wide, warps=warps)
        if M <= 8:                                       # rows 8..15 sit in another accumulator half
            assert torch.equal(alone[0], got[M - 1])     # a row's result does not depend on its companions
    if out_dtype == torch.bfloat16:
        res = rnd(M, N, dtype=torch.bfloat16, seed=44)
        stream = res.clone().to(DEV)
        out = k().gemv(xd, wd, residual=stream, out=stream)
        assert out.data_ptr() == stream.data_ptr()
        want = plain_ops.linear(x, w, None, torch.bfloat16).double() + res.double()
        close(stream, want, torch.bfloat16, "gemv residual epilogue", extra=2.0 ** -8 * want.abs().max().item())


@pytest.mark.parametrize("M", [1, 8, 13])
@pytest.mark.parametrize("I,K,blk", [(128, 64, 128), (8192, 2048, 128), (384, 200, 128), (64, 72, 32), (48, 40, 16)])
def test_gemv_gate_up(M, I, K, blk):
    x = rnd(M, K, dtype=torch.bfloat16, seed=51, scale=2.0)
    wg, wu = rnd(I, K, dtype=torch.bfloat16, seed=52, scale=0.1), rnd(I, K, dtype=torch.bfloat16, seed=53, scale=0.1)
    w = torch.stack([wg.view(-1, blk, K), wu.view(-1, blk, K)], dim=1).reshape(2 * I, K).contiguous()
    g = plain_ops.linear(x, wg, None, torch.bfloat16)
    u = plain_ops.linear(x, wu, None, torch.bfloat16)
    ref = plain_ops.silu_mul(torch.cat([g, u], dim=1))
    for wide in (8, 16, 32):
        if blk % wide:
            continue
        got = k().gemv(x.to(DEV), w.to(DEV), block=blk, wide=wide)
        assert got.shape == (M, I)
        close(got, ref, torch.bfloat16, "gemv gate/up with SiLU-mul", extra=2.0 ** -7 * ref.abs().max().item())


@pytest.mark.parametrize("M,N,K,bias", [(1, 1, 4, False), (1, 4800, 68, True), (4, 33, 60, False), (5, 15, 64, True), (16, 4737, 132, False),
                                        (17, 31, 2048, False), (32, 130, 196, True), (33, 1, 4, False), (33, 65, 20, True),
                                        (64, 127, 2052, False), (65, 16384, 36, False), (200, 2048, 52, True), (333, 130, 16, False)])
def test_gemm_simple_32bit_kernels_sum_in_one_order(M, N, K, bias):
    """32-bit operands in 16-byte rows take kernels of their own (by rows of x, features and SMs); rows that start elsewhere take
    the general one.  All sum an output's products one after the other: the results are equal, and right."""
    x, w = torch.randn(M, K), torch.randn(N, K)
    b = torch.randn(N).to(DEV) if bias else None
    odd = lambda t: torch.cat([t, t[:, :1]], 1).to(DEV)[:, :K]             # rows of K + 1 floats: no 16-byte rows
    got = k().gemm_simple(x.to(DEV), w.to(DEV), b, torch.float32)
    assert torch.equal(got, k().gemm_simple(odd(x), odd(w), b, torch.float32))
    close(got, plain_ops.linear(x, w, None if b is None else b.cpu(), torch.float64), torch.float32, "gemm_simple", scale=None)


@pytest.mark.parametrize("N,K,bias", [(1, 8, True), (127, 72, False), (129, 64, True), (200, 520, False), (130, 2056, True), (2048, 8192, False),
                                      (16384, 256, False), (24000, 512, True)])
def test_gemm_three_does_not_depend_on_the_batch(N, K, bias):
    """32-bit rows against a bfloat16 matrix on the tensor cores: a row's result is the same bits whatever the number of rows (tiles of 16
    to 128 tokens, K walked whole or in a cluster's shares), and as far from 64-bit as 32-bit sums are: up to 16 sums of the tensor cores
    that are cut off, 2^-23 of what was summed each, and half of that for each rounded sum of the blocks of 64.  All together they are
    closer, since roundings of either sign meet: 2^-21.5 = 3.4e-7 of the norm, twice what was measured (1.6e-7 at most) and a seventh of the
    2.4e-6 that the activations' first two terms alone leave in exact arithmetic."""
    x, w = torch.randn(300, K), rnd(N, K, dtype=torch.bfloat16, seed=11)
    b = torch.randn(N).to(DEV) if bias else None
    xd, wd = x.to(DEV), w.to(DEV)
    full = k().linear(xd, wd, b, torch.float32)
    ref = plain_ops.linear(x, w.float(), None if b is None else b.cpu(), torch.float64)
    room = (x.abs().double() @ w.abs().double().t() + (0 if b is None else b.cpu().abs().double())) * 2.0 ** -23 * (16 + K / 128)
    assert ((full.cpu().double() - ref).abs() <= room).all()
    assert (full.cpu().double() - ref).norm() <= 2.0 ** -21.5 * ref.norm()
    for a, m in ((0, 1), (0, 16), (5, 17), (100, 64), (7, 128), (40, 129), (3, 257)):
        assert torch.equal(k().linear(xd[a:a + m], wd, b, torch.float32), full[a:a + m]), m
    odd = torch.cat([x, x[:, :1]], 1).to(DEV)[:, :K]                       # rows that do not start on 16 bytes
    assert torch.equal(k().linear(odd, wd, b, torch.float32), full)
    assert int(k()._status_word(DEV)[0]) == 0


@pytest.mark.parametrize("M", [1, 17, 200])
@pytest.mark.parametrize("N,K,cuts", [(6160, 2048, (0, 6144, 6160)), (1032, 8192, (0, 8, 700, 1032)), (300, 520, (0, 1, 299, 300))])
def test_gemm_three_over_some_rows_of_a_matrix(N, K, cuts, M):
    """The product over some of a matrix's rows takes the whole matrix's shares of K: the bits that the whole product gives those features
    (6,160 x 2,048: 2 shares, its last 16 rows by themselves would take 4)."""
    x, w = torch.randn(M, K, device=DEV), rnd(N, K, dtype=torch.bfloat16, seed=14).to(DEV)
    whole = k().gemm_three(x, w)
    for a, b in zip(cuts, cuts[1:]):
        assert torch.equal(k().gemm_three(x, w[a:b], whole=N), whole[:, a:b]), (a, b)


@pytest.mark.parametrize("N,bias", [(130, True), (2048, False)])
def test_gemm_three_in_waves(N, bias):
    """More tokens than the workspace holds terms of: each the bits it has by itself, on both sides of a wave's end."""
    from fastmlx_b200.kernels.lib import load
    K = 14336
    rows = load("tc").fmx_gemm_three_rows(K)
    x, w = torch.randn(2 * rows + 77, K, device=DEV), rnd(N, K, dtype=torch.bfloat16, seed=16).to(DEV)
    b = torch.randn(N, device=DEV) if bias else None
    full = k().gemm_three(x, w, b)
    for a, m in ((0, 130), (rows - 3, 7), (rows - 1, 1), (2 * rows - 20, 97)):
        assert torch.equal(k().gemm_three(x[a:a + m], w, b), full[a:a + m]), a


def test_gemm_three_infinite_and_huge_activations():
    """An infinity or a NaN stays in its row; values that would round to an infinity in bfloat16 do not."""
    x, w = torch.randn(40, 192), rnd(70, 192, dtype=torch.bfloat16, seed=12)
    x[3, 5], x[9, 0], x[17, 100] = math.inf, -math.inf, math.nan
    x[21] *= 1e-3
    x[21, 7] = 3.4e38
    w[:, 7] = w[:, 7].abs().clamp(0.25, 0.5)
    got = k().linear(x.to(DEV), w.to(DEV), None, torch.float32).cpu()
    ref = x.double() @ w.double().t()
    assert torch.equal(torch.isnan(got), torch.isnan(ref)) and torch.equal(torch.isinf(got), torch.isinf(ref))
    assert torch.equal(got[[3, 9]].sign(), ref[[3, 9]].float().sign())
    fin = torch.isfinite(ref)
    assert ((got.double() - ref).abs()[fin] <= 2.0 ** -19 * (x.double().abs().nan_to_num(posinf=0) @ w.double().abs().t())[fin]).all()


@pytest.mark.parametrize("M,N,K,bias", [(1, 70, 2048, False), (40, 300, 2048, True), (130, 16390, 1096, False), (300, 140, 2056, True)])
def test_linear_with_weights_that_are_not_finite(M, N, K, bias):
    """32-bit rows against a bfloat16 matrix that holds infinities and a NaN: what 64-bit arithmetic gives, an infinity of the right sign and no
    NaN but where an infinity meets a zero, another infinity or a NaN; the other features are the same bits as without them."""
    x, w = torch.randn(M, K), rnd(N, K, dtype=torch.bfloat16, seed=15)
    x[:, 9] = x[:, 9].bfloat16().float()                                   # smaller terms that are zeros
    x[0, 9] = 0.0
    b = torch.randn(N) if bias else None
    bad = w.clone()
    bad[3, 5], bad[60, 9], bad[N - 1, K - 1] = math.inf, -math.inf, math.inf
    bad[7, 100], bad[12, 0], bad[12, 1] = math.nan, math.inf, -math.inf
    run = lambda m: k().linear(x.to(DEV), m.to(DEV), None if b is None else b.to(DEV), torch.float32).cpu()
    got, clean, ref = run(bad), run(w), plain_ops.linear(x, bad.double(), b, torch.float64)
    odd = torch.tensor([3, 7, 12, 60, N - 1])
    assert torch.equal(torch.isnan(got), torch.isnan(ref)) and torch.equal(torch.isinf(got), torch.isinf(ref))
    assert torch.equal(got[:, odd].nan_to_num().sign(), ref[:, odd].nan_to_num().float().sign())
    rest = torch.ones(N, dtype=torch.bool)
    rest[odd] = False
    assert torch.equal(got[:, rest], clean[:, rest])


@pytest.mark.parametrize("ta,tw,tc", [(torch.bfloat16, torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32, torch.float32),
                                      (torch.bfloat16, torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16, torch.bfloat16)])
def test_gemm_simple_mixed_types(ta, tw, tc):
    x, w = rnd(19, 70, dtype=ta, seed=1), rnd(45, 70, dtype=tw, seed=2)
    got = k().gemm_simple(x.to(DEV), w.to(DEV), None, tc)
    close(got, plain_ops.linear(x, w, None, torch.float64), tc, "gemm_simple", scale=None)


# ----------------------------------------------------------------------------- rope + cache write
def _paged(n_rows, lens, page_size, num_pages, seed=0):
    """Block tables that scatter each row's pages over the pool in a shuffled order."""
    g = torch.Generator().manual_seed(seed)
    perm = torch.randperm(num_pages, generator=g).tolist()
    max_blocks = max(-(-n // page_size) for n in lens)
    bt = torch.full((n_rows, max_blocks + 1), -1, dtype=torch.int32)
    for r, n in enumerate(lens):
        for b in range(-(-n // page_size)):
            bt[r, b] = perm.pop()
    return bt


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nh,nkv,hd,rot,trad", [(4, 2, 16, 16, False), (6, 3, 32, 32, False), (5, 1, 48, 48, True),
                                                 (8, 2, 64, 32, False), (3, 3, 128, 128, False), (2, 1, 80, 40, True),
                                                 (4, 0, 32, 32, False), (4, 2, 32, 0, False)])
def test_rope_kv_write(dtype, nh, nkv, hd, rot, trad):
    T, page_size, num_pages = 23, 8, 9
    qkv = rnd(T, (nh + 2 * nkv) * hd, dtype=dtype, seed=1)
    positions = torch.tensor([0, 1, 2, 3, 63, 64, 65, 500, 8191, 8192, 100000, 131071] + list(range(7, 18)), dtype=torch.int32)
    inv_freq = (10000.0 ** (-torch.arange(0, max(rot, 2), 2, dtype=torch.float64) / max(rot, 2))).float()
    slots = torch.randperm(num_pages * page_size, generator=torch.Generator().manual_seed(2))[:T].long()
    slots[5] = -1                                                # a padding token is stored nowhere
    kv_ref = torch.zeros(num_pages, 2, max(nkv, 1), page_size, hd, dtype=dtype)
    kv_dev = kv_ref.clone().to(DEV)
    q_ref = qkv.clone()
    st_ref = torch.zeros(4, dtype=torch.int32)
    plain_ops.rope_kv_write(q_ref, positions, inv_freq, rot, trad, slots, kv_ref if nkv else None, nh, nkv, hd, st_ref)
    q_dev = qkv.clone().to(DEV)
    st = status()
    k().rope_kv_write(q_dev, positions.to(DEV), inv_freq.to(DEV), rot, trad, slots.to(DEV), kv_dev if nkv else None,
                      nh, nkv, hd, st)
    assert st.tolist()[0] == 0
    close(q_dev, q_ref, dtype, "rotated qkv")
    close(kv_dev, kv_ref, dtype, "pages", scale=1.0)


def test_rope_bad_slot_leaves_code():
    qkv = rnd(2, 4 * 16).to(DEV)
    kv = torch.zeros(2, 2, 1, 4, 16, device=DEV)
    st = status()
    k().rope_kv_write(qkv, torch.zeros(2, dtype=torch.int32, device=DEV), torch.ones(8, device=DEV), 16, False,
                      torch.tensor([0, 99], device=DEV), kv, 2, 1, 16, st)
    assert st.tolist()[:2] == [k().BAD_SLOT, 99]


# ----------------------------------------------------------------------------- attention over pages
def _attention_case(dtype, nh, nkv, hd, page_size, rows, window=0, seed=0, spike=None):
    """rows: list of (ctx_before, q_len).  Pages are filled for every position < ctx+q."""
    lens = [c + q for c, q in rows]
    num_pages = sum(-(-n // page_size) for n in lens) + 3
    bt = _paged(len(rows), lens, page_size, num_pages, seed)
    g = torch.Generator().manual_seed(seed + 1)
    kv = torch.randn(num_pages, 2, nkv, page_size, hd, generator=g).to(dtype)
    T = sum(q for _, q in rows)
    q = torch.randn(T, nh * hd, generator=g).to(dtype)
    pos, trow = [], []
    for r, (c, ql) in enumerate(rows):
        pos += list(range(c, c + ql))
        trow += [r] * ql
    if spike is not None:
        # One far key is made to stand out for one query: the query and that key are scaled
        # along a common direction so its score dominates, and its value row is marked.
        t, key_pos, head = spike
        r = trow[t]
        page = int(bt[r, key_pos // page_size])
        gk = head // (nh // nkv)
        d = torch.randn(hd, generator=g)
        d = d / d.norm()
        q[t, head * hd:(head + 1) * hd] = (d * 12.0).to(dtype)
        kv[page, 0, gk, key_pos % page_size] = (d * 12.0).to(dtype)
        kv[page, 1, gk, key_pos % page_size] = torch.full((hd,), 7.0).to(dtype)
    ctx = SimpleNamespace(positions=torch.tensor(pos, dtype=torch.int32), token_row=torch.tensor(trow, dtype=torch.int32),
                          status=torch.zeros(4, dtype=torch.int32))
    grp = SimpleNamespace(block_tables=bt)
    return q, kv, ctx, grp


def _to_dev(ctx, grp):
    return (SimpleNamespace(positions=ctx.positions.to(DEV), token_row=ctx.token_row.to(DEV), status=status(),
                            all_decode=False, max_q_len=0, max_ctx_after=0, row_start=None, row_ctx=None, R=grp.block_tables.shape[0], scratch={}),
            SimpleNamespace(block_tables=grp.block_tables.to(DEV), page_size=None))


ATT_SHAPES = [(4, 2, 16, 16), (6, 3, 32, 16), (5, 1, 48, 8), (8, 8, 64, 32), (12, 4, 128, 64), (3, 3, 80, 16), (2, 1, 256, 16)]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nh,nkv,hd,page_size", ATT_SHAPES)
@pytest.mark.parametrize("window", [0, 24])
def test_paged_attention_simple_mixed_rows(dtype, nh, nkv, hd, page_size, window):
    rows = [(0, 37), (90, 1), (31, 2), (0, 1), (15, 17), (64, 1)]
    q, kv, ctx, grp = _attention_case(dtype, nh, nkv, hd, page_size, rows, window)
    ref = plain_ops.paged_attention(q, kv, ctx, grp, nh, nkv, hd, hd ** -0.5, window)
    dctx, dgrp = _to_dev(ctx, grp)
    got = k().paged_attention_simple(q.to(DEV), kv.to(DEV), dctx, dgrp, nh, nkv, hd, hd ** -0.5, window)
    assert dctx.status.tolist()[0] == 0
    close(got, ref, dtype, "attention", scale=1.0)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("key_pos", [0, 15, 16, 17, 31, 32, 63, 64, 511, 512, 700])
def test_paged_attention_simple_far_key_stands_out(dtype, key_pos):
    """Among 701 keys one is made dominant; a kernel that misses it (a page's edge, a
    chunk's edge) returns something far from its marked value."""
    nh, nkv, hd, page_size = 4, 2, 32, 16
    rows = [(700, 1), (0, 5)]
    q, kv, ctx, grp = _attention_case(dtype, nh, nkv, hd, page_size, rows, spike=(0, key_pos, 3))
    dctx, dgrp = _to_dev(ctx, grp)
    got = k().paged_attention_simple(q.to(DEV), kv.to(DEV), dctx, dgrp, nh, nkv, hd, 1.0, 0)
    ref = plain_ops.paged_attention(q, kv, ctx, grp, nh, nkv, hd, 1.0, 0)
    assert (ref[0, 3 * hd:4 * hd].float() - 7.0).abs().max() < 0.1
    close(got, ref, dtype, "attention with a dominant key", scale=7.0)


@pytest.mark.parametrize("dtype", DTYPES)
def test_paged_attention_simple_window_edge(dtype):
    """The key just outside a window must not count even when it would dominate; the one
    just inside must."""
    nh, nkv, hd, page_size, window = 2, 1, 32, 16, 40
    for key_pos, inside in ((100 - 40, False), (100 - 39, True)):
        rows = [(100, 1)]
        q, kv, ctx, grp = _attention_case(dtype, nh, nkv, hd, page_size, rows, window, spike=(0, key_pos, 1))
        dctx, dgrp = _to_dev(ctx, grp)
        got = k().paged_attention_simple(q.to(DEV), kv.to(DEV), dctx, dgrp, nh, nkv, hd, 1.0, window)
        ref = plain_ops.paged_attention(q, kv, ctx, grp, nh, nkv, hd, 1.0, window)
        assert ((ref[0, hd:].float() - 7.0).abs().max() < 0.1) == inside
        close(got, ref, dtype, "window edge", scale=7.0)


def test_paged_attention_never_reads_unseen_keys():
    """Pages hold NaN wherever a key is not visible: the result must stay finite."""
    nh, nkv, hd, page_size = 4, 2, 32, 16
    rows = [(20, 3), (0, 9)]
    q, kv, ctx, grp = _attention_case(torch.float32, nh, nkv, hd, page_size, rows)
    lens = [c + ql for c, ql in rows]
    poisoned = torch.full_like(kv, float("nan"))
    for r, n in enumerate(lens):
        for j in range(n):
            p = int(grp.block_tables[r, j // page_size])
            poisoned[p, :, :, j % page_size] = kv[p, :, :, j % page_size]
    dctx, dgrp = _to_dev(ctx, grp)
    got = k().paged_attention_simple(q.to(DEV), poisoned.to(DEV), dctx, dgrp, nh, nkv, hd, hd ** -0.5, 0)
    ref = plain_ops.paged_attention(q, kv, ctx, grp, nh, nkv, hd, hd ** -0.5, 0)
    assert torch.isfinite(got).all()
    close(got, ref, torch.float32, "attention", scale=1.0)


def _full_ctx(rows, ctx, grp):
    """A device step context with the row arrays the tiled kernels read."""
    starts, at = [], 0
    for _, ql in rows:
        starts.append(at)
        at += ql
    starts.append(at)
    d, g = _to_dev(ctx, grp)
    d.row_start = torch.tensor(starts, dtype=torch.int32, device=DEV)
    d.row_ctx = torch.tensor([c for c, _ in rows], dtype=torch.int32, device=DEV)
    d.max_q_len = max(ql for _, ql in rows)
    d.max_ctx_after = max(c + ql for c, ql in rows)
    d.all_decode = all(ql == 1 for _, ql in rows)
    d.R = len(rows)
    d.n_splits = 0
    return d, g


# The tiled kernels hand the probabilities to the tensor cores in bfloat16: each p_j carries a
# relative error of 2^-9, so sum_j p_j v_j is off by at most 2^-9 * max|v| on top of the
# rounding of the result itself.
P_ROUNDING = 2.0 ** -9

TILED_SHAPES = [(4, 2, 16, 16), (6, 3, 32, 16), (5, 1, 48, 8), (8, 8, 64, 32), (32, 8, 64, 16), (12, 4, 128, 64),
                (24, 8, 128, 16), (3, 3, 80, 16), (2, 1, 256, 16), (16, 1, 96, 128),
                (12, 1, 64, 16),      # more than 8 query heads to a kv head at a head size with both decode tiles
                (6, 2, 32, 12)]       # pages of no power of two


@pytest.mark.parametrize("nh,nkv,hd,page_size", TILED_SHAPES)
@pytest.mark.parametrize("window", [0, 24, 100])
def test_tiled_prefill_attention_mixed_rows(nh, nkv, hd, page_size, window):
    """Portions of prompts with and without earlier context, single tokens, tiles that end in
    the middle of a portion, rows that span several 64-row and 64-key tiles."""
    rows = [(0, 37), (90, 1), (31, 2), (0, 1), (15, 17), (64, 1), (200, 130), (0, 64), (63, 65)]
    q, kv, ctx, grp = _attention_case(torch.bfloat16, nh, nkv, hd, page_size, rows, window)
    ref = plain_ops.paged_attention(q, kv, ctx, grp, nh, nkv, hd, hd ** -0.5, window)
    dctx, dgrp = _full_ctx(rows, ctx, grp)
    got = k().paged_attention_prefill(q.to(DEV), kv.to(DEV), dctx, dgrp, nh, nkv, hd, hd ** -0.5, window)
    assert dctx.status.tolist()[0] == 0
    close(got, ref, torch.bfloat16, "tiled prefill attention", scale=1.0, extra=P_ROUNDING * kv.abs().max().item())


@pytest.mark.parametrize("nh,nkv,hd,page_size", TILED_SHAPES + [(8, 2, 64, 16), (8, 2, 128, 16)])
@pytest.mark.parametrize("window", [0, 70])
@pytest.mark.parametrize("portion", [17, 130])
def test_mixed_step_attention_takes_two_kernels(nh, nkv, hd, page_size, window, portion):
    """A step whose first rows decode and whose last rows are portions: the dispatch hands the
    decoding rows to the split kernel and the rest to a tiled one (the tensor-memory kernel for
    the 130-token portion where it takes the sizes), into one output, and a single token among
    the portions stays with them."""
    from fastmlx_b200.engine.batch import leading_decode_rows
    rows = [(300, 1), (1000, 1), (63, 1), (0, 1), (0, portion), (90, 1), (31, 2), (200, portion)]
    q, kv, ctx, grp = _attention_case(torch.bfloat16, nh, nkv, hd, page_size, rows, window)
    ref = plain_ops.paged_attention(q, kv, ctx, grp, nh, nkv, hd, hd ** -0.5, window)
    dctx, dgrp = _full_ctx(rows, ctx, grp)
    for name, value in leading_decode_rows([ql for _, ql in rows], [c for c, _ in rows]).items():
        setattr(dctx, name, value)
    assert dctx.decode_rows == 4 and dctx.decode_max_ctx == 1001 and dctx.rest_max_q_len == portion \
        and dctx.rest_max_ctx == 200 + portion
    dctx.scratch = {}
    before = k().launch_count()
    got = k().paged_attention(q.to(DEV), kv.to(DEV), dctx, dgrp, nh, nkv, hd, hd ** -0.5, window)
    assert k().launch_count() - before == 2 and dctx.status.tolist()[0] == 0
    close(got, ref, torch.bfloat16, "mixed step attention", scale=1.0, extra=P_ROUNDING * kv.abs().max().item())


@pytest.mark.parametrize("nh,nkv,hd,page_size", TILED_SHAPES)
@pytest.mark.parametrize("window", [0, 70])
@pytest.mark.parametrize("splits", [1, 2, 5, 8, 9, 32])
def test_split_decode_attention(nh, nkv, hd, page_size, window, splits):
    rows = [(0, 1), (1, 1), (63, 1), (64, 1), (65, 1), (300, 1), (1000, 1), (127, 1)]
    q, kv, ctx, grp = _attention_case(torch.bfloat16, nh, nkv, hd, page_size, rows, window)
    ref = plain_ops.paged_attention(q, kv, ctx, grp, nh, nkv, hd, hd ** -0.5, window)
    dctx, dgrp = _full_ctx(rows, ctx, grp)
    got = k().paged_attention_decode(q.to(DEV), kv.to(DEV), dctx, dgrp, nh, nkv, hd, hd ** -0.5, window, splits=splits)
    assert dctx.status.tolist()[0] == 0
    close(got, ref, torch.bfloat16, "split decode attention", scale=1.0, extra=P_ROUNDING * kv.abs().max().item())
    # up to 8 splits are one thread-block cluster; the same through L2 and tickets, as where no cluster fits
    was = k().decode_attention_clusters(hd, False)
    try:
        again = k().paged_attention_decode(q.to(DEV), kv.to(DEV), dctx, dgrp, nh, nkv, hd, hd ** -0.5, window, splits=splits)
    finally:
        k().decode_attention_clusters(hd, was)
    assert was and dctx.status.tolist()[0] == 0
    close(again, ref, torch.bfloat16, "split decode attention through tickets", scale=1.0, extra=P_ROUNDING * kv.abs().max().item())
    if splits <= 8:
        assert torch.equal(again, got)          # both sum the splits in split order


@pytest.mark.parametrize("seed", range(24))
def test_split_decode_attention_on_random_shapes(seed):
    """Shapes drawn at random: head sizes, heads per kv head up to 16, pages of any size, rows of
    any length with and without a window, every way of splitting (one block, a cluster of up to 8,
    tickets), and the planner's own choice."""
    import random
    rng = random.Random(1000 + seed)
    hd = rng.choice([16, 32, 48, 64, 64, 80, 96, 128, 128])
    nkv = rng.choice([1, 2, 3, 8])
    rep = rng.choice([1, 2, 4, 4, 5, 8, 9, 16])
    nh = nkv * rep
    page_size = rng.choice([4, 8, 12, 16, 16, 32, 64])
    rows = [(rng.choice([0, 1, 15, 16, 17, 63, 64, 65, rng.randrange(100, 3000)]), 1) for _ in range(rng.randint(1, 6))]
    window = rng.choice([0, 0, rng.randrange(1, 200)])
    q, kv, ctx, grp = _attention_case(torch.bfloat16, nh, nkv, hd, page_size, rows, window, seed=seed)
    ref = plain_ops.paged_attention(q, kv, ctx, grp, nh, nkv, hd, hd ** -0.5, window)
    dctx, dgrp = _full_ctx(rows, ctx, grp)
    for splits in (None, 1, rng.randint(2, 8), rng.randint(9, 40)):
        got = k().paged_attention_decode(q.to(DEV), kv.to(DEV), dctx, dgrp, nh, nkv, hd, hd ** -0.5, window, splits=splits)
        assert dctx.status.tolist()[0] == 0
        close(got, ref, torch.bfloat16, f"decode attention nh={nh} nkv={nkv} hd={hd} page={page_size} window={window} "
              f"rows={rows} splits={splits}", scale=1.0, extra=P_ROUNDING * kv.abs().max().item())


@pytest.mark.parametrize("nh,nkv,hd,page_size", TILED_SHAPES)
@pytest.mark.parametrize("rot_frac,traditional", [(1.0, False), (0.5, False), (1.0, True), (0.0, False)])
@pytest.mark.parametrize("splits", [1, 3])
def test_decode_attention_rotates_and_stores_by_itself(nh, nkv, hd, page_size, rot_frac, traditional, splits):
    """The decode kernel given q, k, v as the projection left them: the same bits, in its
    output and in the cache, as the rotary kernel followed by the decode kernel."""
    rows = [(0, 1), (1, 1), (63, 1), (64, 1), (65, 1), (300, 1), (1000, 1), (127, 1)]
    _, kv, ctx, grp = _attention_case(torch.bfloat16, nh, nkv, hd, page_size, rows, 0)
    rot = int(hd * rot_frac) // 2 * 2
    inv = (10000.0 ** (-torch.arange(0, rot, 2, dtype=torch.float64) / max(rot, 1))).float().to(DEV) if rot else None
    qkv = rnd(len(rows), (nh + 2 * nkv) * hd, dtype=torch.bfloat16, seed=77).to(DEV)
    dctx, dgrp = _full_ctx(rows, ctx, grp)
    bt = grp.block_tables
    slots = torch.tensor([int(bt[r, c // page_size]) * page_size + c % page_size for r, (c, _) in enumerate(rows)],
                         dtype=torch.int64, device=DEV)
    # the two kernels
    qkv_a, kv_a = qkv.clone(), kv.to(DEV).clone()
    k().rope_kv_write(qkv_a, dctx.positions, inv, rot, traditional, slots, kv_a, nh, nkv, hd, dctx.status)
    want = k().paged_attention_decode(qkv_a, kv_a, dctx, dgrp, nh, nkv, hd, hd ** -0.5, 0, splits=splits)
    # the one
    qkv_b, kv_b = qkv.clone(), kv.to(DEV).clone()
    got = k().paged_attention_decode(qkv_b, kv_b, dctx, dgrp, nh, nkv, hd, hd ** -0.5, 0, splits=splits,
                                     rope=(inv, rot, traditional, True))
    assert dctx.status.tolist()[0] == 0
    assert torch.equal(kv_a, kv_b), "the cache holds other bits"
    assert torch.equal(got, want)
    assert torch.equal(qkv_b, qkv), "the fused kernel must leave qkv alone"
    # queries only (a layer that reads another layer's cache): the cache stays as it is
    kv_c = kv_a.clone()
    got_q = k().paged_attention_decode(qkv.clone(), kv_c, dctx, dgrp, nh, nkv, hd, hd ** -0.5, 0, splits=splits,
                                       rope=(inv, rot, traditional, False))
    assert torch.equal(kv_c, kv_a) and torch.equal(got_q, want)


TC_SHAPES = [(4, 1, 64, 16), (8, 2, 64, 16), (32, 8, 64, 16), (8, 8, 64, 32), (16, 1, 64, 128), (8, 2, 128, 16),
             (24, 24, 128, 64), (16, 2, 128, 8), (24, 8, 128, 16), (6, 2, 64, 16), (5, 1, 64, 32), (7, 1, 128, 16)]


@pytest.mark.parametrize("variant", [0, 1, 2])
@pytest.mark.parametrize("nh,nkv,hd,page_size", TC_SHAPES)
def test_tensor_memory_prefill_attention(nh, nkv, hd, page_size, variant):
    """The tcgen05 attention kernel on portions with and without earlier context, single
    tokens, rows that end inside a 128-row tile and inside a 128-key tile."""
    rows = [(0, 37), (90, 1), (31, 2), (0, 1), (15, 17), (64, 1), (200, 130), (0, 128), (127, 129), (0, 300)]
    q, kv, ctx, grp = _attention_case(torch.bfloat16, nh, nkv, hd, page_size, rows)
    ref = plain_ops.paged_attention(q, kv, ctx, grp, nh, nkv, hd, hd ** -0.5, 0)
    dctx, dgrp = _full_ctx(rows, ctx, grp)
    assert k().tc_attention_ok(nh, nkv, hd, page_size, 0)
    # variant 0: the library's choice; 1: one query tile per CTA; 2: two where the page size allows that kernel
    got = k().paged_attention_prefill_tc(q.to(DEV), kv.to(DEV), dctx, dgrp, nh, nkv, hd, hd ** -0.5, variant=variant)
    assert dctx.status.tolist()[0] == 0
    close(got, ref, torch.bfloat16, "tensor-memory attention", scale=1.0, extra=P_ROUNDING * kv.abs().max().item())


@pytest.mark.parametrize("ksplits", [2, 3, 4])
@pytest.mark.parametrize("nh,nkv,hd,page_size", [s for s in TC_SHAPES if (128 if s[2] == 64 else 64) % s[3] == 0])
def test_tensor_memory_attention_shares_keys_out(nh, nkv, hd, page_size, ksplits):
    """The keys of a pair of query tiles shared out over several CTAs and combined by a second
    kernel: rows whose keys end in the first share (the others then bring nothing), rows that
    reach into every share, a portion behind a long context, single tokens."""
    rows = [(0, 37), (1500, 130), (90, 1), (700, 2), (0, 300), (2000, 64), (64, 1)]
    q, kv, ctx, grp = _attention_case(torch.bfloat16, nh, nkv, hd, page_size, rows)
    ref = plain_ops.paged_attention(q, kv, ctx, grp, nh, nkv, hd, hd ** -0.5, 0)
    dctx, dgrp = _full_ctx(rows, ctx, grp)
    got = k().paged_attention_prefill_tc(q.to(DEV), kv.to(DEV), dctx, dgrp, nh, nkv, hd, hd ** -0.5, variant=2, ksplits=ksplits)
    assert dctx.status.tolist()[0] == 0
    close(got, ref, torch.bfloat16, f"tensor-memory attention, keys in {ksplits} shares", scale=1.0,
          extra=P_ROUNDING * kv.abs().max().item())
    # one long portion alone: the library plans the shares itself
    rows = [(3000, 200)]
    q, kv, ctx, grp = _attention_case(torch.bfloat16, nh, nkv, hd, page_size, rows, seed=3, spike=(150, 40, nh - 1))
    ref = plain_ops.paged_attention(q, kv, ctx, grp, nh, nkv, hd, hd ** -0.5, 0)
    dctx, dgrp = _full_ctx(rows, ctx, grp)
    from fastmlx_b200.kernels.lib import load
    planned = load(f"attn_hd{hd}").fmx_attn_prefill_tc_plan_splits(1, 200, 3200, nh, nkv, k().num_sms())
    assert planned > 1
    got = k().paged_attention_prefill_tc(q.to(DEV), kv.to(DEV), dctx, dgrp, nh, nkv, hd, hd ** -0.5)
    assert dctx.status.tolist()[0] == 0
    close(got, ref, torch.bfloat16, "tensor-memory attention, planned shares, a far key that stands out", scale=1.0,
          extra=P_ROUNDING * kv.abs().max().item())


@pytest.mark.parametrize("variant", [1, 2])
@pytest.mark.parametrize("key_pos", [0, 15, 16, 127, 128, 129, 255, 256, 511, 700])
def test_tensor_memory_attention_far_key_and_unseen_keys(key_pos, variant):
    """One key among 701 dominates for one head (a tile edge or a page edge that loses it shows
    at once); pages hold NaN wherever a key is out of sight."""
    nh, nkv, hd, page_size = 8, 2, 64, 16
    rows = [(636, 65), (0, 70)]
    q, kv, ctx, grp = _attention_case(torch.bfloat16, nh, nkv, hd, page_size, rows, spike=(64, key_pos, 5))
    ref = plain_ops.paged_attention(q, kv, ctx, grp, nh, nkv, hd, 1.0, 0)
    assert (ref[64, 5 * hd:6 * hd].float() - 7.0).abs().max() < 0.1
    poisoned = torch.full_like(kv, float("nan"))
    for r, (c, ql) in enumerate(rows):
        for j in range(c + ql):
            p = int(grp.block_tables[r, j // page_size])
            poisoned[p, :, :, j % page_size] = kv[p, :, :, j % page_size]
    dctx, dgrp = _full_ctx(rows, ctx, grp)
    got = k().paged_attention_prefill_tc(q.to(DEV), poisoned.to(DEV), dctx, dgrp, nh, nkv, hd, 1.0, variant=variant)
    assert torch.isfinite(got).all()
    close(got, ref, torch.bfloat16, "dominant key", scale=7.0)


def test_decode_padding_rows_read_nothing():
    """A padding row (position -1, block table of -1) gives zeros and no status code."""
    nh, nkv, hd, page_size = 8, 2, 64, 16
    rows = [(100, 1), (0, 1)]
    q, kv, ctx, grp = _attention_case(torch.bfloat16, nh, nkv, hd, page_size, rows)
    ctx.positions[1] = -1
    grp.block_tables[1] = -1
    dctx, dgrp = _full_ctx(rows, ctx, grp)
    got = k().paged_attention_decode(q.to(DEV), kv.to(DEV), dctx, dgrp, nh, nkv, hd, hd ** -0.5, 0, splits=3)
    assert dctx.status.tolist()[0] == 0 and float(got[1].abs().sum()) == 0.0 and torch.isfinite(got).all()


@pytest.mark.parametrize("kernel", ["prefill", "decode"])
@pytest.mark.parametrize("key_pos", [0, 15, 16, 63, 64, 65, 127, 128, 511, 512, 700])
def test_tiled_attention_far_key_stands_out(kernel, key_pos):
    """One key among 701 dominates for one head: a tile edge, a page edge or a split edge
    that loses it shows at once."""
    nh, nkv, hd, page_size = 8, 2, 64, 16
    rows = [(700, 1), (0, 5)] if kernel == "prefill" else [(700, 1), (4, 1)]
    q, kv, ctx, grp = _attention_case(torch.bfloat16, nh, nkv, hd, page_size, rows, spike=(0, key_pos, 5))
    ref = plain_ops.paged_attention(q, kv, ctx, grp, nh, nkv, hd, 1.0, 0)
    assert (ref[0, 5 * hd:6 * hd].float() - 7.0).abs().max() < 0.1
    dctx, dgrp = _full_ctx(rows, ctx, grp)
    if kernel == "prefill":
        got = k().paged_attention_prefill(q.to(DEV), kv.to(DEV), dctx, dgrp, nh, nkv, hd, 1.0, 0)
    else:
        got = k().paged_attention_decode(q.to(DEV), kv.to(DEV), dctx, dgrp, nh, nkv, hd, 1.0, 0, splits=4)
    close(got, ref, torch.bfloat16, "dominant key", scale=7.0)


@pytest.mark.parametrize("kernel", ["prefill", "decode"])
def test_tiled_attention_window_edge_and_unseen_keys(kernel):
    """The key just outside the window must not count, the one just inside must; and pages
    hold NaN wherever a key is out of sight."""
    nh, nkv, hd, page_size, window = 4, 1, 64, 16, 40
    for key_pos, inside in ((100 - 40, False), (100 - 39, True)):
        rows = [(100, 1), (7, 1)]
        q, kv, ctx, grp = _attention_case(torch.bfloat16, nh, nkv, hd, page_size, rows, window, spike=(0, key_pos, 1))
        ref = plain_ops.paged_attention(q, kv, ctx, grp, nh, nkv, hd, 1.0, window)
        assert ((ref[0, hd:2 * hd].float() - 7.0).abs().max() < 0.1) == inside
        poisoned = torch.full_like(kv, float("nan"))
        for r, (c, ql) in enumerate(rows):
            for j in range(max(0, c - window + 1), c + ql):
                p = int(grp.block_tables[r, j // page_size])
                poisoned[p, :, :, j % page_size] = kv[p, :, :, j % page_size]
        dctx, dgrp = _full_ctx(rows, ctx, grp)
        fn = k().paged_attention_prefill if kernel == "prefill" else k().paged_attention_decode
        got = fn(q.to(DEV), poisoned.to(DEV), dctx, dgrp, nh, nkv, hd, 1.0, window)
        assert torch.isfinite(got).all()
        close(got, ref, torch.bfloat16, "window edge", scale=7.0)


# ----------------------------------------------------------------------------- sampling
@pytest.mark.parametrize("V", [131, 320, 1000, 128256])
def test_argmax_first_index_on_ties(V):
    logits = rnd(5, V, seed=3)
    logits[1, 7] = logits[1, V - 2] = 50.0
    logits[2, :] = 0.0
    logits[3, V - 1] = 60.0
    got = k().argmax(logits.to(DEV)).cpu()
    assert got.tolist() == plain_ops.argmax(logits).tolist()
    assert got[1] == 7 and got[2] == 0 and got[3] == V - 1


@pytest.mark.parametrize("rows,V,pad", [(1, 128256, 0), (8, 128256, 0), (3, 50001, 0), (64, 32003, 1), (100, 20000, 3),
                                        (2, 8192, 0)])
def test_argmax_in_chunks(rows, V, pad):
    """Large vocabularies: a row is cut over several blocks.  Equal maxima on both sides of every
    chunk border, rows that do not start on 16 bytes (pad), a width that is no multiple of 4."""
    kk = k()
    chunks = kk.argmax_chunks(rows, V)
    assert chunks > 1
    chunk = ((V + chunks - 1) // chunks + 3) // 4 * 4
    buf = rnd(rows, V + pad, seed=11)
    logits = buf[:, :V]
    for r in range(rows):
        border = chunk * (1 + r % (chunks - 1))
        if r % 3 == 0 and border < V:
            logits[r, border - 1] = logits[r, border] = 70.0          # a tie across a border
        elif r % 3 == 1:
            logits[r, V - 1] = 70.0                                   # the ragged end
        else:
            logits[r, min(V - 1, border + 1)] = 70.0
    dev = buf.to(DEV)[:, :V]
    for _ in range(3):                                                # the tickets come back to zero
        got = kk.argmax(dev).cpu()
        assert got.tolist() == plain_ops.argmax(logits).tolist()
    assert int(kk.argmax_workspace(dev.device)[1].abs().sum()) == 0


@pytest.mark.parametrize("V", [131, 320, 5000, 128256])
def test_temperature_sampling_matches_inverse_cdf(V):
    rows = 24
    logits = rnd(rows, V, seed=5, scale=3.0)
    temps = torch.tensor([0.0, 0.7, 1.0, 1.5] * (rows // 4))
    u = torch.rand(rows, generator=torch.Generator().manual_seed(6))
    u[1], u[2] = 0.0, 0.99999994
    got = k().sample(logits.to(DEV), temps.to(DEV), u.to(DEV)).cpu()
    for r in range(rows):
        if temps[r] == 0:
            assert got[r] == int(torch.argmax(logits[r]))
            continue
        w = torch.softmax(logits[r].double() / temps[r].double(), 0)
        c = torch.cumsum(w, 0)
        i = int(got[r])
        lo, hi = (c[i - 1].item() if i > 0 else 0.0), c[i].item()
        # the chosen token's interval of the CDF holds u, up to 32-bit rounding of the running sum
        assert lo - 1e-4 <= u[r].item() <= hi + 1e-4, (r, i, lo, u[r].item(), hi)


def test_sampling_keep_mask():
    V = 300
    logits = rnd(6, V, seed=8)
    keep = torch.zeros(6, V, dtype=torch.uint8)
    keep[:, 100:110] = 1
    temps = torch.tensor([0.0, 1.0, 1.0, 2.0, 0.5, 1.0])
    u = torch.tensor([0.1, 0.0, 0.999, 0.5, 0.3, 0.7])
    got = k().sample(logits.to(DEV), temps.to(DEV), u.to(DEV), keep.to(DEV)).cpu()
    assert ((got >= 100) & (got < 110)).all()
    assert got.tolist() == plain_ops.sample(logits, temps, u, keep).tolist()


# ----------------------------------------------------------------------------- a wait that runs out
def test_a_wait_that_runs_out_leaves_a_code_and_a_usable_stream():
    """Every wait on a barrier in the tensor-core kernels is bounded.  The library `tc_expiry` is
    the product kernel's source built with a limit of 100,000 clocks and a producer that never
    brings its last block: the issuing thread and the epilogue warps wait for what never comes,
    give up, leave code 5 in the status word, wait for the products already issued, free their
    tensor memory and return.  Nothing faults and nothing is in flight; the next ordinary
    product on the same stream is right."""
    from fastmlx_b200.kernels.lib import call
    M, N, K = 256, 512, 512
    x, w = rnd(M, K, dtype=torch.bfloat16, seed=1).to(DEV), rnd(N, K, dtype=torch.bfloat16, seed=2, scale=0.1).to(DEV)
    out = torch.zeros(M, N, dtype=torch.bfloat16, device=DEV)
    st = status()
    call("tc_expiry", "fmx_gemm_tcgen05", x.data_ptr(), x.stride(0), w.data_ptr(), w.stride(0), out.data_ptr(), out.stride(0),
         None, 0, M, N, K, 256, 0, 0, st.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()                               # returns: the kernel ended by itself
    code, role, block = st.tolist()[:3]
    assert code == 5 and role in (2, 3), (code, role, block)
    st2 = status()
    got = k().gemm_tcgen05(x, w, st2, bn=256)
    torch.cuda.synchronize()
    assert st2.tolist()[0] == 0
    close(got, plain_ops.linear(x.cpu(), w.cpu(), None, torch.bfloat16), torch.bfloat16, "the product after an expired wait")


# ----------------------------------------------------------------------------- the greedy head
@pytest.mark.parametrize("M", [1, 5, 8, 9, 16])
@pytest.mark.parametrize("V,K", [(256, 64), (320, 192), (131, 80), (128256, 2048), (50001, 136)])
def test_greedy_head_chooses_the_largest_logit(M, V, K):
    """The head's product with the greedy choice inside against the logits' argmax; twice in a row
    (its words go back to zero by themselves), and with ties, where the lowest index wins."""
    x = rnd(M, K, dtype=torch.bfloat16, seed=M).to(DEV)
    w = rnd(V, K, dtype=torch.bfloat16, seed=V, scale=0.05).to(DEV)
    w[V - 1] = w[3]                                          # rows 3 and V-1 give equal logits everywhere
    if V > 40:
        x[0] = (w[3].float() * 40).to(torch.bfloat16)        # ... and row 0's largest logit is that pair's
    logits = k().gemv(x, w, out_dtype=torch.float32) if V < 65536 else None
    ref = plain_ops.linear(x.cpu(), w.cpu(), None, torch.float64)
    for _ in range(2):
        ids = k().greedy_head(x, w).cpu()
        for r in range(M):
            got = int(ids[r])
            assert 0 <= got < V
            best = float(ref[r].max())
            assert float(ref[r, got]) >= best - 1e-3 * max(1.0, abs(best)), (r, got, int(ref[r].argmax()))
        if logits is not None:                               # the same sums: the same choice, the first index on ties
            assert ids.tolist() == k().argmax(logits).cpu().tolist()
        if V > 40:
            assert int(ids[0]) == 3
    best_words, ticket = k().greedy_workspace(DEV)
    assert int(ticket) == 0 and int(best_words.abs().sum()) == 0


@pytest.mark.parametrize("rule", ["delta", "plain"])
@pytest.mark.parametrize("lens,H,G,D,P", [((64,), 4, 2, 64, 64), ((65, 1, 97, 31, 128), 4, 2, 64, 48), ((63, 200), 3, 3, 64, 16),
                                          ((32, 33, 7), 4, 1, 128, 128), ((31, 64), 2, 2, 128, 16), ((1, 2, 40, 96), 64, 8, 128, 32),
                                          ((64, 70, 96, 33), 32, 8, 64, 64)])      # (more blocks than two an SM: 32 columns each)
def test_portions_in_runs_of_tokens(rule, lens, H, G, D, P):
    """The kernels that walk runs of 32 tokens as matrix products, against 64-bit arithmetic and beside the walk token by token:
    portions of whole runs and a token more or less, rows too short for them, decays that are zero or nearly one, slots with state
    and slots out of order; what lies behind a slot's matrices stays."""
    torch.manual_seed(D + len(lens))
    starts = [0] + list(torch.tensor(lens).cumsum(0).tolist())
    T, R = starts[-1], len(lens)
    order = list(range(R))[::-1]
    ctx = SimpleNamespace(R=R, row_start=torch.tensor(starts, dtype=torch.int32, device=DEV), max_q_len=max(lens), h_row_start=starts,
                          row_slot=torch.tensor(order, dtype=torch.int32, device=DEV))
    q, kk, v = torch.randn(T, G, D), torch.nn.functional.normalize(torch.randn(T, G, D) + 0.3, dim=-1), torch.randn(T, H, P)
    q = torch.nn.functional.normalize(q, dim=-1)
    decay, w = torch.rand(T, H) ** torch.rand(H), torch.rand(T, H)
    decay[torch.rand(T, H) < 0.05] = 0.0
    decay[:, 0] = 1.0 - 1e-3 * torch.rand(T)
    state = torch.randn(R, H * P * D + 12)
    skip = torch.randn(H)
    if rule == "delta":
        x, gates = torch.cat([q.flatten(1), kk.flatten(1), v.flatten(1)], 1), torch.cat([decay, w], 1)
        walk, runs = k().delta_rule, k().delta_rule_chunks
        call = lambda fn, s: fn(x.to(DEV), gates.to(DEV), ctx, s, H, G, D, P)
    else:
        x, gates = torch.cat([v.flatten(1), kk.flatten(1), q.flatten(1)], 1), torch.cat([w, decay], 1)
        walk, runs = k().ssm_scan, k().ssm_scan_chunks
        call = lambda fn, s: fn(x.to(DEV), gates.to(DEV), skip.to(DEV), ctx, s, H, G, D, P)
    assert k().chunk_scan_takes(ctx, D, P)
    s1, s2 = state.to(DEV), state.to(DEV)
    o1, o2 = call(walk, s1).cpu().double().view(T, H, P), call(runs, s2).cpu().double().view(T, H, P)
    assert torch.equal(s2[:, H * P * D:].cpu(), state[:, H * P * D:])
    bytes_of, least, skips = k().load("chunks").fmx_chunk_scan_bytes, k().chunk_min_tokens(D), () if rule == "delta" else (skip.to(DEV),)
    s3, out, xd, gd = state.to(DEV), torch.zeros(T, H * P, device=DEV), x.to(DEV), gates.to(DEV)
    ws = torch.empty(2 * int(bytes_of(1, 1, H, G, D, int(rule == "delta"))), dtype=torch.uint8, device=DEV)         # two runs at a time
    k().call("chunks", "fmx_chunk_delta_rule" if rule == "delta" else "fmx_chunk_ssm_scan", xd.data_ptr(), gd.data_ptr(), *(t.data_ptr() for t in skips),
             ctx.row_start.data_ptr(), ctx.row_slot.data_ptr(), s3.data_ptr(), s3.stride(0), out.data_ptr(), ws.data_ptr(), ws.numel(), T, R, H, G, D,
             P, R, max(lens), least, k()._stream())
    assert bytes_of(10 ** 7, R, H, G, D, int(rule == "delta")) <= 256 << 20
    for r in range(R):                               # the same bits in waves of two runs; rows too short for runs are left alone
        at, run = slice(starts[r], starts[r + 1]), lens[r] >= least
        assert torch.equal(out[at].cpu().double().view(-1, H, P), o2[at] if run else 0 * o2[at])
        assert torch.equal(s3[order[r]].cpu(), s2[order[r]].cpu() if run else state[order[r]])
    f = lambda t: t.double().repeat_interleave(H // G, 1)
    want, left = torch.empty(T, H, P, dtype=torch.float64), state.double().clone()
    for r in range(R):
        S = left[order[r], :H * P * D].view(H, P, D)
        for t in range(starts[r], starts[r + 1]):
            S = S * decay[t].double()[:, None, None]
            u = v[t].double()
            if rule == "delta":
                u = u - torch.einsum("hpd,hd->hp", S, f(kk[t:t + 1])[0])
            S = S + (w[t].double()[:, None] * u)[:, :, None] * f(kk[t:t + 1])[0][:, None, :]
            want[t] = torch.einsum("hpd,hd->hp", S, f(q[t:t + 1])[0]) + (0 if rule == "delta" else skip.double()[:, None] * v[t].double())
        left[order[r], :H * P * D] = S.flatten()
    # roundings of 2^-24 of the largest value a sum meets, some dozens of which meet in a value at random signs
    for got, ref in ((o2, want), (s2[:, :H * P * D].cpu().double(), left[:, :H * P * D])):
        assert (got - ref).abs().max() < 40 * 2.0 ** -24 * ref.abs().max()
    err = lambda o: ((o - want).norm() / want.norm()).item()
    assert err(o2) < 1.5 * err(o1) + 2e-8
    for r in range(R):                               # rows too short for runs are walked: the same bits
        if lens[r] < k().chunk_min_tokens(D):
            assert torch.equal(o1[starts[r]:starts[r + 1]], o2[starts[r]:starts[r + 1]])


@pytest.mark.parametrize("rule", ["delta", "plain"])
@pytest.mark.parametrize("R,H,G,D,P,lanes,odd", [(3, 4, 2, 128, 128, 0, 0), (37, 2, 2, 64, 50, 0, 0), (5, 4, 1, 100, 33, 0, 0), (2, 2, 1, 30, 17, 0, 1),
                                                 (4, 3, 1, 33, 1, 0, 3), (1, 1, 1, 1, 5, 0, 0), (9, 2, 1, 64, 64, 2, 1), (3, 2, 2, 128, 40, 32, 0)])
def test_recurrence_over_single_tokens(rule, R, H, G, D, P, lanes, odd):
    """Steps of one token a row go through a kernel of their own: the same bits as the walk over the tokens, outputs and states, for states that
    begin on any boundary, sizes that end within a vector, padding rows (slot -1) and slots out of order."""
    torch.manual_seed(R + D)
    slots = torch.randperm(R + 2)[:R].to(torch.int32)
    if R > 2:
        slots[1] = -1
    ctx = lambda longest: SimpleNamespace(R=R, row_start=torch.arange(R + 1, dtype=torch.int32, device=DEV), max_q_len=longest,
                                          row_slot=slots.to(DEV))
    x, gates, skip = torch.randn(R, 2 * G * D + H * P, device=DEV), torch.rand(R, 2 * H, device=DEV), torch.randn(H, device=DEV)
    base = torch.randn(R + 2, H * P * D + 5 + odd, device=DEV)
    got = []
    for longest in (2, 1):
        state = base.clone()
        out = k().delta_rule(x, gates, ctx(longest), state, H, G, D, P, lanes) if rule == "delta" else \
            k().ssm_scan(x, gates, skip, ctx(longest), state, H, G, D, P, lanes)
        got.append((out[(slots >= 0).to(DEV)], state))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert not torch.equal(got[1][1], base) and torch.isfinite(got[1][0]).all()


@pytest.mark.parametrize("rule,D", [("delta", 64), ("delta", 128), ("plain", 64), ("plain", 128), ("channel delta", 64), ("channel delta", 128),
                                    ("channel plain", 64)])
def test_short_rows_join_the_runs_of_a_long_one(rule, D):
    """In a step that goes in runs its rows of 16 tokens and more do, beside shorter ones that are walked; single tokens and short
    steps are walked whole."""
    torch.manual_seed(D)
    lens, H, G, P = (16, 300, 1, 15, 31, 33, 17), 4, 4 if rule.endswith("plain") else 2, 32
    starts, R = [0] + list(torch.tensor(lens).cumsum(0).tolist()), len(lens)
    T, channel, delta = starts[-1], rule.startswith("channel"), rule.endswith("delta")
    ctx = SimpleNamespace(R=R, row_start=torch.tensor(starts, dtype=torch.int32, device=DEV), max_q_len=max(lens), min_q_len=1,
                          row_slot=torch.arange(R, dtype=torch.int32, device=DEV))
    least = k().rows_in_runs(rule, ctx, T, 64, D, P)
    assert least == 16 and k().rows_in_runs(rule, ctx, T, 1, D, P) == 0 and k().rows_in_runs(rule, ctx, T, 64, D, P + 8) == 0
    assert k().rows_in_runs(rule, SimpleNamespace(max_q_len=1), T, 64, D, P) == 0 and k().rows_in_runs(rule, ctx, T, 64, 32, P) == 0
    unit = lambda *s: torch.nn.functional.normalize(torch.randn(*s), dim=-1)
    q, kk, v, w = unit(T, G, D), unit(T, G, D), torch.randn(T, H, P), torch.rand(T, H)
    decay = torch.rand(T, H, D if channel else 1) * 0.2 + 0.8
    x, state = torch.cat([t.flatten(1) for t in ([q, kk, v] if delta or channel else [v, kk, q])], 1).to(DEV), torch.randn(R, H * P * D).to(DEV)
    if channel:
        more, fns = (decay.flatten(1).to(DEV), w.to(DEV) if delta else None), (k().channel_scan, k().channel_scan_chunks)
    elif delta:
        more, fns = (torch.cat([decay.flatten(1), w], 1).to(DEV),), (k().delta_rule, k().delta_rule_chunks)
    else:
        more, fns = (torch.cat([w, decay.flatten(1)], 1).to(DEV), torch.randn(H).to(DEV)), (k().ssm_scan, k().ssm_scan_chunks)
    s1, s2 = state.clone(), state.clone()
    want, got = fns[0](x, *more, ctx, s1, H, G, D, P), fns[1](x, *more, ctx, s2, H, G, D, P, least)
    for r in range(R):
        at = slice(starts[r], starts[r + 1])
        for a, b in ((want[at], got[at]), (s1[r], s2[r])):
            # as in the tests above, with the walk's own roundings
            assert torch.equal(a, b) if lens[r] < least else (a - b).abs().max() < 80 * 2.0 ** -24 * a.abs().max()


@pytest.mark.parametrize("what", ["value", "key", "query", "decay", "weight"])
@pytest.mark.parametrize("form,D,P", [("delta", 64, 48), ("delta", 128, 32), ("plain", 64, 32), ("plain", 128, 48), ("channel delta", 64, 32),
                                      ("channel delta", 128, 48), ("channel plain", 64, 48)])
def test_values_that_are_not_finite_in_runs_of_tokens(form, D, P, what):
    """An infinity or a NaN leaves the same values finite in runs of 32 tokens as in the walk token by token: those of the tokens in
    front of it, also of its own run, of other requests and, where a value holds it, of the other columns."""
    torch.manual_seed(D + P)
    channel, delta = form.startswith("channel"), form.endswith("delta")
    lens = (70, 128) if delta or not channel else (300, 257)
    if channel and D == 64 and delta:
        lens = (140, 128)
    starts, R, H, G = [0] + list(torch.tensor(lens).cumsum(0).tolist()), len(lens), 4, 2 if delta else 4
    T = starts[-1]
    ctx = SimpleNamespace(R=R, row_start=torch.tensor(starts, dtype=torch.int32, device=DEV), max_q_len=max(lens), h_row_start=starts,
                          row_slot=torch.arange(R, dtype=torch.int32, device=DEV))
    unit = lambda *s: torch.nn.functional.normalize(torch.randn(*s), dim=-1)
    q, kk, v, w = unit(T, G, D), unit(T, G, D), torch.randn(T, H, P), torch.rand(T, H) * 0.8 + 0.1
    decay, skip = torch.rand(T, H, D if channel else 1) * 0.3 + 0.7, torch.randn(H)
    for t, bad in ((37, float("inf")), (52, float("nan"))):        # a run's first and second half
        if what == "value":
            v[t, t % H, t % P] = bad
        elif what == "weight":
            w[t, t % H] = float("nan")
        else:
            {"key": kk, "query": q, "decay": decay}[what][t, t % (H if what == "decay" else G), -1] = bad
    if what == "weight" and channel and not delta:
        pytest.skip("no weight")
    order = [q, kk, v] if delta or channel else [v, kk, q]
    x, state = torch.cat([t.flatten(1) for t in order], 1).to(DEV), torch.randn(R, H * P * D).to(DEV)
    s1, s2 = state.clone(), state.clone()
    if channel:
        more = (decay.flatten(1).to(DEV), w.to(DEV) if delta else None, ctx)
        o = [fn(x, *more, s, H, G, D, P) for fn, s in ((k().channel_scan, s1), (k().channel_scan_chunks, s2))]
    else:
        more = (torch.cat([decay.flatten(1), w] if delta else [w, decay.flatten(1)], 1).to(DEV),) + (() if delta else (skip.to(DEV),))
        fns = (k().delta_rule, k().delta_rule_chunks) if delta else (k().ssm_scan, k().ssm_scan_chunks)
        o = [fn(x, *more, ctx, s, H, G, D, P) for fn, s in zip(fns, (s1, s2))]
    for a, b in ((o[0], o[1]), (s1, s2)):
        fine = torch.isfinite(a)
        assert torch.equal(fine, torch.isfinite(b))
        # as in the test above; 2^-24 of the largest value for some dozens of roundings
        assert fine.any() and (a[fine] - b[fine]).abs().max() < 40 * 2.0 ** -24 * a[fine].abs().max()
    assert torch.isfinite(o[1][:37]).all() and not torch.isfinite(o[1]).all()


@pytest.mark.parametrize("lens,ctxs,nh,nkv,hd,page,window,cap,loud", [
    ((64,), (0,), 32, 8, 64, 16, 0, 0.0, 1), ((300, 77, 1, 129), (0, 700, 40, 1033), 32, 8, 64, 16, 100, 30.0, 1),
    ((200, 130), (1500, 0), 12, 4, 64, 8, 200, 5.0, 5), ((33, 65), (7, 130), 6, 2, 64, 64, 17, 0.0, 1), ((70,), (500,), 16, 1, 128, 16, 64, 0.0, 1),
    ((200, 64), (300, 0), 32, 4, 128, 32, 0, 50.0, 3), ((2, 31), (63, 64), 8, 8, 128, 64, 150, 30.0, 20)])
def test_two_term_attention_on_tensor_memory(lens, ctxs, nh, nkv, hd, page, window, cap, loud):
    """Portions with 32-bit queries on tensor memory against 64-bit and beside the `mma.sync` kernel: tiles of tokens and keys with remainders,
    heads that do not fill a tile's rows, pages behind a window given back, unused places that hold NaN, caps that serve as the
    weights' scale and one that does not, scores beyond the short tangent, output rows that do not start on 16 bytes."""
    torch.manual_seed(nh + hd)
    R, starts = len(lens), [0] + list(torch.tensor(lens).cumsum(0).tolist())
    T, blocks = starts[-1], [-(-(c + n) // page) for c, n in zip(ctxs, lens)]
    perm, bt = torch.randperm(sum(blocks) + 3).tolist(), torch.full((R, max(blocks) + 1), -1, dtype=torch.int32)
    kv = torch.full((sum(blocks) + 3, 2, nkv, page, hd), float("nan")).bfloat16()
    K, V = ([torch.randn(c + n, nkv, hd).bfloat16() for c, n in zip(ctxs, lens)] for _ in range(2))
    for r in range(R):
        for b in range(blocks[r]):
            if window and (b + 1) * page <= ctxs[r] - window + 1:
                continue                              # given back
            p = bt[r, b] = perm.pop()
            for i, x in enumerate((K[r], V[r])):
                x = x[b * page:(b + 1) * page]
                kv[p, i, :, :len(x)] = x.transpose(0, 1)
    q = torch.randn(T, nh * hd) * loud
    pos = torch.cat([torch.arange(c, c + n) for c, n in zip(ctxs, lens)])
    ints = lambda x: torch.as_tensor(x, dtype=torch.int32, device=DEV)
    ctx = SimpleNamespace(R=R, T=T, positions=ints(pos), row_start=ints(starts), row_ctx=ints(ctxs), max_q_len=max(lens), status=ints([0] * 4))
    kvd, qd, grp = kv.to(DEV), q.to(DEV), SimpleNamespace(block_tables=bt.to(DEV))
    assert k().wide_tc_ok(kvd, nh, nkv, hd, hd, hd ** -0.5)
    outs = []
    for tc in (False, True):
        wide = torch.zeros(T, nh * hd + 2, dtype=torch.bfloat16, device=DEV)
        k()._wide_launch(qd, kvd, ctx, grp, nh, nkv, hd, hd ** -0.5, cap, window, wide[:, 2:], tc=tc)
        outs.append(wide[:, 2:].cpu().double())
    assert ctx.status.tolist() == [0] * 4
    errs = [0.0, 0.0]
    for r in range(R):
        at, p = slice(starts[r], starts[r + 1]), torch.arange(ctxs[r], ctxs[r] + lens[r])
        k_, v_ = (x[r].double().repeat_interleave(nh // nkv, 1) for x in (K, V))
        qq = q[at].double().view(-1, nh, hd)
        s = torch.einsum("qhd,khd->hqk", qq, k_) * hd ** -0.5
        back = p[:, None] - torch.arange(len(k_))[None]
        hidden = (back < 0) | ((back >= window) if window else False)
        w = torch.softmax((cap * torch.tanh(s / cap) if cap else s).masked_fill(hidden, -float("inf")), -1)
        want = torch.einsum("hqk,khd->qhd", w, v_).flatten(1)
        size = torch.einsum("hqk,khd->qhd", w, v_.abs())
        # operands of two terms are off by 2^-17: a weight, and by the queries a score, by 2^-17 of its products' sizes, which moves a weight by
        # twice that; and the rounding to bfloat16
        products = (torch.einsum("qhd,khd->hqk", qq.abs(), k_.abs()) * hd ** -0.5).masked_fill(hidden, 0.0).amax(-1).T[:, :, None]
        room = 2.0 ** -8 * want.abs() + (2.0 ** -17 * (2 + 2 * products) * size).flatten(1)
        assert ((outs[1][at] - want).abs() <= room).all()
        errs = [e + ((o[at] - want) ** 2).sum().item() for e, o in zip(errs, outs)]
    assert errs[1] <= 1.02 * errs[0]


@pytest.mark.parametrize("hd", [64, 128])
def test_scale_of_capped_weights_on_tensor_memory(hd):
    """How many outputs are not the bfloat16 nearest to 64-bit arithmetic's follows the size of the error in front of that rounding (at 256 keys a
    token, some 0.3 % of them).  Beside the `mma.sync` kernel, whose scale is each row's maximum: 1.05 times as many, where exponents rounded at
    the cap's own scale (2^-19 of a weight, a quarter of what two terms leave of it) made them 1.09 times as many at head size 64."""
    nh, nkv, q_len, c, page, window, cap = 32, 8, 1024, 700, 16, 256, 30.0
    g = torch.Generator().manual_seed(1)
    blocks = -(-(c + q_len) // page)
    kv = torch.randn(blocks, 2, nkv, page, hd, generator=g).bfloat16().to(DEV)
    q = torch.randn(q_len, nh * hd, generator=g).to(DEV)
    ints = lambda x: torch.as_tensor(x, dtype=torch.int32, device=DEV)
    ctx = SimpleNamespace(R=1, T=q_len, positions=ints(list(range(c, c + q_len))), row_start=ints([0, q_len]), row_ctx=ints([c]), max_q_len=q_len,
                          status=ints([0] * 4))
    grp = SimpleNamespace(block_tables=ints(list(range(blocks)))[None])
    K, V = (kv[:, i].permute(0, 2, 1, 3).reshape(blocks * page, nkv, hd)[:c + q_len].double() for i in (0, 1))
    back = torch.arange(c, c + q_len, device=DEV)[:, None] - torch.arange(c + q_len, device=DEV)[None]
    hidden, want = (back < 0) | (back >= window), torch.empty(q_len, nh, hd, dtype=torch.float64, device=DEV)
    for h in range(nh):
        s = cap * torch.tanh(q.double().view(q_len, nh, hd)[:, h] @ K[:, h // (nh // nkv)].t() * hd ** -0.5 / cap)
        want[:, h] = torch.softmax(s.masked_fill(hidden, -float("inf")), -1) @ V[:, h // (nh // nkv)]
    off = []
    for tc in (False, True):
        out = torch.empty(q_len, nh * hd, dtype=torch.bfloat16, device=DEV)
        k()._wide_launch(q, kv, ctx, grp, nh, nkv, hd, hd ** -0.5, cap, window, out, tc=tc)
        off.append(int((out != want.view(q_len, -1).bfloat16()).sum()))
    assert ctx.status.tolist() == [0] * 4 and off[0] < 0.005 * want.numel()
    assert off[1] <= 1.065 * off[0], off


@pytest.mark.parametrize("weights", ["softmax", "sigmoid"])
@pytest.mark.parametrize("window", [0, 20])
def test_capped_scores_do_not_depend_on_later_keys(weights, window):
    """A capped score takes a short form where it is small against the cap.  Which form it takes follows from the score alone: keys behind
    a token, out of its sight and large, leave its output's bits; and both forms, side by side in a tile, stand against 64-bit."""
    nh, nkv, hd, page, T, n, cap = 32, 8, 64, 16, 128, 100, 30.0
    q, kv, ctx, grp = _attention_case(torch.bfloat16, nh, nkv, hd, page, [(0, T)], seed=5)
    q = (q * 4).float()                              # scores of N(0, 4): below 0.8 of the cap
    loud = kv.clone()
    for j in range(n, T):
        loud[int(grp.block_tables[0, j // page]), 0, :, j % page] *= 32
    d, g = _full_ctx([(0, T)], ctx, grp)
    d.T, d.h_row_start = T, [0, T]
    mix, bias = torch.eye(nh) + 0.1 * torch.randn(nh, nh, generator=torch.Generator().manual_seed(6)), torch.full((nh,), -3.0)

    def run(pages):
        if weights == "softmax":
            return k().paged_attention_wide(q.to(DEV), pages.to(DEV), d, g, nh, nkv, hd, hd ** -0.5, cap, window).cpu()
        return k().sigmoid_attention(q.to(DEV), pages.to(DEV), d, g, nh, nkv, hd, hd, hd ** -0.5, cap, window, page, bias.to(DEV), mix.to(DEV)).cpu()
    quiet, got = run(kv), run(loud)
    assert torch.equal(quiet[:n], got[:n]) and not torch.equal(quiet[n:], got[n:])
    K, V = (torch.cat([loud[int(p), i] for p in grp.block_tables[0, :T // page]], 1).double().repeat_interleave(nh // nkv, 0) for i in (0, 1))
    s = torch.einsum("qhd,hkd->hqk", q.double().view(T, nh, hd), K) * hd ** -0.5
    s = cap * torch.tanh(s / cap)
    back = torch.arange(T)[:, None] - torch.arange(T)[None]
    hidden = (back < 0) | ((back >= window) if window else False)
    if weights == "softmax":
        w = torch.softmax(s.masked_fill(hidden, -float("inf")), -1)
        size = torch.einsum("hqk,hkd->qhd", w, V.abs())
    else:
        w = torch.sigmoid(s - 3.0).masked_fill(hidden, 0.0)
        size = torch.einsum("hqk,hkd->qhd", torch.einsum("hg,gqk->hqk", mix.double().abs(), w), V.abs())
        w = torch.einsum("hg,gqk->hqk", mix.double(), w)
    want = torch.einsum("hqk,hkd->qhd", w, V).flatten(1)
    # the rounding to bfloat16; operands of two terms are off by 2^-17: a weight, and by the queries a score, by 2^-17 of its products'
    # sizes, which moves a weight by twice that; three terms (sigmoid): 2^-24 for some dozens of roundings, and a score's 64 products
    products = (torch.einsum("qhd,hkd->hqk", q.double().view(T, nh, hd).abs(), K.abs()) * hd ** -0.5).masked_fill(hidden, 0.0).amax(-1).T[:, :, None]
    eps = 2.0 ** -17 * (2 + 2 * products) if weights == "softmax" else 2.0 ** -24 * (48 + 64 * products)
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + (eps * size).flatten(1)).all()


@pytest.mark.parametrize("lens,ctxs,nh,nkv,hd,vd,page,window,cap", [
    ((4,), (0,), 2, 1, 16, 16, 16, 0, 30.0), ((9, 1, 33), (0, 40, 31), 8, 8, 32, 64, 8, 0, 30.0), ((40, 3, 8), (3, 0, 57), 32, 8, 64, 64, 16, 20, 30.0),
    ((50,), (77,), 6, 3, 48, 32, 16, 0, 0.0), ((17, 5), (200, 0), 12, 3, 64, 16, 5, 0, 2.0), ((264, 31), (0, 700), 32, 8, 64, 64, 16, 0, 30.0),
    ((64, 31), (900, 700), 32, 8, 64, 64, 16, 300, 30.0)])
def test_mixed_heads_on_tensor_cores(lens, ctxs, nh, nkv, hd, vd, page, window, cap):
    """Sigmoid attention with mixed heads over portions with three-term operands, against 64-bit arithmetic and beside the kernel of
    32-bit multiply-adds: tiles of tokens and keys with remainders, rows that stay on the other kernel, fewer heads than a tile
    has, windows, scores far beyond the small tangent's range, pages whose unused places hold NaN, keys shared out over blocks."""
    torch.manual_seed(nh + hd)
    R, starts = len(lens), [0] + list(torch.tensor(lens).cumsum(0).tolist())
    T, blocks = starts[-1], [-(-(c + n) // page) for c, n in zip(ctxs, lens)]
    perm = torch.randperm(sum(blocks) + 3).tolist()
    bt = torch.full((R, max(blocks) + 1), -1, dtype=torch.int32)
    kv = torch.full((sum(blocks) + 3, nkv * page * (hd + vd)), float("nan")).bfloat16()
    K = [torch.randn(c + n, nkv, hd).bfloat16() for c, n in zip(ctxs, lens)]
    V = [torch.randn(c + n, nkv, vd).bfloat16() for c, n in zip(ctxs, lens)]
    for r in range(R):
        for b in range(blocks[r]):
            p = bt[r, b] = perm.pop()
            k_, v_ = K[r][b * page:(b + 1) * page], V[r][b * page:(b + 1) * page]
            kv[p, :nkv * page * hd].view(nkv, page, hd)[:, :len(k_)] = k_.transpose(0, 1)
            kv[p, nkv * page * hd:].view(nkv, page, vd)[:, :len(v_)] = v_.transpose(0, 1)
    kv = (kv.view(-1, 2, nkv, page, hd) if hd == vd else kv).to(DEV)
    q, mix, bias = torch.randn(T, nh * hd) * 2, torch.eye(nh) + 0.1 * torch.randn(nh, nh), torch.randn(nh) * 0.5 - 3
    pos = torch.cat([torch.arange(c, c + n) for c, n in zip(ctxs, lens)])
    ctx = SimpleNamespace(R=R, T=T, positions=pos.int().to(DEV), token_row=torch.arange(R).repeat_interleave(torch.tensor(lens)).int().to(DEV),
                          row_start=torch.tensor(starts, dtype=torch.int32, device=DEV), h_row_start=starts, max_q_len=max(lens),
                          max_ctx_after=max(c + n for c, n in zip(ctxs, lens)), status=torch.zeros(4, dtype=torch.int32, device=DEV))
    run = lambda tc: k().sigmoid_attention(q.to(DEV), kv, ctx, SimpleNamespace(block_tables=bt.to(DEV)), nh, nkv, hd, vd, hd ** -0.5, cap, window,
                                           page, bias.to(DEV), mix.to(DEV), tensor_cores=tc).cpu().double().view(T, nh, vd)
    plan = k().load("chunks").fmx_mixattn_tc_plan(T, R, nh, nkv, hd, vd, ctx.max_q_len, ctx.max_ctx_after, window)
    assert plan >= 1 and (plan > 1 or ctx.max_ctx_after < 256)
    fma, got = run(False), run(None)
    assert ctx.status.tolist()[0] == 0
    want, size = torch.empty(T, nh, vd, dtype=torch.float64), torch.empty(T, nh, vd, dtype=torch.float64)
    for r in range(R):
        at = slice(starts[r], starts[r + 1])
        kk, vv = (t[r].double().repeat_interleave(nh // nkv, 1) for t in (K, V))
        s = torch.einsum("qhd,khd->hqk", q[at].double().view(-1, nh, hd), kk) * hd ** -0.5
        s = cap * torch.tanh(s / cap) if cap else s
        kp, qp = torch.arange(len(kk)), pos[at]
        hidden = (kp[None] > qp[:, None]) | ((kp[None] <= qp[:, None] - window) if window else False)
        w = torch.sigmoid(s + bias.double()[:, None, None]).masked_fill(hidden, 0.0)
        want[at] = torch.einsum("hqk,khd->qhd", torch.einsum("hg,gqk->hqk", mix.double(), w), vv)
        size[at] = torch.einsum("hqk,khd->qhd", torch.einsum("hg,gqk->hqk", mix.double().abs(), w), vv.abs())
    # the rounding to bfloat16, and 2^-24 of what a value's sums add up to for some dozens of roundings in 32-bit
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 48 * 2.0 ** -24 * size).all()
    off = lambda o: (o != want.bfloat16().double()).double().mean().item()
    assert off(got) < off(fma) + 1e-3
    for r in range(R):
        if lens[r] < k().MIXED_TC_MIN_TOKENS:        # these rows run where they ran
            assert torch.equal(got[starts[r]:starts[r + 1]], fma[starts[r]:starts[r + 1]])


@pytest.mark.parametrize("nh,nkv", [(32, 8), (8, 4)])
@pytest.mark.parametrize("dust", [2.0 ** -12, -(2.0 ** -20)])            # a second term of one entry, a third term
def test_mix_without_smaller_terms(nh, nkv, dust):
    """A mix that bfloat16 holds exactly goes without the products of its smaller terms: one entry that has them changes its own head only,
    every other head's values are the same bits."""
    hd, page, T = 64, 16, 45
    q, kv, ctx, grp = _attention_case(torch.bfloat16, nh, nkv, hd, page, [(30, T)], seed=3)
    d, g = _full_ctx([(30, T)], ctx, grp)
    d.T, d.h_row_start = T, [0, T]
    mix, bias = (torch.eye(nh) + 0.1 * torch.randn(nh, nh)).bfloat16().float(), torch.full((nh,), -2.0)
    mix[5, 2] = 0.75
    more = mix.clone()
    more[5, 2] += dust
    assert more[5, 2].bfloat16() != more[5, 2]
    a, b = (k().sigmoid_attention(q.float().to(DEV), kv.to(DEV), d, g, nh, nkv, hd, hd, hd ** -0.5, 0.0, 0, page, bias.to(DEV), m.to(DEV),
                                  tensor_cores=True).view(T, nh, hd) for m in (mix, more))
    others = [h for h in range(nh) if h != 5]
    assert torch.equal(a[:, others], b[:, others]) and torch.isfinite(a).all()
    assert torch.allclose(a[:, 5].float(), b[:, 5].float(), rtol=2.0 ** -7, atol=abs(dust) * 100)


@pytest.mark.parametrize("ctx", [2000, 60000])
@pytest.mark.parametrize("window", [1, 26, 27, 90, 120, 121, 122, 500])
def test_shares_of_a_window_are_no_fewer_than_four_tiles(ctx, window):
    """Behind a window the keys are shared out as behind as much context: 8 tokens meet at most the tiles of 32 that window + 7 keys lie in."""
    plan = k().load("chunks").fmx_mixattn_tc_plan
    most = max((first + window + 6) // 32 + 1 for first in range(32))
    assert plan(64, 1, 32, 8, 64, 64, 64, ctx, window) == max(1, min(most // 4, 32)) < plan(64, 1, 32, 8, 64, 64, 64, ctx, 0)


@pytest.mark.parametrize("cap", [0.0, 30.0])
@pytest.mark.parametrize("where", ["query", "key"])
def test_infinite_scores_saturate_mixed_heads(where, cap):
    """An infinite query or key value makes weights of zero and one, on the tensor cores as with 32-bit multiply-adds."""
    nh, nkv, hd, page, T = 8, 4, 64, 16, 70
    q, kv, ctx, grp = _attention_case(torch.bfloat16, nh, nkv, hd, page, [(30, T)], seed=8)
    q, inf = q.float(), float("inf")
    if where == "query":
        q.view(T, nh, hd)[[3, 40, 41], [0, 5, 7], [0, 17, 63]] = torch.tensor([inf, -inf, inf])
    else:
        for j, g, e, x in ((5, 0, 0, inf), (62, 2, 33, -inf), (90, 3, 63, inf)):
            kv[int(grp.block_tables[0, j // page]), 0, g, j % page, e] = x
            q[:, g * 128 + e] = q[:, g * 128 + e].bfloat16().float()      # no smaller terms
    d, g = _full_ctx([(30, T)], ctx, grp)
    d.T, d.h_row_start = T, [0, T]
    mix, bias = torch.eye(nh) + 0.1 * torch.randn(nh, nh), torch.full((nh,), -2.0)
    want, got = (k().sigmoid_attention(q.to(DEV), kv.to(DEV), d, g, nh, nkv, hd, hd, hd ** -0.5, cap, 0, page, bias.to(DEV), mix.to(DEV),
                                       tensor_cores=tc).cpu().double() for tc in (False, None))
    assert torch.isfinite(want).all() and torch.isfinite(got).all()
    # two roundings to bfloat16, and those of the 32-bit sums
    assert ((got - want).abs() <= 2.0 ** -7 * want.abs() + 2.0 ** -16 * want.abs().max()).all()


@pytest.mark.parametrize("form", ["delta", "ssm", "channel"])
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("lens", [(1,), (1, 1, 1, 1, 1), (2, 1, 3), (5, 40, 1, 17), (700, 4, 3)])
def test_convolutions_by_strips_of_tokens(form, lens, D):
    """The kernels that walk strips of tokens with the last inputs in registers (four taps, channels in fours) beside those token by
    token, which rows of an odd stride take: the same sums in the same order, unit vectors to their sums' rounding, the same slots;
    a row of a captured step that is not there, rows shorter than the taps, strips that hold several rows."""
    torch.manual_seed(len(lens))
    H, G, P, taps = 12, 4, 64, 4
    starts = [0] + list(torch.tensor(lens).cumsum(0).tolist())
    T, R = starts[-1] + 1, len(lens) + 1                               # the last row's slot is -1
    starts.append(T)
    single = max(lens) == 1
    ctx = SimpleNamespace(R=R, max_q_len=max(lens), row_start=torch.tensor(starts, dtype=torch.int32, device=DEV), status=torch.zeros(4, dtype=torch.int32, device=DEV),
                          token_row=torch.arange(R).repeat_interleave(torch.tensor(starts).diff()).int().to(DEV),
                          row_slot=torch.tensor(list(range(R - 1))[::-1] + [-1], dtype=torch.int32, device=DEV))
    C = 2 * G * D + H * P
    width = {"delta": C + 8, "ssm": H * P + C + H, "channel": C + H}[form]
    proj = torch.randn(T, width).bfloat16()
    conv, cb, a_log, dtb = torch.randn(C, taps).to(DEV) * 0.5, torch.randn(C).to(DEV) * 0.1, torch.randn(H).to(DEV), torch.randn(H * D).to(DEV)
    ab, z, off = torch.randn(T, 2 * H).to(DEV), torch.randn(T, H * D).to(DEV), H * P * D
    state = torch.randn(R, off + (taps - 1) * C)

    def run(odd):
        x = torch.zeros(T, width + (1 if odd else (-width) % 4)).bfloat16().to(DEV)
        x[:, :width] = proj.to(DEV)
        s = state.to(DEV)
        if form == "delta":
            out = k().delta_prepare(x, ab, conv, a_log, dtb[:H], ctx, s, off, H, G, D, P, taps)
        elif form == "ssm":
            out = k().ssm_prepare(x, conv, cb, a_log, dtb[:H], ctx, s, off, H, G, D, P, taps)
        else:
            out = k().channel_delta_prepare(x, x[:, C:C + H], z, conv, a_log, dtb, ctx, s, off, H, G, D, P, taps)
        return [t.cpu() for t in out], s.cpu()
    (want, ws), (got, gs) = run(True), run(False)
    assert ctx.status.tolist()[0] == 0 and single == (T == R)
    unit = 0 if form == "ssm" else 2 * G * D
    assert torch.equal(got[0][:, unit:], want[0][:, unit:]) and torch.equal(gs, ws)
    assert (got[0][:, :unit] - want[0][:, :unit]).abs().max() <= 4e-7 if unit else True
    assert (got[0][-1] == 0).all()
    for g, w in zip(got[1:], want[1:]):
        assert (g - w).abs().max() <= 2.0 ** -22 * w.abs().max()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", [4, 36, 512, 516, 2048, 2052])
def test_gated_group_rmsnorm_in_fours(n, dtype):
    """Parts of at most 2,048 values in fours stay in registers; wider ones, and rows that do not start on fours, take the other kernel."""
    T, groups = 5, 3
    y, z, w = rnd(T, groups * n, dtype=torch.float32), rnd(T, groups * n + 3, dtype=dtype, seed=1), 1 + 0.1 * rnd(groups * n, dtype=torch.float32, seed=2)
    zz = z[:, :groups * n]
    got = k().gated_group_rmsnorm(y.to(DEV), zz.contiguous().to(DEV), w.to(DEV), 1e-6, groups, dtype)
    odd = k().gated_group_rmsnorm(y.to(DEV), z.to(DEV)[:, :groups * n], w.to(DEV), 1e-6, groups, dtype)
    want = plain_ops.gated_group_rmsnorm(y, zz, w, 1e-6, groups, torch.float64)
    for o in (got, odd):
        close(o, want, dtype, "gated_group_rmsnorm", scale=None)


@pytest.mark.parametrize("tin,tkv", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.float32, torch.bfloat16)])
@pytest.mark.parametrize("hd,vd,rot,inter,form", [(64, 64, 64, False, "last"), (64, 64, 32, False, "first"), (128, 64, 128, True, "first"),
                                                 (32, 96, 16, False, "none"), (128, 128, 64, False, "whole"), (64, 64, 0, False, "whole keys"),
                                                 (64, 32, 12, True, "last")])
def test_queries_and_keys_in_fours(tin, tkv, hd, vd, rot, inter, form):
    """Queries and keys made ready four values a lane beside the kernels of one value a lane, which rows that do not start on fours
    take: both orders of norm and rotation, norms over the whole projection, values that are the keys, biases, mixed values, partial
    and interleaved rotations, tokens that are stored nowhere."""
    torch.manual_seed(hd + rot)
    T, nh, nkv, page = 7, 6, 3, 4
    from_keys = form == "whole keys"
    width = (nh + nkv) * hd + (0 if from_keys else nkv * vd)
    row = torch.randn(T, width).to(tin)
    slots = torch.tensor([5, 0, 11, -1, 7, 2, 3], device=DEV)
    pos, freq = torch.tensor([0, 3, 900, 17, 4, 1, 8191], dtype=torch.int32, device=DEV), (torch.rand(rot // 2) if rot else torch.zeros(1)).to(DEV)
    whole = form.startswith("whole")
    bias = torch.randn(width).to(DEV) if form in ("first", "whole") else None
    wq, wk = torch.rand(nh * hd if whole else hd).to(DEV) + 0.5, torch.rand(nkv * hd if whole else hd).to(DEV) + 0.5
    first, share = torch.randn(T, nkv * vd).to(tin).to(DEV), torch.tensor([0.3], device=DEV)

    def run(odd):
        x = torch.zeros(T, width + (1 if odd else (-width) % 4)).to(tin).to(DEV)
        x[:, :width] = row.to(DEV)
        kv = torch.zeros(3, nkv * page * (hd + vd), device=DEV).to(tkv)
        status = torch.zeros(4, dtype=torch.int32, device=DEV)
        more = dict(v_first=first, v_share=share) if form == "last" else {}
        q = k().qk_prepare(x, pos, freq, rot, inter, None if form == "none" else 1e-6, slots, kv, nh, nkv, hd, vd, status, bias=bias,
                           q_weight=None if form == "none" else wq, k_weight=None if form == "none" else wk,
                           norm_first=form == "first" or whole, whole=whole, values_from_keys=from_keys, amplitude=1.25, v_scale=0.5, **more)
        return q.cpu(), kv.cpu(), status.tolist()[0]
    (q1, kv1, st1), (q2, kv2, st2) = run(True), run(False)
    assert st1 == st2 == 0
    assert (q1 - q2).abs().max() <= 2.0 ** -21 * q1.abs().max()          # the norms' sums in another order
    assert (kv1.float() - kv2.float()).abs().max() <= (2.0 ** -21 if tkv == torch.float32 else 2.0 ** -7) * kv1.float().abs().max()
    if tkv == torch.bfloat16:
        assert (kv1 != kv2).float().mean() < 2e-3
@pytest.mark.parametrize("delta,lens,H,G,D,P", [
    (True, (128,), 4, 2, 64, 64), (True, (129, 1, 161, 127, 192), 4, 2, 64, 48), (True, (64, 65, 63), 4, 1, 128, 128), (True, (31, 128), 2, 2, 128, 16),
    (True, (3, 72, 96), 32, 8, 128, 96), (False, (256,), 3, 3, 64, 64), (False, (257, 5, 255, 300), 4, 4, 64, 48), (False, (1, 288), 32, 32, 64, 32),
    (True, (128, 130, 160, 129), 32, 8, 64, 64), (False, (256, 257, 288, 256), 32, 32, 64, 64)])          # (more than three: 32 columns each)
def test_channel_decays_in_runs_of_tokens(delta, lens, H, G, D, P):
    """The kernels that walk runs of 32 tokens whose state decays by key channel, against 64-bit arithmetic and beside the walk token
    by token: decays that are zero, that vanish within a run and that are nearly one, portions of whole runs and a token more or
    less, rows too short for runs, a workspace that holds a few runs only."""
    torch.manual_seed(D + len(lens))
    starts, R = [0] + list(torch.tensor(lens).cumsum(0).tolist()), len(lens)
    T, order = starts[-1], list(range(R))[::-1]
    ctx = SimpleNamespace(R=R, row_start=torch.tensor(starts, dtype=torch.int32, device=DEV), max_q_len=max(lens), h_row_start=starts,
                          row_slot=torch.tensor(order, dtype=torch.int32, device=DEV))
    unit = lambda *s: torch.nn.functional.normalize(torch.randn(*s) + 0.2, dim=-1)
    q, kk, v, beta = unit(T, G, D), unit(T, G, D), torch.randn(T, H, P), torch.rand(T, H)
    decay = torch.rand(T, H, D) ** (torch.rand(H, D) * 3)
    decay[torch.rand(T, H, D) < 0.02] = 0.0
    decay[:, 0, ::2] = 1.0 - 1e-3 * torch.rand(T, (D + 1) // 2)
    decay[:, -1, 1::4] = 1e-6
    x, state = torch.cat([q.flatten(1), kk.flatten(1), v.flatten(1)], 1).to(DEV), torch.randn(R, H * P * D + 12)
    g, b = decay.flatten(1).to(DEV), beta.to(DEV) if delta else None
    assert k().channel_scan_takes(ctx, D, P, delta) and not k().channel_scan_takes(ctx, 128, P, False)
    s1, s2, s3 = state.to(DEV), state.to(DEV), state.to(DEV)
    o1 = k().channel_scan(x, g, b, ctx, s1, H, G, D, P).cpu().double().view(T, H, P)
    o2 = k().channel_scan_chunks(x, g, b, ctx, s2, H, G, D, P).cpu().double().view(T, H, P)
    out, one = torch.zeros(T, H * P, device=DEV), int(k().load("chunks").fmx_channel_chunks_bytes(1, 1, H, D, int(delta)))
    ws = torch.empty(2 * one, dtype=torch.uint8, device=DEV)              # two runs at a time
    k().call("chunks", "fmx_channel_chunks", x.data_ptr(), g.data_ptr(), k()._ptr(b), ctx.row_start.data_ptr(), ctx.row_slot.data_ptr(), s3.data_ptr(),
             s3.stride(0), out.data_ptr(), ws.data_ptr(), ws.numel(), T, R, H, G, D, P, R, k().channel_chunks_least(D, delta), k()._stream())
    f = lambda t: t.double().repeat_interleave(H // G, 1)
    qd, kd, want, left = f(q), f(kk), torch.empty(T, H, P, dtype=torch.float64), state.double().clone()
    for r in range(R):
        S = left[order[r], :H * P * D].view(H, P, D)
        for t in range(starts[r], starts[r + 1]):
            S = S * decay[t].double()[:, None, :]
            u = v[t].double()
            if delta:
                u = beta[t].double()[:, None] * (u - torch.einsum("hpd,hd->hp", S, kd[t]))
            S = S + u[:, :, None] * kd[t][:, None, :]
            want[t] = torch.einsum("hpd,hd->hp", S, qd[t])
        left[order[r], :H * P * D] = S.flatten()
    # roundings of 2^-24 of the largest value a sum meets, some dozens of which meet in a value at random signs
    for got, ref in ((o2, want), (s2[:, :H * P * D].cpu().double(), left[:, :H * P * D])):
        assert (got - ref).abs().max() < 40 * 2.0 ** -24 * ref.abs().max()
    err = lambda o: ((o - want).norm() / want.norm()).item()
    assert err(o2) < 1.5 * err(o1) + 2e-8
    assert torch.equal(s2[:, H * P * D:].cpu(), state[:, H * P * D:])
    for r in range(R):
        at = slice(starts[r], starts[r + 1])
        if lens[r] < k().channel_chunks_least(D, delta):        # walked: the same bits; and left alone by the kernel for runs
            assert torch.equal(o1[at], o2[at]) and (out[at] == 0).all() and torch.equal(s3[order[r]].cpu(), state[order[r]])
        else:                                        # in waves of two runs the same bits as in one
            assert torch.equal(out[at].cpu().double().view(-1, H, P), o2[at]) and torch.equal(s3[order[r]], s2[order[r]])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,D,P,rot", [(3, 16, 8, 16), (5, 64, 64, 64), (2, 128, 36, 32), (4, 12, 4, 8), (3, 64, 32, 0)])
def test_retention_prepare_in_fours(dtype, H, D, P, rot):
    """A retention's operands four values a thread: the same bits as the kernel of one value a thread, which rows of an odd stride take."""
    T, width = 9, 2 * H * D + H * P
    x = rnd(T, width, dtype=dtype).to(DEV)
    odd = torch.zeros(T, width + 1, dtype=dtype, device=DEV)
    odd[:, :width] = x
    pos, freq, decay = torch.arange(0, 900, 100, dtype=torch.int32, device=DEV), torch.rand(max(1, rot // 2), device=DEV), torch.rand(H, device=DEV)
    a = k().retention_prepare(x, pos, freq, decay, H, D, P, rot, 0.3)
    b = k().retention_prepare(odd[:, :width], pos, freq, decay, H, D, P, rot, 0.3)
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
