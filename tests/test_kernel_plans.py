"""Host-side arithmetic of the kernels' work division, checked without a GPU."""
import os
import pathlib
import subprocess

import pytest
import torch


def test_short_prompts_go_to_the_library_product():
    """Fewer tiles than about a round of the SMs: the whole-tile kernel would leave most idle."""
    from fastmlx_b200 import kernels as k
    assert k.tc_fills_the_gpu(2048, 2048) and k.tc_fills_the_gpu(8192, 3072) and k.tc_fills_the_gpu(512, 16384)
    assert k.tc_fills_the_gpu(2048, 6144) and not k.tc_fills_the_gpu(2048, 3072)       # 192 tiles: 65 % of two rounds
    assert not k.tc_fills_the_gpu(512, 2048) and not k.tc_fills_the_gpu(1024, 3072) and not k.tc_fills_the_gpu(128, 8192)


def test_no_kernel_is_chosen_by_the_environment():
    """Which kernel runs follows from sizes, types and alignment: no native source reads an environment variable."""
    from fastmlx_b200.csrc import build
    sources = [p for p in pathlib.Path(build.HERE).rglob("*") if p.suffix in (".cu", ".cuh", ".h")]
    assert len(sources) > 40
    assert [p.name for p in sources if "getenv" in p.read_text()] == []


def test_shares_of_the_three_term_product():
    """They follow the matrix, so its rows by themselves would be summed otherwise: at a width of 2,048, all projections of a matrix memory
    (8 heads, 128 x 256) and their gates' alone.  No more than a cluster holds, and no more than there are blocks of K."""
    from fastmlx_b200.kernels import load
    shares = load("tc").fmx_gemm_three_splits
    assert shares(2 * 8 * 128 + 2 * 8 * 256 + 16, 2048) == 2 and shares(16, 2048) == 4
    for N in (1, 128, 129, 2048, 16384, 128256):
        for K in (8, 64, 65, 512, 2048, 8192, 14336):
            assert 1 <= shares(N, K) <= min(8, -(-K // 64))
    assert shares(0, 64) == shares(64, 0) == 0


def test_small_matrices_stay_with_multiply_adds():
    """Where a product of a few tokens is shorter than the three-term product's two kernels the 32-bit path widens the matrix as it did, by the
    whole product's sizes alone; matrices of real widths are kept as they were stored."""
    from fastmlx_b200 import kernels as k
    pays = lambda N, K: k.holds_exactly([torch.ones(N, K, dtype=torch.bfloat16)])
    assert not any(pays(N, K) for N, K in ((16, 64), (320, 80), (2048, 512), (64, 1024), (4096, 1024), (8192, 256)))
    assert all(pays(N, K) for N, K in ((16, 1032), (64, 2048), (2048, 2048), (8192, 1024), (16384, 512)))
    assert not k.three_terms_pay(64, 0) and not k.three_terms_pay(0, 512)
    half = torch.ones(4096, 1024, dtype=torch.bfloat16)
    assert k.holds_exactly([half, half]) and not k.holds_exactly([half])          # rows of one product count together
    big = torch.ones(64, 2048, dtype=torch.bfloat16)
    big[5, 7] = float("inf")
    assert not k.holds_exactly([big]) and not k.holds_exactly([big.float()]) and not k.holds_exactly([torch.ones(64, 2047).bfloat16()])


def test_workspace_of_the_three_term_product_is_bounded():
    """At most 256 MB of terms: more tokens go in waves, as a call and in the native executor's arena."""
    import ctypes
    from fastmlx_b200.engine import native as nat
    from fastmlx_b200.kernels import load
    lib = load("tc")
    for K in (8, 2048, 8192, 14336, 65536):
        rows = lib.fmx_gemm_three_rows(K)
        assert rows % 128 == 0 and rows >= 128
        for M in (1, 333, 8192, 1 << 20):
            assert lib.fmx_gemm_three_bytes(M, K) == 6 * min(M, rows) * K <= 256 << 20
    rt = type("Runtime", (), dict(dtype=torch.float32))()
    b = nat.ProgramBuilder(rt, None)
    x, w = b.reg(14336), torch.zeros(64, 14336, dtype=torch.bfloat16)
    b.op(nat.OP_LINEAR, in0=x, out0=b.reg(64), n=64, k=14336, terms=b.terms(x, w))
    host, table = nat.host_library(), nat.FmxKernelTable()
    for name, _ in table._fields_:
        setattr(table, name, 1)
    ops, regs = (nat.FmxOp * 1)(*b.ops), (nat.FmxReg * len(b.regs))(*[nat.FmxReg(*r) for r in b.regs])
    ex = host.fmx_exec_create(ops, 1, regs, len(b.regs), ctypes.byref(table), 148, None, None, 0)
    assert ex
    for T in (16, 3000, 8192):
        assert host.fmx_exec_arena_bytes(ex, T) <= T * (14336 + 64) * 4 + min(6 * T * 14336, 256 << 20) + 1024
    host.fmx_exec_destroy(ex)


def test_a_refused_launch_of_the_three_term_product_is_an_error(tmp_path):
    """Either of its two kernels: a product over terms that were never written would leave wrong numbers and say nothing."""
    from fastmlx_b200.csrc import build
    try:
        nvcc = build.find_nvcc()
    except build.BuildError:
        pytest.skip("nvcc is not installed")
    here, exe = os.path.dirname(os.path.abspath(__file__)), str(tmp_path / "refused_launch")
    subprocess.run([nvcc, *build.NVCC_FLAGS, "-I", os.path.join(build.HERE, "tc"), os.path.join(here, "refused_launch.cu"),
                    os.path.join(build.HERE, "common", "error.cu"), "-o", exe], check=True)
    lines = [tuple(map(int, l.split())) for l in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()]
    assert lines == [(0, 2), (1, 1), (1, 2)]


@pytest.mark.parametrize("hd,nh,nkv,rows,q,ctx,window,capped,mma,tc", [
    (64, 32, 8, 1, 128, 2000, 64, True, 8.9, 10.9), (64, 16, 16, 1, 128, 2000, 64, True, 8.9, 12.0),
    (64, 16, 16, 1, 512, 2000, 128, True, 11.3, 13.2), (64, 32, 8, 1, 64, 2000, 256, True, 15.0, 14.3),
    (64, 32, 8, 8, 128, 2000, 64, True, 18.9, 13.7), (64, 32, 8, 1, 2048, 2000, 64, True, 29.1, 25.0),
    (64, 16, 1, 1, 512, 0, 0, True, 20.5, 15.3), (64, 32, 8, 1, 64, 0, 0, True, 6.6, 7.9), (64, 32, 8, 1, 64, 512, 0, True, 22.2, 15.8),
    (128, 16, 16, 32, 16, 2000, 128, True, 28.8, 48.4), (128, 16, 16, 1, 512, 2000, 256, True, 20.9, 28.9),
    (128, 32, 8, 1, 64, 2000, 64, True, 12.5, 17.1), (128, 16, 1, 1, 64, 2000, 128, True, 15.3, 18.8),
    (128, 32, 8, 1, 2048, 2000, 128, True, 68.3, 39.5), (128, 32, 8, 1, 128, 2000, 1024, True, 54.2, 44.3),
    (128, 12, 4, 1, 512, 2000, 128, True, 15.7, 23.2), (128, 32, 8, 1, 512, 512, 0, True, 62.5, 40.2),
    (64, 32, 8, 1, 64, 2000, 128, False, 9.8, 12.7)])
def test_two_term_attention_goes_where_it_is_faster(hd, nh, nkv, rows, q, ctx, window, capped, mma, tc):
    """The choice between the two kernels of the two-term attention, at sizes that were timed on both (us): by the keys that a block walks and the
    rows that fill its tile, not by the longest context alone."""
    from fastmlx_b200 import kernels as k
    assert k.wide_tc_pays(hd, nh // nkv, nkv, rows, rows * q, q, ctx + q, window, capped) == (tc < mma)
