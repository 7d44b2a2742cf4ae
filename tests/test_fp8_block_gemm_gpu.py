"""Block-scaled fp8 products (csrc/kernels/gemm_fp8.cu) against float64 at the edges of both kernels: token counts around every tile width of the
decode-shape kernel and the line to the prompt-shape one, output widths that end inside a tile, K that ends inside a block, shares of K of every size."""
import pytest
import torch

from sglang_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 9, 16, 17, 32, 33, 64, 65, 100, 128, 129, 300, 513])
@pytest.mark.parametrize("N,K", [(8, 128), (136, 400), (1024, 2048), (2056, 1152), (4480, 256)])
def test_edges(M, N, K):
    assert ops.load_native()
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N + K)
    kb, nb = (K + 127) // 128, (N + 127) // 128
    xq = (torch.randn(M, K, generator=g, device="cuda") * 40).to(torch.float8_e4m3fn)
    wq = (torch.randn(N, K, generator=g, device="cuda") * 40).to(torch.float8_e4m3fn)
    xs = torch.rand(M, kb, generator=g, device="cuda") * 0.02 + 0.001
    ws = torch.rand(nb, kb, generator=g, device="cuda") * 0.02 + 0.001
    out = torch.full((M, N + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    torch.ops.sglb.gemm_fp8_block(xq, xs, wq, ws, out[:, :N])
    x = xq.double() * xs.double().repeat_interleave(128, 1)[:, :K]
    w = wq.double() * ws.double().repeat_interleave(128, 1)[:, :K].repeat_interleave(128, 0)[:N]
    ref = x @ w.T
    # bf16 output: 7 stored mantissa bits, so half an ulp is at most 2^-8 of a value; the fp32 partial sums stay within 2^-16 of the terms' root sum of squares
    bound = ref.abs() * 2 ** -8 + (x.square() @ w.square().T).sqrt() * 2 ** -16
    assert bool(((out[:, :N].double() - ref).abs() <= bound).all()), float(((out[:, :N].double() - ref).abs() / bound).max())
    assert bool((out[:, N:] == 7).all())


@pytest.mark.parametrize("N,K", [(1024, 4096), (7168, 1024)])
def test_rows_of_one_kernel_are_alike(N, K):
    """from 65 rows on one kernel sums K in sequence: a row's bits do not follow how many others there are"""
    g = torch.Generator(device="cuda").manual_seed(N)
    xq = (torch.randn(200, K, generator=g, device="cuda") * 40).to(torch.float8_e4m3fn)
    wq = (torch.randn(N, K, generator=g, device="cuda") * 40).to(torch.float8_e4m3fn)
    xs = torch.rand(200, K // 128, generator=g, device="cuda") * 0.02 + 0.001
    ws = torch.rand(N // 128, K // 128, generator=g, device="cuda") * 0.02 + 0.001
    whole = torch.empty(200, N, device="cuda", dtype=torch.bfloat16)
    torch.ops.sglb.gemm_fp8_block(xq, xs, wq, ws, whole)
    for M in (65, 96, 128, 129):
        out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
        torch.ops.sglb.gemm_fp8_block(xq[:M], xs[:M], wq, ws, out)
        assert torch.equal(out, whole[:M])
