"""``SGLB_FIXED_ORDER`` (set by --enable-deterministic-inference): a token's row has the same bits alone and inside batches on every side of the lines at
which the kernels' dispatch changes over."""
import pytest
import torch

from sglang_b200 import ops
from sglang_b200.environ import envs
from sglang_b200.ops import moe_ops, quant_ops, torch_ref

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def fixed_order():
    assert ops.load_native()
    with envs.SGLB_FIXED_ORDER.override("1"):
        yield


@pytest.mark.parametrize("N,K", [(1024, 4096), (7168, 1024), (2048, 3584)])
def test_fp8_products(N, K):
    """buckets of 16, 32 and 64 tokens, the line behind them, one row tile and two"""
    g = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randn(300, K, generator=g, device="cuda").to(torch.bfloat16)
    wq, ws = torch_ref.block_quant_weight_fp8(torch.randn(N, K, generator=g, device="cuda") * 0.05, 128, False)
    whole = quant_ops.fp8_block_linear(x, wq, ws)
    for M in (1, 9, 16, 17, 33, 64, 65, 128, 129, 200):
        assert torch.equal(quant_ops.fp8_block_linear(x[:M], wq, ws), whole[:M]), M
        xq, xs = quant_ops.per_token_group_quant_fp8(x[:M])
        out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
        torch.ops.sglb.gemm_fp8_block(xq, xs, wq, ws, out, True)
        assert torch.equal(out, whole[:M]), M


@pytest.mark.parametrize("E,top,H,I", [(8, 2, 1024, 2048), (64, 4, 256, 96)])
@pytest.mark.parametrize("act", [None, ("relu2",), ("clamped_glu", 4.0, 1.702)])
def test_expert_blocks(E, top, H, I, act):
    """row tiles of 16 to 128, shared K, the line between the two kernels"""
    g = torch.Generator(device="cuda").manual_seed(E)
    T = 60 * E // top                                              # beyond the line
    x = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
    w13 = (torch.randn(E, I if act == ("relu2",) else 2 * I, H, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    w2 = (torch.randn(E, H, I, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    w, ids = moe_ops.topk_softmax(torch.randn(T, E, generator=g, device="cuda"), top, True)
    whole = moe_ops.fused_moe(x, w13, w2, w, ids, act=act)
    for M in (1, 5, 2 * E // top, 10 * E // top, 30 * E // top, 47 * E // top, 49 * E // top):
        assert torch.equal(moe_ops.fused_moe(x[:M], w13, w2, w[:M].contiguous(), ids[:M].contiguous(), act=act), whole[:M]), M
