"""``SGLB_FIXED_ORDER`` (set by --enable-deterministic-inference): a token's row has the same bits alone and inside batches on every side of the lines at
which the kernels' dispatch changes over."""
import pytest
import torch

from sglang_b200 import ops
from sglang_b200.environ import envs
from sglang_b200.ops import quant_ops, torch_ref

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
