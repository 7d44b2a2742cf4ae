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


@pytest.mark.parametrize("H,P,N,G", [(2, 64, 128, 2), (2, 128, 64, 1)])
@pytest.mark.parametrize("mode", ["step", "decay", "gates"])
def test_scan(H, P, N, G, mode):
    """a prompt alone, among others, among decode tokens (less than two tokens a request), and cut in two"""
    g = torch.Generator(device="cuda").manual_seed(N)
    lens = [37] + [1] * 60
    T, B = sum(lens), len(lens)
    u = torch.randn(T, H * P + 2 * G * N, generator=g, device="cuda")
    dt = torch.randn(T, H, generator=g, device="cuda")
    gates = torch.rand(T, H, 2, generator=g, device="cuda")
    first = torch.randn(B, H, N, P, generator=g, device="cuda")
    head = torch.rand(3, H, generator=g, device="cuda") * 0.5 + 0.3
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731

    def scan(state, t0, ls, past):
        t1, cu = t0 + sum(ls), [0]
        for n in ls:
            cu.append(cu[-1] + n)
        args, kw = (None, None, None), {}
        if mode == "step":
            args = (dt[t0:t1], head[0], head[1])
        elif mode == "decay":
            kw["decay"] = head[2]
        else:
            kw["gates"] = gates[t0:t1].contiguous()
        return ops.mamba2_scan(u[t0:t1].contiguous(), None, *args, None, state, i32(list(range(len(ls)))), i32([n + past for n in ls]), i32(cu), i32(ls), H, P, N, G, **kw)

    s_all = first.clone()
    y_all = scan(s_all, 0, lens, 50)
    s_one = first[:1].clone()
    assert torch.equal(scan(s_one, 0, lens[:1], 50), y_all[:37]) and torch.equal(s_one[0], s_all[0])
    s_few = first[:5].clone()
    assert torch.equal(scan(s_few, 0, lens[:5], 50), y_all[:41]) and torch.equal(s_few, s_all[:5])
    s_cut = first[:1].clone()
    parts = [scan(s_cut, 0, [13], 50), scan(s_cut, 13, [24], 63)]
    assert torch.equal(torch.cat(parts), y_all[:37]) and torch.equal(s_cut[0], s_all[0])
