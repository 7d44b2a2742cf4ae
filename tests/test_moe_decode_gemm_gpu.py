"""Expert blocks of few rows, against float64: the weight-streaming kernel (csrc/kernels/gemm_grouped_decode.cu) with row tiles of every size and their remainders,
output widths that end inside a tile, shared K, overfull experts, experts of another rank, every epilogue, and both sides of its lines (the blocks here are small or
narrow, which is where it stays ahead of pairs of SMs up to 32 and 48 rows an expert)."""
import pytest
import torch

from sglang_b200 import ops
from sglang_b200.ops import moe_ops

pytestmark = pytest.mark.gpu


def _ref(x, w13, w2, w, ids, off, act, weight_input):
    x, out = x.double(), torch.zeros(x.shape, dtype=torch.float64, device="cuda")
    for e in range(w13.shape[0]):
        t, j = (ids == e + off).nonzero(as_tuple=True)
        if t.numel() == 0:
            continue
        wt = w[t, j].double()[:, None]
        u = (x[t] * (wt if weight_input else 1.0)) @ w13[e].double().T
        if act is None:
            g, u = u.chunk(2, -1)
            h = torch.nn.functional.silu(g) * u
        elif act[0] == "relu2":
            h = u.clamp(min=0).square()
        else:
            g, u = u.chunk(2, -1)
            g, u = g.clamp(max=act[1]), u.clamp(-act[1], act[1])
            h = g * torch.sigmoid(act[2] * g) * (u + 1)
        y = h @ w2[e].double().T
        out.index_add_(0, t, y if weight_input else y * wt)
    return out


@pytest.mark.parametrize("T,E,K,H,I,off,skew", [(1, 8, 2, 512, 256, 0, 0), (9, 8, 2, 160, 96, 0, 0), (20, 8, 2, 4096, 1024, 0, 0), (20, 8, 2, 512, 256, 0, 4), (22, 8, 2, 512, 256, 3, 2), (40, 16, 4, 256, 160, 0, 0),
                                                (64, 8, 2, 512, 416, 0, 3), (130, 8, 2, 512, 256, 4, 0), (190, 8, 2, 256, 128, 0, 0), (194, 8, 2, 256, 128, 0, 0), (250, 8, 2, 256, 128, 0, 0),
                                                (260, 8, 2, 256, 128, 0, 0),
                                                (333, 128, 8, 256, 96, 0, 0), (3, 300, 1, 128, 64, 0, 0), (700, 8, 2, 256, 128, 0, 2), (2100, 128, 8, 128, 64, 0, 0)])
@pytest.mark.parametrize("act", [None, ("relu2",), ("clamped_glu", 4.0, 1.702)])
def test_block(T, E, K, H, I, off, skew, act):
    assert ops.load_native()
    g = torch.Generator(device="cuda").manual_seed(T * 3 + E + H)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x = rnd(T, H).to(torch.bfloat16)
    w13 = (rnd(E, (1 if act and act[0] == "relu2" else 2) * I, H) * H ** -0.5).to(torch.bfloat16)
    w2 = (rnd(E, H, I) * I ** -0.5).to(torch.bfloat16)
    logits = rnd(T, E + off)
    logits[:, off] += skew                       # an expert that most tokens choose needs several row tiles
    w, ids = moe_ops.topk_softmax(logits, K, True)
    for weight_input in ((False, True) if act and act[0] == "relu2" else (False,)):
        y = moe_ops.fused_moe(x, w13, w2, w, ids, off, act, weight_input)
        ref = _ref(x, w13, w2, w, ids, off, act, weight_input)
        # three roundings to bf16 on the way (inner activations, an expert's output, the sum): 2^-9 each in the root mean square, relu2 doubles the first
        err = float((y.double() - ref).norm() / ref.norm())
        assert err < 4 * 2 ** -9, err
        rows = (y.double() - ref).norm(dim=1) / ref.norm(dim=1).clamp(min=float(ref.norm() / T ** 0.5) * 0.05)
        assert float(rows.max()) < 16 * 2 ** -9, float(rows.max())


def test_rows_beyond_the_line_are_alike():
    """from 48 rows an expert on 128-row tiles sum K in sequence: a token's bits do not follow how many others there are"""
    E, K, H, I, T = 8, 2, 4096, 512, 400
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
    w13 = (torch.randn(E, 2 * I, H, generator=g, device="cuda") * H ** -0.5).to(torch.bfloat16)
    w2 = (torch.randn(E, H, I, generator=g, device="cuda") * I ** -0.5).to(torch.bfloat16)
    w, ids = moe_ops.topk_softmax(torch.randn(T, E, generator=g, device="cuda"), K, True)
    whole = moe_ops.fused_moe(x, w13, w2, w, ids)
    for n in (193, 224, 256):
        assert torch.equal(moe_ops.fused_moe(x[:n], w13, w2, w[:n], ids[:n]), whole[:n])
