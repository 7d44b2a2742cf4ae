"""Expert blocks on pairs of SMs (csrc/kernels/gemm_grouped_pair.cu) against float64: rows that fill a tile, miss it by one step of 16 and spill over, every
tile size the round count can choose, widths that end inside a tile, K remainders, experts without rows and of another rank, both lines of its rule."""
import pytest
import torch

from sglang_b200 import ops

pytestmark = pytest.mark.gpu


def run_block(kernel, x, w13, w2, w, ids, off=0, act=None, weight_input=False):
    """the expert block by one of its kernels (0: weights streamed, 1: pairs of SMs, 2: 128-row tiles), whatever its sizes would choose"""
    out = torch.empty_like(x)
    if act is None:
        torch.ops.sglb.moe_grouped_mlp(x, w13, w2, w, ids, out, off, False, 0, kernel)
    elif act[0] == "relu2":
        torch.ops.sglb.moe_grouped_mlp_relu2(x, w13, w2, w, ids, out, off, weight_input, False, 0, kernel)
    else:
        torch.ops.sglb.moe_grouped_mlp_glu(x, w13, w2, w, ids, out, off, act[1], act[2], False, 0, kernel)
    return out


@pytest.mark.parametrize("E,K,H,I,rows", [
    (4, 1, 256, 128, [256, 257, 0, 1]), (4, 1, 128, 64, [512, 240, 16, 15]), (2, 1, 4096, 96, [700, 100]), (3, 1, 160, 416, [0, 0, 90]),
    (8, 1, 2048, 256, [1000] * 8), (8, 1, 512, 1024, [300, 200, 128, 129, 127, 64, 33, 7]), (300, 1, 128, 64, [4] * 300), (8, 1, 256, 2080, [7] * 8), (70, 1, 128, 96, [3] * 69 + [40])])
@pytest.mark.parametrize("act", [None, ("relu2",), ("clamped_glu", 4.0, 1.702)])
@pytest.mark.parametrize("off", [0, 3])
@pytest.mark.parametrize("kernel", [1, 0, 2])
def test_block(E, K, H, I, rows, act, off, kernel):
    assert ops.load_native()
    g = torch.Generator(device="cuda").manual_seed(sum(rows) + E + H)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    ids = torch.cat([torch.full((n,), e + off, dtype=torch.int32) for e, n in enumerate(rows)] + [torch.zeros(5 if off else 0, dtype=torch.int32)]).cuda()
    ids = ids[torch.randperm(ids.numel(), generator=g, device="cuda")][:, None].contiguous()        # (off: five rows of an expert that is not here)
    T = ids.shape[0]
    x, w = rnd(T, H).to(torch.bfloat16), torch.rand(T, 1, generator=g, device="cuda") + 0.1
    w13 = (rnd(E, (1 if act and act[0] == "relu2" else 2) * I, H) * H ** -0.5).to(torch.bfloat16)
    w2 = (rnd(E, H, I) * I ** -0.5).to(torch.bfloat16)
    for weight_input in ((False, True) if act and act[0] == "relu2" else (False,)):
        y = run_block(kernel, x, w13, w2, w, ids, off, act, weight_input)
        ref = torch.zeros(T, H, dtype=torch.float64, device="cuda")
        for e in range(E):
            t = (ids[:, 0] == e + off).nonzero()[:, 0]
            wt = w[t].double()
            u = (x[t].double() * (wt if weight_input else 1.0)) @ w13[e].double().T
            if act is None:
                a, u = u.chunk(2, -1)
                h = torch.nn.functional.silu(a) * u
            elif act[0] == "relu2":
                h = u.clamp(min=0).square()
            else:
                a, u = u.chunk(2, -1)
                a, u = a.clamp(max=act[1]), u.clamp(-act[1], act[1])
                h = a * torch.sigmoid(act[2] * a) * (u + 1)
            o = h @ w2[e].double().T
            ref[t] = o if weight_input else o * wt
        # three roundings to bf16 on the way (inner activations, an expert's output, the sum): 2^-9 each in the root mean square, relu2 doubles the first
        err = float((y.double() - ref).norm() / ref.norm())
        assert err < 4 * 2 ** -9, err
        far = (y.double() - ref).norm(dim=1) / ref.norm(dim=1).clamp(min=float(ref.norm() / T ** 0.5) * 0.05)
        assert float(far.max()) < 16 * 2 ** -9, float(far.max())


@pytest.mark.parametrize("rows", [20, 9, 70, 90, 130])
def test_tiles_of_odd_chunk_counts_in_a_row(rows):
    """one K block a tile, so that the epilogue is behind the products and takes tile after tile: gate and up warps swap values through two buffers, which have to
    alternate across tiles of one, three or five chunks (20, 9: 1, 70 and 90: 3, 130: 5) as well as inside a tile; the same bits every time, and the right ones"""
    assert ops.load_native()
    E, H, I = 300, 64, 1024
    g = torch.Generator(device="cuda").manual_seed(rows)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    ids = torch.arange(E, device="cuda", dtype=torch.int32).repeat_interleave(rows)[torch.randperm(E * rows, generator=g, device="cuda")][:, None].contiguous()
    x, w = rnd(E * rows, H).to(torch.bfloat16), torch.rand(E * rows, 1, generator=g, device="cuda") + 0.1
    w13, w2 = (rnd(E, 2 * I, H) * H ** -0.5).to(torch.bfloat16), (rnd(E, H, I) * I ** -0.5).to(torch.bfloat16)
    first = run_block(1, x, w13, w2, w, ids)
    ref = torch.zeros(E * rows, H, dtype=torch.float64, device="cuda")
    for e in range(E):
        t = (ids[:, 0] == e).nonzero()[:, 0]
        a, u = (x[t].double() @ w13[e].double().T).chunk(2, -1)
        ref[t] = (torch.nn.functional.silu(a) * u) @ w2[e].double().T * w[t].double()
    # three roundings to bf16, as above; a swapped value is as large as what it takes the place of
    err = (first.double() - ref).norm(dim=1) / ref.norm(dim=1).clamp(min=float(ref.norm() / (E * rows) ** 0.5) * 0.05)
    assert float(err.max()) < 16 * 2 ** -9, float(err.max())
    differ = torch.zeros((), dtype=torch.int64, device="cuda")
    for _ in range(300):
        differ += (run_block(1, x, w13, w2, w, ids) != first).sum()
    assert int(differ) == 0


def test_sizes_choose_pairs_and_match_one_order():
    """the dispatch itself reaches the pair kernel; it adds a row's K in sequence, as 128-row tiles do: the same bits"""
    from sglang_b200.ops import moe_ops

    E, H, I, T = 64, 2048, 768, 1300
    g = torch.Generator(device="cuda").manual_seed(2)
    x = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
    w13 = (torch.randn(E, 2 * I, H, generator=g, device="cuda") * H ** -0.5).to(torch.bfloat16)
    w2 = (torch.randn(E, H, I, generator=g, device="cuda") * I ** -0.5).to(torch.bfloat16)
    w, ids = moe_ops.topk_softmax(torch.randn(T, E, generator=g, device="cuda"), 2, True)
    assert torch.ops.sglb.moe_block_plan(2 * T, E, 0, H, I, 0, torch.cuda.get_device_properties(0).multi_processor_count, False) == [1, 16]
    y = moe_ops.fused_moe(x, w13, w2, w, ids)
    assert torch.equal(y, run_block(1, x, w13, w2, w, ids)) and torch.equal(y, run_block(2, x, w13, w2, w, ids))
    # told that twenty times as many experts share the rows, it streams weights in 16-row tiles: other sums of the same products
    z = moe_ops.fused_moe(x, w13, w2, w, ids, num_experts=20 * E)
    assert 0 < float((z.float() - y.float()).norm() / y.float().norm()) < 4 * 2 ** -9
