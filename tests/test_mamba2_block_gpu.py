"""The eight-token form of the Mamba-2 recurrence (csrc/kernels/mamba.cu) against float64: ragged lengths around the block, fresh and continued states,
every source of step and decay, with and without gate and skip; its error must be that of fp32 sums."""
import pytest
import torch

from sglang_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,P,N,G", [(4, 64, 128, 2), (2, 128, 64, 1), (6, 192, 128, 3)])
# (the 64-token form takes 24 tokens a request and 24 more of the first two widths: [40, 1, 65] there, while [40, 1, 29, 1, 65, 1] stays below its line)
@pytest.mark.parametrize("lens", [[2], [7, 1, 8], [9, 16, 17, 3], [40, 1, 65], [40, 1, 29, 1, 65, 1], [47]])
@pytest.mark.parametrize("mode", ["step", "decay", "gates"])
@pytest.mark.parametrize("bf16", [True, False])
def test_against_float64(H, P, N, G, lens, mode, bf16):
    g = torch.Generator(device="cuda").manual_seed(sum(lens) * 13 + H)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    T, B, dt_t = sum(lens), len(lens), torch.bfloat16 if bf16 else torch.float32
    u = torch.nn.functional.silu(rnd(T, H * P + 2 * G * N))
    z = rnd(T, H * P + 8).to(dt_t)[:, : H * P] if mode != "decay" else None
    D = 1 + 0.1 * rnd(H) if mode != "gates" else None
    state = rnd(B + 2, H, N, P)
    s0 = state.double().clone()
    old = [50 if i % 2 else 0 for i in range(B)]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    rows = [B - i for i in range(B)]
    kw, args = {}, (None, None, None)
    if mode == "step":
        raw, bias, A_log = rnd(T, H).to(dt_t), rnd(H) - 3, rnd(H).abs()
        args = (raw, bias, A_log)
        dt = torch.log1p(torch.exp(raw.double() + bias.double()))
        da = torch.exp(-A_log.double().exp() * dt)
    elif mode == "decay":
        kw["decay"] = torch.rand(H, generator=g, device="cuda") * 0.2 + 0.8
        dt, da = torch.ones(T, H, device="cuda", dtype=torch.float64), kw["decay"].double().expand(T, H)
    else:
        kw["gates"] = torch.rand(T, H, 3, generator=g, device="cuda").contiguous()
        da, dt = kw["gates"][..., 0].double(), kw["gates"][..., 1].double()
    y = ops.mamba2_scan(u, z, *args, D, state, i32(rows), i32([a + b for a, b in zip(lens, old)]), i32(cu), i32(lens), H, P, N, G, **kw)
    x, b, c = u.double().split([H * P, G * N, G * N], dim=-1)
    x, b, c = x.view(T, H, P), b.view(T, G, N).repeat_interleave(H // G, 1), c.view(T, G, N).repeat_interleave(H // G, 1)
    ref = torch.empty_like(x)
    for r, n in enumerate(lens):
        S = s0[rows[r]] if old[r] else torch.zeros_like(s0[0])
        for t in range(cu[r], cu[r + 1]):
            S = S * da[t][:, None, None] + (dt[t][:, None] * b[t])[:, :, None] * x[t][:, None, :]
            ref[t] = torch.einsum("hnp,hn->hp", S, c[t])
        s0[rows[r]] = S
    if D is not None:
        ref = ref + D.double()[None, :, None] * x
    ref = ref.view(T, H * P)
    if z is not None:
        ref = ref * torch.nn.functional.silu(z.double())
    # fp32 sums of N products and of up to 65 tokens: a few 2^-24 of the whole in the 2-norm
    for got, want in ((y, ref), (state, s0)):
        assert float((got.double() - want).norm() / want.norm()) < 6e-7, float((got.double() - want).norm() / want.norm())
