"""The 16-byte forms of rotary + KV write, gated activation and fp8 activation quantiser against float64, beside the calls that keep the general form
(partial rotation, odd strides): tails of rows, one token, many heads, both cache types."""
import pytest
import torch

from sglang_b200 import ops
from sglang_b200.ops import quant_ops

pytestmark = pytest.mark.gpu


def _rope(x, cs, rot):
    c, s = (t.double()[:, None, :] for t in cs.chunk(2, dim=-1))
    a, b, rest = x.double().split([rot // 2, rot // 2, x.shape[-1] - rot], dim=-1)
    return torch.cat([a * c - b * s, b * c + a * s, rest], dim=-1)


@pytest.mark.parametrize("T,Hq,Hkv,D,rot,pad", [(1, 32, 8, 128, 128, 0), (3, 4, 1, 64, 64, 0), (5, 16, 8, 256, 256, 0), (129, 64, 8, 128, 128, 8), (7, 8, 2, 128, 64, 0),
                                                (7, 8, 2, 128, 128, 2), (33, 5, 5, 80, 80, 0)])
@pytest.mark.parametrize("fp8", [False, True])
def test_rope_kv_write(T, Hq, Hkv, D, rot, pad, fp8):
    g = torch.Generator(device="cuda").manual_seed(T * D + Hq)
    buf = torch.randn(T, (Hq + 2 * Hkv) * D + pad, generator=g, device="cuda").to(torch.bfloat16)
    qkv = buf[:, : (Hq + 2 * Hkv) * D]
    q, k, v = (t.view(T, -1, D) for t in qkv.split([Hq * D, Hkv * D, Hkv * D], dim=1))
    q0, k0, v0 = q.clone(), k.clone(), v.clone()
    ang = torch.rand(50, rot // 2, generator=g, device="cuda") * 6
    table = torch.cat([ang.cos(), ang.sin()], -1).contiguous()
    pos = torch.randint(0, 50, (T,), generator=g, device="cuda", dtype=torch.int32)
    loc = torch.randperm(T + 9, generator=g, device="cuda")[:T].to(torch.int32)
    dt = torch.float8_e4m3fn if fp8 else torch.bfloat16
    kc, vc = torch.zeros(T + 9, Hkv, D, device="cuda").to(dt), torch.zeros(T + 9, Hkv, D, device="cuda").to(dt)
    ops.rope_kv_write(q, k, v, pos, table, kc, vc, loc, True, 0.5 if fp8 else 1.0, 2.0 if fp8 else 1.0)
    cs = table[pos.long()]
    rq, rk = _rope(q0, cs, rot), _rope(k0, cs, rot)
    # half an ulp of the stored type: 2^-8 (bf16), 2^-4 (e4m3, 2^-10 below its smallest normal), plus fp32 products
    assert bool(((q.double() - rq).abs() <= rq.abs() * 2 ** -8 + 1e-6).all())
    rel, tiny = (2 ** -4, 2 ** -10) if fp8 else (2 ** -8, 1e-6)
    for got, ref, scale in ((kc, rk, 0.5 if fp8 else 1.0), (vc, v0.double(), 2.0 if fp8 else 1.0)):
        r = ref / scale
        assert bool(((got[loc.long()].double() - r).abs() <= r.abs() * rel * 1.001 + tiny).all())
    untouched = torch.ones(T + 9, dtype=torch.bool, device="cuda")
    untouched[loc.long()] = False
    assert float(kc.float()[untouched].abs().max()) == 0.0


@pytest.mark.parametrize("T,I", [(1, 8), (1, 14336), (2, 2056), (300, 4104), (2000, 520)])
def test_silu_and_mul(T, I):
    g = torch.Generator(device="cuda").manual_seed(T + I)
    x = (torch.randn(T, 2 * I, generator=g, device="cuda") * 6).to(torch.bfloat16)
    x[0, :4] = torch.tensor([-100.0, 100.0, 0.0, -87.5], device="cuda")
    a, b = x.double().chunk(2, -1)
    ref = a * torch.sigmoid(a) * b
    out = torch.ops.sglb.act_and_mul
    y = torch.empty(T, I, device="cuda", dtype=torch.bfloat16)
    out(x, y, 0)
    # exp of an fp32 argument up to 100 carries 100 x 2^-24 of itself; the rest is bf16's half ulp
    assert bool(((y.double() - ref).abs() <= ref.abs() * (2 ** -8 + 2e-5) + 1e-37).all())


@pytest.mark.parametrize("M,K,pad", [(1, 128, 0), (3, 8192, 0), (9, 400, 0), (7, 1160, 8), (5, 260, 0), (4, 256, 2), (65, 14336, 0)])
@pytest.mark.parametrize("ue8m0", [False, True])
def test_group_quant(M, K, pad, ue8m0):
    assert ops.load_native()
    g = torch.Generator(device="cuda").manual_seed(M + K)
    x = (torch.randn(M, K + pad, generator=g, device="cuda") * torch.exp(torch.randn(M, 1, generator=g, device="cuda"))).to(torch.bfloat16)[:, :K]
    kg = (K + 127) // 128
    q, s = torch.empty(M, K, device="cuda", dtype=torch.float8_e4m3fn), torch.empty(M, kg, device="cuda")
    torch.ops.sglb.per_token_group_quant_fp8(x, q, s, 128, ue8m0)
    xp = torch.zeros(M, kg * 128, device="cuda", dtype=torch.float64)
    xp[:, :K] = x.double()
    xg = xp.view(M, kg, 128)
    ref = xg.abs().amax(-1).clamp(min=1e-10) / 448.0
    if ue8m0:
        ref = torch.exp2(torch.ceil(torch.log2(ref.float()))).double()
    assert torch.equal(s, ref.float())
    got = torch.zeros_like(xp)
    got[:, :K] = q.double()
    back = got.view(M, kg, 128) * s.double()[..., None]
    # half an ulp of e4m3 (2^-4 of a value, 2^-10 of the scale below the smallest normal), a whole one where the product with 1 / scale lands on a tie
    assert bool(((back - xg).abs() <= xg.abs() * 2 ** -4 * 1.001 + s.double()[..., None] * 2 ** -10).all())


def test_silu_and_mul_rounds_as_the_fused_epilogue():
    """the same bits as the product whose epilogue applies it (csrc/kernels/gemm_tc.cu), which an identity matrix hands exactly the same numbers: every
    gate bf16 has between 2^-20 and 80, times every mantissa"""
    assert ops.load_native()
    gates = torch.arange(-(1 << 15), 1 << 15, device="cuda").to(torch.int16).view(torch.bfloat16)
    gates = gates[(gates.float().abs() < 80) & (gates.float().abs() > 2 ** -20)]
    up = 1 + torch.arange(128, device="cuda").to(torch.bfloat16) / 128
    x = torch.cat([gates[:, None].expand(-1, 128), up[None].expand(gates.numel(), -1)], dim=1).contiguous()
    fused = ops.gemm_tc(x, torch.eye(256, device="cuda", dtype=torch.bfloat16), epilogue=ops.EPI_SILU_SPLIT)
    assert int((ops.silu_and_mul(x) != fused).sum()) == 0
