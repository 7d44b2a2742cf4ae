"""The two-tile prompt attention (csrc/kernels/attention_tc.cu) against float64 and, bit for bit, against the single-tile kernel: ragged requests whose
last pair has one tile, one row or a full pair, cached prefixes that end inside a key tile, group sizes, page sizes, with and without the causal mask."""
import pytest
import torch

from sglang_b200 import ops
from sglang_b200.environ import envs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hq,Hkv,page,copies", [(32, 8, 32, 1), (16, 16, 64, 2), (64, 4, 16, 1), (8, 1, 128, 4), (8, 8, 8, 3)])
@pytest.mark.parametrize("qs,past", [([2500], [0]), ([1, 700, 63, 64, 65, 33, 32, 1100, 31], [0, 0, 5, 130, 0, 127, 128, 1000, 600]), ([129, 2048, 3], [3000, 0, 0])])
@pytest.mark.parametrize("causal", [True, False])
def test_rows(Hq, Hkv, page, copies, qs, past, causal):
    qs, past = qs * copies, past * copies
    D, T, B = 128, sum(qs), len(qs)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert T * Hkv >= 2 * (128 // (Hq // Hkv)) * sms, "not enough query tiles for the kernel under test"
    g = torch.Generator(device="cuda").manual_seed(T + Hq)
    need = [(a + b + page - 1) // page for a, b in zip(qs, past)]
    order = torch.randperm(sum(need), generator=g, device="cuda") + 1
    table = torch.zeros(B + 1, max(need) + 1, dtype=torch.int32, device="cuda")
    off = 0
    for i, n in enumerate(need):
        table[B - i, :n] = order[off:off + n].int()
        off += n
    kv = torch.randn(2, (sum(need) + 1) * page, Hkv, D, generator=g, device="cuda").to(torch.bfloat16)
    q = (torch.randn(T, Hq, D, generator=g, device="cuda") * 2).to(torch.bfloat16)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    cu = [0]
    for a in qs:
        cu.append(cu[-1] + a)

    def attend():
        lse = torch.full((T, Hq), 7.0, device="cuda")
        return ops.paged_attention(q, kv[0], kv[1], table, i32([B - i for i in range(B)]), i32([a + b for a, b in zip(qs, past)]), i32(cu), i32(qs), max(qs),
                                   page, D ** -0.5, causal=causal, lse=lse), lse

    o, lse = attend()
    with envs.SGLB_ATTN_PERSIST.override(False):
        o1, lse1 = attend()                       # one query tile a CTA
    assert torch.equal(o, o1) and torch.equal(lse, lse1)
    for i in range(B // copies):
        L, a = qs[i] + past[i], qs[i]
        pos = torch.arange(L, device="cuda")
        slot = table[B - i].long()[pos // page] * page + pos % page
        k, v = (kv[j][slot].repeat_interleave(Hq // Hkv, 1).double() for j in (0, 1))
        rows = sorted({0, 1, 31, 32, 63, 64, 127, 128, a // 2, a - 2, a - 1} & set(range(a)))
        x = q[cu[i]:cu[i + 1]][rows].double()
        s = torch.einsum("rhd,lhd->hrl", x, k) * D ** -0.5
        if causal:
            s = s.masked_fill(pos[None, None] > (past[i] + torch.tensor(rows, device="cuda"))[None, :, None], float("-inf"))
        ref = torch.einsum("hrl,lhd->rhd", s.softmax(-1), v)
        got = o[cu[i]:cu[i + 1]][rows].double()
        # probabilities and results are rounded to bf16 (2^-9 each in the root mean square)
        assert float((got - ref).norm() / ref.norm()) < 3 * 2 ** -9
        assert float((lse[cu[i]:cu[i + 1]][rows].double() - torch.logsumexp(s, -1).T).abs().max()) < 1e-3
