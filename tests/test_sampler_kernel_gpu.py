"""The cluster sampler (csrc/kernels/sampling.cu) against a float64 oracle that draws with the same counter generator: every row's token and
log-probability, at vocabularies around the slice, warp and vector edges, at several batch sizes, for rows that ask for
different settings."""
import pytest
import torch

from sglang_b200 import ops

pytestmark = pytest.mark.gpu
M64 = (1 << 64) - 1


def _uniform(seed, a, b):
    z = (seed + 0x9E3779B97F4A7C15 * (a + 1) + 0xD1B54A32D192ED03 * (b + 1)) & M64
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & M64
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M64
    z ^= z >> 31
    return (z >> 40) / 16777216.0


def _check_row(logits, temp, top_k, top_p, min_p, u, token, lp):
    l = logits.double()
    V = l.numel()
    d = (l.max() - l) / max(temp, 1e-6)
    r = torch.exp(-d)
    ref_lp = (-d[token] - torch.log(r.sum())).item()
    # fp32 sums of V exponentials whose arguments carry 2^-24 of a logit: 1e-4 covers |logit| / T up to a few hundred
    assert abs(lp - ref_lp) < 1e-4 * max(1.0, abs(ref_lp)) + 1e-4, (lp, ref_lp)
    if top_k == 1:
        assert token == int(torch.argmax(logits))
        return
    # whole groups of equal d fall on one side; the kernel's finest bin is 7.6e-6 wide in d, so keep the oracle's edge fuzzy by twice that
    edges = [float("inf")]
    mass = r.sum()
    keep = torch.ones(V, dtype=torch.bool, device=l.device)
    if 0 < top_k < V:
        e = torch.sort(d).values[top_k - 1].item()
        keep &= d <= e + 2e-5
        mass = r[d <= e].sum()
        edges.append(e)
    if top_p < 1.0:
        sd, idx = torch.sort(d)
        cum = torch.cumsum(torch.where(sd <= edges[-1] + 1e-9, r[idx], torch.zeros_like(sd)), 0)
        n = int((cum < top_p * mass * (1 - 1e-6)).sum())
        edges.append(sd[min(n, V - 1)].item())
        keep &= d <= edges[-1] + 2e-5
    keep &= r >= min_p * (1 - 1e-6)
    assert bool(keep[token]), "token outside the kept set"
    m = torch.where(keep, r, torch.zeros_like(r))
    cum = torch.cumsum(m, 0)
    at = u * cum[-1].item()
    # the fp32 order of the sums moves the drawn point by less than 2e-5 of the total; so do, by their own mass, the elements next to the edge, which
    # the finest bin (and a target rounded to fp32) may put on either side: no more than two of them here
    slack = 2e-5 * cum[-1].item() + (2 * float(torch.exp(torch.tensor(-min(edges)))) if len(edges) > 1 else 0.0)
    assert cum[token].item() - m[token].item() <= at + slack and cum[token].item() >= at - slack, (token, u)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,V,pad", [(1, 7, 0), (3, 2047, 1), (5, 2056, 8), (19, 32000, 0), (23, 65537, 3), (40, 128256, 0), (2, 151936, 5), (2, 420001, 0)])
def test_rows_with_their_own_settings(dtype, B, V, pad):
    g = torch.Generator(device="cuda").manual_seed(B * 131 + V)
    full = torch.randn(B, V + pad, generator=g, device="cuda") * 1.5
    full.scatter_add_(1, torch.randint(0, V, (B, 40), generator=g, device="cuda"), 9 + 2 * torch.randn(B, 40, generator=g, device="cuda"))
    logits = full.to(dtype)[:, :V]
    if V > 64:
        logits[0, V // 2:] = float("-inf")                       # a masked half
    kinds = [(1.0, 1, 1.0, 0.0), (0.7, 1 << 30, 0.9, 0.0), (0.8, 50, 0.95, 0.0), (1.0, 1 << 30, 1.0, 0.05), (1.3, 0, 1.0, 0.0), (1.0, 5, 1.0, 0.0),
             (0.02, 1 << 30, 0.5, 0.0), (1.0, 1 << 30, 0.999, 0.0), (2.0, max(1, V - 1), 0.3, 0.0)]
    rows = [kinds[(i + V) % len(kinds)] for i in range(B)]
    t, k, p, m = (torch.tensor([x[j] for x in rows], device="cuda") for j in range(4))
    lp = torch.empty(B, device="cuda")
    slots = torch.arange(B, device="cuda", dtype=torch.int32).flip(0).contiguous()
    nxt = torch.full((B,), -1, device="cuda", dtype=torch.int32)
    seeds = torch.tensor([[77 + i, i if i % 2 else -1] for i in range(B)], device="cuda", dtype=torch.int64)
    for step in range(3):
        tok = ops.sample(logits, t.float(), k.to(torch.int32), p.float(), m.float(), seeds=seeds, out_slots=slots, next_token_buf=nxt, out_logprobs=lp,
                         global_seed=1234, step=step)
        assert torch.equal(nxt[slots.long()], tok)
        for i in range(B):
            u = _uniform(77 + i, 0, i) if i % 2 else _uniform(1234, i, step)
            _check_row(logits[i].float(), *rows[i], u, int(tok[i]), float(lp[i]))


def test_flat_and_masked_rows():
    """equal logits meet in one bin (top-k keeps the whole tie group); a row with a single finite logit yields it; one without any yields a valid id"""
    V = 50000
    logits = torch.zeros(4, V, device="cuda")
    logits[1] = float("-inf")
    logits[1, 4321] = 3.0
    logits[2] = float("-inf")
    ones = torch.ones(4, device="cuda")
    k = torch.tensor([10, 1 << 30, 1, 1 << 30], device="cuda", dtype=torch.int32)
    tok = ops.sample(logits, ones, k, ones * 0.9, ones * 0, global_seed=5, step=1)
    assert int(tok[1]) == 4321 and 0 <= int(tok[2]) < V
    assert abs(int(tok[0]) - _uniform(5, 0, 1) * V) <= 2 + 1e-5 * V and abs(int(tok[3]) - _uniform(5, 3, 1) * V) <= 2 + 1e-5 * V


@pytest.mark.parametrize("B", [3, 300])
@pytest.mark.parametrize("V", [1, 7, 256, 2047])
def test_short_rows(B, V):
    """most CTAs of a row's cluster have nothing to read and reach the exchange of maxima at once: none may write to a peer that has not started"""
    g = torch.Generator(device="cuda").manual_seed(V)
    one, k = torch.ones(B, device="cuda"), torch.ones(B, device="cuda", dtype=torch.int32)
    for _ in range(20):
        logits = torch.randn(B, V, generator=g, device="cuda")
        assert torch.equal(ops.sample(logits, one, k, one, one * 0, global_seed=3, step=1).long(), logits.argmax(-1))


def test_masked_logits_are_never_drawn():
    """the drawn point at the very end of the kept mass, where rounding decides whether any running sum passes it: the last logit that has mass, not a
    masked one behind it"""
    B, V, live = 512, 3000, 1000
    assert _uniform(11, 0, 24699704) == 1 - 2.0 ** -24
    g = torch.Generator(device="cuda").manual_seed(8)
    logits = torch.randn(B, V, generator=g, device="cuda")
    logits[:, live:] = float("-inf")
    one = torch.ones(B, device="cuda")
    seeds = torch.tensor([[11, 24699704]] * B, device="cuda")
    for p in (1.0, 0.9999999):
        tok = ops.sample(logits, one, one.int() * 0, one * p, one * 0, seeds=seeds, global_seed=1, step=1)
        assert int(tok.max()) < live and int(tok.min()) > live - 50


@pytest.mark.parametrize("V,top_p", [(262144, 0.9), (524288, 0.5), (200000, 0.99999)])
@pytest.mark.parametrize("tail", [0.0, -1.011266])
def test_plateaus(V, top_p, tail):
    """rows whose logits nearly all meet in one bin: their fixed-point mass neither overflows nor, where each rounds down (16200.45 / 16384 of the bin's
    largest), sends the search through every bin: a pass over a row takes some microseconds, so all passes of a bounded search end within two milliseconds"""
    logits = torch.full((2, V), tail, device="cuda")
    logits[:, 5] = 0.0
    one, lp = torch.ones(2, device="cuda"), torch.empty(2, device="cuda")
    draw = lambda: ops.sample(logits, one, one.int() * 0, one * top_p, one * 0, out_logprobs=lp, global_seed=9, step=2)  # noqa: E731
    draw()
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    tok = draw()
    b.record()
    b.synchronize()
    assert a.elapsed_time(b) < 2.0, a.elapsed_time(b)
    for i in range(2):
        _check_row(logits[i], 1.0, 0, top_p, 0.0, _uniform(9, i, 2), int(tok[i]), float(lp[i]))


def test_a_row_does_not_follow_its_batch():
    """a seeded row's token and log-probability, bit for bit, alone and among others"""
    B, V = 40, 128256
    g = torch.Generator(device="cuda").manual_seed(21)
    logits = (torch.randn(B, V, generator=g, device="cuda") * 2).to(torch.bfloat16)
    kinds = [(1.0, 1, 1.0, 0.0), (0.7, 0, 0.9, 0.0), (0.8, 50, 0.95, 0.0), (1.0, 0, 1.0, 0.05), (1.3, 0, 1.0, 0.0)]
    t, k, p, m = (torch.tensor([kinds[i % 5][j] for i in range(B)], device="cuda") for j in range(4))
    seeds = torch.tensor([[77 + i, i] for i in range(B)], device="cuda")
    def draw(n):
        lp = torch.empty(n, device="cuda")
        tok = ops.sample(logits[:n], t[:n].float(), k[:n].int(), p[:n].float(), m[:n].float(), seeds=seeds[:n], out_logprobs=lp, global_seed=4, step=n)
        return tok, lp
    tok, lp = draw(B)
    for n in (1, 5, 8, 9, 17):
        a, b = draw(n)
        assert torch.equal(a, tok[:n]) and torch.equal(b, lp[:n])
