"""The 64-token form of the Mamba-2 recurrence (csrc/kernels/mamba_chunk.cu) against float64: lengths around the chunk, one and two heads a CTA, both state
sizes, every source of step and decay; its error must be that of fp32 sums.  Values that are not finite stay with their column and the tokens behind them."""
import pytest
import torch

from sglang_b200 import ops

pytestmark = pytest.mark.gpu


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def _inputs(H, P, N, G, lens, mode, dt_t, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    T, B = sum(lens), len(lens)
    u = torch.nn.functional.silu(rnd(T, H * P + 2 * G * N))
    z = rnd(T, H * P + 8).to(dt_t)[:, : H * P] if mode != "decay" else None
    D = 1 + 0.1 * rnd(H) if mode != "gates" else None
    state = rnd(B + 2, H, N, P)
    kw, args = {}, (None, None, None)
    if mode == "step":
        raw, bias, A_log = rnd(T, H).to(dt_t), rnd(H) - 3, rnd(H).abs()
        args = (raw, bias, A_log)
        dt = torch.log1p(torch.exp(raw.double() + bias.double()))
        da = torch.exp(-A_log.double().exp() * dt)
    elif mode == "decay":
        kw["decay"] = torch.rand(H, generator=g, device="cuda") * 0.2 + 0.8
        dt, da = torch.ones(T, H, device="cuda", dtype=torch.float64), kw["decay"].double().expand(T, H)
    else:                                                        # (a decay of zero forgets everything: no logarithm of it may be taken)
        kw["gates"] = torch.rand(T, H, 3, generator=g, device="cuda").masked_fill_(torch.rand(T, H, 1, generator=g, device="cuda") < 0.02, 0.0).contiguous()
        da, dt = kw["gates"][..., 0].double(), kw["gates"][..., 1].double()
    old = [50 if i % 2 else 0 for i in range(B)]
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    rows = [B - i for i in range(B)]
    call = lambda st, **more: ops.mamba2_scan(u, z, *args, D, st, _i32(rows), _i32([a + b for a, b in zip(lens, old)]), _i32(cu), _i32(lens),  # noqa: E731
                                              H, P, N, G, **kw, **more)
    return u, z, D, dt, da, state, old, cu, rows, call


def _oracle(H, P, N, G, lens, u, z, D, dt, da, state, old, cu, rows):
    x, b, c = u.double().split([H * P, G * N, G * N], dim=-1)
    x, b, c = x.view(-1, H, P), b.view(-1, G, N).repeat_interleave(H // G, 1), c.view(-1, G, N).repeat_interleave(H // G, 1)
    ref, s0 = torch.empty_like(x), state.double().clone()
    for r, n in enumerate(lens):
        S = s0[rows[r]] if old[r] else torch.zeros_like(s0[0])
        for t in range(cu[r], cu[r + 1]):
            S = S * da[t][:, None, None] + (dt[t][:, None] * b[t])[:, :, None] * x[t][:, None, :]
            ref[t] = torch.einsum("hnp,hn->hp", S, c[t])
        s0[rows[r]] = S
    if D is not None:
        ref = ref + D.double()[None, :, None] * x
    ref = ref.view(-1, H * P)
    return (ref if z is None else ref * torch.nn.functional.silu(z.double())), s0


@pytest.mark.parametrize("H,P,N,G", [(8, 64, 128, 2), (2, 64, 64, 1), (2, 128, 128, 2), (3, 256, 64, 1)])
@pytest.mark.parametrize("lens", [[48], [64], [65, 0, 63], [1, 128, 130, 7], [31, 33, 1, 200]])
@pytest.mark.parametrize("mode", ["step", "decay", "gates"])
@pytest.mark.parametrize("bf16", [True, False])
def test_against_float64(H, P, N, G, lens, mode, bf16):
    u, z, D, dt, da, state, old, cu, rows, call = _inputs(H, P, N, G, lens, mode, torch.bfloat16 if bf16 else torch.float32, sum(lens) * 13 + H)
    ref, s0 = _oracle(H, P, N, G, lens, u, z, D, dt, da, state, old, cu, rows)
    y = call(state)
    # fp32 sums of N products and of up to 64 tokens: a few 2^-24 of the whole in the 2-norm
    for got, want in ((y, ref), (state, s0)):
        assert float((got.double() - want).norm() / want.norm()) < 6e-7, float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("bad", [float("inf"), float("nan"), 3.4e38])
def test_values_that_are_not_finite_stay_behind(bad):
    H, P, N, G, lens = 4, 64, 128, 1, [100, 90]
    u, z, D, dt, da, state, old, cu, rows, call = _inputs(H, P, N, G, lens, "step", torch.float32, 7)
    want, _ = _oracle(H, P, N, G, lens, u, z, D, dt, da, state, old, cu, rows)
    u[30, 5] = bad                                               # request 0, token 30, column 5
    y = call(state)
    hit = torch.zeros_like(y, dtype=torch.bool)
    hit[30:100, 5] = True
    if bad != 3.4e38:                                            # (finite, but its bf16 rounding is not: what follows may come back to numbers)
        assert not torch.isfinite(y[hit]).any()
    assert float((y[~hit].double() - want[~hit]).norm() / want[~hit].norm()) < 6e-7


@pytest.mark.parametrize("bf16", [True, False])
def test_infinite_and_large_gates(bf16):
    """z / (1 + exp(-z)) over the whole range: infinity stays infinite with the sign of what it scales, large negative gates close"""
    H, P, N, G, lens = 4, 64, 128, 1, [100, 90]
    u, z, D, dt, da, state, old, cu, rows, call = _inputs(H, P, N, G, lens, "step", torch.bfloat16 if bf16 else torch.float32, 9)
    z[7], z[8], z[9], z[70], z[71], z[72] = float("inf"), 1e30, -1e30, 20.0, 19.9, 80.0
    z[10, 3], z[120, 5] = float("inf"), float("nan")
    want, _ = _oracle(H, P, N, G, lens, u, z, D, dt, da, state, old, cu, rows)
    y = call(state)
    assert torch.isinf(y[7]).all() and torch.isinf(y[10, 3]) and torch.equal(y[7] > 0, want[7] > 0) and (y[10, 3] > 0) == (want[10, 3] > 0)
    assert torch.equal(torch.isfinite(y), torch.isfinite(want)) and float(y[9].abs().max()) < 1e-30
    for rows_ in (y[8].double() / want[8], y[70:73].double() / want[70:73]):
        assert float((rows_ - 1).abs().median()) < 3e-7              # (a factor of an ulp at most on fp32 sums)
    ok = torch.isfinite(want)
    ok[8] = False
    assert float((y[ok].double() - want[ok]).norm() / want[ok].norm()) < 6e-7


def test_groups_in_slices_and_under_capture(monkeypatch):
    """more chunks of B, C and their products than the workspace holds at once; replayed from a graph, against the token-by-token order"""
    H, P, N, G, lens = 16, 128, 128, 16, [9700, 300]
    u, z, D, dt, da, state, old, cu, rows, call = _inputs(H, P, N, G, lens, "step", torch.bfloat16, 3)
    s1, s2, keep = state.clone(), state.clone(), state.clone()
    monkeypatch.setenv("SGLB_FIXED_ORDER", "1")
    want = call(s1)
    monkeypatch.delenv("SGLB_FIXED_ORDER")
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call(s2)
    torch.cuda.current_stream().wait_stream(side)
    # (index tensors have to exist before the capture)
    rows_t, seq_t, cu_t, q_t = _i32(rows), _i32([a + b for a, b in zip(lens, old)]), _i32(cu), _i32(lens)
    raw, bias, A_log = (torch.randn(sum(lens), H, device="cuda").to(torch.bfloat16), torch.randn(H, device="cuda") - 3, torch.randn(H, device="cuda").abs())
    s3, s4 = keep.clone(), keep.clone()
    eager = ops.mamba2_scan(u, z, raw, bias, A_log, D, s3, rows_t, seq_t, cu_t, q_t, H, P, N, G)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = ops.mamba2_scan(u, z, raw, bias, A_log, D, s4, rows_t, seq_t, cu_t, q_t, H, P, N, G)
    s4.copy_(keep)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, eager) and torch.equal(s3, s4)
    # both orders are fp32 sums: each within a few 2^-24 of the exact one (the token order's chain is 9700 long)
    got = call(keep)
    assert float((got.double() - want.double()).norm() / want.double().norm()) < 3e-6
    assert float((keep.double() - s1.double()).norm() / s1.double().norm()) < 3e-6
    assert torch.equal(s2, keep)


def _values(dist, T, H, P, N, G, g):
    """rows of [x | B | C] whose products add up in every way: independent, of one sign, all alike, alternating, over six decades, one term alone, pairs that cancel"""
    r = torch.randn(T, H * P + 2 * G * N, generator=g, device="cuda")
    b, c = r[:, H * P:H * P + G * N].view(T, G, N), r[:, H * P + G * N:].view(T, G, N)
    if dist == "positive":
        r.abs_()
    elif dist == "ones":
        r.fill_(1.0)
    elif dist == "alternating":
        r.abs_()[:, H * P:].mul_(1.0 - 2.0 * (torch.arange(2 * G * N, device="cuda") % 2))
    elif dist == "mixed":
        r.mul_(10 ** (torch.rand(r.shape, generator=g, device="cuda") * 6 - 3))
    elif dist in ("one term", "one moving term"):
        keep = torch.full((T, G, 1), 3, device="cuda") if dist == "one term" else torch.randint(0, N, (T, G, 1), generator=g, device="cuda")
        hot = torch.zeros(T, G, N, device="cuda").scatter_(2, keep, 1.0)
        b.mul_(hot), c.mul_(hot)
    elif dist == "cancelling":
        b[..., 1::2] = b[..., ::2] * 1.001
        c[..., 1::2] = -c[..., ::2]
    return r


@pytest.mark.parametrize("H,P,N,G", [(8, 64, 128, 2), (4, 128, 128, 2), (4, 64, 64, 2)])
@pytest.mark.parametrize("lens", [[500, 130], [65, 129, 193, 65, 1]])        # (with chunks of a single token)
@pytest.mark.parametrize("mode", ["step", "decay", "one"])
@pytest.mark.parametrize("dist", ["normal", "positive", "ones", "alternating", "mixed", "one term", "one moving term", "cancelling"])
def test_error_against_the_sum_of_magnitudes(H, P, N, G, lens, mode, dist):
    """The constants that carry the accumulator's truncation back were measured on independent values: whatever the sums look like, down to one term and a decay and step
    of exactly 1, an error stays one of fp32 sums.  Scale: the same recurrence over magnitudes, which no cancellation shrinks."""
    g = torch.Generator(device="cuda").manual_seed(len(lens) + N + P)
    T, B = sum(lens), len(lens)
    u, state = _values(dist, T, H, P, N, G, g), torch.randn(B, H, N, P, generator=g, device="cuda")
    args, kw = (None, None, None), {}
    if mode == "step":
        raw, bias, A_log = torch.randn(T, H, generator=g, device="cuda"), torch.randn(H, generator=g, device="cuda") - 3, torch.randn(H, generator=g, device="cuda").abs()
        args = (raw, bias, A_log)
        dt = torch.log1p(torch.exp(raw.double() + bias.double()))
        da = torch.exp(-A_log.double().exp() * dt)
    else:
        kw["decay"] = torch.ones(H, device="cuda") if mode == "one" else torch.rand(H, generator=g, device="cuda") * 0.2 + 0.8
        dt, da = torch.ones(T, H, device="cuda", dtype=torch.float64), kw["decay"].double().expand(T, H)
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    rows, past = list(range(B)), [9] * B
    want, s_want = _oracle(H, P, N, G, lens, u, None, None, dt, da, state, past, cu, rows)
    size, s_size = _oracle(H, P, N, G, lens, u.abs(), None, None, dt, da, state.abs(), past, cu, rows)
    y = ops.mamba2_scan(u, None, *args, None, state, _i32(rows), _i32([n + 9 for n in lens]), _i32(cu), _i32(lens), H, P, N, G, **kw)
    for got, ref, scale in ((y, want, size), (state, s_want, s_size)):
        # magnitudes that decayed below 1e-24 meet the end of the bf16 parts' range (2^-126, 24 bits further down): they count as that
        e = (got.double() - ref).abs() / scale.clamp(min=1e-24)
        # at worst: one accumulator takes up to eight products of the largest part (N / 16) and as many truncations of 2^-24, M and the decays a few more: 2^-20.  In the
        # mean: half an ulp each for the sums of Y1, Y2 and of the state that Y1 reads, and for the factors on them, 2^-22 if all of them lean one way (eight tokens a
        # step come to 1.4e-7 on one term with constant decay; measured here 1.3e-7)
        assert float(e.max()) < 2 ** -20 and float(e.square().mean().sqrt()) < 2 ** -22, (float(e.max()), float(e.square().mean().sqrt()))


def test_more_requests_than_are_ordered():
    """beyond 256 requests none is taken by length, and the split kernel's threads look through several requests each; some are empty"""
    H, P, N, G = 2, 64, 128, 1
    g = torch.Generator().manual_seed(4)
    lens = [0 if i % 7 == 3 else int(n) for i, n in enumerate(torch.randint(1, 90, (300,), generator=g))]
    assert sum(lens) >= 24 * (len(lens) + 1)
    u, z, D, dt, da, state, old, cu, rows, call = _inputs(H, P, N, G, lens, "step", torch.bfloat16, 21)
    ref, s0 = _oracle(H, P, N, G, lens, u, z, D, dt, da, state, old, cu, rows)
    empty = [rows[i] for i, n in enumerate(lens) if n == 0]
    before = state[empty].clone()
    y = call(state)
    assert torch.equal(state[empty], before)
    live = [rows[i] for i, n in enumerate(lens) if n]
    assert float((y.double() - ref).norm() / ref.norm()) < 6e-7
    assert float((state[live].double() - s0[live]).norm() / s0[live].norm()) < 6e-7
