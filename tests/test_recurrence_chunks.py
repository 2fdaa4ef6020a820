"""Walks of a matrix state sixteen tokens at a time against the same rules token by token in 64 bits: portions of one token, of whole chunks and of one
token more, several portions a step, shared q and k, decays near one and near zero, head sizes and columns on both sides of the kernels' variants.

Tolerance: q, k, v are given in bfloat16 and everything behind them is float32; a chunk's products split an operand into three bfloat16 parts, which leaves
2^-25 of a term, so outputs and states of a few hundred terms of size 1 differ by a few 1e-6 of their root mean square."""
import ctypes

import pytest
import torch

from mini_llm_runtime_b200.ops.specs import RecurrenceSpec

pytestmark = pytest.mark.gpu

RULES = {"decay": ("decay", None), "gla": ("decay", "sigmoid_root"), "delta": ("delta", None), "channel_delta": ("delta", "softplus"), "step": ("step", None)}


def make(rule, dim, vdim, heads, group, segments, seed=0, strong=0.0, silu=False):
    """The buffers and the description of a step; `strong` is added to what the decays come from."""
    kind, channel = RULES[rule]
    g = torch.Generator().manual_seed(seed + dim + vdim + heads)
    draw = lambda *shape: torch.randn(*shape, generator=g).cuda()
    rank, rows, qk = 16, sum(segments), heads // group
    ck, cv = qk * dim, 2 * qk * dim
    ca = cv + heads * vdim
    cb = ca + max(rank, heads)
    proj = draw(rows, (cb + heads + 7) // 8 * 8).bfloat16()
    held = dict(decay=(0.9 + 0.0999 * torch.rand(heads, generator=g)).cuda(), a_log=0.5 * draw(heads) + strong, skip=draw(heads),
                dt_bias=0.5 * (draw(heads * dim) if channel else draw(heads)), decay_w=(draw(rank, heads * dim) * rank ** -0.5).bfloat16())
    spec = RecurrenceSpec(decay=held["decay"].data_ptr(), a_log=held["a_log"].data_ptr(), dt_bias=held["dt_bias"].data_ptr(),
                          skip=held["skip"].data_ptr() if rule == "step" else None, decay_w=held["decay_w"].data_ptr() if channel else None,
                          decay_rank=rank if channel else 0, channel_decay=RecurrenceSpec.CHANNEL_DECAY[channel] if channel else 0, heads=heads, qk_heads=qk,
                          dim=dim, vdim=vdim, rule=RecurrenceSpec.RULE[kind], prep=RecurrenceSpec.PREP["unit" if kind == "delta" else None],
                          in_act=int(silu), gate_first=int(rule == "step"), norm_parts=heads, col_q=0, col_k=ck, col_v=cv, col_a=ca, col_b=cb,
                          q_mult=dim ** -0.5, k_mult=1.0 if kind == "delta" else dim ** -0.5, unit_eps=1e-6, eps=1e-5, out_scale=1.0, inv_tau=1 / 16)
    info, first = [], 0
    for i, n in enumerate(segments):
        info.append((first, n, 0, len(segments) - 1 - i))
        first += n
    info = torch.tensor([0] + [v for segment in info for v in segment], dtype=torch.int32, device="cuda")[1:]      # no wider border than an int's, as in a step
    positions = torch.cat([torch.arange(n) for n in segments]).to(torch.int32).cuda()
    state = draw(len(segments), heads * vdim * dim + 3)
    return dict(rule=rule, spec=spec, held=held, proj=proj, info=info, positions=positions, start=state, segments=segments, rank=rank, group=group, silu=silu)


def launch(c, state, chunks=True):
    """The plain outputs (before the read-out), a call that launches the same again, and what that call needs to live."""
    from mini_llm_runtime_b200.ops import native
    s, proj, rows = c["spec"], c["proj"], c["proj"].shape[0]
    f32 = lambda *shape: torch.full(shape, float("nan"), device="cuda")
    out = torch.empty(rows, s.heads * s.vdim, device="cuda", dtype=torch.bfloat16)
    q, k, gates, obuf, df = f32(rows, s.qk_heads * s.dim), f32(rows, s.qk_heads * s.dim), f32(rows, 2 * s.heads), f32(rows, s.heads * s.vdim), f32(rows, s.heads * s.dim)
    common = [ctypes.addressof(s), proj.data_ptr(), proj.stride(0), proj.data_ptr(), proj.stride(0)]
    tail = [out.data_ptr(), out.stride(0), state.data_ptr(), state.stride(0), c["info"].data_ptr(), len(c["segments"]), c["positions"].data_ptr(), rows,
            q.data_ptr(), k.data_ptr(), gates.data_ptr(), obuf.data_ptr(), df.data_ptr(), None, 0]
    held = []
    if chunks:
        places = (rows + 15) // 16 + len(c["segments"])
        held = [f32(places, s.heads * s.dim * 24), f32(places, s.heads * s.dim * 24), f32(places, s.heads * s.dim * 24), f32(rows, s.heads * 16),
                f32(places, s.heads * (s.dim if s.channel_decay else 36))]
        call = lambda: native.call("recurrence", "mlr_linear_recurrence_chunks", *common, *tail, *[t.data_ptr() for t in held], native.stream())
    else:
        call = lambda: native.call("recurrence", "mlr_linear_recurrence_split", *common, 1, *tail, native.stream())
    call()
    torch.cuda.synchronize()
    return obuf, call, (held, q, k, gates, df, out)


def exact(c):
    """Plain outputs and states, token by token in 64 bits."""
    s, h = c["spec"], c["held"]
    x = c["proj"].double()
    silu = (lambda t: t * torch.sigmoid(t)) if c["silu"] else (lambda t: t)
    rows, H, D, V = x.shape[0], s.heads, s.dim, s.vdim
    q = silu(x[:, :s.col_k]).view(rows, -1, D).repeat_interleave(c["group"], 1)
    k = silu(x[:, s.col_k:s.col_v]).view(rows, -1, D).repeat_interleave(c["group"], 1)
    v = silu(x[:, s.col_v:s.col_a]).view(rows, H, V)
    if s.prep == RecurrenceSpec.PREP["unit"]:
        q, k = (t / (t.square().sum(-1, keepdim=True) + s.unit_eps).sqrt() for t in (q, k))
    q, k = q * s.q_mult, k * s.k_mult
    a_log, dt_bias = h["a_log"].double(), h["dt_bias"].double()
    beta = torch.ones(rows, H, dtype=torch.float64, device="cuda")
    if s.channel_decay:
        z = (x[:, s.col_a:s.col_a + c["rank"]] @ h["decay_w"].double() + dt_bias).view(rows, H, D)
        decay = torch.sigmoid(z) ** s.inv_tau if s.channel_decay == 1 else torch.exp(-torch.exp(a_log)[:, None] * torch.nn.functional.softplus(z))
    elif c["rule"] == "decay":
        decay = h["decay"].double()[None, :, None].expand(rows, H, D)
    else:
        dt = torch.nn.functional.softplus(x[:, s.col_a:s.col_a + H] + dt_bias)
        decay = torch.exp(-torch.exp(a_log) * dt)[..., None].expand(rows, H, D)
        if c["rule"] == "step":
            beta = dt
    if c["rule"].endswith("delta"):
        beta = torch.sigmoid(x[:, s.col_b:s.col_b + H])
    out = torch.empty(rows, H, V, dtype=torch.float64, device="cuda")
    states, first = torch.empty(len(c["segments"]), H, V, D, dtype=torch.float64, device="cuda"), 0
    for i, n in enumerate(c["segments"]):
        slot = len(c["segments"]) - 1 - i
        S = c["start"][slot, :H * V * D].view(H, V, D).double()
        for t in range(first, first + n):
            S = S * decay[t][:, None, :]
            u = v[t]
            if c["rule"].endswith("delta"):
                u = u - torch.einsum("hvd,hd->hv", S, k[t])
            S = S + (beta[t][:, None] * u)[..., None] * k[t][:, None, :]
            out[t] = torch.einsum("hvd,hd->hv", S, q[t])
            if c["rule"] == "step":
                out[t] += h["skip"].double()[:, None] * v[t]
        states[slot], first = S, first + n
    return out.view(rows, H * V), states


def distance(got, want):
    return float((got.double() - want).square().mean().sqrt() / want.square().mean().sqrt())


@pytest.mark.parametrize("rule", list(RULES))
@pytest.mark.parametrize("dim,vdim,heads,group,segments,strong,silu", [
    (128, 128, 2, 1, [67], 0.0, False), (128, 16, 4, 2, [16, 1, 33, 15], 0.0, True), (64, 48, 2, 2, [17, 64], 0.0, False),
    (128, 64, 80, 8, [48, 31], 0.0, False),                    # more column tiles than SMs: two a block
    (64, 32, 160, 1, [40], 0.0, True), (128, 32, 2, 1, [100], 4.0, False),     # decays down to exp(-100) and beyond
])
def test_chunks_give_what_the_rules_say(rule, dim, vdim, heads, group, segments, strong, silu):
    c = make(rule, dim, vdim, heads, group, segments, strong=strong, silu=silu)
    state = c["start"].clone()
    got, _, _ = launch(c, state)
    want, want_state = exact(c)
    size = heads * vdim * dim
    assert distance(got, want) < 5e-6
    assert distance(state[:, :size].reshape(want_state.shape), want_state) < 5e-6
    assert torch.equal(state[:, size:], c["start"][:, size:])


def same_kinds(got, want):
    """Whether two tensors have NaN, infinities of each sign and finite numbers at the same places."""
    kind = lambda x: torch.where(torch.isnan(x), 2, torch.where(torch.isinf(x), torch.sign(x), 0)).to(torch.int8)
    return torch.equal(kind(got), kind(want))


@pytest.mark.parametrize("rule", list(RULES))
@pytest.mark.parametrize("dim,vdim,heads", [(64, 32, 2), (128, 64, 80)])       # one and two column tiles a block
@pytest.mark.parametrize("where,value", [("v", "nan"), ("v", "inf"), ("k", "nan"), ("k", "inf"), ("q", "nan"), ("state", "nan"), ("state", "inf")])
def test_a_value_that_is_not_finite_reaches_what_the_rules_say(rule, dim, vdim, heads, where, value):
    """In the middle of a request's second chunk: the tokens before it, other columns (where the rule keeps them apart) and other requests stay what
    they are, infinities stay infinities."""
    c = make(rule, dim, vdim, heads, 1, [40, 20])
    clean, _, _ = launch(c, c["start"].clone())
    if where == "state":
        c["start"][1, 5 * dim + 3] = float(value)              # the first request's column 5 of its first head
    else:
        s = c["spec"]
        c["proj"][24, {"v": s.col_v, "k": s.col_k, "q": s.col_q}[where] + 5] = float(value)
    state = c["start"].clone()
    got, _, _ = launch(c, state)
    want, want_state = exact(c)
    size = heads * vdim * dim
    for ours, true in ((got, want), (state[:, :size].reshape(want_state.shape), want_state)):
        assert same_kinds(ours, true)
        finite = torch.isfinite(true)
        assert distance(ours[finite], true[finite]) < 5e-6
    assert not torch.isfinite(got).all() and torch.isfinite(got[:24] if where != "state" else got[40:]).all()
    assert torch.equal(got[40:], clean[40:]) and torch.equal(got[:, vdim:], clean[:, vdim:])       # the other request, the other heads
    if where in ("v", "state"):
        assert torch.equal(got[:, 32:vdim], clean[:, 32:vdim])             # columns of other blocks


@pytest.mark.parametrize("rule,heads,group,segments,most", [("step", 64, 64, [80, 80], 1), ("step", 64, 64, [256], 2), ("step", 64, 64, [2048], 16), ("step", 128, 128, [700], 8),
                                                            ("decay", 16, 4, [700], 1), ("decay", 16, 4, [2048], 4), ("decay", 48, 3, [2048], 3), ("gla", 64, 64, [2048], 1),
                                                            ("delta", 64, 64, [2048], 1)])
def test_heads_a_block_of_the_preparation(rule, heads, group, segments, most):
    """As many of the heads that share q and k as leave each SM its blocks (148 SMs); q and k of a group are made once whatever it is."""
    from mini_llm_runtime_b200.ops import native
    c = make(rule, 128, 16, heads, group, segments)
    s = c["spec"]
    a_block = native.module("recurrence").mlr_linear_recurrence_chunk_heads(ctypes.addressof(s), sum(segments), len(segments))
    assert a_block == most and group % a_block == 0
    state, (want, want_state) = c["start"].clone(), exact(c)
    got, _, _ = launch(c, state)
    assert distance(got, want) < 5e-6
    assert distance(state[:, :heads * 16 * 128].reshape(want_state.shape), want_state) < 5e-6


def launch_portions(c, state, longest):
    """The outputs of the entry point that chooses the walk; room as a step's description asks for it, with a margin that must stay as it is."""
    from mini_llm_runtime_b200.ops import native
    s, proj, rows, n = c["spec"], c["proj"], c["proj"].shape[0], len(c["segments"])
    f32 = lambda *shape: torch.full(shape, float("nan"), device="cuda")
    out = torch.empty(rows, s.heads * s.vdim, device="cuda", dtype=torch.bfloat16)
    q, k, gates, obuf, df = f32(rows, s.qk_heads * s.dim), f32(rows, s.qk_heads * s.dim), f32(rows, 2 * s.heads), f32(rows, s.heads * s.vdim), f32(rows, s.heads * s.dim)
    pieces = native.module("recurrence").mlr_linear_recurrence_places(ctypes.addressof(s), rows)
    piece_ends = f32(pieces, s.heads * (s.vdim + 1) * s.dim) if pieces else None
    places = (rows + 15) // 16 + min(rows // 4, n)
    held = [f32(places + 1, s.heads * s.dim * 24), f32(places + 1, (s.heads if s.channel_decay else s.qk_heads) * s.dim * 24),
            f32(places + 1, (s.heads if s.channel_decay else s.qk_heads) * s.dim * 24), f32(rows + 1, s.heads * 16), f32(places + 1, s.heads * (s.dim if s.channel_decay else 36))]
    native.call("recurrence", "mlr_linear_recurrence_portions", ctypes.addressof(s), proj.data_ptr(), proj.stride(0), proj.data_ptr(), proj.stride(0),
                out.data_ptr(), out.stride(0), state.data_ptr(), state.stride(0), c["info"].data_ptr(), n, longest, c["positions"].data_ptr(), rows,
                q.data_ptr(), k.data_ptr(), gates.data_ptr(), obuf.data_ptr(), df.data_ptr(), None, 0, piece_ends.data_ptr() if pieces else None, places,
                *[t.data_ptr() for t in held], native.stream())
    torch.cuda.synchronize()
    assert all(torch.isnan(t[-1]).all() for t in held)
    return obuf


@pytest.mark.parametrize("rule,dim,vdim,heads,segments,chunks", [
    ("delta", 128, 128, 16, [1] * 128, False), ("delta", 128, 128, 16, [16] * 64, False), ("delta", 128, 128, 16, [100] + [1] * 28, False),
    ("delta", 128, 128, 16, [2000] + [1] * 40, True), ("delta", 128, 128, 16, [128], True), ("channel_delta", 128, 128, 16, [1] * 256, False),
    ("channel_delta", 128, 128, 16, [700], True), ("gla", 64, 64, 16, [8] * 32, False), ("gla", 128, 128, 16, [3, 900, 1], True), ("decay", 64, 64, 8, [2048], False),
    ("decay", 128, 128, 8, [2048], True), ("decay", 128, 128, 8, [1] * 130, False), ("step", 128, 64, 64, [16] * 40, False), ("step", 128, 64, 64, [600], True),
    ("step", 128, 64, 64, [1] * 128, False), ("step", 128, 64, 64, [127], False),
])
def test_the_walk_is_chosen_by_the_portions_of_a_step(rule, dim, vdim, heads, segments, chunks):
    """Short portions token by token, long ones in chunks (each pair of times beside the rule), in the same bits as the entry points of either walk."""
    from mini_llm_runtime_b200.ops import native
    c = make(rule, dim, vdim, heads, heads if rule == "step" else 1, segments)
    takes = native.module("recurrence").mlr_linear_recurrence_takes_chunks(ctypes.addressof(c["spec"]), len(segments), sum(segments), max(segments))
    assert bool(takes) == chunks
    state, alone = c["start"].clone(), c["start"].clone()
    got = launch_portions(c, state, max(segments))
    if chunks:
        want, _, _ = launch(c, alone)
        assert torch.equal(got, want) and torch.equal(state, alone)
    elif not native.module("recurrence").mlr_linear_recurrence_places(ctypes.addressof(c["spec"]), sum(segments)):
        want, _, _ = launch(c, alone, chunks=False)
        assert torch.equal(got, want) and torch.equal(state, alone)
    else:
        assert distance(got, exact(c)[0]) < 5e-6


@pytest.mark.parametrize("rule,dim,vdim,heads,group,segments", [
    ("decay", 128, 128, 2, 1, [2048]), ("gla", 128, 128, 2, 1, [2048]), ("delta", 128, 128, 2, 1, [2048]), ("channel_delta", 128, 128, 2, 1, [2048]),
    ("step", 128, 64, 2, 2, [1999]), ("delta", 64, 256, 2, 1, [130, 70]), ("channel_delta", 128, 256, 2, 2, [90, 33]), ("delta", 64, 64, 80, 1, [64] * 3),
    ("step", 64, 48, 3, 3, [5, 17, 1] * 100), ("channel_delta", 64, 16, 2, 1, [1, 2, 30] * 110), ("decay", 64, 32, 2, 1, [7] * 300),
])
def test_chunks_are_as_exact_as_the_walk_token_by_token_and_repeat_their_bits(rule, dim, vdim, heads, group, segments):
    """Long portions, columns past the first 128, more than 256 portions.  Both walks add in float32, in other orders, so their distances from 64 bits are
    of one size (1e-8 to 3e-7, chunks at most 1.3 times the other's where measured); limit: three times, and 2e-8 for sums of few terms.  A split
    into two bfloat16 parts instead of three is 16 bits of each operand: 2^-17 of a term, over 4e-6."""
    c = make(rule, dim, vdim, heads, group, segments)
    want, want_state = exact(c)
    size = heads * vdim * dim
    def run(chunks):
        state = c["start"].clone()
        got, _, _ = launch(c, state, chunks=chunks)
        return got, state[:, :size].reshape(want_state.shape)
    (got, state), (by_token, by_token_state) = run(True), run(False)
    assert distance(got, want) < 3 * distance(by_token, want) + 2e-8
    assert distance(state, want_state) < 3 * distance(by_token_state, want_state) + 2e-8
    for _ in range(3):
        again, state_again = run(True)
        assert torch.equal(again, got) and torch.equal(state_again, state)


@pytest.mark.parametrize("rule,rotated,made", [("decay", True, 0), ("gla", False, 1), ("channel_delta", False, 0), ("channel_delta", False, 1)])
def test_both_walks_give_the_same_read_out(rule, rotated, made):
    """Rotated q and k, low-rank decays and gates made by the kernel or beforehand, norm, weight and gate: the entry points differ in the walk alone, so
    their bfloat16 results differ by at most a rounding of values that differ by some 1e-7: one place of eight bits, for few of them."""
    from mini_llm_runtime_b200.ops import native
    dim = vdim = 64
    heads, rank, segments = 2, 16, [70, 100]
    c = make(rule, dim, vdim, heads, 1, segments)
    s, proj, rows = c["spec"], c["proj"], sum(segments)
    g = torch.Generator().manual_seed(5)
    side = torch.randn(rows, heads * vdim, generator=g).cuda().bfloat16()
    weight = (1 + 0.1 * torch.randn(vdim, generator=g)).cuda()
    freq = (100.0 ** (-torch.arange(16) / 16)).cuda()
    gate_w = (torch.randn(rank, heads * vdim, generator=g) * rank ** -0.5).cuda().bfloat16()
    if rotated:
        s.prep, s.rot_dims, s.freq = RecurrenceSpec.PREP["rotate"], 32, freq.data_ptr()
    s.out_weight, s.gate_kind = weight.data_ptr(), 1
    wide = torch.cat([proj, side], 1).contiguous()             # the gate's columns behind the projections
    s.col_gate = proj.shape[1]
    if s.channel_decay:
        s.gate_rank, s.gate_w = rank, gate_w.data_ptr()
    results = []
    for chunks in (True, False):
        f32 = lambda *shape: torch.full(shape, float("nan"), device="cuda")
        out = torch.empty(rows, heads * vdim, device="cuda", dtype=torch.bfloat16)
        state = c["start"].clone()
        q, k, gates, obuf, df, gf = f32(rows, heads * dim), f32(rows, heads * dim), f32(rows, 2 * heads), f32(rows, heads * vdim), f32(rows, heads * dim), f32(rows, heads * vdim)
        if made:
            df.copy_(wide[:, s.col_a:s.col_a + rank].float() @ c["held"]["decay_w"].float())
            gf.copy_(wide[:, s.col_gate:s.col_gate + rank].float() @ gate_w.float())
        common = [ctypes.addressof(s), wide.data_ptr(), wide.stride(0), wide.data_ptr(), wide.stride(0)]
        tail = [out.data_ptr(), out.stride(0), state.data_ptr(), state.stride(0), c["info"].data_ptr(), len(segments), c["positions"].data_ptr(), rows,
                q.data_ptr(), k.data_ptr(), gates.data_ptr(), obuf.data_ptr(), df.data_ptr(), gf.data_ptr(), made]
        places = (rows + 15) // 16 + len(segments)
        held = [f32(places, heads * dim * 24) for _ in range(3)] + [f32(rows, heads * 16), f32(places, heads * (dim if s.channel_decay else 36))]
        if chunks:
            native.call("recurrence", "mlr_linear_recurrence_chunks", *common, *tail, *[t.data_ptr() for t in held], native.stream())
        else:
            native.call("recurrence", "mlr_linear_recurrence_split", *common, 1, *tail, native.stream())
        torch.cuda.synchronize()
        results.append((out.float(), state))
    (got, state), (want, want_state) = results
    assert torch.isfinite(got).all() and float(want.square().mean()) > 0.05
    off = (got - want).abs() > 1e-6 * want.abs().max()
    assert float(off.float().mean()) < 1e-3 and bool(((got - want).abs() <= 2.0 ** -7 * want.abs() + 1e-6).all())
    assert distance(state, want_state.double()) < 1e-6
