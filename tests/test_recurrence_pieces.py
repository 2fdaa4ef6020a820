"""Walks of a matrix state in pieces that run side by side, against the one-kernel form (which its own tests hold to 64 bits): portions that
end inside a piece, portions too short for a second piece beside long ones, head sizes on both sides of the lanes' split, all decays.

Tolerance: both sum in float32; states of a few hundred terms of size 1 differ by a few 1e-6 of their size, normed outputs likewise."""
import ctypes

import pytest
import torch

from mini_llm_runtime_b200.ops.specs import RecurrenceSpec

pytestmark = pytest.mark.gpu


def _call(name, *args):
    from mini_llm_runtime_b200.ops import native
    native.call("recurrence", name, *args)


def _stream():
    from mini_llm_runtime_b200.ops import native
    return native.stream()


@pytest.mark.parametrize("rule,channel,dim,vdim,heads,segments", [
    ("decay", None, 128, 32, 2, [1000]), ("decay", None, 32, 40, 3, [1500, 31, 1300]), ("decay", None, 256, 16, 1, [2049]),
    ("decay", "sigmoid_root", 128, 17, 2, [897, 1100]), ("decay", "sigmoid_root", 64, 16, 2, [771]),
    ("step", None, 64, 24, 4, [1283]), ("step", None, 128, 64, 40, [900]), ("step", None, 128, 16, 2, [769, 1, 2000]),
])
def test_pieces_give_what_the_whole_walk_gives(rule, channel, dim, vdim, heads, segments):
    from mini_llm_runtime_b200.ops import native
    from mini_llm_runtime_b200.ops.specs import RecurrenceSpec
    g = torch.Generator().manual_seed(dim + vdim + len(segments))
    draw = lambda *shape: torch.randn(*shape, generator=g).cuda()
    rank, rows = 8, sum(segments)
    cq, ck, cv, ca = 0, heads * dim, 2 * heads * dim, 2 * heads * dim + heads * vdim
    proj = draw(rows, ca + max(rank, heads) + 8)
    decay, a_log, skip = (0.9 + 0.099 * torch.rand(heads, generator=g)).cuda(), draw(heads), draw(heads)
    dt_bias = draw(heads * dim) if channel else draw(heads)
    decay_w = draw(rank, heads * dim) * rank ** -0.5
    spec = RecurrenceSpec(decay=decay.data_ptr(), a_log=a_log.data_ptr(), dt_bias=dt_bias.data_ptr(), skip=skip.data_ptr() if rule == "step" else None,
                          decay_w=decay_w.data_ptr() if channel else None, decay_rank=rank if channel else 0,
                          channel_decay=RecurrenceSpec.CHANNEL_DECAY[channel] if channel else 0, heads=heads, qk_heads=heads, dim=dim, vdim=vdim,
                          rule=RecurrenceSpec.RULE[rule], gate_first=int(rule == "step"), norm_parts=heads, col_q=cq, col_k=ck, col_v=cv, col_a=ca,
                          q_mult=dim ** -0.5, k_mult=dim ** -0.5, unit_eps=1e-6, eps=1e-5, out_scale=1.0, inv_tau=1 / 16)
    info, first = [], 0
    for i, n in enumerate(segments):
        info.append((first, n, 0, len(segments) - 1 - i))
        first += n
    info = torch.tensor(info, dtype=torch.int32, device="cuda")
    positions = torch.cat([torch.arange(n) for n in segments]).to(torch.int32).cuda()
    start = draw(len(segments), heads * vdim * dim + 3)
    results = []
    for pieces in (False, True):
        state, out, obuf = start.clone(), torch.full((rows, heads * vdim), float("nan"), device="cuda"), torch.empty(rows, heads * vdim, device="cuda")
        common = (ctypes.addressof(spec), proj.data_ptr(), proj.stride(0), proj.data_ptr(), proj.stride(0), 0, out.data_ptr(), out.stride(0),
                  state.data_ptr(), state.stride(0), info.data_ptr(), len(segments))
        if pieces:
            q, k, gates = (torch.empty(rows, w, device="cuda") for w in (heads * dim, heads * dim, 2 * heads))
            df = torch.empty(rows, heads * dim, device="cuda") if channel else None
            ends = torch.full((rows // 128, heads * (vdim + 1) * dim), float("nan"), device="cuda")
            _call("mlr_linear_recurrence_pieces", *common, positions.data_ptr(), rows, q.data_ptr(), k.data_ptr(), gates.data_ptr(), obuf.data_ptr(),
                  df.data_ptr() if channel else None, None, 0, ends.data_ptr(), native.stream())
            assert torch.isfinite(ends).any()              # the pieces' room was used
        else:
            _call("mlr_linear_recurrence", *common, rows, obuf.data_ptr() if rule == "step" else None, None, native.stream())
        results.append((out, state))
    (want, want_state), (got, got_state) = results
    scale = float(want_state.abs().max())
    assert torch.allclose(got_state, want_state, atol=1e-5 * scale, rtol=1e-5)
    assert torch.allclose(got, want, atol=2e-4, rtol=2e-4), float((got - want).abs().max())
    assert torch.equal(got_state[:, heads * vdim * dim:], start[:, heads * vdim * dim:])


def test_the_second_pass_leaves_the_ends_alone():
    """A block of a later piece puts the state before it together from the ends that the first pass left.  It may start after blocks of
    earlier pieces have ended (their number is not bound by what the SMs hold at once), so those must not write ends of their own."""
    g = torch.Generator().manual_seed(7)
    heads, dim, vdim, rows, most, length = 2, 128, 32, 1000, 7, 144          # 7 pieces of 144 tokens, the last shorter
    proj = torch.randn(rows, 2 * heads * dim + heads * vdim, generator=g).cuda()
    decay = torch.tensor([0.99, 0.999], device="cuda")
    spec = RecurrenceSpec(decay=decay.data_ptr(), heads=heads, qk_heads=heads, dim=dim, vdim=vdim, rule=RecurrenceSpec.RULE["decay"], norm_parts=heads,
                          col_k=heads * dim, col_v=2 * heads * dim, q_mult=dim ** -0.5, k_mult=dim ** -0.5, unit_eps=1e-6, eps=1e-5, out_scale=1.0)
    out, obuf = torch.empty(rows, heads * vdim, device="cuda"), torch.empty(rows, heads * vdim, device="cuda")
    q, k = (torch.empty(rows, heads * dim, device="cuda") for _ in range(2))
    ends = torch.full((rows // 128, heads, vdim + 1, dim), float("nan"), device="cuda")
    state = torch.randn(1, heads * vdim * dim, generator=g).cuda()
    positions = torch.arange(rows, dtype=torch.int32, device="cuda")
    info = torch.tensor([[0, rows, 0, 0]], dtype=torch.int32, device="cuda")
    common = (ctypes.addressof(spec), proj.data_ptr(), proj.stride(0), proj.data_ptr(), proj.stride(0), 0, out.data_ptr(), out.stride(0))
    _call("mlr_linear_recurrence_pieces", *common, state.data_ptr(), state.stride(0), info.data_ptr(), 1, positions.data_ptr(), rows, q.data_ptr(),
          k.data_ptr(), None, obuf.data_ptr(), None, None, 0, ends.data_ptr(), _stream())
    for piece in range(1, most - 1):
        alone = torch.zeros(1, heads * vdim * dim, device="cuda")            # the piece from a state of zero
        info = torch.tensor([[piece * length, length, piece * length, 0]], dtype=torch.int32, device="cuda")
        _call("mlr_linear_recurrence", *common, alone.data_ptr(), alone.stride(0), info.data_ptr(), 1, rows, None, None, _stream())
        want = alone.view(heads, vdim, dim)
        off = (ends[:, :, :vdim] - want).abs().amax((1, 2, 3))               # of every place of `ends`
        place = int(off.nan_to_num(float("inf")).argmin())
        assert float(off[place]) <= 1e-5 * float(want.abs().max())
        assert torch.allclose(ends[place, :, vdim], (decay ** length)[:, None].expand(heads, dim), rtol=1e-4)


@pytest.mark.parametrize("rule,dim,vdim,heads,segments,pieces", [("decay", 128, 128, 8, [2048], 16), ("decay", 128, 128, 4, [900, 1400], 8), ("step", 128, 64, 40, [900], 7),
                                                                 ("decay", 64, 16, 2, [800] * 9, 6), ("step", 128, 64, 128, [8192], 1),
                                                                 ("decay", 128, 128, 8, [767], 1), ("decay", 48, 16, 1, [2048], 1), ("delta", 128, 128, 2, [2048], 1)])
def test_room_for_the_ends_is_what_the_walk_uses(rule, dim, vdim, heads, segments, pieces):
    """Room is asked for where a step of these rows can be walked in pieces, bounded by the pieces that are launched, not by the rows."""
    from mini_llm_runtime_b200.ops import native
    g, rows, value = torch.Generator().manual_seed(dim + heads), sum(segments), heads * (vdim + 1) * dim
    draw = lambda *shape: torch.randn(*shape, generator=g).cuda()
    ca = 2 * heads * dim + heads * vdim
    decay, a_log, dt_bias = torch.full((heads,), 0.99, device="cuda"), draw(heads), draw(heads)
    spec = RecurrenceSpec(decay=decay.data_ptr(), a_log=a_log.data_ptr(), dt_bias=dt_bias.data_ptr(), skip=dt_bias.data_ptr(), heads=heads, qk_heads=heads,
                          dim=dim, vdim=vdim, rule=RecurrenceSpec.RULE[rule], gate_first=int(rule == "step"), norm_parts=heads, col_k=heads * dim,
                          col_v=2 * heads * dim, col_a=ca, col_b=ca + heads, q_mult=dim ** -0.5, k_mult=dim ** -0.5, unit_eps=1e-6, eps=1e-5, out_scale=1.0)
    places = native.module("recurrence").mlr_linear_recurrence_places(ctypes.addressof(spec), rows)
    if pieces == 1:
        assert places == 0
        return
    assert len(segments) * pieces <= places <= 8 * 148
    proj, ends = draw(rows, ca + 2 * heads), torch.full((places + 1, value), float("nan"), device="cuda")
    first, info = 0, []
    for i, n in enumerate(segments):
        info.append((first, n, 0, i))
        first += n
    info = torch.tensor(info, dtype=torch.int32, device="cuda")
    state, out, obuf = torch.zeros(len(segments), heads * vdim * dim, device="cuda"), torch.empty(rows, heads * vdim, device="cuda"), torch.empty(rows, heads * vdim, device="cuda")
    q, k, gates, positions = draw(rows, heads * dim), draw(rows, heads * dim), draw(rows, 2 * heads), torch.zeros(rows, dtype=torch.int32, device="cuda")
    _call("mlr_linear_recurrence_pieces", ctypes.addressof(spec), proj.data_ptr(), proj.stride(0), proj.data_ptr(), proj.stride(0), 0, out.data_ptr(),
          out.stride(0), state.data_ptr(), state.stride(0), info.data_ptr(), len(segments), positions.data_ptr(), rows, q.data_ptr(), k.data_ptr(),
          gates.data_ptr(), obuf.data_ptr(), None, None, 0, ends.data_ptr(), _stream())
    used = torch.isfinite(ends).any(1).nonzero().flatten().tolist()
    assert used and max(used) < len(segments) * pieces
