"""Row-wise kernels that keep a row in registers, at the edges of what they take: one to all of a thread's groups of columns, widths that
leave the last group partly empty, one group of columns and many.  Against the same in 64 bits.

Tolerances: sums of at most 16384 products of numbers of size 1 in 32 bits are good to about 1e-6 of their size; results of up to
20 such numbers stay within 1e-4.  bfloat16 rounds by at most 2^-9 of the value: 1e-2 covers it with the float32 error behind it."""
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = {torch.float32: dict(atol=1e-4, rtol=1e-4), torch.bfloat16: dict(atol=1e-2, rtol=1e-2)}


def _call(module, name, *args):
    from mini_llm_runtime_b200.ops import native
    native.call(module, name, *args)


def _draw(seed):
    g = torch.Generator().manual_seed(seed)
    return lambda *shape: torch.randn(*shape, generator=g).cuda()


def _grouped(x, groups, eps):
    parts = x.unflatten(-1, (groups, -1))
    return (parts / (parts.square().mean(-1, keepdim=True) + eps).sqrt()).flatten(-2)


def _near(got, want, dtype):
    assert torch.allclose(got.double(), want, **TOL[dtype]), float((got.double() - want).abs().max())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width", [64, 1020, 1024, 4096, 5120, 16384])
def test_rms_norm(dtype, width):
    from mini_llm_runtime_b200.ops import native
    draw, rows = _draw(width), 5
    h, weight = draw(rows, width), draw(width)
    out = torch.empty(rows, width, dtype=dtype, device="cuda")
    _call("elementwise", "mlr_rmsnorm", h.data_ptr(), None, 1, 0, weight.data_ptr(), 0, out.data_ptr(), native.is_bf16(out), None, rows, width, 1e-5, 0,
          native.stream())
    _near(out, _grouped(h.double(), 1, 1e-5) * weight.double(), dtype)
    # Many rows, which take fewer threads each, give the same bits.
    many, all_out = h.repeat(200, 1), torch.empty(200 * rows, width, dtype=dtype, device="cuda")
    _call("elementwise", "mlr_rmsnorm", many.data_ptr(), None, 1, 0, weight.data_ptr(), 0, all_out.data_ptr(), native.is_bf16(out), None, 200 * rows, width,
          1e-5, 0, native.stream())
    assert torch.equal(all_out, out.repeat(200, 1))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width,states", [(4, 1), (1024, 0), (2052, 3), (4096, 5), (4100, 2), (16384, 1)])
def test_depth_average_and_layer_norm(dtype, width, states):
    from mini_llm_runtime_b200.ops import native
    draw, rows = _draw(width + states), 3
    history, h, d1, d2 = draw(states + 2, rows, width), draw(rows, width), draw(rows, width + 4)[:, :width], draw(rows, width)
    bias, w, b, dwa = draw(width), draw(width), draw(width), draw(states + 1)
    old, before = h.double(), history.clone()
    out = torch.empty(rows, width, dtype=dtype, device="cuda")
    _call("layernorm", "mlr_depth_norm", h.data_ptr(), d1.data_ptr(), d1.stride(0), d2.data_ptr(), d2.stride(0), bias.data_ptr(), history.data_ptr(),
          history.stride(0), states, dwa.data_ptr(), w.data_ptr(), b.data_ptr(), 1e-5, out.data_ptr(), out.stride(0), native.is_bf16(out), None, rows,
          width, 1, native.stream())
    newest = old + d1.double() + d2.double() + bias.double()
    stream = (torch.cat([before[:states].double(), newest[None]]) * dwa.double()[:, None, None]).sum(0)
    centred = stream - stream.mean(-1, keepdim=True)
    want = centred / (centred.square().mean(-1, keepdim=True) + 1e-5).sqrt() * w.double() + b.double()
    _near(history[states], newest, torch.float32)
    assert torch.equal(history[:states], before[:states]) and torch.equal(history[states + 1:], before[states + 1:])
    _near(h, stream, torch.float32)
    _near(out, want, dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width,states,off,gap", [(16388, 1, 0, 0), (20480, 6, 0, 0), (2048, 3, 1, 0), (4100, 5, 2, 0), (1030, 2, 0, 0), (1024, 4, 0, 2), (1028, 5, 0, 0), (2048, 0, 0, 0)])
def test_depth_average_and_layer_norm_of_other_rows(dtype, width, states, off, gap):
    """Rows wider than a thread's registers take, results and norm weights `off` a border, results to add whose rows lie `gap` off one."""
    from mini_llm_runtime_b200.ops import native
    draw, rows = _draw(width + states), 3
    history, h, d1, w = draw(states + 2, rows, width), draw(rows, width), draw(rows, width + gap)[:, :width], draw(width + off)[off:]
    b, dwa = draw(width + off)[off:], draw(states + 1)
    old, before = h.double(), history.clone()
    out = torch.empty(rows, width + off, dtype=dtype, device="cuda")[:, off:]
    _call("layernorm", "mlr_depth_norm", h.data_ptr(), d1.data_ptr(), d1.stride(0), None, 0, None, history.data_ptr(), history.stride(0), states,
          dwa.data_ptr(), w.data_ptr(), b.data_ptr(), 1e-5, out.data_ptr(), out.stride(0), native.is_bf16(out), None, rows, width, 1, native.stream())
    newest = old + d1.double()
    stream = (torch.cat([before[:states].double(), newest[None]]) * dwa.double()[:, None, None]).sum(0)
    centred = stream - stream.mean(-1, keepdim=True)
    want = centred / (centred.square().mean(-1, keepdim=True) + 1e-5).sqrt() * w.double() + b.double()
    _near(history[states], newest, torch.float32)
    assert torch.equal(history[:states], before[:states]) and torch.equal(history[states + 1:], before[states + 1:])
    _near(h, stream, torch.float32)
    _near(out, want, dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width,groups", [(128, 1), (1024, 8), (1152, 3), (2048, 1), (2048, 4), (4096, 32), (5120, 4), (8192, 1)])
def test_grouped_norms_around_a_sub_layer(dtype, width, groups):
    """The result normed and added into the stream, the sum normed, and a result in pieces."""
    from mini_llm_runtime_b200.ops import native
    draw, rows, top = _draw(width + groups), 3, 3
    h, delta, bias, w_post, w_pre = draw(rows, width), draw(rows, width), draw(width), draw(width), draw(width)
    old = h.double()
    out = torch.empty(rows, width, dtype=dtype, device="cuda")
    ends = (rows, width, groups, 1e-5)
    _call("norm_grouped", "mlr_group_rmsnorm", h.data_ptr(), delta.data_ptr(), width, bias.data_ptr(), w_post.data_ptr(), w_pre.data_ptr(), out.data_ptr(),
          width, native.is_bf16(out), None, *ends, 1, native.stream())
    stream = old + _grouped((delta + bias).double(), groups, 1e-5) * w_post.double()
    _near(h, stream, torch.float32)
    _near(out, _grouped(stream, groups, 1e-5) * w_pre.double(), dtype)

    old = h.double()
    _call("norm_grouped", "mlr_group_rmsnorm_sum", h.data_ptr(), 1.5, delta.data_ptr(), width, None, w_post.data_ptr(), None, out.data_ptr(), width,
          native.is_bf16(out), *ends, 1, native.stream())
    stream = _grouped(1.5 * old + delta.double(), groups, 1e-5) * w_post.double()
    _near(h, stream, torch.float32)
    assert torch.equal(out, h.to(dtype))

    y, weights, shared, gate = draw(rows * top, width), draw(rows, top), draw(rows, width), draw(rows)
    place = torch.randperm(rows * top, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(rows, top).cuda()
    place[0, 1] = -1
    old = h.double()
    _call("norm_grouped", "mlr_group_rmsnorm_pieces", h.data_ptr(), y.data_ptr(), width, place.data_ptr(), weights.data_ptr(), top, shared.data_ptr(), width,
          gate.data_ptr(), None, 0, 0, None, w_post.data_ptr(), w_pre.data_ptr(), out.data_ptr(), width, native.is_bf16(out), *ends, 1, native.stream())
    taken = weights.double() * (place >= 0)
    total = (taken[:, :, None] * y.double()[place.clamp(min=0).long()]).sum(1) + gate.double()[:, None] * shared.double()
    stream = old + _grouped(total, groups, 1e-5) * w_post.double()
    _near(h, stream, torch.float32)
    _near(out, _grouped(stream, groups, 1e-5) * w_pre.double(), dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("streams,width", [(1, 1024), (1, 4096), (2, 2052), (3, 4096), (4, 1028), (4, 2048), (4, 4096)])
def test_copies_of_the_stream(dtype, streams, width):
    from mini_llm_runtime_b200.ops import native
    draw, rows = _draw(streams + width), 3
    h, y, scale, norm_w = draw(rows, streams * width), draw(rows, width), draw(width), draw(width)
    mix, w_out, w_in = draw(streams, streams), draw(streams), draw(streams)
    old = h.double().view(rows, streams, width)
    out = torch.empty(rows, width, dtype=dtype, device="cuda")
    _call("streams", "mlr_streams_step", h.data_ptr(), y.data_ptr(), width, scale.data_ptr(), mix.data_ptr(), w_out.data_ptr(), w_in.data_ptr(),
          norm_w.data_ptr(), 1e-5, out.data_ptr(), width, native.is_bf16(out), None, rows, width, streams, native.stream())
    new = torch.einsum("rsw,st->rtw", old, mix.double()) + w_out.double()[None, :, None] * (y.double() * scale.double())[:, None]
    _near(h.view(rows, streams, width), new, torch.float32)
    read = (new * w_in.double()[None, :, None]).sum(1)
    _near(out, _grouped(read, 1, 1e-5) * norm_w.double(), dtype)


def _pieces(draw, rows, top, width, x_dtype):
    """What routed experts leave of a token: pieces (one of them an identity expert's, without a row), a gated shared result, the token
    itself for its identity experts.  The kernels' arguments and the sum in 64 bits."""
    y, weights, shared, gate, passed = draw(rows * top, width), draw(rows, top), draw(rows, width), draw(rows), draw(rows)
    x = draw(rows, width).to(x_dtype)
    place = torch.randperm(rows * top, generator=torch.Generator().manual_seed(2)).to(torch.int32).view(rows, top).cuda()
    place[0, 1] = place[2, 0] = -1
    total = ((weights.double() * (place >= 0))[:, :, None] * y.double()[place.clamp(min=0).long()]).sum(1)
    total = total + gate.double()[:, None] * shared.double() + passed.double()[:, None] * x.double()
    args = (y.data_ptr(), width, place.data_ptr(), weights.data_ptr(), top, shared.data_ptr(), width, gate.data_ptr(), x.data_ptr(), width,
            int(x_dtype is torch.bfloat16), passed.data_ptr())
    return args, total, (y, weights, shared, gate, passed, x, place)


@pytest.mark.parametrize("x_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width,groups", [(1024, 1), (2048, 2), (3200, 5), (4096, 32), (8192, 8), (1000, 4)])
def test_grouped_norm_of_pieces_with_identity_experts(x_dtype, width, groups):
    from mini_llm_runtime_b200.ops import native
    draw, rows, top = _draw(width + groups), 3, 5
    h, w_post, w_pre = draw(rows, width), draw(width), draw(width)
    args, total, held = _pieces(draw, rows, top, width, x_dtype)
    out, old = torch.empty(rows, width, device="cuda"), h.double()
    _call("norm_grouped", "mlr_group_rmsnorm_pieces", h.data_ptr(), *args, w_post.data_ptr(), w_pre.data_ptr(), out.data_ptr(), width, 0, rows, width,
          groups, 1e-5, 1, native.stream())
    stream = old + _grouped(total, groups, 1e-5) * w_post.double()
    _near(h, stream, torch.float32)
    _near(out, _grouped(stream, groups, 1e-5) * w_pre.double(), torch.float32)


@pytest.mark.parametrize("x_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("streams,width,reads", [(1, 4096, True), (2, 1028, True), (4, 2048, False), (4, 4096, True), (3, 4096, False), (2, 8192, True)])
def test_copies_of_the_stream_take_pieces(x_dtype, streams, width, reads):
    """With and without a norm behind the sub-layer."""
    from mini_llm_runtime_b200.ops import native
    draw, rows, top = _draw(streams + width + reads), 3, 5
    h, scale, norm_w = draw(rows, streams * width), draw(width), draw(width)
    mix, w_out, w_in = draw(streams, streams), draw(streams), draw(streams)
    args, total, held = _pieces(draw, rows, top, width, x_dtype)
    out, old = torch.empty(rows, width, device="cuda"), h.double().view(rows, streams, width)
    _call("streams", "mlr_streams_step_pieces", h.data_ptr(), *args, scale.data_ptr(), mix.data_ptr(), w_out.data_ptr(), w_in.data_ptr(), norm_w.data_ptr(),
          1e-5, out.data_ptr() if reads else None, width, 0, rows, width, streams, native.stream())
    new = torch.einsum("rsw,st->rtw", old, mix.double()) + w_out.double()[None, :, None] * (total * scale.double())[:, None]
    _near(h.view(rows, streams, width), new, torch.float32)
    if reads:
        _near(out, _grouped((new * w_in.double()[None, :, None]).sum(1), 1, 1e-5) * norm_w.double(), torch.float32)


@pytest.mark.parametrize("streams,width", [(1, 1024), (4, 2048), (4, 4096)])
def test_copies_of_the_stream_of_wanted_rows(streams, width):
    """A launch over some rows norms what it reads of them and writes nothing back."""
    from mini_llm_runtime_b200.ops import native
    draw = _draw(streams + width)
    h, w_in, norm_w = draw(6, streams * width), draw(streams), draw(width)
    rows = torch.tensor([4, 0, 5], dtype=torch.int32, device="cuda")
    out, before = torch.empty(3, width, device="cuda"), h.clone()
    _call("streams", "mlr_streams_step", h.data_ptr(), None, 0, None, None, None, w_in.data_ptr(), norm_w.data_ptr(), 1e-5, out.data_ptr(), width, 0,
          rows.data_ptr(), 3, width, streams, native.stream())
    read = (h.double().view(6, streams, width)[rows.long()] * w_in.double()[None, :, None]).sum(1)
    _near(out, _grouped(read, 1, 1e-5) * norm_w.double(), torch.float32)
    assert torch.equal(h, before)
