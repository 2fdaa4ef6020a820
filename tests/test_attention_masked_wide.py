"""Masked attention of prompt portions on the tcgen05 kernel: masks, sinks, caps, biases, rotation, gates, values in their keys, sizes that
fill their 64-value pieces and sizes that do not, portions that end inside a tile, pages of several sizes.  Against 64 bits on the same
bfloat16 queries, keys and values; the cache holds NaN wherever nothing was written.

Tolerance: the weights enter as 16 bits and the sums are float32, so a result is good to 2^-15 of the values' size (3) before it is rounded to
bfloat16 (2^-9); queries that the kernel rotates are rounded to bfloat16 behind the rotation in the reference as well, where a last bit
may fall differently: a score of size 5 then moves by 2^-9 of a term of it, which moves a weight by at most a hundredth."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [
    # heads, kv heads, key, value, rotated, window, chunk, kept, sink, softcap, slopes, gate, shared, tokens, first portion, page
    (2, 1, 128, 128, 0, 0, 0, 0, None, 0.0, False, None, False, 300, 170, 16),
    (4, 2, 128, 128, 64, 100, 0, 0, None, 0.0, False, "sigmoid", False, 429, 128, 16),
    (2, 2, 64, 128, 32, 0, 96, 0, "zero", 0.0, False, "silu", False, 260, 131, 8),
    (2, 1, 128, 128, 0, 130, 0, 4, "learned", 30.0, False, None, False, 700, 300, 16),
    (3, 1, 128, 96, 0, 64, 0, 0, "learned", 0.0, False, "sigmoid_head", True, 333, 129, 16),
    (2, 1, 48, 40, 16, 0, 0, 0, None, 5.0, True, None, False, 200, 100, 32),
    (2, 1, 128, 64, 0, 0, 0, 0, None, 0.0, True, None, True, 257, 1, 64),
    (1, 1, 16, 8, 16, 33, 0, 70, None, 0.0, False, "sigmoid", False, 290, 140, 128),
    (2, 1, 64, 24, 0, 1, 0, 0, None, 0.0, False, None, True, 150, 130, 256),
    (1, 1, 80, 120, 0, 0, 64, 0, None, 0.0, False, None, False, 400, 300, 16),
]


@pytest.mark.parametrize("case", CASES, ids=str)
def test_against_64_bits(case):
    from mini_llm_runtime_b200.ops import native
    from mini_llm_runtime_b200.ops.specs import GATES, MaskedAttentionSpec
    H, G, D, V, rot, window, chunk, kept, sink, cap, sloped, gate, shared, T, split, page = case
    g = torch.Generator().manual_seed(T)
    draw = lambda *shape: torch.randn(*shape, generator=g).bfloat16().cuda()
    q, k, v = draw(T, H * D + 8), draw(T, G, D), draw(T, G, V)
    gates = draw(T, H * V) if gate not in (None, "sigmoid_head") else draw(T, H)
    freq = 100.0 ** (-2.0 * torch.arange(rot // 2) / max(rot, 1)).float().cuda()
    sinks, slopes = (torch.randn(H, generator=g) * 2).cuda(), (0.01 * (1 + torch.arange(H)).float()).cuda()
    scale = D ** -0.5 * 1.5
    spec = MaskedAttentionSpec(freq=freq.data_ptr() if rot else None, sinks=sinks.data_ptr() if sink == "learned" else None,
                               slopes=slopes.data_ptr() if sloped else None, heads=H, kv_heads=G, dim=D, vdim=V, rot_dims=rot, window=window, chunk=chunk,
                               sink=int(sink is not None), gate_kind=GATES[gate], shared_kv=int(shared), keep_first=kept, scale=scale, out_scale=0.75,
                               softcap=cap)
    assert native.module("attention_masked_tcgen05").mlr_attention_masked_wide_fit(ctypes.addressof(spec), page) == 1
    used = -(-T // page)
    order = torch.randperm(used + 3, generator=g)[:used]
    cache = torch.full((used + 3, G * page * (D + (0 if shared else V))), float("nan"), dtype=torch.bfloat16, device="cuda")
    for i, p in enumerate(order.tolist()):
        n = min(page, T - i * page)
        cache[p, :G * page * D].view(G, page, D)[:, :n] = k[i * page:i * page + n].transpose(0, 1)
        if not shared:
            cache[p, G * page * D:].view(G, page, V)[:, :n] = v[i * page:i * page + n].transpose(0, 1)
    table = order.to(torch.int32).cuda().view(1, -1).repeat(2, 1).contiguous()
    info = torch.tensor([[0, split, 0, 0], [split, T - split, split, 0]], dtype=torch.int32, device="cuda")
    tiles = torch.tensor([(0, t) for t in range(0, split, 128)] + [(1, t) for t in range(0, T - split, 128)], dtype=torch.int32, device="cuda")
    out, status = torch.full((T, H * V), float("nan"), dtype=torch.bfloat16, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    native.call("attention_masked_tcgen05", "mlr_attention_masked_wide", ctypes.addressof(spec), q.data_ptr(), q.stride(0),
                gates.data_ptr() if gate else None, gates.stride(0) if gate else 0, out.data_ptr(), out.stride(0), cache.data_ptr(), used + 3,
                tiles.data_ptr(), tiles.shape[0], info.data_ptr(), table.data_ptr(), table.stride(0), page, status.data_ptr(), native.stream())
    assert status.item() == 0

    pos = torch.arange(T, device="cuda")
    qd = q[:, :H * D].view(T, H, D).double()
    if rot:
        angle = (pos[:, None].float() * freq).double()
        a, b = qd[..., :rot // 2].clone(), qd[..., rot // 2:rot].clone()
        cs, sn = angle.cos()[:, None], angle.sin()[:, None]
        qd = torch.cat([a * cs - b * sn, b * cs + a * sn, qd[..., rot:]], -1).bfloat16().double()
    kd = k.double().repeat_interleave(H // G, 1)
    vd = (k[..., :V] if shared else v).double().repeat_interleave(H // G, 1)
    s = torch.einsum("ihd,jhd->hij", qd, kd) * scale
    if cap:
        s = cap * torch.tanh(s / cap)
    back = (pos[:, None] - pos[None]).double()
    if sloped:
        s = s - slopes.double()[:, None, None] * back
    lo = torch.zeros(T, dtype=torch.long, device="cuda")
    if window:
        lo = torch.maximum(lo, pos - window + 1)
    if chunk:
        lo = torch.maximum(lo, pos // chunk * chunk)
    seen = (pos[None] <= pos[:, None]) & ((pos[None] >= lo[:, None]) | (pos[None] < kept))
    s = s.masked_fill(~seen, -float("inf"))
    if sink is not None:
        extra = sinks.double() if sink == "learned" else torch.zeros(H, dtype=torch.float64, device="cuda")
        weights = torch.softmax(torch.cat([s, extra[:, None, None].expand(H, T, 1)], -1), -1)[..., :-1]
    else:
        weights = torch.softmax(s, -1)
    want = torch.einsum("hij,jhd->ihd", weights, vd) * 0.75
    if gate == "sigmoid_head":
        want = want * torch.sigmoid(gates.double())[..., None]
    elif gate:
        x = gates.double().view(T, H, V)
        want = want * (torch.sigmoid(x) * x if gate == "silu" else torch.sigmoid(x))
    got = out.double().view(T, H, V)
    assert torch.allclose(got, want, atol=3e-2 if rot else 6e-3, rtol=8e-3), float((got - want).abs().max())
    assert float((got - want).norm() / want.norm()) < 5e-3
