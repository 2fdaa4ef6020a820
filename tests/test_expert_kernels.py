"""Products of routed experts: the pass over the weights of a step's few rows.  Against 64 bits.

Tolerances: operands are bfloat16 and taken as they are, sums are float32: 1e-4 of the results' size (about 1) covers 4096 terms; a
bfloat16 result is rounded by at most 2^-9 of its value."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _call(module, name, *args):
    from mini_llm_runtime_b200.ops import native
    native.call(module, name, *args)


def _stream():
    from mini_llm_runtime_b200.ops import native
    return native.stream()


def _listed(choices, experts, tile_rows):
    """choices [rows, top] (an expert past the last: none).  Tiles, their number, the pairs in the order by expert."""
    tiles, order = [], []
    for e in range(experts):
        pairs = (choices.flatten() == e).nonzero().flatten().tolist()
        for r in range(0, len(pairs), tile_rows):
            tiles.append((e, len(order) + r, min(tile_rows, len(pairs) - r)))
        order += pairs
    on = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    return on(tiles), on([len(tiles)]), order


def _gate(g, u, kind, alpha, limit, offset):
    if kind == 2:
        g, u = (g.clamp(max=limit), u.clamp(-limit, limit)) if limit > 0 else (g, u)
        return g * torch.sigmoid(alpha * g) * (u + offset)
    return g * torch.sigmoid(g) * u


@pytest.mark.parametrize("rows,experts,top,N,K,kind", [(1, 1, 1, 8, 8, 1), (1, 16, 4, 1024, 2048, 1), (3, 5, 3, 36, 520, 2), (8, 16, 8, 512, 4096, 2),
                                                       (8, 2, 1, 300, 1032, 1), (2, 300, 32, 24, 2056, 1)])
def test_few_rows(rows, experts, top, N, K, kind):
    from mini_llm_runtime_b200.ops import native
    g = torch.Generator().manual_seed(rows + N + K)
    draw = lambda *shape, scale=1.0: (torch.randn(*shape, generator=g) * scale).bfloat16().cuda()
    x, w, w2 = draw(rows, K + 8)[:, :K], draw(experts, N, K, scale=K ** -0.5), draw(experts, N, K, scale=K ** -0.5)
    choices = torch.stack([torch.randperm(experts + (top < experts), generator=g)[:top] for _ in range(rows)])
    choices[0, 0] = 0
    choices[0, 1:][choices[0, 1:] == 0] = experts
    tiles, n_tiles, order = _listed(choices, experts, 32)
    source = torch.tensor(order, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    shape = (1.702, 0.7, 1.0) if kind == 2 else (0.0, 0.0, 0.0)
    assert native.module("experts").mlr_experts_few(K, x.stride(0)) == 1
    act = torch.full((rows * top, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    _call("experts", "mlr_experts_product_few", x.data_ptr(), x.stride(0), source.data_ptr(), top, w.data_ptr(), w2.data_ptr(), kind, N, K, act.data_ptr(),
          N, tiles.data_ptr(), n_tiles.data_ptr(), rows, top, *shape, status.data_ptr(), native.stream())
    gathered = x[source.long() // top]
    plain = torch.full((rows * top, N), float("nan"), device="cuda")
    rows_in_order = torch.zeros(rows * top, K, dtype=torch.bfloat16, device="cuda")
    rows_in_order[:len(order)] = gathered
    _call("experts", "mlr_experts_product_few", rows_in_order.data_ptr(), K, None, 1, w.data_ptr(), None, 0, N, K, plain.data_ptr(), N, tiles.data_ptr(),
          n_tiles.data_ptr(), rows, top, 0.0, 0.0, 0.0, status.data_ptr(), native.stream())
    for e, first, count in tiles.tolist():
        a = gathered[first:first + count].double()
        y, up = a @ w[e].double().T, a @ w2[e].double().T
        assert torch.allclose(plain[first:first + count].double(), y, atol=1e-4, rtol=1e-4)
        assert torch.allclose(act[first:first + count].double(), _gate(y, up, kind, *shape), atol=1e-3, rtol=4e-3)
    assert torch.isnan(plain[len(order):]).all() and torch.isnan(act[len(order):].float()).all() and status.item() == 0


@pytest.mark.parametrize("experts,top,lost", [(16, 4, [3]), (16, 16, [0]), (9, 5, [0, 2, 4, 6, 7]), (40, 32, [1, 2, 5])])
def test_few_rows_beside_one_without_scores(experts, top, lost):
    """A token that is all NaN has no best expert and takes the first one `top` times, which then has more rows than the step.  The other
    tokens get the bits that they get beside ordinary tokens, and its own rows are NaN and not what the buffers held before."""
    rows, N, K = 8, 72, 520
    g = torch.Generator().manual_seed(experts + top)
    draw = lambda *shape, scale=1.0: (torch.randn(*shape, generator=g) * scale).bfloat16().cuda()
    plain, w, w2, down = draw(rows, K), draw(experts, N, K, scale=K ** -0.5), draw(experts, N, K, scale=K ** -0.5), draw(experts, K, N, scale=N ** -0.5)
    router, counts = torch.randn(experts, K, generator=g).cuda(), torch.zeros(experts, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    broken = plain.clone()
    broken[lost] = float("nan")
    results = []
    for x in (plain, broken):
        on = lambda n, dtype=torch.int32: torch.full((n,), -1, dtype=dtype, device="cuda")
        chosen, place, row_of_pair, pair_of_row = (on(rows * top) for _ in range(4))
        weights, first_row, tiles, n_tiles = on(rows * top, torch.float32), on(experts + 1), on(3 * (rows * top // 32 + experts)), on(1)
        _call("experts", "mlr_experts_route", x.data_ptr(), K, 1, router.data_ptr(), None, rows, K, experts, experts, 1, 1, top, 0, chosen.data_ptr(),
              weights.data_ptr(), place.data_ptr(), counts.data_ptr(), None, None, 0, _stream())
        _call("experts", "mlr_experts_arrange", counts.data_ptr(), chosen.data_ptr(), place.data_ptr(), experts, rows, top, 32, first_row.data_ptr(),
              tiles.data_ptr(), n_tiles.data_ptr(), row_of_pair.data_ptr(), pair_of_row.data_ptr(), _stream())
        act, y = torch.full((rows * top, N), 7.0, dtype=torch.bfloat16, device="cuda"), torch.full((rows * top, K), 7.0, device="cuda")
        _call("experts", "mlr_experts_product_few", x.data_ptr(), K, pair_of_row.data_ptr(), top, w.data_ptr(), w2.data_ptr(), 1, N, K, act.data_ptr(), N,
              tiles.data_ptr(), n_tiles.data_ptr(), rows, top, 0.0, 0.0, 0.0, status.data_ptr(), _stream())
        _call("experts", "mlr_experts_product_few", act.data_ptr(), N, None, 1, down.data_ptr(), None, 0, K, N, y.data_ptr(), K, tiles.data_ptr(),
              n_tiles.data_ptr(), rows, top, 0.0, 0.0, 0.0, status.data_ptr(), _stream())
        results.append(y[row_of_pair.long()].view(rows, top, K))
        most = int(tiles.view(-1, 3)[:n_tiles.item(), 2].max())
    sound = [r for r in range(rows) if r not in lost]
    assert most > (8 if len(lost) * top > 8 else 1) and status.item() == 0
    assert torch.equal(results[1][sound], results[0][sound])
    assert torch.isnan(results[1][lost]).all()


@pytest.mark.parametrize("rows,experts,top,N,K,kind", [(1, 1, 1, 128, 64, 1), (300, 1, 1, 256, 128, 2), (257, 3, 2, 136, 72, 1), (700, 16, 4, 264, 520, 2),
                                                       (64, 9, 3, 40, 8, 1)])
def test_many_rows_on_two_sms(rows, experts, top, N, K, kind):
    """Tiles that end inside an expert, experts without rows, widths that are no multiple of a tile, rows past the last."""
    from mini_llm_runtime_b200.ops import native
    g = torch.Generator().manual_seed(rows + N + K)
    draw = lambda *shape, scale=1.0: (torch.randn(*shape, generator=g) * scale).bfloat16().cuda()
    x, w, w2, down = draw(rows, K + 8)[:, :K], draw(experts, N, K, scale=K ** -0.5), draw(experts, N, K, scale=K ** -0.5), draw(experts, K, N, scale=N ** -0.5)
    choices = torch.stack([torch.randperm(experts + (top < experts), generator=g)[:top] for _ in range(rows)])
    if experts > 2:
        choices[choices == 1] = experts              # an expert nobody chose
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    shape = (1.702, 0.7, 1.0) if kind == 2 else (0.0, 0.0, 0.0)
    tiles, n_tiles, order = _listed(choices, experts, 256)
    count = len(order)
    source = torch.tensor(order + [0] * (rows * top - count), dtype=torch.int32, device="cuda")
    first_row = torch.tensor([(choices < e).sum().item() for e in range(experts)] + [count], dtype=torch.int32, device="cuda")
    side = torch.full((rows * top, K), float("nan"), dtype=torch.bfloat16, device="cuda")
    _call("experts", "mlr_experts_gather", x.data_ptr(), x.stride(0), source.data_ptr(), rows, top, first_row.data_ptr(), experts, side.data_ptr(), K,
          native.stream())
    gathered = x[source[:count].long() // top]
    assert torch.equal(side[:count], gathered) and torch.isnan(side[count:].float()).all()
    act = torch.full((rows * top, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    _call("gemm_bf16_tcgen05_pair", "mlr_grouped_product_bf16", side.data_ptr(), K, rows, top, w.data_ptr(), w2.data_ptr(), experts, kind, N, K,
          act.data_ptr(), N, tiles.data_ptr(), n_tiles.data_ptr(), *shape, status.data_ptr(), native.stream())
    y = torch.full((rows * top, K), float("nan"), device="cuda")
    _call("gemm_bf16_tcgen05_pair", "mlr_grouped_product_bf16", act.data_ptr(), N, rows, top, down.data_ptr(), None, experts, 0, K, N, y.data_ptr(), K,
          tiles.data_ptr(), n_tiles.data_ptr(), 0.0, 0.0, 0.0, status.data_ptr(), native.stream())
    for e, first, n in tiles.tolist():
        a = gathered[first:first + n].double()
        want = _gate(a @ w[e].double().T, a @ w2[e].double().T, kind, *shape)
        assert torch.allclose(act[first:first + n].double(), want, atol=1e-3, rtol=4e-3)
        assert torch.allclose(y[first:first + n].double(), act[first:first + n].double() @ down[e].double().T, atol=1e-4, rtol=1e-4)
    assert torch.isnan(act[count:].float()).all() and torch.isnan(y[count:]).all() and status.item() == 0


@pytest.mark.parametrize("offset", [1, 3])
def test_the_part_takes_rows_off_16_byte_borders(offset):
    """A caller's activations may be a view that starts anywhere: the first product then leaves the kernel that copies 16 bytes at a time.
    Sums in another order ahead of two roundings to bfloat16 (2^-9 each): a hundredth of the results' size."""
    from mini_llm_runtime_b200.config.base import PartSpec
    from mini_llm_runtime_b200.csrc import build
    from mini_llm_runtime_b200.engine.runtime import Runtime
    from mini_llm_runtime_b200.parts.base import StepContext
    from mini_llm_runtime_b200.parts.experts import RoutedExperts
    rows, width, inter, experts, top = 4, 64, 48, 6, 2
    g = torch.Generator().manual_seed(offset)
    names, tensors = {"router": "r", "correction": "c"}, {"r": torch.randn(experts, width, generator=g), "c": torch.zeros(experts)}
    for e in range(experts):
        for role, shape in (("gate", (inter, width)), ("up", (inter, width)), ("down", (width, inter))):
            names[f"e{e}.{role}"] = f"e{e}.{role}"
            tensors[f"e{e}.{role}"] = torch.randn(*shape, generator=g) * shape[1] ** -0.5
    rt = Runtime(torch.bfloat16)
    part = RoutedExperts(PartSpec("routed_experts", {"hidden_size": width, "intermediate_size": inter, "experts": experts, "top": top}, names))
    build.ensure(part.kernel_modules(rt.dtype) + ["host"])
    part.bind({k: v.bfloat16() for k, v in tensors.items()}, rt)
    step = StepContext(rt=rt, num_rows=rows, segments=[], token_ids=None, positions=None, segment_of_row=None, segment_info=None, slots=None, tables={},
                       page_size=16, status=torch.zeros(1, dtype=torch.int32, device="cuda"))
    x = torch.randn(rows, width + 8, generator=g).bfloat16().cuda()[:, offset:offset + width]
    got, want = part.forward(x, step), part.forward(x.contiguous(), step)
    assert torch.allclose(got, want, atol=1e-2 * float(want.abs().max()), rtol=0)


def test_few_rows_of_two_widths_from_two_threads():
    """The shared memory a launch asks for depends on its K; a thread's smaller launch must not take the limit away under another's larger one."""
    import threading
    rows, N = 4, 32
    status, tiles, n_tiles = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.tensor([0, 0, rows], dtype=torch.int32, device="cuda"), torch.ones(1, dtype=torch.int32, device="cuda")
    errors, results = [], {}

    def launch(K):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                g = torch.Generator().manual_seed(K)
                x, w = (torch.randn(n, K, generator=g).bfloat16().cuda() for n in (rows, N))
                out = torch.empty(rows, N, device="cuda")
                for _ in range(300):
                    _call("experts", "mlr_experts_product_few", x.data_ptr(), K, None, 1, w.data_ptr(), None, 0, N, K, out.data_ptr(), N, tiles.data_ptr(),
                          n_tiles.data_ptr(), rows, 1, 0.0, 0.0, 0.0, status.data_ptr(), _stream())
                torch.cuda.current_stream().synchronize()
                results[K] = (out.double(), x.double() @ w.double().T)
        except Exception as e:
            errors.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=launch, args=(K,)) for K in (512, 4096)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and status.item() == 0
    for got, want in results.values():
        assert torch.allclose(got, want, atol=1e-3, rtol=1e-4)         # sums of up to 4096 products of size 1
