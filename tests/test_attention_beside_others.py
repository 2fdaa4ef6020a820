"""Plain attention of a short prompt portion alone and beside a long one: the step's longest portion decides between the 64-row kernel and the
tcgen05 kernel for all of them, so a portion's rows may differ by the order of their sums.

Tolerance: scores and sums are float32 in both, the weights enter P V as bfloat16 (2^-9 of a weight) and the result is rounded to bfloat16: two roundings of at
most 2^-9 of the values' size (1, averaged over the keys: below 1) each, 4 * 2^-9 covers both sides."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu

PAGE, H, G, D = 16, 8, 2, 128


def attend(segments, qkv, pools):
    """Attention of segments (keys before, rows) whose keys and values lie in `pools` [segment][pages, 2, G, PAGE, D]."""
    from mini_llm_runtime_b200.engine.builder import EagerBuilder
    from mini_llm_runtime_b200.engine.runtime import Runtime
    from mini_llm_runtime_b200.ops.attention import paged_attention
    from mini_llm_runtime_b200.parts.base import Segment, StepContext
    rt = Runtime(torch.bfloat16)
    t = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    segs, info, positions, of_row, row, page, table = [], [], [], [], 0, 0, torch.full((len(segments), max(p.shape[0] for p in pools)), -1, dtype=torch.int32)
    for i, (start, count) in enumerate(segments):
        segs.append(Segment(i, start, count, row))
        info.append((row, count, start, i))
        positions += range(start, start + count)
        of_row += [i] * count
        table[i, :pools[i].shape[0]] = torch.arange(page, page + pools[i].shape[0])
        row, page = row + count, page + pools[i].shape[0]
    step = StepContext(rt=rt, num_rows=row, segments=segs, token_ids=None, positions=t(positions), segment_of_row=t(of_row), segment_info=t(info), slots=None,
                       tables={0: table.cuda()}, page_size=PAGE, status=t([0]))
    out = torch.full((row, H * D), float("nan"), dtype=torch.bfloat16, device="cuda")
    b = EagerBuilder(step)
    paged_attention(b, b.wrap(qkv), b.wrap(out), torch.cat(pools), 0, H, G, D, 0, D ** -0.5)
    assert step.status.item() == 0
    return out


@pytest.mark.parametrize("start,count,other", [(0, 17, (0, 65)), (0, 64, (0, 300)), (500, 40, (100, 129)), (33, 20, (0, 64))])
def test_a_short_portion_alone_and_beside_another(start, count, other):
    g = torch.Generator().manual_seed(count)
    draw = lambda *shape: torch.randn(*shape, generator=g).bfloat16().cuda()
    pools = [draw(-(-(s + n) // PAGE), 2, G, PAGE, D) for s, n in ((start, count), other)]
    qkv = draw(count + other[1], (H + 2 * G) * D)
    alone = attend([(start, count)], qkv[:count], pools[:1])
    beside = attend([(start, count), other], qkv, pools)[:count]
    if other[1] <= 64:
        assert torch.equal(alone, beside)
    else:
        assert torch.allclose(alone.float(), beside.float(), atol=4 * 2.0 ** -9, rtol=4 * 2.0 ** -9)
