"""What parts record for steps of a range of row counts, without a GPU: a program is made of addresses and launches nothing."""
from types import SimpleNamespace

import pytest
import torch

from mini_llm_runtime_b200.engine.builder import ProgramBuilder


def recorder(lo, hi):
    rt = SimpleNamespace(is_bf16=True, use_tcgen05=True, dtype=torch.bfloat16, materialize=lambda b, x: x)
    b = ProgramBuilder(rt, lo, hi, 0, 1, 1 << 20, 16, 0, [])
    b.begin()
    return b


@pytest.mark.parametrize("experts,top,width,inter", [(16, 4, 2048, 1024), (8, 8, 1024, 64)])
def test_many_rows_of_routed_experts_take_no_room_for_the_rows_side_by_side(experts, top, width, inter):
    from mini_llm_runtime_b200.config.base import PartSpec
    from mini_llm_runtime_b200.parts.experts import RoutedExperts
    lo, hi = 64 * experts // top, 8192
    part = RoutedExperts(PartSpec("routed_experts", {"hidden_size": width, "intermediate_size": inter, "experts": experts, "top": top}, {"correction": "c"}))
    part.router = part.correction = part.w_gate = part.w_up = part.w_down = part.counts = torch.zeros(1)
    b = recorder(lo, hi)
    x = b.temp(b.rows, width, torch.bfloat16)
    part.emit(b, x)
    assert b.names.count("mlr_grouped_product_bf16") == 2 and "mlr_experts_gather" in b.names
    # What the step cannot do without: x, the products' two results, the sum; five numbers a pair and the list of tiles.
    needed = hi * (width * 2 + top * (inter * 2 + width * 4) + width * 4) + hi * top * 5 * 4 + 3 * 4 * (hi * top // 32 + experts) + 4 * (experts + 1)
    assert b.workspace_bytes() <= needed + 256 * 16
