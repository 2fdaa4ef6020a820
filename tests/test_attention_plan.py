"""The launch plan of a step's attention, made on the host: which segments go to the few-row kernel, which in tiles of 64 rows and which in
tiles of 128, and which segments and rows the tiles name.  No GPU."""
import pytest

from mini_llm_runtime_b200.engine.executor import plan_attention

SMS = 148


def plan(segments, wide, group=4, small=1):
    """(few-row segments, 64-row tiles, 128-row tiles) of a step with segments (keys before, rows)."""
    values = plan_attention((group, 8, 0, wide, 128, small), segments, 0, SMS)
    lists = values["lists"]
    pairs = lambda at, n: [tuple(lists[at + 2 * i:at + 2 * i + 2]) for i in range(n)]
    few = list(range(len(segments))) if values["n_items"] == len(segments) else lists[values["items_offset"]:values["items_offset"] + values["n_items"]]
    return few, pairs(values["tiles_offset"], values["n_tiles"]), pairs(values["wide_offset"], values["n_wide"])


@pytest.mark.parametrize("segments,wide,tiles,wide_tiles", [
    # 0: none are wide
    ([(0, 129), (0, 17)], 0, [(0, 0), (0, 64), (0, 128), (1, 0)], []),
    # 1: where a portion of the step has more than 64 rows, all of its portions and their remainders
    ([(0, 129), (0, 17)], 1, [], [(0, 0), (0, 128), (1, 0)]),
    ([(0, 65)], 1, [], [(0, 0)]),
    ([(0, 64), (500, 17)], 1, [(0, 0), (1, 0)], []),
    # 2: all portions
    ([(0, 64), (500, 17)], 2, [], [(0, 0), (1, 0)]),
    ([(0, 5)], 2, [], [(0, 0)]),
])
def test_tiles_by_the_lengths_of_a_steps_portions(segments, wide, tiles, wide_tiles):
    few, got, got_wide = plan(segments, wide)
    assert few == [] and sorted(got) == sorted(tiles) and sorted(got_wide) == sorted(wide_tiles)


@pytest.mark.parametrize("wide", [0, 1, 2])
def test_few_rows_go_to_their_own_kernel_beside_tiles(wide):
    few, tiles, wide_tiles = plan([(100, 1), (0, 130), (7, 4), (900, 3)], wide)
    assert few == [0, 2, 3]
    assert sorted(tiles + wide_tiles) == ([(1, 0), (1, 64), (1, 128)] if wide == 0 else [(1, 0), (1, 128)])
    assert plan([(100, 1), (7, 4)], wide) == ([0, 1], [], [])


def test_tiles_with_the_most_keys_come_first():
    assert plan([(0, 200), (1000, 70)], 1)[2] == [(1, 0), (0, 128), (0, 0)]
    assert plan([(0, 200), (1000, 70)], 0)[1] == [(1, 64), (1, 0), (0, 192), (0, 128), (0, 64), (0, 0)]
