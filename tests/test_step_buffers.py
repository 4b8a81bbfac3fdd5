"""The packed metadata of steps: layouts that come back, and ever other ones between them."""

import numpy as np
import pytest
import torch

from test_cache_manager import FULL, WIN, make

from freetoken_b200.cache.manager import NULL_PAGE
from freetoken_b200.engine import step
from freetoken_b200.engine.step import ALIGN, MOST_LAYOUTS, StepBuffers

CPU = torch.device("cpu")


def sections(rng, lens):
    return [(f"s{i}", rng.integers(-1000, 1000, size=n).astype(np.int32)) for i, n in enumerate(lens)]


def check(buffers, secs):
    """Every section where a plain packing has it, with its values."""
    got, at = buffers.upload(secs), 0
    assert list(got) == [name for name, _ in secs]
    for name, arr in secs:
        assert got[name].shape == arr.shape and got[name].is_contiguous() and got[name].storage_offset() == at
        np.testing.assert_array_equal(got[name].numpy(), arr)
        at += -(-max(arr.size, 1) // ALIGN) * ALIGN
    assert buffers.last_upload_bytes == 4 * at
    return got


def test_a_layout_that_comes_back_is_kept_through_ever_other_ones(monkeypatch):
    rng = np.random.default_rng(0)
    buffers, made = StepBuffers(CPU, 1 << 14), []
    real = StepBuffers._layout
    monkeypatch.setattr(StepBuffers, "_layout", lambda self, secs: made.append(len(secs)) or real(self, secs))
    decode = [8, (8, 4), 3, (0, 2), 1]
    for _ in range(2):
        check(buffers, sections(rng, decode))
    assert len(made) == 1
    for n in range(3 * MOST_LAYOUTS):  # prompts of ever other lengths beside the decode steps
        check(buffers, sections(rng, [n + 1, (2, 4), n + 1]))
        check(buffers, sections(rng, decode))
    assert len(made) == 1 and len(buffers._layouts) == 1 and len(buffers._met) <= MOST_LAYOUTS
    for _ in range(2):  # and more of them that come back than are kept
        for n in range(2 * MOST_LAYOUTS):
            for _ in range(2):
                check(buffers, sections(rng, [n + 1]))
    assert len(buffers._layouts) == MOST_LAYOUTS


def test_what_a_step_was_given_keeps_its_place():
    """Views of two steps of one layout are the same memory, whether they were kept or made for the step."""
    rng = np.random.default_rng(1)
    buffers = StepBuffers(CPU, 64)
    first = check(buffers, sections(rng, [5, (3, 4)]))
    for _ in range(3):
        again = check(buffers, sections(rng, [5, (3, 4)]))
        assert all(again[k].data_ptr() == first[k].data_ptr() for k in first)
        again["more"] = None  # (a step's own dictionary)
    with pytest.raises(RuntimeError):
        buffers.upload(sections(rng, [60, 8]))


def test_both_host_buffers_are_waited_for_before_they_are_used_again(monkeypatch):
    """A turn's event is made once, recorded by each of its steps and waited for by the next but one."""
    log = []

    class Event:
        def __init__(self):
            self.name = sum(x[0] == "made" for x in log)
            log.append(("made", self.name))

        def record(self):
            log.append(("record", self.name))

        def synchronize(self):
            log.append(("wait", self.name))

    monkeypatch.setattr(step.torch.cuda, "Event", Event)
    buffers = StepBuffers(CPU, 64)
    buffers.device = type("D", (), dict(type="cuda"))
    for _ in range(4):
        buffers.upload([("a", np.arange(3, dtype=np.int32))])
    assert log == [("made", 0), ("record", 0), ("made", 1), ("record", 1), ("wait", 0), ("record", 0), ("wait", 1), ("record", 1)]


@pytest.mark.parametrize("need", [FULL, WIN], ids=["whole", "windowed"])
def test_entries_of_fresh_pages_taken_together_are_those_taken_one_by_one(need):
    """Portions, decode steps, a closed request: entry after entry leaves the same table, updates and slots."""
    one, many = make([(0, need)], pages=24, seq=32), make([(0, need)], pages=24, seq=32)
    g = one.paged[0]
    g.take_entries = lambda row, block, pages: [g.set_entry(row, block + i, p) for i, p in enumerate(pages)]
    for entries in ([("a", 13), ("b", 5)], [("a", 1), ("b", 1)], [("a", 3), ("c", 9)], None, [("a", 1), ("b", 7), ("d", 4)]):
        seen = []
        for m in (one, many):
            if entries is None:
                m.close("c")
                continue
            for rid, _ in entries:
                if rid not in m.requests:
                    m.open(rid)
            before = {rid: m.requests[rid].length for rid, _ in entries}
            plan = m.begin_step(entries)
            seen.append((plan.slot_maps[0].tolist(), [tuple(map(int, u)) for u in m.take_updates(0)]))
            table, at = m.paged[0].table_host, 0
            for rid, n in entries:
                for pos in range(before[rid], before[rid] + n):
                    page = table[m.requests[rid].row, pos // 4]
                    assert seen[-1][0][at] == (-1 if page == NULL_PAGE else page * 4 + pos % 4)
                    at += 1
            m.end_step()
        np.testing.assert_array_equal(one.paged[0].table_host, many.paged[0].table_host)
        assert entries is None or seen[0] == seen[1]
    for m in (one, many):
        for rid in list(m.requests):
            m.close(rid)
        assert (m.paged[0].table_host == NULL_PAGE).all()
