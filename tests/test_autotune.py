"""CPU: the autotuner's search against a plan that records what it is given:
launches that are alike are timed once, chunks are whole tiles, and a result
stored for other kernels is not applied."""
import json
import types

import pytest


class Plan:
    ewald = True

    def __init__(self, gc, chunks):
        self.gc, self.tuned = gc, [gc.Tuning(8, *chunks, 0, 0, 0)]

    def retune(self, t):
        self.tuned.append(t)

    def tuning(self):
        return self.tuned[-1]


@pytest.fixture
def search(monkeypatch):
    import torch
    from pgrav import autotune as AT, gravcuda as gc
    monkeypatch.setattr(torch.cuda, "Stream", lambda: types.SimpleNamespace(cuda_stream=0))

    def go(chunks, **kw):
        plan, timed = Plan(gc, chunks), []

        def clock(p, stream, reps):
            t = p.tuning()
            timed.append((min(t.warps_per_block, 4), t.warps_per_block * t.blocks_per_sm, t.chunk_p,
                          t.chunk_q, t.chunk_h, t.ewald_side))
            return 1.0 + 0.01 * len(timed)  # the first is the fastest

        monkeypatch.setattr(AT, "_time", clock)
        best, trials = AT.autotune(plan, **kw)
        return best, trials, timed

    return go


@pytest.mark.parametrize("chunks", [(256, 128, 64), (768, 512, 320), (2048, 128, 64)])
def test_alike_launches_are_timed_once_and_chunks_are_whole_tiles(search, chunks):
    best, trials, timed = search(chunks)
    assert len(timed) == len(set(timed))
    assert all(p % 256 == 0 and q % 128 == 0 and h % 64 == 0 for _, _, p, q, h, _ in timed)
    assert len(trials) == 6 + 4 + 4  # what was asked for, timed or not
    assert (best.chunk_p, best.chunk_q, best.chunk_h) == chunks and best.blocks_per_sm == 0


def test_a_result_of_other_kernels_is_searched_again(search, tmp_path):
    cache = str(tmp_path / "c.json")
    old = {"k": {"tuning": [8, 64, 64, 32, 1, 0, 3], "trials": []}}
    json.dump(old, open(cache, "w"))
    best, trials, timed = search((256, 128, 64), cache=cache, key="k")
    assert timed and best.blocks_per_sm == 0
    again, stored, timed = search((256, 128, 64), cache=cache, key="k")
    assert not timed and stored == trials
    assert [getattr(again, f) for f, _ in again._fields_] == [getattr(best, f) for f, _ in best._fields_]
