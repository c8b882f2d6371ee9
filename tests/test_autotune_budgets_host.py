"""The autotuner times both register budgets, and kernels that two candidates share once (no GPU)."""
from spectral_b200 import autotune, configs


def test_default_candidates_name_both_register_budgets():
    # 0 is one or the other by the number of paths, so a list with 0 and 8 misses the 96 registers of large launches
    for layout in ((2, False), (4, False), (8, False), (4, True), (8, True)):
        mega = [c for c in autotune.default_candidates() if c.kernel == "mega" and (c.width, c.quantize) == layout]
        assert {c.occupancy for c in mega} == {5, 8}, layout


class FakeRenderer:
    def __init__(self, scene, cfg, **kw):
        pass

    def __enter__(self):
        return self

    def __exit__(self, *a):
        pass

    def set_launch_config(self, **kw):
        pass

    def check_device(self):
        return 0


def test_candidates_of_the_same_kernels_are_timed_once(monkeypatch):
    s, c, ex = configs.box_scene(width=8, height=8, sphere_slices=8, sphere_stacks=9)
    calls = []
    monkeypatch.setattr(autotune, "Renderer", FakeRenderer)
    monkeypatch.setattr(autotune._lib, "build_bvh_host", lambda *a: None)
    monkeypatch.setattr(autotune, "_time_passes", lambda *a, **k: calls.append(a) or float(len(calls)))
    cands = [autotune.Candidate(2, "default", "wavefront", 128, 0, 1, tb) for tb in (16, 32, 64)]
    cands += [autotune.Candidate(2, t, "mega", 128, 0, occupancy=o) for t in ("default", "speculative") for o in (5, 8)]
    best, table = autotune.tune(s, c, eems=ex["eems"], cmf=ex["cmf"], candidates=cands)
    assert [x for x, _ in table] == cands and best == cands[0]
    assert len(calls) == 3 and [ms for _, ms in table] == [1.0, 1.0, 1.0, 2.0, 3.0, 2.0, 3.0]
    calls.clear()
    tuned = autotune.tune(s, c, eems=ex["eems"], cmf=ex["cmf"], bundles=True)[1]
    assert len(calls) == len({(x.width, x.kernel, x.block_size, x.blocks_per_sm, x.sort_keys,
                               x.occupancy, x.queue_capacity, x.quantize) for x, _ in tuned}) < len(tuned)
