"""A launch choice stored by a library whose loops were other ones is not taken
over: the case is timed anew and the entry replaced."""
import json

from warp_sph_gpt_gb300 import autotune as AT


def test_a_choice_of_other_loops_is_timed_anew(tmp_path):
    path = tmp_path / "tune.json"
    old = {"cell_factor": 1.0, "block_sph": 128, "porosity_variant": 0, "lanes_sph": 32, "ms_per_step": 1.0}
    path.write_text(json.dumps({"case": old, "other": dict(old, loops=AT.LOOPS)}))
    calls = []

    def timer(make_case, cfg):
        calls.append(cfg)
        return 1.0 if cfg["lanes_sph"] == 1 else 2.0

    best = AT.autotune(None, "case", timer=timer, cache_path=path, n_fluid=12500)
    assert calls and best["lanes_sph"] == 1
    n = len(calls)
    assert AT.autotune(None, "case", timer=timer, cache_path=path, n_fluid=12500) == best and len(calls) == n
    assert AT.autotune(None, "other", timer=timer, cache_path=path)["lanes_sph"] == 32 and len(calls) == n
