"""The autotuner times each parameter where it acts: noise in the step times
must not move a class of the reverse sweep (which only a rollout's backward
pass can time) and nothing moves the parameter without effect.  Timings are
faked, so this runs without a GPU."""
import importlib
import re
import sys

import pytest


class FakeTorch:
    class cuda:
        get_device_name = staticmethod(lambda i: "fake")


def table(monkeypatch, tmp_path, step_ms, reverse_ms):
    at = importlib.import_module("fyzzxyzzy-sdk_b200.autotune")
    monkeypatch.setitem(sys.modules, "torch", FakeTorch)
    monkeypatch.setenv("FYZZ_B200_TUNING", "none")
    monkeypatch.setattr(at, "_pkg", lambda: (None, None))
    for name in ("large_scene_specs", "many_scenes_specs", "rollout_specs"):
        monkeypatch.setattr(at, name, lambda scenes: ([], 0), raising=False)
    monkeypatch.setattr(at, "measure", lambda torch, pkg, specs, settle, params, steps: step_ms(params))
    monkeypatch.setattr(at, "measure_reverse", lambda pkg, specs, settle, params, steps=8: reverse_ms(params),
                        raising=False)
    out = tmp_path / "tuning.txt"
    monkeypatch.setattr("sys.argv", ["autotune.py", "--out", str(out)])
    at.main()
    return {line.split()[0]: dict(zip(at.FIELDS, map(int, line.split()[1:])))
            for line in out.read_text().splitlines() if re.match("[a-z]", line)}


DEFAULTS = {"island_thread": 8, "island_warp": 96, "island_cta": 512, "radix_bits": 8, "elem_block": 256,
            "work_queue": 0}


@pytest.mark.parametrize("name,value", [("island_thread", 4), ("island_warp", 32), ("island_cta", 128)])
def test_step_times_do_not_move_what_does_not_act_there(monkeypatch, tmp_path, name, value):
    got = table(monkeypatch, tmp_path, lambda p: 0.9 if p[name] == value else 1.0, lambda p: 1.0)
    assert got == {"large_scene": DEFAULTS, "many_scenes": DEFAULTS}


def test_each_parameter_follows_its_own_timing(monkeypatch, tmp_path):
    got = table(monkeypatch, tmp_path, lambda p: 0.9 if p["elem_block"] == 512 else 1.0,
                lambda p: 0.9 if p["island_cta"] == 256 else 1.0)
    want = dict(DEFAULTS, elem_block=512, island_cta=256)
    assert got == {"large_scene": want, "many_scenes": want}


def test_a_lead_that_does_not_repeat_is_noise(monkeypatch, tmp_path):
    seen = []

    def once_fast(p):
        first = p["radix_bits"] == 9 and seen.count(9) < 2
        seen.append(p["radix_bits"])
        return 0.9 if first else 1.0
    got = table(monkeypatch, tmp_path, once_fast, lambda p: 1.0)
    assert got == {"large_scene": DEFAULTS, "many_scenes": DEFAULTS}
