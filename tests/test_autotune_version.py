"""Saved tuning tables: in tables of version 1 `postpone_min` said when a lane
puts its triangles off (0: never), from version 2 on how many waiting lanes make
a warp test a part-filled round (0: the default). A version-1 threshold is not
read as the other thing; the rest of such an entry is."""
import json

from foundation_gb300 import autotune as AT


def test_version_one_thresholds_are_not_taken_over(tmp_path):
    old = {"17:incoherent:closest": dict(block=64, short_stack=4, refill_min=16, postpone_min=8, sort_bits=9, ms=1.0,
                                         default_ms=2.0),
           "render:8x8:plain": dict(wave_paths=1 << 20, tail_paths=0, ms=1.0)}
    p = tmp_path / "t.json"
    p.write_text(json.dumps({"version": 1, "entries": old}))
    t = AT.TuneTable.load(str(p))
    assert t.entries == {"17:incoherent:closest": dict(old["17:incoherent:closest"], postpone_min=0),
                         "render:8x8:plain": old["render:8x8:plain"]}
    t.entries["17:incoherent:closest"]["postpone_min"] = 8
    t.save(str(p))
    assert json.loads(p.read_text())["version"] == 2
    assert AT.TuneTable.load(str(p)).entries == t.entries
