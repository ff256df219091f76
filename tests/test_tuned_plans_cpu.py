"""What is tuned and generated is what runs, on the CPU.

* The autotuner's stacks lie at the tensor-core widths, where the mixed form runs
  the y and z plans it tunes, and cover every such y and z length; it writes no x
  choices, which no kernel would follow.
* The committed sources of the paired passes are what gen_plans.py writes.
"""

import json
import re
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
PKG = ROOT / "cudadecon_gb300"
sys.path.insert(0, str(PKG))
import autotune as T  # noqa: E402
import gen_plans as G  # noqa: E402


def test_tuner_probes_the_passes_it_tunes():
    src = (PKG / "csrc" / "decon_x_tc.cu").read_text()
    plans = src[src.index("#define CDX_TC_PLANS"):].split("\n\n")[0]
    widths = [int(w) for w in re.findall(r"F\((\d+),", plans)]
    assert sorted(T.TC_WIDTHS) == sorted(widths)
    lens = T.tuned_lengths(G.lengths())
    shapes = T.probe_shapes(lens)
    assert {s[0] for s in shapes} == set(G.lengths()["z"])
    assert {s[1] for s in shapes} == set(G.lengths()["y"])
    assert {s[2] for s in shapes} <= set(widths)


def test_tuner_asks_for_the_mixed_form_and_records_no_x(tmp_path, monkeypatch):
    ran = []

    def fake_run(cmd, check, env, cwd=None):
        ran.append(cmd)
        if "--probe" in cmd:
            shapes = json.loads(Path(cmd[-2]).read_text())
            rows = [{"shape": s, "grid": s, "pass_ms": [1.0] * 9} for s in shapes]
            Path(cmd[-1]).write_text(json.dumps({"device": "fake", "rows": rows}))

    def fake_copy(dst):
        dst.mkdir(parents=True)
        return dst

    monkeypatch.setattr(T.subprocess, "run", fake_run)
    monkeypatch.setattr(T, "scratch_copy", fake_copy)
    monkeypatch.setattr(G, "TUNED", tmp_path / "tuned_plans.json")
    chosen = T.tune(2, 0.02, tmp_path / "work", apply=False)
    assert chosen["x"] == {} and len(chosen["y"]) == len(G.lengths()["y"])
    assert len(chosen["z"]) == len(G.lengths()["z"]) and len(ran) == 6
    assert json.loads((PKG / "tuned_plans.json").read_text())["x"] == {}
    src = (PKG / "autotune.py").read_text()
    assert src.index('set_dft_form("mixed")') < src.index("cdx_RL_device(ctypes")


def test_committed_paired_sources_match_the_generator(tmp_path, monkeypatch):
    (tmp_path / "csrc").mkdir()
    monkeypatch.setattr(G, "HERE", tmp_path)
    monkeypatch.setattr(G, "OUT", tmp_path / "csrc" / "static_plans_gen.cuh")
    monkeypatch.setattr(G, "XDISPATCH", tmp_path / "csrc" / "x_gen_dispatch.h")
    G.generate()
    made = sorted(p.name for p in (tmp_path / "csrc").iterdir())
    units = [f"decon_{a}_gen_{k}.cu" for a, n in (("x", G.X_UNITS), ("y", G.Y_UNITS), ("z", G.Z_UNITS))
             for k in range(n)]
    assert set(made) == {"static_plans_gen.cuh", "x_gen_dispatch.h", "pair_plans_gen.cuh", *units}
    assert sorted(p.name for p in (PKG / "csrc").glob("decon_[xyz]_gen_*.cu")) == sorted(units)
    for n in made:
        assert (tmp_path / "csrc" / n).read_text() == (PKG / "csrc" / n).read_text(), n
