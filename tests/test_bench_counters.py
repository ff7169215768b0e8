"""bench.py's counters (CPU): the kernels it names exist, the committed ncu counts of
this build are the ones it uses, and counts of another build, another form or a kernel
without a summary are not used."""
import json
import os
import re
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402

CSRC = os.path.join(ROOT, "romspath_b200", "csrc")


def test_named_kernels_exist():
    text = "".join(open(os.path.join(CSRC, f)).read() for f in os.listdir(CSRC) if f.endswith(".cu"))
    for ks in bench.KERNELS.values():
        for k in ks:
            assert re.search(rf"__global__[^;{{]*\b{k}\(", text), k


@pytest.fixture
def tree(tmp_path, monkeypatch):
    """A copy of the sources and of summaries made for them."""
    for f in bench.STEP_SOURCES:
        p = tmp_path / "romspath_b200" / "csrc" / f
        p.parent.mkdir(parents=True, exist_ok=True)
        p.write_text(open(os.path.join(CSRC, f)).read())
    (tmp_path / "profiles").mkdir()
    monkeypatch.setattr(bench, "ROOT", str(tmp_path))

    def write(build=None, form="f32", kernels=("k_vturb", "k_advect")):
        b = build or bench.kernel_build()
        t = {k: {"form": form, "particles": 10, "build": b, "ncu_ms": 1.0 + i, "dram_bytes_per_launch": 100 * (i + 1),
                 "lts_bytes_per_launch": 1000 * (i + 1)} for i, k in enumerate(kernels)}
        f = {k: {"form": form, "particles": 10, "build": b, "fp64_flop_per_launch": 7 * (i + 1),
                 "fp64_pipe_active_pct": 30.0 * (i + 1), "source": "s"} for i, k in enumerate(kernels)}
        for n, d in (("traffic", t), ("fp64", f)):
            (tmp_path / "profiles" / f"step_cfg2_{n}.json").write_text(json.dumps({"workload": "cfg2", "kernels": d}))
        return tmp_path

    return write


def test_counters_of_the_exact_step_are_summed_over_its_kernels(tree):
    tree()
    c = bench.step_counters("cfg2", "f32")
    assert (c["dram_bytes"], c["lts_bytes"], c["fp64_flop"], c["particles"]) == (300, 3000, 21, 10)
    assert c["pipe"] == pytest.approx((30.0 * 1.0 + 60.0 * 2.0) / 3.0)


def test_counters_that_are_not_this_builds_are_not_used(tree):
    for kw in ({"build": "0" * 12}, {"kernels": ("k_vturb",)}, {"form": "mixed"}):
        tree(**kw)
        assert bench.step_counters("cfg2", "f32") is None, kw
    d = tree()
    assert bench.step_counters("cfg3", "f32") is None            # no summary of that workload
    src = d / "romspath_b200" / "csrc" / "rp_step.cuh"
    text = src.read_text()
    src.write_text("// a comment\n" + text)
    assert bench.step_counters("cfg2", "f32") is not None        # comments are not the kernels
    src.write_text(text + "\nconstexpr int kOther = 1;\n")
    assert bench.step_counters("cfg2", "f32") is None


def test_committed_counters_are_self_consistent():
    for wl in ("cfg2", "cfg3"):
        T, F = (json.load(open(os.path.join(ROOT, "profiles", f"step_{wl}_{n}.json")))["kernels"]
                for n in ("traffic", "fp64"))
        for k, t in T.items():
            if "build" in t:
                assert F[k]["build"] == t["build"] and F[k]["form"] == t["form"], k
                assert F[k]["fp64_flop_per_launch"] == F[k]["dadd"] + F[k]["dmul"] + 2 * F[k]["dfma"]
                assert t["lts_bytes_per_launch"] > t["dram_bytes_per_launch"] > 0 and t["ncu_ms"] > 0
        assert not any("build" in t for k, t in T.items() if k == "k_step_fused")
