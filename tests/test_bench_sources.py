"""The committed traffic figure of the step kernel goes with the sources it was
captured from, the headers that they include among them."""
import os
import shutil
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCES = ("rod_step_fp64.cu", "rod_math.cuh", "bulk_copy.cuh")


@pytest.mark.parametrize("changed", [*SOURCES, "rod_fast.cuh", "eb_internal.h"])
def test_a_changed_source_or_header_makes_the_figure_stale(changed, tmp_path, monkeypatch):
    sys.path.insert(0, ROOT)
    import bench

    for part in ("profiles", os.path.join("elasticapp_b200", "csrc")):
        shutil.copytree(os.path.join(ROOT, part), tmp_path / part)
    monkeypatch.setattr(bench, "ROOT", str(tmp_path))
    with open(tmp_path / "profiles" / "rod_step_fp64_uneven_batch.txt", encoding="utf-8") as f:
        covered = next(int(line.split(":")[1]) for line in f if line.startswith("elements_per_launch:"))
    traffic, note = bench.profile_traffic("rod_step_fp64", "uneven_batch", SOURCES, covered)
    assert traffic is not None, note
    with open(tmp_path / "elasticapp_b200" / "csrc" / changed, "a", encoding="utf-8") as f:
        f.write("// changed\n")
    traffic, note = bench.profile_traffic("rod_step_fp64", "uneven_batch", SOURCES, covered)
    assert traffic is None and "stale" in note
