"""The measured DRAM bytes and issue counters that bench.py prints beside the evidence kernel belong to the
kernel and to a tiling that exist: the tiling's name follows the default tile rule, and every (tiling, rays
per item) the autotuner may choose has its own figure."""
import json
import re
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("variant,cells,name", [("k3dom", 1 << 19, "16x16x4"), ("k3dom", (1 << 19) - 1, "8x8x4"),
                                                ("dsphdmib", 1 << 17, "16x16x8"), ("dsphdmib", (1 << 17) - 1, "8x8x4")])
def test_default_tiling_name(variant, cells, name):
    import bench
    assert bench.tiling_name(0, variant, cells) == name
    assert [bench.tiling_name(r, variant, cells) for r in (1, 2, 3)] == ["8x8x4", "16x16x4", "16x16x8"]


def test_figures_are_of_the_kernel():
    d = json.loads((ROOT / "profiles" / "bgki_traffic.json").read_text())
    src = (ROOT / "k3dom_b200" / "csrc" / "evidence.cu").read_text()
    assert re.search(r"__global__ void __launch_bounds__\([^)]*\) %s\(" % d["kernel"], src)
    assert d["issue"]["what"].split()[0] == d["kernel"]
    assert set(d["per_tiling"]) == {f"{t}@{c}" for t in ("8x8x4", "16x16x4", "16x16x8") for c in (512, 1024)}
