"""What bench.py reports beside its times: the recorded DRAM traffic belongs to
the launches of the run, and the engine's default grid is the library's."""
import os
import re
from types import SimpleNamespace

import pytest

import bench

WORKLOAD = "pancake14-2bit"


def run(**changes):
    args = dict(workload=WORKLOAD, window_bits=0, far_marks="auto", direction="auto", bottom_up_ratio=0.0)
    tr = bench.LEVEL_TRAFFIC[WORKLOAD]
    st = dict(levels=tr["launches"], window_bits=tr["window_bits"], threads=tr["threads"])
    for k, v in changes.items():
        (st if k in ("levels", "threads") else args)[k] = v
    return bench.recorded_traffic(SimpleNamespace(**args), SimpleNamespace(**st))


def test_traffic_of_the_captured_launches():
    assert run() == run(far_marks="near") == bench.LEVEL_TRAFFIC[WORKLOAD]


@pytest.mark.parametrize("change", [dict(window_bits=16), dict(far_marks="all"), dict(far_marks="none"),
                                    dict(direction="top_down"), dict(bottom_up_ratio=2.0), dict(threads=256),
                                    dict(levels=16), dict(workload="pancake13-3bit")], ids=str)
def test_no_traffic_of_other_launches(change):
    """A window that is asked for reports the size of the automatic one and runs another kernel."""
    assert run(**change) is None


def test_default_engine_grid():
    header = open(os.path.join(bench.REPO, "include", "psb200.h")).read()
    engine = open(os.path.join(bench.REPO, "puzzlesearch_b200", "csrc", "psb_engine.cu")).read()
    blocks = int(re.search(r"kEMinBlocks = (\d+);", engine).group(1))
    assert f"persistent blocks per SM (0 = {blocks})" in header
    assert bench.ENGINE_BLOCKS_PER_SM == blocks
