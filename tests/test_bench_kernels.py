"""The kernels that bench.py's roofline names are those that the batch's gap scores,
score table and tuning reach; a traffic figure belongs to the kernels named."""
import json
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DEFAULT = {"dp_traceback": 3, "rows_max": 8, "bucket_order": 1}


@pytest.mark.parametrize("mode", [0, 1])
def test_default_configuration_is_the_linear_form(native, mode):
    sys.path.insert(0, ROOT)
    import bench
    from pastis_gb300 import capi
    gaps = capi.resolved_gaps(capi.config(mode))[:2]
    dp = bench.alignment_kernels(mode, gaps, DEFAULT)
    assert dp["kernel"] == "k_lin_dp + k_lin_walk"
    assert (dp["cells_per_op"], dp["ops_per_cell"]) == (2, 2)
    traffic = json.load(open(os.path.join(ROOT, "profiles", "traffic.json")))
    assert traffic["xdrop1m" if mode else "sw100k"]["kernel"] == dp["kernel"]


@pytest.mark.parametrize("gaps,scores,tuning,name,per_op", [
    ((-11, -2), (-4, 11), {}, "k_sw_dir + k_tb_sw (tagged 16-bit lanes, two regions per warp)", 2),
    ((-5, -5), (-4, 11), {"dp_traceback": 2}, "k_sw_dir + k_tb_sw (tagged 16-bit lanes)", 2),
    ((-32, -2), (-4, 11), {}, "k_sw_dir + k_tb_sw (16-bit lanes, two regions per warp)", 2),
    ((-32, -40), (-4, 11), {}, "k_sw_dir + k_tb_sw (16-bit lanes, two regions per warp)", 2),
    ((-2, -11), (-40, 32), {}, "k_sw_dir + k_tb_sw (16-bit lanes, two regions per warp)", 2),
    ((-2, -11), (-4, 11), {"rows_max": 7}, "k_sw_dir + k_tb_sw (tagged 16-bit lanes, two regions per warp)", 2),
    ((-2, -11), (-4, 11), {"bucket_order": 0}, "k_sw_dir + k_tb_sw (tagged 16-bit lanes, two regions per warp)", 2),
    ((-2, -11), (-4, 11), {"dp_traceback": 1}, "k_sw_dir + k_tb_sw", 1),
    ((-110, -20), (-40, 110), {}, "k_sw_dir + k_tb_sw", 1),
    ((-2, -11), (-4, 11), {"dp_traceback": 0}, "k_sw", 1),
])
def test_other_forms(native, gaps, scores, tuning, name, per_op):
    sys.path.insert(0, ROOT)
    import bench
    dp = bench.alignment_kernels(0, gaps, dict(DEFAULT, **tuning), scores)
    assert dp["kernel"] == name and dp["cells_per_op"] == per_op
    assert dp["ops_per_cell"] == 4
