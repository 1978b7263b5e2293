"""The relaxation kernel that the benchmark's roofline names, from the launches
per iteration that were counted."""
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


def test_unit_is_what_ran():
    assert bench.sor_unit(4, 128, 3000, 40) == ("sor_resident_kernel", 1.0)
    assert bench.sor_unit(8, 128, 4000, 2) == ("sor_resident_kernel", 1.0)
    assert bench.sor_unit(4, 256, 980, 560) == ("sor_stream_kernel", 2.0)
    # FP32 rows of other lengths, and FP64, run two colour sweeps per iteration
    assert bench.sor_unit(4, 250, 980, 2100) == ("sor_split_kernel", 0.5)
    assert bench.sor_unit(4, 2048, 980, 2100) == ("sor_split_vec_kernel", 0.5)
    assert bench.sor_unit(8, 256, 900, 1900) == ("sor_split_kernel", 0.5)


def test_traffic_figures_belong_to_a_precision():
    assert bench.NCU_DRAM_BYTES_PER_CELL.get(("sor_split_kernel", 4)) is None
    assert bench.NCU_DRAM_BYTES_PER_CELL[("sor_split_kernel", 8)] > 14
