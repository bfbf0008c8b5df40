"""The bench's figures for kernels that leave work out: operations counted at the
reference's samples give an equivalent rate, never a share of a peak, and the density
samples of a step are named as those it determines."""
import pathlib

import numpy as np

import bench


def test_no_fraction_from_work_left_out():
    r = bench.fp32_equivalent(2.0e12, 4.0, 80.0)
    assert r["frac"] is None and r["achieved"] is None
    assert r["reference_equivalent_tflops"] == 500.0  # past the peak: no achieved rate
    assert r["reference_flop_per_launch"] == 2 * 10 ** 12 and "evaluates a part" in r["note"]


def test_samples_are_qualified():
    src = pathlib.Path(bench.__file__).read_text()
    assert src.count('line["density_samples_per_s"]') == src.count('line["density_samples_note"]') == 1


def test_stage_bytes_are_the_bit_planes():
    """A 64^3 chunk's field is 66^2 rows of 16 bytes a plane."""
    res = np.zeros((3, 8), np.int64)
    plane = 3 * 66 * 66 * 16
    assert bench.stage_work("edge_count", res, 3) == bench.stage_work("vox_count", res, 3) == plane
    res[:, 6], res[:, 7] = 100, 50
    assert bench.stage_work("edge_scatter", res, 3) == plane + 12 * 300
    assert bench.stage_work("vox_scatter", res, 3) == plane + 12 * 150
    assert bench.stage_work("hermite", res, 3) is None
