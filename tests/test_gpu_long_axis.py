"""Grids longer than 65535 cells in y, the most blocks of a launch's y axis: a
step of the fast path against the oracle, and the FP32 form's moments against
the fast path's."""
import numpy as np
import pytest

from rhybrid_b200 import abi
from rhybrid_b200 import config as cf

from harness import assert_state_equal, load, run

pytestmark = pytest.mark.gpu

NY = 65536 + 5


def test_fast_step_matches_oracle(port_lib):
    cfg = cf.config_empty_box(3, NY, 3, ppc=0.3)
    assert_state_equal(run(abi.gpu_library(), cfg, 1, fast=True), run(port_lib, cfg, 1, fast=True), "3 x 65541 x 3")


def test_fp32_moments():
    cfg = cf.config_empty_box(3, NY, 3, ppc=0.3)
    grid, pops = cf.initial_state(cfg)
    out = []
    for path in (abi.PATH_FAST, abi.PATH_FP32):
        with abi.Context(abi.gpu_library(), cf.params(cfg), cf.species(cfg), capacity=[pops[0][1].shape[0] + 1024]) as ctx:
            ctx.set_path(path)
            load(ctx, cfg, grid, pops)
            ctx.step(1)
            out.append([ctx.download_array(n).copy() for n in ("cellRhoQi", "cellJi")])
    # a cell's sum of FP32 products of at most 8 ions: positions, weights and sums round to 2^-24 each, and a weight
    # below 1 can be the difference of two positions; 64 roundings of the largest moment bound it
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= 64 * 2.0**-24 * np.abs(a).max()
