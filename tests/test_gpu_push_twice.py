"""A gather takes the deposit of the last push alone: a push that nothing
gathered leaves none of its movers' sums behind. Two pushes and a gather give
the same bits as the same pushes with a gather after each."""
import numpy as np
import pytest

from rhybrid_b200 import abi
from rhybrid_b200 import config as cf

from harness import closed_box_config, load

pytestmark = pytest.mark.gpu


def moments_after_two_pushes(cfg, path, gather_between):
    grid, pops = cf.initial_state(cfg)
    ctx = abi.Context(abi.gpu_library(), cf.params(cfg), cf.species(cfg), capacity=[p.shape[0] + 1024 for _, p in pops])
    try:
        ctx.set_path(path)
        load(ctx, cfg, grid, pops)
        ctx.push()
        if gather_between:
            ctx.accumulate()
        ctx.push()
        ctx.accumulate()
        return [ctx.download_array(n).copy() for n in ("cellRhoQi", "cellJi")]
    finally:
        ctx.close()


@pytest.mark.parametrize("cfg", [closed_box_config(34, 9, 8, ppc=6.0), cf.config_empty_box(33, 7, 6, ppc=6.0)],
                         ids=["closed", "periodic"])
@pytest.mark.parametrize("path", [abi.PATH_FAST, abi.PATH_FP32], ids=["fast", "fp32"])
def test_gather_takes_the_last_push(path, cfg):
    for got, want in zip(moments_after_two_pushes(cfg, path, False), moments_after_two_pushes(cfg, path, True)):
        assert np.array_equal(got.view(np.uint64), want.view(np.uint64))
