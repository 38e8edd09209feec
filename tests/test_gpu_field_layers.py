"""The node and cell passes march layers through shared memory: the field update
is bitwise with the oracle at sizes around a block's 32 x 4 and 32 x 8 (one short
of, exactly and one past a block; the smallest axes), where every block has one
plane, and at sizes where the blocks march two to eight planes and the last ones
fewer, for closed and periodic walls."""
import pytest

from rhybrid_b200 import abi
from rhybrid_b200 import config as cf

from harness import SUM_COUNTERS, assert_state_equal, closed_box_config, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("smooth", [False, True])
@pytest.mark.parametrize("dims", [(3, 3, 3), (31, 4, 9), (32, 8, 3), (33, 9, 8), (64, 5, 17), (5, 7, 33)])
@pytest.mark.parametrize("closed", [False, True])
def test_layers(port_lib, closed, dims, smooth):
    if closed:
        cfg = closed_box_config(nx=dims[0], ny=dims[1], nz=dims[2], ppc=2.0)
    else:
        cfg = cf.config_empty_box(*dims, ppc=2.0).replace(use_electron_pressure=True, electron_temperature=1e5)
    cfg = cfg.replace(electric_field_linear_smoothing_number=1 if smooth else 0,
                      electric_field_smoothing_gauss_sigma=0.8 if smooth else 0.0)
    assert_state_equal(run(abi.gpu_library(), cfg, 3, fast=True), run(port_lib, cfg, 3, fast=True), f"{dims}")


# sizes and the planes per block of the node and of the cell pass there (test_cpu_block_rules.py holds them to the
# rule): two columns of blocks in x at the last one
MARCHED = [((3, 2369, 27), 8, 8), ((3, 2369, 13), 4, 8), ((3, 2369, 7), 2, 4), ((3, 2369, 3), 1, 2),
           ((33, 1185, 13), 4, 8)]


@pytest.mark.parametrize("dims", [d for d, _, _ in MARCHED])
@pytest.mark.parametrize("closed", [False, True])
def test_marched_layers(port_lib, closed, dims):
    if closed:
        cfg = closed_box_config(nx=dims[0], ny=dims[1], nz=dims[2], ppc=0.5).replace(electric_field_smoothing_gauss_sigma=0.0)
    else:
        cfg = cf.config_empty_box(*dims, ppc=0.5).replace(use_electron_pressure=True, electron_temperature=1e5)
    cfg = cfg.replace(electric_field_linear_smoothing_number=0)   # without smoothing: Faraday's law in the cell pass
    got, want = run(abi.gpu_library(), cfg, 2, fast=True), run(port_lib, cfg, 2, fast=True)
    for st in (got, want):   # the removed particles' sums are not the field passes' (test_gpu_removed_sums.py)
        st["counters"] = {k: v for k, v in st["counters"].items() if k.split("[")[0] not in SUM_COUNTERS}
    assert_state_equal(got, want, f"{dims}")


@pytest.mark.parametrize("ppc", [0.5, 1.0, 31.0, 33.0, 65.0])
def test_exact_deposit_batches(port_lib, ppc):
    """The exact path's deposit takes a cell's particles 32 at a time and eight
    cells per block: cells without particles, with part of a batch, with more."""
    cfg = cf.config_empty_box(7, 5, 3, ppc=ppc)
    assert_state_equal(run(abi.gpu_library(), cfg, 3), run(port_lib, cfg, 3), f"exact {ppc}")
