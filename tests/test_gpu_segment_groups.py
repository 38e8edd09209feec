"""The push kernel takes a segment's particles in groups of 32, every species
starting a new group, and skips the wall tests of rows away from the walls. The
fast path is bitwise with the oracle where that can go wrong: species of 31 to
33 and 255 to 257 particles per segment, empty ones between them, the smallest
periodic axes, rows one cell from a wall, two segments per row."""
import dataclasses

import numpy as np
import pytest

from rhybrid_b200 import abi
from rhybrid_b200 import config as cf

from harness import assert_state_equal, closed_box_config, run

pytestmark = pytest.mark.gpu


def split(cfg, pops, counts):
    """The particles of one population dealt to species of counts[s] particles per
    row of cells (the rest to the last), in their order."""
    cnt, p = pops[0]
    cell = np.repeat(np.arange(cfg.ncells), cnt.astype(np.int64))
    row = cell // cfg.nx
    at = np.arange(p.shape[0]) - np.searchsorted(row, row)   # place within the row
    edge = np.cumsum(counts)
    s = np.searchsorted(edge, at, side="right")
    out = []
    for k in range(len(counts) + 1):
        m = s == k
        out.append((np.bincount(cell[m], minlength=cfg.ncells).astype(np.uint32), p[m]))
    return out


@pytest.mark.parametrize("counts", [(31, 33), (32, 0, 1), (0, 255, 0), (256, 0, 32), (257, 31), (1, 0, 0, 64, 7)])
@pytest.mark.parametrize("dims", [(32, 4, 3), (3, 3, 3), (40, 5, 6), (34, 7, 5)])
def test_species_groups(port_lib, counts, dims):
    closed = dims[0] in (34, 40)
    ppc = 700.0 / dims[0]
    if closed:
        cfg = closed_box_config(nx=dims[0], ny=dims[1], nz=dims[2], ppc=ppc, two_species=False)
    else:
        cfg = cf.config_empty_box(*dims, ppc=ppc)
    grid, pops = cf.initial_state(cfg)
    pops = split(cfg, pops, counts)
    base = cfg.populations[0]
    cfg = cfg.replace(populations=[dataclasses.replace(base, name=f"s{k}", charge=1.0 + k % 2) for k in range(len(pops))])
    lib = abi.gpu_library()
    assert_state_equal(run(lib, cfg, 3, grid=grid, pops=pops, fast=True),
                       run(port_lib, cfg, 3, grid=grid, pops=pops, fast=True), f"{dims} {counts}")
