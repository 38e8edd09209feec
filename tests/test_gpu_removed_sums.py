"""The particles removed at the walls and at the obstacle are added to one of
several copies of their sums, by the block that removes them. The first step of
a filled closed box removes every ion of the outermost cells and inside the
sphere: fewer blocks than copies, many more, rows of two segments."""
import numpy as np
import pytest

from rhybrid_b200 import abi
from rhybrid_b200 import config as cf

from harness import closed_box_config, load

pytestmark = pytest.mark.gpu


def first_step(cfg, grid, pops, path):
    ctx = abi.Context(abi.gpu_library(), cf.params(cfg), cf.species(cfg), capacity=[p.shape[0] + 1024 for _, p in pops])
    try:
        ctx.set_path(path)
        load(ctx, cfg, grid, pops)
        ctx.step(1)
        return ctx.counters()
    finally:
        ctx.close()


@pytest.mark.parametrize("dims,ppc", [((12, 10, 9), 4.0), ((34, 7, 6), 20.0), ((65, 9, 8), 3.0), ((31, 8, 33), 40.0)])
def test_removed_sums(dims, ppc):
    cfg = closed_box_config(*dims, ppc=ppc)
    grid, pops = cf.initial_state(cfg)
    # slow ions near their cells' centres: they move by far less than 0.1 cells (1e3 m/s and the
    # fields' 1e8 C/kg x 2e-3 V/m x 0.05 s, 0.05 s long: 600 m), so the removed ones are known
    rng = np.random.default_rng(5)
    pops = [(cnt, np.hstack([rng.uniform(0.35, 0.65, (p.shape[0], 3)) * cfg.dx, rng.uniform(-1e3, 1e3, (p.shape[0], 3)),
                            p[:, 6:]]))
            for cnt, p in pops]
    fast, f32, exact = (first_step(cfg, grid, pops, path) for path in (abi.PATH_FAST, abi.PATH_FP32, abi.PATH_EXACT))
    for s, (cnt, p) in enumerate(pops):
        cell = np.repeat(np.arange(cfg.ncells), cnt.astype(np.int64))
        ijk = np.stack([cell % cfg.nx, cell // cfg.nx % cfg.ny, cell // (cfg.nx * cfg.ny)], axis=1)
        outer = ((ijk == 0) | (ijk == np.array(dims) - 1)).any(axis=1)
        r = np.linalg.norm(np.array([cfg.x_min, cfg.y_min, cfg.z_min]) + ijk * cfg.dx + p[:, :3], axis=1)
        R = cfg.populations[s].obstacle
        w, move = p[:, 6], 2e3
        lo, hi = (w[~outer & (r < R + d)].sum() for d in (-move, move))
        assert outer.any()
        for what, got in (("fast", fast), ("fp32", f32), ("exact", exact)):
            # n terms of one sign in any order: n units of 2^-53
            esc = got[f"particleEscape[{s}]"]
            assert abs(esc - w[outer].sum()) <= p.shape[0] * 2.0**-53 * w[outer].sum(), (what, s)
            assert lo * (1 - 1e-12) <= got[f"particleImpact[{s}]"] <= hi * (1 + 1e-12), (what, s)
        # ions of the outermost cells are not accelerated: v is one FP32 rounding from the FP64 one
        a, b = fast[f"particleEscapeKineticEnergy[{s}]"], f32[f"particleEscapeKineticEnergy[{s}]"]
        assert a > 0 and abs(a - b) <= 1e-5 * a, (s, a, b)
