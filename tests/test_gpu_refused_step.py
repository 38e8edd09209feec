"""A step that is refused after its push (population averages chosen before the
FP32 form, which has none) leaves nothing behind: particles given to the context
afterwards are the ones that the next step moves, as in a context that was never
refused, through every way of giving them."""
import numpy as np
import pytest

from rhybrid_b200 import abi
from rhybrid_b200 import config as cf

from harness import STATE_ARRAYS, closed_box_config, load

pytestmark = pytest.mark.gpu


def as_f32(cfg, counts, p):
    """Records of upload_particles_f32 (cell-unit offsets, velocities) and their weight."""
    return counts, np.hstack([np.minimum(p[:, :3] / cfg.dx, np.float32(1) - np.float32(2.0**-24)), p[:, 3:6]]).astype(np.float32), float(p[0, 6])


def give(ctx, cfg, pops, how):
    for s, (counts, p) in enumerate(pops):
        if how == "upload":
            ctx.upload_particles(s, counts, p)
        elif how == "upload_f32":
            ctx.upload_particles_f32(s, *as_f32(cfg, counts, p))
        else:
            pop = cfg.populations[s]
            ctx.fill_uniform(s, pop.density, pop.temperature, pop.velocity, pop.ppc, seed=7)


@pytest.mark.parametrize("how", ["upload", "upload_f32", "fill"])
@pytest.mark.parametrize("make", [lambda ppc: cf.config_empty_box(33, 9, 8, ppc=ppc),
                                  lambda ppc: closed_box_config(34, 9, 8, ppc=ppc)], ids=["periodic", "closed"])
def test_new_particles_after_a_refused_step(make, how):
    first, cfg = make(11.0), make(3.0)   # more ions first: other segment offsets
    grid, pops = cf.initial_state(cfg)
    _, old = cf.initial_state(first)
    out = []
    for refused in (True, False):
        ctx = abi.Context(abi.gpu_library(), cf.params(cfg), cf.species(cfg), capacity=[p.shape[0] + 1024 for _, p in old])
        try:
            if refused:
                ctx.set_population_averages([0] * len(pops))
            ctx.set_path(abi.PATH_FP32)
            load(ctx, cfg, grid, [])
            if refused:
                give(ctx, first, old, "upload")
                with pytest.raises(abi.RhError) as e:
                    ctx.step(1)
                assert e.value.code == abi.ERR_STATE
                assert sum(ctx.num_particles(s) for s in range(len(old))) <= sum(p.shape[0] for _, p in old)
                ctx.set_population_averages([-1] * len(pops))
            give(ctx, cfg, pops, how)
            n = [ctx.num_particles(s) for s in range(len(pops))]
            ctx.step(3)
            out.append((n, [ctx.download_particles(s) for s in range(len(pops))],
                        {a: ctx.download_array(a).copy() for a in STATE_ARRAYS}))
        finally:
            ctx.close()
    (n0, p0, a0), (n1, p1, a1) = out
    assert n0 == n1
    for (c0, q0), (c1, q1) in zip(p0, p1):
        assert np.array_equal(c0, c1) and np.array_equal(q0.view(np.uint64), q1.view(np.uint64))
    for name in STATE_ARRAYS:
        assert np.array_equal(a0[name].view(np.uint64), a1[name].view(np.uint64)), name
