"""More movers in a step than the mover list holds (2^20 entries for this many
ions): RHGPU_ERR_CAPACITY before anything of the step but its push has run, so
that fields, moments, averages and time still belong to the particles, which
are those of the step before."""
import numpy as np
import pytest

from rhybrid_b200 import abi
from rhybrid_b200 import config as cf

from harness import load

pytestmark = pytest.mark.gpu

ARRAYS = ["faceB", "cellB", "cellRhoQi", "cellJi", "nodeE", "cellUe", "cellAverageB"]


def ions(cfg, ncross, nstay):
    """Counts and records: nstay ions at rest at cell centres, and ncross ions a tenth of a cell from the next one in y
    that move 0.8 cells a step, into another row of dual cells."""
    n = ncross + nstay
    counts = np.full(cfg.ncells, n // cfg.ncells, dtype=np.uint32)
    counts[:n % cfg.ncells] += 1
    p = np.zeros((n, 7))
    p[:, :3] = 0.5 * cfg.dx
    move = np.linspace(0, n - 1, ncross).astype(np.int64)
    p[move, 1] = 0.9 * cfg.dx
    p[move, 4] = 0.8 * cfg.dx / cfg.dt
    p[:, 6] = 1e20
    return counts, p


@pytest.mark.parametrize("path", [abi.PATH_FAST, abi.PATH_FP32], ids=["fast", "fp32"])
def test_overflow_stops_the_step_before_its_moments(path):
    cfg = cf.config_empty_box(40, 30, 24, ppc=1.0).replace(max_ion_velocity=1e9)   # capped at 0.9 dx / dt
    grid, _ = cf.initial_state(cfg)
    few, many = ions(cfg, 200, 50000), ions(cfg, (1 << 20) + 4096, 50000)
    averages = path == abi.PATH_FAST
    out = []
    for overflow in (False, True):
        ctx = abi.Context(abi.gpu_library(), cf.params(cfg), cf.species(cfg), capacity=[many[1].shape[0] + 1024])
        try:
            ctx.set_path(path)
            if averages:
                ctx.set_population_averages([0])
            load(ctx, cfg, grid, [few])
            ctx.step(2)
            if overflow:
                ctx.upload_particles(0, *many)
                uploaded = ctx.download_particles(0)
                assert np.array_equal(uploaded[0], many[0])
                for _ in range(2):   # the state after the error is the one before it
                    with pytest.raises(abi.RhError) as e:
                        ctx.step(1)
                    assert e.value.code == abi.ERR_CAPACITY and "mover list overflow" in str(e.value)
                for a, b in zip(ctx.download_particles(0), uploaded):
                    assert np.array_equal(a, b)
            out.append(({n: ctx.download_array(n).copy() for n in ARRAYS}, ctx.time()[0],
                        ctx.output_averages(cellB=False) if averages else {}))
        finally:
            ctx.close()
    (a0, t0, v0), (a1, t1, v1) = out
    for n in ARRAYS:
        assert np.array_equal(a0[n].view(np.uint64), a1[n].view(np.uint64)), n
    assert t0 == t1
    for n in v0:
        assert np.array_equal(v0[n].view(np.uint64), v1[n].view(np.uint64)), n
