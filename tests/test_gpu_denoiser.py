"""The learned denoiser (rhgpu_dn): its BF16 tensor-core forward and backward
against the numpy oracle (oracle/denoiser.py, same BF16 roundings, float64
accumulation), its training on pairs generated by the method, what the
trained network gains on held-out pairs, and the learned form's step and gate."""
import numpy as np
import pytest

from oracle import denoiser as odn
from rhybrid_b200 import abi
from rhybrid_b200 import config as cf
from rhybrid_b200 import learned

from harness import closed_box_config

pytestmark = pytest.mark.gpu

SHAPE = (6, 7, 9)          # nz, ny, nx
PERIODIC = (1, 0, 1)       # x, y, z


def random_params(rng, scale=0.15):
    p = rng.normal(0.0, scale, odn.PARAMS).astype(np.float32)
    for l in range(3):
        base = l * odn.LAYER
        w = p[base:base + odn.TAPS * odn.C * odn.C].reshape(odn.TAPS, odn.C, odn.C)
        if l == 0:
            w[:, 4:, :] = 0.0
        if l == 2:
            w[:, :, 4:] = 0.0
            p[base + odn.TAPS * odn.C * odn.C + 4:base + odn.LAYER] = 0.0
    return p


def make(lib, sr=2.0, sj=3.0):
    nz, ny, nx = SHAPE
    d = abi.Denoiser(lib, nx, ny, nz, PERIODIC)
    d.set_scales(sr, sj)
    return d


def moments(rng):
    x = rng.normal(0, 1, SHAPE + (4,)).astype(np.float32)
    return x


def to_abi(x, sr, sj):
    """normalized x[.., 4] -> (rho, Ji interleaved) in physical units"""
    rho = (x[..., 0].astype(np.float64) * sr).reshape(-1)
    ji = (x[..., 1:].astype(np.float64) * sj).reshape(-1, 3)
    return rho, ji


def test_forward_matches_oracle():
    rng = np.random.default_rng(11)
    lib = abi.gpu_library()
    d = make(lib)
    try:
        p = random_params(rng)
        d.set_params(p)
        x = moments(rng)
        rho, ji = to_abi(x, 2.0, 3.0)
        ro, jo = d.apply(rho, ji)
        got = np.concatenate([(ro / 2.0).reshape(SHAPE + (1,)), (jo / 3.0).reshape(SHAPE + (3,))], axis=-1)
        want, _ = odn.forward(p, x, PERIODIC, bf16_mode=True)
        err = np.abs(got - want).max() / np.abs(want).max()
        print(f"denoiser forward vs oracle: max rel err {err:.2e}")
        assert err < 1e-2
    finally:
        d.close()


def test_velocity_form_matches_oracle():
    """Velocity form: the network sees rho / sr and (J / rho) / su; it hands back
    rho' = sr x0' and J = rho' su u'. Checked against the oracle's forward on the
    same normalized input."""
    rng = np.random.default_rng(12)
    lib = abi.gpu_library()
    sr, su = 2.0, 3.0
    d = make(lib, sr, su)
    try:
        d.set_velocity_form(True)
        p = random_params(rng)
        d.set_params(p)
        x = moments(rng)
        x[..., 0] = 0.5 + np.abs(x[..., 0])          # positive densities
        rho = (x[..., 0].astype(np.float64) * sr).reshape(-1)
        ji = (x[..., 1:].astype(np.float64) * su * rho.reshape(SHAPE + (1,))).reshape(-1, 3)
        ro, jo = d.apply(rho, ji)
        want, _ = odn.forward(p, x, PERIODIC, bf16_mode=True)
        want = want.astype(np.float64)
        want_rho = (want[..., 0] * sr).reshape(-1)
        want_j = (want[..., :1] * sr * want[..., 1:] * su).reshape(-1, 3)
        err_rho = np.abs(ro - want_rho).max() / np.abs(want_rho).max()
        err_j = np.abs(jo - want_j).max() / np.abs(want_j).max()
        print(f"denoiser velocity form vs oracle: max rel err rho {err_rho:.2e}, J {err_j:.2e}")
        assert err_rho < 1e-2 and err_j < 1e-2
        # a zero network hands the moments back (to FP32 rounding of the normalized values)
        d.set_params(np.zeros(odn.PARAMS, np.float32))
        ro, jo = d.apply(rho, ji)
        assert np.allclose(ro, rho, rtol=1e-6, atol=0)
        assert np.allclose(jo, ji, rtol=2e-6, atol=1e-6 * np.abs(ji).max())
    finally:
        d.close()


def test_keep_mask():
    """Cells of the keep mask hand their moments back unchanged, bit for bit;
    the others get what the unmasked network gives."""
    rng = np.random.default_rng(13)
    lib = abi.gpu_library()
    d = make(lib)
    try:
        d.set_params(random_params(rng))
        rho, ji = to_abi(moments(rng), 2.0, 3.0)
        ro, jo = d.apply(rho, ji)
        keep = (rng.random(rho.size) < 0.4).astype(np.uint8)
        d.set_keep_mask(keep)
        rk, jk = d.apply(rho, ji)
        k = keep.astype(bool)
        assert np.array_equal(rk[k], rho[k]) and np.array_equal(jk[k], ji[k])
        assert np.array_equal(rk[~k], ro[~k]) and np.array_equal(jk[~k], jo[~k])
        d.set_keep_mask(None)
        r2, j2 = d.apply(rho, ji)
        assert np.array_equal(r2, ro) and np.array_equal(j2, jo)
    finally:
        d.close()


def test_gradients_match_oracle():
    rng = np.random.default_rng(12)
    lib = abi.gpu_library()
    d = make(lib)
    try:
        p = random_params(rng)
        d.set_params(p)
        x, t = moments(rng), moments(rng)
        loss, g = d.loss_grad(*to_abi(x, 2.0, 3.0), *to_abi(t, 2.0, 3.0))
        lw, gw = odn.loss_grad(p, x, t, PERIODIC, bf16_mode=True)
        print(f"denoiser loss {loss:.6e} oracle {lw:.6e}")
        assert abs(loss - lw) <= 1e-3 * lw
        for l in range(3):
            sl = slice(l * odn.LAYER, (l + 1) * odn.LAYER)
            e = np.linalg.norm(g[sl] - gw[sl]) / np.linalg.norm(gw[sl])
            print(f"layer {l} gradient rel L2 err {e:.2e}")
            assert e < 2e-2
    finally:
        d.close()


# sizes (nx, ny, nz) and the output slices that a block of the convolutions streams there (test_cpu_block_rules.py holds
# them to the rule): the last block has fewer; two columns of blocks in x at one of them; 14 to 107 rows of gradient
# partials
SLICES = [((3, 173, 27), 2), ((31, 213, 11), 2), ((3, 1581, 5), 3), ((3, 1581, 15), 8), ((3, 1581, 23), 12)]


@pytest.mark.parametrize("dims,periodic", [(d, (1, 0, 1) if q % 2 else (0, 1, 0)) for q, (d, _) in enumerate(SLICES)])
def test_streamed_slices_match_oracle(dims, periodic):
    """Forward (in place, from the moments) and gradients where a block streams
    several slices, to the bounds of the small grid's tests."""
    nx, ny, nz = dims
    rng = np.random.default_rng(nz)
    d = abi.Denoiser(abi.gpu_library(), nx, ny, nz, periodic)
    try:
        d.set_scales(2.0, 3.0)
        p = random_params(rng)
        d.set_params(p)
        x = rng.normal(0, 1, (nz, ny, nx, 4)).astype(np.float32)
        ro, jo = d.apply(*to_abi(x, 2.0, 3.0))
        got = np.concatenate([(ro / 2.0).reshape(nz, ny, nx, 1), (jo / 3.0).reshape(nz, ny, nx, 3)], axis=-1)
        want, _ = odn.forward(p, x, periodic, bf16_mode=True)
        assert np.abs(got - want).max() < 1e-2 * np.abs(want).max()
        t = rng.normal(0, 1, x.shape).astype(np.float32)
        loss, g = d.loss_grad(*to_abi(x, 2.0, 3.0), *to_abi(t, 2.0, 3.0))
        lw, gw = odn.loss_grad(p, x, t, periodic, bf16_mode=True)
        assert abs(loss - lw) <= 1e-3 * lw
        for l in range(3):
            sl = slice(l * odn.LAYER, (l + 1) * odn.LAYER)
            assert np.linalg.norm(g[sl] - gw[sl]) < 2e-2 * np.linalg.norm(gw[sl]), l
    finally:
        d.close()


def test_training_on_method_pairs_gains_on_held_out_pairs():
    """Mars-like geometry (2 % of the cells) at 256 ppc; pairs at 8 ppc (1 in
    32 particles) from 6 states; after training, the denoised moments of a
    held-out pair (a later state) are closer to the 256-ppc moments than the
    raw 8-ppc deposit."""
    from rhybrid_b200 import evaluate
    lib = abi.gpu_library()
    cfg = evaluate.mars_at(256.0, 0.02)
    dn = learned.new_denoiser(lib, cfg, pair_capacity=48)
    try:
        losses, ctx = learned.train_on_run(lib, cfg, dn, factor=32, steps=6, pairs_per_step=8, iters_per_step=80,
                                           lr=2e-3)
        try:
            ctx.step(3)
            dn.add_pair(ctx, 32, 5)
            _, newest = dn.num_pairs()
            e = dn.pair_error(newest)
        finally:
            ctx.close()
        print(f"losses {['%.3e' % l for l in losses]}; held-out: {e}")
        assert losses[-1] < losses[0]
        assert e["dn_rho"] < 0.7 * e["raw_rho"]
        assert e["dn_J"] < 0.7 * e["raw_J"]
    finally:
        dn.close()


def test_learned_form_step_and_gate():
    lib = abi.gpu_library()
    cfg_low = closed_box_config(nx=12, ny=10, nz=9, ppc=8.0, two_species=False)
    cfg_hi = cfg_low.replace(populations=[cfg_low.populations[0].__class__(**{**cfg_low.populations[0].__dict__, "ppc": 64.0})])
    dn = learned.new_denoiser(lib, cfg_low, pair_capacity=0)
    form = learned.LearnedForm(lib, cfg_low, cfg_hi, dn, threshold=0.5)
    try:
        form.step(2)
        e_rho, e_j, on = form.judge()
        assert on and np.isfinite(e_rho) and np.isfinite(e_j)
        # a threshold below the error switches the denoiser off; the run goes on
        form.threshold = 1e-9
        form.step(1)
        _, _, on = form.judge()
        assert not on
        form.step(1)
        assert np.isfinite(form.low.download_array("cellRhoQi")).all()
    finally:
        form.close()
        dn.close()


def test_crop_pairs_and_border_loss():
    """rhgpu_dn_add_crops: crops of a context's (subsample, full) deposits as
    pairs for a crop-sized network. A crop pair's sampling error matches the
    whole grid's in size; crops must lie inside the grid; training on the crops
    with the 3-voxel border left out of the loss lowers the loss, and the
    parameters apply to the whole grid."""
    lib = abi.gpu_library()
    cfg = learned.c4_config(48.0, scale=0.01)
    ctx = learned.filled_context(lib, cfg, seed=11)
    full = abi.Denoiser(lib, cfg.nx, cfg.ny, cfg.nz, cfg.periodic, pair_capacity=1)
    crop = abi.Denoiser(lib, 16, 16, 16, (0, 0, 0), pair_capacity=128)
    try:
        ctx.step(2)
        for dn in (full, crop):
            dn.set_scales(*learned.moment_scales(cfg))
        crop.set_params(learned.init_params(0))
        full.add_pair(ctx, 6, 1)
        org = np.array([[0, 0, 0], [cfg.nx - 16, cfg.ny - 16, cfg.nz - 16], [3, 5, 7]])
        crop.add_crops(ctx, 6, 1, org)
        e_full = full.pair_error(0)["raw_rho"]
        for i in range(3):
            e = crop.pair_error(i)["raw_rho"]
            assert 0.5 * e_full < e < 2.0 * e_full, (e, e_full)
        with pytest.raises(abi.RhError):
            crop.add_crops(ctx, 6, 1, np.array([[cfg.nx - 15, 0, 0]]))
        rng = np.random.default_rng(3)
        for st in range(30):
            ctx.step(1)
            o = np.stack([rng.integers(0, n - 16 + 1, 4) for n in (cfg.nx, cfg.ny, cfg.nz)], axis=1)
            crop.add_crops(ctx, 6, st % 6, o)
        crop.set_loss_border(3)
        first = crop.train(20, 1e-3)
        for _ in range(25):
            last = crop.train(20, 1e-3)
        assert last < 0.7 * first, (first, last)
        full.set_params(crop.params())
        full.add_pair(ctx, 6, 2)
        e = full.pair_error(0)
        assert e["dn_rho"] < e["raw_rho"] and e["dn_J"] < e["raw_J"], e
    finally:
        full.close()
        crop.close()
        ctx.close()
