"""Squarings under a tile plan (only the K-blocks whose operand parts are not zero) against the
full products: the left-out blocks add zeros to the accumulators, so every value is the same
bits (opb_set_band_skip(0) issues every block)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

STRIKES = np.linspace(0.6, 1.4, 5)


def _both(run):
    from oplib_b200 import _lib
    lib = _lib.load()
    out = []
    for skip in (0, 1):
        assert lib.opb_set_band_skip(skip) == 0
        try:
            out.append(run())
            torch.cuda.synchronize()
        finally:
            lib.opb_set_band_skip(1)
        assert lib.opb_tc_error() == 0
    return out


@pytest.mark.parametrize("mode", ["bf16x3", "fp16x3"])
@pytest.mark.parametrize("max_d", [0, 1 << 30])  # parts from the renormalisation kernel, from the epilogues
@pytest.mark.parametrize("n", [1536, 1600, 2048, 2304])  # pair tiles, 128-row tiles, a padded size
def test_planned_squarings_are_bit_identical(cuda, n, max_d, mode):
    from oplib_b200 import _lib
    from oplib_b200.model import Lattice
    lib = _lib.load()
    lat = Lattice.local_vol(n=n, device=cuda)
    assert lib.opb_set_fused_normalisation(max_d) == 0
    try:
        full, planned = _both(lambda: lat.solve(STRIKES, 2, 0.25, 2.0 ** -10, mode=mode, all_states=True)[1])
    finally:
        lib.opb_set_fused_normalisation(-1)
    assert torch.equal(full, planned)


def test_planned_squarings_of_a_stochastic_vol_lattice(cuda):
    from oplib_b200.model import Lattice
    lat = Lattice.stoch_vol(nx=64, nv=32, device=cuda)
    full, planned = _both(lambda: lat.kernel(0.25, 2.0 ** -16, mode="bf16x3"))
    assert torch.equal(full, planned)


@pytest.mark.parametrize("cfg", range(8))
def test_planned_batch_is_bit_identical(cuda, cfg):
    """Every launch configuration, sizes on both of its tile forms and off the grid."""
    from oplib_b200.model import Batch, Lattice
    lats = [Lattice.local_vol(n=n, level=0.12 + 0.03 * i, device=cuda)
            for i, n in enumerate([128, 256, 300, 640, 1024, 1152])]
    bt = Batch(lats, STRIKES, 3, 0.25, 2.0 ** -14, autotune=False)
    bt.set_config(cfg)
    full, planned = _both(lambda: bt.execute().clone())
    assert torch.equal(full, planned)



def test_planned_batch_bermudan_is_bit_identical(cuda):
    from oplib_b200.model import Batch, Lattice
    lats = [Lattice.local_vol(n=n, level=0.12 + 0.03 * i, device=cuda) for i, n in enumerate([128, 300, 1024, 1152])]
    bt = Batch(lats, STRIKES, 3, 0.25, 2.0 ** -14, mode="fp16x3", autotune=False)
    for cfg in (0, 1, 4, 6):
        bt.set_config(cfg)
        full, planned = _both(lambda: bt.execute_bermudan(barrier=0.6).clone())
        assert torch.equal(full, planned)


# what the plan and the kernel have to agree on: the tiles, and the order that a product walks them in
@pytest.mark.parametrize("knob,value,default", [("opb_set_tile_n", 128, 0), ("opb_set_tile_n", 64, 0),
                                                ("opb_set_cta_pair", 0, 1), ("opb_set_group_m", 3, 0),
                                                ("opb_set_group_m", 1, 0), ("opb_set_stage_k", 32, 64)])
@pytest.mark.parametrize("max_d", [0, 1 << 30])
def test_planned_squarings_under_the_tuning_knobs(cuda, knob, value, default, max_d):
    from oplib_b200 import _lib
    from oplib_b200.model import Lattice
    lib = _lib.load()
    lat = Lattice.local_vol(n=2304, device=cuda)
    assert lib.opb_set_fused_normalisation(max_d) == 0 and getattr(lib, knob)(value) == 0
    try:
        full, planned = _both(lambda: lat.solve(STRIKES, 2, 0.25, 2.0 ** -10, mode="bf16x3", all_states=True)[1])
    finally:
        getattr(lib, knob)(default)
        lib.opb_set_fused_normalisation(-1)
    assert torch.equal(full, planned)


@pytest.mark.parametrize("mode", ["bf16x3", "fp16x3"])
@pytest.mark.parametrize("max_d", [0, 1 << 30])
@pytest.mark.parametrize("n,banded", [(1536, True), (1600, False), (2048, True)])
def test_planned_squarings_of_a_dense_generator(cuda, n, banded, max_d, mode):
    """Given densely, a generator starts with every block marked; banded or not, the results are the full
    products'."""
    import ctypes as C
    from oplib_b200 import _lib
    from oplib_b200.model import MODES, Lattice, Plan, bind_stream
    lib = _lib.load()
    lat = Lattice.local_vol(n=n, device=cuda)
    L = torch.zeros(n, n, dtype=torch.float64, device=cuda)
    if banded:
        cols = lat.cols.view(n, 3).long()
        L.scatter_add_(1, cols.clamp(min=0), torch.where(cols >= 0, lat.vals.view(n, 3), 0.0))
    else:
        L = torch.rand(n, n, dtype=torch.float64, device=cuda, generator=torch.Generator(device=cuda).manual_seed(1))
        L -= torch.diag(L.sum(1))
    K = torch.as_tensor(STRIKES, device=cuda)
    desc = lat.desc(Plan(6, float(0.25 / L.diagonal().abs().max()), 0.0), 0.25, 2, K)
    desc.ell_width, desc.gen_cols, desc.gen_vals, desc.gen_dense = 0, None, None, L.data_ptr()
    ws = lat.workspace(len(STRIKES), MODES[mode])

    def run():
        V = torch.empty(2, n, len(STRIKES), dtype=torch.float64, device=cuda)
        q = torch.empty(2, len(STRIKES), dtype=torch.float64, device=cuda)
        bind_stream(cuda)
        assert lib.opb_lattice_solve(C.byref(desc), MODES[mode], ws.data_ptr(), ws.numel(), q.data_ptr(),
                                     V.data_ptr()) == 0
        return V

    assert lib.opb_set_fused_normalisation(max_d) == 0
    try:
        full, planned = _both(run)
    finally:
        lib.opb_set_fused_normalisation(-1)
    assert torch.equal(full, planned)


def _spoiled(lat, how, dt):
    """The lattice with one node's rates far from the quoted state spoiled, and its band as wide as the
    matrix (an entry of rate zero in the far corner), so that band skipping leaves nothing out."""
    from oplib_b200.model import Lattice
    n, w = lat.d, lat.width
    cols, vals = lat.cols.view(n, w), lat.vals.view(n, w).clone()
    cols = torch.cat([cols, torch.full((n, 1), -1, dtype=cols.dtype, device=cols.device)], 1)
    vals = torch.cat([vals, torch.zeros(n, 1, dtype=vals.dtype, device=vals.device)], 1)
    cols[0, w] = n - 1
    row = n - 9
    if how == "grows":  # BF16 parts hold it, but not its square
        vals[row] *= 1e18 / (vals[row].abs().max() * dt)
    elif how == "huge":  # finite, but not in FP16 parts, and not once squared
        vals[row] *= 1e33
    else:
        vals[row, 1] = float(how)
    return Lattice(n, cols.reshape(-1).contiguous(), vals.reshape(-1).contiguous(), lat.x, lat.y0, lat.rate)


@pytest.mark.parametrize("mode", ["bf16x3", "fp16x3"])
@pytest.mark.parametrize("max_d", [0, 1 << 30])
@pytest.mark.parametrize("n,how,niter", [(1600, "nan", 4), (2048, "nan", 3), (1600, "inf", 3), (2048, "huge", 3),
                                         (2048, "grows", 3)])
def test_values_that_are_not_finite_spread_as_in_the_full_products(cuda, n, how, niter, max_d, mode):
    """A zero block has products that are not zero where the other operand is NaN or infinite: from the
    level on at which such a value appears nothing is left out."""
    from oplib_b200 import _lib
    from oplib_b200.model import Lattice, Plan
    lib = _lib.load()
    clean = Lattice.local_vol(n=n, device=cuda)
    plan = Plan(niter, clean.plan(0.25, 2.0 ** -12).dt, 0.0)
    lat = _spoiled(clean, how, plan.dt)
    assert lib.opb_set_fused_normalisation(max_d) == 0
    try:
        full, planned = _both(lambda: lat.solve(STRIKES, 2, 0.01, 0.0, mode=mode, plan=plan, all_states=True)[1])
        quotes, _ = lat.solve(STRIKES, 2, 0.01, 0.0, mode=mode, plan=plan)
    finally:
        lib.opb_set_fused_normalisation(-1)
    assert how == "grows" or not torch.isfinite(full).all()
    torch.testing.assert_close(planned, full, rtol=0, atol=0, equal_nan=True)
    if how == "nan":  # (every state reaches the spoiled one)
        assert torch.isnan(quotes).all()


def test_a_lattice_that_is_not_finite_leaves_the_others_of_a_batch(cuda):
    from oplib_b200.model import Batch, Lattice
    lats = [Lattice.local_vol(n=n, level=0.12 + 0.03 * i, device=cuda) for i, n in enumerate([1152, 700, 256])]
    bt = Batch(lats, STRIKES, 3, 0.25, 2.0 ** -14, autotune=False)
    clean = bt.execute().clone()
    at = lats[0].vals.numel() + 3 * 690 + 1  # the second lattice's node 690
    was = bt.vals[at].clone()
    bt.vals[at] = float("nan")
    for cfg in range(8):
        bt.set_config(cfg)
        got = bt.execute().clone()
        assert torch.isnan(got[1]).all()
        assert torch.equal(got[0], clean[0]) and torch.equal(got[2], clean[2])
    bt.vals[at] = was
    assert torch.equal(bt.execute(), clean)


def test_autotune_runs_every_tile_form_as_often_as_asked(cuda):
    """One run decides nothing: each of the four tile forms is timed reps times over its squarings."""
    import ctypes as C
    from torch.profiler import ProfilerActivity, profile
    from oplib_b200 import _lib
    from oplib_b200.model import Batch, Lattice, bind_stream
    lib = _lib.load()
    lats = [Lattice.local_vol(n=n, device=cuda) for n in (256, 384)]
    bt = Batch(lats, STRIKES, 2, 0.25, 2.0 ** -10, autotune=False)
    levels = max(p.niter for p in bt.plans)
    ms, best, plans = (C.c_float * 8)(), C.c_int(), []
    bind_stream(cuda)
    for reps in (1, 3):
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            assert lib.opb_batch_autotune(bt.plan, reps, ms, C.byref(best)) == 0
            torch.cuda.synchronize()
        plans.append(sum("k_tile_plan" in e.name for e in prof.events()))
        recorded = bool(prof.events())
        assert ms[best.value] == min(ms) and 0 < min(ms) and max(ms) < 1e3
    if not recorded:
        pytest.skip("the profiler recorded no kernels")
    assert plans[1] - plans[0] == 2 * 4 * levels
