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
