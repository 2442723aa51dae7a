"""The quoted row of the chained kernels (solves without all-state values) against the full
chain products, which the same solve runs when it returns every state's value: the row kernel
issues the same products in the same order, so only the order of the FP64 row sums differs
(1e-16 relative; a flipped FP32 rounding moves a quote by under 1e-9)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

STRIKES = np.linspace(0.6, 1.4, 9)


@pytest.mark.parametrize("mode", ["bf16x3", "fp16x3"])
@pytest.mark.parametrize("max_d", [0, 1 << 30])  # normalisation by the kernel, in the epilogues
@pytest.mark.parametrize("n,nmat", [(128, 1), (128, 131), (200, 2), (384, 3), (1024, 4), (1100, 5)])
def test_quoted_row_matches_the_full_products(cuda, n, nmat, max_d, mode):
    from oplib_b200 import _lib
    from oplib_b200.model import Lattice
    lib = _lib.load()
    lat = Lattice.local_vol(n=n, device=cuda)
    assert lib.opb_set_fused_normalisation(max_d) == 0
    try:
        row, _ = lat.solve(STRIKES, nmat, 0.0625, 2.0 ** -12, mode=mode)
        full, V = lat.solve(STRIKES, nmat, 0.0625, 2.0 ** -12, mode=mode, all_states=True)
        torch.cuda.synchronize()
    finally:
        lib.opb_set_fused_normalisation(-1)
    assert lib.opb_tc_error() == 0
    assert torch.equal(full, V[:, lat.y0, :])
    torch.testing.assert_close(row, full, rtol=1e-9, atol=1e-12)


def test_batched_rows_against_fp64(cuda):
    """Sizes from one row tile to seventeen, off the grid too, more maturities than one priced
    group holds: every quote within the library's 1e-5 of the FP64 solve."""
    from oplib_b200 import _lib
    from oplib_b200.model import Batch, Lattice
    from oracle import oracle as O
    lib = _lib.load()
    sizes = [128, 256, 300, 640, 1088]
    nmat, period, dt0 = 130, 1 / 64, 2.0 ** -12
    lats = [Lattice.local_vol(n=n, level=0.15 + 0.02 * i, device=cuda) for i, n in enumerate(sizes)]
    got = Batch(lats, STRIKES, nmat, period, dt0, mode="fp16x3", autotune=False).execute().cpu().numpy()
    assert lib.opb_tc_error() == 0
    for i, (n, lat) in enumerate(zip(sizes, lats)):
        x = O.log_grid(n)
        L = O.lv_generator_fast(x, 0.03 * x, O.lv_sigma(x, level=0.15 + 0.02 * i) * x)
        V, _, _ = O.solve_lattice_fp64(L, x, STRIKES, 0.03, period, nmat, dt0)
        assert np.abs(got[i] - V[:, lat.y0, :]).max() < 1e-5


@pytest.mark.parametrize("n", [384, 640])
def test_batched_rows_with_several_items_a_block(cuda, n):
    """More items than blocks are resident: a block changes lattice (another row in its shared
    memory) and goes on in the ring; equal lattices give equal bits, whichever block had them."""
    from oplib_b200 import _lib
    from oplib_b200.model import Batch, Lattice
    lats = [Lattice.local_vol(n=n, level=0.2 + 0.1 * (i % 2), device=cuda) for i in range(130)]
    got = Batch(lats, STRIKES, 4, 0.125, 2.0 ** -11, mode="bf16x3", autotune=False).execute()
    torch.cuda.synchronize()
    assert _lib.load().opb_tc_error() == 0
    for k in range(2):
        assert torch.equal(got[k::2], got[k:k + 1].expand_as(got[k::2]))
        alone, _ = lats[k].solve(STRIKES, 4, 0.125, 2.0 ** -11, mode="bf16x3")
        assert (got[k] - alone).abs().max() < 1e-5
