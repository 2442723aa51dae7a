"""The training step's fused passes at batches where their row blocks end: one row, short of a
16-row block, one past it, the tensor-core products' smallest batch, a remainder of their slices."""
import numpy as np
import pytest
import torch

from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 15, 17, 100, 128, 384])
def test_gradient_at_block_edges(cuda, B):
    from oplib_b200 import _lib
    from oplib_b200.model import bind_stream
    lib = _lib.load()
    bind_stream(cuda)
    n = lib.opb_mlp_param_count()
    theta = torch.empty(n, device=cuda)
    thb = torch.empty(n, device=cuda)
    assert lib.opb_mlp_init(theta.data_ptr(), 5) == 0
    L, _ = M.layout()
    rng = np.random.default_rng(B)
    for _, o, _, b in L:  # biases as training leaves them
        theta[b[0]:b[1]] = torch.from_numpy(rng.uniform(-0.1, 0.1, o).astype(np.float32)).to(cuda)
    assert lib.opb_mlp_round(theta.data_ptr(), thb.data_ptr(), None) == 0
    X = rng.uniform(-1, 1, (B, 8)).astype(np.float32)
    t = rng.normal(0, 0.5, B).astype(np.float32)
    dX, dt = torch.from_numpy(X).to(cuda), torch.from_numpy(t).to(cuda)
    ws = torch.full((int(lib.opb_mlp_workspace_floats(B)),), float("nan"), device=cuda)
    grad = torch.full((n,), float("nan"), device=cuda)
    loss = torch.zeros(1, dtype=torch.float64, device=cuda)
    assert lib.opb_mlp_loss_grad(thb.data_ptr(), dX.data_ptr(), dt.data_ptr(), B, ws.data_ptr(), grad.data_ptr(),
                                 loss.data_ptr()) == 0
    torch.cuda.synchronize()
    assert lib.opb_tc_error() == 0
    want_loss, want = M.loss_grad(thb.double().cpu().numpy(), X, t)
    want /= B
    # as the step's main test: FP32 accumulation and split products, against the largest entry
    assert abs(float(loss) - want_loss) <= 1e-4 * want_loss
    assert np.abs(grad.cpu().numpy() - want).max() <= 2e-4 * np.abs(want).max()
    # the same inputs give the same bits (every sum has a fixed order)
    again, loss2 = torch.empty_like(grad), torch.zeros_like(loss)
    assert lib.opb_mlp_loss_grad(thb.data_ptr(), dX.data_ptr(), dt.data_ptr(), B, ws.data_ptr(), again.data_ptr(),
                                 loss2.data_ptr()) == 0
    assert torch.equal(grad, again) and torch.equal(loss, loss2)


@pytest.mark.parametrize("off", [1, 2, 3])
@pytest.mark.parametrize("B", [100, 128])  # SIMT products, tensor-core products
def test_networks_at_any_float_address(cuda, B, off):
    """Working weights, inputs, targets and gradient off the 16-byte grid, as the rows of a [members]
    [parameters] array lie (199,937 floats each): the bits of the aligned run."""
    from oplib_b200 import _lib
    from oplib_b200.model import bind_stream
    lib = _lib.load()
    bind_stream(cuda)
    n = lib.opb_mlp_param_count()
    theta = torch.empty(n, device=cuda)
    thb = torch.empty(n, device=cuda)
    assert lib.opb_mlp_init(theta.data_ptr(), 9) == 0
    assert lib.opb_mlp_round(theta.data_ptr(), thb.data_ptr(), None) == 0
    gen = torch.Generator(device=cuda).manual_seed(off)
    thb += 0.01 * torch.randn(n, device=cuda, generator=gen)  # (biases are not zero)
    X = torch.rand(B, 8, device=cuda, generator=gen) * 2 - 1
    t = torch.randn(B, device=cuda, generator=gen)
    ws = torch.empty(int(lib.opb_mlp_workspace_floats(B)), device=cuda)

    def run(o):
        def at(v):
            buf = torch.full((v.numel() + o,), float("nan"), device=cuda)
            buf[o:] = v.reshape(-1)
            return buf[o:]
        w, x, tt, g, y = at(thb), at(X), at(t), at(torch.empty(n, device=cuda)), at(torch.empty(B, device=cuda))
        loss = torch.zeros(1, dtype=torch.float64, device=cuda)
        assert lib.opb_mlp_loss_grad(w.data_ptr(), x.data_ptr(), tt.data_ptr(), B, ws.data_ptr(), g.data_ptr(),
                                     loss.data_ptr()) == 0
        assert lib.opb_mlp_forward(w.data_ptr(), x.data_ptr(), B, ws.data_ptr(), y.data_ptr()) == 0
        torch.cuda.synchronize()
        return g.clone(), y.clone(), loss

    for got, want in zip(run(off), run(0)):
        assert torch.isfinite(want).all() and torch.equal(got, want)
