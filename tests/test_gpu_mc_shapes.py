"""Monte Carlo at the path counts where the launch shape changes (64, 128, 256 threads a block, a
second path a thread) and at the run lengths where the generator's loops end, against the
oracle's paths."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def rows_for(d, nrows, cuda, seed=3):
    from oplib_b200.model import cumulative_rows
    rng = np.random.default_rng(seed)
    P = (rng.random((nrows, d)) ** 8).astype(np.float32)
    P[rng.random((nrows, d)) < 0.3] = 0
    P[0, : d // 2] -= 0.01  # residues below zero count as zero
    dP = torch.from_numpy(P).to(cuda)
    return P, cumulative_rows(dP)


@pytest.mark.parametrize("guided", [True, False])
@pytest.mark.parametrize("nsteps", [1, 226, 228, 453, 455, 623, 624, 625, 1019, 1021, 1300])
def test_run_lengths(cuda, nsteps, guided):
    from oplib_b200.model import guide_table, mc_run
    d, n = 96, 70
    _, C = rows_for(d, d, cuda)
    _, paths = mc_run(C, 40, nsteps, 77, n, guide=guide_table(C) if guided else None, want_paths=True)
    cum = C.cpu().numpy()
    want = np.asarray(O.mc_paths(cum, 40, 77, np.arange(n), nsteps)).T
    assert np.array_equal(paths.cpu().numpy().astype(np.int64), want)


@pytest.mark.parametrize("npaths", [1, 63, 65, 64 * 3552 + 1, 128 * 3552 + 1, 256 * 3552 + 300])
def test_path_counts(cuda, npaths):
    """The payoff sums from the states the same launch shape writes."""
    from oplib_b200.model import guide_table, mc_run
    d, steps = 64, 3
    _, C = rows_for(d, d, cuda)
    x = torch.linspace(0.5, 1.5, d, dtype=torch.float64, device=cuda)
    kw = dict(guide=guide_table(C), x=x, strike=1.0, barrier=0.62, disc=0.97)
    sums, paths = mc_run(C, 30, steps, 5, npaths, want_paths=True, **kw)
    only, _ = mc_run(C, 30, steps, 5, npaths, **kw)
    xv = x[paths.long()]
    bar = torch.where((xv.amin(0) > 0.62) & (xv[-1] > 1.0), 0.97 * (xv[-1] - 1.0), 0.0).sum()
    asi = (0.97 * (xv.mean(0) - 1.0).clamp(min=0)).sum()
    # sums of positive FP64 terms in another order, and the mean's three-term sum
    torch.testing.assert_close(sums, torch.stack([bar, asi]), rtol=1e-11, atol=1e-11)
    assert torch.equal(sums, only)
    first, few = mc_run(C, 30, steps, 5, min(npaths, 200), want_paths=True, **kw)
    assert torch.equal(paths[:, : few.shape[1]], few)  # a path does not depend on the shape


# path counts where a form with more resident blocks takes a wave less, and where it does not
@pytest.mark.parametrize("evaluator,nsteps,npaths,per_sm", [
    (False, 630, 1024 * 148, 4), (False, 630, 1024 * 148 + 1, 6), (False, 630, 262_144, 4), (False, 630, 400_000, 6),
    (True, 630, 1024 * 148 + 1, 6), (True, 5, 1536 * 148, 6), (True, 5, 1536 * 148 + 1, 8), (True, 5, 350_000, 6)])
def test_blocks_an_sm(cuda, evaluator, nsteps, npaths, per_sm):
    """The form that the measured rule names, and the sums of the same paths run in two halves."""
    from torch.profiler import ProfilerActivity, profile
    from oplib_b200 import _lib
    from oplib_b200.model import bind_stream, guide_table
    if torch.cuda.get_device_properties(cuda).multi_processor_count != 148:
        pytest.skip("path counts of 148 SMs")
    lib = _lib.load()
    d = 64
    _, C = rows_for(d, d, cuda)
    g = guide_table(C)
    bind_stream(cuda)
    x = torch.linspace(0.5, 1.5, d, dtype=torch.float64, device=cuda)
    cf = torch.rand(nsteps, d, dtype=torch.float64, device=cuda)
    scratch = torch.empty(2 * lib.opb_mc_scratch_blocks(npaths), dtype=torch.float64, device=cuda)

    def run(path0, n):
        sums = torch.empty(2, dtype=torch.float64, device=cuda)
        args = (C.data_ptr(), d, 1, g.data_ptr(), g.numel() // d, d, 30, nsteps, 5, path0, n, None)
        if evaluator:
            r = lib.opb_mc_mt19937_eval(*args, cf.data_ptr(), None, None, scratch.data_ptr(), sums.data_ptr())
        else:
            r = lib.opb_mc_mt19937(*args, x.data_ptr(), 1.0, 0.52, 0.97, scratch.data_ptr(), sums.data_ptr())
        assert r == 0
        return sums
    halves = run(0, npaths // 2) + run(npaths // 2, npaths - npaths // 2)
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        whole = run(0, npaths)
        torch.cuda.synchronize()
    # sums of non-negative FP64 terms in another order
    torch.testing.assert_close(whole, halves, rtol=1e-11, atol=0)
    if not prof.events():
        pytest.skip("the profiler recorded no kernels")
    ran = [e.name for e in prof.events() if "k_mc<" in e.name]
    assert len(ran) == 1 and f", {per_sm}>" in ran[0]
