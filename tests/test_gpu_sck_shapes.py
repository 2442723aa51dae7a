"""Cumulative rows and guide tables at the widths where their tiles end, against numpy."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def rows_for(d, nrows, cuda, seed=3):
    from oplib_b200.model import cumulative_rows
    rng = np.random.default_rng(seed)
    P = (rng.random((nrows, d)) ** 8).astype(np.float32)
    P[rng.random((nrows, d)) < 0.3] = 0
    P[0, : d // 2] -= 0.01  # residues below zero count as zero
    dP = torch.from_numpy(P).to(cuda)
    return P, cumulative_rows(dP)


@pytest.mark.parametrize("d,nrows", [(1, 1), (3, 5), (128, 4), (513, 7), (1023, 2), (1024, 9), (1025, 6), (2051, 3)])
def test_cumulative_rows_and_guide_at_the_edges(cuda, d, nrows):
    from oplib_b200.model import guide_table
    P, C = rows_for(d, nrows, cuda)
    p = np.where(P > 0, P, np.float32(0))
    acc = np.cumsum(p, axis=1, dtype=np.float32)  # sequential FP32 sums
    with np.errstate(invalid="ignore"):
        want = acc / acc[:, -1:]
    want = np.where(want < 1, want, np.float32(1))
    got = C.cpu().numpy()
    assert np.array_equal(got, want)
    for nb in (1, 64, 1024):
        g = guide_table(C, nb).cpu().numpy().view(np.uint32)
        for r in range(nrows):
            lo = np.searchsorted(got[r], np.arange(nb) / nb, side="right").clip(max=d - 1)
            hi = np.searchsorted(got[r], np.arange(1, nb + 1) / nb, side="left").clip(max=d - 1)
            hi[-1] = d - 1
            assert np.array_equal(g[r] & 0xffff, lo) and np.array_equal(g[r] >> 16, np.maximum(lo, hi))


def test_guide_of_a_row_longer_than_the_staged_one(cuda):
    from oplib_b200.model import guide_table
    d = 12 * 1024 + 5
    _, C = rows_for(d, 2, cuda)
    got = C.cpu().numpy()
    g = guide_table(C, 256).cpu().numpy().view(np.uint32)
    for r in range(2):
        lo = np.searchsorted(got[r], np.arange(256) / 256, side="right").clip(max=d - 1)
        hi = np.searchsorted(got[r], np.arange(1, 257) / 256, side="left").clip(max=d - 1)
        hi[-1] = d - 1
        assert np.array_equal(g[r] & 0xffff, lo) and np.array_equal(g[r] >> 16, np.maximum(lo, hi))


# blocks of 32 rows, their last one short; the widest row they take and one past it; in place
@pytest.mark.parametrize("d,nrows,kernel", [(1, 33, "k_sck_short"), (2, 64, "k_sck_short"), (16, 5000, "k_sck_short"),
                                            (100, 31, "k_sck_short"), (127, 65, "k_sck_short"),
                                            (128, 32, "k_sck_short"), (129, 33, "k_sck_rm")])
def test_short_rows(cuda, d, nrows, kernel):
    from torch.profiler import ProfilerActivity, profile
    from oplib_b200 import _lib
    from oplib_b200.model import bind_stream
    P, C = rows_for(d, nrows, cuda)
    acc = np.cumsum(np.where(P > 0, P, np.float32(0)), axis=1, dtype=np.float32)  # sequential FP32 sums
    with np.errstate(invalid="ignore"):
        want = acc / acc[:, -1:]
    want = np.where(want < 1, want, np.float32(1))
    assert np.array_equal(C.cpu().numpy(), want)
    same = torch.from_numpy(P).to(cuda)
    bind_stream(cuda)
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        assert _lib.load().opb_sck_rm(d, nrows, same.data_ptr(), same.data_ptr()) == 0
        torch.cuda.synchronize()
    assert torch.equal(same, C)
    if not prof.events():
        pytest.skip("the profiler recorded no kernels")
    ran = [e.name for e in prof.events() if "k_sck" in e.name]
    assert len(ran) == 1 and kernel in ran[0]


# tables of many rows: a warp, two, four or eight a row, searched in place or staged; and one of few
@pytest.mark.parametrize("d,nrows,nb,blocks", [(5, 8195, 8, 1025), (64, 2049, 64, 513), (100, 2050, 256, 1025),
                                               (512, 2048, 4096, 2048), (1000, 2060, 128, 1030),
                                               (2100, 2051, 4, 257), (64, 2047, 64, 2047)])
def test_guides_of_many_rows(cuda, tmp_path, d, nrows, nb, blocks):
    import json
    from torch.profiler import ProfilerActivity, profile
    from oplib_b200.model import guide_table
    _, C = rows_for(d, nrows, cuda)
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        g = guide_table(C, nb)
        torch.cuda.synchronize()
    g, got = g.cpu().numpy().view(np.uint32), C.cpu().numpy()
    for r in list(range(0, nrows, 97)) + [nrows - 2, nrows - 1]:
        lo = np.searchsorted(got[r], np.arange(nb) / nb, side="right").clip(max=d - 1)
        hi = np.searchsorted(got[r], np.arange(1, nb + 1) / nb, side="left").clip(max=d - 1)
        hi[-1] = d - 1
        assert np.array_equal(g[r] & 0xffff, lo) and np.array_equal(g[r] >> 16, np.maximum(lo, hi))
    if not prof.events():
        pytest.skip("the profiler recorded no kernels")
    prof.export_chrome_trace(str(tmp_path / "trace.json"))
    events = json.loads((tmp_path / "trace.json").read_text())["traceEvents"]
    grids = [e["args"]["grid"][0] for e in events if e.get("cat") == "kernel" and "k_guide" in e["name"]]
    assert grids == [blocks]
