"""The small-tile FP32 products against the large-tile ones: every kernel sums an output's products
in k order with fma, so the same product gives the same bits whichever runs it (a batch of copies
is large enough for the 128 x 128 tiles); and the grouped products in any order of their task table."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _product(lib, A, B, batch=1):
    M, K = A.shape
    N = B.shape[1]
    C = torch.full((batch, M, N), float("nan"), device=A.device)
    A, B = A.expand(batch, M, K).contiguous(), B.expand(batch, K, N).contiguous()
    assert lib.opb_sgemm_batched_rm(M, N, K, A.data_ptr(), M * K, B.data_ptr(), K * N, C.data_ptr(), M * N, batch) == 0
    torch.cuda.synchronize()
    return C


# the 64 x 32 tiles and the 64 x 64 ones (from 240 of them), whole and ragged, rows on and off the
# 16-byte grid, K of one step, of less and of a remainder
@pytest.mark.parametrize("M,N,K", [(128, 128, 16), (128, 256, 128), (256, 128, 64), (1024, 1024, 48), (33, 65, 19),
                                   (1, 64, 7), (100, 36, 20), (31, 129, 130), (1001, 1003, 33)])
def test_small_tiles_are_bit_identical_to_the_large_ones(cuda, M, N, K):
    from oplib_b200 import _lib
    from oplib_b200.model import bind_stream
    lib = _lib.load()
    bind_stream(cuda)
    g = torch.Generator(device=cuda).manual_seed(M + N + K)
    A = torch.randn(M, K, device=cuda, generator=g)
    B = torch.randn(K, N, device=cuda, generator=g)
    small = _product(lib, A, B)[0]
    if M % 128 == 0 and N % 128 == 0 or K % 4 or N % 4:  # a batch of these runs on the large tiles
        tiles = -(-M // 128) * -(-N // 128)
        large = _product(lib, A, B, batch=-(-150 // tiles))
        assert torch.equal(large, small.expand_as(large))
    # sequential FP32 sums: K roundings of terms of the products' size
    want = A.double() @ B.double()
    bound = (K + 1) * 2.0 ** -24 * (A.double().abs() @ B.double().abs())
    assert bool(((small.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("order", ["rows", "columns", "shuffled"])
@pytest.mark.parametrize("shapes", [[(64, 16, 16)], [(576, 576, 40), (70, 50, 33), (128, 16, 17), (3, 5, 1)]])
def test_grouped_products_in_any_order_of_the_table(cuda, shapes, order):
    from oplib_b200 import _lib
    from oplib_b200.model import bind_stream
    lib = _lib.load()
    bind_stream(cuda)
    g = torch.Generator(device=cuda).manual_seed(7)
    mats, tasks = [], []
    for i, (m, n, k) in enumerate(shapes):
        A = torch.randn(m, k, device=cuda, generator=g)
        B = torch.randn(k, n, device=cuda, generator=g)
        Ac, Bc = A.t().contiguous(), B.t().contiguous()
        C = torch.full((n, m), float("nan"), device=cuda)
        mats.append((A, B, Ac, Bc, C))
        grid = [(bx, by) for bx in range(-(-m // 64)) for by in range(-(-n // 16))]
        if order == "columns":
            grid = sorted(grid, key=lambda t: (t[1], t[0]))
        tasks += [(i, bx, by, m, n, k, Ac.data_ptr(), Bc.data_ptr(), C.data_ptr()) for bx, by in grid]
    if order == "shuffled":
        tasks = [tasks[j] for j in np.random.default_rng(1).permutation(len(tasks))]
    words = lib.opb_sgemm4_task_size() // 8
    rec = np.zeros((len(tasks), words), dtype=np.int64)
    for t, task in enumerate(tasks):
        rec[t, :3] = np.array(task[:6], dtype=np.int32).view(np.int64)
        rec[t, 3:6] = task[6:]
    drec = torch.from_numpy(rec.ravel()).to(cuda)
    ptrs = torch.tensor([drec.data_ptr() + 8 * words * t for t in range(len(tasks))], dtype=torch.int64, device=cuda)
    assert lib.opcuda_sgemm4(len(tasks), ptrs.data_ptr()) == 0
    for A, B, _, _, C in mats:
        assert torch.equal(C.t(), _product(lib, A, B)[0])


@pytest.mark.parametrize("count", [3, 15, 16, 75, 76, 149])  # tasks a block: 1 up to 444, 2 up to 2220, 4 beyond
def test_grouped_products_across_the_table_sizes(cuda, count):
    """Tables of 30 tasks a product (80 x 229 x 37), the last block of a table not full."""
    from oplib_b200 import _lib
    from oplib_b200.model import bind_stream
    lib = _lib.load()
    bind_stream(cuda)
    g = torch.Generator(device=cuda).manual_seed(count)
    m, n, k = 80, 229, 37
    A = torch.randn(count, m, k, device=cuda, generator=g)
    B = torch.randn(count, k, n, device=cuda, generator=g)
    Ac, Bc = A.transpose(1, 2).contiguous(), B.transpose(1, 2).contiguous()
    C = torch.full((count, n, m), float("nan"), device=cuda)
    words = lib.opb_sgemm4_task_size() // 8
    rec = np.zeros((count * 30 - 1, words), dtype=np.int64)  # without the last tile
    for t in range(len(rec)):
        i, bx, by = t // 30, t % 30 // 15, t % 15
        rec[t, :3] = np.array([i, bx, by, m, n, k], dtype=np.int32).view(np.int64)
        rec[t, 3:6] = Ac[i].data_ptr(), Bc[i].data_ptr(), C[i].data_ptr()
    drec = torch.from_numpy(rec.ravel()).to(cuda)
    ptrs = torch.arange(len(rec), dtype=torch.int64, device=cuda) * (8 * words) + drec.data_ptr()
    assert lib.opcuda_sgemm4(len(rec), ptrs.data_ptr()) == 0
    got = C.transpose(1, 2)
    want = torch.stack([_product(lib, A[i], B[i])[0] for i in range(count)])
    want[-1, 64:, 14 * 16:] = float("nan")
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(got.nan_to_num(), want.nan_to_num())


# one 128 x 128 tile an SM, and a second on some; rows on the grid, bases and rows off it
@pytest.mark.parametrize("M,K,off_a,off_b,kernel", [
    (1536, 32, 0, 0, "k_sgemm_pipe"), (1536, 32, 1, 0, "k_sgemm_small"), (1536, 32, 0, 1, "k_sgemm_rm"),
    (1536, 32, 3, 2, "k_sgemm_rm"), (1664, 32, 1, 1, "k_sgemm_small"), (1500, 36, 1, 0, "k_sgemm_rm"),
    (1501, 33, 0, 0, "k_sgemm_rm"), (1001, 33, 0, 0, "k_sgemm_small")])
def test_products_off_the_16_byte_grid(cuda, M, K, off_a, off_b, kernel):
    """The kernel that the measured rule names, and the bits of the product at aligned bases."""
    from torch.profiler import ProfilerActivity, profile
    from oplib_b200 import _lib
    from oplib_b200.model import bind_stream
    lib = _lib.load()
    bind_stream(cuda)
    g = torch.Generator(device=cuda).manual_seed(5)
    A, B = torch.randn(M, K, device=cuda, generator=g), torch.randn(K, M, device=cuda, generator=g)
    want = _product(lib, A, B)[0]

    def at(v, o):
        buf = torch.empty(v.numel() + o, device=cuda)
        buf[o:] = v.reshape(-1)
        return buf[o:]
    a, b, C = at(A, off_a), at(B, off_b), torch.full((M, M), float("nan"), device=cuda)
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        assert lib.opb_sgemm_batched_rm(M, M, K, a.data_ptr(), 0, b.data_ptr(), 0, C.data_ptr(), 0, 1) == 0
        torch.cuda.synchronize()
    assert torch.equal(C, want)
    if not prof.events():
        pytest.skip("the profiler recorded no kernels")
    ran = [e.name for e in prof.events() if "k_sgemm" in e.name]
    assert len(ran) == 1 and kernel in ran[0]
