"""Launches that are set up while the kernel before them runs: chains of solves on two streams, from
two host threads, give the bits of the same solves one after the other."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

STRIKES = np.linspace(0.6, 1.4, 9)


@pytest.mark.parametrize("n,all_states", [(128, False), (512, False), (1000, True), (1664, False)])
def test_two_streams_of_chained_launches(cuda, n, all_states):
    from oplib_b200 import _lib
    from oplib_b200.model import Lattice
    lib = _lib.load()
    lats = [Lattice.local_vol(n=n, level=0.2 + 0.05 * i, device=cuda) for i in range(2)]

    def solve(lat):
        return lat.solve(STRIKES, 4, 0.25, 2.0 ** -12, mode="bf16x3", all_states=all_states)

    want = [solve(lat) for lat in lats]
    torch.cuda.synchronize()
    got, errors = [[], []], []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream(cuda)):
                for _ in range(12):
                    got[i].append(solve(lats[i]))
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and lib.opb_tc_error() == 0
    for i in range(2):
        for q, V in got[i]:
            assert torch.equal(q, want[i][0])
            assert not all_states or torch.equal(V, want[i][1])
