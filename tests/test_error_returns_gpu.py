"""A solve that returns an error has nothing in flight: its buffers are free for
the next one, on whatever stream."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import workloads


@pytest.mark.gpu
@pytest.mark.parametrize("learned", [False, True])
def test_lists_too_large_returns_idle(gpu_lib, learned):
    """A correction radius beyond the whole set makes every leaf a correction
    entry of every other: more than 2^31 - 1 entries, refused once they are
    counted.  The stream is idle on return, and a solve on another stream right
    after gives what it gives alone."""
    torch = pytest.importorskip("torch")
    P = gpu_lib
    dev = torch.device("cuda:0")
    put = lambda b: [torch.from_numpy(np.ascontiguousarray(a)).to(dev) for a in (b.xy, b.cir, b.cor)]  # noqa: E731
    ptr = lambda d: [t.data_ptr() for t in d]  # noqa: E731
    b = workloads().uniform(100_000, seed=31)
    big, small = put(b), put(workloads().lamb_oseen(100_000, seed=32))
    out, alone, after = (torch.empty_like(big[0]) for _ in range(3))
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    P.set_params(11, 33, 0.5)
    P.set_mode(P.MODE_LEARNED if learned else P.MODE_MIXED)
    P.set_mixed_leaf()
    P.set_mixed_params()
    try:
        for _ in range(2):  # the second one with its near-field variant chosen
            P.solve_device(*ptr(small), alone.data_ptr(), 100_000, s2.cuda_stream)
        torch.cuda.synchronize()
        for _ in range(3):
            P.set_mixed_leaf(1)
            P.set_mixed_params(16, 1e6)
            with pytest.raises(P.Tree2DError) as e:
                P.solve_device(*ptr(big), out.data_ptr(), 100_000, s1.cuda_stream)
            assert s1.query()
            assert e.value.code == P.ERR_TOO_LARGE
            P.set_mixed_leaf()
            P.set_mixed_params()
            P.solve_device(*ptr(small), after.data_ptr(), 100_000, s2.cuda_stream)
            torch.cuda.synchronize()
            assert torch.equal(after.view(torch.int64), alone.view(torch.int64))
    finally:
        P.set_mixed_leaf()
        P.set_mixed_params()
        P.clear_params()
        P.set_mode(P.MODE_PLAIN)
