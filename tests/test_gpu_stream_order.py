"""Launches of one default handle of the l2-slot regime that keeps no slots
(N = 61..110), issued on two streams back to back into the same outputs: they
do not overlap, so the outputs are the last launch's, bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [62, 72, 108])
def test_last_launch_wins(cuda, n):
    import torch
    from sunny_gen_eigensolver_b200 import Solver
    from sunny_gen_eigensolver_b200.generators import baseline_problems_torch
    batch = 600
    data = []
    for seed in (1, 2):
        H, S = baseline_problems_torch(n, 50, seed=seed, device="cuda")
        data.append(tuple(x.transpose(-1, -2).contiguous().repeat(batch // 50, 1, 1) for x in (H, S)))
    W = torch.empty((batch, n), dtype=torch.float64, device="cuda")
    U = torch.empty((batch, n, n), dtype=torch.complex128, device="cuda")
    info = torch.empty((batch,), dtype=torch.int32, device="cuda")
    with Solver(n) as s:
        assert s.regime == "l2-slot"
        ref = [s.run_kernel(*d) for d in data]
        torch.cuda.synchronize()
        s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
        for _ in range(3):
            for first, second in ((0, 1), (1, 0)):
                s.launch(*data[first], W, U, info, s1)
                s.launch(*data[second], W, U, info, s2)
                torch.cuda.synchronize()
                assert torch.equal(W, ref[second][0]) and torch.equal(U, ref[second][1]) and torch.equal(info, ref[second][2])
