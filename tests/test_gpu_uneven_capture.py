"""An uneven-size handle in the middle of a stream capture: captured launches and
normal launches on another stream alternate while the capture lasts, and the
replayed graph and the normal launches give the per-size results bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


def test_normal_launches_while_a_capture_lasts(cuda):
    import torch
    from sunny_gen_eigensolver_b200 import Solver, UnevenSolver
    from sunny_gen_eigensolver_b200.generators import baseline_problems_torch
    sizes, batch = [12, 54, 72, 108, 130, 202], 6
    H, S, ref, out = {}, {}, {}, [{}, {}]
    for n in sizes:
        h, s = baseline_problems_torch(n, batch, seed=n, device="cuda")
        H[n], S[n] = h.transpose(-1, -2).contiguous(), s.transpose(-1, -2).contiguous()
        with Solver(n) as one:
            ref[n] = one.run_kernel(H[n], S[n])
        for o in out:
            o[n] = tuple(torch.full_like(x, -7) for x in ref[n])
    W, U, info = ([{n: o[n][k] for n in sizes} for o in out] for k in range(3))
    torch.cuda.synchronize()

    def check(o):
        torch.cuda.synchronize()
        for n in sizes:
            for got, want in zip(o[n], ref[n]):
                assert torch.equal(got, want)
                got.fill_(-7)

    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    with UnevenSolver(sizes) as us:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s1, capture_error_mode="relaxed"):
            us.launch(H, S, W[0], U[0], info[0], s1)
            us.launch(H, S, W[1], U[1], info[1], s2)
            us.launch(H, S, W[0], U[0], info[0], s1)
            us.launch(H, S, W[1], U[1], info[1], s2)
        check(out[1])
        for _ in range(2):
            g.replay()
            check(out[0])
        us.launch(H, S, W[1], U[1], info[1], s1)
        check(out[1])
        del g
