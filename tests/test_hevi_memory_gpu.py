"""The column LU's set-up on a nearly full GPU: the factors have to fit, the band
they are computed in not.  With room for the band (1.53 GB here), the stage
buffers (181 MB) and 350 MB more, where band and factors (0.82 GB) together do
not fit, the solver is made in parts of the lines, and solves bit for bit as
the one made at once."""
import pytest

torch = pytest.importorskip("torch")

NHORZ, NVERT, N = 10, 5, 5


def _solver(dg, lin, Q):
    import cmdg

    return cmdg.ARK2GiraldoKellyConstantinescu(dg, lin, cmdg.LinearBackwardEulerSolver(cmdg.ManyColumnLU()), Q, dt=20.0)


@pytest.mark.gpu
def test_setup_in_parts_of_the_lines():
    import cmdg
    from cmdg import workloads

    dg = workloads.acoustic_wave_model(nhorz=NHORZ, nvert=NVERT, N=N)
    Q0 = workloads.acoustic_wave_state(dg.grid.coordinates(), dg.reference_state()[:, 2])
    Q0 += 1e-3 * torch.rand(Q0.shape, dtype=torch.float64, generator=torch.Generator().manual_seed(3)).numpy()
    Q = torch.from_numpy(Q0).cuda()
    lin = cmdg.DGModel(cmdg.AtmosAcousticGravityLinearModel(dg.balance_law), dg.grid, direction="vertical",
                       state_auxiliary=dg)
    ark = _solver(dg, lin, Q)
    want = ark.backward_euler_solve(torch.zeros_like(Q), Q).clone()
    del ark
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    n, bw, nline = 5 * (N + 1) * NVERT, 5 * (N + 1) - 1, 6 * NHORZ ** 2 * (N + 1) ** 2
    band, buffers = 8 * (2 * bw + 1) * n * nline, 7 * Q.numel() * 8
    free, _total = torch.cuda.mem_get_info()
    ballast = torch.empty(free - band - buffers - (350 << 20), dtype=torch.uint8, device="cuda")
    try:
        got = torch.zeros_like(Q)
        _solver(dg, lin, Q).backward_euler_solve(got, Q)
        torch.cuda.synchronize()
        assert torch.equal(got, want)
    finally:
        del ballast
        torch.cuda.empty_cache()
