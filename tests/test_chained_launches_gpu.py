"""Chained launches (launch.cuh): a kernel may be launched before the one it
reads from has finished, so a missing wait would show as a result that depends
on timing.  Every kind of chain -- stage kernels alone, with the diffusive and
hyperdiffusion passes, on the cubed shell and on grid arrays, HEVI steps --
has to give bit for bit the same state whether its steps are issued back to
back, beside a second model whose kernels fill the GPU, or one at a time with
the device drained in between; on the legacy stream (plain launches) and on a
stream of its own (a captured graph)."""
import pytest

torch = pytest.importorskip("torch")


def _models(kind):
    import cmdg
    from cmdg import workloads

    if kind in ("brick", "brick_fp64", "column"):
        ne = (1, 1, 1) if kind == "column" else (7, 6, 5)
        dg = workloads.bubble_model(ne=ne, N=4, precision="fp64" if kind == "brick_fp64" else "mixed")
        return dg, workloads.rising_bubble(dg.grid.coordinates()), 0.05
    if kind == "les":
        L = (500.0, 400.0, 300.0)
        dg = workloads.les_model(ne=(5, 4, 3), L=L, precision="mixed")
        return dg, workloads.les_initial_state(dg.grid.coordinates(), L, nmodes=4), 0.01
    if kind == "hyper":
        dg = workloads.hyper_bubble_model(ne=(5, 4, 3), N=3, precision="mixed")
        return dg, workloads.rising_bubble(dg.grid.coordinates()), 0.05
    if kind == "arrays":
        dg, _perm, xyz = workloads.bubble_arrays_model(ne=(5, 4, 3), N=3, precision="mixed")
        return dg, workloads.rising_bubble(xyz), 0.05
    if kind == "shell_hyper":
        dg = workloads.gcm_shell_model(nhorz=3, nvert=2, N=3, precision="mixed", tau_hyper=28800.0)
        return dg, workloads.gcm_initial_state(dg.grid.coordinates()), 2.0
    dg = workloads.acoustic_wave_model(nhorz=2, nvert=3, N=4, precision="mixed")
    p_ref = dg.reference_state()[:, 2]
    return dg, workloads.acoustic_wave_state(dg.grid.coordinates(), p_ref), 20.0


def _stepper(dg, Q, dt, kind):
    import cmdg

    if kind == "hevi":
        lin = cmdg.DGModel(cmdg.AtmosAcousticGravityLinearModel(dg.balance_law), dg.grid, direction="vertical",
                           state_auxiliary=dg)
        return cmdg.ARK2GiraldoKellyConstantinescu(
            dg, lin, cmdg.LinearBackwardEulerSolver(cmdg.ManyColumnLU()), Q, dt=dt)
    return cmdg.LSRK54CarpenterKennedy(dg, Q, dt=dt)


@pytest.mark.gpu
@pytest.mark.parametrize("own_stream", [False, True])
@pytest.mark.parametrize("kind", ["brick", "brick_fp64", "column", "les", "hyper", "arrays", "shell_hyper", "hevi"])
def test_back_to_back_steps_equal_drained_steps(kind, own_stream):
    import cmdg
    from cmdg import workloads

    dg, Q0, dt = _models(kind)
    other = workloads.bubble_model(ne=(12, 12, 12), N=4, precision="mixed")
    Qo = other.init_ode_state(workloads.rising_bubble(other.grid.coordinates()))
    lo = cmdg.LSRK54CarpenterKennedy(other, Qo, dt=0.02)

    def state():
        return torch.from_numpy(Q0).cuda() if kind == "hevi" else dg.init_ode_state(Q0)

    steps, results = 6, []
    stream = torch.cuda.Stream() if own_stream else torch.cuda.default_stream()
    for mode in ("drained", "back_to_back", "beside"):
        Q = state()
        solver = _stepper(dg, Q, dt, kind)
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            for _ in range(steps):
                if mode == "beside":
                    cmdg.dostep_(Qo, lo, None, 0.0)
                cmdg.dostep_(Q, solver, None, 0.0)
                if mode == "drained":
                    torch.cuda.synchronize()
        torch.cuda.synchronize()
        results.append(Q.clone())
    assert torch.isfinite(results[0]).all()
    assert torch.equal(results[0], results[1])
    assert torch.equal(results[0], results[2])
