"""Chained launches on the paths that test_chained_launches_gpu.py leaves out:
ensemble chains (members alone and in sets), closures on the cubed shell and on
grid arrays, and filters after steps.  A missing wait would show as a result
that depends on timing: the states have to be bit for bit the same whether the
steps are issued back to back, beside a second model whose kernels fill the
GPU, or with the device drained in between."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


def _closure_shell(turb, precision):
    import cmdg
    from cmdg import workloads

    R = 6.371e6
    model = cmdg.AtmosModel(orientation="sphere", gravity=True,
                            ref_state=cmdg.HydrostaticState(cmdg.IsothermalProfile(285.0)), turbulence=turb, rho_nu=10.0)
    dg = cmdg.DGModel(model, cmdg.CubedShellGrid(3, 3, 2, R, R + 30e3), precision=precision)
    # the closure's horizontal length makes its vertical diffusion stiff
    return dg, workloads.gcm_initial_state(dg.grid.coordinates()), 2.0 if turb == "constant" else 1e-3


def _closure_arrays(turb, precision):
    import cmdg
    from cmdg import workloads

    ne, N, L, per, bnd = (5, 4, 3), 3, 2500.0, (True, True, False), ((0, 0), (0, 0), (1, 2))
    inviscid, perm, xyz = workloads.bubble_arrays_model(ne=ne, N=N, L=L)
    aux7 = np.zeros((xyz.shape[0], 7, xyz.shape[2]))
    aux7[:, 0], aux7[:, 3] = 9.81 * xyz[:, 2], 9.81
    aux7[:, 4:7] = inviscid.reference_state()
    model = cmdg.AtmosModel(orientation="flat", gravity=True,
                            ref_state=cmdg.HydrostaticState(cmdg.DryAdiabaticProfile(300.0, 0.0)), turbulence=turb, rho_nu=2.0)
    vgeo, vmap, bndy, _perm = workloads.brick_grid_arrays(N, ne, (0.0,) * 3, (L,) * 3, per, bnd)
    dg = cmdg.DGModel(model, cmdg.ArraysGrid(N, vgeo, vmap, bndy), precision=precision)
    dg.set_reference(aux7)
    Q = workloads.rising_bubble(xyz)
    Q[:, 1:4] += np.random.default_rng(2).uniform(-1, 1, size=Q[:, 1:4].shape)
    return dg, Q, 0.02


def _passes(kind):
    """The states of a run and the function that issues one step of it."""
    import cmdg
    from cmdg import filters, workloads

    if kind == "ensemble":
        specs = [(8, 8, 8, 4), (3, 4, 5, 3), (2, 3, 2, 3), (9, 8, 8, 4), (4, 4, 4, 5)]
        members = [workloads.bubble_model(ne=s[:3], N=s[3], precision="mixed") for s in specs]
        Qs = [dg.init_ode_state(workloads.rising_bubble(dg.grid.coordinates())) for dg in members]
        regs = [torch.zeros(q.shape, dtype=torch.float64, device=q.device) for q in Qs]
        ens = cmdg.Ensemble(members)
        return Qs, lambda k: ens.lsrk54_step(Qs, regs, [0.02 + 0.01 * (k // 3)] * len(specs))
    if kind == "filtered":
        dg = workloads.bubble_model(ne=(7, 6, 5), N=4, precision="mixed")
        Q0, dt = workloads.rising_bubble(dg.grid.coordinates()), 0.05
    else:
        where, turb, precision = kind.split("_")
        dg, Q0, dt = (_closure_shell if where == "shell" else _closure_arrays)(turb, precision)
    Q = dg.init_ode_state(Q0)
    lsrk = cmdg.LSRK54CarpenterKennedy(dg, Q, dt=dt)
    filt = filters.ExponentialFilter(dg.grid, 0, 18) if kind == "filtered" else None

    def step(_k):
        cmdg.dostep_(Q, lsrk, None, 0.0)
        if filt is not None:
            filters.apply_(Q, None, dg, filt)

    return [Q], step


@pytest.mark.gpu
@pytest.mark.parametrize("own_stream", [False, True])
@pytest.mark.parametrize("kind", ["ensemble", "filtered", "shell_constant_mixed", "shell_smagorinsky_mixed",
                                  "shell_smagorinsky_fp64", "arrays_constant_mixed", "arrays_smagorinsky_fp64"])
def test_back_to_back_steps_equal_drained_steps(kind, own_stream):
    import cmdg
    from cmdg import workloads

    other = workloads.bubble_model(ne=(12, 12, 12), N=4, precision="mixed")
    Qo = other.init_ode_state(workloads.rising_bubble(other.grid.coordinates()))
    lo = cmdg.LSRK54CarpenterKennedy(other, Qo, dt=0.02)
    results = []
    for mode in ("drained", "back_to_back", "beside"):
        Qs, step = _passes(kind)
        start = [q.clone() for q in Qs]
        torch.cuda.synchronize()
        with torch.cuda.stream(torch.cuda.Stream() if own_stream else torch.cuda.default_stream()):
            for k in range(6):
                if mode == "beside":
                    cmdg.dostep_(Qo, lo, None, 0.0)
                step(k)
                if mode == "drained":
                    torch.cuda.synchronize()
        torch.cuda.synchronize()
        assert all(torch.isfinite(q).all() and not torch.equal(q, s) for q, s in zip(Qs, start))
        results.append([q.clone() for q in Qs])
    for r in results[1:]:
        assert all(torch.equal(a, b) for a, b in zip(results[0], r))
