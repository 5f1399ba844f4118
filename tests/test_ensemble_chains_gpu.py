"""Ensembles step large members one by one with the one-model kernel and small
ones in sets: on both sides of the 64,000-node line, alone and mixed, every
member has to step as it does by itself (the same terms in FP32, at most a
different rounding of some sums: relative L2 1e-6 of the step's change, as
between the two kernel families)."""
import pytest

torch = pytest.importorskip("torch")

LARGE4, LARGE5, AT, BELOW, SMALL = (9, 8, 8, 4), (7, 7, 8, 5), (8, 8, 8, 4), (8, 8, 7, 4), (3, 4, 5, 3)


@pytest.mark.gpu
@pytest.mark.parametrize("specs", [[AT], [BELOW], [AT, BELOW], [SMALL, LARGE5, SMALL, AT, LARGE4, BELOW, SMALL]])
@pytest.mark.parametrize("own_stream", [False, True])
def test_members_step_as_by_themselves(specs, own_stream):
    import cmdg
    from cmdg import workloads

    members = [workloads.bubble_model(ne=s[:3], N=s[3], precision="mixed") for s in specs]
    Q0 = [dg.init_ode_state(workloads.rising_bubble(dg.grid.coordinates())) for dg in members]
    dts = [0.01 + 0.002 * m for m in range(len(specs))]
    Qs = [q.clone() for q in Q0]
    regs = [torch.zeros(q.shape, dtype=torch.float64, device=q.device) for q in Qs]
    ens = cmdg.Ensemble(members)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream() if own_stream else torch.cuda.default_stream()):
        ens.lsrk54_step(Qs, regs, dts)
        ens.lsrk54_step(Qs, regs, dts, nsteps=2)
    torch.cuda.synchronize()
    for dg, q0, q, dt in zip(members, Q0, Qs, dts):
        ref = q0.clone()
        solver = cmdg.LSRK54CarpenterKennedy(dg, ref, dt=dt)
        for _ in range(3):
            cmdg.dostep_(ref, solver, None, 0.0)
        change = (ref.double() - q0.double()).norm()
        scale = torch.maximum(change, 1e-1 * ref.double().norm())  # FP32 states: rounding is relative to the state
        assert float((q.double() - ref.double()).norm() / scale) < 1e-6
