"""Calls of an ensemble on a stream of its own, with time steps and numbers of
steps that change from call to call: the launch parameters of a call may not
reach the GPU while the steps before still read theirs.  The states equal the
default stream's bit for bit."""
import pytest

torch = pytest.importorskip("torch")


def _ensemble(specs):
    import cmdg
    from cmdg import workloads

    members = [workloads.bubble_model(ne=s[:3], N=s[3], precision="mixed") for s in specs]
    Qs = [dg.init_ode_state(workloads.rising_bubble(dg.grid.coordinates())) for dg in members]
    regs = [torch.zeros(q.shape, dtype=torch.float64, device=q.device) for q in Qs]
    return cmdg.Ensemble(members), Qs, regs


@pytest.mark.gpu
def test_changing_and_repeated_calls_give_the_default_streams_states():
    specs = [(3, 4, 5, 3), (8, 8, 8, 4), (2, 3, 2, 5)]
    calls = [(1e-2, 1), (1e-2, 1), (1e-2, 1), (2e-2, 1), (1e-2, 2), (1e-2, 2), (1e-2, 2), (1e-2, 1), (3e-2, 2), (3e-2, 1)]
    out = []
    for stream in (torch.cuda.default_stream(), torch.cuda.Stream()):
        ens, Qs, regs = _ensemble(specs)
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            for dt, nsteps in calls:
                ens.lsrk54_step(Qs, regs, [dt] * len(specs), nsteps=nsteps)
        torch.cuda.synchronize()
        out.append([q.clone() for q in Qs])
    for a, b in zip(*out):
        assert torch.isfinite(a).all() and torch.equal(a, b)
