"""Calls of an ensemble on a stream of its own, with time steps and numbers of
steps that change from call to call.  The launch parameters of a call may not
reach the GPU while the steps before still read theirs: the states equal the
default stream's bit for bit.  Repeated calls replay a captured graph, calls
that change something launch directly: a dt that changes on every call (an
adaptive step) may not cost the capture of a graph that is used once."""
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


@pytest.mark.gpu
def test_a_changing_dt_costs_no_capture():
    """24 members of 64,000 nodes: a step is 120 launches.  Issued directly they
    take at most 2.5 us each and the upload of their parameters some 30 us, in
    all below 1.6 times the replayed graph's 240 us; capture and instantiation
    of the 120 nodes come to more than that step again."""
    specs = [(8, 8, 8, 4)] * 24
    ens, Qs, regs = _ensemble(specs)
    times = {}
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        for changing in (False, True):
            best = float("inf")
            for block in range(6):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                for k in range(20):
                    ens.lsrk54_step(Qs, regs, [1e-3 * (1 + 1e-3 * (k if changing else 0))] * len(specs))
                b.record()
                torch.cuda.synchronize()
                best = min(best, a.elapsed_time(b) / 20)
            times[changing] = best
    assert times[True] <= 1.6 * times[False], times
