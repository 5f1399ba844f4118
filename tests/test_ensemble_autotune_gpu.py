"""The ensemble autotuner times what a step runs: sets of small members stage by
stage, large members by the one-model kernel, every chain's five stages before
the next chain's.

Tilings apply to sets, so an order whose members are all large keeps its
tiling and reports no candidates.  The per-order family's time is that of a
replayed step: within a fifth of a measured one (the timer, and a register
that is written where B dt = 0 rounds nothing away)."""
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
@pytest.mark.parametrize("own_stream", [False, True])
def test_orders_without_sets_keep_their_tiling(own_stream):
    specs = [(8, 8, 8, 4), (9, 8, 8, 4), (3, 4, 5, 3), (4, 3, 2, 3), (4, 4, 4, 5)]
    ens, Qs, regs = _ensemble(specs)
    before = [q.clone() for q in Qs]
    ens.set_tiling(7, 13)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream() if own_stream else torch.cuda.default_stream()):
        ms, choice = ens.autotune(Qs, regs, reps=2)
    torch.cuda.synchronize()
    assert choice[4] == (7, 13) and all(m == 0 for m in ms[4])
    for N in (3, 5):
        assert choice[N][0] in (1, 2, 4, 8, 16) and choice[N][1] in (-1, 0) and all(m > 0 for m in ms[N])
    assert ms["per_order"] > 0 and all(m > 0 for m in ms["persistent"])
    for q, b in zip(Qs, before):
        assert torch.equal(q, b)


@pytest.mark.gpu
def test_the_reported_time_is_a_steps():
    """12 members of 216,000 nodes: one chain's buffers (22 MB) stay in L2 from
    stage to stage, those of a stage of every member (260 MB) do not."""
    specs = [(12, 12, 12, 4)] * 12
    ens, Qs, regs = _ensemble(specs)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        ms, _ = ens.autotune(Qs, regs, reps=10)
        ens.set_kernel("per_order")
        best = float("inf")
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                ens.lsrk54_step(Qs, regs, [1e-3] * len(specs))
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) / 10)
    assert abs(5 * ms["per_order"] / best - 1) <= 0.2, (5 * ms["per_order"], best)
