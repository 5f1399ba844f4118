"""Chained launches on meshes of fewer elements than SMs (launch.cuh): every CTA
has an SM of its own, so a step's time does not depend on the number of
elements, unless a kernel's CTAs were launched onto SMs that others still
held.  Two CTAs on one SM of an FP64-bound kernel take twice as long.  Bound:
a fifth more than the mesh of a quarter of the elements takes (the larger
one's memory traffic and the timer are below a tenth)."""
import pytest

torch = pytest.importorskip("torch")


def _step_us(dg, Q, dt):
    import cmdg

    lsrk = cmdg.LSRK54CarpenterKennedy(dg, Q, dt=dt)
    stream, best = torch.cuda.Stream(), float("inf")
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            cmdg.dostep_(Q, lsrk, None, 0.0, nsteps=10)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) * 100)
    return best


def _case(kind, big, N):
    from cmdg import workloads

    if kind == "les":
        L = (500.0, 400.0, 300.0)
        dg = workloads.les_model(ne=(6, 5, 4) if big else (3, 3, 3), N=N, L=L)
        return dg, workloads.les_initial_state(dg.grid.coordinates(), L, nmodes=2), 1e-3
    if kind == "hyper":
        dg = workloads.hyper_bubble_model(ne=(6, 5, 4) if big else (3, 3, 3), N=N)
        return dg, workloads.rising_bubble(dg.grid.coordinates()), 1e-3
    dg = workloads.gcm_shell_model(nhorz=3 if big else 2, nvert=2, N=N, tau_hyper=28800.0)
    return dg, workloads.gcm_initial_state(dg.grid.coordinates()), 1.0


@pytest.mark.gpu
@pytest.mark.parametrize("kind,N", [("les", 3), ("les", 5), ("hyper", 4), ("hyper", 5), ("shell_hyper", 4), ("shell_hyper", 5)])
def test_small_meshes_keep_one_cta_per_sm(kind, N):
    if torch.cuda.get_device_properties(0).multi_processor_count < 120:
        pytest.skip("needs an SM per element")
    small, big = (_step_us(dg, dg.init_ode_state(Q), dt) for dg, Q, dt in (_case(kind, b, N) for b in (False, True)))
    assert big <= 1.2 * small, (small, big)
