"""Stage kernels walk the elements forward in the odd stages and backward in the
even ones; a tendency walks them forward.  A low-storage Runge-Kutta step built
from tendencies has to equal the fused step on meshes of one element, a prime
number of them and uneven boxes.  FP64: the two differ in the rounding of the
stage sums only, a few 1e-16 per stage and amplified by at most the step's
acoustic Courant number: 1e-13 of each field's acoustic scale (momentum: rho c)."""
import pytest

torch = pytest.importorskip("torch")

A = (0.0, -567301805773 / 1357537059087, -2404267990393 / 2016746695238, -3550918686646 / 2091501179385,
     -1275806237668 / 842570457699)
B = (1432997174477 / 9575080441755, 5161836677717 / 13612068292357, 1720146321549 / 2090206949498,
     3134564353537 / 4481467310338, 2277821191437 / 14882151754819)


def _case(kind, N):
    from cmdg import workloads

    if kind == "shell":
        dg = workloads.gcm_shell_model(nhorz=2, nvert=3, N=N, precision="fp64")
        return dg, workloads.gcm_initial_state(dg.grid.coordinates()), 1.0
    if kind == "arrays":
        dg, _perm, xyz = workloads.bubble_arrays_model(ne=(5, 3, 2), N=N, precision="fp64")
        return dg, workloads.rising_bubble(xyz), 0.02
    if kind == "les":
        L = (500.0, 400.0, 300.0)
        dg = workloads.les_model(ne=(5, 3, 2), N=N, L=L, precision="fp64")
        return dg, workloads.les_initial_state(dg.grid.coordinates(), L, nmodes=4), 0.01
    dg = workloads.bubble_model(ne=(1, 1, 1) if kind == "one" else (7, 1, 5), N=N, precision="fp64")
    return dg, workloads.rising_bubble(dg.grid.coordinates()), 0.02


@pytest.mark.gpu
@pytest.mark.parametrize("N", [2, 3, 4, 5])
@pytest.mark.parametrize("kind", ["one", "brick", "les", "arrays", "shell"])
def test_fused_step_equals_step_from_tendencies(kind, N):
    import cmdg

    dg, Q0, dt = _case(kind, N)
    Q = dg.init_ode_state(Q0)
    ref, reg, T = Q.clone(), torch.zeros_like(Q), torch.zeros_like(Q)
    for a, b in zip(A, B):
        dg(T, ref, None, 0.0)
        reg = T + a * reg
        ref = ref + b * dt * reg
    cmdg.dostep_(Q, cmdg.LSRK54CarpenterKennedy(dg, Q, dt=dt), None, 0.0)
    torch.cuda.synchronize()
    rho = float(ref[:, 0].abs().max())
    for rows, scale in (((0,), rho), ((1, 2, 3), 340.0 * rho), ((4,), float(ref[:, 4].abs().max()))):
        d = float((Q[:, rows] - ref[:, rows]).abs().max())
        assert d <= 1e-13 * scale, (kind, N, rows, d)
