"""Members of an ensemble step as they do by themselves, field by field: density,
momentum and energy each against its own change, from a bubble with winds and a
pressure wave at an acoustic Courant number of 0.4, so that every field changes
far above rounding.

Bound: the two kernels sum the same terms in different orders.  A nodal sum of
3 (N + 1) + 20 products in FP32 whose magnitudes exceed the result up to
20-fold differs by at most 40 * 20 * 2^-24 < 5e-5 of the change, and storing the
state in FP32 five times per step adds an ulp each: 3 steps, 15 * 2^-23 of the
field."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

L = 2500.0


def _state(dg):
    from cmdg import workloads

    xyz = dg.grid.coordinates()
    Q = workloads.rising_bubble(xyz)
    x, y, z = (2 * np.pi * xyz[:, d] / L for d in range(3))
    wind = 5.0 * np.stack((np.sin(x + y), np.cos(y) * np.sin(0.5 * z), 0.3 * np.sin(0.5 * z) * np.cos(x)), axis=1)
    Q[:, 4] += 0.5 * Q[:, 0] * (wind ** 2).sum(axis=1) + 2.5 * 200.0 * np.sin(x) * np.cos(0.5 * z)
    Q[:, 1:4] = Q[:, 0][:, None] * wind
    return Q


@pytest.mark.gpu
@pytest.mark.parametrize("specs", [[(8, 8, 8, 4)], [(8, 8, 7, 4)], [(10, 10, 10, 3), (9, 9, 9, 3)], [(7, 7, 8, 5), (6, 6, 6, 5)],
                                   [(3, 4, 5, 3), (9, 8, 8, 4), (2, 3, 2, 5), (8, 8, 7, 4), (10, 10, 10, 3)]])
def test_every_field_steps_as_by_itself(specs):
    import cmdg
    from cmdg import workloads

    members = [workloads.bubble_model(ne=s[:3], N=s[3], precision="mixed") for s in specs]
    Q0 = [dg.init_ode_state(_state(dg)) for dg in members]
    dts = [dg.courant_dt(q, 0.4) for dg, q in zip(members, Q0)]
    Qs = [q.clone() for q in Q0]
    regs = [torch.zeros(q.shape, dtype=torch.float64, device=q.device) for q in Qs]
    ens = cmdg.Ensemble(members)
    ens.lsrk54_step(Qs, regs, dts)
    ens.lsrk54_step(Qs, regs, dts, nsteps=2)
    for dg, q0, q, dt in zip(members, Q0, Qs, dts):
        ref = q0.clone()
        lsrk = cmdg.LSRK54CarpenterKennedy(dg, ref, dt=dt)
        for _ in range(3):
            cmdg.dostep_(ref, lsrk, None, 0.0)
        for rows in ((0,), (1, 2, 3), (4,)):
            a, b, c = (t[:, rows].double() for t in (q, ref, q0))
            change, size = float((b - c).norm()), float(b.norm())
            assert change > 1e-4 * size
            assert float((a - b).norm()) <= 5e-5 * change + 15 * 2.0 ** -23 * size, rows
