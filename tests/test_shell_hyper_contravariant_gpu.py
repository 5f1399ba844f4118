"""Hyperdiffusion on the cubed shell: the passes hand contravariant components
J dxi_d/dx . grad from one to the next, and a face takes the neighbour's
component along the neighbour's own direction, with a sign where two lower (or
two upper) faces meet across a panel edge.  2 x 2 elements per panel meet every
pairing of panels on every element; with and without xi3 terms.

FP64 rounding: three chained derivatives on each side of the comparison, each
amplifying rounding by at most 2 max|D| Nq < 200, stay below 1e-9 of the
fields' scale (2e-16 * 200^3 = 2e-9 is the bound for worst-case alignment)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

TAU = 3600.0


@pytest.mark.gpu
@pytest.mark.parametrize("direction", ["horizontal", "every"])
@pytest.mark.parametrize("N", [2, 3, 4, 5])
def test_shell_hyperdiffusive_tendency_across_panels(N, direction):
    import cmdg
    import oracle as O
    from cmdg import workloads

    R = O.EARTH["planet_radius"]
    om = O.OracleModel(N, shell=dict(nhorz=2, nvert=2, r_inner=R, r_outer=R + 30e3), orientation="sphere",
                       gravity=True, ref_state=True, profile="isothermal", T_surface=285.0,
                       hyperdiffusion="dry_biharmonic", tau_hyper=TAU, hyper_direction=direction)
    dg = workloads.gcm_shell_model(nhorz=2, nvert=2, N=N, precision="fp64", tau_hyper=TAU,
                                   diffusion_direction=direction)
    Q = workloads.gcm_initial_state(dg.grid.coordinates(), seed=5)
    Q[:, 1:4] += np.random.default_rng(7).uniform(-0.5, 0.5, size=Q[:, 1:4].shape)
    ref = om.tendency(Q)
    dQ = dg.new_state(torch.float64)
    dg(dQ, dg.init_ode_state(Q), None, 0.0)
    got = dQ.cpu().numpy()
    for rows in ((0,), (1, 2, 3), (4,)):
        a, b = got[:, rows], ref[:, rows]
        assert np.abs(a - b).max() < 2e-9 * np.abs(b).max(), (rows, np.abs(a - b).max() / np.abs(b).max())
