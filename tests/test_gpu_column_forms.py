"""The column kernels, the adjoint's scatter and the EOS at the sizes where their forms change.

Up to a number of columns a column's levels are shared by several threads (w, K_u and K_v,
the back substitution, the closure, the tracer solve) and its components by two (the
momentum solve); above it a thread takes a column. Fields equal the oracle's bit for bit on both sides of the
limit, at level counts around the chunk of levels.
"""

import numpy as np
import pytest

from oracle import ocean_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mxl", ["integral", "recursive"])
@pytest.mark.parametrize("nx,ny,nz", [
    (256, 192, 3), (256, 193, 3),   # the limit of the few-column forms, and just above it
    (128, 192, 2), (193, 128, 2),   # half of it (K_u, K_v)
    (45, 3, 33), (33, 5, 8), (7, 4, 1), (64, 2, 41),  # part-filled warps; around a chunk of levels
    # the kernels' own limits, which depend on the levels: few of them, one CTA of rows an SM
    (224, 128, 24), (225, 128, 24), (256, 144, 16), (256, 145, 16), (128, 32, 8), (128, 65, 8), (128, 129, 7),
    (41, 30, 90), (41, 30, 128),
])
def test_column_forms_match_oracle(nx, ny, nz, mxl):
    from hydrostatic_ocean_core_benchmark_b200 import cases
    from hydrostatic_ocean_core_benchmark_b200.stepper import OceanStepper
    s = cases.seamount_basin(nx=nx, ny=ny, nz=nz, seed=nx + ny, solver_kind="pcg_jacobi", rtol=1e-10,
                             mxl=mxl)
    p = s.params
    geo = orc.Geometry(p, s.H, s.mask, s.dzr)
    b = orc.buoyancy(p.eos, s.T, s.S, geo.zc, p.g, p.rho0, p.alpha_t, p.beta_s, p.t0, p.s0) * geo.mask3
    ref = orc.OracleStepper(p, s.H, s.mask, dzr=s.dzr, taux_c=s.taux_c, tauy_c=s.tauy_c)
    st = OceanStepper(p, s.H, s.mask, dzr=s.dzr, taux_c=s.taux_c, tauy_c=s.tauy_c)
    st.set_state(eta=s.eta, u=s.u, v=s.v, b=b, T=s.T, S=s.S)
    state = orc.OracleState(s.u, s.v, b, s.eta, s.T, s.S)
    for step in range(2):
        state = ref.step(state)
        st.step(1)
        got = st.get_state()
        for f in ("eta", "u", "v", "b", "T", "S", "e"):
            assert np.array_equal(got[f], getattr(state, f)), f"step {step + 1}: {f} differs"
    st.close()


# one cell a thread up to 2 x 148 x 8 x 256 cells, four above; the last leaves each remainder of four blocks' widths
@pytest.mark.parametrize("n", [1, 255, 257, 769, 1023, 1024, 1025, 606208, 606209, 606977, 700001])
@pytest.mark.parametrize("kind", ["linear", "seos", "teos10"])
def test_density_matches_oracle(kind, n):
    import torch
    from hydrostatic_ocean_core_benchmark_b200 import _lib
    rng = np.random.default_rng(n)
    T, S, z = 2.0 + 18.0 * rng.random(n), 33.0 + 3.0 * rng.random(n), 4000.0 * rng.random(n)
    if kind == "teos10":
        want = orc.rho_teos10(T, S, z)
    else:
        want = orc.rho_anomaly(kind, T, S, z, 1025.0, 2.0e-4, 7.4e-4, 10.0, 35.0)
    dT, dS, dz = (torch.as_tensor(a, device="cuda:0") for a in (T, S, z))
    out = torch.full((n + 4,), -7.0, dtype=torch.float64, device="cuda:0")
    stream = torch.cuda.current_stream()
    _lib.check(_lib.load().oc_density(("linear", "seos", "teos10").index(kind), 1025.0, 2.0e-4, 7.4e-4, 10.0, 35.0,
                                      dT.data_ptr(), dS.data_ptr(), dz.data_ptr(), out.data_ptr(), n,
                                      stream.cuda_stream), None, "oc_density")
    got = out.cpu().numpy()
    assert np.array_equal(got[:n], want)
    assert np.all(got[n:] == -7.0)
