"""The momentum and tracer kernels where a tile's levels are all full, and where they stop being so.

Those levels take the short form (thicknesses from the level table, face masks as bits);
the levels below, and tiles that touch a shallow column, the general one. Fields equal
the oracle's bit for bit in both and across the change, for walls and periodic edges,
every advection and face rule, horizontal mixing, and any number of levels per CTA.
"""

import numpy as np
import pytest

from oracle import ocean_oracle as orc

pytestmark = pytest.mark.gpu

NX, NY, NZ = 70, 21, 11


def _case(bc_x, bc_y, advection, face_rule, mix, tracers, closure, shallow):
    from hydrostatic_ocean_core_benchmark_b200.params import OceanParams
    p = OceanParams(nx=NX, ny=NY, nz=NZ, lx=4.0e3 * NX, ly=3.5e3 * NY, h0=2000.0, nu=1e-3, kappa=1e-3, tau_x=0.1,
                    tau_y=-0.05, bottom_drag=1e-3, scheme_name="theta", theta=0.6, n_picard=2,
                    solver_kind="pcg_jacobi", rtol=1e-12, dt=60.0, bc_x=bc_x, bc_y=bc_y, eos="teos10", pgf="keep",
                    advection=advection, tracers=tracers, closure=closure, face_rule=face_rule, a_h=mix, k_h=mix,
                    q_heat=20.0, q_salt=1e-7)
    rng = np.random.default_rng(5)
    H = np.full((NY, NX), 2000.0)
    if shallow:
        H[4:9, 50:58] = 700.0       # a tile, and its neighbours' rings, with partial columns
        H[15, 3] = 130.0            # one wet level
        H[0:3, 30:40] = 1990.0      # a partial bottom level
        # just outside the first tile's ring: the outermost faces of the ring are shallower than its columns
        H[5, 34] = 500.0
        H[10, 20] = 600.0
    mask = np.ones((NY, NX))
    if shallow:
        mask[18, 10:14] = 0.0       # land
    dzr = 60.0 * 1.12 ** np.arange(NZ)
    dzr *= 2000.0 / dzr.sum()
    geo = orc.Geometry(p, H, mask, dzr)
    m3 = geo.mask3
    T = (10.0 + rng.standard_normal(m3.shape)) * m3
    S = (35.0 + 0.1 * rng.standard_normal(m3.shape)) * m3
    S[:, :, :20] = 35.0 * m3[:, :, :20]  # uniform: zero differences in the limiter
    # velocities on closed faces too: a caller may give them, and the step carries them
    u, v = 0.2 * rng.standard_normal(m3.shape) * m3, 0.2 * rng.standard_normal(m3.shape) * m3
    eta = 0.1 * rng.standard_normal((NY, NX))
    b = orc.buoyancy(p.eos, T, S, geo.zc, p.g, p.rho0, p.alpha_t, p.beta_s, p.t0, p.s0) * m3
    return p, H, mask, dzr, orc.OracleState(u, v, b, eta, T if tracers == "TS" else None, S if tracers == "TS" else None)


@pytest.mark.parametrize("bc_x,bc_y,advection,face_rule,mix,tracers,closure,shallow,levels", [
    ("closed", "closed", "up3_tvd", "min", 0.0, "TS", "tke", True, (3, 4)),
    ("periodic", "closed", "up3_tvd", "harmonic", 50.0, "TS", "none", True, (NZ, NZ)),
    ("closed", "periodic", "up3", "mean", 50.0, "TS", "none", True, (1, 1)),
    ("periodic", "periodic", "up3_tvd", "min", 0.0, "TS", "none", False, (NZ, 5)),
    ("closed", "closed", "centered2", "harmonic", 0.0, "buoyancy", "none", True, (4, 2)),
    ("periodic", "periodic", "upwind1", "min", 30.0, "TS", "none", False, (2, 3)),
    ("closed", "closed", "none", "mean", 30.0, "buoyancy", "none", False, (5, NZ)),
])
def test_full_levels_match_oracle(bc_x, bc_y, advection, face_rule, mix, tracers, closure, shallow, levels):
    from hydrostatic_ocean_core_benchmark_b200.stepper import OceanStepper
    p, H, mask, dzr, state = _case(bc_x, bc_y, advection, face_rule, mix, tracers, closure, shallow)
    ref = orc.OracleStepper(p, H, mask, dzr=dzr)
    st = OceanStepper(p, H, mask, dzr=dzr)
    tuned = OceanStepper(p, H, mask, dzr=dzr)
    tuned.set_tiling(*levels)
    for s in (st, tuned):
        s.set_state(eta=state.eta, u=state.u, v=state.v, b=state.b, T=state.T, S=state.S)
    for step in range(3):
        state = ref.step(state)
        for s in (st, tuned):
            s.step(1)
            got = s.get_state()
            for f in ("eta", "u", "v", "b") + (("T", "S") if tracers == "TS" else ()):
                assert np.array_equal(got[f], getattr(state, f)), f"step {step + 1}: {f} differs"
    assert st.solve_log() == ref.solve_log
    st.close()
    tuned.close()


@pytest.mark.parametrize("face_rule", ["harmonic", "mean", "min"])
def test_mixed_full_levels_do_not_depend_on_the_tiling(face_rule):
    """A slab of levels starts with fluxes formed from the columns' own thicknesses, and
    the levels below carry those of the level table: the FP32 step's bits are the same
    wherever slabs start, in tiles of full, partial and mixed columns."""
    from hydrostatic_ocean_core_benchmark_b200.stepper import OceanStepper
    nx, ny = 100, 40
    p = _case("closed", "periodic", "up3_tvd", face_rule, 50.0, "TS", "none", True)[0].replace(
        nx=nx, ny=ny, lx=4.0e3 * nx, ly=3.5e3 * ny, nu=2.0e3, kappa=2.0e3)  # large explicit fluxes between levels
    H, mask = np.full((ny, nx), 2000.0), np.ones((ny, nx))
    H[14:18, 45:60] = 700.0
    rng = np.random.default_rng(2)
    shape = (NZ, ny, nx)
    u, v = 0.2 * rng.standard_normal(shape), 0.2 * rng.standard_normal(shape)
    T, S = 10.0 + rng.standard_normal(shape), 35.0 + 0.1 * rng.standard_normal(shape)
    eta = 0.1 * rng.standard_normal((ny, nx))
    dzr = 60.0 + 200.0 * np.random.default_rng(3).random(NZ)
    dzr *= 2000.0 / dzr.sum()
    d = dzr.astype(np.float32)
    if face_rule == "harmonic":  # levels where the fp64 mean rounded to FP32 is another number
        assert np.any((2.0 * dzr * dzr / (dzr + dzr)).astype(np.float32) != np.float32(2.0) * d * d / (d + d))
    fields = []
    for levels in (None, (1, 1), (3, 4), (4, 3), (NZ, NZ)):
        st = OceanStepper(p, H, mask, dzr=dzr, precision="mixed")
        if levels:
            st.set_tiling(*levels)
        st.set_state(eta=eta, u=u, v=v, T=T, S=S)
        st.step(3)
        fields.append(st.get_state())
        st.close()
    for f in ("eta", "u", "v", "b", "T", "S"):
        assert np.all(np.isfinite(fields[0][f]))
        for other in fields[1:]:
            assert np.array_equal(fields[0][f], other[f]), f"{f} depends on the levels per CTA"
