"""The Helmholtz solve at the sizes where its launch form changes, against the oracle.

PCG-Jacobi runs on one CTA, on one cluster of CTAs or on every SM, and keeps all,
some or only the search direction in shared memory; the leaf sums are folded in a
perfect tree in which grids of other sizes leave slots empty. Iteration counts and
solutions are the oracle's bit for bit in every form.
"""

import subprocess
import sys
from pathlib import Path
from types import SimpleNamespace

import numpy as np
import pytest

from oracle import ocean_oracle as orc

pytestmark = pytest.mark.gpu


def _system(nx, ny, seed, walls=False):
    rng = np.random.default_rng(seed)
    dx, dy = 4.0e6 / nx, 5.0e6 / ny
    mask = np.ones((ny, nx))
    mask[ny // 4:ny // 3, nx // 5:nx // 2] = 0.0
    ku = (0.5 + 0.5 * rng.random((ny, nx))) * mask * np.roll(mask, -1, 1)
    kv = (0.5 + 0.5 * rng.random((ny, nx))) * mask * np.roll(mask, -1, 0)
    if walls:
        ku[:, -1] = 0.0
        kv[-1, :] = 0.0
    return dx, dy, 0.4 * dx * dy, ku, kv, mask, rng.standard_normal((ny, nx)) * mask


@pytest.mark.parametrize("nx,ny", [
    (8, 4), (9, 7), (128, 4), (32, 64),   # one CTA, from less than one leaf to its largest
    (45, 46), (41, 640), (640, 41),       # one cluster; short and long rows
    (251, 187), (256, 256),               # uneven leaves; the largest cluster
    (257, 256), (512, 512),               # every SM, all vectors on the chip
    (1000, 720),                          # r and A p on the chip
    (1300, 1260), (5000, 300),            # only the window of p; rows longer than a range
    (600, 2), (3001, 3),                  # a window that would meet itself: the general kernel
])
def test_pcg_jacobi_forms_match_oracle(nx, ny):
    from hydrostatic_ocean_core_benchmark_b200.solvers_var import HelmholtzVar
    dx, dy, coef, ku, kv, mask, rhs = _system(nx, ny, 100 * nx + ny)
    solver = HelmholtzVar(SimpleNamespace(nx=nx, ny=ny, dx=dx, dy=dy), coef, ku, kv, mask, kind="pcg_jacobi",
                          rtol=1e-10)
    ref = orc.Helmholtz(nx, ny, 4.0e6, 5.0e6, coef, ku, kv, mask, "pcg_jacobi", 1e-10, 2000)
    for r in (rhs, rhs[::-1].copy() * mask, np.zeros_like(rhs)):
        x, rep = solver.solve(r)
        xr, itr, ok = ref.solve(r)
        assert rep.iterations == itr and rep.converged == ok
        assert np.array_equal(x, xr)
    solver.close()


@pytest.mark.parametrize("nx,ny", [(40, 30), (120, 130), (400, 390)])
def test_pcg_jacobi_stops_at_max_iter(nx, ny):
    """A solve that does not converge leaves its last iterate and says so, in every form."""
    from hydrostatic_ocean_core_benchmark_b200.solvers_var import HelmholtzVar
    dx, dy, coef, ku, kv, mask, rhs = _system(nx, ny, nx)
    solver = HelmholtzVar(SimpleNamespace(nx=nx, ny=ny, dx=dx, dy=dy), coef, ku, kv, mask, kind="pcg_jacobi",
                          rtol=1e-12, max_iter=3)
    ref = orc.Helmholtz(nx, ny, 4.0e6, 5.0e6, coef, ku, kv, mask, "pcg_jacobi", 1e-12, 3)
    x, rep = solver.solve(rhs)
    xr, itr, ok = ref.solve(rhs)
    assert not ok and not rep.converged and rep.iterations == itr == 3
    assert np.array_equal(x, xr)
    solver.close()


@pytest.mark.parametrize("kind,nx,ny", [("pcg_rbgs", 50, 34), ("pcg_rbgs", 251, 187), ("rbgs", 37, 29),
                                        ("multigrid", 24, 16), ("multigrid", 152, 104)])
def test_uneven_leaf_trees_match_oracle(kind, nx, ny):
    """Grids whose leaf tree is not perfect, through the other solvers (closed at the
    edges: across the wrap of an odd size, neighbours have the same colour)."""
    from hydrostatic_ocean_core_benchmark_b200.solvers_var import HelmholtzVar
    dx, dy, coef, ku, kv, mask, rhs = _system(nx, ny, nx + ny, walls=True)
    solver = HelmholtzVar(SimpleNamespace(nx=nx, ny=ny, dx=dx, dy=dy), coef, ku, kv, mask, kind=kind, rtol=1e-10)
    ref = orc.Helmholtz(nx, ny, 4.0e6, 5.0e6, coef, ku, kv, mask, kind, 1e-10, 2000)
    x, rep = solver.solve(rhs)
    xr, itr, ok = ref.solve(rhs)
    assert rep.iterations == itr and rep.converged == ok
    assert np.array_equal(x, xr)
    solver.close()


@pytest.mark.parametrize("nx,ny", [
    (6, 4), (62, 30), (64, 40), (40, 64),  # one CTA: tiny, an odd coarsest level, the largest
    (66, 40), (52, 50),                               # just above it
    (128, 96), (128, 128),                            # tiles over one-CTA coarse levels
    (300, 14), (75, 77), (290, 142),                  # a coarsest level on the grid: even; odd; below a finer one
    (384, 256), (384, 272),                           # 32 x 32 tiles
    (384, 512), (256, 640),                           # 128 x 16 tiles with their x and b kept, the test piped
    (512, 512),                                       # the same, the residual formed in the up phase
    (512, 520), (1024, 400),                          # a partial last row of tiles; more tiles than SMs
])
def test_multigrid_forms_match_oracle(nx, ny):
    """The V-cycle on one CTA and on tiles of every form (those of a B200's 148 SMs)."""
    from hydrostatic_ocean_core_benchmark_b200.solvers_var import HelmholtzVar
    dx, dy, coef, ku, kv, mask, rhs = _system(nx, ny, nx + 7 * ny, walls=True)
    solver = HelmholtzVar(SimpleNamespace(nx=nx, ny=ny, dx=dx, dy=dy), coef, ku, kv, mask, kind="multigrid",
                          rtol=1e-8, max_iter=6)
    ref = orc.Helmholtz(nx, ny, 4.0e6, 5.0e6, coef, ku, kv, mask, "multigrid", 1e-8, 6)
    for r in (rhs, np.zeros_like(rhs), rhs[:, ::-1].copy()):
        x, rep = solver.solve(r)
        xr, itr, ok = ref.solve(r)
        assert rep.iterations == itr and rep.converged == ok
        assert np.array_equal(x, xr)
    solver.close()


@pytest.mark.parametrize("kind,nx,ny", [("pcg_jacobi", 40, 30), ("pcg_jacobi", 120, 130), ("pcg_jacobi", 400, 390),
                                        ("pcg_jacobi", 1000, 720), ("pcg_jacobi", 5000, 300),
                                        ("multigrid", 48, 40), ("multigrid", 256, 192)])
def test_a_solve_in_place_gives_the_same_solution(kind, nx, ny):
    """x may be the right-hand side's own device array."""
    import ctypes as C
    import torch
    from hydrostatic_ocean_core_benchmark_b200.solvers_var import HelmholtzVar
    dx, dy, coef, ku, kv, mask, rhs = _system(nx, ny, nx, walls=True)
    solver = HelmholtzVar(SimpleNamespace(nx=nx, ny=ny, dx=dx, dy=dy), coef, ku, kv, mask, kind=kind, rtol=1e-9)
    want, rep = solver.solve(rhs)
    a = torch.as_tensor(rhs, device="cuda:0").contiguous()
    its, conv = C.c_int32(), C.c_int32()
    solver._check(solver.lib.oc_helm_solve(solver.h, a.data_ptr(), a.data_ptr(), 1, C.byref(its), C.byref(conv),
                                           torch.cuda.current_stream().cuda_stream), "oc_helm_solve")
    assert its.value == rep.iterations
    assert np.array_equal(a.cpu().numpy(), want)
    solver.close()


@pytest.mark.parametrize("nx,ny", [(40, 30), (120, 130), (400, 390), (1000, 720), (5000, 300)])
def test_pcg_jacobi_warm_start(nx, ny):
    """The mixed-precision step's solves start from the elevation they are given, in every
    form: one step's elevation against that of PCG-RBGS (the general kernel). Both stop at
    |r| <= rtol |b| and A - 1 is positive, so they are within 2 rtol |b| <= 2 rtol |A| |x|."""
    from hydrostatic_ocean_core_benchmark_b200 import cases
    from hydrostatic_ocean_core_benchmark_b200.stepper import OceanStepper
    rtol, got = 1e-9, {}
    y, x = np.mgrid[0:ny, 0:nx]
    eta = 0.3 * np.sin(3.0 * x / nx) * np.cos(5.0 * y / ny)
    for kind in ("pcg_jacobi", "pcg_rbgs"):
        s = cases.seamount_basin(nx=nx, ny=ny, nz=2, seed=4, dt=120.0, solver_kind=kind, rtol=rtol, n_picard=1,
                                 closure="none")
        p = s.params
        st = OceanStepper(p, s.H, s.mask, dzr=s.dzr, taux_c=s.taux_c, tauy_c=s.tauy_c, precision="mixed")
        st.set_state(eta=eta, u=s.u, v=s.v, T=s.T, S=s.S)
        st.step(1)
        got[kind] = st.get_state()["eta"]
        assert st.stats()["solver_failures"] == 0
        st.close()
    norm_A = 1.0 + 4.0 * p.g * (p.theta * p.dt) ** 2 * float(s.H.max()) * (1.0 / p.dx ** 2 + 1.0 / p.dy ** 2)
    err = np.linalg.norm(got["pcg_jacobi"] - got["pcg_rbgs"])
    assert err <= 2.0 * rtol * norm_A * np.linalg.norm(got["pcg_rbgs"])
    # and the step moved the elevation by much more than that
    assert np.linalg.norm(got["pcg_rbgs"] - eta) > 1e3 * err


# run in a process of its own: a solver built earlier may have raised the kernels'
# shared-memory allowance for all that follow
FRESH_SOLVE = """
import sys
from types import SimpleNamespace
import numpy as np
from hydrostatic_ocean_core_benchmark_b200.solvers_var import HelmholtzVar
from oracle import ocean_oracle as orc
from tests.test_gpu_helm_forms import _system
nx, ny = int(sys.argv[1]), int(sys.argv[2])
dx, dy, coef, ku, kv, mask, rhs = _system(nx, ny, nx + ny, walls=True)
solver = HelmholtzVar(SimpleNamespace(nx=nx, ny=ny, dx=dx, dy=dy), coef, ku, kv, mask, kind="multigrid", rtol=1e-8,
                      max_iter=4)
x, rep = solver.solve(rhs)
xr, itr, ok = orc.Helmholtz(nx, ny, 4.0e6, 5.0e6, coef, ku, kv, mask, "multigrid", 1e-8, 4).solve(rhs)
assert rep.iterations == itr and rep.converged == ok
assert np.array_equal(x, xr)
"""

FRESH_ENSEMBLE = """
import sys
from tests.test_gpu_ensemble import _member, _same
from hydrostatic_ocean_core_benchmark_b200.stepper import OceanEnsemble
sizes = [(int(sys.argv[1]), int(sys.argv[2]), 3, seed) for seed in (1, 2)]
together, alone = [_member(*s) for s in sizes], [_member(*s) for s in sizes]
OceanEnsemble(together).step(2)
for a, b in zip(together, alone):
    b.step(2)
    _same(a, b, "ensemble member")
"""


@pytest.mark.parametrize("script,nx,ny", [
    (FRESH_SOLVE, 104, 104), (FRESH_SOLVE, 52, 52), (FRESH_SOLVE, 26, 26), (FRESH_SOLVE, 80, 172),
    (FRESH_SOLVE, 108, 128), (FRESH_ENSEMBLE, 104, 104),
], ids=lambda a: {FRESH_SOLVE: "solve", FRESH_ENSEMBLE: "ensemble"}.get(a, a))
def test_multigrid_near_the_default_shared_memory_limit(script, nx, ny):
    """Solvers whose dynamic shared memory is under 48 KB and whose dynamic and static
    shared memory together are not (46,480 to 48,896 bytes beside 2.8 KB)."""
    r = subprocess.run([sys.executable, "-c", script, str(nx), str(ny)], capture_output=True, text=True, timeout=300,
                       cwd=Path(__file__).resolve().parents[1])
    assert r.returncode == 0, r.stderr[-2000:]
