"""The workloads this framework is timed on: what its users run, over the range they run it.

Six kinds of work, each through the package's public entry points:

* ``step``: a forecast window -- a state uploaded from device tensors, a number of
  model steps, the state read back. Sizes, schemes, solvers and options follow the
  repository's recipes (``cases.py``, ``config/*.toml``) and its tests and benchmark.
* ``ensemble``: several members of uneven grids advanced by one recorded graph.
* ``adjoint``: the gradient of a short run with respect to the initial temperature and
  the surface stress field.
* ``helmholtz``: the free-surface solver on its own, on device arrays.
* ``density``: an equation of state over flat arrays.
* ``thomas``: the batched column solve on device arrays.

Inputs are seeded: a basin over Gaussian seamounts with stretched levels, a stratified
T/S profile with noise, a smooth current, a raised surface and a wind-mixed layer of
turbulent energy, so that a first step meets the values of a running model.
"""

import ctypes as C
import math

import numpy as np
import torch

from hydrostatic_ocean_core_benchmark_b200 import _lib
from hydrostatic_ocean_core_benchmark_b200 import cases as recipes
from hydrostatic_ocean_core_benchmark_b200.adjoint import OceanRollout, rollout_apply
from hydrostatic_ocean_core_benchmark_b200.params import OceanParams
from hydrostatic_ocean_core_benchmark_b200.stepper import OceanEnsemble, OceanStepper

DEV = "cuda:0"
CELL = 3906.25  # horizontal spacing [m] of the 512 x 512 basin, kept for the other sizes


def listed():
    return [
        # one call per step on a small test-sized basin: launches and latency
        _step("step_48x48x12_single", 48, 48, 12, steps=1, graph=False),
        # the lock-exchange channel: a narrow periodic-index domain, PCG-Jacobi, linear EOS
        {"name": "step_channel_128x4x32", "kind": "step", "recipe": "channel", "nx": 128, "ny": 4, "nz": 32,
         "steps": 10, "graph": True, "scheme": "theta", "solver": "pcg_jacobi", "closure": "none", "mxl": "integral",
         "advection": "up3_tvd", "eos": "linear", "face_rule": "min", "mix": 0.0, "precision": "fp64"},
        # an ordinary basin, as ensemble members and tests have it
        _step("step_128x128x50", 128, 128, 50, steps=4),
        # the benchmark's basin
        _step("step_512x512x50", 512, 512, 50, steps=4),
        # the same with the 3D state in FP32
        _step("step_512x512x50_mixed", 512, 512, 50, steps=4, precision="mixed"),
        # odd sizes, the reference's default solver, other advection, mixing length, face rule and viscosity
        _step("step_251x187x37_pcg", 251, 187, 37, steps=2, solver="pcg_jacobi", advection="up3", mxl="recursive",
              face_rule="harmonic", mix=100.0),
        # the explicit free surface (no elliptic solve), without a closure, centred advection
        _step("step_384x320x30_fb", 384, 320, 30, steps=4, scheme="fb", closure="none", advection="centered2",
              eos="seos"),
        # the split-explicit scheme with its barotropic substeps
        _step("step_200x160x40_split", 200, 160, 40, steps=2, scheme="split_explicit"),
        # members of uneven grids advanced together
        {"name": "ensemble_8", "kind": "ensemble", "members": 8, "lo": 4, "hi": 12, "nz": 24, "steps": 4},
        # the gradient of a five-step run
        {"name": "adjoint_256x256x32", "kind": "adjoint", "nx": 256, "ny": 256, "nz": 32, "steps": 5},
        # the free-surface system alone, on a size with no power of two in it
        {"name": "helmholtz_pcg_1000x720", "kind": "helmholtz", "nx": 1000, "ny": 720, "solver": "pcg_jacobi",
         "rtol": 1.0e-10},
        # the equation of state over a large flat array
        {"name": "density_teos10_2e7", "kind": "density", "n": 20000003, "eos": 2},
    ]


def _step(name, nx, ny, nz, steps, graph=True, scheme="theta", solver="multigrid", closure="tke", mxl="integral",
          advection="up3_tvd", eos="teos10", face_rule="min", mix=0.0, precision="fp64"):
    case = {"kind": "step", "recipe": "basin", "nx": nx, "ny": ny, "nz": nz, "steps": steps, "graph": graph,
            "scheme": scheme, "solver": solver, "closure": closure, "mxl": mxl, "advection": advection, "eos": eos,
            "face_rule": face_rule, "mix": mix, "precision": precision}
    if name:
        case["name"] = name
    return case


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.random()
    if pick < 0.64:
        while True:
            nx, ny, nz = _log(rng, 32, 512), _log(rng, 32, 512), _log(rng, 8, 64)
            solver = rng.choice(["multigrid", "multigrid", "pcg_jacobi"])
            if solver == "multigrid":  # sizes the hierarchy halves down to at most 15
                q = 2 ** max(0, math.ceil(math.log2(max(nx, ny) / 15.0)))
                nx, ny = max(8, round(nx / q)) * q, max(8, round(ny / q)) * q
            if nx <= 512 and ny <= 512 and nx * ny * nz <= 9_000_000:
                break
        scheme = rng.choice(["theta"] * 6 + ["fb", "split_explicit"])
        precision = rng.choice(["fp64", "fp64", "mixed"]) if scheme == "theta" else "fp64"
        advection = rng.choice(["up3_tvd", "up3_tvd", "up3", "centered2"])
        return _step(None, nx, ny, nz, steps=rng.choice([1, 2, 4]), graph=rng.random() < 0.7, scheme=scheme,
                     solver=solver, closure=rng.choice(["tke", "tke", "none"]),
                     mxl=rng.choice(["integral", "integral", "recursive"]), advection=advection,
                     eos=rng.choice(["teos10", "teos10", "seos", "linear"]),
                     face_rule=rng.choice(["min", "min", "mean", "harmonic"]),
                     mix=rng.choice([0.0, 0.0, 100.0]), precision=precision)
    if pick < 0.72:
        return {"kind": "ensemble", "members": rng.randint(2, 8), "lo": 3, "hi": rng.randint(5, 10),
                "nz": rng.randint(12, 40), "steps": rng.choice([2, 4])}
    if pick < 0.80:
        return {"kind": "adjoint", "nx": 2 * _log(rng, 20, 128), "ny": 2 * _log(rng, 20, 128),
                "nz": _log(rng, 8, 32), "steps": rng.randint(2, 5)}
    if pick < 0.89:
        return {"kind": "helmholtz", "nx": _log(rng, 48, 1400), "ny": _log(rng, 48, 1400),
                "solver": rng.choice(["pcg_jacobi", "pcg_jacobi", "pcg_rbgs", "pcg_refined"]),
                "rtol": rng.choice([1.0e-8, 1.0e-10, 1.0e-12])}
    if pick < 0.95:
        return {"kind": "density", "n": _log(rng, 1000, 20_000_000), "eos": rng.choice([0, 1, 2])}
    return {"kind": "thomas", "n": _log(rng, 8, 120), "ncols": _log(rng, 500, 300_000)}


# ------------------------------------------------------------------ inputs
def _rng(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _layers(H, dzr, min_partial):
    """Wet mask, level-centre depth of the z-level cells (float64, on the GPU)."""
    edge = torch.cumsum(dzr, 0) - dzr
    dz = torch.minimum((H[None] - edge[:, None, None]).clamp_min(0.0), dzr[:, None, None])
    dz = torch.where(dz < min_partial * dzr[:, None, None], torch.zeros((), dtype=dz.dtype, device=DEV), dz)
    return (dz > 0.0).double(), torch.cumsum(dz, 0) - dz + 0.5 * dz


def _basin(nx, ny, nz, seed, **over):
    """Parameters, bathymetry, levels and wind of a seeded seamount basin."""
    opts = dict(nx=nx, ny=ny, nz=nz, lx=CELL * nx, ly=CELL * ny, h0=4000.0, nu=1.0e-3, kappa=1.0e-3, tau_x=0.1,
                scheme_name="theta", theta=0.6, n_picard=2, solver_kind="multigrid", rtol=1.0e-12, max_iter=2000,
                dt=600.0, bc_x="closed", bc_y="closed", eos="teos10", pgf="keep", advection="up3_tvd", tracers="TS",
                closure="tke", mxl="integral")
    opts.update(over)
    p = OceanParams(**opts)
    # seamounts of the benchmark's heights, their radii in proportion to the basin
    s = min(p.lx, p.ly) / 2.0e6
    H = recipes.seamount_bathymetry(p, np.random.default_rng(seed), r_lo=5.0e4 * s, r_hi=2.0e5 * s)
    dzr = recipes.stretched_levels(nz, float(H.max()))
    y = (np.arange(ny) + 0.5) * p.dy
    taux = np.repeat(0.1 * np.cos(2.0 * np.pi * y / p.ly)[:, None], nx, axis=1)
    return p, H, dzr, taux


def _state(p, H, dzr, seed, mixed_layer=True):
    """A running model's fields: stratification with noise, a smooth current decaying with
    depth, a raised surface, and turbulent energy and viscosity of a wind-mixed layer."""
    g = _rng(seed)
    m3, zc = _layers(torch.from_numpy(H).to(DEV), torch.from_numpy(dzr).to(DEV), p.min_partial)
    nz, ny, nx = zc.shape

    def noise():
        return torch.randn(zc.shape, generator=g, device=DEV, dtype=torch.float64)

    T = (2.0 + 18.0 * torch.exp(-zc / 800.0) + 0.01 * noise()) * m3
    S = (35.0 + 0.5 * torch.exp(-zc / 500.0) + 0.001 * noise()) * m3
    x = (torch.arange(nx, device=DEV, dtype=torch.float64) + 0.5)[None, :] * (2.0 * math.pi / nx)
    y = (torch.arange(ny, device=DEV, dtype=torch.float64) + 0.5)[:, None] * (2.0 * math.pi / ny)
    ph = torch.rand(6, generator=g, device=DEV, dtype=torch.float64) * 2.0 * math.pi
    wall_x = torch.ones(nx, device=DEV, dtype=torch.float64)
    wall_y = torch.ones(ny, device=DEV, dtype=torch.float64)
    if p.bc_x == "closed":
        wall_x[-1] = 0.0
    if p.bc_y == "closed":
        wall_y[-1] = 0.0
    decay = torch.exp(-zc / 600.0)
    mu = m3 * torch.roll(m3, -1, 2) * wall_x
    mv = m3 * torch.roll(m3, -1, 1) * wall_y[:, None]
    u = (0.1 * torch.sin(2.0 * y + ph[0]) * torch.cos(x + ph[1]) * decay + 1.0e-3 * noise()) * mu
    v = (0.1 * torch.sin(3.0 * x + ph[2]) * torch.cos(y + ph[3]) * decay + 1.0e-3 * noise()) * mv
    eta = 0.05 * torch.sin(x + ph[4]) * torch.cos(2.0 * y + ph[5])
    st = {"eta": eta, "u": u, "v": v, "T": T, "S": S}
    if mixed_layer:
        zi = torch.from_numpy(np.concatenate([[0.0], np.cumsum(dzr)])).to(DEV)[:, None, None]
        fade = torch.exp(-zi / 40.0) * (1.0 + 0.2 * torch.sin(x + y + ph[0]))
        st["e"] = p.e_min + 2.0e-3 * fade.expand(nz + 1, ny, nx)
        st["km"] = p.nu + 0.02 * fade.expand(nz + 1, ny, nx)
        st["kh"] = p.kappa + 0.02 * fade.expand(nz + 1, ny, nx)
    return {k: f.contiguous() for k, f in st.items()}


def _buffers(p):
    n2, n3, ni = (p.ny, p.nx), (p.nz, p.ny, p.nx), (p.nz + 1, p.ny, p.nx)
    shapes = {"eta": n2, "u": n3, "v": n3, "b": n3, "T": n3, "S": n3, "e": ni, "km": ni, "kh": ni}
    return {k: torch.empty(s, device=DEV, dtype=torch.float64) for k, s in shapes.items()}


def _step_params(case):
    over = dict(scheme_name=case["scheme"], solver_kind=case["solver"], closure=case["closure"], mxl=case["mxl"],
                advection=case["advection"], eos=case["eos"], face_rule=case["face_rule"], a_h=case["mix"],
                k_h=case["mix"])
    # dt of the benchmark; the explicit surface, and PCG-Jacobi runs, keep to a few gravity-wave steps
    wave = CELL / math.sqrt(2.0 * 9.80616 * 4000.0)
    if case["scheme"] == "fb":
        over["dt"] = 0.5 * wave
    elif case["solver"] == "pcg_jacobi" and case["scheme"] == "theta":
        over["dt"] = 4.0 * wave
    else:
        over["dt"] = 300.0
    return over


def _channel(case, seed):
    s = recipes.lock_exchange_channel(nx=case["nx"], ny=case["ny"], nz=case["nz"])
    g = _rng(seed)
    T = torch.from_numpy(s.T).to(DEV)
    T = T + 0.01 * torch.randn(T.shape, generator=g, device=DEV, dtype=torch.float64)
    st = {"eta": torch.from_numpy(s.eta).to(DEV), "u": torch.from_numpy(s.u).to(DEV),
          "v": torch.from_numpy(s.v).to(DEV), "T": T.contiguous(), "S": torch.from_numpy(s.S).to(DEV)}
    return s, st


def _solver_handle(case, seed):
    """A free-surface system of the reference cases' conditioning with an island, on the device."""
    rng = np.random.default_rng(seed)
    nx, ny = case["nx"], case["ny"]
    dx = 4.0e6 / max(nx, ny)
    mask = np.ones((ny, nx))
    mask[ny // 4:ny // 3, nx // 5:nx // 2] = 0.0
    ku = (0.5 + 0.5 * rng.random((ny, nx))) * mask * np.roll(mask, -1, 1)
    kv = (0.5 + 0.5 * rng.random((ny, nx))) * mask * np.roll(mask, -1, 0)
    rhs = rng.standard_normal((ny, nx)) * mask
    return dx, 0.5 * dx * dx, ku, kv, mask, rhs


class _Helm:
    """A handle of the standalone solver (oc_helm_*)."""

    def __init__(self, case, seed):
        dx, coef, ku, kv, mask, rhs = _solver_handle(case, seed)
        self.lib, self.h = _lib.load(), C.c_void_p()
        kinds = {"pcg_jacobi": 0, "pcg_rbgs": 1, "multigrid": 3, "pcg_refined": 4}
        cfg = _lib.OcHelmConfig(nx=case["nx"], ny=case["ny"], dx=dx, dy=dx, coef=coef, solver=kinds[case["solver"]],
                                rtol=case["rtol"], max_iter=2000, device=0)
        _lib.check(self.lib.oc_helm_create(C.byref(cfg), ku.ctypes.data, kv.ctypes.data, mask.ctypes.data,
                                           C.byref(self.h)), None, "oc_helm_create")
        self.rhs = torch.from_numpy(rhs).to(DEV)
        self.x = torch.empty_like(self.rhs)

    def solve(self):
        its, conv = C.c_int32(), C.c_int32()
        _lib.check(self.lib.oc_helm_solve(self.h, self.rhs.data_ptr(), self.x.data_ptr(), 1, C.byref(its),
                                          C.byref(conv), torch.cuda.current_stream().cuda_stream), None, "oc_helm_solve")
        return {"x": self.x, "iterations": its.value, "converged": conv.value}

    def __del__(self):
        if getattr(self, "h", None):
            self.lib.oc_helm_destroy(self.h)
            self.h = None


def _thomas_inputs(case, seed):
    g = _rng(seed)
    shape = (case["n"], case["ncols"])
    a, c, r = (torch.rand(shape, generator=g, device=DEV, dtype=torch.float64) for _ in range(3))
    return -a, 1.0 + a + c, -c, r - 0.5


def prepare(case, seed):
    torch.cuda.set_device(0)
    kind = case["kind"]
    if kind == "step":
        if case["recipe"] == "channel":
            s, state = _channel(case, seed)
            p, H, dzr, taux = s.params, s.H, s.dzr, None
        else:
            p, H, dzr, taux = _basin(case["nx"], case["ny"], case["nz"], seed, **_step_params(case))
            state = _state(p, H, dzr, seed, mixed_layer=case["closure"] == "tke")
        st = OceanStepper(p, H, np.ones_like(H), dzr=dzr, taux_c=taux, precision=case["precision"])
        return {"kind": kind, "st": st, "state": state, "out": _buffers(p), "steps": case["steps"],
                "graph": case["graph"]}
    if kind == "ensemble":
        rng = np.random.default_rng(seed + 5)
        members, states, outs = [], [], []
        # the members' sizes belong to the case (a seed changes their fields, not their work)
        sizes = np.random.default_rng(1000 * case["members"] + case["hi"]).integers(case["lo"], case["hi"] + 1,
                                                                                   (case["members"], 2))
        for ix, iy in sizes:
            s = int(rng.integers(1 << 30))
            p, H, dzr, taux = _basin(32 * int(ix), 32 * int(iy), case["nz"], s, dt=300.0)
            members.append(OceanStepper(p, H, np.ones_like(H), dzr=dzr, taux_c=taux))
            states.append(_state(p, H, dzr, s))
            outs.append({k: v for k, v in _buffers(p).items() if k in ("eta", "u", "v", "T", "S", "e")})
            members[-1].set_state(**states[-1])
        return {"kind": kind, "members": members, "ens": OceanEnsemble(members), "states": states, "outs": outs,
                "steps": case["steps"]}
    if kind == "adjoint":
        p, H, dzr, taux = _basin(case["nx"], case["ny"], case["nz"], seed, closure="none", dt=300.0,
                                 solver_kind="pcg_jacobi" if case["nx"] % 16 or case["ny"] % 16 else "multigrid")
        if p.solver_kind == "pcg_jacobi":
            p = p.replace(dt=4.0 * CELL / math.sqrt(2.0 * 9.80616 * 4000.0))
        state = _state(p, H, dzr, seed, mixed_layer=False)
        g = _rng(seed + 1)
        weights = torch.randn(state["T"].shape, generator=g, device=DEV, dtype=torch.float64)
        ro = OceanRollout(p, H, np.ones_like(H), dzr=dzr, n_steps=case["steps"], every=5)
        return {"kind": kind, "ro": ro, "state": state, "taux": torch.from_numpy(taux).to(DEV), "weights": weights}
    if kind == "helmholtz":
        return {"kind": kind, "helm": _Helm(case, seed)}
    if kind == "density":
        g = _rng(seed)
        T, S, z = (torch.rand(case["n"], generator=g, device=DEV, dtype=torch.float64) for _ in range(3))
        T, S, z = 30.0 * T, 30.0 + 10.0 * S, 5000.0 * z
        return {"kind": kind, "lib": _lib.load(), "in": (T, S, z), "rho": torch.empty_like(T), "n": case["n"],
                "eos": case["eos"]}
    ins = tuple(t.contiguous() for t in _thomas_inputs(case, seed))
    return {"kind": kind, "lib": _lib.load(), "in": ins, "x": torch.empty_like(ins[3]), "n": case["n"],
            "ncols": case["ncols"]}


# ------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    stream = torch.cuda.current_stream()
    if kind == "step":
        st = state["st"]
        st.set_state_async(stream, **state["state"])
        st.step(state["steps"], stream=stream, graph=state["graph"])
        st.get_state_async(stream, state["out"])
        return state["out"]
    if kind == "ensemble":
        for st, s in zip(state["members"], state["states"]):
            st.set_state_async(stream, **s)
        state["ens"].step(state["steps"], stream=stream)
        for st, o in zip(state["members"], state["outs"]):
            st.get_state_async(stream, o)
        return state["outs"]
    if kind == "adjoint":
        T0 = state["state"]["T"].detach().requires_grad_(True)
        taux = state["taux"].detach().requires_grad_(True)
        out = rollout_apply(state["ro"], T0, taux, state["state"])
        objective = (out["T"] * state["weights"]).sum() + (out["eta"] ** 2).sum()
        gT, gtau = torch.autograd.grad(objective, (T0, taux))
        return {"gT": gT, "gtau": gtau, "final": {k: v.detach() for k, v in out.items()}}
    if kind == "helmholtz":
        return state["helm"].solve()
    if kind == "density":
        T, S, z = state["in"]
        _lib.check(state["lib"].oc_density(state["eos"], 1025.0, 2.0e-4, 7.4e-4, 10.0, 35.0, T.data_ptr(),
                                           S.data_ptr(), z.data_ptr(), state["rho"].data_ptr(), state["n"],
                                           stream.cuda_stream), None, "oc_density")
        return state["rho"]
    sub, diag, sup, rhs = state["in"]
    _lib.check(state["lib"].oc_thomas(sub.data_ptr(), diag.data_ptr(), sup.data_ptr(), rhs.data_ptr(),
                                      state["x"].data_ptr(), state["n"], state["ncols"], stream.cuda_stream), None,
               "oc_thomas")
    return state["x"]


# ------------------------------------------------------------------ what a pass cannot do without
def _step_work(cells, columns, steps, word, closure, solves):
    """Per step: the prognostic fields read and written once (u, v, T, S; the buoyancy in
    fp64; with a closure e, K_m and K_h too), the surface and its elliptic system once per
    solve; about 700 operations per cell (two TVD momentum fields and two tracers, their
    column solves, the EOS) and 300 more for the closure."""
    fields = 2 * 4 * word + 2 * 8 + (2 * 3 * word if closure else 0)
    return {"bytes": steps * (cells * fields + columns * 8 * (2 + 6 * solves)),
            "flops": steps * (cells * (700 + (300 if closure else 0)) + columns * 100 * solves)}


def work(case):
    kind = case["kind"]
    if kind == "step":
        cols = case["nx"] * case["ny"]
        return _step_work(cols * case["nz"], cols, case["steps"], 4 if case["precision"] == "mixed" else 8,
                          case["closure"] == "tke", 2 if case["scheme"] == "theta" else 0)
    if kind == "ensemble":
        sizes = np.random.default_rng(1000 * case["members"] + case["hi"]).integers(case["lo"], case["hi"] + 1,
                                                                                   (case["members"], 2))
        cols = int(sum(1024 * int(a) * int(b) for a, b in sizes))
        return _step_work(cols * case["nz"], cols, case["steps"], 8, True, 2)
    if kind == "adjoint":
        cols = case["nx"] * case["ny"]
        w = _step_work(cols * case["nz"], cols, case["steps"], 8, False, 2)
        # the forward run, the segment's recomputation, and the adjoint steps (about two steps' work)
        return {"bytes": 4 * w["bytes"], "flops": 4 * w["flops"]}
    if kind == "helmholtz":
        n = case["nx"] * case["ny"]
        return {"bytes": 5 * 8 * n, "flops": 25 * 25 * n}  # K_u, K_v, mask, rhs in, x out; about 25 iterations
    if kind == "density":
        return {"bytes": 32 * case["n"], "flops": (6, 20, 110)[case["eos"]] * case["n"]}
    n = case["n"] * case["ncols"]
    return {"bytes": 40 * n, "flops": 9 * n}


def tolerance(case):
    """The fp64 paths give NumPy's bits, so their outputs do not change at all."""
    kind = case["kind"]
    if kind == "adjoint":
        # its transposed stencils add with fp64 atomics, in an order that changes from run to run:
        # two runs on the same inputs were 6e-7 apart (2.5e-5 at the worst value)
        return {"rel": 2.5e-6, "max": 1.0e-4}
    if kind == "step" and case["precision"] == "mixed":
        # FP32 state: another order of an FP32 expression moves the fields by their rounding,
        # which the limiters and the closure's clips carry on
        return {"rel": 2.0e-4, "max": 0.3}
    if kind == "helmholtz" and case["solver"] == "pcg_refined":
        return {"rel": 4.0 * case["rtol"], "max": 400.0 * case["rtol"], "differ": 0.0}
    return "exact"


# ------------------------------------------------------------------ the same in 64 bits, without the package
def _density64(eos, T, S, z):
    """The published polyTEOS10-bsq, the simplified EOS and the linear one (Roquet et al. 2015)."""
    if eos == 0:
        return 1025.0 * (-2.0e-4 * (T - 10.0) + 7.4e-4 * (S - 35.0))
    if eos == 1:
        Ta, Sa = T - 10.0, S - 35.0
        return (-1.6550e-1 * (1.0 + 0.5 * 5.9520e-2 * Ta + 1.4970e-4 * z) * Ta
                + 7.6554e-1 * (1.0 - 0.5 * 7.4914e-4 * Sa - 1.1090e-5 * z) * Sa - 2.4341e-3 * Ta * Sa)
    zh, ss, tt = z * 1.0e-4, torch.sqrt((S + 32.0) * (0.875 / 35.16504)), T * 0.025

    def horner(x, *c):  # highest power first
        acc = torch.zeros_like(x) + c[0]
        for a in c[1:]:
            acc = acc * x + a
        return acc

    r0 = horner(zh, -1.7243708991e-03, 1.5616995503e-02, 6.4326772569e-02, 2.2601900708e-01, -5.2099962525e+00,
                4.6494977072e+01, 0.0)
    rz3 = 3.7969820455e-01 * tt - 1.8507636718e-02 * ss - 2.3342758797e-02
    rz2 = horner(tt, -1.2419983026e+00, -2.1311365518e-01 * ss + 2.0564311499e+00,
                 horner(ss, 2.5019633803e+00, -4.9527603989e+00, 2.0660924175e+00))
    rz1 = horner(tt, 5.5927935970e-01, -5.5077101279e-01 * ss - 2.4649669534e+00,
                 horner(ss, -1.8795372996e+00, 3.5063081279e+00, 6.7080479603e+00),
                 horner(ss, -6.5399043664e-01, 5.0042598061e+00, -4.4870114575e+00, -1.3336301113e+01),
                 horner(ss, 6.6051753097e+00, -3.0938076334e+01, 5.0774768218e+01, -4.2549998214e+01,
                        1.9681925209e+01))
    rz0 = horner(tt, -1.9098268277e-01, 4.5111434961e-01 * ss + 5.4048723791e-01,
                 horner(ss, -5.3563304045e+00, 1.1311538584e+01, -8.3627885467e+00),
                 horner(ss, -3.1742946532e+00, 1.9717078466e+01, -3.3449108469e+01, 2.1661789529e+01),
                 horner(ss, -5.4723692739e+00, 2.9130021253e+01, -6.0362551501e+01, 6.1548258127e+01,
                        -3.7074170417e+01),
                 horner(ss, -1.9193502195e+00, 1.7681814114e+01, -5.6888046321e+01, 8.1770425108e+01,
                        -6.5281885265e+01, 2.6010145068e+01),
                 horner(ss, -6.0579916612e+01, 4.3227585684e+02, -1.2849161071e+03, 2.0375295546e+03,
                        -1.7864682637e+03, 8.6672408165e+02, 8.0189615746e+02))
    return ((rz3 * zh + rz2) * zh + rz1) * zh + rz0 + r0


def _helmholtz64(case, seed):
    """The system's solution by conjugate gradients to the last digits."""
    dx, coef, ku, kv, mask, rhs = (torch.from_numpy(a).to(DEV) if isinstance(a, np.ndarray) else a
                                   for a in _solver_handle(case, seed))

    def A(x):
        fx = ku * (torch.roll(x, -1, 1) - x)
        fy = kv * (torch.roll(x, -1, 0) - x)
        return x - coef / (dx * dx) * (fx - torch.roll(fx, 1, 1) + fy - torch.roll(fy, 1, 0))

    b = rhs * mask
    x, r = torch.zeros_like(b), b.clone()
    p, rr = r.clone(), float((b * b).sum())
    stop = 1.0e-32 * rr
    for _ in range(400):
        q = A(p)
        alpha = rr / float((p * q).sum())
        x, r = x + alpha * p, r - alpha * q
        new = float((r * r).sum())
        if new <= stop:
            break
        p, rr = r + (new / rr) * p, new
    return {"x": x, "iterations": None, "converged": None}


def _thomas64(case, seed):
    sub, diag, sup, rhs = _thomas_inputs(case, seed)
    c, d = [sup[0] / diag[0]], [rhs[0] / diag[0]]
    for k in range(1, case["n"]):
        den = diag[k] - sub[k] * c[-1]
        c.append(sup[k] / den)
        d.append((rhs[k] - sub[k] * d[-1]) / den)
    x = [d[-1]]
    for k in range(case["n"] - 2, -1, -1):
        x.append(d[k] - c[k] * x[-1])
    return torch.stack(x[::-1])


def exact(case, seed):
    """A whole model step, its ensemble and its adjoint have no short plain form; their fp64
    outputs are compared bit for bit instead."""
    kind = case["kind"]
    if kind == "density":
        g = _rng(seed)
        T, S, z = (torch.rand(case["n"], generator=g, device=DEV, dtype=torch.float64) for _ in range(3))
        return _density64(case["eos"], 30.0 * T, 30.0 + 10.0 * S, 5000.0 * z)
    if kind == "helmholtz":
        return _helmholtz64(case, seed)
    if kind == "thomas":
        return _thomas64(case, seed)
    return None
