"""What a user of this solver has it do, through the public entry points: the
cases its speed is measured on, over the range of sizes that real surveys have.

The solves.  A survey program holds one handle per mesh
(maple3dmt_gb300.solver.ForwardSolverFV) and calls it once per model: new
conductivity in (set_sigma), impedances, fields and gradients out.  The
handle is what such a program keeps, so one handle per mesh and parameter set
is shared here by every state on that mesh, and each pass sets its own state's
conductivity first; the models, data and sources come from the seed.  The
mixed-precision solver (precision=1, what the benchmark and the integration
notes run) is used at every size, the library's default all-FP64 solver on the
small mesh.

Tolerance.  The solves stop at a relative true residual of 1e-12 instead of the
1e-7 of a field inversion: gradients checked against finite differences and
comparisons between codes need tight solves (the repository's own checks run
1e-10 and less), and at 1e-12 the returned FP64 numbers are determined by the
problem and no longer by the path the iteration took.  The kernels and their
shares are the same as at 1e-7, with one or two more refinement steps.

Meshes: the uniform-halfspace mesh of the repository (levels 3/5) and the
layered-earth survey meshes at levels 4/5 to 6/7 (about 20 k to 1.7 M edges).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from maple3dmt_gb300 import mesh, workloads
from maple3dmt_gb300.learned import Cnn
from maple3dmt_gb300.solver import solver_for_survey

TOL = 1e-12
MAXITER = 20000


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------

def _survey(what, lo, hi, side, nf, fmin, fmax, **more):
    return {"what": what, "lo": lo, "hi": hi, "side": side, "nf": nf, "fmin": fmin, "fmax": fmax, **more}


def listed():
    return [
        # inner product of two short device vectors for two systems: a latency-bound call
        {"name": "dot-small", "what": "dot", "n": 4099, "K": 2},
        # the same for 16 systems on the edges of the benchmark mesh: pure bandwidth
        {"name": "dot-large", "what": "dot", "n": 1687305, "K": 16},
        # model regularisation of one inversion step on the benchmark mesh:
        # objective and gradient, W^T W x, CmCm^T x (host vectors in and out)
        {"name": "regularisation", **_survey("reg", 6, 7, 11, 8, 0.01, 100.0)},
        # one frequency on the small halfspace mesh, the library's default FP64 solver
        {"name": "forward-small-fp64", "what": "single", "half": True, "lo": 3, "hi": 5, "side": 5, "nf": 1,
         "fmin": 1.0, "fmax": 1.0, "precision": 0},
        # one frequency on a small survey mesh (a quick look at a model): latency and launches count
        {"name": "forward-small", **_survey("single", 4, 5, 5, 1, 0.5, 0.5, precision=1)},
        # forward modelling of a survey with the fields read back, five frequencies
        {"name": "forward-fields", **_survey("forward", 5, 6, 7, 5, 0.01, 100.0, precision=1)},
        # many right-hand sides at one frequency (an odd number), as a Jacobian build asks for them
        {"name": "many-rhs", **_survey("rhs", 5, 6, 7, 1, 0.3, 0.3, precision=1, nrhs=11)},
        # data misfit gradient of an inversion step, mid-size mesh two levels deep, three frequencies
        {"name": "gradient-mid", **_survey("gradient", 5, 7, 9, 3, 0.03, 30.0, precision=1)},
        # the same on the benchmark mesh (1.7 M edges), four frequencies over its range
        {"name": "gradient-large", **_survey("gradient", 6, 7, 11, 4, 0.01, 100.0, precision=1)},
        # forward solve and per-station gradients of one frequency, three station sources
        {"name": "station-gradients", **_survey("stations", 5, 7, 11, 1, 1.0, 1.0, precision=1, nsrc=3)},
        # Gauss-Newton: background fields and one J^T W^2 J v product, two frequencies
        {"name": "gauss-newton", **_survey("gn", 5, 6, 7, 2, 0.1, 10.0, precision=1)},
        # the learned preconditioner's network on one batch: forward pass and all gradients
        {"name": "network", "what": "cnn", "n": 4, "grid": 32},
    ]


def draw(rng):
    what = rng.choice(["dot", "reg", "single", "forward", "rhs", "gradient", "gradient", "stations", "gn", "cnn"])
    if what == "dot":
        return {"what": what, "n": int(round(4096 * 2.0 ** rng.uniform(0.0, 8.7))), "K": rng.choice([2, 4, 8, 16])}
    if what == "cnn":
        return {"what": what, "n": rng.randint(1, 4), "grid": rng.choice([16, 32])}
    lo, hi = rng.choice([(4, 5), (4, 6), (5, 6), (5, 7)])
    side = rng.randint(4, 11)
    fmin = round(10.0 ** rng.uniform(-2.0, 0.0), 5)
    if what in ("single", "rhs", "stations"):
        c = _survey(what, lo, hi, side, 1, fmin, fmin, precision=1)
    else:
        fmax = round(fmin * 10.0 ** rng.uniform(1.0, 3.0), 5)
        nf = rng.randint(2, 4) if what == "gn" else rng.randint(1, 8)
        c = _survey(what, lo, hi, side, nf, fmin, fmax if nf > 1 else fmin, precision=1)
    if what == "rhs":
        c["nrhs"] = rng.randint(1, 20)
    if what == "stations":
        c["nsrc"] = rng.randint(1, 9)
    if what == "reg":
        del c["precision"]
    return c


# --------------------------------------------------------------------------
# meshes and handles
# --------------------------------------------------------------------------

_surveys: dict = {}
_handles: dict = {}


def _freqs(case):
    if case["nf"] == 1:
        return np.array([case["fmin"]])
    return np.logspace(math.log10(case["fmin"]), math.log10(case["fmax"]), case["nf"])


def _mesh_key(case):
    return (bool(case.get("half")), case["lo"], case["hi"], case["side"], case["nf"], case["fmin"], case["fmax"])


def _mesh(case):
    key = _mesh_key(case)
    if key not in _surveys:
        if key[0]:
            sv = mesh.halfspace_survey(min_level=case["lo"], max_level=case["hi"], n_side=case["side"],
                                       freqs=_freqs(case))
        else:
            sv = mesh.layered_block_survey(min_level=case["lo"], max_level=case["hi"], n_side=case["side"],
                                           freqs=_freqs(case))
        _surveys[key] = sv
    return _surveys[key]


def _handle(case):
    """The handle a program keeps for this mesh; the three used last are held."""
    key = (_mesh_key(case), case.get("precision", 1))
    s = _handles.pop(key, None)
    if s is None:
        while len(_handles) >= 3:
            _handles.pop(next(iter(_handles))).close()
        s = solver_for_survey(_mesh(case), bicgstab_tol=TOL, bicgstab_maxiter=MAXITER,
                              precision=case.get("precision", 1))
        if case["what"] == "reg":
            s.reg_setup()
    _handles[key] = s
    return s


def _model(sv, rng):
    """The survey's earth with a random log-conductivity perturbation (std 0.3) of its earth cells."""
    sig = np.array(sv.sigma, copy=True)
    earth = sv.leaves.cell_type == 0
    sig[earth] *= 10.0 ** rng.normal(0.0, 0.3, int(earth.sum()))
    return sig


def _weights(rng):
    """Weights of the 6-layer network (8 -> 32 -> ... -> 6 channels), laid out
    [layer][tap][out][in] and zero-padded to 32 channels, as read from a file."""
    w = np.zeros((6, 27, 32, 32), np.float32)
    b = np.zeros((6, 32), np.float32)
    for l, (ci, co) in enumerate([(8, 32)] + 4 * [(32, 32)] + [(32, 6)]):
        w[l, :, :co, :ci] = rng.normal(0.0, math.sqrt(2.0 / (27 * ci)), (27, co, ci))
        b[l, :co] = rng.normal(0.0, 0.01, co)
    return w, b


# --------------------------------------------------------------------------
# prepare, run
# --------------------------------------------------------------------------

def prepare(case, seed):
    rng = np.random.default_rng([seed, 17])
    st = {"case": case, "what": case["what"]}
    if case["what"] == "dot":
        g = torch.Generator(device="cuda").manual_seed(seed)
        shape = (case["n"], case["K"], 2)
        st["x"] = torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)
        st["y"] = torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)
        st["out"] = torch.zeros((case["K"], 2), device="cuda", dtype=torch.float64)
        small = {"what": "dot", "half": True, "lo": 3, "hi": 5, "side": 5, "nf": 1, "fmin": 1.0, "fmax": 1.0}
        st["solver"] = _handle(small)
        torch.cuda.synchronize()
        return st
    if case["what"] == "cnn":
        net = Cnn(layers=6, c_in=8, hidden=32, c_out=6)
        net.set_weights(*_weights(rng))
        shape = (case["n"],) + (case["grid"],) * 3
        st["net"] = net
        st["x"] = rng.standard_normal(shape + (8,), dtype=np.float32)
        st["dy"] = rng.standard_normal(shape + (6,), dtype=np.float32)
        return st
    sv = _mesh(case)
    st["solver"] = _handle(case)
    st["freqs"] = _freqs(case)
    ns, nf = len(sv.stations), case["nf"]
    st["sigma"] = _model(sv, rng)
    if case["what"] == "reg":
        na = st["solver"].n_active
        st["x"] = rng.normal(size=na)
        st["ref"] = np.full(na, math.log(0.01))
    elif case["what"] in ("gradient", "gn"):
        st["obs"], st["err"] = workloads.halfspace_data(sv.stations, st["freqs"], seed=seed)
        st["dsigma"] = st["sigma"] * rng.normal(0.0, 0.1, len(st["sigma"]))
    elif case["what"] == "stations":
        st["wr"] = workloads.station_sources(ns, rng)[rng.choice(ns, size=case["nsrc"], replace=False)]
    elif case["what"] == "rhs":
        ne = st["solver"].ne
        b = np.zeros((case["nrhs"], ne), np.complex128)
        for row in b:   # a source on a few edges of the survey, as a Jacobian column has
            at = rng.choice(ne, size=64, replace=False)
            row[at] = rng.normal(size=64) + 1j * rng.normal(size=64)
        st["b"] = b
    return st


def run(st):
    what, s = st["what"], st.get("solver")
    if what == "dot":
        s.dot_batched(st["x"].data_ptr(), st["y"].data_ptr(), st["case"]["n"], st["case"]["K"], st["out"].data_ptr())
        return st["out"]
    if what == "cnn":
        y = st["net"].forward(st["x"])
        dw, db, dx = st["net"].backward(st["x"], st["dy"])
        return {"y": y, "dw": dw, "db": db, "dx": dx}
    if what == "reg":
        v, g = s.reg_evaluate(np.log(st["sigma"]), st["ref"])
        return {"value": v, "grad": g, "wtw": s.reg_apply_wtw(st["x"]), "cmcmt": s.reg_apply_cmcmt(st["x"])}
    s.set_sigma(st["sigma"])
    f = st["freqs"]
    if what == "single":
        Z = s.compute_single_frequency(f[0])
        return {"Z": Z, "E1": s.background_E(0), "E2": s.background_E(1)}
    if what == "forward":
        Z, E = s.forward_batch(f, with_fields=True)
        return {"Z": Z, "E": E}
    if what == "rhs":
        s.factorize_frequency(f[0])
        return {"x": s.solve_rhs_batch(st["b"])}
    if what == "gradient":
        Z, g = s.gradient_batch(f, st["obs"], st["err"])
        return {"Z": Z, "g": g}
    if what == "stations":
        Z = s.compute_single_frequency(f[0])
        return {"Z": Z, "g": s.station_gradients(st["wr"])}
    Z = s.forward_batch(f)   # Gauss-Newton
    return {"Z": Z, "JtJv": s.jtjv_batch(f, st["dsigma"], st["err"], inner_tol=TOL)}


# --------------------------------------------------------------------------
# work, exact
# --------------------------------------------------------------------------

def work(case):
    if case["what"] == "dot":
        n, K = case["n"], case["K"]
        return {"bytes": 32.0 * n * K + 16 * K, "flops": 8.0 * n * K}
    if case["what"] == "cnn":
        vox = case["n"] * case["grid"] ** 3
        macs = vox * 27.0 * (8 * 32 + 4 * 32 * 32 + 32 * 6)
        # forward, then the backward pass with its own forward: one pass for
        # the activations, one for the input and one for the weight gradients
        return {"bytes": 4.0 * vox * (8 + 6 + 8 + 6 + 8) + 2 * 4.0 * 6 * (27 * 32 * 32 + 32), "flops": 2.0 * 4 * macs}
    nc = _mesh(case).leaves.n_cells
    ne = 3.1 * nc   # edges of an octree mesh, near enough
    if case["what"] == "reg":
        # ln sigma in, gradient out, four active-cell vectors; the face adjacency
        # (six neighbours, index and weight) once per operator
        return {"bytes": 8.0 * nc * 7 + 3 * 12.0 * 6 * nc, "flops": 2.0 * 7 * 5 * nc}
    fwd = 2 * case["nf"]
    more = {"single": 0, "forward": 0, "rhs": case.get("nrhs", 0) - fwd, "gradient": fwd,
            "stations": 2 * case.get("nsrc", 0), "gn": 2 * fwd}[case["what"]]
    n_rhs = fwd + more
    # per right-hand side one source read and one field written; the operator
    # (12 off-diagonal entries a row, value and column, and the diagonal pair) once
    # a batch of 16; one product per right-hand side as the least arithmetic
    batches = -(-n_rhs // 16)
    return {"bytes": ne * (32.0 * n_rhs + batches * (12 * 12.0 + 16)) + 24.0 * nc, "flops": ne * n_rhs * (12 * 4.0 + 8)}


def exact(case, seed):
    """In FP64: the inner products, and the network's forward values; the solves have no reference outside this package."""
    if case["what"] == "dot":
        st = {}
        g = torch.Generator(device="cuda").manual_seed(seed)
        shape = (case["n"], case["K"], 2)
        for k in ("x", "y"):
            st[k] = torch.view_as_complex(torch.randn(shape, generator=g, device="cuda", dtype=torch.float64))
        return torch.view_as_real((st["x"].conj() * st["y"]).sum(0))
    if case["what"] == "cnn":
        rng = np.random.default_rng([seed, 17])
        w, b = _weights(rng)
        x = rng.standard_normal((case["n"],) + (case["grid"],) * 3 + (8,), dtype=np.float32)
        x = torch.from_numpy(x).cuda().double().permute(0, 4, 1, 2, 3)
        w, b = torch.from_numpy(w).cuda().double(), torch.from_numpy(b).cuda().double()
        for l, (ci, co) in enumerate([(8, 32)] + 4 * [(32, 32)] + [(32, 6)]):
            k = w[l, :, :co, :ci].permute(1, 2, 0).reshape(co, ci, 3, 3, 3)
            x = torch.nn.functional.conv3d(x, k, b[l, :co], padding=1)
            if l < 5:
                x = x.relu()
        return {"y": x.permute(0, 2, 3, 4, 1).contiguous(), "dw": None, "db": None, "dx": None}
    return None
