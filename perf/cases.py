"""Performance cases: what a program built on this framework has it do, through the public entry
points (``caffe_old_b200.solver``, ``precond`` and the C ABI's Krylov solves).

Families, by the field "do":

* ``step``   time steps / outer iterations of a flow solver (Simple, Piso, IbPiso) in each form of
             its pressure solve (plain FP64, mixed precision, learned preconditioner): a pass loads a
             restart state from pinned host memory, advances ``steps`` steps and reads u and p back.
* ``psolve`` one pressure-correction solve of the time loop (the phase "solve_pcorr" of a handle whose
             system is assembled), solution read back: what dominates a step of the largest lattices.
* ``ksp7``   the stand-alone Krylov solve of a 7-point system held in device memory.
* ``csr``    SparseMatrix::solve: a compressed-row system handed over in host memory.
* ``train``  optimiser steps of the preconditioner network on stored pairs: forward, backward, weight
             gradient and update.

Linear solves of the PISO flows run to the 1e-8 of the benchmark configurations (their correctors
leave the fields much closer than that), with the round-off floor of the cavities' second corrector
as the absolute tolerance.  SIMPLE takes one correction per iteration, so its solves run to 1e-11:
fields of two builds then agree to well below the 1e-8 that a solve's tolerance would leave.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from caffe_old_b200 import _lib, cases as C, precond as P
from caffe_old_b200.solver import make_solver

# Arrays that make up a restart state: everything a step reads that it does not form itself.
RESTART = ("u", "p", "gradP", "massFlowI", "massFlowJ", "massFlowK") + tuple(f"pPatch{f}" for f in range(6))
# Field bytes of one cell that a step reads and writes once: u, p, grad p, d and three face fluxes.
STEP_BYTES = 2 * 8 * (3 + 1 + 3 + 1 + 3)


def listed():
    return [
        # the SIMPLE configuration of the 2-D cavity (Re 100): small systems, the latency of a solve's iterations
        dict(name="simple_2d_64", do="step", flow="simple2d", nI=64, nJ=64, nK=1, form="fp64", steps=5),
        # the same on a ragged, larger 2-D lattice
        dict(name="simple_2d_210x130", do="step", flow="simple2d", nI=210, nJ=130, nK=1, form="fp64", steps=2),
        # a coarse 3-D cavity as a parameter study runs it: PISO, Jacobi-CG
        dict(name="piso_3d_28x24x20", do="step", flow="piso", nI=28, nJ=24, nK=20, form="fp64", steps=4),
        # the 3-D PISO cavity configuration (128^3, Re 400): the plain FP64 form at production size
        dict(name="piso_3d_128", do="step", flow="piso", nI=128, nJ=128, nK=128, form="fp64", steps=2),
        # the skewed cavity configuration: non-orthogonal terms and the mixed-precision pressure solve
        dict(name="skewed_mixed_128", do="step", flow="skewed", nI=128, nJ=128, nK=128, form="mixed", steps=2),
        # the immersed sphere in plain FP64 (BiCGStab, ghost rows) on the benchmark's host-comparison lattice
        dict(name="ib_fp64_72x48x48", do="step", flow="ib", nI=72, nJ=48, nK=48, form="fp64", steps=1),
        # the same flow, mixed precision, odd sizes
        dict(name="ib_mixed_75x39x41", do="step", flow="ib", nI=75, nJ=39, nK=41, form="mixed", steps=1),
        # the immersed sphere with the learned preconditioner: a whole step at 3.1M cells
        dict(name="ib_learned_192x128x128", do="step", flow="ib", nI=192, nJ=128, nK=128, form="learned_mixed", steps=1),
        # one pressure solve of the benchmark's 25.2M-cell sphere, learned preconditioner
        dict(name="ib_psolve_384x256x256", do="psolve", flow="ib", nI=384, nJ=256, nK=256, form="learned_mixed"),
        # a caller's own symmetric 7-point system in device memory, ragged
        dict(name="ksp7_cg_101x67x53", do="ksp7", nI=101, nJ=67, nK=53, method="cg_jacobi"),
        # SparseMatrix::solve from host rows (the reference's 2-D systems)
        dict(name="csr_bicgstab_90x70", do="csr", nI=90, nJ=70, method="bicgstab_jacobi"),
        # fine-tuning the shipped preconditioner network on a new, smaller case
        dict(name="train_128x64x64", do="train", flow="ib", nI=128, nJ=64, nK=64, steps=2, batch=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sphere_lattice(rng, lo, hi):
    """A lattice of the 8x4x4 box with nJ in [lo, hi]; its cell centres are off the planes through the
    sphere's centre (where the search for the cells around an image point ends on round-off) and
    the cell count is a multiple of 4."""
    nJ = 2 * _log_int(rng, lo / 2, hi / 2)
    nI = int(nJ * rng.uniform(1.3, 1.5))
    return dict(flow="ib", nI=nI + 1 if nI % 4 == 2 else nI, nJ=nJ, nK=max(lo, nJ - 2 * rng.randrange(4)))


def draw(rng):
    do = rng.choice(["step"] * 7 + ["psolve", "ksp7", "csr", "train"])
    if do == "psolve":
        return dict(do="psolve", form="learned_mixed", **_sphere_lattice(rng, 48, 256))
    if do == "ksp7":
        return dict(do="ksp7", nI=_log_int(rng, 8, 160), nJ=_log_int(rng, 8, 128), nK=_log_int(rng, 1, 100),
                    method=rng.choice(["cg_jacobi", "bicgstab_jacobi"]))
    if do == "csr":
        return dict(do="csr", nI=_log_int(rng, 10, 240), nJ=_log_int(rng, 10, 160), method=rng.choice(["cg_jacobi", "bicgstab_jacobi"]))
    if do == "train":
        return dict(do="train", steps=rng.choice([1, 2, 3]), batch=rng.choice([2, 4]), **_sphere_lattice(rng, 40, 80))
    flow = rng.choice(["simple2d", "piso", "skewed", "ib", "ib"])
    if flow == "simple2d":
        return dict(do="step", flow=flow, nI=_log_int(rng, 16, 256), nJ=_log_int(rng, 16, 160), nK=1, form="fp64", steps=rng.choice([1, 2, 4]))
    if flow in ("piso", "skewed"):
        n = [_log_int(rng, 10, 128) for _ in range(3)]
        return dict(do="step", flow=flow, nI=n[0], nJ=n[1], nK=n[2], form="fp64" if flow == "piso" else rng.choice(["mixed", "fp64"]), steps=rng.choice([1, 2]))
    form = rng.choice(["fp64", "mixed", "learned_mixed"])
    return dict(do="step", form=form, steps=1, **_sphere_lattice(rng, 40, 128 if form == "learned_mixed" else 52))


def _flow_case(case, seed):
    """Nodes and case of a flow: the repository's configurations with the viscosity from the seed."""
    dims = (case["nI"], case["nJ"], case["nK"])
    scale = float(np.random.default_rng(seed).uniform(0.8, 1.25))
    flow, form = case["flow"], case.get("form", "fp64")
    if flow == "simple2d":
        _, spec, _ = C.config1_cavity2d(8)
        nodes = C.cartesian_nodes(dims, (1.0, dims[1] / dims[0], 1.0 / dims[0]))
        spec = spec.replace(mom_rtol=1e-11, p_rtol=1e-11, p_atol=1e-17)
    elif flow == "piso":
        _, spec, _ = C.config2_cavity3d(8)
        nodes = C.cartesian_nodes(dims, (1.0, 1.0, 1.0))
        spec = spec.replace(p_atol=1e-16)
    elif flow == "skewed":
        _, spec, _ = C.config3_skewed(8)
        nodes = C.skewed_nodes(dims, (1.0, 1.0, 1.0), 30.0, 0.1, seed)
        spec = spec.replace(p_atol=1e-16)
    else:
        _, spec, _ = C.config5_sphere((8, 8, 8), re=300.0)
        nodes = C.cartesian_nodes(dims, (8.0, 4.0, 4.0))
    return nodes, spec.replace(mu=spec.mu * scale, p_form=form)


def _make_flow(case, seed):
    nodes, spec = _flow_case(case, seed)
    s = make_solver(nodes, spec)
    if case.get("form") == "learned_mixed":
        # the benchmark's settings of the shipped network: levels from 2 on, short FGMRES cycles
        P.set_params(s, P.load_default())
        P.set_mode(s, "network")
        last = min(P.trained_last_level(), len(P.pyramid_dims(s.shape)) - 1)
        P.set_options(s, "auto", 2, 5)
        P.set_net_levels(s, 2, max(last, 2))
    return s


def _start_velocity(case, seed):
    """A smooth seeded motion, one plane per component (zero on the walls of a cavity; the
    immersed-boundary flows start at the inlet velocity with a small disturbance)."""
    nI, nJ, nK = case["nI"], case["nJ"], case["nK"]
    rng = np.random.default_rng(seed + 1)
    x = [(np.arange(n) + 0.5) / n for n in (nI, nJ, nK)]
    u = np.zeros((3, nK, nJ, nI))
    for q in range(2 if nK == 1 else 3):
        a = rng.uniform(-0.05, 0.05, size=3)
        for m in range(3):
            f = [np.sin(np.pi * (m + 1 + (d == q)) * x[d]) if n > 1 else np.ones(1) for d, n in enumerate((nI, nJ, nK))]
            u[q] += a[m] * f[0][None, None, :] * f[1][None, :, None] * f[2][:, None, None]
    if case["flow"] == "ib":
        u *= 0.1
        u[0] += 1.0
    return u


def _pinned(n):
    return torch.zeros(int(n), dtype=torch.float64, pin_memory=True)


def _prepare_flow(case, seed):
    s = _make_flow(case, seed)
    restart = {name: _pinned(s.size_of(name)) for name in RESTART}
    restart["u"].copy_(torch.from_numpy(_start_velocity(case, seed).reshape(-1)))
    return s, restart


def _load(s, restart):
    for name, v in restart.items():
        s.set_from_ptr(name, v.data_ptr(), v.numel())


def _seven_point(dims, seed):
    """A symmetric 7-point diffusion system with seeded smooth coefficients and walls at fixed value
    on three sides, a known solution and its right-hand side (device tensors)."""
    nI, nJ, nK = dims
    g = torch.Generator(device="cuda").manual_seed(seed)
    ax = [torch.arange(n, dtype=torch.float64, device="cuda") / n for n in (nK, nJ, nI)]
    ph = torch.rand(6, generator=g, device="cuda", dtype=torch.float64) * 6.28
    k = 1.0 + 0.4 * torch.sin(6.28 * ax[0] + ph[0])[:, None, None] * torch.cos(6.28 * ax[1] + ph[1])[None, :, None] * torch.sin(6.28 * ax[2] + ph[2])[None, None, :]
    z = torch.zeros_like(k)
    aE, aN, aT = z.clone(), z.clone(), z.clone()
    aE[:, :, :-1] = 0.5 * (k[:, :, 1:] + k[:, :, :-1])
    aN[:, :-1, :] = 0.5 * (k[:, 1:, :] + k[:, :-1, :])
    aT[:-1] = 0.5 * (k[1:] + k[:-1])
    aW, aS, aB = z.clone(), z.clone(), z.clone()
    aW[:, :, 1:], aS[:, 1:, :], aB[1:] = aE[:, :, :-1], aN[:, :-1, :], aT[:-1]
    wall = z.clone()
    wall[:, :, 0] += 2.0 * k[:, :, 0]
    wall[:, 0, :] += 2.0 * k[:, 0, :]
    wall[0] += 2.0 * k[0] if nK > 1 else 0.0
    aP = -(aE + aW + aN + aS + aT + aB + wall)
    x = torch.sin(3.0 * ax[0] + ph[3])[:, None, None] * torch.cos(4.0 * ax[1] + ph[4])[None, :, None] * torch.sin(5.0 * ax[2] + ph[5])[None, None, :]
    x = x + 0.01 * torch.randn(x.shape, generator=g, device="cuda", dtype=torch.float64)
    b = aP * x
    b[:, :, :-1] += aE[:, :, :-1] * x[:, :, 1:]
    b[:, :, 1:] += aW[:, :, 1:] * x[:, :, :-1]
    b[:, :-1, :] += aN[:, :-1, :] * x[:, 1:, :]
    b[:, 1:, :] += aS[:, 1:, :] * x[:, :-1, :]
    b[:-1] += aT[:-1] * x[1:]
    b[1:] += aB[1:] * x[:-1]
    return torch.stack([aP, aE, aW, aN, aS, aT, aB]).reshape(7, -1), b.reshape(-1), x.reshape(-1)


def _csr_rows(coef, dims):
    """The same system in compressed rows, as SparseMatrix holds it on the host."""
    nI, nJ, nK = dims
    n = nI * nJ * nK
    c = np.arange(n, dtype=np.int64)
    i, j = c % nI, (c // nI) % nJ
    off = [0, 1, -1, nI, -nI]
    keep = [np.ones(n, bool), i < nI - 1, i > 0, j < nJ - 1, j > 0]
    mask = np.stack(keep, axis=1)
    cols = np.stack([c + o for o in off], axis=1)[mask]
    vals = np.stack([coef[q] for q in range(5)], axis=1)[mask]
    ptr = np.zeros(n + 1, dtype=np.int32)
    np.cumsum(mask.sum(axis=1), out=ptr[1:])
    return ptr, cols.astype(np.int32), np.ascontiguousarray(vals)


def prepare(case, seed):
    do = case["do"]
    if do == "step":
        s, restart = _prepare_flow(case, seed)
        return dict(case=case, s=s, restart=restart, out={k: _pinned(s.size_of(k)) for k in ("u", "p")})
    if do == "psolve":
        s, restart = _prepare_flow(case, seed)
        _load(s, restart)
        for ph in ("save_u0", "ib_field", "ib_coeffs", "assemble_momentum", "solve_momentum", "momentum_post", "assemble_pcorr"):
            s.phase(ph)
        return dict(case=case, s=s, out={"pCorr": _pinned(s.size_of("pCorr"))})
    if do == "ksp7":
        coef, b, x = _seven_point((case["nI"], case["nJ"], case["nK"]), seed)
        return dict(case=case, coef=coef.contiguous(), b=b.contiguous(), x=torch.zeros_like(x))
    if do == "csr":
        dims = (case["nI"], case["nJ"], 1)
        coef, b, _ = _seven_point(dims, seed)
        return dict(case=case, rows=_csr_rows(coef.cpu().numpy(), dims), b=b.cpu().numpy())
    s = make_solver(*_flow_case(case, seed))
    _load(s, {"u": torch.from_numpy(_start_velocity(case, seed).reshape(-1))})
    for ph in ("save_u0", "ib_field", "ib_coeffs", "assemble_momentum", "solve_momentum", "momentum_post", "assemble_pcorr"):
        s.phase(ph)
    P.add_random_pairs(s, 8, seed=seed & 0xFFFF)
    return dict(case=case, s=s, params=P.load_default())


def run(state):
    case = state["case"]
    do = case["do"]
    if do in ("step", "psolve"):
        s = state["s"]
        if do == "step":
            _load(s, state["restart"])
            for _ in range(case["steps"]):
                s.solve()
        else:
            s.phase("solve_pcorr")
        for name, v in state["out"].items():
            s.get_to_ptr(name, v.data_ptr(), v.numel())
        return state["out"]
    if do == "ksp7":
        x = state["x"]
        it, rr = ctypes.c_int(0), ctypes.c_double(0.0)
        st = _lib.lib().caffe_ksp7_solve_device(case["nI"], case["nJ"], case["nK"], state["coef"].data_ptr(), state["b"].data_ptr(), x.data_ptr(),
                                                C.KSP_METHODS[case["method"]], 1e-12, 20000, torch.cuda.current_stream().cuda_stream,
                                                ctypes.byref(it), ctypes.byref(rr))
        if st != 0:
            raise RuntimeError(f"ksp7 solve: status {st}")
        return x
    if do == "csr":
        x, _, _, st = _lib.csr_solve(*state["rows"], state["b"], method=case["method"], rtol=1e-12)
        if st != 0:
            raise RuntimeError(f"csr solve: status {st}")
        return x
    params, loss = P.train(state["s"], state["params"], steps=case["steps"], batch=case["batch"], lr=1e-5, seed=3)
    return {"params": params, "loss": loss}


def work(case):
    """What a pass cannot do without: fields and systems read and written once (a Krylov solve's own
    sweeps over the system are the path's, not the task's), the network's multiplications."""
    n = case["nI"] * case["nJ"] * case.get("nK", 1)
    do = case["do"]
    if do == "step":
        return {"bytes": float(n * case["steps"] * STEP_BYTES), "flops": 400.0 * n * case["steps"]}
    if do == "psolve":
        return {"bytes": 48.0 * n, "flops": 13.0 * n}
    if do == "ksp7":
        return {"bytes": 72.0 * n, "flops": 13.0 * n}
    if do == "csr":
        return {"bytes": (5 * 12 + 4 + 16) * float(n), "flops": 10.0 * n}
    # 4 layers of 27 x 16 x 16 on every coarse level (1/8 + 1/64 + ...), two signs, forward, backward and weights
    cells = n / 7.0 * case["steps"] * case["batch"]
    return {"bytes": cells * 2 * 4 * 32 * 4, "flops": cells * 2 * 4 * 2 * 27 * 256 * 3}


def exact(case, seed):
    """The Krylov solves' known solutions; the flow and training outputs have no closed form."""
    if case["do"] == "ksp7":
        return _seven_point((case["nI"], case["nJ"], case["nK"]), seed)[2]
    if case["do"] == "csr":
        return _seven_point((case["nI"], case["nJ"], 1), seed)[2].cpu().numpy()
    return None
