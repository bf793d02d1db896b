"""The work this library is used for, as timed cases: what a program hands to the public entry
points, one pass through them, and the outputs of that pass.

``kind`` names the entry point:

* ``matvec``  ``MatrixFreeKff.matvec``: the FP64 operator product of the Krylov solves and the guard.
* ``fused``   ``FusedMatvec.matvec_full``: the FP32 product, or the one with BF16 operands.
* ``solve``   ``GuardedFloorPolicy.run``: one guarded solve of one density state (hierarchy setup,
              probe, preserve / escalate rule, FP64 guard), in the FP64 or the mixed-precision form, with
              the plain damped-Jacobi stack or the drivers' canonical one.
* ``batch``   ``BatchedFloorPolicy.run_many_native``: several states in flight on one GPU.
* ``simp``    the design update around a solve: density filter, filtered sensitivities and the OC
              bisection, without or with the Heaviside projection.
* ``train``   one Adam step of the floor proposer on a mini-batch.
* ``propose`` the floor proposer on one state: pooling and one forward pass.

States are those of the benchmark and of the proposer's training set: elements void with probability
p, smoothed by the cone filter, SIMP exponent 3, on the cantilever of the presets.
"""

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "solver-admissibility-and-guarded-floor-selection_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from gpu_fem.bc_generator import generate_bc  # noqa: E402
from gpu_fem.cuda_fused_matvec import FusedMatvec  # noqa: E402
from gpu_fem.floor_proposer import FloorProposerNet  # noqa: E402
from gpu_fem.paper4 import CANONICAL_STACK, PLAIN_JACOBI_STACK  # noqa: E402
from gpu_fem.policy import BatchedFloorPolicy, GuardedFloorPolicy  # noqa: E402
from gpu_fem.presets import cantilever_spec  # noqa: E402
from gpu_fem.pub_simp_solver import KE_UNIT_3D, _edof_table_3d  # noqa: E402
from gpu_fem.simp_loop import OCUpdater, cone_filter  # noqa: E402
from gpu_fem.solver_v2 import MatrixFreeKff  # noqa: E402

PENAL, FLOOR, RADIUS = 3.0, 1e-12, 1.5


def listed():
    return [
        # the smallest preset: a call is launch latency
        {"name": "matvec_24x12x6", "kind": "matvec", "nx": 24, "ny": 12, "nz": 6},
        # the largest grid of the SIMP loop and of the benchmark's scaling workload
        {"name": "matvec_200x100x50", "kind": "matvec", "nx": 200, "ny": 100, "nz": 50},
        # the 2M-element preset, whose extents fit no tile
        {"name": "fused_fp32_252x126x63", "kind": "fused", "nx": 252, "ny": 126, "nz": 63, "dtype": "fp32"},
        {"name": "fused_bf16_80x40x20", "kind": "fused", "nx": 80, "ny": 40, "nz": 20, "dtype": "bf16"},
        # the plain FP64 method on the medium preset
        {"name": "solve_fp64_80x40x20", "kind": "solve", "nx": 80, "ny": 40, "nz": 20, "precision": "fp64",
         "stack": "plain", "void_p": 0.35, "radius": 1.5, "restart": 300},
        # the reference drivers' default stack (Chebyshev, line search, inner FGMRES, root-local FGMRES)
        {"name": "solve_canonical_80x40x20", "kind": "solve", "nx": 80, "ny": 40, "nz": 20, "precision": "fp64",
         "stack": "canonical", "void_p": 0.2, "radius": 1.5, "restart": 300},
        # the benchmark's state: 512,000 elements, mixed precision
        {"name": "solve_mixed_160x80x40", "kind": "solve", "nx": 160, "ny": 80, "nz": 40, "precision": "mixed",
         "stack": "plain", "void_p": 0.35, "radius": 1.5, "restart": 300},
        # the SIMP loop's solve: 1,000,000 elements, restart 100, iterative coarsest solve; the displacement
        # field is kept in FP32 as for display and storage (the fixed-count coarse PCG stops unconverged and
        # carries rounding into the digits beyond those that the solve's tolerance defines)
        {"name": "solve_mixed_200x100x50", "kind": "solve", "nx": 200, "ny": 100, "nz": 50, "precision": "mixed",
         "stack": "plain", "void_p": 0.2, "radius": 1.5, "restart": 100, "keep": "fp32"},
        # the batching workload: states of the smaller mesh of the floor study, eight in flight
        {"name": "batch_mixed_45x30x30", "kind": "batch", "nx": 45, "ny": 30, "nz": 30, "states": 16, "width": 8},
        # the design update of one SIMP iteration at 1M elements
        {"name": "simp_update_200x100x50", "kind": "simp", "nx": 200, "ny": 100, "nz": 50, "rmin": 1.5,
         "projected": False},
        # the proposer's training step at its training batch, and its use inside a guarded solve
        {"name": "train_128", "kind": "train", "batch": 128},
        {"name": "propose_80x40x20", "kind": "propose", "nx": 80, "ny": 40, "nz": 20},
    ]


def _grid(rng, lo, hi, odd=True):
    """A cantilever grid of about lo..hi elements (log-uniform), extents near 4 : 2 : 1."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    s = (n / 8.0) ** (1.0 / 3.0)
    dims = [max(4, int(round(f * s * rng.uniform(0.85, 1.15)))) for f in (4, 2, 1)]
    if not odd:  # hierarchies are built on grids that halve
        dims = [max(m, int(round(d / m)) * m) for d, m in zip(dims, (8, 4, 2))]
    return {"nx": dims[0], "ny": dims[1], "nz": dims[2]}


def draw(rng):
    kind = rng.choice(("matvec", "matvec", "fused", "fused", "solve", "solve", "solve", "simp", "train", "propose"))
    if kind == "matvec":
        return {"kind": kind, **_grid(rng, 1500, 1_000_000)}
    if kind == "fused":
        return {"kind": kind, **_grid(rng, 1500, 2_000_000), "dtype": rng.choice(("fp32", "bf16"))}
    if kind == "solve":
        return {"kind": kind, **_grid(rng, 1700, 500_000, odd=False), "precision": rng.choice(("fp64", "mixed")),
                "stack": "plain", "void_p": round(rng.uniform(0.1, 0.4), 3),
                "radius": round(rng.uniform(1.5, 2.5), 1), "restart": rng.choice((100, 300))}
    if kind == "simp":
        return {"kind": kind, **_grid(rng, 20_000, 1_000_000), "rmin": round(rng.uniform(1.2, 2.5), 1),
                "projected": rng.random() < 0.3}
    if kind == "train":
        return {"kind": kind, "batch": int(round(math.exp(rng.uniform(math.log(16), math.log(128)))))}
    return {"kind": kind, **_grid(rng, 1700, 1_000_000)}


# ------------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _cone(x, dims, r, transpose=False):
    """The row-normalised cone filter (weight r - dist, the element itself r) by plain torch, 64 bits."""
    h = int(math.floor(r))
    a = torch.arange(-h, h + 1, device="cuda", dtype=torch.float64)
    d = torch.sqrt(a[:, None, None] ** 2 + a[None, :, None] ** 2 + a[None, None, :] ** 2)
    off = [(i - h, j - h, k - h) for i in range(2 * h + 1) for j in range(2 * h + 1) for k in range(2 * h + 1)]
    w = torch.where(d <= r - 1e-10, r - d, torch.zeros_like(d)).reshape(-1).tolist()

    def conv(v):
        p = torch.nn.functional.pad(v.reshape(dims), (h,) * 6)
        out = torch.zeros(dims, dtype=torch.float64, device="cuda")
        for (i, j, k), c in zip(off, w):
            if c != 0.0:
                out += c * p[h + i:h + i + dims[0], h + j:h + j + dims[1], h + k:h + k + dims[2]]
        return out.reshape(-1)

    rows = conv(torch.ones(math.prod(dims), dtype=torch.float64, device="cuda"))
    return conv(x / rows) if transpose else conv(x) / rows


def _density(dims, p, r, gen):
    solid = (torch.rand(math.prod(dims), dtype=torch.float64, device="cuda", generator=gen) >= p).double()
    return _cone(solid, dims, r)


def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _mesh(case):
    dims = _dims(case)
    bc = generate_bc(cantilever_spec(*dims))
    edof = torch.as_tensor(_edof_table_3d(*dims), device="cuda")
    return dims, np.asarray(bc.free_dofs), bc.ndof, edof


def _policy(case):
    kw = dict(penal=PENAL, tol=1e-6, restart=case.get("restart", 300), maxiter=300, probe_iters=100, probe_r50=50,
              raised_rho_mins=(1e-3, 1e-2))
    if case.get("stack") == "canonical":
        return dict(kw, stack=dict(CANONICAL_STACK), cycle_precision="fp64")
    mixed = case.get("precision", "mixed") == "mixed"
    return dict(kw, stack=dict(PLAIN_JACOBI_STACK, fine_smoother="fp32" if mixed else "fp64"),
                cycle_precision="fp32" if mixed else "fp64")


def prepare(case, seed):
    g, kind = _gen(seed), case["kind"]
    if kind in ("matvec", "fused"):
        dims, free, ndof, edof = _mesh(case)
        E = FLOOR + (1.0 - FLOOR) * _density(dims, 0.35, RADIUS, g) ** PENAL
        if kind == "matvec":
            free_t = torch.as_tensor(free.astype(np.int64), device="cuda")
            op = MatrixFreeKff(edof, torch.as_tensor(KE_UNIT_3D, device="cuda"), free_t, free.size, ndof,
                               grid_dims=dims)
            u = torch.randn(free.size, dtype=torch.float64, device="cuda", generator=g)
            return {"kind": kind, "op": op, "E": E, "u": u}
        u = torch.zeros(ndof, dtype=torch.float32, device="cuda")
        free_t = torch.as_tensor(free.astype(np.int64), device="cuda")
        u[free_t] = torch.randn(free.size, dtype=torch.float32, device="cuda", generator=g)
        op = FusedMatvec(edof, torch.as_tensor(KE_UNIT_3D, device="cuda"), ndof)
        return {"kind": kind, "op": op, "E": E.float(), "u": u, "dtype": case["dtype"]}
    if kind == "solve":
        dims = _dims(case)
        return {"kind": kind, "pol": GuardedFloorPolicy(cantilever_spec(*dims), **_policy(case)),
                "keep": case.get("keep", "fp64"), "density": _density(dims, case["void_p"], case["radius"], g)}
    if kind == "batch":
        dims = _dims(case)
        pol = BatchedFloorPolicy(case["width"], cantilever_spec(*dims), **_policy(case))
        return {"kind": kind, "pol": pol,
                "densities": [_density(dims, (0.2, 0.35, 0.5)[k % 3], RADIUS, g) for k in range(case["states"])]}
    if kind == "simp":
        dims = _dims(case)
        rho, dc = _design(case, seed)
        ones = torch.ones(math.prod(dims), dtype=torch.float64, device="cuda")
        return {"kind": kind, "oc": OCUpdater(), "dims": dims, "rmin": case["rmin"], "projected": case["projected"],
                "rho": rho, "dc": dc, "vol_w": cone_filter(ones, dims, case["rmin"], transpose=True)}
    if kind == "train":
        x, f, y = _samples(case["batch"], g)
        return {"kind": kind, "net": FloorProposerNet(max_batch=case["batch"], seed=int(seed) & 0xFFFF),
                "x": x, "f": f, "y": y}
    dims = _dims(case)
    feats = torch.rand((1, 2), dtype=torch.float32, device="cuda", generator=g) * 0.5
    return {"kind": kind, "net": FloorProposerNet.load(max_batch=1), "dims": dims, "feats": feats,
            "density": _density(dims, 0.35, RADIUS, g)}


def _design(case, seed):
    """A design in the middle of an optimisation: densities around the volume fraction of 0.3, and
    sensitivities over several decades, as element energies are."""
    g, n = _gen(seed), case["nx"] * case["ny"] * case["nz"]
    rho = (0.3 + 0.15 * torch.randn(n, dtype=torch.float64, device="cuda", generator=g)).clamp(1e-3, 1.0)
    dc = -torch.exp(1.5 * torch.randn(n, dtype=torch.float64, device="cuda", generator=g))
    return rho, dc


def _samples(batch, g):
    """Pooled densities (means near 0.65 as the masks pool to), probe features and rung labels."""
    x = (0.65 + 0.2 * torch.randn((batch, 4096), device="cuda", generator=g)).clamp(0.0, 1.0)
    f = torch.stack([-torch.rand(batch, device="cuda", generator=g),
                     torch.rand(batch, device="cuda", generator=g)], dim=1)
    y = torch.randint(0, 3, (batch,), device="cuda", generator=g).to(torch.int32)
    return x, f, y


# ------------------------------------------------------------------------- one pass
def _row(r):
    """The decisions of a guarded solve."""
    return [int(r["total_iters"]), int(r["solve_iters"]), int(r["n_floor_attempts"]), int(r["solve_converged"]),
            int(round(-math.log10(r["recommended_rho_min"])))]


def run(s):
    kind = s["kind"]
    if kind == "matvec":
        return s["op"].matvec(s["u"], s["E"])
    if kind == "fused":
        return s["op"].matvec_full(s["u"], s["E"], dtype=s["dtype"])
    if kind == "solve":
        r = s["pol"].run(s["density"])
        x = s["pol"].last_x
        return {"x": x.float() if s["keep"] == "fp32" else x, "row": _row(r)}
    if kind == "batch":
        rows = s["pol"].run_many_native(s["densities"])
        return {"x": list(s["pol"].last_xs), "row": np.array([_row(r) for r in rows], dtype=np.int64)}
    if kind == "simp":
        rho_f = cone_filter(s["rho"], s["dims"], s["rmin"])
        if s["projected"]:
            out = s["oc"].projected(s["dims"], s["rmin"], s["rho"], rho_f, s["dc"], 4.0, 0.5, 0.3, 0.2)
        else:
            dc = cone_filter(s["dc"], s["dims"], s["rmin"], transpose=True)
            out = s["oc"](s["rho"], dc, s["vol_w"], 0.3, 0.2)
        return {"rho_f": rho_f, "rho_new": out[0], "change": out[1], "lm": out[2], "steps": out[3]}
    if kind == "train":
        loss, grad = s["net"].loss_grad(s["x"], s["f"], s["y"], want_grad=True)
        s["net"].adam_step(2e-3)
        return {"loss": np.float32(loss), "grad": grad}
    x = FloorProposerNet.pool(s["density"], s["dims"])
    return {"x": x, "prob": s["net"].forward(x.reshape(1, -1), s["feats"])}


# ------------------------------------------------------------------------- bytes and operations
def work(case):
    """Inputs read once and outputs written once; the operations of the method's own arithmetic: an
    element product in the stiffness's symmetry-reduced form is 312 of them (dense: 1,152)."""
    kind = case["kind"]
    if kind == "train":
        n = case["batch"]
        return {"bytes": 4.0 * (4096 * n + 2 * 49017), "flops": 3.0 * 2 * _macs() * n}
    ne = case["nx"] * case["ny"] * case["nz"]
    ndof = 3 * (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    if kind == "matvec":
        return {"bytes": 8.0 * ne + 16.0 * ndof, "flops": 312.0 * ne}
    if kind == "fused":
        per = 1152.0 if case["dtype"] == "bf16" else 312.0
        return {"bytes": 4.0 * ne + 8.0 * ndof, "flops": per * ne}
    if kind in ("solve", "batch"):
        # the filtered states take about eight iterations; one multiplies by the operator once in the Krylov
        # space and eleven times in the V-cycle's smoothing and residual, and keeps two vectors, read back once
        it = 8 * case.get("states", 1)
        return {"bytes": case.get("states", 1) * (8.0 * ne + 16.0 * ndof) + it * 4 * 8.0 * ndof,
                "flops": it * 12 * 312.0 * ne}
    if kind == "simp":
        return {"bytes": 8.0 * ne * 5, "flops": ne * (60 * 12.0 + 4 * 19)}
    return {"bytes": 8.0 * ne + 2.0 * 49017, "flops": 2.0 * _macs() + ne}


def _macs():
    return 27.0 * (16 * 4096 + 16 * 16 * 512 + 16 * 32 * 64 + 32 * 32 * 8) + 3 * 34


# ------------------------------------------------------------------------- the same in 64 bits
def _product(dims, E, u, ke):
    """K(E) u over all degrees of freedom: gather, dense element product, scatter-add."""
    edof = torch.as_tensor(_edof_table_3d(*dims), device="cuda").long()
    y = torch.zeros_like(u)
    for a in range(0, edof.shape[0], 1 << 18):
        e = edof[a:a + (1 << 18)]
        y.index_add_(0, e.reshape(-1), ((u[e] @ ke.T) * E[a:a + (1 << 18), None]).reshape(-1))
    return y


def _bisect(volume, target):
    l1, l2, steps = 0.0, 1e9, 0
    for _ in range(100):
        lm = 0.5 * (l1 + l2)
        steps += 1
        if volume(lm) > target:
            l1 = lm
        else:
            l2 = lm
        if l2 - l1 < 1e-9:
            break
    return lm, steps


def exact(case, seed):
    kind, g = case["kind"], _gen(seed)
    if kind in ("matvec", "fused"):
        dims, free, ndof, _ = _mesh(case)
        E = FLOOR + (1.0 - FLOOR) * _density(dims, 0.35, RADIUS, g) ** PENAL
        free_t = torch.as_tensor(free.astype(np.int64), device="cuda")
        ke = torch.as_tensor(KE_UNIT_3D, device="cuda", dtype=torch.float64)
        u = torch.zeros(ndof, dtype=torch.float64, device="cuda")
        if kind == "matvec":
            u[free_t] = torch.randn(free.size, dtype=torch.float64, device="cuda", generator=g)
            return _product(dims, E, u, ke)[free_t]
        u[free_t] = torch.randn(free.size, dtype=torch.float32, device="cuda", generator=g).double()
        if case["dtype"] == "bf16":  # operands rounded to bfloat16, as the entry point defines its product
            u, ke = u.to(torch.bfloat16).double(), ke.float().to(torch.bfloat16).double()
        return _product(dims, E.float().double(), u, ke)
    if kind == "simp":
        dims, r, move, beta, eta = _dims(case), case["rmin"], 0.2, 4.0, 0.5
        rho, dc = _design(case, seed)
        rho_f = _cone(rho, dims, r)
        n = rho.numel()
        if case["projected"]:
            tbe, den = math.tanh(beta * eta), math.tanh(beta * eta) + math.tanh(beta * (1 - eta))
            dh = beta * (1.0 - torch.tanh(beta * (rho_f - eta)) ** 2) / den
            dcd, dv = _cone(dc * dh, dims, r, True), _cone(dh, dims, r, True).clamp_min(1e-12)
        else:
            dcd, dv = _cone(dc, dims, r, True), torch.ones_like(rho)
        dcd = dcd.clamp_max(-1e-12)

        def candidate(lm):
            v = rho * torch.sqrt(-dcd / (lm * dv))
            return torch.minimum(torch.maximum(v, rho - move), rho + move).clamp(1e-3, 1.0)

        def volume(lm):
            f = _cone(candidate(lm), dims, r) if case["projected"] else candidate(lm) * vol_w
            return float((tbe + torch.tanh(beta * (f - eta))).sum()) / den if case["projected"] else float(f.sum())

        vol_w = None if case["projected"] else _cone(torch.ones_like(rho), dims, r, True)
        lm, steps = _bisect(volume, 0.3 * n)
        new = candidate(lm)
        return {"rho_f": rho_f, "rho_new": new, "change": float((new - rho).abs().max()), "lm": lm, "steps": steps}
    if kind == "train":
        x, f, y = _samples(case["batch"], g)
        theta = _weights(FloorProposerNet(max_batch=1, seed=int(seed) & 0xFFFF).get_params())
        for t in theta:
            t.requires_grad_(True)
        loss = torch.nn.functional.cross_entropy(_logits(theta, x.double(), f.double()), y.long())
        grads = torch.autograd.grad(loss, theta)
        return {"loss": np.float64(loss.item()), "grad": torch.cat([v.reshape(-1) for v in grads]).cpu().numpy()}
    if kind == "propose":
        dims = _dims(case)
        feats = torch.rand((1, 2), dtype=torch.float32, device="cuda", generator=g) * 0.5
        d = _density(dims, 0.35, RADIUS, g)
        x = torch.nn.functional.adaptive_avg_pool3d(d.reshape(1, 1, *dims), 16).reshape(-1)
        theta = _weights(FloorProposerNet.load(max_batch=1).get_params())
        logits = _logits(theta, x.float().double().reshape(1, -1), feats.double())
        return {"x": x, "prob": torch.softmax(logits, dim=1)}
    return None  # a guarded solve stops at its tolerance: its answer has no value of its own in 64 bits


def _weights(params):
    """The parameters in their layout (weights rounded to bfloat16, as the network reads them; biases FP32)."""
    p = torch.as_tensor(np.asarray(params), device="cuda")
    out, o = [], 0
    for cin, cout in ((1, 16), (16, 16), (16, 32), (32, 32)):
        for n, shape in ((cout * cin * 27, (cout, cin, 3, 3, 3)), (cout, (cout,))):
            v = p[o:o + n].reshape(shape)
            out.append((v.to(torch.bfloat16) if len(shape) > 1 else v).double())
            o += n
    out.append(p[o:o + 102].reshape(3, 34).to(torch.bfloat16).double())
    out.append(p[o + 102:o + 105].double())
    return out


def _logits(t, x, f):
    h = x.reshape(-1, 1, 16, 16, 16)
    for i, stride in enumerate((1, 2, 2, 2)):
        h = torch.relu(torch.nn.functional.conv3d(h, t[2 * i], t[2 * i + 1], stride=stride, padding=1))
    z = torch.cat([h.mean(dim=(2, 3, 4)), f], dim=1)
    return z @ t[8].T + t[9]
