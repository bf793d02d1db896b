"""The BF16 operator on a stiffness that is off its reflection symmetry by less than the accepted
1e-9, with mirrored entries on two sides of a bf16 rounding boundary: the product is that of one
rounded matrix (the entries of the first corner, mirrored), with no term lost.

Entries of 1 + 2^-8 + 2^-24 lie halfway between two floats; the lower is a bf16 tie that rounds
down to 1, the upper rounds to 1 + 2^-7.  The product sums at most 8 x 24 terms in FP32: 1e-5 of
the largest entry is some hundred roundings, against 4e-3 for a lost 2^-8.  In a process of its
own: the meshes alive on a device share one stiffness."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_SCRIPT = r"""
import sys
import numpy as np
import torch
sys.path[:0] = [{root!r}, {pkg!r}]
from gpu_fem.cuda_fused_matvec import FusedMatvec
from gpu_fem.pub_simp_solver import KE_UNIT_3D, _edof_table_3d

dims = (5, 4, 3)
base = 1.0 + 2.0 ** -8 + 2.0 ** -24
ke = KE_UNIT_3D * (base / KE_UNIT_3D[0, 0])
for a in range(8):  # the xx entries of the nodes, corner 0 among the lower ones
    ke[3 * a, 3 * a] = base + (1e-10 if a % 2 else 0.0)
keb = torch.as_tensor(ke, dtype=torch.float32).to(torch.bfloat16).double().numpy()
assert keb[0, 0] == 1.0 and keb[3, 3] == 1.0 + 2.0 ** -7
for a in range(8):
    keb[3 * a, 3 * a] = 1.0
edof = _edof_table_3d(*dims)
ndof = int(edof.max()) + 1
rng = np.random.default_rng(1)
E = (0.5 + rng.random(edof.shape[0])).astype(np.float32)
u = torch.as_tensor(rng.standard_normal(ndof), dtype=torch.float32)
ub = u.to(torch.bfloat16).double().numpy()
ref = np.zeros(ndof)
np.add.at(ref, edof, (ub[edof] @ keb.T) * E.astype(np.float64)[:, None])
op = FusedMatvec(torch.as_tensor(edof, device="cuda"), torch.as_tensor(ke, device="cuda"), ndof)
got = op.matvec_full(u.cuda(), torch.as_tensor(E, device="cuda"), dtype="bf16").double().cpu().numpy()
err = np.abs(got - ref).max() / np.abs(ref).max()
assert err <= 1e-5, err
print("ok")
"""


def test_mirrored_entries_that_round_apart(cuda):
    code = _SCRIPT.format(root=ROOT, pkg=os.path.join(ROOT, "solver-admissibility-and-guarded-floor-selection_b200"))
    res = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600)
    assert res.returncode == 0 and res.stdout.strip().endswith("ok"), res.stdout + res.stderr
