"""Programmatic dependent launch of direct calls (marked gpu): the same bits as plain launches, and
inputs rewritten on the stream between calls are read as they are at each call."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from gpu_cases import case, volume_case

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CALLS = """
import sys
import numpy as np, torch
sys.path[:0] = sys.argv[2:4]
from gpu_cases import case, volume_case
from trajsparsenufft_b200 import autograd as tad, synth
from trajsparsenufft_b200.operator import Batch, Plan
out, plans = [], []
for traj, x, s, n, g, c, j in (case("small")[:7], case("c16")[:7], volume_case("vol64c8")):
    plan = Plan.from_trajectory(traj, im_size=n, grid_size=g, coils=c, width=j)
    xt, st = torch.from_numpy(x).cuda(), torch.from_numpy(s).cuda()
    w = torch.linspace(0.5, 1.5, len(traj), device="cuda")
    y = plan.forward(xt, st)
    a = plan.adjoint(y, st)
    rho = plan.rdot(a, a)
    q, t, gamma = plan.normal(a, st, density=w, lam=1e-4, coils=True, pq=True)
    x1, r1, p1, rho1, parts = plan.cg_step(rho, gamma, xt, a, a, q, norm_parts=True)
    out += [y, a, plan.forward((st * xt).contiguous()), plan.adjoint(y), q, t, gamma, x1, r1, p1, rho1]
    out += list(plan.normal(p1, st, lam=1e-4, pq=True, p_norm_parts=parts))[::2]
    out.append(plan.cg_sense(y, st, density=w, iters=3, sync=False)[0])
    yl, sl = y.clone().requires_grad_(True), st.clone().requires_grad_(True)
    tad.cg_sense(yl, sl, tad.PlanOps(plan), density=w, iters=3, checkpoint=2).abs().pow(2).sum().backward()
    out += [yl.grad, sl.grad]
    plans.append((plan, y, st))
out += Batch([p for p, _, _ in plans]).cg_sense([y for _, y, _ in plans], [s for _, _, s in plans], iters=3, sync=False)[0]
np.savez(sys.argv[1], *[v.detach().cpu().numpy() for v in out])
"""


def test_plain_and_programmatic_launches_give_the_same_bits(tmp_path):
    """Every direct call, a solve, a gradient and a batch, of images and a volume, with TSN_PDL=0 and
    without it (read once per process)."""
    tests = Path(__file__).resolve().parent
    got = []
    for name, env in (("plain", {"TSN_PDL": "0"}), ("programmatic", {})):
        path = tmp_path / f"{name}.npz"
        base = {k: v for k, v in os.environ.items() if k != "TSN_PDL"}
        subprocess.run([sys.executable, "-c", CALLS, str(path), str(tests), str(tests.parent)], env={**base, **env},
                       check=True, timeout=300)
        got.append(np.load(path))
    assert len(got[0].files) == len(got[1].files) == 3 * 16 + 3
    for k in got[0].files:
        assert got[0][k].tobytes() == got[1][k].tobytes(), k


@pytest.mark.parametrize("volume", [False, True])
def test_inputs_rewritten_between_calls(volume):
    """Images, maps, k-space and density rewritten in place between direct calls, with and without
    waiting in between: a kernel that starts early reads nothing that is still being written.  The
    operator whose panel scale the caller has (forward rows as the first kernel) follows a rewrite of
    the maps directly."""
    from trajsparsenufft_b200.operator import Plan
    traj, x, s, n, g, c, j = (volume_case("vol64") if volume else case("headline"))[:7]
    plan = Plan.from_trajectory(traj, im_size=n, grid_size=g, coils=c, width=j)
    gen = torch.Generator(device="cuda").manual_seed(1)
    new = [[torch.randn(sh, dtype=dt, device="cuda", generator=gen) for sh, dt in
            ((x.shape, torch.complex64), (s.shape, torch.complex64), ((c, len(traj)), torch.complex64),
             ((len(traj),), torch.float32))] for _ in range(4)]
    bufs = [torch.empty_like(v) for v in new[0]]
    img, maps, y, w = bufs
    parts = torch.empty(1, dtype=torch.float64, device="cuda")
    runs = []
    for wait in (True, False):
        out = []
        sync = torch.cuda.synchronize if wait else (lambda: None)
        torch.cuda.synchronize()
        for vals in new:
            def put(*which):
                sync()
                for k in which:
                    bufs[k].copy_(vals[k])
                sync()
            put(0, 1)
            out.append(plan.forward(img, maps))
            put(2, 1)
            out.append(plan.adjoint(y, maps))
            put(3)
            out += plan.normal(img, maps, density=w, lam=1e-4, coils=True, pq=True)
            parts.copy_(plan.rdot(img, img).reshape(1))
            maps.neg_()
            put(1)
            out.append(plan.normal(img, maps, density=w, lam=1e-4, p_norm_parts=parts)[0])
            for b in bufs:  # a read that comes late would see zeros
                b.zero_()
        torch.cuda.synchronize()
        runs.append(out)
    for a, b in zip(*runs):
        assert torch.equal(torch.view_as_real(a) if a.is_complex() else a, torch.view_as_real(b) if b.is_complex() else b)
