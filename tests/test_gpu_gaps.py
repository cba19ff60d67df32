"""Grid cells that no sample touches (marked gpu): the operator leaves them out of the FFT
stages' writes and (volumes) reads, by the longest unused run of each grid line and by whole
unused lines and planes.  Trajectories that leave most of the grid unused, on one side of the
centre, around it, and wrapping past the grid's edge, against the FP64 Kaiser-Bessel operator:
within 2^-11, the largest relative rounding of an FP16 coefficient."""
import numpy as np
import pytest

from gpu_cases import rel_l2
from oracle import operator as oop

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

BOXES = {"corner": ((0.05, 0.2), (-0.4, -0.1), (0.2, 0.3)), "line": ((-0.5, 0.5), (0.0, 0.004), (-0.1, 0.1)),
         "edge": ((0.44, 0.5), (-0.5, -0.46), (-0.5, 0.5)), "one cell": ((0.1, 0.1), (0.2, 0.2), (-0.3, -0.3))}


@pytest.mark.parametrize("dims,n,g,c", [(2, 60, 128, 8), (2, 128, 256, 4), (2, 92, 256, 16), (3, 28, 128, 4)])
@pytest.mark.parametrize("box", BOXES)
def test_operator_with_unused_grid(dims, n, g, c, box):
    from trajsparsenufft_b200.operator import Plan
    rng = np.random.default_rng(n)
    traj = np.stack([rng.uniform(*b, 700) for b in BOXES[box][:dims]], axis=1).astype(np.float32)
    plan = Plan.from_trajectory(traj, im_size=n, grid_size=g, coils=c, width=4)
    ref = (oop.KbSenseOperator3 if dims == 3 else oop.KbSenseOperator)(traj, n, g, 4, workers=4)
    cplx = lambda *sh: (rng.standard_normal(sh) + 1j * rng.standard_normal(sh)).astype(np.complex64)
    x, s, y = cplx(*[n] * dims), cplx(c, *[n] * dims), cplx(c, len(traj))
    xt, st, yt = (torch.from_numpy(v).cuda() for v in (x, s, y))
    for _ in range(2):  # the second pass reads what the first left in the workspaces
        assert rel_l2(plan.forward(xt, st).cpu().numpy(), ref.forward(x, s)) <= 2.0 ** -11
        assert rel_l2(plan.adjoint(yt, st).cpu().numpy(), ref.adjoint(y, s)) <= 2.0 ** -11
