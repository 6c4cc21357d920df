"""The reverse stage at the orders that test_adjoint.py leaves out, on both
sides of the element counts at which its blocks change form (152 SMs), and on
meshes of more elements than blocks fit, so that blocks take several.

dJ/deps node by node against torch's tape gradient of the oracle's operator
(tests/tape_maxwell.py, as in test_adjoint.py: 1e-9 of the largest entry, J to
1e-12): smooth fields everywhere, J = sum bm1 |E|^2 over the whole box,
permittivity varying node by node, mixed walls."""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from adjoint_autograd import BoxProblem  # noqa: E402
from helpers import smooth_fields  # noqa: E402
from test_adjoint import PEC, PER, SOURCE, make_tape, problem_data, tape_J  # noqa: E402

pytestmark = pytest.mark.gpu


# small meshes; N=7 to 152 and N=5 to 456 elements a thread per task; N=4, 3:
# more than the resident blocks, N=6, 7, 8: more than 608, 608 and 304
@pytest.mark.parametrize("N,nel,nsteps", [(2, (2, 3, 2), 8), (5, (2, 2, 3), 8), (8, (2, 2, 2), 6),
                                          (7, (8, 19, 1), 2), (7, (9, 17, 1), 2), (5, (12, 38, 1), 2),
                                          (5, (1, 457, 1), 2), (2, (16, 16, 16), 2), (3, (13, 13, 13), 2),
                                          (4, (11, 12, 13), 2), (6, (8, 9, 9), 2), (7, (8, 9, 9), 2),
                                          (8, (7, 7, 7), 2)])
def test_gradient_node_by_node(N, nel, nsteps):
    bc = (PEC, PER, PEC)
    ref, eps, _, _, _, dt, xyz = problem_data(N, nel, bc, seed=90 + N)
    H0, E0 = smooth_fields(ref, N)
    jw = ref.d("bm1").copy()
    pb = BoxProblem(N, nel, (0, 0, 0), (1, 1, 1), bc, H0, E0, jw, nsteps, dt, source=SOURCE)
    J, grad = pb.gradient(eps)
    tm = make_tape(ref, xyz)
    eps_t = torch.tensor(eps, requires_grad=True)
    Jt = tape_J(tm, eps_t, H0, E0, jw, nsteps, dt)
    Jt.backward()
    assert J == pytest.approx(Jt.item(), rel=1e-12)
    gt = eps_t.grad.numpy()
    assert np.abs(grad - gt).max() <= 1e-9 * np.abs(gt).max()
    assert np.count_nonzero(gt) > 0.9 * gt.size
    ref.close()
