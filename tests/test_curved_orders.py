"""The curvilinear kernels at the orders and element counts the parity tests
of test_gpu_curved.py leave out: the smallest row lengths, N=6, one element,
and more elements than blocks fit; one step from random fields against the
oracle at the forms' bars (FP64 1e-12, mixed 1e-9)."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import gpu_from_ref, make_ref, random_fields, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,tol", [("fused64", 1e-12), ("mixed", 1e-9)])
@pytest.mark.parametrize("N,nel,bc", [(2, (2, 3, 1), (0, 1, 0)), (3, (1, 1, 1), (0, 0, 0)),
                                      (3, (9, 9, 9), (1, 0, 1)), (6, (2, 3, 2), (1, 1, 0)),
                                      (7, (3, 1, 2), (0, 0, 0))])
@pytest.mark.parametrize("materials", [False, True])
def test_curved_step(form, tol, N, nel, bc, materials):
    eps = (lambda x, y, z: 1.0 + 0.5 * np.sin(2 * x) ** 2) if materials else None
    ref = make_ref(N, nel, (0, 0, 0), (1, 1, 1), bc, eps=eps, deform=0.04)
    H, E = random_fields(ref.npts, 8)
    src = dict(xc=(0.4, 0.5, 0.6), sigma=0.2, amp=1.0, f0=2.0, t0=0.1)
    with gpu_from_ref(ref, form) as g:
        ref.set_state(H, E); g.set_state(H, E)
        ref.set_source(**src); g.set_source(**src)
        dt = 0.2 * ref.dxmin()
        ref.op_rk(0.0, dt)
        g.run(1, 0.0, dt)
        assert rel_err(*g.get_state(), ref.hn, ref.en) <= tol
    ref.close()
