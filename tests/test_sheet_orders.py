"""Graphene sheet, incident field and PML together (cases.GrapheneSheet) at the
orders that test_graphene.py leaves out: three steps of the fused forms
against the oracle at their bars, per step FP64 1e-12, mixed 1e-9."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import gpu_from_box
from test_graphene import CS, make_case, setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,tol", [("fused64", 1e-12), ("mixed", 1e-9)])
@pytest.mark.parametrize("N", [2, 3, 5, 6, 7, 8])
def test_sheet_per_step(form, tol, N):
    ref = make_case(N)
    with gpu_from_box(ref, form) as g:
        setup(ref, None, N)
        setup(ref, g, N)
        for step in range(3):
            ref.op_rk(step * CS.dt, CS.dt)
            g.run(1, step * CS.dt, CS.dt)
            got = np.concatenate(g.get_state())
            want = np.concatenate([ref.hn, ref.en])
            assert np.abs(got - want).max() <= (step + 1) * tol * np.abs(want).max()
    ref.close()
