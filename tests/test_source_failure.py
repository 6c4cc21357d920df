"""A nekgpu_set_source that fails for lack of memory, after the arrays of the
source before it were given back: the context steps on without a source."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import random_fields
from nekcem_gb300 import MaxwellGPU, NekgpuError

pytestmark = pytest.mark.gpu
SOURCE = dict(xc=(0.4, 0.5, 0.6), sigma=0.2, amp=1.0, f0=2.0, t0=0.1)


@pytest.mark.parametrize("form", ["fused64", "mixed", "mixed_naive"])
def test_failed_source_leaves_no_source(form, monkeypatch):
    args = (4, (3, 3, 3), (0, 0, 0), (1, 1, 1), (0, 1, 0))
    with MaxwellGPU.from_box(*args, form=form) as g, MaxwellGPU.from_box(*args, form=form) as plain:
        H, E = random_fields(g.npts, 12)
        for x in (g, plain):
            x.set_state(H, E)
        g.set_source(**SOURCE)
        monkeypatch.setenv("NEKGPU_MEM_BUDGET_MB", "0")
        with pytest.raises(NekgpuError) as e:
            g.set_source(**SOURCE)
        assert e.value.status == -4
        monkeypatch.delenv("NEKGPU_MEM_BUDGET_MB")
        for x in (g, plain):
            x.run(2, 0.0, 1e-4)
        np.testing.assert_array_equal(np.concatenate(g.get_state()), np.concatenate(plain.get_state()))
        g.set_source(**SOURCE)  # and takes a new one
        g.run(1, 0.0, 1e-4)
        plain.run(1, 0.0, 1e-4)
        assert not np.array_equal(g.get_state()[1], plain.get_state()[1])
