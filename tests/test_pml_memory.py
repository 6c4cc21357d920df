"""What the PML adds to a fused context's device memory: thirteen coefficients
and twelve auxiliary values per node of a PML element, two integers per
element; sigma, which only the host reads back, stays there."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import gpu_from_ref, make_ref
from nekcem_gb300 import MaxwellGPU

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["fused64", "mixed"])
def test_pml_device_memory_and_sigma(form):
    N, nel = 4, (4, 5, 6)
    ref = make_ref(N, nel, (0, 0, 0), (1, 1, 1), (2, 1, 0), pml=(1, 3.0, 1e-6))
    n3 = (N + 1) ** 3
    with gpu_from_ref(ref, form) as g:
        # without PML, with face coefficients as the PML walls have them
        with MaxwellGPU.from_box(N, nel, (0, 0, 0), (1, 1, 1), (0, 1, 0), form=form,
                                 permittivity=1.0 + ref.coords()[0]) as plain:
            added = g.device_bytes() - plain.device_bytes()
        nodes = 2 * 5 * 6 * n3
        assert added <= 8 * 25 * nodes + 2 * 4 * g.nelt + 4096
        np.testing.assert_array_equal(g.array("pmlsigma"), ref.d("pmlsigma"))
    ref.close()
