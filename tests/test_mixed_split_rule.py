"""The mixed stage on both sides of the element counts at which its rule for
meshes of few elements changes form (152 SMs), with and without PML, one step
against the oracle, and two threads per line bit for bit against one.

Tolerance: the form's bar against the oracle, 1e-9 per step."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import gpu_from_box, gpu_from_ref, make_ref, random_fields, rel_err
from nekcem_gb300 import MaxwellGPU

pytestmark = pytest.mark.gpu


# N=7: two slabs to 114 elements, then two threads per line to 152; N=6: three
# slabs to 101; N=5: three to 152; N=4: two to 152; N=3: two to 456 (with PML 228)
@pytest.mark.parametrize("N,nel", [(7, (2, 57, 1)), (7, (5, 23, 1)), (7, (8, 19, 1)), (7, (9, 17, 1)),
                                   (6, (2, 51, 1)), (5, (9, 17, 1)), (4, (8, 19, 1)), (4, (9, 17, 1)),
                                   (3, (12, 19, 1)), (3, (1, 229, 1)), (3, (8, 57, 1)), (3, (1, 457, 1))])
@pytest.mark.parametrize("pml", [False, True])
def test_rule_edges(N, nel, pml):
    ref = make_ref(N, nel, (0, 0, 0), (1.0, 1.4, 0.7), (0, 2 if pml else 1, 1),
                   eps=None if pml else (lambda x, y, z: 1.0 + 0.5 * np.sin(3 * x) ** 2),
                   pml=(2, 3.0, 1e-6) if pml else None)
    H, E = random_fields(ref.npts, 16)
    with (gpu_from_ref if pml else gpu_from_box)(ref, "mixed") as g:
        ref.set_state(H, E); g.set_state(H, E)
        dt = 0.1 * ref.dxmin()
        ref.op_rk(0.0, dt)
        g.run(1, 0.0, dt)
        assert rel_err(*g.get_state(), ref.hn, ref.en) <= 1e-9
        if pml:
            for name in ("pmlbn", "pmldn"):
                want = ref.d(name)
                assert np.max(np.abs(g.array(name) - want)) <= 1e-9 * np.max(np.abs(want))
    ref.close()


def test_two_threads_per_line_are_bitwise_one():
    """1920 elements step unsplit on the device; the host-field step runs them
    as 16 ranges of 120"""
    with MaxwellGPU.from_box(7, (16, 8, 15), (0, 0, 0), (1, 1.2, 0.9), (0, 1, 0), form="mixed") as g:
        H, E = random_fields(g.npts, 4)
        dt = 2e-5
        g.set_state(H, E)
        g.run(2, 0.0, dt)
        want = g.get_state()
        h, e = H.copy(), E.copy()
        for step in range(2):
            g.op_rk_host(h, e, step * dt, dt)
        np.testing.assert_array_equal(h, want[0])
        np.testing.assert_array_equal(e, want[1])
