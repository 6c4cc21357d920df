"""The mixed stage on meshes of few elements, whose k-slabs go to several
blocks: one step against the oracle on both sides of the split rule's element
counts (152 SMs), with the extension terms, and bit for bit against the
unsplit kernel.

Tolerance: the form's bar against the oracle, 1e-9 per step (contractions
carried to ~2^-34 of sum|D||u|)."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import gpu_from_box, gpu_from_ref, make_ref, random_fields, rel_err
from nekcem_gb300 import MaxwellGPU

pytestmark = pytest.mark.gpu


# N=8, 7: four slabs up to 38 elements, two up to 76; N=6 three to 101, two to
# 152; N=5 three to 152, two to 228; N=4 two to 228; N=3 two to 456
@pytest.mark.parametrize("N,nel", [(8, (1, 1, 1)), (8, (2, 19, 1)), (8, (3, 13, 1)), (8, (7, 11, 1)),
                                   (7, (2, 19, 1)), (7, (3, 13, 1)), (7, (4, 19, 1)), (7, (7, 11, 1)),
                                   (6, (1, 101, 1)), (6, (2, 51, 1)), (6, (9, 17, 1)), (5, (8, 19, 1)),
                                   (5, (9, 17, 1)), (5, (12, 19, 1)), (4, (12, 19, 1)), (4, (1, 229, 1)),
                                   (3, (8, 57, 1)), (2, (2, 2, 2))])
@pytest.mark.parametrize("materials", [False, True])
def test_split_rule_edges(N, nel, materials):
    eps = (lambda x, y, z: 1.0 + 0.5 * np.sin(3 * x) ** 2) if materials else None
    ref = make_ref(N, nel, (0, 0, 0), (1.0, 1.4, 0.7), (0, 1, 0), eps=eps)
    H, E = random_fields(ref.npts, 6)
    src = dict(xc=(0.4, 0.5, 0.3), sigma=0.2, amp=1.0, f0=2.0, t0=0.1)
    with gpu_from_box(ref, "mixed") as g:
        ref.set_state(H, E); g.set_state(H, E)
        ref.set_source(**src); g.set_source(**src)
        dt = 0.2 * ref.dxmin()
        ref.op_rk(0.0, dt)
        g.run(1, 0.0, dt)
        assert rel_err(*g.get_state(), ref.hn, ref.en) <= 1e-9
    ref.close()


@pytest.mark.parametrize("form,tol", [("fused64", 1e-12), ("mixed", 1e-9)])
@pytest.mark.parametrize("N,nel", [(7, (2, 4, 2)), (7, (4, 4, 4)), (8, (2, 4, 3)), (5, (6, 6, 6))])
def test_pml_and_currents_per_step(form, tol, N, nel):
    """PML at both y ends and a Drude slab, auxiliary fields included; the
    oracle's own arrays handed over, so that its sigma comes back as given"""
    ref = make_ref(N, nel, (0, 0, 0), (1, 1, 1), (1, 2, 1), pml=(1, 3.0, 1e-6))
    x, y, _ = ref.coords()
    idx = np.nonzero((x < 0.5) & (y > 0.3) & (y < 0.7))[0].astype(np.int32)
    rng = np.random.default_rng(3)
    par = rng.uniform(0.5, 2.0, (2, ref.npts))
    H, E = random_fields(ref.npts, 5)
    dt = 0.1 * ref.dxmin()
    with gpu_from_ref(ref, form) as g:
        ref.set_drude(par[0], par[1], idx)
        g.set_dispersive(g.DRUDE, par, idx)
        ref.set_state(H, E); g.set_state(H, E)
        for step in range(2):
            ref.op_rk(step * dt, dt)
            g.run(1, step * dt, dt)
        assert rel_err(*g.get_state(), ref.hn, ref.en) <= 2 * tol
        for name, want in (("pmlbn", ref.d("pmlbn")), ("pmldn", ref.d("pmldn"))):
            assert np.max(np.abs(g.array(name) - want)) <= 2 * tol * np.max(np.abs(want))
        np.testing.assert_array_equal(g.array("pmlsigma"), ref.d("pmlsigma"))
    ref.close()


@pytest.mark.parametrize("N", [3, 4, 5, 6, 7, 8])
def test_split_is_bitwise_the_unsplit_kernel(N):
    """1024 elements step unsplit on the device; the host-field step runs them
    as 16 ranges of 64, which the rule splits"""
    nel = (16, 8, 8)
    with MaxwellGPU.from_box(N, nel, (0, 0, 0), (1, 1.2, 0.9), (0, 1, 0), form="mixed") as g:
        H, E = random_fields(g.npts, 4)
        dt = 1e-3 / N ** 2
        g.set_state(H, E)
        g.run(2, 0.0, dt)
        want = g.get_state()
        h, e = H.copy(), E.copy()
        for step in range(2):
            g.op_rk_host(h, e, step * dt, dt)
        np.testing.assert_array_equal(h, want[0])
        np.testing.assert_array_equal(e, want[1])
