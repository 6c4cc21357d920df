"""The fused FP64 form's integer contractions (nekgpu_fixed.cuh) where they
can go wrong: the element counts on both sides of the split rule, the
reference's GLL orders with odd and even rows, fields spread over many
binades, lines that hold infinities, NaNs and huge values, and a D that does
not fit the fixed-point table.

Tolerance: a step's five stages each round the residual of at most ~40 terms
and the update in FP64, ~1e-14 of the largest value at these sizes; 1e-12 is
the form's bar against the oracle everywhere in this suite."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import gpu_from_box, make_ref, oracle_arrays, random_fields, rel_err
from nekcem_gb300 import MaxwellGPU, NekgpuError

pytestmark = pytest.mark.gpu


def one_step(ref, g, H, E, dt):
    ref.set_state(H, E)
    g.set_state(H, E)
    ref.op_rk(0.0, dt)
    g.run(1, 0.0, dt)
    return rel_err(*g.get_state(), ref.hn, ref.en)


# one element, five slabs, two slabs (76 of 152 SMs), unsplit just above, and
# more elements than one wave of blocks
@pytest.mark.parametrize("nel", [(1, 1, 1), (3, 3, 3), (4, 19, 1), (7, 11, 1), (9, 9, 8)])
@pytest.mark.parametrize("N", [2, 3, 7, 8])
def test_split_rule_edges(nel, N):
    ref = make_ref(N, nel, (0, 0, 0), (1.0, 1.3, 0.8), (0, 1, 0),
                   eps=lambda x, y, z: 1.0 + 0.5 * np.sin(2 * x) ** 2)
    with gpu_from_box(ref, "fused64") as g:
        assert one_step(ref, g, *random_fields(ref.npts, 3), 0.2 * ref.dxmin()) <= 1e-12
    ref.close()


@pytest.mark.parametrize("nel", [(2, 2, 2), (5, 4, 5)])
@pytest.mark.parametrize("decades", [0, 20, 300])
def test_wide_range_fields(nel, decades):
    """values spread over up to 300 decades inside the elements, zeros among them"""
    ref = make_ref(7, nel, (0, 0, 0), (1, 1, 1), (1, 0, 1))
    rng = np.random.default_rng(5)
    H, E = (rng.standard_normal((3, ref.npts)) * 10.0 ** (-decades * rng.random((3, ref.npts)))
            for _ in range(2))
    H[:, ::7] = 0.0
    E[1] = 0.0
    with gpu_from_box(ref, "fused64") as g:
        assert one_step(ref, g, H, E, 0.2 * ref.dxmin()) <= 1e-12
    ref.close()


@pytest.mark.parametrize("nel", [(2, 2, 2), (5, 4, 5)])
@pytest.mark.parametrize("scale", [1e-290, 1e-200, 1e200, 1e303])
def test_extreme_scales(nel, scale):
    """the step is linear: fields scaled by a power of ten, up to where lines
    leave the integer form for FP64"""
    ref = make_ref(5, nel, (0, 0, 0), (1, 1, 1), (0, 1, 0))
    H, E = random_fields(ref.npts, 9)
    with gpu_from_box(ref, "fused64") as g:
        assert one_step(ref, g, H * scale, E * scale, 0.2 * ref.dxmin()) <= 1e-12
    ref.close()


@pytest.mark.parametrize("nel", [(2, 2, 2), (5, 4, 5)])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_non_finite_value_spreads_along_its_lines_only(nel, bad):
    n = 6
    ref = make_ref(n - 1, nel, (0, 0, 0), (1, 1, 1), (1, 1, 1))
    H, E = random_fields(ref.npts, 2)
    v = 2 + n * 3 + n * n * 2  # an interior node of element 1
    H1 = H.copy()
    H1[2, n ** 3 + v] = bad
    dt = 0.2 * ref.dxmin()
    out = []
    for h in (H, H1):
        with gpu_from_box(ref, "fused64") as g:
            g.set_state(h, E)
            g.stage(1, 0.0, dt)
            out.append(np.concatenate(g.get_state()))
            if h is H1:
                with pytest.raises(NekgpuError):
                    g.check_blowup()
    ok = np.isfinite(out[1])
    # H_z is differentiated along r (into E_y) and s (into E_x); no other line holds the value
    hit = np.zeros((6, ref.nelt, n, n, n), dtype=bool)
    hit[4, 1, 2, 3, :] = True
    hit[3, 1, 2, :, 2] = True
    hit[2, 1, 2, 3, 2] = True
    hit = hit.reshape(6, -1)
    np.testing.assert_array_equal(out[1][~hit], out[0][~hit])
    # (the derivative's own diagonal entry is zero: 0 times NaN or infinity)
    assert not ok[hit].any()
    ref.close()


@pytest.mark.parametrize("nel", [(2, 2, 2), (5, 4, 5)])
@pytest.mark.parametrize("power", [-150, -40, 0, 30])
def test_scaled_derivative_matrix(nel, power):
    """dxm1 scaled by a power of two, inside the fixed-point table's range and
    outside it, against the plain form on the same arrays"""
    ref = make_ref(6, nel, (0, 0, 0), (1, 1, 1), (0, 1, 0))
    arrays = oracle_arrays(ref)
    arrays["dxm1"] = arrays["dxm1"] * 2.0 ** power
    H, E = random_fields(ref.npts, 4)
    dt = 0.2 * ref.dxmin() * 2.0 ** min(0, -power)
    got = {}
    for form in ("plain", "fused64"):
        with MaxwellGPU.from_arrays(arrays, ref.n, ref.nelt, form=form) as g:
            g.set_state(H, E)
            g.run(1, 0.0, dt)
            got[form] = g.get_state()
    assert rel_err(*got["fused64"], *got["plain"]) <= 1e-12
    ref.close()
