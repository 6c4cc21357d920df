"""A derivative matrix of large entries on large fields, where the exponents
of the fixed-point contractions (nekgpu_fixed.cuh) would leave FP64's range:
the lines overflow as FP64 sums do, and the blow-up check sees it."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import make_ref, oracle_arrays, random_fields
from nekcem_gb300 import MaxwellGPU, NekgpuError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("deform", [0.0, 0.04])
@pytest.mark.parametrize("nel", [(2, 2, 2), (5, 4, 5)])
@pytest.mark.parametrize("power,scale", [(30, 1e302), (40, 1e302), (60, 1e297), (100, 1e285)])
def test_overflowing_lines_overflow(nel, power, scale, deform):
    """dxm1 times 2^power on fields of the given scale, both within what the
    integers take one without the other, the derivatives 1e312 and more:
    non-finite where the plain form's FP64 sums are, and only there"""
    ref = make_ref(6, nel, (0, 0, 0), (1, 1, 1), (0, 1, 0), deform=deform)
    arrays = oracle_arrays(ref)
    arrays["dxm1"] = arrays["dxm1"] * 2.0 ** power
    H, E = random_fields(ref.npts, 4)
    finite = {}
    for form in ("plain", "fused64"):
        with MaxwellGPU.from_arrays(arrays, ref.n, ref.nelt, form=form) as g:
            g.set_state(H * scale, E * scale)
            g.stage(1, 0.0, 1e-4)
            finite[form] = np.isfinite(np.concatenate(g.get_state()))
            with pytest.raises(NekgpuError):
                g.check_blowup()
    assert not finite["plain"].all()
    np.testing.assert_array_equal(finite["fused64"], finite["plain"])
    ref.close()
