"""The mixed general sweep over face lists with entries that a caller may hand in.

Groups of faces are left out by bounds over their normals; a face that is no
number must not take its neighbours along.
"""
import numpy as np
import pytest

from test_gpu_flux64_groups import flat_grid

pytestmark = pytest.mark.gpu

LIMB = dict(ldc=[0.4, 0.1, 0.05, 0.02], spin=1.1, vfac=1e-3, xcofm=0.2)


def entries(nent):
    ph = np.linspace(0, 1, nent, endpoint=False)
    si, ci = np.sin(np.radians(85.0)), np.cos(np.radians(85.0))
    return dict(ex=si * np.cos(2 * np.pi * ph), ey=-si * np.sin(2 * np.pi * ph),
                ez=np.full(nent, ci), phin=ph)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("column", ["dx", "dy", "dz"])
@pytest.mark.parametrize("n,face", [(1, 0), (63, 20), (64, 63), (65, 64), (1500, 777)])
def test_a_face_that_is_no_number_spoils_no_other(engine_mixed, column, value, n, face):
    flat, ph = flat_grid(n, n // 2, False), entries(257)
    flat[column][face] = value
    flat["flux"][face] = 0.0
    a = engine_mixed.sum_star_multi(0, flat, ph, ltype=1, **LIMB)
    for k in ("dx", "dy", "dz"):
        flat[k][face] = 0.0
    b = engine_mixed.sum_star_multi(0, flat, ph, ltype=1, **LIMB)
    # an infinite normal times no flux is no number where the face is seen
    clean = np.full(257, True) if np.isnan(value) else ~np.isnan(a)
    np.testing.assert_array_equal(a[clean], b[clean])
