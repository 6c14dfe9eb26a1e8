"""Small visibility calls, whose tiles are split over several warps: sizes over the
range in which the split goes from 8 to 1, whole and masked parts in one call,
against the oracle's edges."""
import numpy as np
import pytest

from visacd_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu,nv", [(3, 3), (10, 5), (14, 9), (14, 10), (14, 11), (14, 14), (15, 14), (20, 14), (21, 14),
                                   (28, 14), (29, 14), (39, 14), (40, 14), (41, 14)])
def test_split_tiles_equal_oracle(ctx, orc, nu, nv):
    v, t = mg.torus(nu=nu, nv=nv, seed=nu)
    cv, ct = mg.offset_cage(v, t, 0.03)
    _, want, _ = orc.visibility(v, t, cv, ct)
    a, b = ctx.bvh(v, t), ctx.bvh(cv, ct)
    new = np.zeros(len(v), np.uint8)
    new[::3] = 1
    whole, masked = ctx.visibility_batch([(v, a, b, None), (v, a, b, new)])[0]
    np.testing.assert_array_equal(whole, want)
    np.testing.assert_array_equal(masked, want[(new[want[:, 0]] | new[want[:, 1]]).astype(bool)])
