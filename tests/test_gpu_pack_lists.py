"""The packer's shared candidate lists where they can go wrong: fewer particles than a warp or a
block takes, one more than a whole number of blocks, and radii spread over a factor of ten (cells
with tens of small particles: more pairs of a large one than are listed at a time), by brute force
over all pairs and the wall. Bound: the generator stops below a relative overlap of 2e-4 in the
last force pass; the update behind it moves a particle by less than that again (4e-4)."""
import numpy as np
import pytest

import rfdem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,rmin,phi", [(2, 0.8, 0.1), (5, 0.8, 0.2), (31, 0.8, 0.3), (33, 0.5, 0.3), (641, 0.5, 0.45),
                                        (1500, 0.1, 0.45), (4000, 0.1, 0.45)])
def test_pack_lists(cuda, n, rmin, phi):
    R, rad, D, H, mo = rfdem.pack_cylinder(n, 0.25, rmin=rmin, rmax=1.0, aspect=1.5, phi=phi, seed=n + 3,
                                           dist="log-uniform")
    assert mo < 2e-4
    P = R.reshape(3, n)
    assert np.all(np.sqrt(P[0] ** 2 + P[1] ** 2) + rad <= 0.5 * D + 4e-4 * rad)
    assert np.all(np.abs(P[2]) + rad <= 0.5 * H + 4e-4 * rad)
    dd = np.sqrt(((P.T[:, None, :] - P.T[None, :, :]) ** 2).sum(-1))
    np.fill_diagonal(dd, np.inf)
    ov = (rad[:, None] + rad[None, :] - dd) / np.minimum(rad[:, None], rad[None, :])
    assert ov.max() < 4e-4
    R2 = rfdem.pack_cylinder(n, 0.25, rmin=rmin, rmax=1.0, aspect=1.5, phi=phi, seed=n + 3, dist="log-uniform")[0]
    assert np.array_equal(R, R2)
