"""The md_* row kernels at the edges of their tiling: rows shorter than a warp, longer than
one and longer than the staged ones, particle counts off the rows a warp takes, slots
scattered over the row, contacts and broken bonds; bit for bit against the oracle."""
import numpy as np
import pytest

import mdcall as mc
import rfdem

pytestmark = pytest.mark.gpu


def _state(K, d, h):
    """A specimen squeezed so that its broken pairs overlap, its rows' slots scattered over
    K slots, random bond state, velocities and spins (some particles at rest)."""
    t, R = rfdem.make_test(rfdem.RF_TEST_UNIAXIAL, d, h, seed=0xB2000000 + K)
    t.K = K
    N = R.size // 3
    rng = np.random.default_rng(K)
    c = np.repeat(np.array([t.S.center.x, t.S.center.y, t.S.center.z], np.float32), N)
    R = (c + np.float32(0.985) * (R - c)).astype(np.float32)
    _, _, CIs, pnC = mc.oracle_cells(t, R)
    so, IL = mc.oracle_list_construct(t, R, CIs, pnC)
    assert so == 0
    ty, iL, S = np.zeros(N * K, np.uint8), np.zeros(N * K, np.float32), mc.zeros_state(N, K)
    IL, ty, iL, S = mc.oracle_bonds_delete(t, R, IL, ty, iL, S, np.float32(t.Po.b_dd), np.float32(t.Po.aa_farcut), True,
                                           False)
    order = np.argsort(rng.random((N, K)), 1)
    perm = lambda a: np.take_along_axis(a.reshape(N, K), order, 1).reshape(-1).copy()   # noqa: E731
    IL, ty, iL = perm(IL), perm(ty), perm(iL)
    ty[rng.random(N * K) < 0.2] = 0
    live = np.repeat(IL != rfdem.EMPTY, 3)
    for k in ("Oijt", "Mijn", "Mijt"):
        S[k] = (rng.normal(scale=1e-4, size=3 * N * K) * live).astype(np.float32)
    n = rng.normal(size=(N * K, 3))
    S["Rij"] = ((n / np.linalg.norm(n, axis=1, keepdims=True)).reshape(-1) * live).astype(np.float32)
    V, W = (rng.normal(scale=1e-3, size=3 * N).astype(np.float32) for _ in range(2))
    for a in range(3):
        W[a * N: a * N + 40] = 0.0          # the rolling rule's clear
    return t, R, V, W, IL, ty, iL, S, CIs, pnC


@pytest.mark.parametrize("K,d,h", [(18, 5.0, 6.0), (32, 9.0, 13.0), (33, 7.0, 9.0), (70, 6.0, 5.0), (600, 4.0, 4.0)])
def test_row_kernels_bitexact(cuda, K, d, h):
    t, R, V, W, IL, ty, iL, S, CIs, pnC = _state(K, d, h)
    N = R.size // 3
    g = mc.gpu_forces(cuda, t, R, V, W, IL, ty, iL, S)
    o = mc.oracle_forces(t, R, V, W, IL, ty, iL, S)
    for k in ["F", "M", "ty", "Rij", "Oijt", "Mijn", "Mijt"]:
        assert np.array_equal(g[k].view(np.uint8), o[k].view(np.uint8)), k
    assert np.abs(o["M"]).max() > 0 and np.abs(o["Oijt"]).max() > 0
    # holes to refill, then links to delete
    rng = np.random.default_rng(1)
    holes = IL.copy()
    live = np.nonzero(holes != rfdem.EMPTY)[0]
    holes[rng.choice(live, size=max(1, len(live) // 50), replace=False)] = rfdem.EMPTY
    st, ILg, tyg = mc.gpu_reconstruct(cuda, t, R, CIs, pnC, holes, ty)
    so, ILo, tyo = mc.oracle_reconstruct(t, R, CIs, pnC, holes, ty)
    assert st == so and np.array_equal(ILg, ILo) and np.array_equal(tyg, tyo)
    R2 = R + rng.normal(scale=0.12, size=R.size).astype(np.float32)
    a = mc.gpu_bonds_delete(cuda, t, R2, IL, ty, iL, S, 0.0, np.float32(t.Po.aa_farcut), False, True)
    b = mc.oracle_bonds_delete(t, R2, IL, ty, iL, S, 0.0, np.float32(t.Po.aa_farcut), False, True)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    for k in ["Rij", "Oijt", "Mijn", "Mijt"]:
        assert np.array_equal(a[3][k], b[3][k])


def test_cells_crowded_and_out_of_grid(cuda):
    """Cell lists with cells of more than a warp's ids, exactly a warp's, and particles outside
    the grid (the tail bin, ordered by key and id)."""
    t, R = rfdem.make_test(rfdem.RF_TEST_UNIAXIAL, 9.0, 14.0)
    N = R.size // 3
    rng = np.random.default_rng(4)
    X = R.reshape(3, N).copy()
    p = rng.permutation(N)
    X[:, p[:100]] = X[:, p[100]:p[100] + 1]
    X[:, p[101:133]] = np.array([[t.C.a * 1.5]] * 3, np.float32)
    X[2, p[200:260]] = 1e4 * (1 + np.arange(60) % 7)
    R2 = X.reshape(-1).copy()
    st, CI, CIs, pnC = mc.gpu_cells(cuda, t, R2)
    so, CIo, CIso, pnCo = mc.oracle_cells(t, R2)
    assert st == so != 0
    assert np.array_equal(CI, CIo) and np.array_equal(CIs, CIso) and np.array_equal(pnC, pnCo)
