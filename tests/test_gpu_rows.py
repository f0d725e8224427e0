"""Rows, bonds and candidate lists of a fresh engine at the sizes its kernels can go wrong at
(one particle, around a warp's and a CTA's particles, short rows): the reference model against
the md_* construction sequence it replaces, slot for slot; the extended model against the
oracle's start state; and one step of every particles-a-warp variant against the oracle."""
import numpy as np
import pytest

import extspec
import mdcall as mc
import oracle
import rfdem

pytestmark = pytest.mark.gpu


def _cut(t, R, n):
    """The first n particles of a specimen."""
    N = R.size // 3
    n = min(n, N)
    R = R.reshape(3, N)[:, :n].reshape(-1).copy()
    t.N = n
    t.bloks = n // 1024 + 1
    return t, R


@pytest.mark.parametrize("n,K", [(1, 32), (2, 32), (31, 32), (33, 20), (128, 32), (129, 18), (585, 24)])
def test_fresh_rows_match_md_sequence(cuda, n, K):
    t, R = rfdem.make_test(rfdem.RF_TEST_UNIAXIAL, 9.0, 14.0, seed=0xB2000000 + n, K=K)
    t, R = _cut(t, R, n)
    N = R.size // 3
    e = rfdem.Engine(mc.clone(t), R)
    st = e.export()
    bonds = e.counters()["bonds"]
    e.close()
    _, _, CIs, pnC = mc.oracle_cells(t, R)
    s, IL = mc.gpu_list_construct(cuda, t, R, CIs, pnC)
    assert s == 0
    ty, iL, S = np.zeros(N * K, np.uint8), np.zeros(N * K, np.float32), mc.zeros_state(N, K)
    IL, ty, iL, S = mc.gpu_bonds_delete(cuda, t, R, IL, ty, iL, S, np.float32(t.Po.b_dd), np.float32(t.Po.aa_farcut))
    assert np.array_equal(st["IL"].astype(np.uint64), IL.astype(np.uint64))
    assert np.array_equal(st["ILtype"], ty) and np.array_equal(st["iL"], iL)
    assert bonds == int(ty.sum()) and not st["Oijt"].any() and not st["Rij"].any()


@pytest.mark.parametrize("n,gap", [(2, 0.0), (33, 0.05), (300, 0.0), (300, 0.05)])
def test_fresh_rows_extended_match_oracle(cuda, n, gap):
    t, R, rad, x = extspec.ext_case(rfdem.RF_TEST_UNIAXIAL, 6.0, 10.0, min_stress=1e3)
    t, R = _cut(t, R, n)
    rad = rad[:int(t.N)].copy()
    x.list_gap = gap
    o = oracle.run_ext(mc.clone(t), x, R, rad, 0)
    e = rfdem.Engine(mc.clone(t), R, ext=x, radius=rad)
    st = e.export()
    e.close()
    assert np.array_equal(st["IL"].astype(np.uint64), o["IL"]) and np.array_equal(st["ILtype"], o["ILtype"])


@pytest.mark.parametrize("d,h,steps", [(9.0, 14.0, 300), (21.0, 26.0, 40), (34.0, 44.0, 10), (41.0, 70.0, 6)])
def test_step_variants_bitexact(cuda, d, h, steps):
    """Specimens on both sides of the sizes at which the step takes 4, 8, 16 and 32 particles a warp."""
    t, R = rfdem.make_test(rfdem.RF_TEST_UNIAXIAL, d, h, seed=0xB2000000 + 5, max_strain=1.0, v_load=-1e-3)
    _, st = mc.oracle_state_after(t, R, steps)
    e = rfdem.Engine(mc.clone(t), R)
    e.step(steps)
    out = e.export()
    e.close()
    for k in ("R", "V", "W", "IL", "ILtype", "Rij", "Oijt", "Mijn", "Mijt"):
        assert np.array_equal(np.asarray(out[k], st[k].dtype), st[k]), k
