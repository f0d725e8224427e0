"""Specimens whose particles have more neighbours than a row has slots (K < 32): rows are cut at
K and the overflow is reported. Rows, masks and steps of both models against the md_* construction
sequence and the oracle, which cut in the same place."""
import numpy as np
import pytest

import extspec
import mdcall as mc
import oracle
import rfdem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [8, 12, 16])
def test_cut_rows_reference_model(cuda, K):
    t, R = rfdem.make_test(rfdem.RF_TEST_UNIAXIAL, 9.0, 14.0, seed=0xB2000000 + K, K=K, max_strain=1.0, v_load=-1e-3)
    N = R.size // 3
    _, _, CIs, pnC = mc.oracle_cells(t, R)
    s, IL = mc.gpu_list_construct(cuda, t, R, CIs, pnC)
    assert s == rfdem.RF_ERR_ROW_OVERFLOW
    ty, iL, S = np.zeros(N * K, np.uint8), np.zeros(N * K, np.float32), mc.zeros_state(N, K)
    IL, ty, iL, S = mc.gpu_bonds_delete(cuda, t, R, IL, ty, iL, S, np.float32(t.Po.b_dd), np.float32(t.Po.aa_farcut))
    e = rfdem.Engine(mc.clone(t), R)
    st, n = e.export(), e.counters()
    assert e.sync()[1].error == rfdem.RF_ERR_ROW_OVERFLOW
    assert np.array_equal(st["IL"].astype(np.uint64), IL.astype(np.uint64))
    assert np.array_equal(st["ILtype"], ty) and np.array_equal(st["iL"], iL)
    assert n["occupied"] == int((IL != rfdem.EMPTY).sum()) and n["bonds"] == int(ty.sum())
    _, want = mc.oracle_state_after(t, R, 20)
    e.step(20)
    assert e.sync()[1].error == rfdem.RF_ERR_ROW_OVERFLOW
    out, n = e.export(), e.counters()
    e.close()
    for k in ("R", "V", "W", "IL", "ILtype", "Rij", "Oijt", "Mijn", "Mijt"):
        assert np.array_equal(np.asarray(out[k], want[k].dtype), want[k]), k
    assert n["occupied"] == int((want["IL"] != oracle.EMPTY64).sum())


@pytest.mark.parametrize("K,gap", [(4, 0.05), (8, 0.0), (12, 0.0), (16, 0.0)])
def test_cut_rows_extended_model(cuda, K, gap):
    t, R, rad, x = extspec.ext_case(rfdem.RF_TEST_UNIAXIAL, 6.0, 10.0, min_stress=1e3, K=K)
    x.list_gap = gap
    e = rfdem.Engine(mc.clone(t), R, ext=x, radius=rad)
    for steps in (0, 20):
        o = oracle.run_ext(mc.clone(t), x, R, rad, steps)
        assert o["status"] == rfdem.RF_ERR_ROW_OVERFLOW
        if steps:
            e.step(steps)
        assert e.sync()[1].error == rfdem.RF_ERR_ROW_OVERFLOW
        st, n = e.export(), e.counters()
        assert np.array_equal(st["IL"].astype(np.uint64), o["IL"]) and np.array_equal(st["ILtype"], o["ILtype"])
        assert n["occupied"] == int((o["IL"] != oracle.EMPTY64).sum()) and n["bonds"] == int(o["ILtype"].sum())
        assert np.array_equal(e.positions_f64(), o["R"])
    e.close()
