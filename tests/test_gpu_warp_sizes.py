"""The extended model's step at every number of particles a warp takes (4 up to about 7,100
particles, 8 up to 28,400, 16 up to 56,800, 32 beyond): explicit steps and FIRE increments of one
specimen against the oracle, and batches whose specimens share CTAs against the oracle and against
the same specimens alone. The other tests of the extended model run specimens of 4."""
import numpy as np
import pytest

import extspec
import mdcall as mc
import oracle
import rfdem
from test_gpu_batch import _check_against_oracle

pytestmark = pytest.mark.gpu

# Fragments of these violent windows may move more than half the lists' skin between two looks at
# it; the engine reports that (RF_ERR_CAPACITY, 6) and goes on.
STATUS = (0, 6)
SIZES = [(rfdem.RF_TEST_UNIAXIAL, 21.0, 30.0), (rfdem.RF_TEST_BRAZIL, 52.0, 20.0), (rfdem.RF_TEST_UNIAXIAL, 41.0, 55.0)]
IDS = ["8", "16", "32"]


@pytest.mark.parametrize("tuned", [False, True], ids=["default", "autotuned"])
@pytest.mark.parametrize("kind,d,h", SIZES, ids=IDS)
def test_explicit_steps_bitexact(cuda, kind, d, h, tuned):
    """A strained specimen: bonds break, pairs overlap and links come and go within 40 steps."""
    t, R, rad, x = extspec.ext_case(kind, d, h, min_stress=1e3, max_strain=1.0)
    x.list_gap = 0.05
    strain, steps = (-0.02, 0.01, -0.04), 40
    o = oracle.run_ext(mc.clone(t), x, R, rad, steps, strain=strain)
    e = rfdem.Engine(mc.clone(t), R, ext=x, radius=rad)
    e.affine_strain(*strain)
    if tuned:
        e.autotune(20)
    e.step(steps)
    _, res = e.sync()
    st, R64, curve = e.export(), e.positions_f64(), e.curve()
    e.close()
    np.testing.assert_allclose(curve, o["curve"], rtol=1e-9, atol=1e-12)    # (FP64 sums in another order)
    N, K = int(t.N), int(t.K)
    bonds, contacts = extspec.pair_counts(o["R"], N, K, o["IL"], o["ILtype"], rad)
    start = oracle.run_ext(mc.clone(t), x, R, rad, 0)
    assert o["broken"] > N and contacts > N // 4 and bonds > N // 8 and (start["IL"] != o["IL"]).any()
    assert o["status"] == 0 and res.error in STATUS and res.steps == steps and res.broken_bonds == o["broken"]
    assert np.array_equal(R64, o["R"]), np.abs(R64 - o["R"]).max()
    assert np.array_equal(st["V"], o["V"])
    assert np.array_equal(st["IL"].astype(np.uint64), o["IL"]) and np.array_equal(st["ILtype"], o["ILtype"])


@pytest.mark.parametrize("kind,d,h", SIZES, ids=IDS)
def test_fire_increments_vs_oracle(cuda, kind, d, h):
    """Two increments of 20 iterations each. The arithmetic is the oracle's up to the order of the
    FP64 sums, which reaches the motion through FP32 FIRE scalars: 6e-8 an iteration of a motion of
    2e-4 of the specimen, 5e-10 of it over 40."""
    t, R, rad, x = extspec.ext_case(kind, d, h, min_stress=1e3)
    e = rfdem.Engine(mc.clone(t), R, ext=x, radius=rad)
    p = e.relax_params(max_iter=20, strain_inc=1e-4)
    res = [e.load_increment(p) for _ in range(2)]
    Re = e.positions_f64()
    e.close()
    o = oracle.qs_ext(mc.clone(t), x, R, rad, p, 2)
    assert [r.iterations for r in res] == o["iters"].tolist() and all(r.error == 0 for r in res)
    ext = float(np.ptp(R))
    assert np.max(np.abs(o["R"] - R)) > 1e-5 * ext
    assert np.max(np.abs(Re - o["R"])) < 1e-8 * ext, np.abs(Re - o["R"]).max() / ext
    for r, s, q in zip(res, o["stress"], o["residual"]):
        assert abs(r.stress - s) <= 1e-4 * abs(s) and abs(r.residual - q) <= 1e-4 * q


@pytest.mark.parametrize("nspec", [10, 24, 40], ids=IDS)
def test_batches(cuda, nspec):
    """Weak specimens of three sizes (none a multiple of 128 particles) under a fast platen: 60
    explicit steps with breaking bonds and contacts, bit for bit the oracle's, then two FIRE
    increments of the damaged specimens, each as in an engine of its own (bounds of the batched
    FIRE test)."""
    po = rfdem.granite_potential()
    specs = []
    for q in range(nspec):
        d, h = [(12.0, 18.0), (11.0, 19.0), (13.0, 16.0)][q % 3]
        R0, rad = extspec.lattice_ext(rfdem.RF_TEST_UNIAXIAL, d, h, seed=0xB2000000 + 100 + q)
        t, R = rfdem.make_test_ext(rfdem.RF_TEST_UNIAXIAL, R0, rad, 0.5, v_load=-5e-2, min_stress=1e3, max_strain=1.0)
        specs.append((t, R, rad, extspec.stiff_params(seed=0xB2000000 + 200 + q, weibull_m=3.0, sigma_c=po.m_Ec * 0.05,
                                                      tau_c=po.m_Gc * 0.05)))
    assert all(int(s[0].N) % 128 for s in specs)
    e = rfdem.BatchEngine([s[0] for s in specs], [s[3] for s in specs], [s[1] for s in specs], [s[2] for s in specs])
    steps = 60
    e.step(steps)
    _check_against_oracle(e, specs, [steps] * nspec)
    c = e.counters()
    assert c["contacts"] > 100 * nspec and e.sync()[1].broken_bonds > 1000 * nspec
    p = e.relax_params(max_iter=30, strain_inc=1e-4)
    res = [e.load_increment(p) for _ in range(2)]
    Rall = e.positions_f64()
    for q in range(0, nspec, 3 if nspec < 30 else 5):
        t, R, rad, x = specs[q]
        first, m, off, tq = e.spec_info(q)
        Rq = R.reshape(3, m).copy()
        Rq[0] += off
        a = rfdem.Engine(mc.clone(tq), Rq.reshape(-1), ext=x, radius=rad)
        a.step(steps)
        ra = [a.load_increment(p) for _ in range(2)]
        Ra = a.positions_f64()
        a.close()
        ext = float(np.ptp(Rq[2]))
        Re = Rall.reshape(3, e.N)[:, first:first + m].reshape(-1)
        for k in range(2):
            assert res[k][q].error in STATUS and res[k][q].iterations == ra[k].iterations
            assert abs(res[k][q].stress - ra[k].stress) <= 1e-6 * abs(ra[k].stress)
        assert np.max(np.abs(Re - Ra)) < 1e-7 * ext, (q, np.abs(Re - Ra).max() / ext)
    e.close()


def test_two_large_specimens(cuda):
    """A batch whose specimens' sums take the paths of many CTAs (more than 256 each, in several FIRE
    groups) and meet in one CTA: explicit steps and load curves against the oracle, then FIRE
    increments as in an engine of their own."""
    specs = []
    for q, (d, h) in enumerate([(34.0, 44.0), (33.0, 45.0)]):
        R0, rad = extspec.lattice_ext(rfdem.RF_TEST_UNIAXIAL, d, h, seed=0xB2000000 + 300 + q)
        t, R = rfdem.make_test_ext(rfdem.RF_TEST_UNIAXIAL, R0, rad, 0.5, v_load=-5e-2, min_stress=1e3, max_strain=1.0)
        specs.append((t, R, rad, extspec.stiff_params(seed=0xB2000000 + 310 + q)))
    assert all(int(s[0].N) > 256 * 128 and int(s[0].N) % 128 for s in specs)
    e = rfdem.BatchEngine([s[0] for s in specs], [s[3] for s in specs], [s[1] for s in specs], [s[2] for s in specs])
    steps = 40
    e.step(steps)
    _check_against_oracle(e, specs, [steps] * 2)
    curves = [e.curve_spec(q) for q in range(2)]
    p = e.relax_params(max_iter=12, strain_inc=1e-4)
    res = [e.load_increment(p) for _ in range(2)]
    Rall = e.positions_f64()
    for q, (t, R, rad, x) in enumerate(specs):
        first, m, off, tq = e.spec_info(q)
        Rq = R.reshape(3, m).copy()
        Rq[0] += off
        o = oracle.run_ext(mc.clone(tq), x, Rq.reshape(-1), rad, steps)
        assert (o["curve"] != 0).any(0).all()
        np.testing.assert_allclose(curves[q], o["curve"], rtol=1e-9, atol=1e-12)
        a = rfdem.Engine(mc.clone(tq), Rq.reshape(-1), ext=x, radius=rad)
        a.step(steps)
        ra = [a.load_increment(p) for _ in range(2)]
        Ra = a.positions_f64()
        a.close()
        for k in range(2):
            assert res[k][q].iterations == ra[k].iterations
            assert abs(res[k][q].stress - ra[k].stress) <= 1e-6 * abs(ra[k].stress)
            assert abs(res[k][q].residual - ra[k].residual) <= 1e-6 * ra[k].residual
        Re = Rall.reshape(3, e.N)[:, first:first + m].reshape(-1)
        assert np.max(np.abs(Re - Ra)) < 1e-7 * float(np.ptp(Rq[2]))
    e.close()


@pytest.mark.parametrize("kind,d,h,steps", [(rfdem.RF_TEST_UNIAXIAL, 21.0, 26.0, 40), (rfdem.RF_TEST_BRAZIL, 52.0, 20.0, 20),
                                            (rfdem.RF_TEST_UNIAXIAL, 41.0, 70.0, 6)], ids=IDS)
def test_reference_model_load_curves(cuda, kind, d, h, steps):
    t, R = rfdem.make_test(kind, d, h, seed=0xB2000000 + 5, max_strain=1.0, v_load=-1e-2)
    n, _, curve, status = oracle.run_f(mc.clone(t), R, steps)
    assert n == steps and status == 0 and np.abs(curve[:, 1:]).max(0).all()
    e = rfdem.Engine(t, R)
    e.step(steps)
    got = e.curve()
    e.close()
    np.testing.assert_allclose(got, curve, rtol=1e-9, atol=1e-12)
