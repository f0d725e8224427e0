"""The FIRE loop's graph body holds several iterations, and what follows an update that asks for new
candidate lists leaves without doing anything. The plain launches (RF_ENGINE_NO_GRAPH) look for a
rebuild before every iteration: both must give the same bits, through rebuilds inside an increment."""
import numpy as np
import pytest

import extspec
import mdcall as mc
import rfdem
from test_gpu_batch import _specimens

pytestmark = pytest.mark.gpu

FIELDS = ("R", "V", "W", "IL", "ILtype", "Rij", "Oijt", "Mijn", "Mijt")


def _increments(make, n, **params):
    e = make()
    p = e.relax_params(**params)
    res = [e.load_increment(p) for _ in range(n)]
    if not isinstance(res[0], list):
        res = [[r] for r in res]
    log = [(r.iterations, r.converged, r.residual, r.stress, r.error) for rk in res for r in rk]
    out = e.export()
    out["R64"] = e.positions_f64()
    n_rebuilds, graph = e.counters()["rebuilds"], e.uses_graph()
    e.close()
    return log, out, n_rebuilds, graph


def _compare(make, monkeypatch, n, **params):
    log, a, na, graph = _increments(make, n, **params)
    assert graph
    monkeypatch.setenv("RF_ENGINE_NO_GRAPH", "1")
    log2, b, nb, graph2 = _increments(make, n, **params)
    assert not graph2
    print("iterations", [q[0] for q in log], "rebuilds", na)
    assert log == log2
    assert na == nb > 2 * n                          # (one at each start; the rest inside)
    for k in FIELDS + ("R64",):
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("kind,d,h", [(rfdem.RF_TEST_UNIAXIAL, 6.0, 10.0), (rfdem.RF_TEST_BRAZIL, 10.0, 4.0),
                                      (rfdem.RF_TEST_UNIAXIAL, 21.0, 30.0)], ids=["uniaxial", "brazil", "9k"])
def test_graph_body_equals_plain_launches(cuda, monkeypatch, kind, d, h):
    t, R, rad, x = extspec.ext_case(kind, d, h, min_stress=1e3)
    _compare(lambda: rfdem.Engine(mc.clone(t), R, ext=x, radius=rad), monkeypatch, 3, max_iter=1500,
             strain_inc=2e-2 if kind == rfdem.RF_TEST_UNIAXIAL else 1e-2)


def test_graph_body_equals_plain_launches_batch(cuda, monkeypatch):
    specs = _specimens()
    _compare(lambda: rfdem.BatchEngine([mc.clone(s[0]) for s in specs], [s[3] for s in specs], [s[1] for s in specs],
                                       [s[2] for s in specs]), monkeypatch, 3, max_iter=1500, strain_inc=2e-2)
