"""The step rule where the sums of an attempt overflow (src/pdhg/pdhg.cu:770-794):
an infinite dy . A dx beside finite norms gives etabar = 0 and a rejected step, on
the cluster kernel and on the grid-wide ones."""
import numpy as np
import pytest

from igaos_gb300 import generators as G

pytestmark = pytest.mark.gpu


def overflowing_lp():
    """4 x 4, all ones, A~ = A, ||A~|| = 4, eta = 0.3, omega = 1 (no row bounds of
    size): the first step moves x by 0.3 |c| and y by 2.4 times that; dx^2, dy^2 and
    dy . A dx are 4, 23 and 38 times its square."""
    dx = 2.5e153
    i, j = np.divmod(np.arange(16), 4)
    inf = np.full(4, np.inf)
    return G.from_triplets(4, 4, j, i, np.ones(16), np.full(4, -dx / 0.3), -inf, inf, np.zeros(4), np.zeros(4))


@pytest.mark.parametrize("cluster", ["1", "0"])
def test_infinite_product_is_a_rejected_step(native, orc, monkeypatch, cluster):
    from igaos_gb300 import capi
    monkeypatch.setenv("IGAOS_PDHG_CLUSTER", cluster)
    lp = overflowing_lp()
    olp = orc.lp_from(lp)
    sd = orc.scale(olp, *orc.ruiz(olp))
    with capi.Problem(lp) as P:
        _, eta0, omega0 = P.step_init()
        assert abs(eta0 - 0.3) < 1e-12 and omega0 == 1.0
        z = lambda: np.zeros(4)
        st = dict(x=z(), y=z(), xavg=z(), yavg=z(), axcur=z(), eta=eta0, omega=omega0, k=1, hn=0)
        got = P.iterate(st, 1, "fp64")
    want, attempts = orc.iterate(olp, sd, st, 1)
    assert got["attempts"] == attempts == 2
    assert np.all(np.abs(want["x"]) < 1e150)
    for key in ("x", "y", "xavg", "yavg"):
        assert np.allclose(got[key], want[key], rtol=1e-12, atol=0.0), key
    assert got["eta"] == want["eta"] and got["k"] == want["k"]
