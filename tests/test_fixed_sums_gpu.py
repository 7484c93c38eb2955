"""The passes with fixed-point sums against the oracle, at the edges of the
rule that picks them (levels, tracers, del4) and with values they leave to
FP64: magnitudes beyond the words' range, zeros beside them, NaN and
infinities."""
import numpy as np
import pytest

import omega_playground_gb300 as og
from helpers import rel_diff
from test_config_matrix_gpu import ALL, build, state

pytestmark = pytest.mark.gpu

# the parity bound of every tendency test: maximum difference over maximum
TOL = 1e-12


def tendency(cfg, K, T, edit=None, nx=10, ny=8):
    mesh, params, model, omd = build(nx, ny, K, dict(cfg, T=T))
    x = state(mesh, T, 31)
    if edit:
        edit(*x)
    S, D = og.ShallowWaterState(mesh, params), og.ShallowWaterState(mesh, params)
    S.upload(*x)
    model.compute_tendency(D, S, 0.0)
    return D.download(), omd.compute_tendency(*x)


@pytest.mark.parametrize("K", [1, 2, 3, 31, 32, 65])
@pytest.mark.parametrize("T,del4", [(0, True), (1, True), (2, False),
                                    (3, False), (5, True), (8, True)])
def test_rule_edges(K, T, del4):
    cfg = ALL if del4 else dict(ALL, eddy_diff4=0.0)
    got, want = tendency(cfg, K, T)
    for g, w in zip(got, want):
        assert rel_diff(g, w) <= TOL


@pytest.mark.parametrize("del4", [True, False])
def test_magnitudes_beyond_the_words(del4):
    """Each tracer is held to its own scale: far below and far above the
    range of the words, and mixed with zeros and tiny values."""
    def edit(h, vn, tr):
        tr[1] *= 1e-100
        tr[2] *= 1e28
        tr[3][::2] = 0.0
        tr[3][1::4] *= 1e-97
        tr[4] = 0.0
        vn[::3] = 0.0
        vn[1::7] *= 1e-99

    cfg = ALL if del4 else dict(ALL, eddy_diff4=0.0)
    got, want = tendency(cfg, 33, 5, edit)
    assert rel_diff(got[0], want[0]) <= TOL
    assert rel_diff(got[1], want[1]) <= TOL
    for g, w in zip(got[2], want[2]):
        assert rel_diff(g, w) <= TOL
    assert not got[2][4].any()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("field", ["tr", "vn"])
def test_not_finite(bad, field):
    """A value that is not finite reaches exactly the elements it reaches in
    the oracle, and no other changes."""
    def edit(h, vn, tr):
        if field == "tr":
            tr[1, 37, 5] = bad
        else:
            vn[101, 5] = bad

    got, want = tendency(ALL, 33, 3, edit)
    for g, w in zip(got, want):
        fine = np.isfinite(w)
        np.testing.assert_array_equal(np.isfinite(g), fine)
        assert rel_diff(np.where(fine, g, 0), np.where(fine, w, 0)) <= TOL
