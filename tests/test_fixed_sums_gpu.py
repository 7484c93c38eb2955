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


# 3 nx ny K edge-levels on either side of the sizes at which the joint small
# launches end (2^16) and the PV, vertex and divergence sums begin (2^17)
@pytest.mark.parametrize("nx,ny,K", [(26, 28, 30), (26, 28, 31), (40, 34, 32),
                                     (40, 34, 33), (43, 64, 16), (210, 210, 1),
                                     (150, 146, 2)])
@pytest.mark.parametrize("T", [0, 2, 5])
def test_size_rule_edges(nx, ny, K, T):
    got, want = tendency(ALL if T else dict(ALL, eddy_diff4=0.0), K, T,
                         nx=nx, ny=ny)
    for g, w in zip(got, want):
        assert rel_diff(g, w) <= TOL


@pytest.mark.parametrize("T", [1, 5])
def test_large_with_magnitudes_beyond_the_words(T):
    """The velocity sums where the model has them in fixed point: zeros, tiny
    and mixed magnitudes beside ordinary ones."""
    def edit(h, vn, tr):
        vn[::3] = 0.0
        vn[1::7] *= 1e-99
        vn[2::11] *= 1e-9
        vn[:, 7] = 0.0
        tr[0][::2] = 0.0

    got, want = tendency(ALL, 33, T, edit, nx=40, ny=34)
    for g, w in zip(got, want):
        assert rel_diff(g, w) <= TOL


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("field", ["tr", "vn", "h"])
def test_large_not_finite(bad, field):
    def edit(h, vn, tr):
        if field == "tr":
            tr[0, 37, 5] = bad
        elif field == "vn":
            vn[101, 5] = bad
        else:
            h[55, 5] = bad

    got, want = tendency(ALL, 33, 2, edit, nx=40, ny=34)
    for g, w in zip(got, want):
        fine = np.isfinite(w)
        np.testing.assert_array_equal(np.isfinite(g), fine)
        assert rel_diff(np.where(fine, g, 0), np.where(fine, w, 0)) <= TOL


@pytest.mark.parametrize("shape,K,T", [((8, 6), 1, 9), ((40, 34), 33, 2),
                                       ((40, 34), 33, 6), ((26, 28), 30, 3)])
@pytest.mark.parametrize("size", [1, 12])
def test_batch_shapes_are_bitwise_alike(shape, K, T, size):
    """Members with and without words, with one and two elements a thread in
    the word-sum passes: every launch shape gives the single step's bits."""
    import torch
    members, single = [], []
    for i in range(size):
        k, t = max(1, K - 3 * (i % 5)), max(0, T - i % 3)
        mesh, params, model, _ = build(*shape, k, dict(ALL, T=t))
        x = state(mesh, t, 40 + i)
        a = og.ShallowWaterState(mesh, params)
        a.upload(*x)
        og.RK4Stepper(model).do_step(0.0, 1.0, a)
        single.append(a.download())
        members.append((mesh, params, model, x))
    states = [og.ShallowWaterState(m[0], m[1]) for m in members]
    b = og.Batch([m[2] for m in members], states, "rk4")
    for cfg in (None, 0, 4, 5, b.config_count() - 1):
        if cfg is not None:
            b.set_config(cfg)
        for s, m in zip(states, members):
            s.upload(*m[3])
        b.step(0.0, 1.0, 1)
        torch.cuda.synchronize()
        for s, want in zip(states, single):
            for g, w in zip(s.download(), want):
                np.testing.assert_array_equal(g, w)


@pytest.mark.parametrize("del4", [True, False])
def test_one_update_where_two_tracers_leave_the_words(del4):
    """A tracer whose own value alone is out of range keeps its sum; the same
    cell's other tracer, with such a neighbour, takes FP64.  Each is updated
    once."""
    cfg = ALL if del4 else dict(ALL, eddy_diff4=0.0)
    mesh, params, model, omd = build(10, 8, 33, dict(cfg, T=5))
    h, vn, tr = state(mesh, 5, 31)
    tr[1, 37, 5] = 1e150
    tr[2, 38, 5] = 1e150  # the east neighbour of 37
    S = og.ShallowWaterState(mesh, params)
    S.upload(h, vn, tr)
    og.LSRKStepper(model, 1).do_step(0.0, 1.0, S)
    want = omd.step(h.copy(), vn.copy(), tr.copy(), 0.0, 1.0, 1, kind="lsrk",
                    nstages=1)
    got = S.download()
    for g, w in zip(got[:2], want[:2]):
        assert rel_diff(g, w) <= TOL
    for g, w in zip(got[2], want[2]):
        assert rel_diff(g, w) <= TOL


@pytest.mark.parametrize("T,del4", [(1, True), (3, True), (3, False)])
def test_bad_weights_beside_finite_elements_in_a_batch(T, del4):
    """Batches large enough for two elements a thread in the word-sum passes:
    a cell whose weights are not finite skips its sums, and the thread's next
    element has the single step's bits all the same."""
    import torch
    cfg = ALL if del4 else dict(ALL, eddy_diff4=0.0)
    members, single = [], []
    for i in range(4):
        mesh, params, model, _ = build(40, 34, 33, dict(cfg, T=T))
        h, vn, tr = state(mesh, T, 60 + i)
        vn[i::37, 3::5] = np.nan
        vn[9::53, i] = np.inf
        vn[20::71, 2 * i + 1] = 1e-200  # F, and so the weight, below 2^-400
        a = og.ShallowWaterState(mesh, params)
        a.upload(h, vn, tr)
        og.LSRKStepper(model, 1).do_step(0.0, 1.0, a)
        single.append(a.download())
        assert np.isfinite(single[-1][2]).any()
        members.append((mesh, params, model, (h, vn, tr)))
    states = [og.ShallowWaterState(m[0], m[1]) for m in members]
    for s, m in zip(states, members):
        s.upload(*m[3])
    b = og.Batch([m[2] for m in members], states, "lsrk", 1)
    b.step(0.0, 1.0, 1)
    torch.cuda.synchronize()
    for s, want in zip(states, single):
        for g, w in zip(s.download(), want):
            np.testing.assert_array_equal(g, w)


@pytest.mark.parametrize("del4", [True, False])
def test_small_products_beside_calm_edges(del4):
    """Tracers whose products are near the words' lower end, beside zeros under
    larger weights (calm edges of every smaller magnitude): each tracer within
    the bound of its own scale, and updated once."""
    cfg = (ALL if del4 else
           dict(f0=1e-4, grav=9.81, visc_del2=1e3, visc_del4=1e9))
    mesh, params, model, omd = build(10, 8, 33, dict(cfg, T=5))
    h, vn, tr = state(mesh, 5, 31)
    for j, f in enumerate((1e-20, 1e-40, 0.0, 1e-60)):
        vn[j::5] *= f
    tr[1] *= 1e-70
    tr[2] *= 1e-80
    tr[3] *= 1e-90
    tr[1:4, ::3] = 0.0
    S = og.ShallowWaterState(mesh, params)
    S.upload(h, vn, tr)
    og.LSRKStepper(model, 1).do_step(0.0, 1.0, S)
    want = omd.step(h.copy(), vn.copy(), tr.copy(), 0.0, 1.0, 1, kind="lsrk",
                    nstages=1)
    got = S.download()
    for g, w in zip(got[:2], want[:2]):
        assert rel_diff(g, w) <= TOL
    for g, w in zip(got[2], want[2]):
        assert rel_diff(g, w) <= TOL


@pytest.mark.parametrize("stepper,nstages", [("lsrk", 1), ("rk4", 4)])
def test_taped_and_recomputed_pv_sums_agree(stepper, nstages):
    """Fluxes F that the words hold with products F Q that they do not: the
    edge pass takes both sums in FP64, and a gradient that reads the first one
    (the thickness gradient without the pressure term) does not depend on
    which steps the schedule tapes while it advances."""
    mesh, params, model, _ = build(40, 34, 33, dict(f0=1e-4, grav=9.81, T=0))
    model.m_ssh_grad_edge.m_enabled = False
    h, vn, tr = state(mesh, 0, 5)
    h[:] = 1000.0
    vn *= 1e-88
    seeds = [np.zeros_like(h), vn / np.abs(vn).max(), tr]
    grads, taped = [], []
    for nsnap in (1, 2, 12):
        adj = og.Adjoint(model, nsnap, stepper, nstages)
        x, xn, lam = (og.ShallowWaterState(mesh, params) for _ in range(3))
        x.upload(h, vn, tr)
        lam.upload(*seeds)
        adj.forward(x, 0.0, 1.0, 6, xn)
        adj.backward(lam)
        grads.append(lam.download())
        taped.append(og.adjoint_plan(6, nsnap, nstages)[1])
    assert len(set(taped)) > 1 and np.abs(grads[0][0]).max() > 0
    for g in grads[1:]:
        for a, b in zip(g, grads[0]):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("T", [0, 2])
def test_host_chunks_of_a_model_without_pv_words(T):
    """One TRiSK weight out of range: the model's PV sums are FP64, its vertex
    and divergence sums fixed-point still, and so are those of level chunks
    small enough for the joint launches."""
    import pyoracle
    from test_general_mesh_gpu import TABLES, models
    om = pyoracle.OracleMesh(40, 34, 1e4, 33)
    t = om.tables
    t["weights_on_edge"][7, 1] = 1e-130
    gm = og.MPASMesh.from_tables({n: t[n] for n in TABLES}, 33)
    _, gp, model = models(om, gm, T)
    x = state(gm, T, 3)
    S = og.ShallowWaterState(gm, gp)
    S.upload(*x)
    og.RK4Stepper(model).step(S, 0.0, 1.0, 1)
    hs = og.HostStepper(model, "rk4", 4, 8)
    arrs = hs.pinned_state()
    for a, b in zip(arrs, x):
        a[...] = b
    hs.step(*arrs, 0.0, 1.0, 1)
    for g, w in zip(arrs, S.download()):
        np.testing.assert_array_equal(g, w)


def test_equal_models_sum_alike_whatever_memory_is_free():
    """The words are chosen by the model's size, not by the free memory: a
    second model beside less free memory gives the first one's bits.  Where the
    words do not fit at all the model runs in FP64, within the parity bound."""
    import torch
    T, mb = 8, 1 << 20
    mesh, params, model, _ = build(128, 128, 64, dict(ALL, T=T))
    S, D = og.ShallowWaterState(mesh, params), og.ShallowWaterState(mesh, params)
    S.upload(*state(mesh, T, 31))
    model.compute_tendency(D, S, 0.0)
    want = D.download()
    cl = 8 * mesh.m_ncells * mesh.m_nlayers
    words, rest = 22 * cl, 43 * cl  # of both fluxes, 8 tracers and Laplacians

    def with_free(nbytes):
        torch.cuda.empty_cache()
        fill = torch.empty(torch.cuda.mem_get_info()[0] - nbytes,
                           dtype=torch.uint8, device="cuda")
        other = og.ShallowWaterModel(mesh, params)
        other.compute_tendency(D, S, 0.0)
        got = D.download()
        del other, fill
        torch.cuda.empty_cache()
        return got

    for g, w in zip(with_free(3 * words + 64 * mb), want):
        np.testing.assert_array_equal(g, w)
    for g, w in zip(with_free(rest + 96 * mb), want):
        assert rel_diff(g, w) <= TOL
    for g, w in zip(with_free(8 * (words + rest)), want):
        np.testing.assert_array_equal(g, w)


def _mesh_bytes(nx, K, edit=None):
    """Device memory of a mesh's tables."""
    import torch
    from test_general_mesh_gpu import TABLES
    h = og.PlanarHexagonalMesh(nx, nx, 1e4, K)
    t = {n: np.array(h.tables[n]) for n in TABLES}
    if edit:
        edit(t)
    del h
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    gm = og.MPASMesh.from_tables(t, K)
    assert gm.handle
    return before - torch.cuda.mem_get_info()[0]


def test_tables_are_kept_only_where_they_are_read():
    """The tables of the fixed-point sums (about 700 B per cell): not on a
    mesh of one level or below the size rule, nor with a weight they cannot
    hold."""
    cells, mb = 300 * 300, 1 << 20
    one = _mesh_bytes(300, 1)
    large = _mesh_bytes(300, 2)
    assert large - one >= 600 * cells
    small = _mesh_bytes(64, 8)  # below 2^17 edge-levels
    assert small <= one * 64 * 64 / cells + 32 * mb

    def edit(t):
        t["weights_on_edge"][7, 1] = 1e-130
        t["area_triangle"][5] *= 1e-70

    rejected = _mesh_bytes(300, 2, edit)
    # ten weights an edge instead of eight where the edit adds a ninth
    assert rejected - one <= 24 * 3 * cells + 8 * mb


def test_a_tendency_gradient_launches_no_pass_for_the_pv_sums():
    """One gradient of one tendency has no tape to fill: its launches are the
    same on either side of the size rule, and the dot product with the
    tangent-linear model holds."""
    counts = []
    for K in (32, 33):
        mesh, params, model, _ = build(40, 34, K, dict(ALL, T=2))
        adj = og.Adjoint(model, 1)
        x, dx, mu, lam, jd = (og.ShallowWaterState(mesh, params)
                              for _ in range(5))
        x.upload(*state(mesh, 2, 31))
        d, m = state(mesh, 2, 41), state(mesh, 2, 51)
        d = d[0] - 1000.0, 0.1 * d[1], d[2] - 1000.0
        m = m[0] - 1000.0, m[1], 1e-3 * m[2]
        dx.upload(*d)
        mu.upload(*m)
        n = og.kernel_launches()
        adj.adj_tendency(x, mu, lam)
        counts.append(og.kernel_launches() - n)
        adj.tlm_tendency(x, dx, jd)
        lhs = sum(float(np.sum(a * b)) for a, b in zip(jd.download(), m))
        rhs = sum(float(np.sum(a * b)) for a, b in zip(lam.download(), d))
        assert abs(lhs - rhs) <= 1e-12 * max(abs(lhs), abs(rhs))
    assert counts[0] == counts[1]


def test_not_finite_under_a_zero_kite_area():
    """A thickness that is not finite reaches the potential vorticity of a
    vertex through a kite area of zero too (0 x is NaN in FP64)."""
    from test_general_mesh_gpu import TABLES, models
    import pyoracle
    om = pyoracle.OracleMesh(40, 34, 1e4, 33)
    t = om.tables
    t["kiteareas_on_vertex"][::2, 1] = 0.0
    gm = og.MPASMesh.from_tables({n: t[n] for n in TABLES}, 33)
    _, gp, model = models(om, gm, 0)
    h, vn, _ = state(gm, 0, 3)
    h[55, 5], h[700, 9] = np.nan, np.inf
    S, D = og.ShallowWaterState(gm, gp), og.ShallowWaterState(gm, gp)
    S.upload(h, vn)
    model.compute_tendency(D, S, 0.0)
    q = model.aux("q_vertex").reshape(gm.m_nvertices, 33)
    k, cv = t["kiteareas_on_vertex"], t["cells_on_vertex"]
    with np.errstate(invalid="ignore"):
        hv = sum(k[:, j, None] * h[cv[:, j]] for j in range(3))
    assert (~np.isfinite(hv)).any(axis=1)[::2].any()
    np.testing.assert_array_equal(np.isnan(q), ~np.isfinite(hv))


def _beyond(mesh, T, seed, bad=None):
    """A state with magnitudes beyond the words, and some values `bad`."""
    h, vn, tr = state(mesh, T, seed)
    tr[1] *= 1e-100
    tr[2, ::2] = 0.0
    tr[2, 1::4] *= 1e-97
    vn[::3] = 0.0
    vn[1::7] *= 1e-99
    if bad is not None:
        tr[0, 7, 3] = bad
        vn[11, 2] = bad
    return h, vn, tr


@pytest.mark.parametrize("bad", [None, np.nan])
@pytest.mark.parametrize("shape,K", [((10, 8), 33), ((24, 20), 37)])
def test_noalloc_tendency_beyond_the_words(shape, K, bad):
    from test_zz_no_alloc import _noalloc
    mesh, params, model, _ = build(*shape, K, dict(ALL, T=3))
    S, A, B = (og.ShallowWaterState(mesh, params) for _ in range(3))
    S.upload(*_beyond(mesh, 3, 31, bad))
    model.compute_tendency(A, S, 0.0)
    assert _noalloc(mesh, params, S, B) == 0
    og.sync()
    want, got = A.download(), B.download()
    for g, w in zip([*got[:2], *got[2]], [*want[:2], *want[2]]):
        fine = np.isfinite(w)
        np.testing.assert_array_equal(np.isfinite(g), fine)
        assert rel_diff(np.where(fine, g, 0), np.where(fine, w, 0)) <= TOL


@pytest.mark.parametrize("shape,K", [((10, 8), 33), ((40, 34), 33)])
def test_taped_steps_beyond_the_words(shape, K):
    """Adjoints of such states: an ensemble's members bitwise equal to single
    adjoints, the taped forward bitwise equal to the plain stepper."""
    members, want = [], []
    for i in range(3):
        mesh, params, model, _ = build(*shape, K - i, dict(ALL, T=3))
        x, mu = _beyond(mesh, 3, 31 + i), state(mesh, 3, 51 + i)
        adj = og.Adjoint(model, 2)
        S, F, L, P = (og.ShallowWaterState(mesh, params) for _ in range(4))
        S.upload(*x)
        P.upload(*x)
        L.upload(*mu)
        adj.forward(S, 0.0, 1.0, 4, F)
        adj.backward(L)
        og.RK4Stepper(model).step(P, 0.0, 1.0, 4)
        for g, w in zip(F.download(), P.download()):
            np.testing.assert_array_equal(g, w)
        want.append((F.download(), L.download()))
        members.append((model, adj, S, F, L, x, mu))
    ens = og.AdjointEnsemble([m[1] for m in members])
    for _, _, S, _, L, x, mu in members:
        S.upload(*x)
        L.upload(*mu)
    ens.forward([m[2] for m in members], 0.0, 1.0, 4, [m[3] for m in members])
    ens.backward([m[4] for m in members])
    og.sync()
    for m, w in zip(members, want):
        for got, ref in zip((m[3].download(), m[4].download()), w):
            for g, r in zip(got, ref):
                assert np.isfinite(r).all()
                np.testing.assert_array_equal(g, r)
