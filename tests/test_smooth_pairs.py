"""The two-walks-per-lane passes of the smoothed form where they can go wrong: bins with one,
two, odd and just over a warp's lineages, one candidate and one more than a warp's lanes, types
whose walks fall back to one at a time (quiescent, zero mean, the FP64 form), against the FP64
CPU restatement with the tolerances of tests/test_smooth.py; and Gauss-Newton systems of one to
eight types against their Jacobian."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("candidates", [1, 32, 33, 65])
@pytest.mark.parametrize("h", [0.5, 1e-7])  # 1e-7: beyond the grid form's error bound
def test_passes_at_their_edges(engine, candidates, h):
    import smooth_ref
    import torch
    from procell.smooth import Smooth
    bins = [(900.0, 1), (300.0, 2), (77.0, 3), (640.0, 31), (37.0, 33), (1.5, 5), (150.0, 65), (0.6, 4), (20.0, 129)]
    sets = [[[0.5, 30.0, 6.0], [0.3, 45.0, 18.0], [0.2, -1.0, -1.0]], [[0.6, 25.0, 12.0], [0.4, 0.0, 1.0], [0.0, 40.0, 4.0]],
            [[0.2, 60.0, 1.0], [0.5, 21.0, 9.0], [0.3, 33.0, 3.0]]]
    rng = np.random.default_rng(3)
    sm = Smooth(engine, bins, n_types=3, t_max=140.0, phi=1.0, h=h, paths=1, seed=99)
    g3 = rng.normal(size=(3, sm.n_values))
    E_ref, G_ref, vals, J_ref = smooth_ref.forward_backward(bins, 140.0, 1.0, h, 1, 99, sets, g3, with_jacobian=True)
    pick = np.arange(candidates) % 3
    P = torch.tensor(np.array(sets)[pick], dtype=torch.float64, device="cuda")
    E = sm.forward(P).cpu().numpy()
    G = sm.backward(P, torch.tensor(g3[pick], device="cuda")).cpu().numpy()
    EJ, J = (x.cpu().numpy() for x in sm.jacobian(P))
    sm.sync()
    sm.close()
    assert np.array_equal(vals, sm.values)
    for got, ref, atol in ((E, E_ref, 1e-9), (EJ, E_ref, 1e-9), (G, G_ref, 1e-7), (J, J_ref, 1e-7)):
        assert np.allclose(got, ref[pick], rtol=2e-5, atol=atol * np.abs(ref).max())
        for k in range(3):  # equal candidates, equal results, wherever they stand
            same = got[pick == k]
            assert np.array_equal(same, np.broadcast_to(same[:1], same.shape))


@pytest.mark.parametrize("depth", [1, 33, 63])  # 63: the most generations a bin may have
@pytest.mark.parametrize("lineages", [2, 35])
def test_pairs_against_single_walks(engine, depth, lineages):
    """The same lineages in one bin (walked in pairs) and in one bin each (walked alone; values a
    little apart, so that every lineage's results can be told). A weight has the same factors
    either way, so the sums differ by their roundings, 2^-24 of the sum of magnitudes per term, and
    by what pairs add below the stopping level, e^-40 cells (times a tangent below 1e5). Types that
    divide to the end, that stop on the way, and with factors below the normal floats."""
    import torch
    from procell.smooth import Smooth
    v = 1.5 * 2.0 ** depth
    apart = [v * (1.0 + i / 1024.0) for i in range(lineages)]
    P = torch.tensor([[[0.5, 2.1, 0.2], [0.3, 9.0, 3.0], [0.2, 300.0, 10.0]]], dtype=torch.float64, device="cuda")
    rng = np.random.default_rng(depth)
    gen_grad = rng.normal(size=depth + 1) * 0.5 ** np.arange(depth + 1)
    E, J, G = [], [], []
    for bins in ([(v, lineages)], [(a, 1) for a in apart]):
        sm = Smooth(engine, bins, n_types=3, t_max=140.0, phi=1.0, h=0.5, paths=1, seed=17)
        values = list(sm.values)
        idx = np.array([[values.index(x / 2.0 ** g) for g in range(depth + 1)] for x, _ in bins])
        grad = np.zeros((1, sm.n_values))
        grad[0, idx] = gen_grad
        e, j = (x.cpu().numpy() for x in sm.jacobian(P))
        E.append((sm.forward(P).cpu().numpy()[0, idx], e[0, idx]))
        J.append(j[0, idx])
        G.append(sm.backward(P, torch.tensor(grad, device="cuda")).cpu().numpy()[0])
        sm.sync()
        sm.close()
    eps = (lineages + 2) * 2.0 ** -24
    for pair, single in zip(*E):
        assert np.all(np.abs(pair[0] - single.sum(0)) <= eps * single.sum(0) + 1e-15)
    mags = np.abs(J[1]).sum(0)
    assert np.all(np.abs(J[0][0] - J[1].sum(0)) <= eps * mags + 1e-10)
    terms = np.einsum("g,gkq->kq", np.abs(gen_grad), mags)
    assert np.all(np.abs(G[0] - G[1]) <= (64 * lineages + 2) * 2.0 ** -24 * terms + 1e-10)


@pytest.mark.parametrize("types", [1, 2, 5, 8])
def test_gauss_newton_of_every_width(engine, types):
    import torch
    from procell.smooth import Smooth
    rng = np.random.default_rng(types)
    bins = [(float(v), int(f)) for v, f in zip(np.exp(rng.uniform(0, 7, 41)), rng.integers(1, 9, 41))]
    sm = Smooth(engine, bins, n_types=types, t_max=150.0, phi=1.0, h=0.5, paths=1, seed=5)
    P = np.empty((3, types, 3))
    P[..., 0] = rng.dirichlet(np.ones(types), 3)
    P[..., 1] = rng.uniform(25, 70, (3, types))
    P[..., 2] = 0.2 * P[..., 1]
    P = torch.tensor(P, device="cuda")
    target = torch.tensor(rng.lognormal(2.0, 1.0, sm.n_values), device="cuda")
    loss, jtj, jtr = sm.gauss_newton(P, target)
    E, J = sm.jacobian(P)
    r = torch.log1p(E) - torch.log1p(target)
    Js = (J / (1.0 + E)[:, :, None, None]).reshape(3, sm.n_values, -1)
    # FP64 sums of at most 600 terms in another order
    assert torch.allclose(loss, (r ** 2).sum(1), rtol=1e-12)
    assert torch.allclose(jtj, torch.einsum("cvp,cvq->cpq", Js, Js), rtol=1e-11, atol=1e-12 * float(jtj.abs().max()))
    assert torch.allclose(jtr, torch.einsum("cvp,cv->cp", Js, r), rtol=1e-11, atol=1e-12 * float(jtr.abs().max()))
    sm.close()


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan, 1e300])  # 1e300: infinite once in FP32
def test_gradient_that_is_not_finite_where_no_cell_is(engine, bad):
    """A loss may have an infinite or undefined gradient at an expected count of 0 (sqrt(E), xlogy);
    a generation none of whose lineages has any weight adds nothing to the adjoint, whatever its
    gradient, for even and odd numbers of lineages alike. The values of weight 0 are those of the
    lineages walked alone. Tolerance as in test_pairs_against_single_walks."""
    import torch
    from procell.smooth import Smooth
    depth, cand = 11, 64
    v = 1.5 * 2.0 ** depth
    rng = np.random.default_rng(8)
    mean = np.exp(rng.uniform(np.log(8.0), np.log(70.0), cand))
    P = torch.tensor(np.stack([np.ones(cand), mean, 0.5 * mean], 1)[:, None, :], device="cuda")
    hit = 0
    for lineages in (2, 3, 6):
        apart = [v * (1.0 + i / 1024.0) for i in range(lineages)]
        sm = Smooth(engine, [(a, 1) for a in apart], n_types=1, t_max=140.0, phi=1.0, h=0.5, paths=1, seed=23)
        values = list(sm.values)
        idx = np.array([[values.index(x / 2.0 ** g) for g in range(depth + 1)] for x in apart])
        E, J = (x.cpu().numpy() for x in sm.jacobian(P))
        sm.sync()
        sm.close()
        empty = E[:, idx].sum(1) == 0.0  # [candidate, generation]
        terms = np.abs(J[:, idx]).sum(1)[:, :, 0]  # [candidate, generation, parameter]
        sm = Smooth(engine, [(v, lineages)], n_types=1, t_max=140.0, phi=1.0, h=0.5, paths=1, seed=23)
        values = list(sm.values)
        at = np.array([values.index(v / 2.0 ** g) for g in range(depth + 1)])
        gen_grad = rng.normal(size=depth + 1) * 0.5 ** np.arange(depth + 1)
        got = []
        for there in (0.0, bad):
            grad = np.zeros((cand, sm.n_values))
            grad[:, at] = np.where(empty, there, gen_grad)
            got.append(sm.backward(P, torch.tensor(grad, device="cuda")).cpu().numpy()[:, 0])
        sm.sync()
        sm.close()
        later = empty & (np.cumsum(~empty, 1) > 0) & (np.cumsum(~empty[:, ::-1], 1)[:, ::-1] > 0)
        hit += int(later.any(1).sum())  # a generation of weight 0 between two others
        tol = (64 * lineages + 2) * 2.0 ** -24 * np.einsum("g,cgq->cq", np.abs(gen_grad), terms) + 1e-10
        assert np.all(np.isfinite(got[1]))
        assert np.all(np.abs(got[1] - got[0]) <= tol)
    assert hit > 0


@pytest.mark.parametrize("predraw", [1, 0])
@pytest.mark.parametrize("extra", [23, 24, 25, 63])  # the plan's rows are one more: pairs up to 24 rows
def test_adjoint_of_plans_with_a_deep_bin(engine, predraw, extra):
    """The same bins in a plan by themselves (pairs) and with a brighter bin behind them, whose depth
    decides how the whole plan is walked and whose own gradient is 0: the same lineages, so the same
    adjoint up to rounding. Tolerance as in test_pairs_against_single_walks."""
    import torch
    from procell.smooth import Smooth
    bins = [(900.0, 35), (77.0, 3), (3.0, 4), (150.0, 64)]
    P = torch.tensor([[[0.5, 22.0, 4.0], [0.5, 35.0, 14.0]], [[0.3, 60.0, 3.0], [0.7, 18.0, 9.0]]], device="cuda",
                     dtype=torch.float64)
    rng = np.random.default_rng(extra)
    engine.set_option("smooth_predraw", predraw)
    try:
        sm = Smooth(engine, bins, n_types=2, t_max=140.0, phi=1.0, h=0.5, paths=1, seed=31)
        values, g = list(sm.values), rng.normal(size=(2, sm.n_values))
        J = sm.jacobian(P)[1].cpu().numpy()
        alone = sm.backward(P, torch.tensor(g, device="cuda")).cpu().numpy()
        sm.sync()
        sm.close()
        sm = Smooth(engine, bins + [(1.5 * 2.0 ** extra, 2)], n_types=2, t_max=140.0, phi=1.0, h=0.5, paths=1, seed=31)
        grad = np.zeros((2, sm.n_values))
        grad[:, [list(sm.values).index(v) for v in values]] = g
        both = sm.backward(P, torch.tensor(grad, device="cuda")).cpu().numpy()
        sm.sync()
        sm.close()
    finally:
        engine.set_option("smooth_predraw", 1)
    terms = np.einsum("cv,cvkq->ckq", np.abs(g), np.abs(J))
    assert np.all(np.abs(both - alone) <= (64 * 64 + 2) * 2.0 ** -24 * terms + 1e-10)


def test_a_neighbour_whose_gradient_is_not_finite(engine):
    """It changes no other candidate's adjoint, not in the last bit."""
    import torch
    from procell.smooth import Smooth
    rng = np.random.default_rng(12)
    bins = [(float(v), int(f)) for v, f in zip(np.exp(rng.uniform(0, 8, 23)), rng.integers(1, 40, 23))]
    sm = Smooth(engine, bins, n_types=2, t_max=140.0, phi=1.0, h=0.5, paths=1, seed=3)
    P = np.empty((40, 2, 3))
    P[..., 0] = rng.dirichlet(np.ones(2), 40)
    P[..., 1] = rng.uniform(15, 60, (40, 2))
    P[..., 2] = 0.3 * P[..., 1]
    P = torch.tensor(P, device="cuda")
    g = torch.tensor(rng.normal(size=(40, sm.n_values)), device="cuda")
    want = sm.backward(P, g).cpu().numpy()
    for odd in (0, 17, 39):
        h = g.clone()
        h[odd, ::5] = float("inf")
        got = sm.backward(P, h).cpu().numpy()
        others = np.arange(40) != odd
        assert np.array_equal(got[others], want[others]), odd
        assert not np.all(np.isfinite(got[odd]))
    sm.sync()
    sm.close()
