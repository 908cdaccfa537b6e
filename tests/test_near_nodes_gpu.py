"""Direct lists through interpolation nodes (near_nodes.cu) against float64, over the node counts and the shapes of boxes."""
import pytest
import torch

from cases import rel_l2

pytestmark = pytest.mark.gpu

# Relative to the 2-norm of the product, normal weights: a fifth of the interpolation bound 4e-7, and roundings of 6e-8 in moments and
# expansions that Lagrange weights of either sign enlarge (12 for nine nodes in three dimensions) and random signs keep to a few.
TOL = 1.2e-6


def _used(plan):
    return plan.timings()["direct_launches"] > 0 and plan.last_work()["pairs"] == 0 and not any(plan.direct_variants().values())


def _plan(X, ls, leaf, nodes, cuda):
    from f3m_b200 import engine
    return engine.Plan(X.to(cuda), None, engine.make_params(ls, leaf, nodes, False, 0.15, nodes))


# edge over lengthscale -> nodes per axis 7, 8, 9, 10, 11, 12, 13; far fields stay empty: every pair of boxes holds fewer than 2 P points
@pytest.mark.parametrize("edge", [0.5, 0.7, 1.0, 1.3, 1.6, 1.95, 2.3])
@pytest.mark.parametrize("shape", ["long", "short"])
def test_against_float64(edge, shape, cuda):
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(int(100 * edge))
    level = 1 if shape == "long" else 2     # boxes of 4000 points (summed in parts) or of 480
    X = torch.rand(32003 if shape == "long" else 30707, 3, generator=g) + 1.3   # coordinates that are large against the boxes
    n = X.shape[0]
    side = float((X.max(0).values - X.min(0).values).max()) * 1.01
    ls = side / 2 ** level / edge
    b = torch.randn(n, 1, generator=g)
    plan = _plan(X, ls, 2000.0 if shape == "long" else 300.0, 5000 if shape == "long" else 1000, cuda)
    out = plan.apply(b.to(cuda))
    assert plan.stats()["levels"] == level and plan.stats()["far_box_pairs"] == 0
    assert _used(plan)
    Xd = X.to(cuda).double()
    exact = engine.rbf_dense(Xd, Xd, b.to(cuda).double(), ls)
    assert rel_l2(out.cpu(), exact.cpu()) <= TOL
    again = plan.apply(b.to(cuda))          # the ordered rows are kept in the plan
    assert torch.equal(out, again)
    half = n // 2 + 3
    parts = plan.apply(b.to(cuda), row_range=(0, half)) + plan.apply(b.to(cuda), row_range=(half, n))   # slices sum the pairs
    assert rel_l2(out.cpu(), parts.cpu()) <= TOL + rel_l2(parts.cpu(), exact.cpu())


@pytest.mark.parametrize("edge", [0.5, 0.7, 1.0, 1.3, 1.6, 1.95, 2.3])
def test_uneven_boxes(edge, cuda):
    """Boxes of some tens to four thousand points, far pairs beside the direct ones: against the same lists summed pair by pair."""
    g = torch.Generator().manual_seed(int(100 * edge))
    n = 1500011
    X = torch.rand(n, 3, generator=g) ** 1.4 + 1.3
    b = torch.rand(n, 1, generator=g) + 0.5
    plan = _plan(X, 1.01 / 16 / edge, 6000.0, 216, cuda)
    assert plan.stats()["levels"] == 4
    out = plan.apply(b.to(cuda))
    assert plan.timings()["direct_launches"] > 0 and plan.last_work()["pairs"] < plan.stats()["direct_pairs"] // 2
    assert torch.equal(plan.apply(b.to(cuda)), out)
    parts = plan.apply(b.to(cuda), row_range=(0, 700001)) + plan.apply(b.to(cuda), row_range=(700001, n))
    assert plan.last_work()["pairs"] > 0
    assert rel_l2(out.cpu(), parts.cpu()) <= 2 * TOL


def test_weights_that_are_not_finite(cuda):
    """An infinite weight gives what the pairs give: infinity, and NaN rows for a NaN weight."""
    g = torch.Generator().manual_seed(3)
    X = torch.rand(30707, 3, generator=g)
    plan = _plan(X, 0.25, 300.0, 1000, cuda)
    b = torch.rand(30707, 1, generator=g) + 0.5
    plan.apply(b.to(cuda))
    assert _used(plan)
    for value in (float("inf"), float("nan"), 3e38):
        c = b.clone()
        c[777] = value
        out = plan.apply(c.to(cuda))
        half = 15000
        parts = plan.apply(c.to(cuda), row_range=(0, half)) + plan.apply(c.to(cuda), row_range=(half, 30707))
        assert torch.equal(torch.isnan(out), torch.isnan(parts)) and torch.equal(torch.isinf(out), torch.isinf(parts))
        assert not torch.isfinite(out).all() or value == 3e38
    plan.apply(b.to(cuda))
    assert _used(plan)


def test_small_workspace_sums_the_pairs(cuda):
    """A workspace without room for the moments: the product is there all the same."""
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(4)
    X = torch.rand(32003, 3, generator=g).to(cuda)
    b = torch.rand(32003, 1, generator=g).to(cuda)
    prm = engine.make_params(0.22, 2000.0, 5000, False, 0.15, 5000)
    want = engine.kmvm(X, None, b, prm)
    for mb in (64, 8, 6, 5, 4):
        ws = torch.empty(mb << 20, dtype=torch.uint8, device=cuda)
        try:
            out = engine.kmvm_ws(X, None, b, prm, ws)
        except RuntimeError as e:
            assert "workspace" in str(e)
            continue
        assert rel_l2(out.cpu(), want.cpu()) <= TOL


def _mixture(n, g, width=0.06):
    return torch.rand(20, 3, generator=g)[torch.randint(0, 20, (n,), generator=g)] + torch.randn(n, 3, generator=g) * width


@pytest.mark.parametrize("n,p,ls", [(400_000, 6, 0.16), (500_000, 8, 0.25)])
def test_products_that_end_above_the_exact_level(n, p, ls, cuda):
    """The level whose children's interpolation is exact: its near pairs through more nodes, nothing below it is visited."""
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(p)
    X = _mixture(n, g).to(cuda)
    b = (torch.rand(n, 1, generator=g) + 0.5).to(cuda)
    plan = engine.Plan(X, None, engine.make_params(ls, 100.0, p ** 3, False, 0.15, p ** 3))
    out = plan.apply(b)
    cut = plan.last_work()["cut_level"]
    assert 0 < cut < plan.stats()["levels"] and plan.timings()["direct_launches"] > 0
    half = n // 2 + 1
    parts = plan.apply(b, row_range=(0, half)) + plan.apply(b, row_range=(half, n))   # slices visit all levels
    # positive weights: the bound of the far pairs that are replaced (1.2e-7) besides those above
    assert rel_l2(out.cpu(), parts.cpu()) <= 2 * TOL
    assert torch.equal(plan.apply(b), out)
    c = b.clone()
    c[n // 3] = float("inf")
    assert not torch.isfinite(plan.apply(c)).all()
    assert torch.equal(plan.apply(b), out)


def test_one_product_that_ends_above_the_exact_level(cuda):
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(11)
    n = (1 << 21) + 77
    X = _mixture(n, g).to(cuda)
    b = (torch.rand(n, 1, generator=g) + 0.5).to(cuda)
    prm = engine.make_params(0.16, 100.0, 216, False, 0.15, 216)
    plan = engine.Plan(X, None, prm)
    want = plan.apply(b)
    assert 0 < plan.last_work()["cut_level"] < plan.stats()["levels"] and plan.timings()["direct_launches"] > 0
    out = engine.kmvm(X, None, b, prm)
    assert rel_l2(out.cpu(), want.cpu()) <= TOL
    assert torch.equal(engine.kmvm(X, None, b, prm), out)
    rows = torch.arange(0, n, n // 300, device=cuda)
    exact = engine.rbf_dense(X[rows].double(), X.double(), b.double(), 0.16)
    assert rel_l2(out[rows].cpu(), exact.cpu()) <= 1.2 * rel_l2(want[rows].cpu(), exact.cpu()) + TOL
    # a weight of infinity: its neighbourhood is summed pair by pair
    b[5] = float("inf")
    out = engine.kmvm(X, None, b, prm)
    assert not torch.isfinite(out[5]).any()


@pytest.mark.parametrize("edge", [0.55, 1.09, 1.6])
def test_few_weights_are_summed_pair_by_pair(edge, cuda):
    """A column of K: entries far below 1 keep their digits, which interpolation against the kernel's largest value does not give."""
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(int(100 * edge))
    X = torch.rand(30707, 3, generator=g) + 1.3
    n = X.shape[0]
    ls = float(torch.tensor(float((X.max(0).values - X.min(0).values).max()) * 1.01 / 4 / edge, dtype=torch.float32))
    plan = _plan(X, ls, 300.0, 1000, cuda)
    Xd = X.to(cuda).double()
    for count in (1, n // 100):
        b = torch.zeros(n, 1, device=cuda)
        b[torch.randperm(n, generator=g)[:count].to(cuda)] = 0.75
        out = plan.apply(b)
        assert plan.last_work()["pairs"] == plan.stats()["direct_pairs"]
        exact = engine.rbf_dense(Xd, Xd, b.double(), ls)
        seen = exact > 1e-20
        # exponents are differences of numbers up to 64 (in powers of two), good to some three roundings of them
        assert float(((out.double() - exact).abs() / exact)[seen].max()) <= 2e-5
    b = torch.rand(n, 1, device=cuda) + 0.5
    plan.apply(b)
    assert _used(plan)


@pytest.mark.parametrize("edge", [0.55, 1.09])
def test_targets_beside_dense_boxes(edge, cuda):
    """Rows of single targets around two boxes of 2e4 points each: their error stays below the bound times the sum of the weights."""
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(int(100 * edge))
    dense = torch.rand(40000, 3, generator=g) * 0.25
    dense[20000:, 0] += 0.25
    X = torch.cat([dense, torch.rand(600, 3, generator=g), torch.zeros(1, 3), torch.ones(1, 3)]).to(cuda)
    b = (torch.rand(X.shape[0], 1, generator=g) + 0.5).to(cuda)
    b[40000:] *= 1e-3
    ls = float(torch.tensor(1.01 / 4 / edge, dtype=torch.float32))
    plan = engine.Plan(X, None, engine.make_params(ls, 21000.0, 45000, False, 0.15, 45000))
    out = plan.apply(b)
    assert _used(plan)
    exact = engine.rbf_dense(X[40000:].double(), X.double(), b.double(), ls)
    assert float((out[40000:].double() - exact).abs().max()) <= TOL * float(b.sum())


# A last level whose two lists both qualify for box moments (boxes of a tenth of a lengthscale) while one of them, or both, or none goes
# through nodes: every pair is summed once.  Against slices of the rows, which take no nodes.
@pytest.mark.parametrize("n,nodes,small,ls,leaf,by_nodes", [(3_000_000, 27, 27, 1.7, 1000.0, "keep"), (3_000_000, 27, 27, 3.0, 1000.0, "keep"),
                                                            (8_000_000, 27, 27, 0.9, 1000.0, "keep"), (2_000_000, 27, 300, 1.5, 1000.0, "both"),
                                                            (3_000_000, 8, 200, 1.7, 1000.0, None),
                                                            (3_000_000, 8, 8, 1.7, 1000.0, None), (1_000_000, 27, 27, 2.0, 1000.0, None)])
def test_one_list_through_nodes_and_one_through_moments(n, nodes, small, ls, leaf, by_nodes, cuda):
    from f3m_b200 import engine
    g = torch.Generator(device=cuda).manual_seed(3)
    X = torch.randn(n, 3, device=cuda, generator=g)
    b = torch.rand(n, 1, device=cuda, generator=g) + 0.5
    plan = engine.Plan(X, None, engine.make_params(ls, leaf, nodes, False, 0.15, small))
    last = plan.level(plan.stats()["levels"])
    assert last["n_small"] > 0 and last["n_keep"] > 0
    out = plan.apply(b)
    v, launches = plan.direct_variants(), plan.timings()["direct_launches"]
    assert plan.last_work()["cut_level"] == 0
    half = n // 2 + 1
    parts = plan.apply(b, row_range=(0, half)) + plan.apply(b, row_range=(half, n))
    # positive weights; both forms of a list are good to some 3e-7 of its sum
    assert rel_l2(out.cpu(), parts.cpu()) <= 1e-6
    assert rel_l2(engine.kmvm(X, None, b, engine.make_params(ls, leaf, nodes, False, 0.15, small)).cpu(), parts.cpu()) <= 1e-6
    assert plan.direct_variants()["moments"] > 0
    if by_nodes:
        assert v["moments"] > 0 and launches > v["mufu"] + v["direct"] + v["moments"]   # a launch without a count is the nodes'
