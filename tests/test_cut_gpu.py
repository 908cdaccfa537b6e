"""Products that end at the level whose interpolation is exact for every pair, against the same lists without the cut."""
import pytest
import torch

from cases import rel_l2

pytestmark = pytest.mark.gpu

# Positive weights, so that no sum cancels: the cut's bound 1.2e-7, the near sums' own 2.4e-7, and the rounding of the Lagrange
# values and translations, some tens of roundings of 6e-8 on either side.
TOL = 2e-6


def _points(n, d, dist, g):
    if dist == "uniform":
        return torch.rand(n, d, generator=g)
    if dist == "normal":
        return torch.randn(n, d, generator=g)
    centre = torch.rand(10, d, generator=g) * 10 - 5     # a mixture: empty boxes, neighbours on several levels
    return torch.randn(n, d, generator=g) * 0.5 + centre[torch.randint(0, 10, (n,), generator=g)]


@pytest.mark.parametrize("d,p,n,m,R,ls,dist", [(3, 6, 600011, 0, 1, 1.0, "uniform"), (3, 8, 400000, 0, 1, 0.7, "uniform"), (3, 5, 500000, 0, 1, 40.0, "normal"),
                                               (3, 6, 700001, 0, 1, 30.0, "mixture"), (2, 6, 900000, 0, 1, 0.3, "uniform"), (3, 6, 500000, 300007, 1, 1.5, "uniform"),
                                               (3, 6, 300000, 0, 1, 1000.0, "uniform"), (4, 4, 300000, 0, 3, 8.0, "uniform")])
def test_cut_equals_the_full_lists(d, p, n, m, R, ls, dist, cuda):
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(n + d)
    X = _points(n, d, dist, g).to(cuda)
    Y = (_points(m, d, dist, g) * 0.9 + 0.037).to(cuda) if m else None
    b = (torch.rand(m or n, R, generator=g) + 0.5).to(cuda)
    plan = engine.Plan(X, Y, engine.make_params(ls, 300.0, p ** d, False, 0.15, p ** d))
    out = plan.apply(b)
    cut = plan.timings()["direct_launches"] == 0
    half = n // 2 + 7
    parts = plan.apply(b, row_range=(0, half)) + plan.apply(b, row_range=(half, n))   # slices keep all levels and lists
    assert plan.timings()["direct_launches"] > 0
    print(f"cut {cut}: rel-L2 against the full lists {rel_l2(out.cpu(), parts.cpu()):.2e}")
    assert cut
    assert rel_l2(out.cpu(), parts.cpu()) <= TOL
    again = plan.apply(b)                                       # the plan's list of the cut level, used again
    assert torch.equal(again, out) if d == 3 else rel_l2(again.cpu(), out.cpu()) <= 2e-7
    rows = torch.arange(0, n, n // 400, device=cuda)
    exact = engine.rbf_dense(X[rows].double(), (X if Y is None else Y).double(), b.double(), ls)
    assert rel_l2(out[rows].cpu(), exact.cpu()) <= max(TOL, 1.2 * rel_l2(parts[rows].cpu(), exact.cpu()))


def test_no_cut_where_the_interpolation_is_not_exact(cuda):
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(5)
    X = torch.rand(400000, 3, generator=g).to(cuda)
    b = torch.randn(400000, 1, generator=g).to(cuda)
    for ls, p in ((0.1, 6), (1.0, 3)):
        plan = engine.Plan(X, None, engine.make_params(ls, 300.0, p ** 3, False, 0.15, p ** 3))
        plan.apply(b)
        assert plan.timings()["direct_launches"] > 0


def test_result_larger_than_the_cache(cuda):
    """More rows than two windows of the result's permutation, the last window and the last rows ragged."""
    from f3m_b200 import engine
    n = 2 * (16 << 20) + 4099
    g = torch.Generator(device=cuda).manual_seed(9)
    X = torch.rand(n, 3, device=cuda, generator=g)
    b = torch.rand(n, 1, device=cuda, generator=g) + 0.5
    out = engine.kmvm(X, None, b, engine.make_params(1.0, 1000.0, 216, False, 0.15, 216))
    rows = torch.tensor([0, 1, 2, (16 << 20) - 1, 16 << 20, (32 << 20) - 1, 32 << 20, n - 4, n - 3, n - 2, n - 1], device=cuda)
    exact = engine.rbf_dense(X[rows].double(), X.double(), b.double(), 1.0)
    assert ((out[rows].double() - exact).abs() / exact).max().item() <= 2e-6
    assert torch.isfinite(out).all() and (out > 0).all()


def test_more_source_parts_than_a_grid_dimension(cuda):
    """Half of 1.4e8 sources in one octant of a tree that its few targets keep to one level: 68 000 parts of a box."""
    from f3m_b200 import engine
    g = torch.Generator(device=cuda).manual_seed(12)
    m = 140_000_000
    Y = torch.rand(m, 3, device=cuda, generator=g)
    Y[: m // 2] *= 0.5
    X = torch.rand(2000, 3, device=cuda, generator=g)
    b = torch.rand(m, 1, device=cuda, generator=g) + 0.5
    plan = engine.Plan(X, Y, engine.make_params(1.0, 1000.0, 512, False, 0.15, 512))   # too narrow for moments, exact on eight nodes
    out = plan.apply(b)
    assert plan.stats()["levels"] == 1 and plan.timings()["direct_launches"] == 0
    exact = engine.rbf_dense(X[:64].double(), Y.double(), b.double(), 1.0)
    assert rel_l2(out[:64].cpu(), exact.cpu()) <= TOL


# boxes of many parts: the sources of a cut level (one set, a mixture, two sets), of the last level, and of box moments
@pytest.mark.parametrize("d,p,n,m,ls,leaf,dist", [(3, 6, 600011, 0, 1.0, 300.0, "uniform"), (3, 6, 700001, 0, 30.0, 300.0, "mixture"),
                                                  (3, 4, 20000, 2000003, 1.0, 64.0, "uniform"), (4, 6, 100000, 0, 0.5, 8000.0, "uniform"),
                                                  (3, 3, 3000, 300007, 2.0, 1000.0, "uniform")])
def test_a_kept_plan_repeats_bit_for_bit(d, p, n, m, ls, leaf, dist, cuda):
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(n + d)
    X = _points(n, d, dist, g).to(cuda)
    Y = _points(m, d, dist, g).to(cuda) if m else None
    b = torch.randn(m or n, 1, generator=g).to(cuda)
    plan = engine.Plan(X, Y, engine.make_params(ls, leaf, p ** d, False, 0.15, p ** d))
    out = plan.apply(b)
    for _ in range(5):
        assert torch.equal(plan.apply(b), out)
