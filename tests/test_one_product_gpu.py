"""Calls that build a tree for one product: it may end at the level where the product does, and b may be sorted with the points."""
import pytest
import torch

from cases import rel_l2

pytestmark = pytest.mark.gpu
N = (1 << 21) + 4099      # from 2^21 points on


# positive weights; the two products differ in the level their sources are interpolated at and in the order of sums: some tens of roundings
TOL = 2e-6


@pytest.mark.parametrize("d,p,n,m,R,ls,dist,leaf", [(3, 6, N, 0, 1, 1.0, "uniform", 1000.0),       # ends early, two passes of short digits
                                                    (3, 4, N, 0, 1, 0.3, "uniform", 1000.0),       # does not, two passes of long ones
                                                    (3, 5, N, 0, 1, 0.5, "mixture", 1000.0),       # sorted again to the full depth
                                                    (2, 6, N, N + 1, 1, 0.8, "uniform", 300.0),    # two sets, b with the sources
                                                    (3, 5, N, N - 3, 1, 0.4, "uniform", 1000.0), (3, 6, N, 0, 2, 1.0, "uniform", 1000.0),
                                                    (1, 6, N, 0, 1, 0.2, "uniform", 20000.0), (5, 3, N, 0, 1, 3.0, "uniform", 3000.0),
                                                    (4, 4, N, 0, 3, 12.0, "uniform", 1000.0), (3, 8, N, 0, 1, 1e4, "uniform", 1000.0),
                                                    (3, 6, (1 << 21) - 1, 0, 1, 1.0, "uniform", 1000.0), (3, 6, N, 5000, 1, 1.0, "uniform", 1000.0)])
def test_one_product_equals_the_plans(d, p, n, m, R, ls, dist, leaf, cuda):
    from f3m_b200 import engine
    g = torch.Generator(device=cuda).manual_seed(n % 1000 + d)
    X = torch.rand(n, d, device=cuda, generator=g)
    if dist == "mixture":
        X = X * 0.05 + torch.rand(10, d, device=cuda, generator=g)[torch.randint(0, 10, (n,), device=cuda, generator=g)]
    Y = torch.rand(m, d, device=cuda, generator=g) * 0.9 + 0.03 if m else None
    b = torch.rand(m or n, R, device=cuda, generator=g) + 0.5
    prm = engine.make_params(ls, leaf, p ** d, False, 0.15, p ** d)
    out = engine.kmvm(X, Y, b, prm)
    plan = engine.Plan(X, Y, prm)
    assert rel_l2(out.cpu(), plan.apply(b).cpu()) <= TOL
    host = engine.kmvm_host(X.cpu(), None if Y is None else Y.cpu(), b.cpu(), prm)
    assert rel_l2(host, out.cpu()) <= TOL
    if d == 3 and R == 1:
        assert torch.equal(engine.kmvm(X, Y, b, prm), out)
    else:
        assert rel_l2(engine.kmvm(X, Y, b, prm).cpu(), out.cpu()) <= 2e-7


def test_rows_of_b_follow_their_points(cuda):
    """Weights that name their rows, points on a line: every row of the result is its own weight and its neighbours'."""
    from f3m_b200 import engine
    n = N
    g = torch.Generator(device=cuda).manual_seed(1)
    X = torch.rand(n, 3, device=cuda, generator=g)
    b = torch.zeros(n, 1, device=cuda)
    rows = torch.randperm(n, device=cuda, generator=g)[:64]
    b[rows, 0] = torch.arange(1, 65, device=cuda, dtype=torch.float32)
    out = engine.kmvm(X, None, b, engine.make_params(1.0, 1000.0, 216, False, 0.15, 216))
    exact = engine.rbf_dense(X[rows].double(), X[rows].double(), b[rows].double(), 1.0)
    assert rel_l2(out[rows].cpu(), exact.cpu()) <= 2e-5     # six nodes per axis at l = 1: 2.5e-6 of the dense product and more for few weights


@pytest.mark.parametrize("n", [(1 << 21) - 1, (1 << 21) + 4099])   # both sides of the size from which wide digits take fewer blocks
@pytest.mark.parametrize("d,leaf,scale", [(3, 3e4, 1.0), (3, 4e3, 1.0), (3, 500.0, 1.0), (3, 60.0, 1.0), (2, 200.0, 1.0), (5, 3000.0, 1.0),
                                          (3, 1000.0, 0.02)])
def test_sorted_order_of_all_digit_widths(n, d, leaf, scale, cuda):
    """The sorted points fill their boxes, box by box: 9 to 30 key bits in one to three passes of six to ten."""
    from f3m_b200 import _lib, engine
    g = torch.Generator(device=cuda).manual_seed(n % 1000 + d)
    X = torch.rand(n, d, device=cuda, generator=g)
    if scale < 1.0:   # clustered: sorted again to the full key depth
        X = X * scale + torch.rand(10, d, device=cuda, generator=g)[torch.randint(0, 10, (n,), device=cuda, generator=g)]
    plan = engine.Plan(X, None, engine.make_params(1.0, leaf, 8, False, 0.15, 8))
    L = plan.stats()["levels"]
    perm = torch.from_numpy(plan.array(L, 0, _lib.ARR_SORTED_INDEX)).long().to(cuda)
    assert torch.equal(torch.sort(perm).values, torch.arange(n, device=cuda))
    off = torch.from_numpy(plan.array(L, 0, _lib.ARR_BOX_OFFSETS)).long().to(cuda)
    box = torch.repeat_interleave(torch.arange(off.numel() - 1, device=cuda), off.diff())
    ctr = torch.from_numpy(plan.array(L, 0, _lib.ARR_BOX_CENTERS)).to(cuda)
    lo, hi = X.min(0).values, X.max(0).values
    half = (hi - lo).max() * 1.01 / 2 ** (L + 1)
    # float32 centres and cells: a few roundings of coordinates of size one
    assert ((X[perm] - ctr[box]).abs() <= half + 4e-6).all()


@pytest.mark.parametrize("n,ls", [(3_000_000, 10.0), (10_000_000, 10.0), (10_000_000, 3.0)])
def test_full_boxes_lose_no_precision(n, ls, cuda):
    """A tree that ends at boxes of 2e4 to 1.2e6 points: its product is no further from float64 than that of a kept plan, whose sources are
    interpolated in smaller ones.  A wide kernel makes one error of all rows, so it is the mean over many right-hand sides that tells:
    two means over 300 differ by 6 per cent in one standard deviation."""
    from f3m_b200 import engine
    g = torch.Generator(device=cuda).manual_seed(99)
    X = torch.rand(n, 3, device=cuda, generator=g) * 12 ** 0.5
    prm = engine.make_params(ls, 1000.0, 216, False, 0.15, 216)
    plan = engine.Plan(X, None, prm)
    rows = torch.randperm(n, device=cuda, generator=g)[:8]
    K = torch.exp(-((X[rows].double()[:, None, :] - X.double()[None]) ** 2).sum(-1) / (2 * ls * ls))
    one = kept = 0.0
    for _ in range(300):
        b = torch.randn(n, 1, device=cuda, generator=g)
        exact = K @ b.double()
        one += float((engine.kmvm(X, None, b, prm)[rows] - exact).square().sum())
        kept += float((plan.apply(b)[rows] - exact).square().sum())
    assert 0 < plan.last_work()["cut_level"] < plan.stats()["levels"]
    assert one ** 0.5 <= 1.15 * kept ** 0.5, ((one / 2400 / n) ** 0.5, (kept / 2400 / n) ** 0.5)
