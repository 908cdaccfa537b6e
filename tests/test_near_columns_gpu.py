"""Direct sums with several columns (split TF32 contraction) against float64 and against single columns."""
import pytest
import torch

from cases import rel_l2

pytestmark = pytest.mark.gpu


# every pair summed directly (small_field_points covers all): expanded form for narrow boxes, difference form for wide ones
@pytest.mark.parametrize("d,n,m,R,ls", [(1, 3001, 0, 2, 0.3), (2, 1537, 900, 8, 0.5), (3, 5000, 0, 3, 0.4), (3, 5000, 0, 8, 0.05), (3, 63, 4001, 9, 0.4),
                                        (4, 2000, 17, 8, 0.6), (4, 2000, 0, 5, 0.15), (5, 1999, 0, 8, 0.9), (5, 4000, 2500, 7, 0.25), (3, 12, 11, 2, 0.5)])
def test_columns_against_float64(d, n, m, R, ls, cuda):
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(d * n + R)
    X = torch.rand(n, d, generator=g).to(cuda)
    Y = torch.rand(m, d, generator=g).to(cuda) if m else None
    b = (torch.rand(m or n, R, generator=g) + 0.5).to(cuda)
    plan = engine.Plan(X, Y, engine.make_params(ls, 5.0 if min(n, m or n) < 100 else 100.0, 8 ** d, False, 0.15, 10 ** 6))
    out = plan.apply(b)
    st = plan.stats()
    assert st["far_box_pairs"] == 0 and st["direct_pairs"] == n * (m or n)
    exact = engine.rbf_dense(X.double(), (X if Y is None else Y).double(), b.double(), ls)
    # positive terms; exponent of the expanded form: d + 1 roundings of a number below 2 d (side / ls)^2 in the worst pair
    assert rel_l2(out.cpu(), exact.cpu()) <= 5e-6
    # and no further off than the single-column kernel, which splits nothing
    one = torch.cat([plan.apply(b[:, r:r + 1].contiguous()) for r in range(R)], 1)
    e_one, e_all = rel_l2(one.cpu(), exact.cpu()), rel_l2(out.cpu(), exact.cpu())
    print(f"columns {e_all:.2e}, one by one {e_one:.2e}")
    assert e_all <= 1.2 * e_one + 2e-7, (e_all, e_one)


@pytest.mark.parametrize("d,ls,leaf,dist", [(4, 1.0, 60.0, "normal"), (5, 1.0, 200.0, "normal"), (3, 0.1, 20.0, "uniform"), (5, 0.8, 40.0, "uniform")])
def test_columns_of_trees_with_short_boxes(d, ls, leaf, dist, cuda):
    """Boxes of one to a few dozen points at several levels, slices of the rows included."""
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(7 + d)
    n = 20011
    X = (torch.randn(n, d, generator=g) if dist == "normal" else torch.rand(n, d, generator=g)).to(cuda)
    b = torch.randn(n, 8, generator=g).to(cuda)
    plan = engine.Plan(X, None, engine.make_params(ls, leaf, 3 ** d, False, 0.15, 3 ** d))
    out = plan.apply(b)
    one = torch.cat([plan.apply(b[:, r:r + 1].contiguous()) for r in range(8)], 1)
    assert rel_l2(out.cpu(), one.cpu()) <= 2e-6
    cuts = (0, 5, 1000, 1017, n)
    parts = sum(plan.apply(b, row_range=(lo, hi)) for lo, hi in zip(cuts, cuts[1:]))
    assert rel_l2(parts.cpu(), out.cpu()) <= 1e-6
