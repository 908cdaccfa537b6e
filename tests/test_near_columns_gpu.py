"""Direct sums with several columns against float64 and against single columns."""
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
    # and no further off than the single-column kernel
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


# short boxes at the last levels of a tree: narrow ones in the expanded form, wide ones (short lengthscale) in the difference form; columns
# that fill a block of eight, parts of one, and a block and a single column; two point sets; slices that cut boxes
@pytest.mark.parametrize("d,n,m,R,ls,leaf", [(3, 60000, 0, 8, 0.1, 20.0), (3, 60000, 0, 5, 0.01, 20.0), (3, 50021, 40009, 9, 0.02, 20.0), (4, 50021, 0, 8, 0.5, 20.0),
                                             (4, 50021, 0, 7, 0.05, 20.0), (4, 40009, 50021, 6, 0.1, 20.0), (5, 60000, 0, 8, 0.5, 20.0), (5, 60000, 0, 2, 0.5, 20.0),
                                             (5, 60000, 0, 3, 0.1, 20.0), (5, 50021, 60000, 8, 0.1, 20.0), (5, 50021, 60000, 4, 0.1, 20.0)])
def test_columns_of_many_short_boxes(d, n, m, R, ls, leaf, cuda):
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(31 + d + R)
    X = torch.rand(n, d, generator=g).to(cuda)
    Y = (torch.rand(m, d, generator=g) * 0.97 + 0.011).to(cuda) if m else None
    b = (torch.rand(m or n, R, generator=g) + 0.5).to(cuda)
    plan = engine.Plan(X, Y, engine.make_params(ls, leaf, 2 ** d, False, 0.15, 2 ** d))
    cuts = (0, 5, 1000, 1017, n)
    parts = sum(plan.apply(b, row_range=(lo, hi)) for lo, hi in zip(cuts, cuts[1:]))
    assert plan.last_work()["column_launches"] > 0
    wide = plan.direct_variants()["direct"] > 0
    assert wide == (ls <= 0.1 and (d, ls) != (3, 0.1)), plan.direct_variants()
    one = torch.cat([sum(plan.apply(b[:, r:r + 1].contiguous(), row_range=(lo, hi)) for lo, hi in ((0, 7), (7, n))) for r in range(R)], 1)
    assert plan.last_work()["column_launches"] == 0
    assert rel_l2(parts.cpu(), one.cpu()) <= 2e-6
    whole = plan.apply(b)
    assert rel_l2(whole.cpu(), one.cpu()) <= 2e-6


# NaN as arithmetic on the GPU makes it (all mantissa bits set) and as the host writes it, and infinities
@pytest.mark.parametrize("bits", [0x7fffffff, 0x7fc00000, 0x7f800000, -0x00800000])
@pytest.mark.parametrize("d,n,ls,leaf,dist", [(4, 20011, 1.0, 60.0, "normal"), (3, 60000, 0.05, 20.0, "uniform")])
def test_columns_keep_non_finite_weights(bits, d, n, ls, leaf, dist, cuda):
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(7 + d)
    X = (torch.randn(n, d, generator=g) if dist == "normal" else torch.rand(n, d, generator=g)).to(cuda)
    b = torch.zeros(n, 8, dtype=torch.int32)
    b[4321, 3] = bits
    b = b.view(torch.float32).to(cuda)
    plan = engine.Plan(X, None, engine.make_params(ls, leaf, 3 ** d, False, 0.15, 3 ** d))
    out = plan.apply(b)
    assert plan.last_work()["column_launches"] > 0
    one = plan.apply(b[:, 3:4].contiguous())[:, 0]
    assert not one.isfinite().all()
    assert torch.equal(out[:, 3].isnan(), one.isnan()) and torch.equal(out[:, 3].isinf(), one.isinf())
    others = out[:, [0, 1, 2, 4, 5, 6, 7]]
    assert torch.equal(others, torch.zeros_like(others))


def _one_level(n, d, g):
    """Points whose boxes at level 1 are all neighbours (in the first three dimensions; four offsets of one box would be far)."""
    X = torch.rand(n, d, generator=g)
    X[:, 3:] *= 0.4
    return X


# every pair in the boxes of one level, so that the sums are exact: two to nine columns, boxes of one to 600 points, the lists that the
# costs send to the stream of sources (expanded form up to some fifty sources per box, difference form)
@pytest.mark.parametrize("d,n,m,R,ls", [(2, 200, 0, 8, 0.6), (2, 63, 30, 3, 0.6), (2, 1537, 900, 8, 0.1), (3, 400, 0, 7, 0.7), (3, 130, 0, 2, 0.7), (3, 5000, 0, 9, 0.05),
                                        (3, 1200, 900, 4, 0.1), (4, 400, 0, 8, 0.9), (4, 200, 0, 5, 0.2), (5, 500, 0, 8, 1.0), (5, 500, 1999, 6, 0.3),
                                        (5, 300, 250, 3, 1.0), (3, 12, 11, 2, 0.5), (3, 1700, 0, 8, 0.3)])
def test_stream_of_sources_against_float64(d, n, m, R, ls, cuda):
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(d * n + R)
    X = _one_level(n, d, g).to(cuda)
    Y = _one_level(m, d, g).to(cuda) if m else None
    b = (torch.rand(m or n, R, generator=g) + 0.5).to(cuda)
    plan = engine.Plan(X, Y, engine.make_params(ls, 5.0, 2 ** d, False, 0.15, 10 ** 6))
    out = plan.apply(b)
    assert plan.last_work()["column_launches"] > 0
    assert plan.stats()["direct_pairs"] == n * (m or n) == plan.last_work()["pairs"]
    exact = engine.rbf_dense(X.double(), (X if Y is None else Y).double(), b.double(), ls)
    one = torch.cat([plan.apply(b[:, r:r + 1].contiguous()) for r in range(R)], 1)
    e_one, e_all = rel_l2(one.cpu(), exact.cpu()), rel_l2(out.cpu(), exact.cpu())
    print(f"columns {e_all:.2e}, one by one {e_one:.2e}")
    assert e_all <= 5e-6 and e_all <= 1.2 * e_one + 2e-7, (e_all, e_one)    # bounds of test_columns_against_float64


@pytest.mark.parametrize("value", [8e37, 2.0 ** -120])
def test_stream_of_sources_at_the_ends_of_the_exponent_range(value, cuda):
    """Neither a huge value nor a tiny one loses digits on its way through the columns (the expanded form holds terms of up to
    2^(d/4) times a value)."""
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(19)
    X = _one_level(400, 5, g).to(cuda)
    b = torch.zeros(400, 8, device=cuda)
    b[77, 5] = value * (1.0 if value > 1 else 1.2345678)
    plan = engine.Plan(X, None, engine.make_params(1.0, 5.0, 32, False, 0.15, 10 ** 6))
    out = plan.apply(b)
    assert plan.last_work()["column_launches"] > 0 and plan.stats()["far_box_pairs"] == 0
    exact = engine.rbf_dense(X.double(), X.double(), b.double(), 1.0)
    assert ((out[:, 5].double() - exact[:, 5]).abs() <= 2e-6 * exact[:, 5]).all()


def test_long_boxes_stay_with_the_tiles(cuda):
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(20)
    for d, R, ls in ((3, 8, 1.0), (3, 3, 1.0), (1, 8, 0.01)):
        X = torch.rand(200_000, d, generator=g).to(cuda)     # enough targets for tiles on every SM
        plan = engine.Plan(X, None, engine.make_params(ls, 5.0, 2 ** d, False, 0.15, 10 ** 6, flags=2))
        plan.apply(torch.rand(200_000, R, device=cuda))
        assert plan.last_work()["column_launches"] == 0 and plan.last_work()["pairs"] == 200_000 ** 2


# lists of more than 1e8 pairs are cut into parts; siblings whose rows are equal are summed as one box (nodes large: all of them) or keep
# their own rows (normal points, few nodes: rows differ); tiles of every number of rows; four columns and eight
@pytest.mark.parametrize("d,n,R,ls,leaf,nodes,dist", [(2, 60011, 8, 0.05, 300.0, 1000, "normal"), (3, 90011, 4, 0.7, 60.0, 64, "normal"),
                                                      (4, 70003, 8, 1.0, 60.0, 81, "normal"), (4, 70003, 3, 0.1, 60.0, 16, "uniform"),
                                                      (5, 90001, 2, 1.0, 200.0, 243, "normal"), (5, 60001, 7, 0.5, 40.0, 32, "normal")])
def test_groups_and_parts_of_long_lists(d, n, R, ls, leaf, nodes, dist, cuda):
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(41 + d + R)
    X = (torch.randn(n, d, generator=g) if dist == "normal" else torch.rand(n, d, generator=g)).to(cuda)
    b = (torch.rand(n, R, generator=g) + 0.5).to(cuda)
    plan = engine.Plan(X, None, engine.make_params(ls, leaf, nodes, False, 0.15, nodes))
    assert plan.stats()["direct_pairs"] > 2e8
    cuts = (0, 5, 1000, 1017, n // 2 + 3, n)
    parts = sum(plan.apply(b, row_range=(lo, hi)) for lo, hi in zip(cuts, cuts[1:]))
    assert plan.last_work()["column_launches"] > 0
    one = torch.cat([sum(plan.apply(b[:, r:r + 1].contiguous(), row_range=(lo, hi)) for lo, hi in ((0, 7), (7, n))) for r in range(R)], 1)
    assert rel_l2(parts.cpu(), one.cpu()) <= 2e-6    # as in test_columns_of_many_short_boxes
    assert rel_l2(plan.apply(b).cpu(), one.cpu()) <= 2e-6


# Lists of more than 1e8 pairs are cut into parts (ten here): the parts' sums are added in one order, however their warps end.  Lengthscales
# of an eighth of a box: far pairs (whose moments are summed in any order) are below 1e-13 of a row's own weight.
@pytest.mark.parametrize("d,R", [(3, 8), (3, 3), (3, 9), (2, 2), (2, 8)])
def test_parts_of_long_lists_repeat_bit_by_bit(d, R, cuda):
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(d + R)
    n = 60007
    ls = 1.01 / (4 if d == 3 else 8) / 8
    X = torch.rand(n, d, generator=g).to(cuda)
    b = (torch.rand(n, R, generator=g) + 0.5).to(cuda)
    plan = engine.Plan(X, None, engine.make_params(ls, 2000.0, 3 ** d, False, 0.15, 3 ** d))
    assert plan.stats()["direct_pairs"] > 200_000_000
    out = plan.apply(b)
    assert plan.last_work()["column_launches"] > 0
    for _ in range(6):
        assert torch.equal(plan.apply(b), out)
    exact = engine.rbf_dense(X.double(), X.double(), b.double(), ls)
    # ex2.approx 2.4e-7, exponents of the difference form to d + 2 roundings of a number whose share x e^-x is below 0.4
    assert rel_l2(out.cpu(), exact.cpu()) <= 2e-6


@pytest.mark.parametrize("d,n,R", [(5, 200003, 8), (4, 300007, 3), (4, 300007, 9), (3, 300007, 2)])
def test_parts_of_long_lists_of_uneven_trees(d, n, R, cuda):
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(d)
    X = torch.randn(n, d, generator=g).to(cuda)
    b = (torch.rand(n, R, generator=g) + 0.5).to(cuda)
    plan = engine.Plan(X, None, engine.make_params(0.3 if d == 3 else 1.0, 200.0 if d == 3 else 1000.0, 3 ** d, False, 0.15, 3 ** d))
    assert plan.stats()["direct_pairs"] > 200_000_000
    out = plan.apply(b)
    assert plan.last_work()["column_launches"] > 0
    one = torch.cat([plan.apply(b[:, r:r + 1].contiguous()) for r in range(R)], 1)
    assert rel_l2(out.cpu(), one.cpu()) <= 2e-6
    cuts = (0, 1017, n // 2 + 1, n)
    parts = sum(plan.apply(b, row_range=(lo, hi)) for lo, hi in zip(cuts, cuts[1:]))
    assert rel_l2(parts.cpu(), out.cpu()) <= 1e-6
