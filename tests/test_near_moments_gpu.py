"""Near sums through box moments against the sums over the pairs."""
import pytest
import torch

from cases import rel_l2

pytestmark = pytest.mark.gpu


def _both(X, Y, b, ls, leaf, nodes, cuda):
    """The default product, and the one whose lists are all summed pair by pair (the tensor-core flag keeps moments out)."""
    from f3m_b200 import _lib, engine
    out, forms = [], []
    for flags in (0, _lib.FLAG_NEAR_TENSOR_CORES):
        plan = engine.Plan(X.to(cuda), None if Y is None else Y.to(cuda), engine.make_params(ls, leaf, nodes, False, 0.15, nodes, flags=flags))
        out.append(plan.apply(b.to(cuda)).cpu())
        forms.append(plan.direct_variants())
    assert forms[1]["moments"] == 0
    return out, forms[0], plan


def _weights(n, R, g):
    # positive, so that no sum cancels: truncation 1.2e-7, ex2.approx 2.4e-7 on either side, and FP32 sums of blocks of at most a few
    # hundred terms, each below 1e-6 of the (positive) result
    return torch.rand(n, R, generator=g) + 0.5


TOL = 2e-6


# degrees 2, 3, 4, 5, 6 as the boxes widen; one column, a partial block of four, and a block of four and one column
@pytest.mark.parametrize("d,ls,R", [(1, 0.4, 1), (1, 0.05, 5), (2, 3.0, 1), (2, 0.5, 2), (2, 0.2, 3), (3, 4.0, 1), (3, 1.6, 5), (3, 0.9, 1),
                                    (3, 0.7, 4), (3, 0.5, 1), (3, 0.42, 2), (4, 4.0, 1), (4, 2.5, 3), (5, 6.0, 1), (5, 4.0, 2)])
def test_moments_equal_pair_sums(d, ls, R, cuda):
    g = torch.Generator().manual_seed(10 * d + R)
    n = 30011
    X = torch.rand(n, d, generator=g)
    (a, b), forms, _ = _both(X, None, _weights(n, R, g), ls, 300.0, 3 ** d if d > 3 else 4 ** d, cuda)
    assert forms["moments"] > 0, forms
    assert rel_l2(a, b) <= TOL


def test_moments_at_the_corners_of_the_boxes(cuda):
    """Every point within a hair of a corner of its finest box: the exponents reach the bound the degree is chosen by."""
    g = torch.Generator().manual_seed(3)
    corner = torch.randint(0, 9, (40000, 3), generator=g).float() / 8.0
    X = (corner + (torch.rand(40000, 3, generator=g) - 0.5) * 1e-3)
    (a, b), forms, _ = _both(X, None, _weights(40000, 1, g), 0.8, 300.0, 64, cuda)
    assert forms["moments"] > 0, forms
    assert rel_l2(a, b) <= TOL


@pytest.mark.parametrize("n,m", [(1, 70000), (31, 40000), (129, 3000), (40000, 1500), (70001, 33), (31, 400_000), (200, 1_000_003)])
def test_moments_of_two_point_sets(n, m, cuda):
    """Source boxes of very different length (a warp, 256 threads, parts of more than 16 384 rows) and few targets."""
    g = torch.Generator().manual_seed(n + m)
    X, Y = torch.rand(n, 3, generator=g), torch.rand(m, 3, generator=g)
    if m >= 400_000:
        Y[: m // 3] *= 0.5     # one octant holds several times the others' sources
    if n == 1:
        X = torch.cat([X, X + 0.2])
    (a, b), forms, plan = _both(X, Y, _weights(m, 1, g), 2.0, 20.0 if min(n, m) > 20 else 1.0, 27, cuda)
    if m >= 400_000:
        assert forms["moments"] > 0 and plan.level(1)["max_count_y"] > 2 * 16384, forms
    assert torch.isfinite(a).all()
    assert rel_l2(a, b) <= TOL


def test_moments_of_a_slice_and_short_boxes(cuda):
    """Rows outside the slice stay untouched; boxes with fewer sources than the polynomial has terms keep the pair form."""
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(8)
    X = torch.rand(30000, 3, generator=g)
    b = _weights(30000, 1, g)
    plan = engine.Plan(X.to(cuda), None, engine.make_params(1.6, 300.0, 64, False, 0.15, 64))
    full = plan.apply(b.to(cuda))
    cuts = (0, 1, 63, 12345, 30000)
    parts = sum(plan.apply(b.to(cuda), row_range=(lo, hi)) for lo, hi in zip(cuts, cuts[1:]))
    assert plan.direct_variants()["moments"] > 0
    assert rel_l2(parts.cpu(), full.cpu()) <= 5e-7
    X = torch.rand(30000, 5, generator=g)    # one or two points per box against 21 terms
    (a, p), forms, plan = _both(X, None, b, 6.0, 20.0, 32, cuda)
    assert forms["moments"] == 0 and forms["poly2"] + forms["poly3"] > 0, forms
    assert rel_l2(a, p) <= TOL


def test_moments_only_where_they_take_less_time(cuda):
    """Lists of a few pairs on upper levels and short boxes with several columns stay with the pairs; long boxes take moments whatever the
    number of columns."""
    from f3m_b200 import engine
    g = torch.Generator(device=cuda).manual_seed(5)
    for d, n, ls, leaf, R, most in ((1, 1000000, 0.3, 200.0, 8, 2), (1, 1000000, 0.3, 200.0, 1, 7), (3, 1000000, 0.3, 200.0, 8, 0), (3, 1000000, 0.3, 200.0, 4, 0)):
        X = torch.randn(n, d, device=cuda, generator=g)
        plan = engine.Plan(X, None, engine.make_params(ls, leaf, 3 ** d, False, 0.15, 3 ** d))
        plan.apply(torch.randn(n, R, device=cuda, generator=g), row_range=(0, n - 1))
        assert plan.direct_variants()["moments"] <= most, (d, R, plan.direct_variants())
    X = torch.rand(300000, 2, device=cuda, generator=g)
    plan = engine.Plan(X, None, engine.make_params(1.0, 200.0, 9, False, 0.15, 9))
    for R in (1, 4, 8):
        plan.apply(torch.randn(300000, R, device=cuda, generator=g), row_range=(0, 299999))
        assert plan.direct_variants()["moments"] > 0 and plan.last_work()["pairs"] == 0


@pytest.mark.parametrize("ls", [0.42, 0.9, 4.0])
@pytest.mark.parametrize("exponent", [-30, 30])
def test_moments_do_not_depend_on_the_unit_of_length(ls, exponent, cuda):
    """Points and lengthscale in another unit (a power of two, so that every rounding is the same)."""
    g = torch.Generator().manual_seed(17)
    X = torch.rand(30011, 3, generator=g)
    b = _weights(30011, 1, g)
    unit = 2.0 ** exponent
    (a, _), forms, _ = _both(X, None, b, ls, 300.0, 64, cuda)
    (c, p), scaled, _ = _both(X * unit, None, b, ls * unit, 300.0, 64, cuda)
    assert forms == scaled and forms["moments"] > 0, (forms, scaled)
    assert rel_l2(c, p) <= TOL and rel_l2(c, a) <= 1e-7


def test_moments_of_an_infinite_weight(cuda):
    """Every pair is summed directly and every term of the kernel is positive: the sums over an infinite weight are infinite, those
    over a NaN are NaN, and the other columns do not notice."""
    g = torch.Generator().manual_seed(18)
    X = torch.rand(3000, 3, generator=g)
    for R in (1, 3):
        b = _weights(3000, R, g)
        ref, forms, plan = _both(X, None, b, 1.6, 1000.0, 27, cuda)
        assert forms["moments"] > 0 and plan.stats()["far_box_pairs"] == 0
        for bad in (float("inf"), float("-inf"), float("nan")):
            c = b.clone()
            c[1234, R - 1] = bad
            (a, p), _, _ = _both(X, None, c, 1.6, 1000.0, 27, cuda)
            want = torch.full((3000,), bad)
            assert torch.equal(torch.nan_to_num(a[:, -1], 7.0), torch.nan_to_num(want, 7.0))
            assert torch.equal(a[:, :-1], ref[0][:, :-1])
