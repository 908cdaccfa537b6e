"""Small calls: tiles of 4 to 32 target rows, lists written on a bound of their length, cubes that stay on the device."""
import pytest
import torch

from cases import rel_l2

pytestmark = pytest.mark.gpu


# tiles of 4 rows (up to 4735 targets), 8, 16, 32 and full ones; boxes of one point to some thousand, sources in halves of 96 pairs
@pytest.mark.parametrize("n,m,leaf", [(9, 40, 4.0), (300, 0, 100.0), (2000, 0, 1000.0), (4735, 0, 1000.0), (4739, 0, 200.0), (9470, 3, 1.0),
                                      (9481, 0, 50.0), (20011, 0, 3000.0), (37887, 2500, 300.0), (37889, 0, 1000.0), (75801, 500, 100.0), (31, 20000, 5.0)])
def test_short_tiles_against_float64(n, m, leaf, cuda):
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(n)
    X = torch.rand(n, 3, generator=g).to(cuda)
    Y = torch.rand(m, 3, generator=g).to(cuda) if m else None
    b = (torch.rand(m or n, 1, generator=g) + 0.5).to(cuda)
    plan = engine.Plan(X, Y, engine.make_params(0.5, leaf, 8, False, 0.15, 10 ** 6))
    out = plan.apply(b)
    assert plan.stats()["levels"] > 0
    if n <= 9470 and plan.stats()["levels"] <= 2:     # boxes too wide for moments, calls too small for nodes
        assert plan.direct_variants()["mufu"] > 0 and plan.last_work()["pairs"] == plan.stats()["direct_pairs"]
    exact = engine.rbf_dense(X.double(), (X if Y is None else Y).double(), b.double(), 0.5)
    st = plan.stats()
    if st["far_box_pairs"] == 0:
        assert st["direct_pairs"] == n * (m or n)
        # positive terms: ex2.approx 2.4e-7 and d + 1 roundings of exponents below 16
        assert rel_l2(out.cpu(), exact.cpu()) <= 1.5e-6
    assert torch.equal(plan.apply(b), out)
    half = n // 2
    parts = plan.apply(b, row_range=(0, half)) + plan.apply(b, row_range=(half, n))
    assert rel_l2(parts.cpu(), out.cpu()) <= 1.5e-6


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("n", [5, 3000, 70000])
def test_cubes_that_are_not_finite(n, bad, cuda):
    """The sort runs before the host sees the cube: an invalid one ends in an error all the same, and the next call is right."""
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(2)
    X = torch.rand(n, 3, generator=g)
    Y = X[: n // 2 + 1].clone()
    b = torch.ones(n, 1).to(cuda)
    prm = engine.make_params(0.7, 3.0, 27, False, 0.15, 27)
    good = engine.kmvm(X.to(cuda), None, b, prm)
    for where in (0, n // 2, n - 1):
        Z = X.clone()
        Z[where, 1] = bad
        with pytest.raises(RuntimeError, match="non-finite"):
            engine.kmvm(Z.to(cuda), None, b, prm)
        with pytest.raises(RuntimeError, match="non-finite"):
            engine.kmvm(Y.to(cuda), Z.to(cuda), b, prm)
    with pytest.raises(RuntimeError, match="degenerate"):
        engine.kmvm(torch.full((n, 3), 0.5, device=cuda), None, b, prm)
    again = engine.kmvm(X.to(cuda), None, b, prm)
    assert torch.equal(good, again)


@pytest.mark.parametrize("shift", [0.0, 3e4, 1e6, 1.6e7])
@pytest.mark.parametrize("d", [1, 2, 3])
def test_lists_hold_every_pair_whatever_the_centres(d, shift, cuda):
    """Far from the origin the centres of small boxes are rounded and more boxes count as near than a lattice allows."""
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(d)
    n = 20000
    X = ((torch.rand(n, d, generator=g) + shift).unique(dim=0)).to(cuda)
    if X.shape[0] < 30:
        X = torch.cat([X, X + 1.0])
    n = X.shape[0]
    plan = engine.Plan(X, None, engine.make_params(1.0, max(4.0, n / 200), 2, False, 0.15, 2))
    st = plan.stats()
    covered = 0
    for level in range(1, st["levels"] + 1):
        import numpy as np
        from f3m_b200 import _lib
        counts = np.diff(plan.array(level, 0, _lib.ARR_BOX_OFFSETS)).astype(np.int64)
        for cls in ("far", "small") + (("keep",) if level == st["levels"] else ()):
            p = plan.pairs(level, cls)
            covered += int((counts[p[:, 0]] * counts[p[:, 1]]).sum())
    assert st["levels"] == 0 or covered == n * n
