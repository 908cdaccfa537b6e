"""P2M and L2P of one column in three dimensions at the edges of their chunks: two point sets so far apart that every pair of boxes of
level 1 is far, box by box with a chosen number of points, against the same algorithm in float64."""
import pytest
import torch

from cases import rel_l2

pytestmark = pytest.mark.gpu

# Interpolation weighs its terms with either sign: the Lebesgue constant of eight nodes is 2.3, so 12 over three axes on the sources'
# and as much on the targets' side.  The sums of a few roundings (6e-8 each) that the moments and values carry are random and
# mostly cancel: 12 * 4 of them.
TOL = 12 * 4 * 6e-8
TAILS = [33, 59, 60, 61, 64, 65, 121, 241]   # a warp takes 56 to 64 points at a time, a CTA four times that


def _octants(counts, side, shift, g):
    parts = []
    for o, n in enumerate(counts):
        lo = torch.tensor([(o >> k) & 1 for k in range(3)]) * 0.5 * side
        parts.append(torch.rand(n, 3, generator=g) * 0.46 * side + lo + 0.02 * side)
    X = torch.cat(parts)
    X[0], X[-1] = 0.0, side           # the cube's corners: both sets get the same edge
    return (X[torch.randperm(X.shape[0], generator=g)] + shift).contiguous()


@pytest.mark.parametrize("p", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("tails", ["targets", "sources", "blocks"])
def test_chunks_of_points(p, tails, cuda):
    from f3m_b200 import engine
    from oracle.f3m_oracle import f3m_kmvm
    g = torch.Generator().manual_seed(10 * p)
    full = [2 * p ** 3 + 500 + 3 * o for o in range(8)]
    long = [2047, 2048, 2049, 1919, 1920, 1921, 4097, 8193]   # sums are taken out of the registers every 1920 to 2048 points
    nx, ny = {"targets": (TAILS, full), "sources": (full, TAILS), "blocks": (full, long)}[tails]
    X, Y = _octants(nx, 1.0, 0.0, g), _octants(ny, 1.0, 3.0, g)
    b = torch.rand(Y.shape[0], 1, generator=g) + 0.5
    prm = dict(ls=2.0, min_points=30.0, nr_of_interpolation=p ** 3, var_compression=False, eff_var_limit=0.15, small_field_points=8)
    plan = engine.Plan(X.to(cuda), Y.to(cuda), engine.make_params(2.0, 30.0, p ** 3, False, 0.15, 8))
    assert plan.stats()["levels"] == 1 and plan.level(1)["n_far"] == 64
    out = plan.apply(b.to(cuda)).cpu()
    ref = f3m_kmvm(X, Y, b, dtype=torch.float64, **prm)
    assert rel_l2(out, ref) <= TOL
    again = plan.apply(b.to(cuda)).cpu()
    assert torch.equal(out, again)


# Positive weights under a kernel that is wide against the boxes: what is left are the roundings of the Lagrange rows (six per pair of
# points, one per side and axis), of moments and of expansions.  Mean over ten right-hand sides.  Rows of plain products of differences, whose sum is off one
# by some 1e-7: 2.2, 2.0, 2.2, 1.5e-7; normalised by division 1.3, 1.4, 1.7, 1.2e-7; rows that sum to one 1.0, 1.0, 1.4, 1.0e-7.
@pytest.mark.parametrize("d,n,R,ls,bound", [(3, 1_000_000, 1, 10.0, 1.4e-7), (3, 1_000_000, 1, 4.0, 1.4e-7), (3, 300_000, 3, 4.0, 1.75e-7),
                                            (2, 300_000, 3, 4.0, 1.2e-7)])
def test_rows_sum_to_one(d, n, R, ls, bound, cuda):
    from f3m_b200 import engine
    g = torch.Generator(device=cuda).manual_seed(99)
    X = torch.rand(n, d, device=cuda, generator=g) * 12 ** 0.5
    plan = engine.Plan(X, None, engine.make_params(ls, 1000.0, 6 ** d, False, 0.15, 6 ** d))
    rows = torch.randperm(n, device=cuda, generator=g)[:64]
    K = torch.exp(-((X[rows].double()[:, None, :] - X.double()[None]) ** 2).sum(-1) / (2 * ls * ls))
    err = ref = 0.0
    for _ in range(10):
        b = torch.rand(n, R, device=cuda, generator=g) + 0.5
        exact = K @ b.double()
        err += float((plan.apply(b)[rows] - exact).square().sum())
        ref += float(exact.square().sum())
    assert plan.last_work()["cut_level"] > 0          # every pair through the rows
    assert (err / ref) ** 0.5 <= bound, (err / ref) ** 0.5
