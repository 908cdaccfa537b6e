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
