"""The exact dense products at the edges of their tiles, slices and column blocks."""
import pytest
import torch

from cases import rel_l2

pytestmark = pytest.mark.gpu


# tiles of 256 targets and 256 sources, slices of an even number of sources, column blocks 1, 2, 3, 4, 8 and 8 + 1
@pytest.mark.parametrize("n,m,d,R", [(1, 1, 3, 1), (1, 40001, 2, 3), (255, 257, 1, 2), (256, 512, 3, 4), (257, 255, 4, 8), (700, 31, 5, 5),
                                     (40001, 33, 3, 1), (3000, 64, 2, 9), (5003, 20001, 3, 3), (129, 1000, 5, 6)])
def test_dense_products(n, m, d, R, cuda):
    from f3m_b200 import engine
    g = torch.Generator().manual_seed(n + m + R)
    X, Y, b = torch.rand(n, d, generator=g).to(cuda), torch.rand(m, d, generator=g).to(cuda), (torch.rand(m, R, generator=g) + 0.5).to(cuda)
    r2 = torch.zeros(n, m, dtype=torch.float64, device=cuda)
    for k in range(d):
        r2 += (X[:, None, k].double() - Y[None, :, k].double()) ** 2
    K = torch.exp(-r2 / (2 * 0.6 ** 2))
    # positive terms: exponential 2.4e-7, its argument a few roundings of at most 7, sums of 256 terms
    out = engine.rbf_dense(X, Y, b, 0.6)
    assert rel_l2(out.cpu(), (K @ b.double()).cpu()) <= 2e-6
    grad = engine.rbf_dense(X, Y, b, 0.6, grad=True)
    assert rel_l2(grad.cpu(), ((K * r2) @ b.double() / 0.6 ** 3).cpu()) <= 2e-6
    assert torch.equal(out, engine.rbf_dense(X, Y, b, 0.6))   # slices are added in a fixed order


def test_dense_extreme_values(cuda):
    """A pair far apart underflows to zero, an odd source count adds a partner of weight zero, and a point at infinity (distance
    infinite to every source) keeps its row at zero without touching the others."""
    from f3m_b200 import engine
    X = torch.tensor([[0.0, 0.0], [1e4, 0.0], [float("inf"), 0.0]], device=cuda)
    Y = torch.tensor([[0.0, 0.0], [0.5, 0.0], [1.0, 0.0]], device=cuda)
    out = engine.rbf_dense(X, Y, torch.ones(3, 1, device=cuda), 1.0).cpu()
    assert abs(float(out[0, 0]) - 2.489027668) <= 1e-5 and float(out[1, 0]) == 0.0 and float(out[2, 0]) == 0.0


@pytest.mark.parametrize("n,R,most", [(300_000, 8, 0), (100_000, 8, 3)])
def test_dense_scratch_pays(n, R, most, cuda):
    """Partial sums are kept only where slices shorten the call: enough targets fill the GPU without them."""
    from f3m_b200 import engine
    X = torch.rand(n, 3, device=cuda)
    b = torch.rand(n, R, device=cuda)
    torch.cuda.synchronize()
    engine.release_cached_memory()
    before = torch.cuda.mem_get_info()[0]
    out = engine.rbf_dense(X, X, b, 0.6)
    torch.cuda.synchronize()
    held = before - torch.cuda.mem_get_info()[0] - out.numel() * 4
    assert held <= most * n * R * 4 + (8 << 20), held


def test_dense_gradient_of_an_odd_count_far_from_the_origin(cuda):
    """The partner of the last source weighs nothing, wherever the points lie."""
    from f3m_b200 import engine
    X = torch.full((3, 2), 1e20, device=cuda)
    b = torch.ones(3, 1, device=cuda)
    assert torch.equal(engine.rbf_dense(X, X, b, 1.0, grad=True), torch.zeros(3, 1, device=cuda))
    assert torch.equal(engine.rbf_dense(X, X, b, 1.0), torch.full((3, 1), 3.0, device=cuda))
