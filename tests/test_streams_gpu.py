"""A plan is finished when it is handed out: its products may run on other streams, and what it gives back may be taken by them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# a second set below the leaf size: no level is built, and the build's last kernels (box starts and links of the first set) follow the
# last count that the host reads
@pytest.mark.parametrize("n,m", [(3_000_017, 200), (200, 3_000_017), (3_000_017, 0)])
def test_a_plan_built_on_one_stream_and_applied_on_another(n, m, cuda):
    from f3m_b200 import engine
    g = torch.Generator(device=cuda).manual_seed(5)
    X = torch.rand(n, 3, device=cuda, generator=g)
    Y = torch.rand(m, 3, device=cuda, generator=g) if m else None
    b = torch.rand(m or n, 1, device=cuda, generator=g) + 0.5
    prm = engine.make_params(0.3, 1000.0, 64, False, 0.15, 64)
    want = engine.Plan(X, Y, prm).apply(b)
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(3):
        with torch.cuda.stream(first):
            plan = engine.Plan(X, Y, prm)
            assert not m or first.query()          # no kernel of the build is left on its stream (an event may be)
        assert plan.stats()["levels"] == (0 if m else 4)
        with torch.cuda.stream(second):
            out = plan.apply(b)
        assert torch.equal(out, want)


def test_plans_dropped_at_once(cuda):
    """The blocks and scratch words of a dropped plan go to the next one, on another stream, while the device has work queued."""
    from f3m_b200 import engine
    g = torch.Generator(device=cuda).manual_seed(6)
    X, Y = torch.rand(2_000_003, 3, device=cuda, generator=g), torch.rand(150, 3, device=cuda, generator=g)
    prm = engine.make_params(0.3, 1000.0, 64, False, 0.15, 64)
    small = engine.make_params(0.3, 50.0, 64, False, 0.15, 64)
    Z = X[:5000].clone()
    b = torch.rand(5000, 1, device=cuda, generator=g)
    want = engine.kmvm(Z, None, b, small)
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(4):
        with torch.cuda.stream(first):
            engine.Plan(X, Y, prm)
            assert first.query()
        with torch.cuda.stream(second):
            plan = engine.Plan(Z, None, small)
            assert plan.stats()["levels"] > 0
            assert torch.equal(plan.apply(b), want)


@pytest.mark.parametrize("n,m", [(50_000, 0), (2_000_003, 0), (2_000_003, 100)])
def test_the_time_of_a_build_is_there_when_the_plan_is(n, m, cuda):
    from f3m_b200 import engine
    X = torch.rand(n, 3, device=cuda)
    Y = torch.rand(m, 3, device=cuda) if m else None
    prm = engine.make_params(0.3, 1000.0, 64, False, 0.15, 64)
    for _ in range(20):
        plan = engine.Plan(X, Y, prm)
        ms = plan.stats()["build_ms"]
        assert ms > 0
        plan.apply(torch.ones(m or n, 1, device=cuda))
        assert plan.stats()["build_ms"] == ms == plan.timings()["build"]
