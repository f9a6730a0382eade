"""Inputs of a differentiable problem that torch changes, or whose memory it
gives away, right after update(): the library reads them as they were.  Its stream
is kept busy for some 0.1 s first, so that its copies come late."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("change", ["in place", "freed"])
def test_inputs_as_they_were_at_the_call(change):
    torch = pytest.importorskip("torch")
    import ugcore_gb300 as ug
    from ugcore_gb300 import problems
    from ugcore_gb300.adjoint import DifferentiableProblem
    ctx = ug.Context(0)
    cfg = problems.config("c3", nref=4)
    p = DifferentiableProblem(ctx, cfg)
    rng = np.random.default_rng(1)
    m0 = torch.tensor(rng.normal(size=p.num_elements), device="cuda")
    f0 = torch.tensor(rng.uniform(-1, 1, p.n), device="cuda")
    p.update(m0.clone(), f0.clone())
    want = p.solve_u().cpu().numpy()
    p.update(torch.zeros_like(m0), torch.ones_like(f0))
    assert not np.array_equal(p.solve_u().cpu().numpy(), want)
    m, f = m0.clone(), f0.clone()
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream)):
        torch.cuda._sleep(200_000_000)
    p.update(m, f)
    if change == "in place":
        m.add_(1.0)
        f.neg_()
    else:
        p._inputs = None
        del m, f
        junk = [torch.full_like(m0, 7.0) for _ in range(4)] + [torch.full_like(f0, 7.0) for _ in range(4)]
    assert np.array_equal(p.solve_u().cpu().numpy(), want)
