"""GPU: a plan's evaluations in a caller's CUDA graph.  What the captured launches point to -- leaf
offsets, workspaces, task lists -- stays as it was for the life of the plan, whatever the plan
evaluates before a replay; an evaluation that still has to be prepared is refused, not captured."""
import pytest

from matrox_ru_b200 import _lib, hgemm as H

pytestmark = pytest.mark.gpu
PRECISIONS = ["fp64", "split_bf16"]


@pytest.fixture(scope="module")
def torch():
    import torch as t
    assert t.cuda.is_available(), "GPU tests need a CUDA device"
    from matrox_ru_b200 import build
    build.build()
    return t


@pytest.mark.parametrize("precision", PRECISIONS)
def test_replay_after_other_column_counts(torch, small_cases, precision):
    """More column counts, in both directions and layouts, than task lists or entries are kept for,
    up to wider ones that replace every workspace."""
    cds, r = small_cases["ragged"], 24
    plan = H.Plan(cds, precision, adjoint=True)
    plan.set_permutation(cds.perm)
    W = torch.randn(cds.n, r, dtype=torch.float64, device="cuda")
    calls = [lambda w, y: plan.evaluate(w.view(-1), r, out=y.view(-1)),
             lambda w, y: plan.adjoint(w.view(-1), r, out=y.view(-1)),
             lambda w, y: plan.evaluate_ordered(w, out=y),
             lambda w, y: plan.adjoint_ordered(w, out=y, accumulate=True)]
    Ys = [torch.zeros_like(W) for _ in calls]
    for f, y in zip(calls, Ys):
        f(W, y)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        for f, y in zip(calls, Ys):
            f(W, y)
    for k in (1, 3, 9, 17, 33, 50, 65, 70, 100, 129, 140, 200, 300):
        V = torch.randn(cds.n, k, dtype=torch.float64, device="cuda")
        plan.evaluate(V.view(-1), k)
        plan.adjoint(V.view(-1), k)
        plan.evaluate_ordered(V)
    for seed in range(2):
        torch.manual_seed(seed)
        W.normal_()
        want = []
        for f, y in zip(calls, Ys):
            y.normal_()
            want.append(f(W, y.clone()))
        g.replay()
        torch.cuda.synchronize()
        for a, b in zip(Ys, want):
            assert torch.equal(a.view(-1), b.reshape(-1))
    plan.status()


@pytest.mark.parametrize("precision", PRECISIONS)
def test_unprepared_evaluations_are_refused_under_capture(torch, small_cases, precision):
    """Neither a first evaluation nor a wider one allocates into a capture, which stays usable."""
    cds = small_cases["h2b"]
    plan = H.Plan(cds, precision, adjoint=True)
    W = torch.randn(cds.n * 90, dtype=torch.float64, device="cuda")
    Y, Z = torch.empty_like(W), torch.empty_like(W)

    def refused(call, r):
        with pytest.raises(_lib.MxbError) as e:
            call(W, r, out=Y)
        assert e.value.code == _lib.MXB_ERR_UNSUPPORTED

    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        refused(plan.evaluate, 8)
        Z.copy_(W)
    want = plan.evaluate(W, 8).clone()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        refused(plan.evaluate, 90)
        refused(plan.adjoint, 8)
        plan.evaluate(W, 8, out=Y)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(Y[:want.numel()], want)
    plan.status()


@pytest.mark.parametrize("precision", PRECISIONS)
def test_a_recorded_plan_does_not_grow(torch, small_cases, precision):
    """Only what the captured evaluation uses is kept: a loop over more column counts than a plan keeps
    entries for holds no more memory after many rounds than after a few."""
    cds, counts = small_cases["h2b"], range(4, 64, 5)
    plan = H.Plan(cds, precision)
    W = torch.randn(cds.n * 64, dtype=torch.float64, device="cuda")
    Y = torch.empty_like(W)
    plan.evaluate(W, 24, out=Y)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        plan.evaluate(W, 24, out=Y)

    def free_after(rounds):
        for _ in range(rounds):
            for r in counts:
                plan.evaluate(W, r, out=Y)
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    first = free_after(3)
    assert free_after(400) >= first - (4 << 20)
    plan.status()
