"""GPU: split-BF16 evaluations in one flow launch (every pass in one launch, units waiting on
per-node counters) against the same plans with a launch per pass.  The products, their order and
the splits are the same, so results are bit-identical at every column count and layout."""
import dataclasses

import numpy as np
import pytest

from matrox_ru_b200 import _lib, hgemm as H, structure as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as t
    assert t.cuda.is_available(), "GPU tests need a CUDA device"
    from matrox_ru_b200 import build
    build.build()
    return t


def results(torch, cds, mode, r, hooks=0):
    """Forward and transposed products, leaf-blocked and in caller order, plain and accumulated."""
    plan = H.Plan(cds, mode, adjoint=True)
    plan.set_test_hooks(hooks)
    plan.set_permutation(cds.perm)
    g = torch.Generator(device="cuda")
    g.manual_seed(r)
    out = []
    for _ in range(2):  # the second set of operands takes the launches prepared for the first
        W = torch.randn(cds.n * r, dtype=torch.float64, device="cuda", generator=g)
        Y = torch.randn(cds.n * r, dtype=torch.float64, device="cuda", generator=g)
        out += [plan.evaluate(W, r), plan.adjoint(W, r)]
        for accumulate in (False, True):
            out.append(plan.evaluate(W, r, out=Y.clone(), accumulate=accumulate))
        if hooks:
            continue  # the one-launch mode takes leaf-blocked operands
        rows, cols = W.view(cds.n, r), W.view(r, cds.n).t()
        out += [plan.evaluate_ordered(rows), plan.evaluate_ordered(cols, out=Y.clone().view(r, cds.n).t(), accumulate=True),
                plan.adjoint_ordered(rows), plan.adjoint_ordered(cols)]
    plan.status()
    return plan.info()["launches"], out


@pytest.mark.parametrize("r", [1, 16, 17, 64, 65, 100, 128])
@pytest.mark.parametrize("name", ["hss", "h2b", "ragged"])
def test_flow_equals_separate_launches(torch, small_cases, monkeypatch, name, r):
    for mode in ("split_bf16", "split_bf16_far6"):
        n, flow = results(torch, small_cases[name], mode, r)
        assert n <= 2, (mode, n)
        monkeypatch.setenv("MXB_TC_FLOW", "0")
        n, separate = results(torch, small_cases[name], mode, r)
        monkeypatch.delenv("MXB_TC_FLOW")
        assert n > 2
        for k, (a, b) in enumerate(zip(flow, separate)):
            assert torch.equal(a, b), (mode, k)


@pytest.mark.parametrize("r, width", [(130, 64), (257, 64), (6001, 128)])
def test_flow_beyond_one_column_tile(torch, small_cases, monkeypatch, r, width):
    """Several column tiles, the last one narrow, at both tile widths; W split by a launch before
    and (the one-launch mode) by units of the flow launch."""
    cds = small_cases["ragged"]
    n, flow = results(torch, cds, "split_bf16_x6", r)
    assert n <= 2
    n, one = results(torch, cds, "split_bf16_x6", r, _lib.DEBUG_ONE_LAUNCH)
    assert n == 1
    plan = H.Plan(cds, "split_bf16_x6")
    assert {x["width"] for x in plan.profile(torch.zeros(cds.n * r, dtype=torch.float64, device="cuda"), r)
            if x["phase"] != "split_w"} == {width}
    monkeypatch.setenv("MXB_TC_FLOW", "0")
    n, separate = results(torch, cds, "split_bf16_x6", r)
    assert n > 2
    for k, (a, b) in enumerate(zip(flow, separate)):
        assert torch.equal(a, b), k
    for k, (a, b) in enumerate(zip(one, separate[:4] + separate[8:12])):
        assert torch.equal(a, b), k


def test_flow_batch_equals_plans_alone(torch, small_cases):
    cases = [("h2b", "split_bf16", 40), ("ragged", "split_bf16_far6", 128), ("hss", "split_bf16_x6", 3)]
    plans = [H.Plan(small_cases[n], m) for n, m, _ in cases]
    W = [torch.randn(p.n * r, dtype=torch.float64, device="cuda") for p, (_, _, r) in zip(plans, cases)]
    alone = [p.evaluate(w, r).clone() for p, w, (_, _, r) in zip(plans, W, cases)]
    for one_launch in (False, True):
        batch = H.Batch(plans)
        batch.set_one_launch(one_launch)
        for _ in range(2):
            got = batch.evaluate(W, [r for _, _, r in cases])
        batch.status()
        assert batch.info()["launches"] == (1 if one_launch else 2)
        for a, b in zip(got, alone):
            assert torch.equal(a, b)


@pytest.mark.parametrize("precision", ["split_bf16", "fp64"])
def test_replay_of_a_captured_evaluation(torch, small_cases, precision):
    """A plan's launches in a caller's graph: other buffers than the first evaluation's, replayed on
    new values."""
    cds, r = small_cases["h2b"], 24
    plan = H.Plan(cds, precision)
    W = torch.randn(cds.n * r, dtype=torch.float64, device="cuda")
    plan.evaluate(W, r)
    Ws, Ys = torch.empty_like(W), torch.empty_like(W)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        plan.evaluate(Ws, r, out=Ys)
    for seed in range(2):
        torch.manual_seed(seed)
        Ws.normal_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(Ys, plan.evaluate(Ws, r))
    plan.status()


@pytest.mark.parametrize("hooks", [0, _lib.DEBUG_ONE_LAUNCH])
def test_in_place_without_diagonal_blocks(torch, small_cases, hooks):
    """Y = W on near lists without a leaf's own block: a Y block is written once the W it replaces
    has been split, as with a launch per pass."""
    full, r = small_cases["h2b"], 100
    keep = np.flatnonzero((full.npairx != full.npairy) & (full.npairx % 2 == 0))
    cds = dataclasses.replace(full, npairx=full.npairx[keep], npairy=full.npairy[keep], Dptr=full.Dptr[keep])
    plan = H.Plan(cds, "split_bf16", adjoint=True)
    plan.set_test_hooks(hooks)
    W = torch.randn(cds.n * r, dtype=torch.float64, device="cuda")
    for call in (plan.evaluate, plan.adjoint):
        want = call(W, r).clone()
        assert plan.info()["launches"] == 1
        for _ in range(20):
            x = W.clone()
            call(x, r, out=x)
            assert torch.equal(x, want)
    plan.status()


@pytest.mark.parametrize("r", [1, 100])
def test_nodes_in_many_far_lists(torch, monkeypatch, r):
    """An adjoint with a node in very many far lists, whose launches are timed instead of taken for
    granted, and its forward product: the same as in separate launches."""
    X = S.gaussian_mixture(24000, 8, 8, 0.0, 4.0, 0.5, None, seed=2)
    cds = S.build_cds(X, S.KernelSpec("gaussian", 1.0), leaf_size=32, budget=0.008, tol=1e-3, max_rank=24, id_on_gpu=True)
    assert np.bincount(cds.fpairy).max() > 60
    W = torch.randn(cds.n * r, dtype=torch.float64, device="cuda")
    got = []
    for flow in ("1", "0"):
        monkeypatch.setenv("MXB_TC_FLOW", flow)
        plan = H.Plan(cds, "split_bf16", adjoint=True)
        got.append([plan.evaluate(W, r), plan.adjoint(W, r), plan.adjoint(W, r)])
        plan.status()
    for a, b in zip(*got):
        assert torch.equal(a, b)
