"""GPU: the FP64 dataflow launch at the edges of its column tiles (8, 16 and 32 wide variants), with
sums cut along K, odd ranks and leaves, operands that are only 8-byte aligned, and a wait that
runs out."""
import copy

import numpy as np
import pytest

import oracle as O
from matrox_ru_b200 import _lib, hgemm as H, structure as S

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the FP64 parity bar of the other GPU tests


@pytest.fixture(scope="module")
def torch():
    import torch as t
    assert t.cuda.is_available(), "GPU tests need a CUDA device"
    from matrox_ru_b200 import build
    build.build()
    return t


@pytest.fixture(scope="module")
def tall():
    """Leaves of several row tiles and near lists long enough to be cut along K."""
    X = S.gaussian_mixture(1501, 3, 3, 0.0, 2.0, 0.3, None, seed=5)
    return S.build_cds(X, S.KernelSpec("gaussian", 0.4), leaf_size=200, budget=0.9, tol=1e-7, max_rank=149)


@pytest.mark.parametrize("r", [1, 8, 9, 16, 17, 32, 33, 100])
@pytest.mark.parametrize("name", ["tall", "ragged"])
def test_column_tile_edges(torch, small_cases, tall, name, r):
    cds = tall if name == "tall" else small_cases[name]
    rng = np.random.default_rng(r)
    TW, Y0 = rng.standard_normal((2, cds.n * r))
    plan = H.Plan(cds, "fp64")
    room = torch.zeros(2 * cds.n * r + 3, dtype=torch.float64, device="cuda")
    w, y = room[1:1 + cds.n * r], room[2 + cds.n * r:2 + 2 * cds.n * r]  # 8-byte aligned
    w.copy_(torch.as_tensor(TW))
    for call, want in ((plan.evaluate, O.eval_h2b(cds, TW, r)), (plan.adjoint, O.adjoint(cds, TW, r))):
        for accumulate in (False, True):
            y.copy_(torch.as_tensor(Y0))
            call(w, r, out=y, accumulate=accumulate)
            ref = want + Y0 if accumulate else want
            assert np.abs(y.cpu().numpy() - ref).max() <= TOL * np.abs(ref).max()
            assert room[0] == 0 and room[1 + cds.n * r] == 0 and room[-1] == 0  # nothing else written
    plan.status()


def test_changing_column_counts_on_one_plan(torch, tall):
    """Buffers and counters grow and are reused across right-hand-side counts and directions."""
    plan = H.Plan(tall, "fp64")
    for r in (3, 70, 16, 1, 70):
        TW = np.random.default_rng(r).standard_normal(tall.n * r)
        w = torch.as_tensor(TW, device="cuda")
        got, adj = plan.evaluate(w, r).cpu().numpy(), plan.adjoint(w, r).cpu().numpy()
        want, wadj = O.eval_h2b(tall, TW, r), O.adjoint(tall, TW, r)
        assert np.abs(got - want).max() <= TOL * np.abs(want).max()
        assert np.abs(adj - wadj).max() <= TOL * np.abs(wadj).max()


def test_wait_that_runs_out_reports_timeout(torch, tall):
    r = 16
    TW = np.random.default_rng(0).standard_normal(tall.n * r)
    w = torch.as_tensor(TW, device="cuda")
    plan = H.Plan(tall, "fp64")
    plan.set_test_hooks(0, wait_cycles=1)  # the first wait that is not already over gives up
    plan.evaluate(w, r)
    with pytest.raises(_lib.MxbError) as e:
        plan.status()
    assert e.value.code == _lib.MXB_ERR_TIMEOUT
    plan.set_test_hooks(0)
    want = O.eval_h2b(tall, TW, r)
    assert np.abs(plan.evaluate(w, r).cpu().numpy() - want).max() <= TOL * np.abs(want).max()
    plan.status()


@pytest.mark.parametrize("r", [5, 16, 70])
def test_waits_of_any_limit_end_with_a_status(torch, tall, r):
    """Limits from nothing to a few polls: some lanes of a warp find a barrier complete where others
    give up.  Every such evaluation returns, with a timeout or with the product, and the plan
    computes correctly after it."""
    TW = np.random.default_rng(r).standard_normal(tall.n * r)
    w = torch.as_tensor(TW, device="cuda")
    plan = H.Plan(tall, "fp64")
    want = O.eval_h2b(tall, TW, r)
    for limit in (1, 30, 100, 300, 1000, 3000, 10000, 30000):
        plan.set_test_hooks(0, wait_cycles=limit)
        got = plan.evaluate(w, r).cpu().numpy()
        try:
            plan.status()
        except _lib.MxbError as e:
            assert e.code == _lib.MXB_ERR_TIMEOUT
        else:
            assert np.abs(got - want).max() <= TOL * np.abs(want).max()
    plan.set_test_hooks(0)
    assert np.abs(plan.evaluate(w, r).cpu().numpy() - want).max() <= TOL * np.abs(want).max()
    plan.status()


def test_timeout_outlives_the_workspaces_it_happened_in(torch, tall):
    """A timed-out evaluation, then one that needs more counters and partial tiles (the workspaces
    are replaced) and one in the other direction: status() still reports the first."""
    rng = np.random.default_rng(2)
    plan = H.Plan(tall, "fp64")
    w = torch.as_tensor(rng.standard_normal(tall.n * 8), device="cuda")
    plan.set_test_hooks(0, wait_cycles=1)
    plan.evaluate(w, 8)
    plan.set_test_hooks(0)
    TW = rng.standard_normal(tall.n * 200)
    wide = torch.as_tensor(TW, device="cuda")
    got = plan.evaluate(wide, 200).cpu().numpy()
    plan.adjoint(wide, 200)
    want = O.eval_h2b(tall, TW, 200)
    assert np.abs(got - want).max() <= TOL * np.abs(want).max()
    with pytest.raises(_lib.MxbError) as e:
        plan.status()
    assert e.value.code == _lib.MXB_ERR_TIMEOUT
    plan.status()


@pytest.mark.parametrize("r", [5, 16, 40])
@pytest.mark.parametrize("name", ["hss", "h2b", "ragged"])
def test_infinities_stay_infinities(torch, small_cases, name, r):
    """Ranks and leaves off the multiples of 8 on positive blocks: an infinite right-hand side gives
    infinities, as the oracle's loops do, and NaN only where it gives NaN (the padding of the 8 x 8
    sub-blocks multiplies nothing that is not finite)."""
    cds = copy.copy(small_cases[name])
    for pool in ("D", "B", "VT"):
        setattr(cds, pool, np.abs(getattr(cds, pool)) + 0.125)
    TW = np.random.default_rng(r).standard_normal((cds.n, r))
    TW[3, 0], TW[-2, 1], TW[5, 2], TW[5, 3] = np.inf, -np.inf, np.nan, 1e307
    lo = cds.leaf_lids_offset
    TW = np.concatenate([TW[lo[i]:lo[i + 1]].reshape(-1, order="F") for i in range(cds.nleaf)])
    plan = H.Plan(cds, "fp64")
    w = torch.as_tensor(TW, device="cuda")
    with np.errstate(all="ignore"):
        for call, want in ((plan.evaluate, O.eval_h2b(cds, TW, r)), (plan.adjoint, O.adjoint(cds, TW, r))):
            got = call(w, r).cpu().numpy()
            assert np.isinf(want).any() and np.isnan(want).any()
            assert np.array_equal(np.isnan(got), np.isnan(want))
            assert np.array_equal(np.isposinf(got), np.isposinf(want))
            assert np.array_equal(np.isneginf(got), np.isneginf(want))
            ok = np.isfinite(want)
            assert np.abs(got[ok] - want[ok]).max() <= TOL * np.abs(want[ok]).max()
    plan.status()


@pytest.fixture(scope="module")
def short():
    """Blocks of at most 16 and of at most 32 rows: the variants of 128 and of 64 columns (the first too
    small for them but with very many columns)."""
    out = {}
    for leaf, n, budget in ((16, 999, 0.05), (16, 8000, 0.0), (16, 7999, 0.008), (32, 16000, 0.0), (32, 15999, 0.008)):
        X = S.gaussian_mixture(n, 4, 4, 0.0, 3.0, 0.4, None, seed=n)
        out[leaf, n] = S.build_cds(X, S.KernelSpec("gaussian", 1.0), leaf_size=leaf, budget=budget, tol=1e-7, max_rank=leaf - n % 3)
    return out


@pytest.mark.parametrize("r", [3, 33, 64, 65, 100, 128, 129, 200, 300])
@pytest.mark.parametrize("key", [(16, 8000), (16, 7999), (32, 16000), (32, 15999)])
def test_short_blocks(torch, short, key, r):
    cds = short[key]
    rng = np.random.default_rng(r)
    TW, Y0 = rng.standard_normal((2, cds.n * r))
    plan = H.Plan(cds, "fp64")
    room = torch.zeros(2 * cds.n * r + 3, dtype=torch.float64, device="cuda")
    w, y = room[1:1 + cds.n * r], room[2 + cds.n * r:2 + 2 * cds.n * r]  # 8-byte aligned
    w.copy_(torch.as_tensor(TW))
    for call, want in ((plan.evaluate, O.eval_h2b(cds, TW, r)), (plan.adjoint, O.adjoint(cds, TW, r))):
        for accumulate in (False, True):
            y.copy_(torch.as_tensor(Y0))
            call(w, r, out=y, accumulate=accumulate)
            ref = want + Y0 if accumulate else want
            assert np.abs(y.cpu().numpy() - ref).max() <= TOL * np.abs(ref).max()
            assert room[0] == 0 and room[1 + cds.n * r] == 0 and room[-1] == 0  # nothing else written
    plan.status()
    width = {x["width"] for x in plan.profile(w, r)}
    assert width == {8 if r <= 8 else 32 if r <= 32 else 64 if key[0] == 32 or r <= 64 else 128}


@pytest.mark.parametrize("name,r", [("ragged", 13000), ("short", 13000), ("short", 52010)])
def test_many_tiles(torch, small_cases, short, name, r):
    """Fused sums, and units of two column tiles (the last size; an odd number of tiles)."""
    cds = small_cases["ragged"] if name == "ragged" else short[16, 999]
    rng = np.random.default_rng(r)
    TW, Y0 = rng.standard_normal((2, cds.n * r))
    plan = H.Plan(cds, "fp64")
    w, y = torch.as_tensor(TW, device="cuda"), torch.as_tensor(Y0, device="cuda")
    want = O.eval_h2b(cds, TW, r)
    got = plan.evaluate(w, r).cpu().numpy()
    assert np.abs(got - want).max() <= TOL * np.abs(want).max()
    got = plan.adjoint(w, r, out=y, accumulate=True).cpu().numpy()
    want = O.adjoint(cds, TW, r) + Y0
    assert np.abs(got - want).max() <= TOL * np.abs(want).max()
    plan.status()
