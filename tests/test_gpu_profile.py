"""GPU: launch-by-launch timing (mxb_plan_profile / mxb_batch_profile).  The per-launch
algorithmic flops must add up exactly to the reference's flop model (computeFlops,
matroxTest-V1/compression.h:1079-1130, restated by mxb_plan_flops), and the profiled
evaluation must leave the ordinary result in Y."""
import numpy as np
import pytest

from matrox_ru_b200 import _lib, hgemm as H
from test_f64_schedule import TILE_W, WSKEL, schedule

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as t
    assert t.cuda.is_available(), "GPU tests need a CUDA device"
    from matrox_ru_b200 import build
    build.build()
    return t


@pytest.mark.parametrize("precision", ["fp64", "split_bf16", "split_bf16_far6", "split_bf16_x6"])
@pytest.mark.parametrize("name", ["hss", "h2b", "ragged"])
def test_profile_flops_and_result(torch, small_cases, name, precision):
    cds = small_cases[name]
    r = 72
    plan = H.Plan(cds, precision)
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    TW = torch.randn(cds.n * r, dtype=torch.float64, device="cuda", generator=g)
    want = plan.evaluate(TW, r)
    out = torch.full_like(want, 7.0)  # overwritten by the profiled evaluation
    recs = plan.profile(TW, r, out=out)
    torch.cuda.synchronize()
    plan.status()
    # one record per op; ops chained into the launch before them (device-side level barriers)
    # report ms 0, the launch's own record covers them
    assert sum(not x["chained"] for x in recs) == plan.info()["launches"]
    assert sum(x["flops"] for x in recs) == plan.flops(r) == cds.flops(r)
    for x in recs:
        assert (x["ms"] > 0.0) != x["chained"]
        assert x["issued_flops"] >= x["flops"]
        assert x["units"] > 0 or x["flops"] == 0  # units without items zero their output
    phases = {x["phase"] for x in recs}
    if precision == "fp64":
        assert phases <= {"up", "far_down", "near_leaf_down"}
    else:
        assert phases <= {"split_w", "up", "far", "far_near", "down", "near", "leaf_down"}
        # the far couplings of all depths run as one launch, joined by the near field when
        # both use the same number of products
        assert sum(x["phase"] in ("far", "far_near") for x in recs) == 1
        assert ("near" in phases) == (precision == "split_bf16_far6")
        k = 6.0 if precision == "split_bf16_x6" else None
        if k:
            for x in recs:
                assert x["issued_flops"] >= k * x["flops"]
    torch.testing.assert_close(out, want, rtol=1e-13, atol=1e-13 * float(want.abs().max()))


def test_batch_profile(torch, small_cases):
    cases = [(small_cases["h2b"], 40), (small_cases["ragged"], 200), (small_cases["hss"], 96)]
    plans = [H.Plan(c, "split_bf16") for c, _ in cases]
    batch = H.Batch(plans)
    TWs = [torch.randn(c.n * r, dtype=torch.float64, device="cuda") for c, r in cases]
    want = batch.evaluate(TWs, [r for _, r in cases])
    outs = [torch.zeros_like(w) for w in want]
    recs = batch.profile(TWs, [r for _, r in cases], outs)
    batch.status()
    assert sum(not x["chained"] for x in recs) == batch.info()["launches"]
    assert sum(x["flops"] for x in recs) == sum(c.flops(r) for c, r in cases)
    for o, w in zip(outs, want):
        torch.testing.assert_close(o, w, rtol=1e-13, atol=1e-13 * float(w.abs().max()))


@pytest.mark.parametrize("r,widths", [(1, (8,)), (13, (16,)), (100, (32, 64, 128))])
@pytest.mark.parametrize("name", ["h2b", "ragged"])
def test_fp64_profile_is_of_the_launch_that_ran(torch, small_cases, name, r, widths):
    """Width, units and issued flops of the one launch's column tiles and task list, and its passes'
    spans, which make up the launch."""
    cds = small_cases[name]
    recs = H.Plan(cds, "fp64").profile(torch.randn(cds.n * r, dtype=torch.float64, device="cuda"), r)
    tasks, items, counts = schedule(_lib.load(), cds, False, r)
    ncol, nb = int(counts[4]), -(-r // 8)
    width = recs[0]["width"]
    assert width in widths and all(x["width"] == width for x in recs) and ncol == -(-8 * nb // width)
    assert sum(x["units"] for x in recs) == len(tasks) * ncol
    up = [x for x in recs if x["phase"] == "up"]
    assert sum(x["units"] for x in up) == ncol * int(np.isin(tasks["kind"], (TILE_W, WSKEL)).sum())
    # a warp multiplies its share of a tile's 8-row sub-blocks in pairs
    warps = {8: 4, 16: 4, 32: 2, 64: 1, 128: 1}[width]
    issued = 0
    for t in tasks:
        m8 = int(t["m8"])
        rows = sum(16 * -(-(m8 * (w + 1) // warps - m8 * w // warps) // 2) for w in range(warps))
        issued += 2 * rows * 8 * int(items["k8"][t["item0"]:t["item0"] + t["nitem"]].sum()) * 8 * nb
    assert sum(x["issued_flops"] for x in recs) == issued
    assert all(x["level_ms"] > 0 for x in recs)
    assert 0.5 * recs[0]["ms"] < sum(x["level_ms"] for x in recs) < 1.1 * recs[0]["ms"] + 0.01


def test_flow_profile_counts_what_is_issued(torch, small_cases):
    """A flow launch: products of whole 16-column groups only, and the passes' spans inside it."""
    cds = small_cases["ragged"]
    plan = H.Plan(cds, "split_bf16_x6")
    recs = {r: plan.profile(torch.randn(cds.n * r, dtype=torch.float64, device="cuda"), r) for r in (5, 16, 64)}
    issued = {r: sum(x["issued_flops"] for x in v) for r, v in recs.items()}
    assert issued[5] == issued[16] and issued[64] == 4 * issued[16]
    for v in recs.values():
        launch = sum(x["ms"] for x in v)
        assert plan.info()["launches"] == 1
        assert all(x["level_ms"] > 0 for x in v)
        assert 0.3 * launch < sum(x["level_ms"] for x in v) < 1.1 * launch + 0.01
