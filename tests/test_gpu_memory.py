"""GPU: device memory that runs out.  The call reports it and the plan goes on working."""
import numpy as np
import pytest

import oracle as O
from matrox_ru_b200 import _lib, hgemm as H, structure as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as t
    assert t.cuda.is_available(), "GPU tests need a CUDA device"
    from matrox_ru_b200 import build
    build.build()
    return t


def fill(torch, leave):
    """Device memory down to `leave` bytes, held by the tensor returned."""
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")


@pytest.mark.parametrize("precision", ["fp64", "split_bf16"])
def test_workspaces_that_do_not_fit(torch, small_cases, precision):
    """A wider evaluation that finds no memory for its workspaces, then the earlier column count."""
    cds, r, wide = small_cases["h2b"], 16, 60000
    TW = np.random.default_rng(1).standard_normal(cds.n * r)
    want = O.eval_h2b(cds, TW, r)
    plan = H.Plan(cds, precision)
    w = torch.as_tensor(TW, device="cuda")
    plan.evaluate(w, r)
    W, Y = torch.zeros(2, cds.n * wide, dtype=torch.float64, device="cuda")
    hog = fill(torch, 64 << 20)
    with pytest.raises(_lib.MxbError) as e:
        plan.evaluate(W, wide, out=Y)
    assert e.value.code == _lib.MXB_ERR_NOMEM
    got = plan.evaluate(w, r).cpu().numpy()
    plan.status()
    del hog, W, Y
    torch.cuda.empty_cache()
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)


def test_plan_creation_needs_little_more_than_the_plan(torch):
    """FP64 plans copy a host CDS through a bounded staging buffer, in several pieces, not beside a
    second copy of it.  170 MB of near blocks, 110 MB to spare."""
    X = S.gaussian_mixture(16384, 3, 3, 0.0, 2.0, 0.3, None, seed=5)
    cds = S.build_cds(X, S.KernelSpec("gaussian", 0.4), leaf_size=256, budget=0.1, tol=1e-3, max_rank=9)
    size = 8 * (cds.D.size + cds.B.size + cds.VT.size)
    assert size > 160e6
    H.Plan(cds, "fp64").close()  # loads the kernels
    torch.zeros(1, device="cuda")
    hog = fill(torch, size + (110 << 20))
    plan = H.Plan(cds, "fp64")
    del hog
    torch.cuda.empty_cache()
    TW = np.random.default_rng(1).standard_normal(cds.n * 3)
    got = plan.evaluate(torch.as_tensor(TW, device="cuda"), 3).cpu().numpy()
    want = O.eval_h2b(cds, TW, 3)
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
