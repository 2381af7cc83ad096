"""GPU: device memory that runs out.  The call reports it and the plan goes on working."""
import numpy as np
import pytest

import oracle as O
from matrox_ru_b200 import _lib, hgemm as H

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
