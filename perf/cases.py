"""The workloads whose time is followed, as a user's program runs them through `matrox_ru_b200`.

A case names a kernel matrix (points, kernel, leaf size, near-field budget, maximum rank), the
number of right-hand sides and the entry point; `prepare` gives what such a program holds before
the call: the plan of the compressed matrix and its operands.  The compressed matrix (the CDS)
depends on the case alone, as a user compresses once and evaluates many times; right-hand sides
come from the seed.  The compression here is a quick stand-in for the ID build: tree and
interaction lists are the package's, skeletons are a random subset of the candidate points and
the projections interpolate from them, so block shapes, ranks and value ranges are the real
ones while a matrix of 65536 points is ready in about a second.
"""
import functools
import math

import numpy as np
import torch

from matrox_ru_b200 import hgemm as H
from matrox_ru_b200 import structure as S
from matrox_ru_b200._lib import FLAG_OUTPUT_IS_ZERO

DEV = "cuda"


def listed():
    return [
        # the smallest use: one matrix-vector product of a small model (launch latency)
        dict(name="evaluate fp64 1024x1", kind="evaluate", precision="fp64", n=1024, d=4, kernel="gaussian", h=1.0,
             leaf=64, budget=0.2, rank=48, nrhs=1),
        # a small model applied to a few columns in the caller's point order, tensor cores
        dict(name="ordered split 2048x32", kind="ordered", precision="split_bf16", n=2048, d=4, kernel="gaussian",
             h=1.0, leaf=64, budget=0.2, rank=48, nrhs=32),
        # plain HSS in FP64: d = 8, leaf 128, 256 right-hand sides
        dict(name="hss fp64 16384x256", kind="evaluate", precision="fp64", n=16384, d=8, kernel="gaussian", h=1.0,
             leaf=128, budget=0.0, rank=128, nrhs=256),
        # one product inside an iterative solver (conjugate gradients) on the full-size matrix
        dict(name="matvec fp64 65536x1", kind="evaluate", precision="fp64", n=65536, d=28, kernel="gaussian", h=2.0,
             leaf=256, budget=0.03, rank=256, nrhs=1),
        # the headline workload, FP64 and split-BF16
        dict(name="h2b fp64 65536x1024", kind="evaluate", precision="fp64", n=65536, d=28, kernel="gaussian", h=2.0,
             leaf=256, budget=0.03, rank=256, nrhs=1024),
        dict(name="h2b split 65536x1024", kind="evaluate", precision="split_bf16", n=65536, d=28, kernel="gaussian",
             h=2.0, leaf=256, budget=0.03, rank=256, nrhs=1024),
        # ragged leaves and columns, caller's point order, six products in the far couplings
        dict(name="ordered far6 30011x130", kind="ordered", precision="split_bf16_far6", n=30011, d=18, kernel="imq",
             h=1.5, leaf=250, budget=0.05, rank=200, nrhs=130),
        # a kernel-ridge training step: loss and gradient by autograd, FP32 operands
        dict(name="gradient split 65536x64", kind="gradient", precision="split_bf16", n=65536, d=18, kernel="gaussian",
             h=1.5, leaf=256, budget=0.03, rank=256, nrhs=64),
        # the transposed product in FP64
        dict(name="adjoint fp64 32768x64", kind="adjoint", precision="fp64", n=32768, d=18, kernel="gaussian", h=1.5,
             leaf=256, budget=0.05, rank=256, nrhs=64),
        # many uneven matrices in one launch sequence
        dict(name="batch of 12", kind="batch", precision="split_bf16", count=12, n_lo=4096, n_hi=16384, leaf=256,
             budget=0.03, rank=256, nrhs_lo=32, nrhs_hi=512, one_launch=False, geometry=3),
        # the reference-signature call on pinned host arrays, copies included
        dict(name="dropin hss 16384x256", kind="dropin", precision="fp64", n=16384, d=8, kernel="gaussian", h=1.0,
             leaf=128, budget=0.0, rank=128, nrhs=256),
        # the compression of one tree level: sample matrices and their column IDs
        dict(name="compress 32 of 1024x512", kind="compress", nodes=32, cols=512, d=28, kernel="gaussian", h=2.0,
             tol=1e-5, rank=256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["evaluate", "evaluate", "evaluate", "ordered", "ordered", "gradient", "adjoint", "batch",
                       "dropin", "compress"])
    kernel = rng.choice(["gaussian", "gaussian", "imq"])
    if kind == "compress":
        cols = _log_int(rng, 48, 512)
        return dict(kind=kind, nodes=rng.randint(4, 32), cols=cols, d=rng.choice([8, 18, 28]), kernel=kernel,
                    h=round(rng.uniform(1.5, 3.0), 2), tol=1e-7, rank=max(16, cols // rng.choice([2, 2, 3, 4])))
    if kind == "batch":
        lo = _log_int(rng, 1024, 6000)
        return dict(kind=kind, precision="split_bf16", count=rng.randint(3, 12), n_lo=lo, n_hi=min(16384, 4 * lo),
                    leaf=rng.randint(100, 256), budget=0.03, rank=rng.randint(64, 256), nrhs_lo=rng.randint(8, 48),
                    nrhs_hi=rng.randint(64, 512), one_launch=rng.random() < 0.3, geometry=rng.randint(0, 1 << 20))
    split = rng.choice(["split_bf16", "split_bf16", "split_bf16_far6", "split_bf16_x6"])
    precision = split if rng.random() < 0.55 else "fp64"
    n = _log_int(rng, 1024, 16384 if kind == "dropin" else 65536)
    leaf = rng.randint(48, 128) if n < 8192 else rng.randint(100, 256) if n <= 16384 else rng.randint(180, 256)
    leaves = 2 ** math.ceil(math.log2(n / leaf))
    hss = rng.random() < 0.25
    return dict(kind=kind, precision=precision, n=n, d=rng.choice([4, 8, 18, 28, 54]), kernel=kernel,
                h=round(rng.uniform(0.5, 3.0), 2), leaf=leaf, budget=0.0 if hss else max(0.03, 4.0 / leaves),
                rank=rng.randint(max(24, leaf // 2), leaf), nrhs=_log_int(rng, 1, 512 if kind == "dropin" else 1024))


# ---- the compressed matrix -------------------------------------------------------------------

def _kernel(d2, kind, h):
    return torch.exp(d2 * (-0.5 / (h * h))) if kind == "gaussian" else 1.0 / torch.sqrt(1.0 + d2 / (h * h))


def _padded(sets):
    size = np.array([len(s) for s in sets], np.int64)
    idx = np.zeros((len(sets), max(1, int(size.max(initial=0)))), np.int64)
    for i, s in enumerate(sets):
        idx[i, :len(s)] = s
    return torch.as_tensor(idx, device=DEV), torch.as_tensor(size, device=DEV)


def _blocks(X, rows, cols, kind, h):
    """K(X[rows_b], X[cols_b]) for padded index sets, as (b, columns, rows)."""
    P, Q = X[cols], X[rows]
    d2 = torch.baddbmm(((P * P).sum(2)[:, :, None] + (Q * Q).sum(2)[:, None, :]), P, Q.transpose(1, 2), alpha=-2.0)
    return _kernel(d2.clamp_(min=0.0), kind, h)


def _pool(X, sets, pairs_x, pairs_y, kind, h):
    """Kernel blocks of the pairs packed back to back, each column-major; and their offsets."""
    idx, size = _padded(sets)
    px, py = torch.as_tensor(pairs_x.astype(np.int64), device=DEV), torch.as_tensor(pairs_y.astype(np.int64), device=DEV)
    ofs = torch.cat([torch.zeros(1, dtype=torch.int64, device=DEV), torch.cumsum(size[px] * size[py], 0)]).cpu().numpy()
    pool = torch.empty(int(ofs[-1]), dtype=torch.float64, device=DEV)
    width = idx.shape[1]
    lane = torch.arange(width, device=DEV)
    step = max(1, (1 << 24) // (width * width))
    for a in range(0, len(pairs_x), step):
        b = min(len(pairs_x), a + step)
        K = _blocks(X, idx[px[a:b]], idx[py[a:b]], kind, h)
        keep = (lane[None, :] < size[py[a:b]][:, None])[:, :, None] & (lane[None, :] < size[px[a:b]][:, None])[:, None, :]
        pool[int(ofs[a]):int(ofs[b])] = K[keep]
    return pool, ofs[:-1].astype(np.uint64)


@functools.lru_cache(maxsize=16)
def _matrix(n, d, kernel, h, leaf, budget, rank):
    """(CDS without pool values, (D, B, VT) on the device)."""
    rng = np.random.default_rng([n, d, leaf, rank])
    Xh = S.gaussian_mixture(n, d, 16, -2.0, 2.0, 0.3, 1.0, seed=n + d)
    tree = S.build_tree(Xh, leaf)
    near = S.near_lists(tree, budget)
    far = S.far_lists(tree, near)
    nn, nl = tree.numnodes, tree.nleaf
    hss = all(len(x) == 1 for x in near)
    X = torch.as_tensor(Xh, device=DEV)
    leaves = [np.asarray(tree.lids[tree.leaf_node(i)], np.int64) for i in range(nl)]
    Ddim = np.array([len(x) for x in leaves], np.int32)
    lm = np.full(nn, -1, np.int32)
    lm[tree.first_leaf:] = np.arange(nl)
    inner = np.arange(nn) < tree.first_leaf
    lch = np.where(inner, 2 * np.arange(nn) + 1, -1).astype(np.int32)
    rch = np.where(inner, 2 * np.arange(nn) + 2, -1).astype(np.int32)
    # ranks: most nodes at the maximum, some below, as the ID leaves them
    skel, slen, proj = [np.zeros(0, np.int64)] * nn, np.zeros(nn, np.int32), [None] * nn
    for lev in range(tree.depth, 0, -1):
        nodes = range((1 << lev) - 1, (1 << (lev + 1)) - 1)
        cand = [leaves[lm[v]] if lch[v] < 0 else np.concatenate([skel[lch[v]], skel[rch[v]]]) for v in nodes]
        pick = []
        for c in cand:
            r = rank if rng.random() < 0.85 else int(rng.uniform(0.7, 1.0) * rank)
            pick.append(rng.permutation(len(c))[:max(1, min(r, len(c)))])
        ci, cs = _padded(cand)
        si, ss = _padded([c[p] for c, p in zip(cand, pick)])
        lane = torch.arange(si.shape[1], device=DEV)
        live = (lane[None, :] < ss[:, None]).to(torch.float64)
        Kss = _blocks(X, si, si, kernel, h) * live[:, :, None] * live[:, None, :]
        Kss += torch.diag_embed(1.0 - live + 1e-3)
        Ksc = _blocks(X, ci, si, kernel, h) * live[:, :, None]
        P = torch.cholesky_solve(Ksc, torch.linalg.cholesky(Kss))
        for q, v in enumerate(nodes):
            skel[v], slen[v] = cand[q][pick[q]], len(pick[q])
            Pv = P[q, :slen[v], :len(cand[q])].clone()
            Pv[:, torch.as_tensor(pick[q], device=DEV)] = torch.eye(int(slen[v]), dtype=torch.float64, device=DEV)
            proj[v] = Pv.t().contiguous().reshape(-1)
    levelset, idx = S.levelsets_top_down(tree)
    clevelset, wpart, cidx = S.coarsened_levels(tree)
    VTptr, off = np.zeros(nn, np.int32), 0
    for v in cidx.tolist():
        VTptr[v] = off
        off += proj[v].numel()
    VT = torch.cat([proj[v] for v in cidx.tolist()]) if off else torch.zeros(1, dtype=torch.float64, device=DEV)
    if hss:
        npx = np.arange(nl, dtype=np.int32)
        npy = npx.copy()
        fpx = np.arange(1, nn, dtype=np.int32)
        fpy = np.array([v - 1 if v % 2 == 0 else v + 1 for v in range(1, nn)], np.int32)
        nblockset = nblocks = fblockset = fblocks = np.array([0], np.int32)
    else:
        nblockset, nblocks, npx, npy = S.blocked_near(tree, near)
        fblockset, fblocks, fpx, fpy = S.blocked_far(tree, far)
    D, Dptr = _pool(X, leaves, npx, npy, kernel, h)
    B, Bptr = _pool(X, skel, fpx, fpy, kernel, h)
    lofs = np.concatenate([[0], np.cumsum(Ddim.astype(np.int64))]).astype(np.int64)
    cds = S.CDS(n=n, nleaf=nl, numnodes=nn, depth=tree.depth, is_hss=hss, D=np.empty(D.numel()), Dptr=Dptr,
                B=np.empty(B.numel()), Bptr=Bptr, VT=np.empty(VT.numel()), VTptr=VTptr, lchildren=lch, rchildren=rch,
                levelset=levelset, idx=idx, Ddim=Ddim, lm=lm, slen=slen, nblockset=nblockset, nblocks=nblocks,
                npairx=npx, npairy=npy, fblockset=fblockset, fblocks=fblocks, fpairx=fpx, fpairy=fpy, wpart=wpart,
                clevelset=clevelset, cidx=cidx, perm=np.concatenate(leaves), leaf_lids_offset=lofs, skels=skel)
    return cds, (D, B, VT)


def _matrix_of(c):
    return _matrix(c["n"], c["d"], c["kernel"], c["h"], c["leaf"], c["budget"], c["rank"])


@functools.lru_cache(maxsize=4)
def _host_matrix_of(*key):
    """The same matrix with its values on the host, for the reference-signature calls."""
    cds, (D, B, VT) = _matrix(*key)
    H.cache_invalidate()  # values change under the pools' addresses
    cds.D[:], cds.B[:], cds.VT[:] = D.cpu().numpy(), B.cpu().numpy(), VT.cpu().numpy()
    return cds


def _members(c):
    """The matrices of a batch: (matrix case, precision)."""
    rng = np.random.default_rng(c["geometry"])
    out = []
    for i in range(c["count"]):
        n = int(round(math.exp(rng.uniform(math.log(c["n_lo"]), math.log(c["n_hi"])))))
        leaves = 2 ** math.ceil(math.log2(n / c["leaf"]))
        out.append(dict(n=n, d=int(rng.choice([8, 18, 28, 54])), kernel="imq" if rng.random() < 0.5 else "gaussian",
                        h=float(np.round(rng.uniform(0.5, 3.0), 2)), leaf=c["leaf"],
                        budget=c["budget"] if i % 3 else max(c["budget"], 4.0 / leaves), rank=c["rank"],
                        nrhs=int(round(math.exp(rng.uniform(math.log(c["nrhs_lo"]), math.log(c["nrhs_hi"]))))),
                        precision="split_bf16_far6" if i % 4 == 3 else c["precision"]))
    return out


# ---- what a program holds, and its call --------------------------------------------------------

def _randn(seed, *shape, dtype=torch.float64):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return torch.randn(*shape, dtype=dtype, device=DEV, generator=g)


def _samples(c, seed):
    """Points and, per node of a level, sample rows and candidate columns (index arrays)."""
    n = max(4096, c["cols"] * 32)
    X = S.gaussian_mixture(n, c["d"], 16, -2.0, 2.0, 0.3, 1.0, seed=seed)
    order = np.argsort(X[:, 0], kind="stable")
    rng = np.random.default_rng(seed)
    ragged = np.random.default_rng(c["cols"]).integers(0, 1 + c["cols"] // 8, c["nodes"])
    rows, cols = [], []
    for b in range(c["nodes"]):
        m = c["cols"] - int(ragged[b])  # unevenly filled nodes, the same ones for every seed
        a = b * c["cols"]
        near, rest = order[a + c["cols"]:a + c["cols"] + m], np.delete(order, np.s_[a:a + 2 * c["cols"]])
        if len(near) < m:
            near = order[a - m:a]
        cols.append(order[a:a + m].astype(np.int64))
        rows.append(np.concatenate([near, rng.permutation(rest)[:m]]).astype(np.int64))
    return X, rows, cols


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "compress":
        X, rows, cols = _samples(c, seed)
        return dict(case=c, X=torch.as_tensor(X, device=DEV), rows=rows, cols=cols,
                    kernel=S.KernelSpec(c["kernel"], c["h"]))
    if kind == "batch":
        plans, W, out, nrhs = [], [], [], []
        for i, m in enumerate(_members(c)):
            cds, pools = _matrix_of(m)
            plans.append(H.Plan(cds, m["precision"], pools=pools))
            nrhs.append(m["nrhs"])
            W.append(_randn(seed * 64 + i, m["n"] * m["nrhs"], dtype=torch.float32).to(torch.float64))
            out.append(torch.empty_like(W[-1]))
        batch = H.Batch(plans)
        if c["one_launch"]:
            batch.set_one_launch(True)
        return dict(case=c, batch=batch, W=W, out=out, nrhs=nrhs)
    n, r = c["n"], c["nrhs"]
    if kind == "dropin":
        cds = _host_matrix_of(c["n"], c["d"], c["kernel"], c["h"], c["leaf"], c["budget"], c["rank"])
        H.set_precision(c["precision"])
        H.set_flags(FLAG_OUTPUT_IS_ZERO)  # the output array is zeroed by its owner
        W = torch.empty(n * r, dtype=torch.float64, pin_memory=True)
        W.copy_(_randn(seed, n * r))
        Y = torch.zeros(n * r, dtype=torch.float64, pin_memory=True)
        total = int(cds.slen.astype(np.int64).sum()) * r
        return dict(case=c, cds=cds, W=W.numpy(), Y=Y.numpy(), hold=(W, Y), wskel=np.zeros(total), uskel=np.zeros(total))
    cds, pools = _matrix_of(c)
    plan = H.Plan(cds, c["precision"], pools=pools, adjoint=kind in ("adjoint", "gradient"))
    if kind == "gradient":
        return dict(case=c, ev=H.Evaluator(cds, c["precision"], plan=plan),
                    W=_randn(seed, n, r, dtype=torch.float32).requires_grad_(),
                    T=_randn(seed + (1 << 32), n, r, dtype=torch.float32))
    if kind == "ordered":
        return dict(case=c, ev=H.Evaluator(cds, c["precision"], plan=plan), W=_randn(seed, n, r))
    W = _randn(seed, n * r)
    return dict(case=c, plan=plan, W=W, out=torch.empty_like(W))


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "evaluate":
        return state["plan"].evaluate(state["W"], c["nrhs"], out=state["out"])
    if kind == "adjoint":
        return state["plan"].adjoint(state["W"], c["nrhs"], out=state["out"])
    if kind == "ordered":
        return state["ev"](state["W"])
    if kind == "gradient":
        Y = H.kernel_matvec(state["ev"], state["W"])
        loss = 0.5 * (Y - state["T"]).square().sum()
        return {"loss": loss.detach(), "gradient": torch.autograd.grad(loss, state["W"])[0]}
    if kind == "batch":
        return state["batch"].evaluate(state["W"], state["nrhs"], state["out"])
    if kind == "dropin":
        call = H.parHSSGEMM if state["cds"].is_hss else H.CBHGEMM
        call(state["cds"], state["W"], state["Y"], c["nrhs"], state["wskel"], state["uskel"])
        return state["Y"]
    K, _ = H.kernel_matrices(state["X"], state["kernel"], state["rows"], state["cols"])
    return H.batched_id(K, [(len(a), len(b)) for a, b in zip(state["rows"], state["cols"])], c["tol"], c["rank"])


def work(case):
    c = case
    if c["kind"] == "compress":
        m, k = 2 * c["cols"], c["rank"]
        qr = 4.0 * m * c["cols"] * k - 2.0 * k * k * (m + c["cols"]) + 4.0 / 3.0 * k ** 3
        return {"bytes": c["nodes"] * (3 * c["cols"] * c["d"] * 8 + k * c["cols"] * 8),
                "flops": c["nodes"] * (m * c["cols"] * 3.0 * c["d"] + qr + k * k * c["cols"])}
    total = {"bytes": 0, "flops": 0}
    for m in _members(c) if c["kind"] == "batch" else [c]:
        cds, _ = _matrix_of(m)
        # values of the matrix: FP64, or the two and three bf16 parts of the split modes
        near, far = (8, 8) if m["precision"] == "fp64" else (6, 6) if m["precision"] == "split_bf16_x6" else \
            (4, 6) if m["precision"] == "split_bf16_far6" else (4, 4)
        held = near * cds.D.size + far * cds.B.size + (8 if m["precision"] == "fp64" else 6) * cds.VT.size
        if c["kind"] == "gradient":
            total["bytes"] += 2 * held + 3 * 4 * m["n"] * m["nrhs"]
            total["flops"] += 2 * cds.flops(m["nrhs"])
        else:
            total["bytes"] += held + 2 * 8 * m["n"] * m["nrhs"]
            total["flops"] += cds.flops(m["nrhs"])
    return total


# ---- the same results in plain FP64 ------------------------------------------------------------

def _product(cds, pools, W, transposed=False):
    """K~ W (or K~^T W) in FP64, W and the result with rows in tree order."""
    D, B, VT = pools
    rows = [slice(int(a), int(b)) for a, b in zip(cds.leaf_lids_offset[:-1], cds.leaf_lids_offset[1:])]
    s, m = cds.slen.astype(int), cds.Ddim.astype(int)

    def block(pool, ofs, r, c):
        A = pool[int(ofs):int(ofs) + int(r) * int(c)].view(int(c), int(r))
        return A if transposed else A.t()

    w, u = [None] * cds.numnodes, [None] * cds.numnodes
    P = [None] * cds.numnodes
    for v in range(cds.numnodes - 1, 0, -1):
        l, r = cds.lchildren[v], cds.rchildren[v]
        k = m[cds.lm[v]] if l < 0 else s[l] + s[r]
        P[v] = VT[int(cds.VTptr[v]):int(cds.VTptr[v]) + int(s[v] * k)].view(int(k), int(s[v])).t()
        w[v] = P[v] @ (W[rows[cds.lm[v]]] if l < 0 else torch.cat([w[l], w[r]]))
        u[v] = torch.zeros_like(w[v])
    for k in range(len(cds.fpairx)):
        x, y = int(cds.fpairx[k]), int(cds.fpairy[k])
        to, of = (y, x) if transposed else (x, y)
        u[to] += block(B, cds.Bptr[k], s[x], s[y]) @ w[of]
    Y = torch.zeros_like(W)
    for k in range(len(cds.npairx)):
        x, y = int(cds.npairx[k]), int(cds.npairy[k])
        to, of = (y, x) if transposed else (x, y)
        Y[rows[to]] += block(D, cds.Dptr[k], m[x], m[y]) @ W[rows[of]]
    for v in range(1, cds.numnodes):
        t = P[v].t() @ u[v]
        if cds.lchildren[v] < 0:
            Y[rows[cds.lm[v]]] += t
        else:
            l, r = int(cds.lchildren[v]), int(cds.rchildren[v])
            u[l] += t[:s[l]]
            u[r] += t[s[l]:]
    return Y


def _unblock(cds, TW, r):
    return torch.cat([TW[int(a) * r:int(b) * r].view(r, int(b - a)).t()
                      for a, b in zip(cds.leaf_lids_offset[:-1], cds.leaf_lids_offset[1:])])


def _block(cds, W):
    return torch.cat([W[int(a):int(b)].t().reshape(-1)
                      for a, b in zip(cds.leaf_lids_offset[:-1], cds.leaf_lids_offset[1:])])


def _pivoted_id(A, tol, rank):
    """Projection of a column-pivoted QR, for a batch of equally sized matrices (b, m, n)."""
    b, m, n = A.shape
    A = A.clone()
    at = torch.arange(b, device=A.device)
    R, piv = torch.zeros(b, min(rank, m, n), n, dtype=A.dtype, device=A.device), []
    diag = []
    for k in range(R.shape[1]):
        q2 = A.square().sum(1)
        for p in piv:
            q2[at, p] = -1.0
        p = q2.argmax(1)
        q = A[at, :, p]
        nrm = q.norm(dim=1)
        q = q / nrm.clamp(min=1e-300)[:, None]
        R[:, k] = torch.einsum("bm,bmn->bn", q, A)
        A -= q[:, :, None] * R[:, k][:, None, :]
        piv.append(p)
        diag.append(nrm)
    diag, piv = torch.stack(diag, 1), torch.stack(piv, 1)
    out = []
    for i in range(b):
        low = torch.nonzero(diag[i] / diag[i, 0] < tol)
        k = max(1, int(low[0]) if len(low) else R.shape[1])
        pk = piv[i, :k]
        R11 = torch.triu(R[i, :k][:, pk])
        P = torch.linalg.solve_triangular(R11, R[i, :k], upper=True)
        P[:, pk] = torch.eye(k, dtype=A.dtype, device=A.device)
        out.append(P)
    return out


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "compress":
        Xh, rows, cols = _samples(c, seed)
        X = torch.as_tensor(Xh, device=DEV)
        P = []
        for a, b in zip(rows, cols):
            R, Q = X[torch.as_tensor(a, device=DEV)], X[torch.as_tensor(b, device=DEV)]
            d2 = sum((R[:, k, None] - Q[None, :, k]).square() for k in range(c["d"]))
            P += [(None, _pivoted_id(_kernel(d2, c["kernel"], c["h"])[None], c["tol"], c["rank"])[0])]
        return P
    if kind == "batch":
        out = []
        for i, m in enumerate(_members(c)):
            cds, pools = _matrix_of(m)
            W = _randn(seed * 64 + i, m["n"] * m["nrhs"], dtype=torch.float32).to(torch.float64)
            out.append(_block(cds, _product(cds, pools, _unblock(cds, W, m["nrhs"]))))
        return out
    cds, pools = _matrix_of(c)
    n, r = c["n"], c["nrhs"]
    perm = torch.as_tensor(cds.perm, device=DEV)
    if kind == "gradient":
        W = _randn(seed, n, r, dtype=torch.float32).to(torch.float64)
        T = _randn(seed + (1 << 32), n, r, dtype=torch.float32).to(torch.float64)
        E = _product(cds, pools, W[perm]) - T[perm]
        G = torch.empty_like(W)
        G[perm] = _product(cds, pools, E, transposed=True)
        return {"loss": 0.5 * E.square().sum(), "gradient": G}
    if kind == "ordered":
        Y = torch.empty(n, r, dtype=torch.float64, device=DEV)
        Y[perm] = _product(cds, pools, _randn(seed, n, r)[perm])
        return Y
    W = _randn(seed, n * r)
    Y = _block(cds, _product(cds, pools, _unblock(cds, W, r), transposed=kind == "adjoint"))
    return Y
