"""CPU: the task list of the FP64 launch (its host scheduler, through the test hook
``mxb_debug_f64_schedule``; no device needed), run here in claim order on sub-block arrays laid
out as the kernel's.

Every unit must find its inputs written by earlier units (the launch's waits then end), count
exactly the writers it waits for, stay inside the pools and buffers, and the list as a whole must
give the oracle's product, forward and transposed, whole and cut along K.
"""
import ctypes

import numpy as np
import pytest

import oracle as O
from matrox_ru_b200 import _lib, build, hgemm as H, structure as S

TASK = np.dtype([("out", "<i8"), ("item0", "<i4"), ("nitem", "<i4"), ("rows", "<i4"), ("r8", "<i4"), ("m8", "<i4"),
                 ("stages", "<i4"), ("sig", "<i4"), ("old_dep", "<i4"), ("old_need", "<i4"), ("piece_ctr", "<i4"),
                 ("piece", "<i4"), ("npiece", "<i4"), ("kind", "<i2"), ("beta", "<i2"), ("slot", "<i4")])
ITEM = np.dtype([("a_off", "<u8"), ("lda", "<i4"), ("k8", "<i4"), ("b_base", "<i8"), ("dep", "<i4"), ("need", "<i4"),
                 ("a_pool", "<i2"), ("trans", "<i2"), ("b_buf", "<i2"), ("pad", "<i2")])
Y, WSKEL, USKEL, TILE_W = 0, 1, 2, 3


@pytest.fixture(scope="module")
def lib():
    build.build()
    return _lib.load()


def schedule(lib, cds, adjoint, nrhs):
    keep = []
    desc = H.cds_desc(cds, keep)
    tasks, items = np.zeros(1 << 16, TASK), np.zeros(1 << 18, ITEM)
    counts = np.zeros(9, np.int64)
    rc = lib.mxb_debug_f64_schedule(ctypes.byref(desc), int(adjoint), nrhs, tasks.ctypes.data, tasks.size,
                                    items.ctypes.data, items.size, counts.ctypes.data)
    assert rc == 0, lib.mxb_last_error()
    return tasks[:counts[0]], items[:counts[1]], counts


def c8(n):
    return (int(n) + 7) // 8


def pools(cds, counts):
    """The CDS as 8 x 8 sub-blocks, in the layout's order."""
    out = [[], [], []]

    def add(q, A):
        m, k = c8(A.shape[0]), c8(A.shape[1])
        P = np.zeros((8 * m, 8 * k))
        P[:A.shape[0], :A.shape[1]] = A
        out[q] += [P[8 * i:8 * i + 8, 8 * j:8 * j + 8] for j in range(k) for i in range(m)]

    def block(pool, ofs, r, c):
        return pool[int(ofs):int(ofs) + int(r) * int(c)].reshape(int(r), int(c), order="F")

    for k in range(cds.ncount):
        add(0, block(cds.D, cds.Dptr[k], cds.Ddim[cds.npairx[k]], cds.Ddim[cds.npairy[k]]))
    for k in range(cds.fcount):
        add(1, block(cds.B, cds.Bptr[k], cds.slen[cds.fpairx[k]], cds.slen[cds.fpairy[k]]))
    for v in range(1, cds.numnodes):
        if cds.slen[v] == 0:
            continue
        l, r = cds.lchildren[v], cds.rchildren[v]
        if l < 0:
            add(2, block(cds.VT, cds.VTptr[v], cds.slen[v], cds.Ddim[cds.lm[v]]))
        else:
            P = block(cds.VT, cds.VTptr[v], cds.slen[v], cds.slen[l] + cds.slen[r])
            add(2, P[:, :cds.slen[l]])
            add(2, P[:, cds.slen[l]:])
    for q in range(3):
        assert len(out[q]) == counts[6 + q]
    return out


def execute(lib, cds, TW, r, adjoint):
    tasks, items, counts = schedule(lib, cds, adjoint, r)
    pool = pools(cds, counts)
    ncol, nctr, slots, bk8 = int(counts[4]), int(counts[2]), int(counts[3]), int(counts[5])
    nb = c8(r)
    rows8 = [sum(c8(m) for m in cds.Ddim), sum(c8(s) for s in cds.slen)]
    buf = [np.full((8 * rows8[0], 8 * nb), np.nan), np.full((8 * rows8[1], 8 * nb), np.nan),
           np.full((8 * rows8[1], 8 * nb), np.nan)]
    lo = cds.leaf_lids_offset
    W = [TW[int(lo[i]) * r:int(lo[i + 1]) * r].reshape(-1, r, order="F") for i in range(cds.nleaf)]
    out = [np.full((int(m), r), np.nan) for m in cds.Ddim]
    ctr = np.zeros((nctr, ncol), np.int64)
    partial, arrived = {}, {}
    for t in tasks:
        for col in range(ncol):
            a8, b8 = nb * col // ncol, nb * (col + 1) // ncol
            cs = slice(8 * a8, 8 * b8)
            assert 0 < b8 - a8 <= 8 and t["m8"] <= 8
            if t["kind"] == TILE_W:
                i = int(t["out"])
                tile = np.zeros((8 * c8(cds.Ddim[i]), 8 * nb))
                tile[:cds.Ddim[i], :r] = W[i]
                a, b = 8 * int(t["r8"]), 8 * int(t["r8"] + t["m8"])
                buf[0][8 * int(t["slot"]) + a:8 * int(t["slot"]) + b, cs] = tile[a:b, cs]
                ctr[t["sig"], col] += 4
                continue
            acc, stages = np.zeros((8 * t["m8"], 8 * (b8 - a8))), 0
            for it in items[t["item0"]:t["item0"] + t["nitem"]]:
                if it["dep"] >= 0:
                    assert ctr[it["dep"], col] == it["need"]  # written before, and counted in full
                stages += -(-int(it["k8"]) // bk8)
                src = pool[it["a_pool"]]
                for k in range(it["k8"]):
                    ofs = int(it["a_off"])
                    blk = [src[ofs + (t["r8"] + i) * it["lda"] + k].T if it["trans"] else
                           src[ofs + k * it["lda"] + t["r8"] + i] for i in range(t["m8"])]
                    b = int(it["b_base"]) + k
                    acc += np.concatenate(blk) @ buf[it["b_buf"]][8 * b:8 * b + 8, cs]
            assert stages == t["stages"]
            if t["npiece"] > 1:
                key = (int(t["piece_ctr"]), col)
                assert key[0] + 4 <= nctr and t["slot"] + t["npiece"] <= slots
                partial.setdefault(key, {})[int(t["piece"])] = acc
                arrived[key] = arrived.get(key, 0) + 1
                if arrived[key] < t["npiece"]:
                    continue
                acc = sum(partial[key][p] for p in range(int(t["npiece"])))
            if t["old_dep"] >= 0:
                assert ctr[t["old_dep"], col] == t["old_need"]
            if t["kind"] == Y:
                i, r0 = int(t["out"]), 8 * int(t["r8"])
                n = min(len(acc), int(cds.Ddim[i]) - r0)
                v = acc[:n, :max(0, min(8 * b8, r) - 8 * a8)]
                dst = out[i][r0:r0 + n, 8 * a8:min(8 * b8, r)]
                dst[:] = dst + v if t["beta"] == 1 else v
            else:
                r0 = 8 * (int(t["out"]) + int(t["r8"]))
                dst = buf[t["kind"]][r0:r0 + len(acc), cs]
                assert dst.shape == acc.shape
                dst[:] = dst + acc if t["beta"] == 1 else acc
            if t["sig"] >= 0:
                ctr[t["sig"], col] += 4
    return np.concatenate([o.reshape(-1, order="F") for o in out]), tasks


def cases(small):
    yield from small.items()
    X = S.gaussian_mixture(1500, 3, 3, 0.0, 2.0, 0.3, None, seed=5)  # tall leaves: several row tiles, K pieces
    yield "tall", S.build_cds(X, S.KernelSpec("gaussian", 0.4), leaf_size=200, budget=0.9, tol=1e-7, max_rank=150)


@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("r", [1, 9, 30, 65, 130])
def test_schedule_gives_the_product(lib, small_cases, r, adjoint):
    cut = 0
    for name, cds in cases(small_cases):
        TW = np.random.default_rng(r).standard_normal(cds.n * r)
        got, tasks = execute(lib, cds, TW, r, adjoint)
        want = O.adjoint(cds, TW, r) if adjoint else O.eval_h2b(cds, TW, r)
        assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max(), name
        cut += int((tasks["npiece"] > 1).sum())
    assert cut > 0  # some sum was cut along K


@pytest.mark.parametrize("adjoint", [False, True])
def test_schedule_of_many_tiles(lib, small_cases, adjoint):
    """So many columns that far and down products, and near and leaf down products, are one sum: each
    Y and each skeleton block is written once."""
    r = 13000
    cds = small_cases["ragged"]
    TW = np.random.default_rng(r).standard_normal(cds.n * r)
    got, tasks = execute(lib, cds, TW, r, adjoint)
    want = O.adjoint(cds, TW, r) if adjoint else O.eval_h2b(cds, TW, r)
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
    assert (tasks["old_dep"] == -1).all() and (tasks["beta"] != 1).all()
    few = schedule(lib, cds, adjoint, 100)[0]
    assert (few["beta"] == 1).any() and len(few) > len(tasks)
