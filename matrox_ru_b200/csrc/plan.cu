// Plan: validated structure, creation, and the calls that FP64 (f64_engine.cu) and split-BF16
// (split_bf16.cu) plans share; and the launch-per-pass task lists that mxb_evaluate_noalloc runs.
// Schedule of one such evaluation (the reference runs the same four phases,
// symGen/HGEMM_gen.h:125-236, but as thousands of separate DGEMM calls):
//   1. leaf up        wskel[v] = P_v W[leaf v]                          (one launch)
//   2. transfer up    wskel[v] = P_v [wskel[l]; wskel[r]]    one launch per height, bottom-up
//   3. far + down     uskel[c] = sum_y B_cy wskel[y] + P_p[:, c]^T uskel[p]
//                                                            one launch per depth, top-down
//   4. near + leaf down  Y[x] (+)= sum_y D_xy W[y] + P_x^T uskel[x]        (one launch)
// Phase 3 fuses the far coupling with the downward transfer and phase 4 fuses the near
// field with the leaf projection, so each skeleton block and each Y block is written
// exactly once per evaluation.  The adjoint reuses phases 1-2 on G and runs phases 3-4
// with every near block and far coupling transposed.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>
#include <numeric>
#include <string>
#include <vector>

#include "matrox_b200.h"
#include "mxb_internal.h"
#include "f64_engine.h"
#include "plan.h"

namespace mxb {

namespace {
thread_local std::string g_last_error;
}

void set_error(const std::string &msg) { g_last_error = msg; }
const char *last_error() { return g_last_error.c_str(); }

#define MXB_CUDA(call)                                                                    \
    do {                                                                                  \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess) {                                                          \
            set_error(std::string(#call) + ": " + cudaGetErrorString(e_));                \
            return MXB_ERR_CUDA;                                                          \
        }                                                                                 \
    } while (0)

Plan::~Plan()
{
    clear_graphs();
    f64_destroy(*this);
    free_split_bf16();
    for (void *p : allocations) cudaFree(p);
}

int Plan::alloc(void **p, size_t bytes)
{
    if (bytes == 0) bytes = 16;
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) {
        *p = nullptr;
        (void)cudaGetLastError();  // not for the check behind the next launch
        set_error(std::string("cudaMalloc(") + std::to_string(bytes) + "): " + cudaGetErrorString(e));
        return e == cudaErrorMemoryAllocation ? MXB_ERR_NOMEM : MXB_ERR_CUDA;
    }
    allocations.push_back(*p);
    device_bytes += bytes;
    return MXB_OK;
}

void Plan::release(void *q, size_t bytes)
{
    if (!q || recorded) return;
    cudaFree(q);
    allocations.erase(std::remove(allocations.begin(), allocations.end(), q), allocations.end());
    device_bytes -= std::max<size_t>(bytes, 16);
}

void Plan::record()
{
    recorded = true;
    for (int slot = 0; slot < 2; ++slot) {
        if (ofs[slot] != &ofs_own[slot]) continue;
        ofs_kept.push_back(std::move(ofs_own[slot]));
        ofs_own[slot] = Offsets{};
        ofs[slot] = &ofs_kept.back();
    }
}

int is_capturing(cudaStream_t stream, bool *yes)
{
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    MXB_CUDA(cudaStreamIsCapturing(stream, &st));
    *yes = st != cudaStreamCaptureStatusNone;
    return MXB_OK;
}

int refuse_unprepared()
{
    set_error("the first evaluation of a column count, direction or layout cannot be captured: evaluate it once before");
    return MXB_ERR_UNSUPPORTED;
}

// ---------------------------------------------------------------------------------------
// validation of the host structure
// ---------------------------------------------------------------------------------------

static int fail(const std::string &m)
{
    set_error(m);
    return MXB_ERR_STRUCTURE;
}

static int arg_fail(const std::string &m)
{
    set_error(m);
    return MXB_ERR_ARG;
}

int Plan::validate(const mxb_cds_desc &d)
{
    if (d.nleaf < 1 || d.numnodes < 1 || d.ncount < 0 || d.fcount < 0) {
        set_error("nleaf, numnodes must be >= 1 and pair counts >= 0");
        return MXB_ERR_ARG;
    }
    if (!d.D || !d.Dptr || !d.lchildren || !d.rchildren || !d.lm || !d.slen || !d.Ddim ||
        (d.ncount && (!d.npairx || !d.npairy)) || (d.fcount && (!d.fpairx || !d.fpairy || !d.B || !d.Bptr)) ||
        (d.numnodes > 1 && (!d.VT || !d.VTptr))) {
        set_error("null array in CDS description");
        return MXB_ERR_ARG;
    }
    nleaf = d.nleaf;
    numnodes = d.numnodes;
    is_hss = d.is_hss;
    Ddim.assign(d.Ddim, d.Ddim + nleaf);
    slen.assign(d.slen, d.slen + numnodes);
    lch.assign(d.lchildren, d.lchildren + numnodes);
    rch.assign(d.rchildren, d.rchildren + numnodes);
    lm.assign(d.lm, d.lm + numnodes);
    parent.assign(numnodes, -1);
    for (int i = 0; i < nleaf; ++i)
        if (Ddim[i] < 1) return fail("Ddim[" + std::to_string(i) + "] < 1");
    std::vector<int> leafseen(nleaf, 0);
    for (int v = 0; v < numnodes; ++v) {
        if (slen[v] < 0) return fail("negative rank at node " + std::to_string(v));
        const int l = lch[v], r = rch[v];
        if ((l == -1) != (r == -1)) return fail("node " + std::to_string(v) + " has one child");
        if (l == -1) {
            if (lm[v] < 0 || lm[v] >= nleaf) return fail("leaf " + std::to_string(v) + " has no leaf index");
            if (leafseen[lm[v]]++) return fail("leaf index used twice");
        } else {
            if (l < 0 || l >= numnodes || r < 0 || r >= numnodes || l == r || l == v || r == v)
                return fail("child index out of range at node " + std::to_string(v));
            if (parent[l] != -1 || parent[r] != -1) return fail("node with two parents");
            parent[l] = v;
            parent[r] = v;
        }
    }
    for (int i = 0; i < nleaf; ++i)
        if (!leafseen[i]) return fail("leaf index " + std::to_string(i) + " unused");
    root = -1;
    for (int v = 0; v < numnodes; ++v)
        if (parent[v] == -1) {
            if (root != -1) return fail("more than one root");
            root = v;
        }
    if (root == -1) return fail("no root");
    // depth (from root) and height (from leaves); detects cycles by counting visits
    depth.assign(numnodes, -1);
    height.assign(numnodes, 0);
    std::vector<int> order;
    order.reserve(numnodes);
    order.push_back(root);
    depth[root] = 0;
    for (size_t i = 0; i < order.size(); ++i) {
        const int v = order[i];
        if (lch[v] != -1) {
            for (int c : {lch[v], rch[v]}) {
                if (depth[c] != -1) return fail("cycle in tree");
                depth[c] = depth[v] + 1;
                order.push_back(c);
            }
        }
    }
    if ((int)order.size() != numnodes) return fail("tree does not span all nodes");
    for (int i = numnodes - 1; i >= 0; --i) {
        const int v = order[i];
        if (lch[v] != -1) height[v] = 1 + std::max(height[lch[v]], height[rch[v]]);
    }
    bfs = order;

    // ranks of leaves may not exceed their sizes' usefulness but any s >= 0 is allowed;
    // check projection extents
    VT_len = d.VT_len;
    for (int v = 0; v < numnodes; ++v) {
        if (v == root || slen[v] == 0) continue;
        const uint64_t cols = (lch[v] == -1) ? (uint64_t)Ddim[lm[v]] : (uint64_t)slen[lch[v]] + slen[rch[v]];
        if (d.VTptr[v] < 0 || (uint64_t)d.VTptr[v] + (uint64_t)slen[v] * cols > d.VT_len)
            return fail("projection of node " + std::to_string(v) + " exceeds VT");
    }
    if (slen[root] != 0 && lch[root] != -1) {
        // the reference never projects the root (cacheSkeldim starts at node 1)
    }
    VTptr.assign(d.VTptr ? d.VTptr : nullptr, d.VTptr ? d.VTptr + numnodes : nullptr);
    if (VTptr.empty()) VTptr.assign(numnodes, 0);

    near_x.assign(d.npairx, d.npairx + d.ncount);
    near_y.assign(d.npairy, d.npairy + d.ncount);
    near_off.assign(d.Dptr, d.Dptr + d.ncount);
    for (int k = 0; k < d.ncount; ++k) {
        const int x = near_x[k], y = near_y[k];
        if (x < 0 || x >= nleaf || y < 0 || y >= nleaf) return fail("near pair out of range");
        if (near_off[k] + (uint64_t)Ddim[x] * Ddim[y] > d.D_len) return fail("near block exceeds D");
    }
    far_x.assign(d.fpairx, d.fpairx + d.fcount);
    far_y.assign(d.fpairy, d.fpairy + d.fcount);
    far_off.assign(d.Bptr, d.Bptr + d.fcount);
    for (int k = 0; k < d.fcount; ++k) {
        const int x = far_x[k], y = far_y[k];
        if (x < 0 || x >= numnodes || y < 0 || y >= numnodes) return fail("far pair out of range");
        if (x == root || y == root) {
            if (slen[root] != 0) return fail("far pair touches the root");
        }
        if (far_off[k] + (uint64_t)slen[x] * slen[y] > d.B_len) return fail("far block exceeds B");
    }
    D_len = d.D_len;
    B_len = d.B_len;
    rows_total = 0;
    leaf_row.resize(nleaf);
    for (int i = 0; i < nleaf; ++i) {
        leaf_row[i] = rows_total;
        rows_total += Ddim[i];
    }
    skel_row.assign(numnodes, 0);
    skel_total = 0;
    for (int v : bfs) {
        skel_row[v] = skel_total;
        skel_total += slen[v];
    }
    return MXB_OK;
}

// ---------------------------------------------------------------------------------------
// task lists
// ---------------------------------------------------------------------------------------

void Plan::add_task(std::vector<Task> &tasks, int16_t c_kind, int64_t c_row, int ldc, int M,
                    int item0, int nitem, int16_t beta, int tile)
{
    for (int m0 = 0; m0 < M; m0 += tile) {
        Task t{};
        t.c_row = c_row;
        t.ldc = ldc;
        t.M = M;
        t.m0 = m0;
        t.item0 = item0;
        t.nitem = nitem;
        t.c_kind = c_kind;
        t.beta = beta;
        tasks.push_back(t);
    }
}

static Item make_item(int16_t pool, uint64_t a_off, int lda, int K, int trans, int16_t b_kind,
                      int64_t b_row, int ldb)
{
    Item it{};
    it.a_pool = pool;
    it.a_off = a_off;
    it.lda = lda;
    it.K = K;
    it.trans = (int16_t)trans;
    it.b_kind = b_kind;
    it.b_row = b_row;
    it.ldb = ldb;
    return it;
}

void Plan::build_tasks(int tile)
{
    items.clear();
    tasks.clear();
    launches_fwd.clear();
    launches_adj.clear();
    auto begin_launch = [&](std::vector<Launch> &L, int kind, int level) {
        Launch l{};
        l.task0 = (int)tasks.size();
        l.kind = kind;
        l.level = level;
        L.push_back(l);
    };
    auto end_launch = [&](std::vector<Launch> &L) {
        L.back().ntasks = (int)tasks.size() - L.back().task0;
        if (L.back().ntasks == 0) {
            L.pop_back();
            return;
        }
        // longest tasks first: the CTAs of a launch start in task order, so the last wave holds
        // the shortest tasks (each task owns its output tile, so the order changes no result)
        auto cost = [&](const Task &t) {
            int64_t k = 0;
            for (int q = t.item0; q < t.item0 + t.nitem; ++q) k += items[q].K;
            return k;
        };
        std::stable_sort(tasks.begin() + L.back().task0, tasks.end(),
                         [&](const Task &a, const Task &b) { return cost(a) > cost(b); });
    };
    // per-node far lists (forward: pairs (c, y) for output c; adjoint: pairs (x, c))
    std::vector<std::vector<int>> far_out(numnodes), far_in(numnodes);
    for (size_t k = 0; k < far_x.size(); ++k) {
        far_out[far_x[k]].push_back((int)k);
        far_in[far_y[k]].push_back((int)k);
    }
    std::vector<std::vector<int>> near_out(nleaf), near_in(nleaf);
    for (size_t k = 0; k < near_x.size(); ++k) {
        near_out[near_x[k]].push_back((int)k);
        near_in[near_y[k]].push_back((int)k);
    }
    int maxh = 0, maxd = 0;
    for (int v = 0; v < numnodes; ++v) {
        maxh = std::max(maxh, height[v]);
        maxd = std::max(maxd, depth[v]);
    }
    auto projects = [&](int v) { return v != root && slen[v] > 0; };

    // phases 1-2: up-sweep, shared by forward and adjoint
    std::vector<Launch> up;
    for (int h = 0; h <= maxh; ++h) {
        begin_launch(up, MXB_PHASE_UP, h);
        for (int v : bfs) {
            if (height[v] != h || !projects(v)) continue;
            const int s = slen[v];
            const int item0 = (int)items.size();
            if (lch[v] == -1) {
                const int leaf = lm[v];
                items.push_back(make_item(2, (uint64_t)VTptr[v], s, Ddim[leaf], 0, KIND_W, leaf, Ddim[leaf]));
            } else {
                const int l = lch[v], r = rch[v];
                if (slen[l] > 0)
                    items.push_back(make_item(2, (uint64_t)VTptr[v], s, slen[l], 0, KIND_WSKEL, skel_row[l], slen[l]));
                if (slen[r] > 0)
                    items.push_back(make_item(2, (uint64_t)VTptr[v] + (uint64_t)s * slen[l], s, slen[r], 0,
                                              KIND_WSKEL, skel_row[r], slen[r]));
            }
            add_task(tasks, KIND_WSKEL, skel_row[v], s, s, item0, (int)items.size() - item0, 0, tile);
        }
        end_launch(up);
    }
    launches_fwd = up;
    launches_adj = up;

    // phase 3: far + down, top-down by depth
    auto down_item = [&](int c) -> bool {
        const int p = parent[c];
        if (p < 0 || !projects(p) || slen[c] == 0) return false;
        const uint64_t off = (uint64_t)VTptr[p] + (c == rch[p] ? (uint64_t)slen[p] * slen[lch[p]] : 0);
        items.push_back(make_item(2, off, slen[p], slen[p], 1, KIND_USKEL, skel_row[p], slen[p]));
        return true;
    };
    for (int adj = 0; adj < 2; ++adj) {
        std::vector<Launch> &L = adj ? launches_adj : launches_fwd;
        for (int dd = 1; dd <= maxd; ++dd) {
            begin_launch(L, MXB_PHASE_FAR_DOWN, dd);
            for (int c : bfs) {
                if (depth[c] != dd || !projects(c)) continue;
                const int item0 = (int)items.size();
                if (!adj) {
                    for (int k : far_out[c]) {
                        const int y = far_y[k];
                        if (slen[y] == 0) continue;
                        items.push_back(make_item(1, far_off[k], slen[c], slen[y], 0, KIND_WSKEL, skel_row[y], slen[y]));
                    }
                } else {
                    for (int k : far_in[c]) {
                        const int x = far_x[k];
                        if (slen[x] == 0) continue;
                        items.push_back(make_item(1, far_off[k], slen[x], slen[x], 1, KIND_WSKEL, skel_row[x], slen[x]));
                    }
                }
                down_item(c);
                add_task(tasks, KIND_USKEL, skel_row[c], slen[c], slen[c], item0, (int)items.size() - item0, 0, tile);
            }
            end_launch(L);
        }
        // phase 4: near + leaf down
        begin_launch(L, MXB_PHASE_NEAR_LEAF_DOWN, 0);
        for (int v : bfs) {
            if (lch[v] != -1) continue;
            const int x = lm[v];
            const int item0 = (int)items.size();
            if (!adj) {
                for (int k : near_out[x]) {
                    const int y = near_y[k];
                    items.push_back(make_item(0, near_off[k], Ddim[x], Ddim[y], 0, KIND_W, y, Ddim[y]));
                }
            } else {
                for (int k : near_in[x]) {
                    const int xx = near_x[k];
                    items.push_back(make_item(0, near_off[k], Ddim[xx], Ddim[xx], 1, KIND_W, xx, Ddim[xx]));
                }
            }
            if (projects(v)) items.push_back(make_item(2, (uint64_t)VTptr[v], slen[v], slen[v], 1, KIND_USKEL, skel_row[v], slen[v]));
            add_task(tasks, KIND_Y, x, Ddim[x], Ddim[x], item0, (int)items.size() - item0, 2, tile);
        }
        end_launch(L);
    }
}

uint64_t Plan::flops(int nrhs) const
{
    uint64_t f = 0;
    for (int v = 0; v < numnodes; ++v) {
        if (v == root) continue;
        const uint64_t s = (uint64_t)slen[v];
        if (lch[v] == -1) f += 2 * s * nrhs * (uint64_t)Ddim[lm[v]];
        else f += 2 * s * ((uint64_t)slen[lch[v]] + slen[rch[v]]) * nrhs;
    }
    f *= 2;
    for (size_t k = 0; k < near_x.size(); ++k) f += 2ull * Ddim[near_x[k]] * Ddim[near_y[k]] * nrhs;
    for (size_t k = 0; k < far_x.size(); ++k) f += 2ull * slen[far_x[k]] * slen[far_y[k]] * nrhs;
    return f;
}

// ---------------------------------------------------------------------------------------
// creation, scratch, evaluation
// ---------------------------------------------------------------------------------------

int Plan::create(const mxb_cds_desc &d, int prec, Plan **out)
{
    const int flags = prec & ~0xFF;
    prec &= 0xFF;
    if (prec < MXB_PREC_FP64 || prec > MXB_PREC_SPLIT_BF16_X6 || (flags & ~MXB_PLAN_ADJOINT)) {
        set_error("unknown precision mode");
        return MXB_ERR_ARG;
    }
    std::unique_ptr<Plan> p(new Plan());
    p->precision = prec;
    p->want_adjoint = (flags & MXB_PLAN_ADJOINT) && prec != MXB_PREC_FP64;  // FP64 plans always have it
    MXB_CUDA(cudaGetDevice(&p->device));
    int rc = p->validate(d);
    if (rc) return rc;
    if (prec == MXB_PREC_FP64) {
        rc = f64_create(*p, d.D, d.B, d.VT);
        if (rc) return rc;
    } else {
        // FP64 CDS for the tiling (host or device arrays: cudaMemcpyDefault follows the pointers)
        rc = p->alloc((void **)&p->dD, std::max<uint64_t>(d.D_len, 1) * sizeof(double));
        if (rc) return rc;
        MXB_CUDA(cudaMemcpy(p->dD, d.D, d.D_len * sizeof(double), cudaMemcpyDefault));
        rc = p->alloc((void **)&p->dB, std::max<uint64_t>(d.B_len, 1) * sizeof(double));
        if (rc) return rc;
        if (d.B_len) MXB_CUDA(cudaMemcpy(p->dB, d.B, d.B_len * sizeof(double), cudaMemcpyDefault));
        rc = p->alloc((void **)&p->dVT, std::max<uint64_t>(d.VT_len, 1) * sizeof(double));
        if (rc) return rc;
        if (d.VT_len) MXB_CUDA(cudaMemcpy(p->dVT, d.VT, d.VT_len * sizeof(double), cudaMemcpyDefault));
    }
    rc = p->alloc((void **)&p->ofs_own[0].dev, 2 * (size_t)p->nleaf * sizeof(int32_t));
    if (rc) return rc;
    p->ofs_own[1].dev = p->ofs_own[0].dev + p->nleaf;
    if (prec != MXB_PREC_FP64) {
        rc = p->setup_split_bf16(d);
        if (rc) return rc;
    }
    // The uploads above are synchronous copies from pageable memory, which may return before
    // their DMA has landed; the evaluations that follow run on the caller's streams, which do
    // not wait for the legacy stream.  Wait for every copy here.
    MXB_CUDA(cudaDeviceSynchronize());
    *out = p.release();
    return MXB_OK;
}

void Plan::clear_graphs() { clear_split_graphs(); }

// Per-leaf offsets for one call; packed offsets when the caller passes none.
int Plan::stage_offsets(int slot, const int32_t *given, int nrhs, cudaStream_t stream)
{
    std::vector<int32_t> want(nleaf);
    if (given) {
        std::memcpy(want.data(), given, sizeof(int32_t) * nleaf);
        for (int i = 0; i < nleaf; ++i)
            if (want[i] < 0) return fail("negative leaf offset");
    } else {
        for (int i = 0; i < nleaf; ++i) {
            const int64_t o = leaf_row[i] * (int64_t)nrhs;
            if (o > INT32_MAX) return fail("packed leaf offsets overflow int32");
            want[i] = (int32_t)o;
        }
    }
    if (ofs[slot] && ofs[slot]->host == want) return MXB_OK;
    for (const Offsets &k : ofs_kept)
        if (k.host == want) {
            ofs[slot] = &k;
            return MXB_OK;
        }
    Offsets &own = ofs_own[slot];
    if (own.host != want) {
        bool capturing = false;
        int rc = is_capturing(stream, &capturing);
        if (rc) return rc;
        if (capturing) return refuse_unprepared();
        if (!own.dev) {
            rc = alloc((void **)&own.dev, sizeof(int32_t) * nleaf);
            if (rc) return rc;
        }
        own.host = std::move(want);
        MXB_CUDA(cudaMemcpyAsync(own.dev, own.host.data(), sizeof(int32_t) * nleaf, cudaMemcpyHostToDevice, stream));
        MXB_CUDA(cudaStreamSynchronize(stream));
    }
    ofs[slot] = &own;
    return MXB_OK;
}

int Plan::run(bool adjoint, const double *dW, double *dY, int nrhs, const int32_t *wofs, const int32_t *yofs,
              int accumulate, cudaStream_t stream)
{
    if (nrhs < 1) {
        set_error("nrhs must be >= 1");
        return MXB_ERR_ARG;
    }
    if (!dW || !dY) {
        set_error("null device operand");
        return MXB_ERR_ARG;
    }
    int cur = -1;
    MXB_CUDA(cudaGetDevice(&cur));
    if (cur != device) {
        set_error("plan used on a different device than it was created on");
        return MXB_ERR_ARG;
    }
    int rc = stage_offsets(0, wofs, nrhs, stream);
    if (rc) return rc;
    rc = stage_offsets(1, yofs, nrhs, stream);
    if (rc) return rc;
    if (precision != MXB_PREC_FP64) return run_split_bf16(adjoint, dW, dY, nrhs, accumulate, stream);
    return f64_evaluate(*this, adjoint, dW, dY, ofs[0]->dev, ofs[1]->dev, nrhs, accumulate, stream);
}

// The caller's point order: perm[t] is the row of W / Y holding tree position t (the `lids`
// order of matroxTest-V1/hcds.h:766-788).  Host or device array; checked to be a permutation.
int Plan::set_permutation(const int32_t *perm)
{
    if (!perm) return arg_fail("null permutation");
    const int64_t n = rows_total;
    std::vector<int32_t> h((size_t)n + nleaf + 1);
    MXB_CUDA(cudaMemcpy(h.data(), perm, sizeof(int32_t) * (size_t)n, cudaMemcpyDefault));
    std::vector<char> seen((size_t)n, 0);
    for (int64_t t = 0; t < n; ++t) {
        const int32_t q = h[(size_t)t];
        if (q < 0 || q >= n || seen[(size_t)q]) return arg_fail("perm is not a permutation of the plan's rows");
        seen[(size_t)q] = 1;
    }
    for (int i = 0; i <= nleaf; ++i) h[(size_t)n + i] = (int32_t)(i < nleaf ? leaf_row[i] : n);
    if (!dTree) {
        int rc = alloc((void **)&dTree, h.size() * sizeof(int32_t));
        if (rc) return rc;
    }
    MXB_CUDA(cudaMemcpy(dTree, h.data(), h.size() * sizeof(int32_t), cudaMemcpyHostToDevice));
    MXB_CUDA(cudaDeviceSynchronize());  // a pageable upload may return before it lands
    return MXB_OK;
}

// dY (+)= K~ dW (or K~^T) with dW / dY in the caller's point order.  Split-BF16 plans gather
// W's rows inside the launch that splits W into operand tiles and scatter Y's rows in the
// epilogues that write Y: no extra pass over either matrix (the adjoint at N = 65536, 64 columns
// lost 21 us to each permutation).  FP64 plans permute into leaf-blocked copies, evaluate, and
// permute back.
int Plan::run_ordered(bool adjoint, const double *dW, int64_t w_rs, int64_t w_cs, double *dY, int64_t y_rs,
                      int64_t y_cs, int nrhs, int accumulate, cudaStream_t stream)
{
    if (!dTree) return arg_fail("no point order set (mxb_plan_set_permutation)");
    if (!dW || !dY || nrhs < 1) return arg_fail("bad caller-order operands");
    const int64_t n = rows_total;
    // distinct elements must not alias: one stride has to step over the whole other extent
    auto separated = [&](int64_t rs, int64_t cs) {
        return rs >= 1 && cs >= 1 && (rs >= (int64_t)nrhs * cs || cs >= n * rs);
    };
    if (!separated(w_rs, w_cs) || !separated(y_rs, y_cs)) return arg_fail("caller-order strides overlap");
    if (precision != MXB_PREC_FP64) {
        int cur = -1;
        MXB_CUDA(cudaGetDevice(&cur));
        if (cur != device) return arg_fail("plan used on a different device than it was created on");
        int rc = stage_offsets(0, nullptr, nrhs, stream);
        if (!rc) rc = stage_offsets(1, nullptr, nrhs, stream);
        if (rc) return rc;
        const CallerOrder o{dTree, dTree + n, w_rs, w_cs, y_rs, y_cs};
        return run_split_bf16(adjoint, dW, dY, nrhs, accumulate, stream, &o);
    }
    const size_t need = (size_t)std::max<int64_t>(n, 1) * nrhs;
    if (need > order_elems) {
        bool capturing = false;
        int rc = is_capturing(stream, &capturing);
        if (rc) return rc;
        if (capturing) return refuse_unprepared();
        for (double **q : {&dTW, &dTY}) {
            release(*q, order_elems * sizeof(double));
            *q = nullptr;
        }
        order_elems = 0;
        rc = alloc((void **)&dTW, need * sizeof(double));
        if (!rc) rc = alloc((void **)&dTY, need * sizeof(double));
        if (rc) return rc;
        order_elems = need;
    }
    int rc = stage_offsets(0, nullptr, nrhs, stream);  // packed blocks of the leaf-blocked copies
    if (rc) return rc;
    MXB_CUDA(launch_permute(dTree, dTree + n, ofs[0]->dev, nleaf, n, dW, dTW, w_rs, w_cs, nrhs, 0, 0, stream));
    rc = run(adjoint, dTW, dTY, nrhs, nullptr, nullptr, 0, stream);
    if (rc) return rc;
    MXB_CUDA(launch_permute(dTree, dTree + n, ofs[1]->dev, nleaf, n, dTY, dY, y_rs, y_cs, nrhs, 1, accumulate,
                            stream));
    return MXB_OK;
}

// Timing of the forward evaluation by launches and passes (mxb_plan_profile).
int Plan::profile(const double *dW, double *dY, int nrhs, cudaStream_t stream, mxb_op_profile *out, int cap,
                  int *nops)
{
    int rc = run(false, dW, dY, nrhs, nullptr, nullptr, 0, stream);  // checks, offsets, tuning
    if (rc) return rc;
    if (precision != MXB_PREC_FP64) return batch_profile(split_bf16_batch(*this), &dW, &dY, &nrhs, stream, out, cap, nops);
    return f64_profile(*this, dW, dY, ofs[0]->dev, ofs[1]->dev, nrhs, stream, out, cap, nops);
}

std::vector<float> pass_spans(const std::vector<unsigned long long> &ends)
{
    const int n = (int)ends.size() - 1;
    std::vector<float> ms(n, 0.f);
    if (ends[0] == ~0ull) return ms;
    std::vector<int> by(n);
    for (int k = 0; k < n; ++k) by[k] = k;
    std::stable_sort(by.begin(), by.end(), [&](int a, int b) { return ends[a + 1] < ends[b + 1]; });
    unsigned long long last = ends[0];
    for (int k : by) {
        if (!ends[k + 1]) continue;
        const unsigned long long end = std::max(ends[k + 1], last + 1);
        ms[k] = (float)((double)(end - last) * 1e-6);
        last = end;
    }
    return ms;
}

int Plan::read_workspaces(int nrhs, const int32_t *wsko, double *wskel, const int32_t *usko, double *uskel)
{
    if (precision != MXB_PREC_FP64) {
        set_error("skeleton workspaces are kept by FP64 plans only");
        return MXB_ERR_UNSUPPORTED;
    }
    std::vector<double> w, u;
    const int rc = f64_read_skeletons(*this, nrhs, w, u);
    if (rc) return rc;
    for (int v = 0; v < numnodes; ++v) {
        const size_t n = (size_t)slen[v] * nrhs;
        if (!n) continue;
        if (wskel && wsko) std::memcpy(wskel + wsko[v], w.data() + skel_row[v] * nrhs, n * sizeof(double));
        if (uskel && usko) std::memcpy(uskel + usko[v], u.data() + skel_row[v] * nrhs, n * sizeof(double));
    }
    return MXB_OK;
}

}  // namespace mxb
