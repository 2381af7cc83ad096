// Batched column interpolative decomposition (ID) on the GPU: the compression step of the
// CDS, matroxTest-V1/compression.h:446-523 `decomposition`, which the reference runs on the
// host per tree node with LAPACKE_dgeqp3 followed by cblas_dtrsm.
//
// Two kernels do it: a cluster of blocks per node (below), and, for ranks above 512, very tall nodes
// and levels of many small ones (choose_cluster), one CTA per node matrix A (nrows x ncols, column-major, nrows samples of the kernel against
// ncols candidate points), in place in global memory:
//   1. Householder QR with column pivoting.  The pivot of step i is the first column of
//      largest remaining norm; the norms are downdated after every step and recomputed where
//      the downdate has cancelled (LAPACK's dlaqp2 / dlaqps recurrence, tolerance
//      sqrt(machine epsilon)).
//   2. The reference's rank rule: s is the first s >= 1 with |R[s,s] / R[0,0]| < tol, at most
//      max_rank and at most min(nrows, ncols).  The QR stops there: only R[0:s, :] is needed.
//   3. P (s x ncols) with R11 P[:, piv] = R[0:s, :] by back substitution (upper triangular
//      R11), columns in parallel.  If R[0,0] == 0 (a zero matrix), P = 0: the reference then
//      returns R's upper rows, which are zero, without the solve.
// The factorisation is a sequence of rank-1 steps over the trailing matrix, each bound by
// the memory traffic of that matrix (L2 for a few nodes in flight, HBM beyond).
#include <algorithm>
#include <cfloat>
#include <climits>
#include <string>
#include <type_traits>
#include <vector>

#include "matrox_b200.h"
#include "mxb_internal.h"

namespace mxb {
namespace {

constexpr int MAX_COLS = 8192;  // shared memory holds 20 bytes per column

struct IdJob {
    uint64_t a_off;    // A: nrows x ncols, column-major (leading dimension nrows)
    uint64_t p_off;    // P and its scratch: pmax x ncols each, pmax = min(max_rank, ncols)
    uint64_t piv_off;  // ncols pivots
    int32_t nrows, ncols;
    int32_t panel, pad;  // columns per panel (cluster kernel)
};

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum over the block; every thread gets the result.  `red` holds WARPS + 1 doubles.
template <int THREADS>
__device__ double block_sum(double v, double *red)
{
    constexpr int WARPS = THREADS / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_sum(v);
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0) {
        double t = lane < WARPS ? red[lane] : 0.0;
        t = warp_sum(t);
        if (lane == 0) red[WARPS] = t;
    }
    __syncthreads();
    const double r = red[WARPS];
    __syncthreads();  // red is reused by the next call
    return r;
}

// First index of the largest value in x[lo, hi); every thread gets it.
template <int THREADS>
__device__ int block_argmax(const double *x, int lo, int hi, double *redv, int *redi)
{
    constexpr int WARPS = THREADS / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double bv = -1.0;
    int bi = hi;
    for (int j = lo + threadIdx.x; j < hi; j += THREADS)
        if (x[j] > bv) {  // ascending j per thread: the first of equal values stays
            bv = x[j];
            bi = j;
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) {
            bv = ov;
            bi = oi;
        }
    }
    if (lane == 0) {
        redv[warp] = bv;
        redi[warp] = bi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < WARPS; ++w)
            if (redv[w] > redv[0] || (redv[w] == redv[0] && redi[w] < redi[0])) {
                redv[0] = redv[w];
                redi[0] = redi[w];
            }
        redi[WARPS] = redi[0] < hi ? redi[0] : lo;
    }
    __syncthreads();
    const int r = redi[WARPS];
    __syncthreads();
    return r;
}

// THREADS: 256 when the launch has enough nodes to fill the GPU, 1024 (more warps on the
// trailing columns of one node) when it has fewer nodes than SMs.
template <int THREADS>
__global__ void __launch_bounds__(THREADS) id_qrcp_kernel(const IdJob *__restrict__ jobs, double *__restrict__ A,
                                                          double *__restrict__ P, double *__restrict__ Z,
                                                          int32_t *__restrict__ piv, int32_t *__restrict__ rank,
                                                          double tol, int max_rank)
{
    constexpr int WARPS = THREADS / 32;
    extern __shared__ double sm[];
    __shared__ double red[WARPS + 1];
    __shared__ int redi[WARPS + 1];
    __shared__ double s_beta, s_tau, s_scale;
    const IdJob jb = jobs[blockIdx.x];
    const int ns = jb.nrows, nc = jb.ncols;
    const int pmax = min(max_rank, nc);
    double *a = A + jb.a_off;
    double *vn1 = sm, *vn2 = sm + nc;
    int *jp = reinterpret_cast<int *>(sm + 2 * nc);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double tol3z = sqrt(DBL_EPSILON / 2);  // sqrt of LAPACK's relative machine epsilon

    // ---- column norms ----
    for (int j = warp; j < nc; j += WARPS) {
        const double *col = a + (size_t)j * ns;
        double t = 0.0;
        for (int r = lane; r < ns; r += 32) t += col[r] * col[r];
        t = warp_sum(t);
        if (lane == 0) vn1[j] = vn2[j] = sqrt(t);
    }
    for (int j = threadIdx.x; j < nc; j += THREADS) jp[j] = j;
    __syncthreads();

    // ---- pivoted Householder QR up to the rank ----
    const int kmax = min(ns, nc);
    int s = min(kmax, max_rank);
    double r00 = 0.0;
    for (int i = 0; i < kmax; ++i) {
        if (i >= max_rank) break;  // s = max_rank
        const int p = block_argmax<THREADS>(vn1, i, nc, red, redi);
        if (p != i) {
            double *ci = a + (size_t)i * ns, *cp = a + (size_t)p * ns;
            for (int r = threadIdx.x; r < ns; r += THREADS) {
                const double t = ci[r];
                ci[r] = cp[r];
                cp[r] = t;
            }
            if (threadIdx.x == 0) {
                const int tj = jp[i];
                jp[i] = jp[p];
                jp[p] = tj;
                vn1[p] = vn1[i];
                vn2[p] = vn2[i];
            }
        }
        __syncthreads();
        // reflector for a[i:, i] (dlarfg): beta = -sign(alpha) |x|, v = x[1:] / (alpha - beta)
        double *ci = a + (size_t)i * ns;
        double x2 = 0.0;
        for (int r = i + 1 + threadIdx.x; r < ns; r += THREADS) x2 += ci[r] * ci[r];
        x2 = block_sum<THREADS>(x2, red);
        if (threadIdx.x == 0) {
            const double alpha = ci[i];
            const double xnorm = sqrt(x2);
            if (xnorm == 0.0) {
                s_beta = alpha;
                s_tau = 0.0;
                s_scale = 0.0;
            } else {
                const double beta = -copysign(hypot(alpha, xnorm), alpha);
                s_beta = beta;
                s_tau = (beta - alpha) / beta;
                s_scale = 1.0 / (alpha - beta);
            }
        }
        __syncthreads();
        const double beta = s_beta, tau = s_tau, scale = s_scale;
        // the rank rule looks at R[i, i] = beta
        if (i == 0) {
            r00 = beta;
        } else if (r00 != 0.0 && fabs(beta / r00) < tol) {
            s = i;
            break;
        }
        if (tau != 0.0)
            for (int r = i + 1 + threadIdx.x; r < ns; r += THREADS) ci[r] *= scale;
        __syncthreads();
        if (threadIdx.x == 0) ci[i] = beta;
        // apply I - tau v v^T (v = [1; a[i+1:, i]]) to the columns right of i, one warp per
        // column, then downdate that column's norm
        for (int j = i + 1 + warp; j < nc; j += WARPS) {
            double *cj = a + (size_t)j * ns;
            double w = 0.0;
            if (tau != 0.0) {
                for (int r = i + 1 + lane; r < ns; r += 32) w += ci[r] * cj[r];
                w = warp_sum(w) + cj[i];
                w *= tau;
                for (int r = i + 1 + lane; r < ns; r += 32) cj[r] -= w * ci[r];
            }
            __syncwarp();
            double rij = cj[i];
            if (lane == 0 && tau != 0.0) {
                rij -= w;
                cj[i] = rij;
            }
            rij = __shfl_sync(0xffffffffu, rij, 0);
            const double v1 = vn1[j];
            bool recompute = false;
            if (v1 != 0.0) {
                double t = fabs(rij) / v1;
                t = fmax(0.0, (1.0 + t) * (1.0 - t));
                const double q = v1 / vn2[j];
                if (t * q * q <= tol3z) recompute = true;
                else if (lane == 0) vn1[j] = v1 * sqrt(t);
            }
            if (recompute) {  // uniform across the warp
                double t = 0.0;
                for (int r = i + 1 + lane; r < ns; r += 32) t += cj[r] * cj[r];
                t = warp_sum(t);
                if (lane == 0) vn1[j] = vn2[j] = i + 1 < ns ? sqrt(t) : 0.0;
            }
        }
        __syncthreads();
    }
    s = max(1, min(s, pmax));

    // ---- outputs: rank, pivots, P = R11^{-1} R[0:s, :] with columns in pivot order ----
    int32_t *pv = piv + jb.piv_off;
    for (int j = threadIdx.x; j < nc; j += THREADS) pv[j] = jp[j];
    if (threadIdx.x == 0) rank[blockIdx.x] = s;
    double *pout = P + jb.p_off;  // s x nc, leading dimension s
    if (r00 == 0.0) {
        for (int e = threadIdx.x; e < s * nc; e += THREADS) pout[e] = 0.0;
        return;
    }
    // z[k][j] (row-major, j fastest: coalesced across the threads) = R[k, j]
    double *z = Z + jb.p_off;
    for (int k = 0; k < s; ++k)
        for (int j = threadIdx.x; j < nc; j += THREADS)
            z[(size_t)k * nc + j] = (j >= k || j >= s) ? a[k + (size_t)j * ns] : 0.0;
    __syncthreads();
    // back substitution, all columns at once: x_k = z_k / R[k,k], then z_t -= x_k R[t,k], t < k
    for (int k = s - 1; k >= 0; --k) {
        const double *rk = a + (size_t)k * ns;  // column k of R11
        double *zk = z + (size_t)k * nc;
        for (int j = threadIdx.x; j < nc; j += THREADS) {
            const double x = zk[j] / rk[k];
            zk[j] = x;
            for (int t = 0; t < k; ++t) z[(size_t)t * nc + j] -= x * rk[t];
        }
    }
    __syncthreads();
    for (int k = 0; k < s; ++k)
        for (int j = threadIdx.x; j < nc; j += THREADS) pout[k + (size_t)jp[j] * s] = z[(size_t)k * nc + j];
}

// ---------------------------------------------------------------------------------------
// the cluster kernel
// ---------------------------------------------------------------------------------------
// A node is factored by a cluster of 1 - 8 blocks, each owning every C-th column.  Instead of
// applying every reflector to the whole trailing matrix (two reads and a write of it per
// column), columns stay as they were at the start of a panel: with the panel's orthonormal
// vectors q in shared memory, step i orthogonalises the pivot column against them (twice where it cancels), and
// row i of R is q_i^T A, one read of the trailing matrix.  Every PANEL columns (or when a norm
// downdate has cancelled, as LAPACK's dlaqps does) the panel is subtracted from the trailing
// columns in one pass.  R is the same as Householder's up to the signs of its rows, which
// P = R11^{-1} R does not depend on.
//
// Bound by the L2 reads of the trailing matrix (97 GB/s per SM, 7.5 us of a column's 15 us at
// 1024 x 512 with 4 blocks) and by the elections, reductions and barriers of each column (~6 us).
// One launch, one block per node -> this and id_solve_kernel: 32 nodes of 1024 x 512, rank 256,
// 46.5 -> 4.9 ms; 2 nodes 40.8 -> 3.1 ms; 32 of 512 x 256 13.0 -> 2.2 ms; 31 of 200 x 100, rank 50,
// 1.0 -> 0.8 ms.
constexpr int CL_THREADS = 512, CL_WARPS = CL_THREADS / 32, PANEL = 16, MAX_CLUSTER = 8;

struct Candidate {
    double norm;
    int32_t pos, col, flag, pad;
};

__device__ __forceinline__ uint32_t cluster_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_size()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(r));
    return r;
}
// every thread of the cluster; orders shared and global memory between its blocks
__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// Shared memory of the cluster kernel, in doubles, for ns rows, nc columns, C blocks and panels of nb.
__host__ __device__ inline size_t cl_smem_doubles(int ns, int nc, int C, int nb)
{
    const size_t ld = ((size_t)ns + 1) & ~size_t(1), nl = ((size_t)nc + C - 1) / C;
    return (size_t)nb * ld + ld                      // panel vectors, work vector
           + 2 * nl                                  // vn1, vn2
           + 2 * PANEL + CL_WARPS * PANEL * 4        // coefficients
           + 2 * CL_WARPS + 4                        // reductions
           + (size_t)CL_WARPS * 3 + 2 * MAX_CLUSTER * 3  // candidates: per warp, per block (two slots)
           + nl + (size_t)nc + 3;                    // active list and places in it, jp and pos
}

// acc[c] = sum over rows of q[r] * column c, c < W.
template <bool VEC, int W>
__device__ __forceinline__ void dots_of(const double *__restrict__ q, const double *const (&col)[4], int ns, int lane,
                                        double (&acc)[4])
{
#pragma unroll
    for (int c = 0; c < W; ++c) acc[c] = 0.0;
    if constexpr (VEC) {
        const int n2 = ns >> 1;
        int r = lane;
        for (; r + 96 < n2; r += 128) {  // 4 W loads of 16 bytes in flight
            double2 x[4][W];
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int c = 0; c < W; ++c) x[u][c] = __ldcg(reinterpret_cast<const double2 *>(col[c]) + r + 32 * u);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const double2 w = *(reinterpret_cast<const double2 *>(q) + r + 32 * u);
#pragma unroll
                for (int c = 0; c < W; ++c) acc[c] = fma(w.y, x[u][c].y, fma(w.x, x[u][c].x, acc[c]));
            }
        }
        for (; r < n2; r += 32) {
            const double2 w = *(reinterpret_cast<const double2 *>(q) + r);
#pragma unroll
            for (int c = 0; c < W; ++c) {
                const double2 x = __ldcg(reinterpret_cast<const double2 *>(col[c]) + r);
                acc[c] = fma(w.y, x.y, fma(w.x, x.x, acc[c]));
            }
        }
    } else {
        for (int r = lane; r < ns; r += 32) {
            const double w = q[r];
#pragma unroll
            for (int c = 0; c < W; ++c) acc[c] = fma(w, __ldcg(col[c] + r), acc[c]);
        }
    }
#pragma unroll
    for (int c = 0; c < W; ++c) acc[c] = warp_sum(acc[c]);
}

template <bool VEC>
__device__ __forceinline__ void dots_of(int width, const double *__restrict__ q, const double *const (&col)[4], int ns,
                                        int lane, double (&acc)[4])
{
    switch (width) {
    case 1: return dots_of<VEC, 1>(q, col, ns, lane, acc);
    case 2: return dots_of<VEC, 2>(q, col, ns, lane, acc);
    case 3: return dots_of<VEC, 3>(q, col, ns, lane, acc);
    default: return dots_of<VEC, 4>(q, col, ns, lane, acc);
    }
}

__global__ void __launch_bounds__(CL_THREADS, 1) id_cluster_kernel(const IdJob *__restrict__ jobs, double *__restrict__ A,
                                                                   double *__restrict__ Z, int32_t *__restrict__ piv,
                                                                   int32_t *__restrict__ rank, double tol, int max_rank)
{
    extern __shared__ __align__(16) double sm[];
    const uint32_t C = cluster_size(), me = cluster_rank();
    const IdJob jb = jobs[blockIdx.x / C];
    const int ns = jb.nrows, nc = jb.ncols, nb = jb.panel;
    const int pmax = min(max_rank, nc);
    const int ld = (ns + 1) & ~1, nl = (nc + (int)C - 1) / (int)C;
    double *a = A + jb.a_off;
    double *z = Z + jb.p_off;  // R, column-major: entry (k, j) at j * pmax + k
    double *Q = sm, *v = Q + (size_t)nb * ld, *vn1 = v + ld, *vn2 = vn1 + nl;
    double *coef = vn2 + nl, *dots = coef + PANEL, *wcoef = dots + PANEL, *red = wcoef + CL_WARPS * PANEL * 4;
    Candidate *wcand = reinterpret_cast<Candidate *>(red + 2 * CL_WARPS + 4), *ccand = wcand + CL_WARPS;
    int *act = reinterpret_cast<int *>(ccand + 2 * MAX_CLUSTER), *place = act + nl, *jp = place + nl, *pos = jp + nc;
    int *nact_s = pos + nc;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double tol3z = sqrt(DBL_EPSILON / 2);
    const bool vec = !(ns & 1) && !(reinterpret_cast<uintptr_t>(a) & 15);

    // own columns: j = me + C * l, l < count; l indexes vn1 and vn2
    const int count = (nc - (int)me + (int)C - 1) / (int)C;
    for (int j = tid; j < nc; j += CL_THREADS) jp[j] = pos[j] = j;
    for (int l = tid; l < count; l += CL_THREADS) act[l] = place[l] = l;
    if (tid == 0) *nact_s = count;
    for (int l = warp; l < count; l += CL_WARPS) {
        const double *col = a + (size_t)(me + C * l) * ns;
        double t = 0.0;
        for (int r = lane; r < ns; r += 32) t = fma(col[r], col[r], t);
        t = warp_sum(t);
        if (lane == 0) vn1[l] = vn2[l] = sqrt(t);
    }
    __syncthreads();
    if (C > 1) cluster_barrier();  // every block runs before another writes to its shared memory

    const int kmax = min(ns, nc);
    int s = min(kmax, max_rank), i0 = 0, slot = 0;
    double r00 = 0.0;
    bool flagged = false;  // some own column's norm has to be recomputed

    // best own column (largest norm, then first position) to every block; all blocks then agree
    auto better = [](double x, int p, const Candidate &o) { return x > o.norm || (x == o.norm && p < o.pos); };
    // the warp's best: norms are >= 0 where a candidate exists, so their bits order like integers
    auto warp_best = [&](Candidate &c) {
        const bool have = c.norm >= 0.0;
        const uint32_t hi = have ? (uint32_t)__double2hiint(c.norm) : 0u, lo = have ? (uint32_t)__double2loint(c.norm) : 0u;
        const uint32_t mh = __reduce_max_sync(0xffffffffu, hi);
        const uint32_t ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
        const bool top = have && hi == mh && lo == ml;
        const int p = __reduce_min_sync(0xffffffffu, top ? c.pos : INT_MAX);
        const unsigned who = __ballot_sync(0xffffffffu, top && c.pos == p);
        c.col = who ? __shfl_sync(0xffffffffu, c.col, __ffs(who) - 1) : -1;
        c.norm = who ? __hiloint2double((int)mh, (int)ml) : -1.0;
        c.pos = p;
    };
    auto elect = [&](bool flag) {
        Candidate c{-1.0, INT_MAX, -1, 0, 0};
        const int n = *nact_s;
        for (int t = tid; t < n; t += CL_THREADS) {
            const int l = act[t], j = (int)(me + C * l);
            const double x = vn1[l];
            if (x >= 0.0 && better(x, pos[j], c)) c.norm = x, c.pos = pos[j], c.col = j;
        }
        warp_best(c);
        if (lane == 0) wcand[warp] = c;
        __syncthreads();
        if (warp == 0) {
            c = lane < CL_WARPS ? wcand[lane] : Candidate{-1.0, INT_MAX, -1, 0, 0};
            warp_best(c);
            c.flag = flag ? 1 : 0;
            Candidate *dst = ccand + slot * MAX_CLUSTER + me;
            if (C == 1) {
                if (lane == 0) *dst = c;
            } else if (lane < (int)C) {
                uint32_t at;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(at)
                             : "r"((uint32_t)__cvta_generic_to_shared(dst)), "r"(lane));
                asm volatile("st.shared::cluster.f64 [%0], %1;\n" ::"r"(at), "d"(c.norm) : "memory");
                asm volatile("st.shared::cluster.v2.s32 [%0], {%1, %2};\n" ::"r"(at + 8), "r"(c.pos), "r"(c.col) : "memory");
                asm volatile("st.shared::cluster.s32 [%0], %1;\n" ::"r"(at + 16), "r"(c.flag) : "memory");
            }
        }
        if (C == 1) __syncthreads();
        else cluster_barrier();
        Candidate best = ccand[slot * MAX_CLUSTER];
        for (uint32_t b = 1; b < C; ++b) {
            const Candidate o = ccand[slot * MAX_CLUSTER + b];
            const int f = best.flag | o.flag;
            if (better(o.norm, o.pos, best)) best = o;
            best.flag = f;
        }
        slot ^= 1;
        return best;
    };
    // subtract the panel [i0, i1) from the own active columns; recompute flagged norms
    auto subtract_panel = [&](int i1) {
        const int kp = i1 - i0, n = *nact_s;
        double *wc = wcoef + warp * PANEL * 4;
        for (int t = warp * 4; t < n; t += CL_WARPS * 4) {
            double *col[4];
            int l[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                l[c] = act[min(t + c, n - 1)];
                col[c] = a + (size_t)(me + C * l[c]) * ns;
            }
            for (int e = lane; e < kp * 4; e += 32) {
                const int k = e >> 2, c = e & 3;
                wc[k * 4 + c] = t + c < n ? z[(size_t)(me + C * act[min(t + c, n - 1)]) * pmax + i0 + k] : 0.0;
            }
            __syncwarp();
            double sq[4] = {0.0, 0.0, 0.0, 0.0};
            auto rows = [&](auto rn, int r0) {  // rows r0, r0 + 32, ...: their loads in flight together
                constexpr int R = decltype(rn)::value;
                double x[R][4];
#pragma unroll
                for (int u = 0; u < R; ++u)
#pragma unroll
                    for (int c = 0; c < 4; ++c) x[u][c] = __ldcg(col[c] + r0 + 32 * u);
                for (int k = 0; k < kp; ++k) {
                    double f[4], w[R];
#pragma unroll
                    for (int c = 0; c < 4; ++c) f[c] = wc[k * 4 + c];
#pragma unroll
                    for (int u = 0; u < R; ++u) w[u] = Q[(size_t)k * ld + r0 + 32 * u];
#pragma unroll
                    for (int u = 0; u < R; ++u)
#pragma unroll
                        for (int c = 0; c < 4; ++c) x[u][c] = fma(-w[u], f[c], x[u][c]);
                }
#pragma unroll
                for (int u = 0; u < R; ++u)
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        if (t + c < n) col[c][r0 + 32 * u] = x[u][c];
                        sq[c] = fma(x[u][c], x[u][c], sq[c]);
                    }
            };
            int r = lane;
            for (; r + 96 < ns; r += 128) rows(std::integral_constant<int, 4>{}, r);
            for (; r < ns; r += 32) rows(std::integral_constant<int, 1>{}, r);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const double t2 = warp_sum(sq[c]);
                if (lane == 0 && t + c < n && vn1[l[c]] < 0.0) vn1[l[c]] = vn2[l[c]] = i1 < ns ? sqrt(t2) : 0.0;
            }
            __syncwarp();
        }
        __syncthreads();
        i0 = i1;
    };

    for (int i = 0; i < kmax && i < max_rank; ++i) {
        Candidate best = elect(flagged);
        if (best.flag || i - i0 >= nb) {
            subtract_panel(i);
            flagged = false;
            best = elect(false);
        }
        // the pivot, as a swap of columns i and best.pos of the permuted matrix
        const int p = best.col >= 0 ? best.col : jp[i], pp = best.col >= 0 ? best.pos : i;
        __syncthreads();  // jp[i] is read by all before it changes
        if (tid == 0) {
            const int q = jp[i];
            jp[i] = p;
            jp[pp] = q;
            pos[p] = i;
            pos[q] = pp;
            if (p % (int)C == (int)me) {  // no longer active
                const int n = *nact_s - 1, t = place[p / (int)C], l = act[n];
                act[t] = l;
                place[l] = t;
                *nact_s = n;
            }
        }
        // v = column p less its components along the panel, twice
        const int kp = i - i0;
        const double *ap = a + (size_t)p * ns, *zp = z + (size_t)p * pmax + i0;
        if (tid < kp) coef[tid] = __ldcg(zp + tid);
        for (int r = tid; r < ns; r += CL_THREADS) v[r] = __ldcg(ap + r);
        __syncthreads();
        // less its components c along the panel, and the square of what is left
        auto reduce_against = [&](const double *c) {
            double sq = 0.0;
            for (int r = tid; r < ns; r += CL_THREADS) {
                double x = v[r];
                for (int k = 0; k < kp; ++k) x = fma(-Q[(size_t)k * ld + r], c[k], x);
                v[r] = x;
                sq = fma(x, x, sq);
            }
            sq = warp_sum(sq);
            if (lane == 0) red[warp] = sq;
            __syncthreads();
            double t = 0.0;
#pragma unroll
            for (int w = 0; w < CL_WARPS; ++w) t += red[w];
            return t;
        };
        double left = reduce_against(coef);
        if (kp > 0) {
            double gone = 0.0;
            for (int k = 0; k < kp; ++k) gone = fma(coef[k], coef[k], gone);
            if (!(left > 0.0625 * gone)) {
                // more than 94 % of the column lay in the panel: what is left has lost digits, and a
                // second pass makes it orthogonal to the panel again
                for (int k = warp; k < kp; k += CL_WARPS) {
                    double t = 0.0;
                    for (int r = lane; r < ns; r += 32) t = fma(Q[(size_t)k * ld + r], v[r], t);
                    t = warp_sum(t);
                    if (lane == 0) dots[k] = t;
                }
                __syncthreads();
                left = reduce_against(dots);
            }
        }
        const double rii = sqrt(left);
        if (i == 0) {
            r00 = rii;
        } else if (r00 != 0.0 && rii / r00 < tol) {
            s = i;
            break;
        }
        double *q = Q + (size_t)kp * ld;
        const double inv = rii > 0.0 ? 1.0 / rii : 0.0;
        for (int r = tid; r < ns; r += CL_THREADS) q[r] = v[r] * inv;
        if (tid == 0 && me == 0) z[(size_t)p * pmax + i] = rii;
        __syncthreads();
        // row i of R over the own active columns, and their norms downdated
        const int n = *nact_s;
        bool flag = false;
        const int rounds = (n + 4 * CL_WARPS - 1) / (4 * CL_WARPS);
        const int width = n ? (n + CL_WARPS * rounds - 1) / (CL_WARPS * rounds) : 1;  // columns of a warp at a time
        for (int t = warp * width; t < n; t += CL_WARPS * width) {
            const double *col[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) col[c] = a + (size_t)(me + C * act[min(t + c, n - 1)]) * ns;
            double acc[4] = {0.0, 0.0, 0.0, 0.0};
            if (vec) dots_of<true>(width, q, col, ns, lane, acc);
            else dots_of<false>(width, q, col, ns, lane, acc);
            if (lane < width && t + lane < n) {
                const double rij = lane == 0 ? acc[0] : (lane == 1 ? acc[1] : (lane == 2 ? acc[2] : acc[3]));
                const int l = act[t + lane];
                z[(size_t)(me + C * l) * pmax + i] = rij;
                const double v1 = vn1[l];
                if (v1 != 0.0) {
                    double x = fabs(rij) / v1;
                    x = fmax(0.0, (1.0 + x) * (1.0 - x));
                    const double y = v1 / vn2[l];
                    if (x * y * y <= tol3z) {
                        vn1[l] = -1.0;
                        flag = true;
                    } else {
                        vn1[l] = v1 * sqrt(x);
                    }
                }
            }
        }
        flagged = __syncthreads_or(flag) != 0;
    }
    s = max(1, min(s, pmax));
    __syncthreads();
    if (me == 0) {
        int32_t *pv = piv + jb.piv_off;
        for (int j = tid; j < nc; j += CL_THREADS) pv[j] = jp[j];
        if (tid == 0) rank[blockIdx.x / C] = s;
    }
    if (C > 1) cluster_barrier();  // no block leaves while another may still write to its shared memory
}

// P = R11^{-1} R with columns at their places, from the cluster kernel's R: a warp solves four columns
// at a time, 32 rows of R11 per register.  NR: registers per column (s <= 32 NR).
template <int NR>
__device__ void solve_columns(const double *__restrict__ z, const int32_t *__restrict__ piv, const double *__restrict__ inv,
                              double *__restrict__ pout, int s, int nc, int pmax, int j0, int step, int lane)
{
    for (int q = s + 4 * j0; q < nc; q += 4 * step) {
        double x[4][NR];
        int col[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            col[c] = piv[min(q + c, nc - 1)];
#pragma unroll
            for (int u = 0; u < NR; ++u) {
                const int t = lane + 32 * u;
                x[c][u] = t < s ? z[(size_t)col[c] * pmax + t] : 0.0;
            }
        }
#pragma unroll
        for (int u = NR - 1; u >= 0; --u) {
            if (32 * u >= s) continue;
            for (int l = min(31, s - 1 - 32 * u); l >= 0; --l) {
                const int k = 32 * u + l;
                const double *rk = z + (size_t)piv[k] * pmax;  // column k of R11
                double r[NR];
#pragma unroll
                for (int w = 0; w <= u; ++w) r[w] = lane + 32 * w < k ? rk[lane + 32 * w] : 0.0;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const double xk = __shfl_sync(0xffffffffu, x[c][u], l) * inv[k];
                    if (lane == l) x[c][u] = xk;
#pragma unroll
                    for (int w = 0; w <= u; ++w) x[c][w] = fma(-xk, r[w], x[c][w]);
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (q + c < nc)
#pragma unroll
                for (int u = 0; u < NR; ++u) {
                    const int t = lane + 32 * u;
                    if (t < s) pout[(size_t)col[c] * s + t] = x[c][u];
                }
    }
}

constexpr int SOLVE_THREADS = 128, SOLVE_MAX = 512;  // largest rank of the cluster path

__global__ void __launch_bounds__(SOLVE_THREADS) id_solve_kernel(const IdJob *__restrict__ jobs, const double *__restrict__ Z,
                                                                 double *__restrict__ P, const int32_t *__restrict__ piv_all,
                                                                 const int32_t *__restrict__ rank, int max_rank)
{
    __shared__ double inv[SOLVE_MAX];
    const IdJob jb = jobs[blockIdx.x];
    const int nc = jb.ncols, pmax = min(max_rank, nc), s = rank[blockIdx.x];
    const double *z = Z + jb.p_off;
    double *pout = P + jb.p_off;
    const int32_t *piv = piv_all + jb.piv_off;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = SOLVE_THREADS / 32;
    const bool zero = z[(size_t)piv[0] * pmax] == 0.0;  // R[0, 0]
    for (int k = threadIdx.x; k < s; k += SOLVE_THREADS) inv[k] = 1.0 / z[(size_t)piv[k] * pmax + k];
    __syncthreads();
    const int w = blockIdx.y * warps + warp, nw = gridDim.y * warps;
    // skeleton columns: the identity (all zeros for a zero matrix)
    for (int k = w; k < (zero ? nc : s); k += nw)
        for (int t = lane; t < s; t += 32) pout[(size_t)piv[k] * s + t] = (!zero && t == k) ? 1.0 : 0.0;
    if (zero) return;
    if (s <= 64) solve_columns<2>(z, piv, inv, pout, s, nc, pmax, w, nw, lane);
    else if (s <= 128) solve_columns<4>(z, piv, inv, pout, s, nc, pmax, w, nw, lane);
    else if (s <= 256) solve_columns<8>(z, piv, inv, pout, s, nc, pmax, w, nw, lane);
    else solve_columns<16>(z, piv, inv, pout, s, nc, pmax, w, nw, lane);
}

void cluster_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute *attr, int count, int C, size_t smem, cudaStream_t s)
{
    cfg.gridDim = dim3((unsigned)(count * C), 1, 1);
    cfg.blockDim = dim3(CL_THREADS, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)C;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
}

// Blocks per node for the cluster kernel (0: it does not take these nodes), the nodes' panel widths
// and the shared memory: the most blocks for which every node's cluster is resident at once, each
// with at least 16 columns.  Ranks above SOLVE_MAX, and nodes so tall that shared memory holds
// fewer than 4 panel vectors (above ~5500 rows), stay with the kernel of one block per node.  So do
// levels of many small nodes, whose columns wait for one block's steps either way: that kernel's
// blocks are half as large and a step has fewer barriers.  Kernel of one block per node / this one:
// 256 threads and more nodes than SMs: 2048 nodes of 64 x 32 0.98 / 1.99 ms; 300 of 128 x 64 0.85 /
// 1.44, of 160 x 80 1.26 / 1.31, of 200 x 100 2.09 / 1.92; 1024 of 200 x 100 5.04 / 6.69, of 224 x 112
// 6.91 / 5.47; 256 of 512 x 256 34.9 / 7.0.
int choose_cluster(std::vector<IdJob> &jobs, int max_rank, int maxc, int sms, size_t &smem_doubles)
{
    constexpr size_t LIMIT = 225 * 1024 / sizeof(double);
    if (std::min(max_rank, maxc) > SOLVE_MAX) return 0;
    if (cudaFuncSetAttribute(id_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(LIMIT * sizeof(double))) !=
        cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    int64_t largest = 0;
    for (const IdJob &j : jobs) largest = std::max(largest, (int64_t)j.nrows * j.ncols);
    const int count = (int)jobs.size();
    const bool many_small = count >= sms && (largest <= 128 * 64 || (count > 3 * sms && largest <= 200 * 100));
    for (int C = MAX_CLUSTER; C >= 1; C >>= 1) {
        if (C > 1 && maxc < 16 * C) continue;
        smem_doubles = 0;
        bool fits = true;
        for (IdJob &j : jobs) {
            const size_t base = cl_smem_doubles(j.nrows, j.ncols, C, 0), ld = ((size_t)j.nrows + 1) & ~size_t(1);
            const size_t room = base < LIMIT ? (LIMIT - base) / ld : 0;
            j.panel = (int)std::min<size_t>(PANEL, room);
            fits = fits && j.panel >= std::min(4, std::min(j.nrows, j.ncols));
            smem_doubles = std::max(smem_doubles, cl_smem_doubles(j.nrows, j.ncols, C, j.panel));
        }
        if (!fits) continue;
        if (C == 1) return many_small ? 0 : 1;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        cluster_config(cfg, attr, count, C, smem_doubles * sizeof(double), nullptr);
        int resident = 0;
        if (cudaOccupancyMaxActiveClusters(&resident, id_cluster_kernel, &cfg) != cudaSuccess) {
            (void)cudaGetLastError();
            continue;
        }
        if (resident >= count) return C;
    }
    return 0;
}

int fail_id(const std::string &m, int code = MXB_ERR_ARG)
{
    set_error("mxb_batched_id: " + m);
    return code;
}

}  // namespace
}  // namespace mxb

using namespace mxb;

extern "C" int32_t mxb_batched_id(double *dA, const int32_t *nrows, const int32_t *ncols, int32_t count, double tol,
                                  int32_t max_rank, int32_t *dRank, int32_t *dPiv, double *dP, void *stream)
{
    if (count < 0) return fail_id("negative count");
    if (count == 0) return MXB_OK;
    if (!dA || !nrows || !ncols || !dRank || !dPiv || !dP) return fail_id("null argument");
    if (max_rank < 1) return fail_id("max_rank must be >= 1");
    if (!(tol >= 0.0)) return fail_id("tolerance must be >= 0");
    std::vector<IdJob> jobs((size_t)count);
    uint64_t a = 0, p = 0, q = 0;
    int maxc = 1;
    for (int b = 0; b < count; ++b) {
        const int ns = nrows[b], nc = ncols[b];
        if (ns < 1 || nc < 1) return fail_id("empty matrix");
        if (nc > MAX_COLS) return fail_id("more than " + std::to_string(MAX_COLS) + " columns", MXB_ERR_UNSUPPORTED);
        jobs[b] = IdJob{a, p, q, ns, nc, 0, 0};
        a += (uint64_t)ns * nc;
        p += (uint64_t)std::min(max_rank, nc) * nc;
        q += (uint64_t)nc;
        maxc = std::max(maxc, nc);
    }
    cudaStream_t s = (cudaStream_t)stream;
    int dev = 0, sms = 148;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    size_t cl_smem = 0;
    const int cluster = choose_cluster(jobs, max_rank, maxc, sms, cl_smem);
    IdJob *dJobs = nullptr;
    double *dZ = nullptr;
    if (e == cudaSuccess) e = cudaMallocAsync(&dJobs, jobs.size() * sizeof(IdJob), s);
    if (e == cudaSuccess) e = cudaMallocAsync(&dZ, std::max<uint64_t>(p, 1) * sizeof(double), s);
    if (cluster) {
        const size_t smem = cl_smem * sizeof(double);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(dJobs, jobs.data(), jobs.size() * sizeof(IdJob), cudaMemcpyHostToDevice, s);
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        cluster_config(cfg, attr, count, cluster, smem, s);
        if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, id_cluster_kernel, (const IdJob *)dJobs, dA, dZ, dPiv, dRank, tol, max_rank);
        if (e == cudaSuccess) {
            const unsigned groups = (unsigned)std::min(64, (maxc + 15) / 16);
            id_solve_kernel<<<dim3((unsigned)count, groups), SOLVE_THREADS, 0, s>>>(dJobs, dZ, dP, dPiv, dRank, max_rank);
            e = cudaGetLastError();
        }
    } else {
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(dJobs, jobs.data(), jobs.size() * sizeof(IdJob), cudaMemcpyHostToDevice, s);
        const size_t smem = (size_t)maxc * (2 * sizeof(double) + sizeof(int));
        const bool wide = count < sms;
        if (e == cudaSuccess)
            e = wide ? cudaFuncSetAttribute(id_qrcp_kernel<1024>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
                     : cudaFuncSetAttribute(id_qrcp_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess) {
            if (wide)
                id_qrcp_kernel<1024><<<(unsigned)count, 1024, smem, s>>>(dJobs, dA, dP, dZ, dPiv, dRank, tol, max_rank);
            else
                id_qrcp_kernel<256><<<(unsigned)count, 256, smem, s>>>(dJobs, dA, dP, dZ, dPiv, dRank, tol, max_rank);
            e = cudaGetLastError();
        }
    }
    if (dJobs) cudaFreeAsync(dJobs, s);
    if (dZ) cudaFreeAsync(dZ, s);
    if (e != cudaSuccess) return fail_id(cudaGetErrorString(e), MXB_ERR_CUDA);
    return MXB_OK;
}
