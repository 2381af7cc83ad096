// FP64 evaluation (Y = K~ W, and its adjoint) as ONE persistent launch on the FP64 tensor path.
//
// tcgen05.mma has no f64 kind, so FP64 products use the DMMA instruction mma.sync.m16n8k8.f64.
//
// Layout.  Every operand the products read is kept in DMMA fragment order, as 8 x 8 sub-blocks
// of 64 doubles (512 bytes):
//   A (the CDS, tiled once at plan creation): row-major sub-blocks, sub-block columns outermost,
//     so a pipeline stage of a row tile is one run per sub-block column.  A lane takes the pair
//     (k = 2a, 2a + 1) of its row as one 16-byte shared-memory read: the two DMMA steps of a
//     sub-block use k = 2a and k = 2a + 1 (any order of k, the same for A and B, sums the same
//     products).  A transposed product reads the same sub-blocks with k = a and k = a + 4,
//     8-byte reads of 32 consecutive doubles: one copy of the CDS serves both directions.
//   B (W, wskel, uskel): column-major sub-blocks, column sub-blocks of one row sub-block
//     contiguous; element (k, n) at n * 8 + (k ^ 4 ((n >> 1) & 1)), which makes both read orders
//     free of bank conflicts.  The skeleton vectors are written this way by the epilogue that
//     computes them; W is rewritten by tasks of the same launch.
// A stage is then filled by a few 1-D bulk copies on an mbarrier, issued by one warp, and the
// product warps execute nothing but shared-memory reads and DMMAs.
//
// Schedule.  The tasks of all passes (rewriting W, up-sweep, far couplings, near field,
// down-sweep, leaf down) form one list; a unit is a task and a column tile (two where there are very
// many), claimed in list order.  Units wait on per-node counters for the blocks they read, so no pass waits for the
// last tile of the pass before.  The list comes from a list-scheduling simulation on the host
// (longest remaining path first), every unit's inputs come earlier in it and a block runs its
// units in claim order, so every wait ends; each is bounded all the same.  A long sum (a node
// in many near or far lists) is cut along K into pieces whose partial tiles the last piece
// adds up in piece order, so the result does not depend on timing.
//
// What bounds it: the DMMA pipe from about 32 right-hand sides on (91 % active), the number of tiles
// where blocks are short, HBM (the CDS, read once) below, and for small matrices the chain of node to node hops
// (2 - 3 us each: publish, poll, load, multiply).  Measured on one B200, launch per pass with
// cp.async tiles -> one dataflow launch: N = 65536 H2-b, 1024 right-hand sides 25.6 -> 23.1 ms
// (34.1 TFLOP/s), 1 right-hand side 2560 -> 460 us (5.8 TB/s); N = 16384 HSS, 256 right-hand
// sides 511 -> 349 us; N = 32768 adjoint, 64 right-hand sides (long near lists) 2940 -> 695 us;
// N = 1024, 1 right-hand side 102 -> 30 us.
#include <algorithm>
#include <cstring>
#include <queue>
#include <string>

#include "f64_engine.h"
#include "plan.h"
#include "tc_common.cuh"

namespace mxb {
namespace {

enum : int16_t { F64_Y = 0, F64_WSKEL = 1, F64_USKEL = 2, F64_TILE_W = 3 };
enum { BUF_W = 0, BUF_WSKEL = 1, BUF_USKEL = 2 };
enum { CTL_CLAIM = 0, CTL_EXIT = 1, CTL_FIRST = 16 };

constexpr int WARPS = 4, THREADS = (WARPS + 1) * 32, RING = 4;
constexpr int EAGER = 64;  // polls of a node counter before the first pause

// BN: right-hand sides of a column tile.  M8: sub-block rows of a row tile.  BK8: sub-block columns of
// A per stage.  64 rows x 32 columns for tall blocks: with 64 columns a unit takes twice as long on a
// shared SM, which the tree sweeps wait for (N = 65536, 1024 right-hand sides: 24.2 ms against 23.3
// ms; N = 16384 HSS, 256: 376 against 354 us), and 16 re-reads A too often (418 us).  The same area as
// 32 x 64 and 16 x 128 for short blocks (shape_for).  Stages of 4 sub-block columns beat 2 (24.8 ms)
// because a warp pays ~100 cycles to move to the next stage; 3 blocks of 12 product warps per SM
// beat 4 without fragment double-buffering (26.4 ms) and 2 (25 ms).
template <int BN, int M8_ = 8>
struct Cfg {
    static constexpr int M8 = M8_, N8 = BN / 8;
    static constexpr int WN = M8 < 8 ? 4 : (N8 >= 4 ? 2 : 1), WM = WARPS / WN;  // product warps: rows x columns
    static constexpr int MI = M8 / WM, NJ = N8 / WN;              // sub-blocks per warp
    static constexpr int BK8 = M8 == 2 ? 2 : 4;
    static constexpr int A_BYTES = BK8 * M8 * 512, B_BYTES = BK8 * N8 * 512;
    static constexpr int STAGE = A_BYTES + B_BYTES;
    static constexpr int STAGES = 3;
    static constexpr int CTAS = N8 >= 2 ? 3 : 4;                  // resident per SM
    static constexpr int SMEM = STAGES * STAGE + 1024;            // + barriers and the unit ring
};

struct Args {
    const double *pool[3];
    double *buf[3];
    const double *W;
    double *Y;
    const int32_t *wofs, *yofs;
    const F64Task *tasks;
    const F64Item *items;
    double *partial;
    int *ctl, *err;
    long long wait_cycles;
    int units, ncol, group, nb, nrhs, beta, nctr;  // group: column tiles of a unit (at most 32)
    // profiling (null otherwise): [0] the earliest block's start, [1 + p] the time the last tile of
    // pass p was written (%globaltimer, ns); the pass of each task
    unsigned long long *pass_ns;
    const uint8_t *pass_of;
};

struct Unit {  // ring slot: one column tile of the claimed unit
    F64Task task;
    int32_t col, n8_0, n8;
    int32_t live;   // 0: no more units, 1: more column tiles of the unit follow, 2: its last one
    int32_t index;  // of the task
    int32_t col0;   // the unit's first column tile
};

// Two stacked 8 x 8 sub-blocks of A (rows g and g + 8 of a lane's fragment) times one of B.
__device__ __forceinline__ void dmma(double (&c)[2], double (&d)[2], const double (&a0)[2], const double (&a1)[2],
                                     const double (&b)[2])
{
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+d"(c[0]), "+d"(c[1]), "+d"(d[0]), "+d"(d[1])
                 : "d"(a0[0]), "d"(a1[0]), "d"(a0[1]), "d"(a1[1]), "d"(b[0]), "d"(b[1]));
}

__device__ __forceinline__ int b_elem(int k, int n) { return n * 8 + (k ^ (((n >> 1) & 1) << 2)); }

template <int BN, int M8>
__global__ void __launch_bounds__(THREADS, Cfg<BN, M8>::CTAS) f64_dataflow_kernel(const Args g)
{
    using C = Cfg<BN, M8>;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + C::STAGES * C::STAGE);
    uint64_t *empty = full + C::STAGES;
    uint64_t *ufull = empty + C::STAGES;
    uint64_t *uempty = ufull + RING;
    Unit *ring = reinterpret_cast<Unit *>(uempty + RING);
    volatile int *meta = reinterpret_cast<volatile int *>(ring + RING);  // per stage: sub-block columns | trans << 8
    volatile int *abort_word = meta + C::STAGES;
    int *last_cta = const_cast<int *>(abort_word) + 1;
    static_assert(sizeof(Unit) == 88 && (2 * C::STAGES + 2 * RING) * 8 + RING * 88 + C::STAGES * 4 + 8 <= 1024, "");

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int *counters = g.ctl + CTL_FIRST;
    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; ++s) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], WARPS);
        }
        for (int i = 0; i < RING; ++i) {
            tc::mbar_init(&ufull[i], 1);
            tc::mbar_init(&uempty[i], WARPS);
        }
        *abort_word = 0;
        tc::fence_mbar_init();
    }
    __syncthreads();
    if (g.pass_ns && threadIdx.x == 0) atomicMin(g.pass_ns, tc::globaltimer_ns());

    if (warp == WARPS) {
        // ---------------- producer: claims units, fills the stages ----------------
        uint32_t st = 0;  // stages filled
        int slot = 0;
        const int ngroup = (g.ncol + g.group - 1) / g.group;  // units of a task
        bool ok = true, more = true;
        while (ok && more) {
            // claimed once the loads of the unit before are on their way, not earlier: a unit held
            // back behind another would keep the units that read it waiting
            int u = 0;
            if (lane == 0) u = atomicAdd(g.ctl + CTL_CLAIM, 1);
            u = __shfl_sync(0xffffffffu, u, 0);
            const int t = u / ngroup, col0 = (u - t * ngroup) * g.group;
            const bool done = u >= g.units;
            const int col1 = done ? col0 + 1 : min(g.ncol, col0 + g.group);
            const int word = !done && lane < 16 ? __ldg(reinterpret_cast<const int *>(g.tasks + t) + lane) : 0;
            for (int col = col0; col < col1 && ok; ++col) {
                const int i = slot % RING;
                ok = __all_sync(0xffffffffu, tc::mbar_wait(&uempty[i], ((slot / RING) & 1) ^ 1, abort_word, g.wait_cycles));
                if (!ok) break;
                ++slot;
                Unit &un = ring[i];
                // column tiles of nearly equal width: sub-blocks [n8_0, n8_0 + n8)
                const int n8_0 = (int)((long long)g.nb * col / g.ncol);
                const int n8 = (int)((long long)g.nb * (col + 1) / g.ncol) - n8_0;
                if (lane < 16) reinterpret_cast<int *>(&un.task)[lane] = word;
                if (lane == 16) un.col = col;
                if (lane == 17) un.n8_0 = n8_0;
                if (lane == 18) un.n8 = n8;
                if (lane == 19) un.live = done ? 0 : 1 + (col + 1 == col1);
                if (lane == 20) un.index = t;
                if (lane == 21) un.col0 = col0;
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(tc::smem_u32(&ufull[i])) : "memory");
                if (done) {
                    more = false;
                    break;
                }
                const int item0 = un.task.item0, nitem = un.task.nitem, r8 = un.task.r8, m8 = un.task.m8;
                for (int q = 0; q < nitem && ok; ++q) {
                    const F64Item it = g.items[item0 + q];
                    const double *a0 = it.a_pool == 0 ? g.pool[0] : (it.a_pool == 1 ? g.pool[1] : g.pool[2]);
                    const double *b0 = it.b_buf == 0 ? g.buf[0] : (it.b_buf == 1 ? g.buf[1] : g.buf[2]);
                    const uint8_t *A = reinterpret_cast<const uint8_t *>(a0 + it.a_off * 64);
                    const uint8_t *B = reinterpret_cast<const uint8_t *>(b0 + (it.b_base * g.nb + n8_0) * 64);
                    // stage f of the item: the CDS side (and the byte count of both), then B
                    auto load_a = [&](uint32_t f, int k0) {
                        const int s = f % C::STAGES, nk = min(C::BK8, it.k8 - k0);
                        uint8_t *sa = smem + s * C::STAGE;
                        if (lane == 0) {
                            meta[s] = nk | (it.trans << 8);
                            tc::mbar_expect_tx(&full[s], (uint32_t)(nk * (m8 + n8) * 512));
                        }
                        __syncwarp();
                        if (it.trans) {  // one run per sub-block row of the tile
                            if (lane < m8)
                                tc::bulk_g2s(sa + lane * C::BK8 * 512, A + ((size_t)(r8 + lane) * it.lda + k0) * 512,
                                             (uint32_t)nk * 512, &full[s]);
                        } else if (lane < nk) {  // one run per sub-block column of the stage
                            tc::bulk_g2s(sa + lane * C::M8 * 512, A + ((size_t)(k0 + lane) * it.lda + r8) * 512,
                                         (uint32_t)m8 * 512, &full[s]);
                        }
                    };
                    auto load_b = [&](uint32_t f, int k0) {
                        const int s = f % C::STAGES, nk = min(C::BK8, it.k8 - k0);
                        if (lane < nk)
                            tc::bulk_g2s(smem + s * C::STAGE + C::A_BYTES + lane * C::N8 * 512,
                                         B + (size_t)(k0 + lane) * g.nb * 512, (uint32_t)n8 * 512, &full[s]);
                    };
                    int ahead = 0;  // sub-block columns whose A is on its way
                    if (it.dep >= 0) {
                        const int *ctr = counters + it.dep * g.ncol + col;
                        // every lane takes its own acquire: each issues copies of its own
                        if (__all_sync(0xffffffffu, tc::counter_reached(ctr, it.need))) {
                            tc::fence_async_global();
                        } else {
                            // B is not written yet: fill the free stages with A meanwhile
                            for (uint32_t f = st; ahead < it.k8 && f < st + C::STAGES; ++f, ahead += C::BK8) {
                                if (!__all_sync(0xffffffffu, tc::mbar_try_wait(&empty[f % C::STAGES], ((f / C::STAGES) & 1) ^ 1))) break;
                                load_a(f, ahead);
                            }
                            ok = __all_sync(0xffffffffu, tc::wait_counter(ctr, it.need, abort_word, g.wait_cycles, EAGER));
                        }
                    }
                    for (int k0 = 0; k0 < it.k8; k0 += C::BK8, ++st) {
                        if (k0 >= ahead) {
                            if (ok) ok = __all_sync(0xffffffffu, tc::mbar_wait(&empty[st % C::STAGES], ((st / C::STAGES) & 1) ^ 1,
                                                                            abort_word, g.wait_cycles));
                            if (!ok) break;
                            load_a(st, k0);
                        }
                        load_b(st, k0);  // also after a failed wait: a stage that was begun is filled
                    }
                }
            }
        }
        if (!ok && lane == 0) *abort_word = 1;
        __syncwarp();
        // every filled stage has landed before the block may exit
        for (uint32_t f = st > C::STAGES ? st - C::STAGES : 0; f < st; ++f) {
            volatile int never = 0;
            tc::mbar_wait(&full[f % C::STAGES], (f / C::STAGES) & 1, &never, tc::WAIT_CYCLES);
        }
    } else {
        // ---------------- product warps ----------------
        const int wm = warp / C::WN, wn = warp % C::WN;
        const int fr = lane >> 2, fa = lane & 3;  // fragment row (A) or column (B), and k
        uint32_t st = 0, pend = 0;  // pend: column tiles of the unit written, not counted yet
        for (int slot = 0;; ++slot) {
            const int ri = slot % RING;
            if (!tc::mbar_wait_warp(&ufull[ri], (slot / RING) & 1, abort_word, g.wait_cycles)) {
                *abort_word = 1;
                break;
            }
            const Unit &un = ring[ri];
            if (!un.live) break;
            const int m8 = un.task.m8, n8 = un.n8, stages = un.task.stages;
            // this warp's sub-blocks: rows [mb, mb + mi), columns [jb, jb + nj)
            const int mb = m8 * wm / C::WM, mi = m8 * (wm + 1) / C::WM - mb;
            const int jb = n8 * wn / C::WN, nj = n8 * (wn + 1) / C::WN - jb;
            double acc[C::MI][C::NJ][2];
#pragma unroll
            for (int i = 0; i < C::MI; ++i)
#pragma unroll
                for (int j = 0; j < C::NJ; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
            // an accumulating unit starts from the old output, read while its first stages load
            // (written by another unit of this launch where old_dep says so)
            auto old_output = [&](const Unit &u) -> bool {
                if (u.task.old_dep >= 0) {
                    if (!__all_sync(0xffffffffu, tc::wait_counter(counters + u.task.old_dep * g.ncol + u.col, u.task.old_need,
                                                                  abort_word, g.wait_cycles, EAGER)))
                        return false;
                }
                if (u.task.kind == F64_Y) {
                    const int rows = u.task.rows;
                    const int r0 = (u.task.r8 + mb) * 8 + fr, c0 = (u.n8_0 + jb) * 8 + 2 * fa;
                    const double *Y = g.Y + g.yofs[u.task.out] + r0 + (size_t)c0 * rows;
#pragma unroll
                    for (int j = 0; j < C::NJ; ++j, Y += (size_t)8 * rows)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            if (j >= nj || c0 + 8 * j + e >= g.nrhs) break;
#pragma unroll
                            for (int i = 0; i < C::MI; ++i)
                                if (i < mi && r0 + 8 * i < rows) acc[i][j][e] = Y[(e ? rows : 0) + 8 * i];
                        }
                } else {
                    const double *row = g.buf[BUF_USKEL] + ((u.task.out + u.task.r8 + mb) * (int64_t)g.nb + u.n8_0 + jb) * 64;
                    const int e0 = b_elem(fr, 2 * fa), e1 = b_elem(fr, 2 * fa + 1);
#pragma unroll
                    for (int i = 0; i < C::MI; ++i, row += (size_t)g.nb * 64) {
                        if (i >= mi) break;
#pragma unroll
                        for (int j = 0; j < C::NJ; ++j)
                            if (j < nj) {
                                acc[i][j][0] = row[j * 64 + e0];
                                acc[i][j][1] = row[j * 64 + e1];
                            }
                    }
                }
                return true;
            };
            bool ok = true;
            const int kind = un.task.kind, beta = un.task.beta == 2 ? g.beta : un.task.beta;
            if (beta && kind != F64_TILE_W && un.task.npiece == 1) ok = old_output(un);
            for (int q = 0; q < stages && ok; ++q, ++st) {
                const int s = st % C::STAGES;
                if (!tc::mbar_wait_warp(&full[s], (st / C::STAGES) & 1, abort_word, g.wait_cycles)) {
                    ok = false;
                    break;
                }
                const int mt = meta[s], nk = mt & 0xFF;
                const double *sa = reinterpret_cast<const double *>(smem + s * C::STAGE);
                const double *sb = reinterpret_cast<const double *>(smem + s * C::STAGE + C::A_BYTES);
                // ALL: every sub-block of the warp's tile and of the stage exists; the fragments of the
                // next sub-block column are then read while this one's products run
                auto products = [&](auto trans, auto whole) {
                    constexpr bool T = decltype(trans)::value, ALL = decltype(whole)::value;
                    const int sw = ((fr >> 1) & 1) << 2;
                    const double *pb = sb + jb * 64 + fr * 8 + (T ? fa ^ sw : (2 * fa) ^ sw);
                    const double *pa = T ? sa + mb * C::BK8 * 64 + fr + fa * 8 : sa + mb * 64 + fr * 8 + fa * 2;
                    const int hop = T ? ((fa + 4) ^ sw) - (fa ^ sw) : 0;
                    double a[2][C::MI][2], b[2][C::NJ][2];
                    auto fetch = [&](int k, int h) {
#pragma unroll
                        for (int j = 0; j < C::NJ; ++j) {
                            if (!ALL && j >= nj) break;
                            const double *q = pb + (k * C::N8 + j) * 64;
                            if constexpr (T) {
                                b[h][j][0] = q[0];
                                b[h][j][1] = q[hop];
                            } else {
                                const double2 v = *reinterpret_cast<const double2 *>(q);
                                b[h][j][0] = v.x;
                                b[h][j][1] = v.y;
                            }
                        }
                        // rows come in pairs: past an odd count the stage holds older values, whose
                        // products are never stored
#pragma unroll
                        for (int i = 0; i < C::MI; ++i) {
                            if (!ALL && (i & ~1) >= mi) break;
                            if constexpr (T) {
                                a[h][i][0] = pa[(i * C::BK8 + k) * 64];
                                a[h][i][1] = pa[(i * C::BK8 + k) * 64 + 32];
                            } else {
                                const double2 v = *reinterpret_cast<const double2 *>(pa + (k * C::M8 + i) * 64);
                                a[h][i][0] = v.x;
                                a[h][i][1] = v.y;
                            }
                        }
                    };
                    auto multiply = [&](int h) {
#pragma unroll
                        for (int i = 0; i < C::MI; i += 2) {
                            if (!ALL && i >= mi) break;
#pragma unroll
                            for (int j = 0; j < C::NJ; ++j) {
                                if (!ALL && j >= nj) break;
                                dmma(acc[i][j], acc[i + 1][j], a[h][i], a[h][i + 1], b[h][j]);
                            }
                        }
                    };
                    if constexpr (ALL) {
                        fetch(0, 0);
#pragma unroll
                        for (int k = 0; k < C::BK8; ++k) {
                            if (k + 1 < C::BK8) fetch(k + 1, (k + 1) & 1);
                            multiply(k & 1);
                        }
                    } else {
                        for (int k = 0; k < nk; ++k) {
                            fetch(k, 0);
                            multiply(0);
                        }
                    }
                };
                const bool whole = mi == C::MI && nj == C::NJ && nk == C::BK8;
                if (mt >> 8) {
                    if (whole) products(std::true_type{}, std::true_type{});
                    else products(std::true_type{}, std::false_type{});
                } else {
                    if (whole) products(std::false_type{}, std::true_type{});
                    else products(std::false_type{}, std::false_type{});
                }
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(tc::smem_u32(&empty[s])) : "memory");
            }
            if (!ok) {
                *abort_word = 1;
                break;
            }
            const int col = un.col, n8_0 = un.n8_0, sig = un.task.sig;
            bool write = true;
            if (un.task.npiece > 1) {
                // K piece: leave the partial tile; the last piece of the tile to arrive adds all of
                // them in piece order
                constexpr int PER = C::MI * C::NJ * 2 * 32;  // partial values per warp
                const size_t stride = (size_t)g.ncol * WARPS * PER;
                double *base = g.partial + ((size_t)un.task.slot * g.ncol + col) * WARPS * PER + warp * PER + lane;
                double *mine = base + un.task.piece * stride;
#pragma unroll
                for (int i = 0; i < C::MI; ++i)
#pragma unroll
                    for (int j = 0; j < C::NJ; ++j) {
                        __stcg(mine + ((i * C::NJ + j) * 2) * 32, acc[i][j][0]);
                        __stcg(mine + ((i * C::NJ + j) * 2 + 1) * 32, acc[i][j][1]);
                    }
                __threadfence();
                __syncwarp();
                int seen = 0;
                if (lane == 0) seen = atomicAdd(counters + un.task.piece_ctr * g.ncol + col * WARPS + warp, 1);
                write = __shfl_sync(0xffffffffu, seen, 0) == un.task.npiece - 1;
                if (write) {
                    __threadfence();
#pragma unroll
                    for (int i = 0; i < C::MI; ++i)
#pragma unroll
                        for (int j = 0; j < C::NJ; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
                    if (beta && !old_output(un)) {
                        *abort_word = 1;
                        break;
                    }
                    for (int p = 0; p < un.task.npiece; ++p) {
                        const double *src = base + p * stride;
#pragma unroll
                        for (int i = 0; i < C::MI; ++i)
#pragma unroll
                            for (int j = 0; j < C::NJ; ++j) {
                                acc[i][j][0] += __ldcg(src + ((i * C::NJ + j) * 2) * 32);
                                acc[i][j][1] += __ldcg(src + ((i * C::NJ + j) * 2 + 1) * 32);
                            }
                    }
                }
            }
            if (write) {
                if (kind == F64_Y) {
                    const int rows = un.task.rows;
                    const int r0 = (un.task.r8 + mb) * 8 + fr, c0 = (n8_0 + jb) * 8 + 2 * fa;
                    double *Y = g.Y + g.yofs[un.task.out] + r0 + (size_t)c0 * rows;
#pragma unroll
                    for (int j = 0; j < C::NJ; ++j, Y += (size_t)8 * rows)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            if (j >= nj || c0 + 8 * j + e >= g.nrhs) break;
                            double *y = Y + (e ? rows : 0);
#pragma unroll
                            for (int i = 0; i < C::MI; ++i)
                                if (i < mi && r0 + 8 * i < rows) y[8 * i] = acc[i][j][e];
                        }
                } else if (kind == F64_TILE_W) {
                    // W (column-major, leading dimension rows) -> sub-blocks of this column tile; a
                    // warp takes 32 rows of 16 columns at a time, all its loads in flight (k past
                    // the leaf and columns past nrhs are zero)
                    const int rows = un.task.rows, r8 = un.task.r8;
                    const double *W = g.W + g.wofs[un.task.out];
                    double *dst = g.buf[BUF_W] + un.task.slot * (int64_t)g.nb * 64;
                    const int nj2 = (n8 + 1) >> 1, steps = (m8 + 3) / 4 * nj2;
                    for (int x = warp; x < steps; x += WARPS) {
                        const int kq = x / nj2, j = 2 * (x - kq * nj2);
                        const int k = r8 * 8 + kq * 32 + lane;
                        double v[16];
#pragma unroll
                        for (int n = 0; n < 16; ++n) {
                            const int c = (n8_0 + j) * 8 + n;
                            v[n] = (k < rows && c < g.nrhs) ? W[(size_t)k + (size_t)c * rows] : 0.0;
                        }
                        if (k < (r8 + m8) * 8) {
                            double *blk = dst + ((int64_t)(k >> 3) * g.nb + n8_0 + j) * 64;
#pragma unroll
                            for (int n = 0; n < 16; ++n)
                                if (j + n / 8 < n8) blk[n / 8 * 64 + b_elem(k & 7, n & 7)] = v[n];
                        }
                    }
                } else {
                    double *buf = kind == F64_WSKEL ? g.buf[BUF_WSKEL] : g.buf[BUF_USKEL];
                    double *row = buf + ((un.task.out + un.task.r8 + mb) * (int64_t)g.nb + n8_0 + jb) * 64;
                    const int e0 = b_elem(fr, 2 * fa), e1 = b_elem(fr, 2 * fa + 1);
                    // rows past the block are K padding of the units that read it: zero, not the sum
                    // of zeros times what may be infinite
                    const int left = un.task.rows - (un.task.r8 + mb) * 8 - fr;
#pragma unroll
                    for (int i = 0; i < C::MI; ++i, row += (size_t)g.nb * 64) {
                        if (i >= mi) break;
                        const bool in = 8 * i < left;
#pragma unroll
                        for (int j = 0; j < C::NJ; ++j)
                            if (j < nj) {
                                row[j * 64 + e0] = in ? acc[i][j][0] : 0.0;
                                row[j * 64 + e1] = in ? acc[i][j][1] : 0.0;
                            }
                    }
                }
                if (sig >= 0) pend |= 1u << (col - un.col0);
                if (g.pass_ns && lane == 0) atomicMax(g.pass_ns + 1 + g.pass_of[un.index], tc::globaltimer_ns());
            }
            if (un.live == 2 && pend) {  // one fence for all column tiles of the unit
                asm volatile("fence.proxy.async.global;\n" ::: "memory");
                __threadfence();
                __syncwarp();
                if ((pend >> lane) & 1) atomicAdd(counters + sig * g.ncol + un.col0 + lane, 1);
                pend = 0;
            }
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(tc::smem_u32(&uempty[ri])) : "memory");
        }
    }
    __syncwarp();
    __syncthreads();
    // the last block out leaves the claim counter and every other counter at zero for the next launch
    if (threadIdx.x == 0) {
        if (*abort_word) atomicExch(g.err, MXB_ERR_TIMEOUT);
        __threadfence();
        *last_cta = atomicAdd(g.ctl + CTL_EXIT, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (*last_cta) {
        __threadfence();
        for (int i = threadIdx.x; i < g.nctr; i += THREADS) counters[i] = 0;
        if (threadIdx.x == 0) g.ctl[CTL_CLAIM] = g.ctl[CTL_EXIT] = 0;
    }
}

// CDS blocks (column-major) -> sub-blocks, one job per block.
struct PoolJob {
    const double *src;  // device address
    uint64_t dst;       // sub-block offset from the first pool
    int32_t ld, rows, cols, pad;
};

// A warp writes four sub-blocks (32 rows of 8 columns) at a time: reads of 32 consecutive rows.
__global__ void __launch_bounds__(256) f64_tile_pool_kernel(const PoolJob *__restrict__ jobs, double *__restrict__ dst)
{
    const PoolJob j = jobs[blockIdx.x];
    const int m8 = (j.rows + 7) >> 3, k8 = (j.cols + 7) >> 3, mq = (m8 + 3) >> 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int x = blockIdx.y * 8 + warp; x < mq * k8; x += gridDim.y * 8) {
        const int q = x % mq, k = x / mq;
        const int r = q * 32 + lane;
        double v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e)
            v[e] = (r < j.rows && k * 8 + e < j.cols) ? j.src[(size_t)r + (size_t)(k * 8 + e) * j.ld] : 0.0;
        if (r < m8 * 8) {
            double *o = dst + (j.dst + (uint64_t)k * m8 + (r >> 3)) * 64 + (r & 7) * 8;
#pragma unroll
            for (int e = 0; e < 8; e += 2) *reinterpret_cast<double2 *>(o + e) = make_double2(v[e], v[e + 1]);
        }
    }
}

int fail(const std::string &m, int code = MXB_ERR_CUDA)
{
    (void)cudaGetLastError();  // reported here, not by the next launch
    set_error(m);
    return code;
}

#define F64_CUDA(call)                                                                    \
    do {                                                                                  \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess) return fail(std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

int sm_count()
{
    static int n[128];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 128) return 148;
    if (!n[dev] && cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
    return n[dev];
}

template <int BN, int M8 = 8>
int launch(const Args &a, cudaStream_t stream)
{
    using C = Cfg<BN, M8>;
    static bool configured[128];
    int dev = 0;
    F64_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 128) return fail("device index out of range");
    if (!configured[dev]) {
        F64_CUDA(cudaFuncSetAttribute(f64_dataflow_kernel<BN, M8>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
        configured[dev] = true;
    }
    const int grid = std::min(a.units, sm_count() * C::CTAS);
    f64_dataflow_kernel<BN, M8><<<grid, THREADS, C::SMEM, stream>>>(a);
    F64_CUDA(cudaGetLastError());
    return MXB_OK;
}

struct Shape {  // of the kernel variant and task list that run `nb` column sub-blocks
    int bn, m8, bk8, ctas, wm, ncol;
    bool fused = false;  // far and down, near and leaf down in one sum each
    int group = 1;       // column tiles of a unit
};

template <int BN, int M8 = 8>
Shape shape_of(int nb)
{
    using C = Cfg<BN, M8>;
    return {BN, M8, C::BK8, C::CTAS, C::WM, (nb + C::N8 - 1) / C::N8};
}

// Row tiles of a block; tiles of all output blocks of an evaluation.
int row_tiles_of(int rows, int m8) { return std::max(1, ((rows + 7) / 8 + m8 - 1) / m8); }
int64_t tiles_of(const Plan &p, const Shape &s)
{
    int64_t n = 0;
    for (int v : p.Ddim) n += 3 * row_tiles_of(v, s.m8);  // W, near field, leaf down
    for (int v : p.slen) n += 3 * row_tiles_of(v, s.m8);  // up, far, down
    return n * s.ncol;
}

// Columns: the narrowest variant that holds all of them (8, 16), else tiles of at most 32: below 17
// right-hand sides the launch is bound by the CDS bytes, and a wider tile only adds padding products (16
// right-hand sides, N = 32768: 237 us; 32: 382 us).
//
// Short blocks: a tile of 64 rows is mostly empty, and an evaluation is as many tiles, of 2 - 3 us each
// whatever they hold.  Flatter, wider tiles where they cut the number of tiles by more than a quarter:
// HSS of N = 16384, 1000 right-hand sides, leaves of 16 points 1804 -> 588 us (16 x 128), of 32 points
// 1486 -> 917 (32 x 64; N = 65536, 512 columns 2159 -> 1309).  Not below 8 tiles per block, where more
// blocks at work count for more: N = 4096, leaves of 32, 64 columns (5 per block) 55.5 us against 57.8,
// 100 columns (10) 68.6 against 65.8.
//
// Many tiles per block (of those resident): the launch is bound by tiles, not by the path through the
// tree.  From 128 on, a block's far and down products, and its near and leaf down products, are one
// sum, which a short path needs in two units: the far and near parts run while the sweeps arrive (N
// = 16384 HSS, 256 columns, 41 per block: 347 us).  N = 65536 HSS, leaves of 64, 1000 columns 3273 ->
// 2872 us, of 256 9371 -> 9106; H2-b, leaves of 256, 1024 columns (726 per block) 23.36 -> 23.14 ms.
// From 512 on, a unit is two column tiles: one claim and one publication for both (2872 -> 2758 us,
// 23.14 -> 23.07 ms; at 330 per block 4560 -> 4623).
Shape shape_for(const Plan &p, int nb)
{
    if (nb <= 1) return shape_of<8>(nb);
    if (nb <= 2) return shape_of<16>(nb);
    Shape best = shape_of<32>(nb);
    int64_t tiles = tiles_of(p, best);
    const bool many = tiles >= 8 * (int64_t)sm_count() * best.ctas;
    for (const Shape &s : {shape_of<64, 4>(nb), shape_of<128, 2>(nb)}) {
        const int64_t n = tiles_of(p, s);
        if (!many || 4 * n >= 3 * tiles) continue;
        best = s;
        tiles = n;
    }
    const int64_t per_block = tiles / (sm_count() * best.ctas);
    best.fused = per_block >= 128;
    best.group = per_block >= 512 ? std::min(2, best.ncol) : 1;
    return best;
}

// A group of the schedule: the tasks of one output block in one pass, and the groups it reads.
struct Group {
    int task0, ntask, dep0, ndep;
};

}  // namespace

// ---------------------------------------------------------------------------------------
// creation: the CDS into sub-blocks
// ---------------------------------------------------------------------------------------

namespace {

// Where every block of the CDS goes (host only), and where it comes from.
struct BlockSource {
    uint64_t src;  // element offset in the caller's pool
    uint64_t dst;  // sub-block offset in the pool
    int32_t ld, rows, cols;
    uint64_t end() const { return src + (uint64_t)(cols - 1) * ld + rows; }
};

void layout(Plan &p, std::vector<BlockSource> (&blocks)[3], uint64_t (&used)[3])
{
    F64Engine &E = *(p.f64 = new F64Engine());
    auto ceil8 = [](int64_t v) { return (int32_t)((v + 7) / 8); };
    auto add = [&](int pool, uint64_t src, int ld, int rows, int cols) {
        F64Block b;
        b.off = used[pool];
        b.m8 = ceil8(rows);
        b.k8 = ceil8(cols);
        used[pool] += (uint64_t)b.m8 * b.k8;
        if (rows > 0 && cols > 0) blocks[pool].push_back(BlockSource{src, b.off, ld, rows, cols});
        return b;
    };
    for (size_t k = 0; k < p.near_x.size(); ++k)
        E.near.push_back(add(0, p.near_off[k], p.Ddim[p.near_x[k]], p.Ddim[p.near_x[k]], p.Ddim[p.near_y[k]]));
    for (size_t k = 0; k < p.far_x.size(); ++k)
        E.far.push_back(add(1, p.far_off[k], p.slen[p.far_x[k]], p.slen[p.far_x[k]], p.slen[p.far_y[k]]));
    E.proj_l.resize(p.numnodes);
    E.proj_r.resize(p.numnodes);
    for (int v = 0; v < p.numnodes; ++v) {
        if (v == p.root || p.slen[v] <= 0) continue;
        const int s = p.slen[v];
        if (p.lch[v] == -1) {
            E.proj_l[v] = add(2, (uint64_t)p.VTptr[v], s, s, p.Ddim[p.lm[v]]);
        } else {
            const int l = p.slen[p.lch[v]], r = p.slen[p.rch[v]];
            E.proj_l[v] = add(2, (uint64_t)p.VTptr[v], s, s, l);
            E.proj_r[v] = add(2, (uint64_t)p.VTptr[v] + (uint64_t)s * l, s, s, r);
        }
    }
    E.leaf8.resize(p.nleaf);
    for (int i = 0; i < p.nleaf; ++i) {
        E.leaf8[i] = E.leaf8_total;
        E.leaf8_total += ceil8(p.Ddim[i]);
    }
    E.node8.assign(p.numnodes, 0);
    for (int v : p.bfs) {
        E.node8[v] = E.node8_total;
        E.node8_total += ceil8(p.slen[v]);
    }
}

}  // namespace

// Device memory for the tiling besides the pools, at most: pools on the host go through it piece by
// piece (a block larger than it alone), so a plan needs little more than its own size.  Mapping and
// unmapping it costs more than the copies it saves: 72 MB of CDS take 6.8 - 7.5 ms in pieces of 8
// MB, 7.1 - 7.4 in 64, 8.1 in 1; 2.8 MB take 0.7 ms in pieces of 1 MB and 1.3 ms in one.
constexpr size_t STAGING_BYTES = 8 << 20, SMALL_STAGING_BYTES = 1 << 20;

int f64_create(Plan &p, const double *D, const double *B, const double *VT)
{
    std::vector<BlockSource> blocks[3];
    uint64_t used[3] = {0, 0, 0};
    layout(p, blocks, used);
    F64Engine &E = *p.f64;
    const double *src[3] = {D, B, VT};
    // one allocation for the pools and the error word, and one for the tiling.  The error word
    // stays where it is until the plan is destroyed: it holds a failure until it is asked for, also
    // where the workspaces of the failed evaluation have been replaced since.
    const uint64_t total = used[0] + used[1] + used[2];
    int rc = p.alloc((void **)&E.pool[0], total * 512 + 512);
    if (rc) return rc;
    E.pool[1] = E.pool[0] + used[0] * 64;
    E.pool[2] = E.pool[1] + used[1] * 64;
    E.err = reinterpret_cast<int *>(E.pool[0] + total * 64);
    F64_CUDA(cudaMemset(E.err, 0, sizeof(int)));
    // pieces: runs of blocks whose part of the caller's pool fits the staging, several pools together
    // where they do.  The caller's pool is read in place where this device holds it.
    struct Copy {
        const double *from;
        size_t to, len;  // elements
    };
    struct Piece {
        std::vector<Copy> copies;
        size_t job0, jobs;
    };
    std::vector<PoolJob> jobs;
    std::vector<Piece> pieces(1, Piece{{}, 0, 0});
    std::vector<std::pair<const double *, uint64_t>> from;  // per job: the pool (null: the staging), and where in it
    size_t fill = 0, staging = 0;
    const size_t room = (total * 512 <= STAGING_BYTES ? SMALL_STAGING_BYTES : STAGING_BYTES) / sizeof(double);
    uint64_t first = 0;        // of the pool's sub-blocks
    for (int q = 0; q < 3; first += used[q++]) {
        std::vector<BlockSource> &bl = blocks[q];
        cudaPointerAttributes at{};
        bool here = false;
        if (!bl.empty() && cudaPointerGetAttributes(&at, src[q]) != cudaSuccess) (void)cudaGetLastError();
        else here = at.type == cudaMemoryTypeDevice && at.device == p.device;
        if (!here)
            std::sort(bl.begin(), bl.end(), [](const BlockSource &a, const BlockSource &b) { return a.src < b.src; });
        for (size_t i = 0; i < bl.size();) {
            size_t n = 1;
            uint64_t end = bl[i].end();
            auto joins = [&](uint64_t e) { return here || std::max(end, e) - bl[i].src <= room; };
            while (i + n < bl.size() && joins(bl[i + n].end())) end = std::max(end, bl[i + n++].end());
            if (!here) {
                const size_t len = (size_t)(end - bl[i].src);
                if (fill && fill + len > room) {
                    pieces.push_back(Piece{{}, jobs.size(), 0});
                    fill = 0;
                }
                pieces.back().copies.push_back(Copy{src[q] + bl[i].src, fill, len});
            }
            for (size_t k = i; k < i + n; ++k) {
                jobs.push_back(PoolJob{nullptr, first + bl[k].dst, bl[k].ld, bl[k].rows, bl[k].cols, 0});
                from.push_back({here ? src[q] : nullptr, here ? bl[k].src : fill + (bl[k].src - bl[i].src)});
            }
            pieces.back().jobs += n;
            if (!here) {
                fill += (size_t)(end - bl[i].src);
                staging = std::max(staging, fill);
            }
            i += n;
        }
    }
    if (jobs.empty()) return MXB_OK;
    const size_t job_bytes = (jobs.size() * sizeof(PoolJob) + 255) / 256 * 256;
    uint8_t *work = nullptr;
    cudaError_t e = cudaMalloc(&work, job_bytes + staging * sizeof(double));
    double *stage = reinterpret_cast<double *>(work + job_bytes);
    for (size_t k = 0; k < jobs.size(); ++k) jobs[k].src = (from[k].first ? from[k].first : stage) + from[k].second;
    if (e == cudaSuccess) e = cudaMemcpy(work, jobs.data(), jobs.size() * sizeof(PoolJob), cudaMemcpyHostToDevice);
    for (const Piece &pc : pieces) {  // (on the legacy stream: a piece's copies wait for the kernel before)
        for (const Copy &c : pc.copies)
            if (e == cudaSuccess) e = cudaMemcpy(stage + c.to, c.from, c.len * sizeof(double), cudaMemcpyDefault);
        if (e != cudaSuccess || !pc.jobs) continue;
        f64_tile_pool_kernel<<<dim3((unsigned)pc.jobs, 4), 256>>>(reinterpret_cast<PoolJob *>(work) + pc.job0, E.pool[0]);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);
    if (work) cudaFree(work);
    if (e == cudaErrorMemoryAllocation) return fail("tiling the CDS: out of device memory", MXB_ERR_NOMEM);
    if (e != cudaSuccess) return fail(std::string("tiling the CDS: ") + cudaGetErrorString(e));
    return MXB_OK;
}

// ---------------------------------------------------------------------------------------
// schedule
// ---------------------------------------------------------------------------------------

namespace {

// Tasks in claim order for one direction and column count; see the file comment.  Built at the first
// evaluation of each, so the lists are flat arrays and the workers are kept by integer times: N =
// 65536 with leaves of 256 points, 10075 tasks, 0.75 ms (2.5 ms with vectors of tasks and readers per
// group and a heap of workers); the first product with one column after creation 2.0 ms (3.3).
int build_schedule(Plan &p, bool adjoint, const Shape &sh, std::vector<F64Task> &out, std::vector<F64Item> &items,
                   int &nctr, int64_t &slots)
{
    F64Engine &E = *p.f64;
    auto projects = [&](int v) { return v != p.root && p.slen[v] > 0; };
    auto has_down = [&](int v) { return p.parent[v] >= 0 && projects(p.parent[v]); };
    auto ceil8 = [](int v) { return (v + 7) / 8; };
    auto row_tiles = [&](int rows) { return row_tiles_of(rows, sh.m8); };
    // counters (times the column count): per leaf W tiled and near field written; per node
    // wskel, far part and uskel written
    const int c_w = 0, c_near = p.nleaf, c_up = 2 * p.nleaf, c_far = c_up + p.numnodes, c_u = c_far + p.numnodes;
    nctr = c_u + p.numnodes;
    const bool fused = sh.fused;
    std::vector<Group> G;
    std::vector<F64Task> all;
    std::vector<int> deps;
    G.reserve(3 * (size_t)p.nleaf + 3 * (size_t)p.numnodes);
    all.reserve(4 * G.capacity());
    deps.reserve(p.near_x.size() + p.far_x.size() + 2 * G.capacity());
    items.reserve(p.near_x.size() + p.far_x.size() + G.capacity());
    std::vector<int> g_w(p.nleaf, -1), g_near(p.nleaf, -1), g_up(p.numnodes, -1), g_far(p.numnodes, -1), g_u(p.numnodes, -1);
    const int WR = WARPS;  // every product warp of a tile counts itself
    auto stages_of = [&](int k8) { return (k8 + sh.bk8 - 1) / sh.bk8; };
    // A group is begun, given the groups and blocks it reads, and ended with its output rows.  Every
    // group reads only groups begun before it.
    int item0 = 0, dep0 = 0, stages = 0;
    auto begin_group = [&]() {
        item0 = (int)items.size();
        dep0 = (int)deps.size();
        stages = 0;
    };
    auto reads_group = [&](int g) {
        if (g >= 0 && std::find(deps.begin() + dep0, deps.end(), g) == deps.end()) deps.push_back(g);
    };
    auto reads = [&](const F64Block &a, int pool, int trans, int buf, int dep, int need, int group, int64_t base) {
        F64Item it{};
        it.a_off = a.off;
        it.lda = a.m8;
        it.k8 = trans ? a.m8 : a.k8;
        if (it.k8 <= 0) return;
        it.b_base = base;
        it.dep = dep;
        it.need = need;
        it.a_pool = (int16_t)pool;
        it.trans = (int16_t)trans;
        it.b_buf = (int16_t)buf;
        items.push_back(it);
        stages += stages_of(it.k8);
        reads_group(group);
    };
    auto end_group = [&](int kind, int64_t o, int rows, int beta, int sig, int old_dep, int old_need, int slot) {
        F64Task t{};
        t.out = o;
        t.item0 = item0;
        t.nitem = (int)items.size() - item0;
        t.stages = stages;
        t.rows = rows;
        t.sig = sig;
        t.old_dep = old_dep;
        t.old_need = old_need;
        t.piece_ctr = -1;
        t.npiece = 1;
        t.kind = (int16_t)kind;
        t.beta = (int16_t)beta;
        t.slot = slot;
        const int m8 = ceil8(rows), T = row_tiles(rows);
        G.push_back(Group{(int)all.size(), T, dep0, (int)deps.size() - dep0});
        for (int i = 0; i < T; ++i) {  // row tiles of nearly equal height
            t.r8 = (int)((int64_t)m8 * i / T);
            t.m8 = (int)((int64_t)m8 * (i + 1) / T) - t.r8;
            all.push_back(t);
        }
        return (int)G.size() - 1;
    };
    auto reads_w = [&](const F64Block &a, int pool, int trans, int leaf) {
        reads(a, pool, trans, BUF_W, c_w + leaf, WR * row_tiles(p.Ddim[leaf]), g_w[leaf], E.leaf8[leaf]);
    };
    auto reads_up = [&](const F64Block &a, int pool, int trans, int v) {  // (nothing writes the root's block)
        reads(a, pool, trans, BUF_WSKEL, g_up[v] < 0 ? -1 : c_up + v, WR * row_tiles(p.slen[v]), g_up[v], E.node8[v]);
    };
    auto reads_u = [&](const F64Block &a, int pool, int trans, int v) {
        reads(a, pool, trans, BUF_USKEL, c_u + v, WR * row_tiles(p.slen[v]), g_u[v], E.node8[v]);
    };
    for (int i = 0; i < p.nleaf; ++i) {
        begin_group();
        g_w[i] = end_group(F64_TILE_W, i, p.Ddim[i], 0, c_w + i, -1, 0, (int)E.leaf8[i]);
    }
    for (auto it = p.bfs.rbegin(); it != p.bfs.rend(); ++it) {  // children before parents
        const int v = *it;
        if (!projects(v)) continue;
        begin_group();
        if (p.lch[v] == -1) {
            reads_w(E.proj_l[v], 2, 0, p.lm[v]);
        } else {
            if (p.slen[p.lch[v]] > 0) reads_up(E.proj_l[v], 2, 0, p.lch[v]);
            if (p.slen[p.rch[v]] > 0) reads_up(E.proj_r[v], 2, 0, p.rch[v]);
        }
        g_up[v] = end_group(F64_WSKEL, E.node8[v], p.slen[v], 0, c_up + v, -1, 0, 0);
    }
    // the pairs of each output block: far by node, near by leaf
    auto by_output = [](const std::vector<int> &x, int n, std::vector<int> &first, std::vector<int> &pair) {
        first.assign(n + 1, 0);
        for (int v : x) ++first[v + 1];
        for (int i = 0; i < n; ++i) first[i + 1] += first[i];
        pair.resize(x.size());
        std::vector<int> at(first.begin(), first.end() - 1);
        for (size_t k = 0; k < x.size(); ++k) pair[at[x[k]]++] = (int)k;
    };
    std::vector<int> far0, far_of, near0, near_of;
    by_output(adjoint ? p.far_y : p.far_x, p.numnodes, far0, far_of);
    by_output(adjoint ? p.near_y : p.near_x, p.nleaf, near0, near_of);
    auto reads_far = [&](int v) {
        for (int q = far0[v]; q < far0[v + 1]; ++q) {
            const int k = far_of[q], o = adjoint ? p.far_x[k] : p.far_y[k];
            if (p.slen[o] > 0) reads_up(E.far[k], 1, adjoint ? 1 : 0, o);
        }
    };
    for (int v : p.bfs) {
        if (!projects(v) || (fused && has_down(v))) continue;
        begin_group();
        reads_far(v);
        if ((int)items.size() == item0 && has_down(v)) continue;
        g_far[v] = end_group(F64_USKEL, E.node8[v], p.slen[v], 0, has_down(v) ? c_far + v : c_u + v, -1, 0, 0);
        if (!has_down(v)) g_u[v] = g_far[v];
    }
    for (int v : p.bfs) {  // parents before children
        if (!projects(v) || !has_down(v)) continue;
        const int q = p.parent[v];
        const bool far = g_far[v] >= 0;
        begin_group();
        if (fused) reads_far(v);
        reads_u(v == p.rch[q] ? E.proj_r[q] : E.proj_l[q], 2, 1, q);
        reads_group(g_far[v]);
        g_u[v] = end_group(F64_USKEL, E.node8[v], p.slen[v], far ? 1 : 0, c_u + v, far ? c_far + v : -1,
                           WR * row_tiles(p.slen[v]), 0);
    }
    std::vector<int> leaf_node(p.nleaf, -1);
    for (int v = 0; v < p.numnodes; ++v)
        if (p.lch[v] == -1) leaf_node[p.lm[v]] = v;
    for (int i = 0; i < p.nleaf; ++i) {
        begin_group();
        for (int q = near0[i]; q < near0[i + 1]; ++q) {
            const int k = near_of[q];
            reads_w(E.near[k], 0, adjoint ? 1 : 0, adjoint ? p.near_x[k] : p.near_y[k]);
        }
        const int v = leaf_node[i];
        if (fused && projects(v)) reads_u(E.proj_l[v], 2, 1, v);
        g_near[i] = end_group(F64_Y, i, p.Ddim[i], 2, c_near + i, -1, 0, 0);
        if (fused || !projects(v)) continue;
        begin_group();
        reads_u(E.proj_l[v], 2, 1, v);
        reads_group(g_near[i]);
        end_group(F64_Y, i, p.Ddim[i], 1, -1, c_near + i, WR * row_tiles(p.Ddim[i]), 0);
    }

    // Long sums are cut along K where one would keep a block busy for a large part of the
    // launch: pieces of about an eighth of a block's share of all stages, at least 256 deep
    // (N = 32768 adjoint, 64 right-hand sides: 707 us when this was chosen; a third of the share:
    // 800 us; sixteenths only add partial tiles).
    const int blocks = sm_count() * sh.ctas, ngroup = (int)G.size();
    int64_t total = 0;
    for (const F64Task &t : all) total += (int64_t)t.stages * sh.ncol;
    const int chunk = (int)std::max<int64_t>(32 / sh.bk8, total / (8 * (int64_t)blocks));
    slots = 0;
    std::vector<F64Item> src;
    std::vector<F64Task> tiles, range;
    for (Group &g : G) {
        const F64Task t0 = all[g.task0];
        if (t0.stages <= chunk + chunk / 2) continue;
        const int n = (t0.stages + chunk - 1) / chunk;
        // item ranges of the pieces, cut at stage boundaries
        src.assign(items.begin() + t0.item0, items.begin() + t0.item0 + t0.nitem);
        range.assign(n, t0);
        int q = 0, off = 0;
        for (int i = 0; i < n; ++i) {
            F64Task &r = range[i];
            int want = (int)((int64_t)t0.stages * (i + 1) / n) - (int)((int64_t)t0.stages * i / n);
            r.item0 = (int)items.size();
            r.stages = want;
            while (want > 0) {
                F64Item it = src[q];
                const int have = stages_of(it.k8 - off), take = std::min(want, have);
                it.a_off += it.trans ? (uint64_t)off : (uint64_t)off * it.lda;
                it.b_base += off;
                it.k8 = std::min(take * sh.bk8, it.k8 - off);
                items.push_back(it);
                want -= take;
                off += take * sh.bk8;
                if (take == have) {
                    ++q;
                    off = 0;
                }
            }
            r.nitem = (int)items.size() - r.item0;
        }
        tiles.assign(all.begin() + g.task0, all.begin() + g.task0 + g.ntask);
        g.task0 = (int)all.size();
        g.ntask *= n;
        for (const F64Task &base : tiles) {
            for (int i = 0; i < n; ++i) {
                F64Task t = range[i];
                t.r8 = base.r8;
                t.m8 = base.m8;
                t.piece = i;
                t.npiece = n;
                t.piece_ctr = nctr;
                t.slot = (int)slots;
                all.push_back(t);
            }
            nctr += WARPS;  // one arrival counter per product warp
            slots += n;
        }
    }

    // List scheduling, longest remaining path first among the groups whose inputs are written.  A
    // worker stands for the blocks that run one task's column tiles side by side; it claims its
    // next task once the loads of the current one are issued, STAGES before its products end.
    // Times in stages of a busy SM (1.0 - 1.5 us): writing a tile out and publishing it takes
    // about EPILOGUE, seeing it and loading from it about LATENCY.
    const int EPILOGUE = sh.bn == 8 ? 4 : 2, LATENCY = 2, DEPTH = 3;
    std::vector<int> prio(ngroup, 0), ready_at(ngroup, 0), unplaced(ngroup), con0(ngroup + 1, 0), cons(deps.size());
    for (int i = ngroup - 1; i >= 0; --i) {  // (readers come after what they read)
        const Group &g = G[i];
        int cost = 0;
        for (int t = g.task0; t < g.task0 + g.ntask; ++t) cost = std::max(cost, all[t].stages);
        prio[i] += cost + EPILOGUE + LATENCY;
        unplaced[i] = g.ndep;
        for (int d = g.dep0; d < g.dep0 + g.ndep; ++d) {
            prio[deps[d]] = std::max(prio[deps[d]], prio[i]);
            ++con0[deps[d] + 1];
        }
    }
    for (int i = 0; i < ngroup; ++i) con0[i + 1] += con0[i];
    {
        std::vector<int> at(con0.begin(), con0.end() - 1);
        for (int i = 0; i < ngroup; ++i)
            for (int d = G[i].dep0; d < G[i].dep0 + G[i].ndep; ++d) cons[at[deps[d]]++] = i;
    }
    // the highest priority, then the first group; the earliest time, then the first group
    std::priority_queue<std::pair<int, int>> ready, waiting;
    // Workers by the time they claim at, which only grows: lists per time, walked in order.
    const int nworker = std::max(1, blocks / sh.ncol);
    std::vector<int> at(1, 0), next(nworker), free_at(nworker, 0);  // first worker of a time, the one after
    for (int w = 0; w < nworker; ++w) next[w] = w + 1 < nworker ? w + 1 : -1;
    int now = 0;
    for (int i = 0; i < ngroup; ++i)
        if (!unplaced[i]) waiting.push({0, -i});
    out.clear();
    out.reserve(all.size());
    for (int placed = 0; placed < ngroup; ++placed) {
        while (at[now] < 0) ++now;
        while (!waiting.empty() && -waiting.top().first <= now) {
            const int i = -waiting.top().second;
            waiting.pop();
            ready.push({prio[i], -i});
        }
        int i;
        if (!ready.empty()) {
            i = -ready.top().second;
            ready.pop();
        } else if (!waiting.empty()) {
            i = -waiting.top().second;
            waiting.pop();
        } else {
            return fail("FP64 schedule: a block's inputs are never written", MXB_ERR_STRUCTURE);
        }
        const Group &g = G[i];
        int finish = 0;
        for (int t = g.task0; t < g.task0 + g.ntask; ++t) {
            while (at[now] < 0) ++now;
            const int w = at[now], load = std::max(now, ready_at[i]);
            const int end = std::max(load + 1, free_at[w]) + all[t].stages, claim = std::max(load, end - DEPTH);
            at[now] = next[w];
            if (claim >= (int)at.size()) at.resize(claim + claim / 2 + 1, -1);
            next[w] = at[claim];
            at[claim] = w;
            free_at[w] = end + EPILOGUE;
            finish = std::max(finish, free_at[w]);
            out.push_back(all[t]);
        }
        for (int q = con0[i]; q < con0[i + 1]; ++q) {
            const int c = cons[q];
            ready_at[c] = std::max(ready_at[c], finish + LATENCY);
            if (--unplaced[c] == 0) waiting.push({-ready_at[c], -c});
        }
    }
    return MXB_OK;
}

// Task lists of a plan, in bytes, above which the oldest go (N = 65536 with leaves of 256 points: 1.4
// MB each).  Those a caller's graph may replay stay.
constexpr size_t SCHEDULE_BYTES = 64 << 20;

int schedule_for(Plan &p, bool adjoint, const Shape &sh, bool capturing, F64Engine::Schedule **out)
{
    F64Engine &E = *p.f64;
    for (F64Engine::Schedule &s : E.schedules)
        if (s.adjoint == adjoint && s.ncol == sh.ncol && s.bn == sh.bn) {
            *out = &s;
            return MXB_OK;
        }
    if (capturing) return refuse_unprepared();
    std::vector<F64Task> tasks;
    std::vector<F64Item> items;
    F64Engine::Schedule s;
    s.adjoint = adjoint;
    s.ncol = sh.ncol;
    s.bn = sh.bn;
    int rc = build_schedule(p, adjoint, sh, tasks, items, s.nctr, s.slots);
    if (rc) return rc;
    s.ntasks = (int)tasks.size();
    if ((int64_t)s.ntasks * sh.ncol > 0x3FFFFFFF) return fail("too many work units", MXB_ERR_UNSUPPORTED);
    const size_t tb = tasks.size() * sizeof(F64Task), ib = items.size() * sizeof(F64Item);
    s.bytes = tb + ib;
    size_t held = s.bytes;
    for (const F64Engine::Schedule &o : E.schedules) held += o.bytes;
    for (size_t i = 0; i < E.schedules.size() && held > SCHEDULE_BYTES;) {
        if (E.schedules[i].recorded) {
            ++i;
            continue;
        }
        held -= E.schedules[i].bytes;
        cudaFree(E.schedules[i].tasks);
        E.schedules.erase(E.schedules.begin() + i);
    }
    std::vector<uint8_t> both(tb + ib);
    std::memcpy(both.data(), tasks.data(), tb);
    if (ib) std::memcpy(both.data() + tb, items.data(), ib);
    cudaError_t e = cudaMalloc(&s.tasks, std::max<size_t>(both.size(), 16));
    if (e == cudaSuccess) e = cudaMemcpy(s.tasks, both.data(), both.size(), cudaMemcpyHostToDevice);
    // the launch's stream does not wait for the legacy stream, and a copy from pageable memory
    // may return before it has landed
    if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);
    if (e != cudaSuccess) {
        if (s.tasks) cudaFree(s.tasks);
        return fail(std::string("FP64 schedule: ") + cudaGetErrorString(e),
                    e == cudaErrorMemoryAllocation ? MXB_ERR_NOMEM : MXB_ERR_CUDA);
    }
    s.items = reinterpret_cast<F64Item *>(s.tasks + tasks.size());
    E.schedules.push_back(s);
    *out = &E.schedules.back();
    return MXB_OK;
}

}  // namespace

// ---------------------------------------------------------------------------------------
// evaluation
// ---------------------------------------------------------------------------------------

namespace {

int evaluate(Plan &p, bool adjoint, const double *dW, double *dY, const int32_t *wofs, const int32_t *yofs, int nrhs,
             int accumulate, cudaStream_t stream, unsigned long long *pass_ns, const uint8_t *pass_of)
{
    F64Engine &E = *p.f64;
    const int nb = (nrhs + 7) / 8;
    const Shape sh = shape_for(p, nb);
    bool capturing = false;
    int rc = is_capturing(stream, &capturing);
    if (rc) return rc;
    F64Engine::Schedule *s = nullptr;
    rc = schedule_for(p, adjoint, sh, capturing, &s);
    if (rc) return rc;
    if (nb > E.buf_nb) {
        if (capturing) return refuse_unprepared();
        p.release(E.buf[0], (size_t)(E.leaf8_total + 2 * E.node8_total) * E.buf_nb * 512);
        E.buf[0] = nullptr;
        E.buf_nb = 0;
        rc = p.alloc((void **)&E.buf[0], (size_t)(E.leaf8_total + 2 * E.node8_total) * nb * 512);
        if (rc) return rc;
        E.buf[1] = E.buf[0] + (size_t)E.leaf8_total * nb * 64;
        E.buf[2] = E.buf[1] + (size_t)E.node8_total * nb * 64;
        E.buf_nb = nb;
    }
    // counters (zero between launches: each launch's last block clears what it used), then the
    // partial tiles
    const size_t ctl = ((CTL_FIRST + (size_t)s->nctr * sh.ncol) * sizeof(int) + 511) / 512 * 512;
    const size_t partial = (size_t)s->slots * sh.ncol * 8 * sh.m8 * sh.bn * sizeof(double);
    if (ctl > E.ctl_bytes || partial > E.partial_bytes) {
        const size_t c = std::max(ctl, E.ctl_bytes), q = std::max(partial, E.partial_bytes);
        if (capturing) return refuse_unprepared();
        p.release(E.ctl, E.ctl_bytes + E.partial_bytes);
        E.ctl = nullptr;
        E.ctl_bytes = E.partial_bytes = 0;
        rc = p.alloc((void **)&E.ctl, c + q);
        if (rc) return rc;
        F64_CUDA(cudaMemset(E.ctl, 0, c));
        F64_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
        E.ctl_bytes = c;
        E.partial_bytes = q;
    }
    if (capturing) {
        s->recorded = true;
        p.record();
    }
    Args a{};
    for (int q = 0; q < 3; ++q) {
        a.pool[q] = E.pool[q];
        a.buf[q] = E.buf[q];
    }
    a.W = dW;
    a.Y = dY;
    a.wofs = wofs;
    a.yofs = yofs;
    a.tasks = s->tasks;
    a.items = s->items;
    a.partial = reinterpret_cast<double *>(E.ctl + E.ctl_bytes / sizeof(int));
    a.ctl = E.ctl;
    a.err = E.err;
    // ~2 s, and longer for evaluations that themselves take that long
    a.wait_cycles = p.debug_wait_cycles > 0 ? p.debug_wait_cycles : tc::WAIT_CYCLES + (long long)(p.flops(nrhs) / 500);
    a.units = s->ntasks * ((sh.ncol + sh.group - 1) / sh.group);
    a.ncol = sh.ncol;
    a.group = sh.group;
    a.nb = nb;
    a.nrhs = nrhs;
    a.beta = accumulate ? 1 : 0;
    a.nctr = s->nctr * sh.ncol;
    a.pass_ns = pass_ns;
    a.pass_of = pass_of;
    switch (sh.bn) {
    case 8: return launch<8>(a, stream);
    case 16: return launch<16>(a, stream);
    case 32: return launch<32>(a, stream);
    case 64: return launch<64, 4>(a, stream);
    default: return launch<128, 2>(a, stream);
    }
}

// Rows of the products that a variant's warps issue for a tile of m8 sub-block rows: its share of
// them in pairs, per warp.
int issued_rows(const Shape &s, int m8)
{
    int rows = 0;
    for (int w = 0; w < s.wm; ++w) rows += (m8 * (w + 1) / s.wm - m8 * w / s.wm + 1) / 2 * 16;
    return rows;
}

}  // namespace

int f64_evaluate(Plan &p, bool adjoint, const double *dW, double *dY, const int32_t *wofs, const int32_t *yofs,
                 int nrhs, int accumulate, cudaStream_t stream)
{
    return evaluate(p, adjoint, dW, dY, wofs, yofs, nrhs, accumulate, stream, nullptr, nullptr);
}

// The one launch of a forward evaluation by passes: a record per up-sweep height (the rewriting of W
// with the first), far + down depth, and the near field with leaf down.  Flops come from the
// structure, units and issued flops from the task list that ran, spans from the kernel's own timer.
int f64_profile(Plan &p, const double *dW, double *dY, const int32_t *wofs, const int32_t *yofs, int nrhs,
                cudaStream_t stream, mxb_op_profile *out, int cap, int *nops)
{
    F64Engine &E = *p.f64;
    const int nb = (nrhs + 7) / 8;
    const Shape sh = shape_for(p, nb);
    F64Engine::Schedule *s = nullptr;
    int rc = schedule_for(p, false, sh, false, &s);
    if (rc) return rc;
    std::vector<F64Task> tasks(s->ntasks);
    std::vector<F64Item> items((s->bytes - tasks.size() * sizeof(F64Task)) / sizeof(F64Item));
    F64_CUDA(cudaMemcpy(tasks.data(), s->tasks, tasks.size() * sizeof(F64Task), cudaMemcpyDeviceToHost));
    if (!items.empty())
        F64_CUDA(cudaMemcpy(items.data(), s->items, items.size() * sizeof(F64Item), cudaMemcpyDeviceToHost));

    std::vector<mxb_op_profile> rec;
    auto record = [&](int phase, int level) {
        mxb_op_profile o{};
        o.phase = phase;
        o.level = level;
        o.width = sh.bn;
        o.chained = rec.empty() ? 0 : 1;
        rec.push_back(o);
        return (int)rec.size() - 1;
    };
    auto projects = [&](int v) { return v != p.root && p.slen[v] > 0; };
    int top = 0, deep = 0;
    for (int v = 0; v < p.numnodes; ++v)
        if (projects(v)) {
            top = std::max(top, p.height[v]);
            deep = std::max(deep, p.depth[v]);
        }
    std::vector<int> up(top + 1, -1), down(deep + 1, -1);
    for (int h = 0; h <= top; ++h)
        for (int v = 0; v < p.numnodes && up[h] < 0; ++v)
            if (projects(v) && p.height[v] == h) up[h] = record(MXB_PHASE_UP, h);
    for (int d = 1; d <= deep; ++d)
        for (int v = 0; v < p.numnodes && down[d] < 0; ++v)
            if (projects(v) && p.depth[v] == d) down[d] = record(MXB_PHASE_FAR_DOWN, d);
    const int near = record(MXB_PHASE_NEAR_LEAF_DOWN, 0);
    for (int v = 0; v < p.numnodes; ++v) {
        if (!projects(v)) continue;
        const bool leaf = p.lch[v] == -1;
        const double cols = leaf ? p.Ddim[p.lm[v]] : p.slen[p.lch[v]] + p.slen[p.rch[v]];
        rec[up[p.height[v]]].flops += 2.0 * p.slen[v] * cols * nrhs;
        if (leaf) rec[near].flops += 2.0 * p.slen[v] * cols * nrhs;
        if (p.parent[v] >= 0 && projects(p.parent[v]))
            rec[down[p.depth[v]]].flops += 2.0 * p.slen[v] * p.slen[p.parent[v]] * nrhs;
    }
    for (size_t k = 0; k < p.far_x.size(); ++k)
        if (projects(p.far_x[k])) rec[down[p.depth[p.far_x[k]]]].flops += 2.0 * p.slen[p.far_x[k]] * p.slen[p.far_y[k]] * nrhs;
    for (size_t k = 0; k < p.near_x.size(); ++k) rec[near].flops += 2.0 * p.Ddim[p.near_x[k]] * p.Ddim[p.near_y[k]] * nrhs;

    std::vector<int> node_at(E.node8_total + 1, -1);  // by sub-block row
    for (int v = 0; v < p.numnodes; ++v)
        if (projects(v)) node_at[E.node8[v]] = v;
    std::vector<uint8_t> pass(tasks.size());
    for (size_t t = 0; t < tasks.size(); ++t) {
        const F64Task &tk = tasks[t];
        const int k = tk.kind == F64_TILE_W ? 0 : tk.kind == F64_Y ? near
                      : tk.kind == F64_WSKEL ? up[p.height[node_at[tk.out]]] : down[p.depth[node_at[tk.out]]];
        pass[t] = (uint8_t)std::min(k, 255);
        rec[k].units += sh.ncol;
        for (int q = tk.item0; q < tk.item0 + tk.nitem; ++q)
            rec[k].issued_flops += 2.0 * issued_rows(sh, tk.m8) * (8.0 * items[q].k8) * (8.0 * nb);
    }

    // [start, passes], then the pass of each task
    std::vector<unsigned long long> ends(rec.size() + 1, 0);
    const size_t times = ends.size() * sizeof(unsigned long long);
    uint8_t *work = nullptr;
    F64_CUDA(cudaMalloc(&work, times + pass.size()));
    cudaEvent_t ev[2] = {nullptr, nullptr};
    cudaError_t e = cudaMemcpy(work + times, pass.data(), pass.size(), cudaMemcpyHostToDevice);
    for (cudaEvent_t &x : ev)
        if (e == cudaSuccess) e = cudaEventCreate(&x);
    for (int rep = 0; rep < 2 && !rc && e == cudaSuccess; ++rep) {
        cudaMemsetAsync(work, 0, times, stream);
        cudaMemsetAsync(work, 0xff, sizeof(unsigned long long), stream);  // start: minimum of
        cudaEventRecord(ev[0], stream);
        rc = evaluate(p, false, dW, dY, wofs, yofs, nrhs, 0, stream, reinterpret_cast<unsigned long long *>(work), work + times);
        cudaEventRecord(ev[1], stream);
        e = cudaStreamSynchronize(stream);
    }
    float ms = 0.f;
    if (!rc && e == cudaSuccess) e = cudaEventElapsedTime(&ms, ev[0], ev[1]);
    if (!rc && e == cudaSuccess) e = cudaMemcpy(ends.data(), work, times, cudaMemcpyDeviceToHost);
    for (cudaEvent_t x : ev)
        if (x) cudaEventDestroy(x);
    cudaFree(work);
    if (rc) return rc;
    if (e != cudaSuccess) return fail(std::string("profile: ") + cudaGetErrorString(e));
    const std::vector<float> spans = pass_spans(ends);
    for (size_t k = 0; k < rec.size(); ++k) {
        rec[k].ms = k ? 0.f : ms;
        rec[k].level_ms = spans[k];
        if (out && (int)k < cap) out[k] = rec[k];
    }
    if (nops) *nops = (int)rec.size();
    return MXB_OK;
}

int f64_status(Plan &p)
{
    if (!p.f64 || !p.f64->err) return MXB_OK;
    int h = 0;
    F64_CUDA(cudaMemcpy(&h, p.f64->err, sizeof(int), cudaMemcpyDeviceToHost));
    if (!h) return MXB_OK;
    F64_CUDA(cudaMemset(p.f64->err, 0, sizeof(int)));
    F64_CUDA(cudaDeviceSynchronize());
    return fail("an FP64 kernel wait timed out (MXB_ERR_TIMEOUT)", h);
}

// The last evaluation's skeleton vectors, node-blocked column-major (as skel_row * nrhs).
int f64_read_skeletons(Plan &p, int nrhs, std::vector<double> &w, std::vector<double> &u)
{
    F64Engine &E = *p.f64;
    const int64_t nb = (nrhs + 7) / 8;
    if (nb > E.buf_nb) return fail("no evaluation with this nrhs has run on the plan", MXB_ERR_ARG);
    F64_CUDA(cudaDeviceSynchronize());
    std::vector<double> h((size_t)E.node8_total * nb * 64);
    for (int which = 0; which < 2; ++which) {
        std::vector<double> &o = which ? u : w;
        o.assign((size_t)p.skel_total * nrhs, 0.0);
        F64_CUDA(cudaMemcpy(h.data(), E.buf[which ? BUF_USKEL : BUF_WSKEL], h.size() * sizeof(double), cudaMemcpyDeviceToHost));
        for (int v = 0; v < p.numnodes; ++v)
            for (int c = 0; c < nrhs; ++c)
                for (int r = 0; r < p.slen[v]; ++r)
                    o[(size_t)p.skel_row[v] * nrhs + (size_t)c * p.slen[v] + r] =
                        h[((size_t)(E.node8[v] + r / 8) * nb + c / 8) * 64 + (c % 8) * 8 + ((r % 8) ^ ((((c % 8) >> 1) & 1) << 2))];
    }
    return MXB_OK;
}

void f64_destroy(Plan &p)
{
    if (!p.f64) return;
    for (F64Engine::Schedule &s : p.f64->schedules) cudaFree(s.tasks);
    delete p.f64;
    p.f64 = nullptr;
}

}  // namespace mxb

// Test hook (no counterpart in the reference): the task list of the FP64 launch; host code only.
extern "C" int32_t mxb_debug_f64_schedule(const mxb_cds_desc *desc, int32_t adjoint, int32_t nrhs, void *tasks,
                                          int64_t task_cap, void *items, int64_t item_cap, int64_t *counts)
{
    if (!desc || nrhs < 1 || !tasks || !items || !counts) {
        mxb::set_error("bad FP64 schedule arguments");
        return MXB_ERR_ARG;
    }
    mxb::Plan p;
    int rc = p.validate(*desc);
    if (rc) return rc;
    std::vector<mxb::BlockSource> blocks[3];
    uint64_t used[3] = {0, 0, 0};
    mxb::layout(p, blocks, used);
    const mxb::Shape sh = mxb::shape_for(p, (nrhs + 7) / 8);
    std::vector<mxb::F64Task> t;
    std::vector<mxb::F64Item> it;
    int nctr = 0;
    int64_t slots = 0;
    rc = mxb::build_schedule(p, adjoint != 0, sh, t, it, nctr, slots);
    if (rc) return rc;
    const int64_t c[9] = {(int64_t)t.size(), (int64_t)it.size(), nctr, slots, sh.ncol, sh.bk8,
                          (int64_t)used[0], (int64_t)used[1], (int64_t)used[2]};
    std::memcpy(counts, c, sizeof(c));
    if ((int64_t)t.size() > task_cap || (int64_t)it.size() > item_cap) {
        mxb::set_error("output arrays too short");
        return MXB_ERR_ARG;
    }
    std::memcpy(tasks, t.data(), t.size() * sizeof(mxb::F64Task));
    std::memcpy(items, it.data(), it.size() * sizeof(mxb::F64Item));
    return MXB_OK;
}
