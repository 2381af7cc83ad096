// FP64 evaluation engine of a plan: the CDS in DMMA fragment order and one persistent
// dataflow launch per evaluation (f64_engine.cu).
#pragma once
#include <cstdint>
#include <vector>

#include "matrox_b200.h"
#include "mxb_internal.h"

namespace mxb {

struct Plan;

// One block of the CDS in fragment order: 8 x 8 sub-blocks of 64 doubles (row-major), the
// sub-block of rows 8 i.. and columns 8 j.. at 64 * (off + j * m8 + i) doubles of its pool.
struct F64Block {
    uint64_t off = 0;  // in 64-double sub-blocks
    int32_t m8 = 0;    // sub-block rows
    int32_t k8 = 0;    // sub-block columns
};

struct F64Task {       // one row tile (or one K piece of it) of one output block; 64 bytes
    int64_t out;       // leaf index (Y, W tiles) or sub-block row base in the skeleton buffer
    int32_t item0, nitem;
    int32_t rows;      // rows of the whole output block (its leading dimension in Y)
    int32_t r8;        // first sub-block row of this tile
    int32_t m8;        // sub-block rows of this tile (<= 8)
    int32_t stages;    // pipeline stages of the tile's items
    int32_t sig;       // counter raised when the tile is written (times ncol, + column), or -1
    int32_t old_dep;   // counter to reach before the old output is read back, or -1
    int32_t old_need;
    int32_t piece_ctr; // K pieces: arrival counters of the tile (times ncol; 4 per column), or -1
    int32_t piece, npiece;
    int16_t kind;      // F64_*
    int16_t beta;      // 0 overwrite, 1 accumulate, 2 the launch's argument
    int32_t slot;      // K pieces: first partial slot of the tile; W tiles: sub-block row base of the leaf
};
static_assert(sizeof(F64Task) == 64, "F64Task layout");

struct F64Item {       // one product op(A) B of a task; 40 bytes
    uint64_t a_off;    // sub-block (0, 0) of A in its pool
    int32_t lda;       // sub-block rows of A's block
    int32_t k8;        // inner sub-blocks of this item
    int64_t b_base;    // sub-block row base of B in its buffer
    int32_t dep;       // counter of B's producer (times ncol, + column), or -1
    int32_t need;
    int16_t a_pool, trans, b_buf, pad0;
};
static_assert(sizeof(F64Item) == 40, "F64Item layout");

struct F64Engine {
    // ---- structure (host) ----
    std::vector<F64Block> near, far;           // per pair
    std::vector<F64Block> proj_l, proj_r;      // per node: P_v (leaf: proj_l) or its two halves
    std::vector<int64_t> leaf8, node8;         // sub-block row bases of leaves / nodes
    int64_t leaf8_total = 0, node8_total = 0;
    // ---- device ----
    double *pool[3] = {nullptr, nullptr, nullptr};  // near, far, projections
    double *buf[3] = {nullptr, nullptr, nullptr};   // W, wskel, uskel sub-blocks
    int64_t buf_nb = 0;                             // column sub-blocks the buffers hold
    int *ctl = nullptr;                             // claim, exits, counters; then partial tiles
    int *err = nullptr;                             // sticky error word, behind the pools
    size_t ctl_bytes = 0, partial_bytes = 0;
    struct Schedule {                               // tasks in claim order for one column count
        bool adjoint = false;
        int ncol = 0, bn = 0;
        int ntasks = 0, nctr = 0;
        int64_t slots = 0;                          // partial slots (times ncol)
        size_t bytes = 0;                           // of tasks and items
        bool recorded = false;                      // in a caller's capture: kept (see Plan::recorded)
        F64Task *tasks = nullptr;                   // followed by the items
        F64Item *items = nullptr;
    };
    std::vector<Schedule> schedules;
};

int f64_create(Plan &p, const double *D, const double *B, const double *VT);
int f64_evaluate(Plan &p, bool adjoint, const double *dW, double *dY, const int32_t *wofs, const int32_t *yofs,
                 int nrhs, int accumulate, cudaStream_t stream);
int f64_profile(Plan &p, const double *dW, double *dY, const int32_t *wofs, const int32_t *yofs, int nrhs,
                cudaStream_t stream, mxb_op_profile *out, int cap, int *nops);
int f64_status(Plan &p);
int f64_read_skeletons(Plan &p, int nrhs, std::vector<double> &w, std::vector<double> &u);
void f64_destroy(Plan &p);

}  // namespace mxb
