// Kernel argument blocks and the internal entry points shared by the
// single-model calls (rf.cu, se.cu) and the batched launch (batch.cu).
#pragma once

#include "common.cuh"

namespace portal {

// Everything the radiation-field kernel reads or writes for one model.
struct RFArgs {
    int N, bulk, L, nvel, nch, ndir, n_depth;
    float dx32;
    const double *__restrict__ pos;
    const double *__restrict__ bvec;
    double *frames;                   // (N, 13) node frames (k_line_table)
    const double *__restrict__ ab;
    const float4 *__restrict__ cellv;
    // the walk's tables (ctx.cu): a block of slots per node, in groups of 4
    const int *__restrict__ wstart;     // (N) first group of each node's block
    const int2 *__restrict__ whead;     // per group; a block's first: (degree, node)
    const float4 *__restrict__ wedge;   // per slot: the edge record
    const int *__restrict__ wnext;      // per slot: the neighbour's first group
    const float4 *__restrict__ ltab;
    const double *__restrict__ dirs;  // (ndir, 6): mu, sin th, cos ph, sin ph, w, w*c_in/sqrt2
    const float *__restrict__ chq;    // (nch) 2 nv / nvel
    const float *__restrict__ chw;    // (nch) exp(-q0^2) * 2/(sqrt(pi) nvel)
    const float *__restrict__ bb;     // (L) black_body(2.73 K) per line: the incoming intensity
    double gx, gy, gz;
    // star mode: each node's ray set from star_all (nth x nph bands around the
    // star direction), star rays end on the star and start from B(T_star)
    int star, nth, nph;
    double xs, ys, zs, Rs;
    const float *__restrict__ bbs;    // (L) black_body(T_star) per line
    double *J0, *J2;
    double *JE, *LS;                  // split field (accelerated Lambda iteration) or null
    int *status;
    int *segs;                        // (N) ray segments of each node (sum of node_count) or null
    float *kmom;                      // (6, N) second moment sum w I n n of line 1 (xx yy zz xy xz yz) or null
    int2 *walk;
    unsigned long long *counters;
    // items of rays (small clouds), and what they leave for k_rf_finish -- per
    // (node, ray, line) channel sums (three planes with a split field), ray
    // directions, segments per ray (-1: a walk past n_depth)
    int items32, items16;   // items of rays: so many of 32, then of 16, the rest of 8
    float *vray;
    float4 *dray;
    int *iseg;
};

// Everything the SE kernel reads or writes for one model.
struct SEArgs {
    int N, bulk, c_dim, n_trans, nlev, L, c_temp, c_num, c_par, nent;
    int n_feat;                         // features per node: NF per transition + depolarisation
    int n_dep, depol;                   // (level, K >= 2) depolarisation rates, mode (0 off)
    const double *__restrict__ dep_tab; // (c_temp, n_dep) D^(K) coefficients [cm^3/s] or null
    const double *__restrict__ J0;
    const double *__restrict__ J2;
    const double *__restrict__ JE;      // J0_eff (r_num, N) or null
    const double *__restrict__ LS;      // L* (r_num, N) or null
    const double *__restrict__ h2;
    const double *__restrict__ tkin;
    const double *__restrict__ ab;
    // per transition
    const int *__restrict__ tr_rad;
    const int *__restrict__ tr_col;
    const double *__restrict__ tr_nu;
    const double *__restrict__ tr_A;
    const double *__restrict__ tr_B21;
    const double *__restrict__ col_temps;
    const double *__restrict__ Cji;
    // program over the matrix entries
    const int *__restrict__ ent_off;
    const int *__restrict__ ent_pos;
    const int *__restrict__ term_f;
    const double *__restrict__ term_c;
    const int *__restrict__ norm_col;   // (nlev) count_array
    const double *__restrict__ norm_val;
    const int *__restrict__ pack;       // (2 nlev) rho index or -1
    const int *__restrict__ row_off;    // (c_dim + 1) entries of each matrix row,
    const int *__restrict__ row_ent;    // ascending column (the rates' summation order)
    const int4 *__restrict__ sp_rec;    // the matrix's entries, most terms first: (row | column << 16, first term,
                                        // terms << 16 | entry, -1), row 1 the normalisation's (.., 0, entry, level)
    const int *__restrict__ sp_off;     // (c_dim + 1) the entries' row offsets,
    const int *__restrict__ sp_col;     // columns
    const unsigned short *__restrict__ sp_map;  // entry at each place, nnz: none (c_dim <= 96)
    int nnz;
    double *pops;                       // (N, 2 nlev) column-major
    double *jj20;                       // (N, L) or null
    double *rates;                      // (N, 3, 2 nlev) column-major or null
    int *status;
    int *nfail;
    const unsigned long long *skip;     // the solve is left out where this is not 0 (null: never)
    double *a64;                        // FP64 matrices (entries, then dense), one slot of a64_stride doubles per team
    size_t a64_stride;
    int fp64_only;                      // factorise every system in FP64 (no FP32 LU)
};

// A batched launch: work items (model, node) over many models, the models'
// argument blocks in device memory.
struct RFBatch {
    const RFArgs *models;
    const int2 *items;
    long long n_items;
    unsigned long long *queue;   // [0] next item, [1] segments walked
    int2 *walk;                  // per warp: 32 rays x n_depth
    int n_depth;
    int nch;                     // velocity channels and their tables (the same for every model)
    const float *chq, *chw;
    int max_group;               // widest line group
    int rt;                      // remainder channel integrated lanes-over-lines
    int split;                   // the models have split fields
    size_t warp_bytes;           // dynamic shared memory per warp (largest model)
};
struct SEBatch {
    const SEArgs *models;
    const int2 *items;
    long long n_items;
    size_t team_bytes;           // dynamic shared memory per node solved (largest model)
    double *a64;                 // FP64 matrices, one slot of a64_stride doubles per node solved
    size_t a64_stride;           // largest model's nnz + c_dim^2
    int max_dim;                 // largest model's c_dim
    bool gauss;                  // every model's system is inverted
};

// rf.cu
int rf_prepare(portal_ctx *c, int nth, int nph, int nvel, const double *gvec, double dx, int n_depth,
               bool split, RFArgs *a);
int rf_pass(portal_ctx *c, const RFArgs &a, int max_group, bool dust, cudaStream_t s);
// the single-model kernel for groups of nlg lines (1..10, with dust 1..5); FLAT:
// its items are ranges of rays, not nodes
template <bool FLAT> const void *rf_kernel_one(int nlg, bool split);    // one slot of channels
template <bool FLAT> const void *rf_kernel_even(int nlg);               // an even number of slots
template <bool FLAT> const void *rf_kernel_even_split(int nlg);
template <bool FLAT> const void *rf_kernel_any(int nlg);                // any, split or not
template <bool FLAT> const void *rf_kernel_dust(int nlg, int slots);    // slots 1: one, 2: an even number, 0: any
template <> const void *rf_kernel_one<false>(int nlg, bool split);
template <> const void *rf_kernel_one<true>(int nlg, bool split);
template <> const void *rf_kernel_even<false>(int nlg);
template <> const void *rf_kernel_even<true>(int nlg);
template <> const void *rf_kernel_even_split<false>(int nlg);
template <> const void *rf_kernel_even_split<true>(int nlg);
template <> const void *rf_kernel_any<false>(int nlg);
template <> const void *rf_kernel_any<true>(int nlg);
template <> const void *rf_kernel_dust<false>(int nlg, int slots);
template <> const void *rf_kernel_dust<true>(int nlg, int slots);
const void *rf_batch_even();                       // the batched kernel's instantiations
const void *rf_batch_any(bool dust, bool one_slot, bool split);
size_t rf_walk_records(int n_depth);     // walk scratch per warp, int2 records
// the batched launch: its shape for these models (max_group: the widest line
// group wanted), and the blocks per SM the kernel reaches with it
void rf_batch_shape(RFBatch *bw, const int *lines, int n_models, int nch, bool dust, int max_group, bool split);
int rf_line_group(int lines, int max_group, bool dust);   // the groups' width for a model of so many lines
int rf_batch_blocks_per_sm(const RFBatch &bw, bool dust, int *blocks);
int rf_batch_launch(cudaStream_t s, int grid, bool dust, const RFBatch &bw);
constexpr int RF_BATCH_WARPS = 4;        // warps per block of the batched launch
// se.cu
int se_prepare(portal_ctx *c, int kmax, SEArgs *a, size_t *warp_bytes);
int se_batch_pass(portal_ctx *c, cudaStream_t s);
int se_batch_launch(cudaStream_t s, int grid, int warps_per_block, const SEBatch &bw);
int se_batch_blocks_per_sm(int warps_per_block, size_t team_bytes, int max_dim, bool gauss, int *blocks);
bool se_gauss(const portal_ctx *c);            // the prepared system is inverted,
size_t se_gauss_team_bytes(const portal_ctx *c);   // and its shared memory per node
int se_batch_team(int max_dim, bool gauss);        // warps per node of the batched solve
size_t se_matrix_doubles(const portal_ctx *c);  // matrix slot of the prepared SE program

}  // namespace portal
