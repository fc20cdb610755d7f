// Polarized statistical equilibrium of every node: make_AC + get_rhovec +
// the packing of trace_node.
//
// Reference: trace_node main_sub.f90:93-137, make_AC miscellaneous.f90:288-392,
// all_transitions :394-460, setup_count_array :206-239, get_rhovec
// em_coefs.f90:115-201, setup_stateq pop_eqs.f90:361-653 and the coupling
// constants pop_eqs.f90:1-359.
//
// Every entry of the SE matrix is a linear combination of seven per-node,
// per-transition quantities
//     f0 = B21 J0,  f1 = B21 J2,  f2 = A21,  f3 = C21 (n_H2, T),
//     f4 = C21 exp(-h nu / k T),  f5 = B21 J0_eff,  f6 = A21 (1 - L*)
// with node-independent coefficients built from the Wigner coupling
// constants.  f5 and f6 serve the couplings between K = 0 components
// (populations) only.  Without a local operator J0_eff = J0 and L* = 0, so
// they equal f0 and f2 exactly and the matrix is setup_stateq's.  With one
// (the accelerated Lambda iteration) J0 = J0_eff + L* S is split into the
// field of everything but the node's own emission and the node's own
// contribution L* S, and the net radiative rates of the K = 0 equations,
// (B_lu n_l - B_ul n_u) J0 - A n_u, become (B_lu n_l - B_ul n_u) J0_eff -
// A (1 - L*) n_u (Rybicki & Hummer 1991, A&A 245, 171: the preconditioned
// rate equations), still linear in the populations.  At the fixed point
// (S unchanged) both forms are the same equations.  The host turns setup_stateq's loops into that program once per
// (molecule, kmax): a CSR list over matrix entries of (feature, coefficient)
// terms.  The kernel (one warp per node or a team of four) evaluates the
// features, assembles the matrix's entries (FP64), replaces row 1 by the
// normalisation sum sqrt(2J+1) rho^0_0 = 1, inverts a row-scaled FP32 copy by
// Gauss-Jordan elimination with partial pivoting (up to 96 unknowns; above,
// FP32 LU factors) and refines the solution of A rho = e_1 with FP64
// residuals.  Should the refinement stall (FP32 too inaccurate for the
// matrix's condition) the node is factorised in FP64 on the device and
// flagged.
//
// Depolarising collisions (portal_set_depolarization; off by default, as
// main_sub.f90:96 passes D0 = 0): setup_stateq's col_dep slot
// (pop_eqs.f90:642-648) holds D^(K)(level) = n_H2 1e-6 times the
// coefficient de_polarization tabulates (depol.f90:242-317), interpolated in
// T as make_depolarization_temp does (depol.f90:319-360).  Each (level, K >=
// 2) rate is one more per-node feature after the transitions' ones; mode 2
// keeps a second copy that stands for col_dep read where the reference does
// not assign it (its last assigned value, carried through the loop), which
// the extra_info rates leave out as the reference's C_mat does.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>

#include "internal.cuh"

namespace portal {
void coupling_constants(int which, int j, int k, int j2, int k2, double *c0, double *c2);
double wigner3j(int tj1, int tj2, int tj3, int tm1, int tm2, int tm3);
double wigner6j(int tj1, int tj2, int tj3, int tj4, int tj5, int tj6);
}
using namespace portal;

namespace {

constexpr double A_TO_B = 6.781962e49;  // pop_eqs.f90:419
constexpr double HK = 4.79924e-11;      // pop_eqs.f90:535

// In-place LU with partial pivoting of the n x n column-major matrix M
// (pivot: the first row of largest modulus, as LAPACK's IDAMAX picks).
// Returns false if a pivot is zero.
template <typename T>
__device__ bool warp_lu(int n, T *M, int *piv, int lane) {
    bool ok = true;
    for (int k = 0; k < n; k++) {
        T best = (T)-1;
        int bi = n;
        for (int i = k + lane; i < n; i += 32) {
            T v = fabs(M[i + (size_t)n * k]);
            if (v > best) { best = v; bi = i; }
        }
        for (int o = 16; o >= 1; o >>= 1) {
            T ob = __shfl_xor_sync(0xffffffffu, best, o);
            int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
        if (bi >= n) bi = k;  // NaN column: no row qualified; keep the diagonal
        if (lane == 0) piv[k] = bi;
        if (!(best > (T)0)) { ok = false; }
        if (bi != k)
            for (int j = lane; j < n; j += 32) {
                T t = M[k + (size_t)n * j];
                M[k + (size_t)n * j] = M[bi + (size_t)n * j];
                M[bi + (size_t)n * j] = t;
            }
        __syncwarp();
        const T d = M[k + (size_t)n * k];
        const T r = (d != (T)0) ? (T)1 / d : (T)0;
        for (int i = k + 1 + lane; i < n; i += 32) M[i + (size_t)n * k] *= r;
        __syncwarp();
        for (int i = k + 1 + lane; i < n; i += 32) {
            const T lik = M[i + (size_t)n * k];
            if (lik != (T)0)
                for (int j = k + 1; j < n; j++) M[i + (size_t)n * j] -= lik * M[k + (size_t)n * j];
        }
        __syncwarp();
    }
    return ok;
}

// Solve (LU) x = P b in place in b (length n, shared memory), one warp.
// The pivots are applied in shared memory; then lane l holds b[l + 32 m] in
// register br[m], and step k broadcasts b[k] = br[k / 32] of lane k % 32
// with a shuffle.  The steps run in blocks of 32 under an unrolled loop over
// the register index, so every register is named at compile time (a
// run-time index would put br in local memory).  The per-element operations
// are those of the plain forward and back substitution (b[i] -= M[i,k] b[k];
// b[k] /= M[k,k]).  MR rows per lane: n <= 32 MR.
template <typename T, typename V, int MR>
__device__ void warp_lu_solve(int n, const T *M, const int *piv, V *b, int lane) {
    if (lane == 0)
        for (int k = 0; k < n; k++)
            if (piv[k] != k) { V t = b[k]; b[k] = b[piv[k]]; b[piv[k]] = t; }
    __syncwarp();
    V br[MR];
#pragma unroll
    for (int m = 0; m < MR; m++) br[m] = (lane + 32 * m < n) ? b[lane + 32 * m] : (V)0;
#pragma unroll
    for (int kb = 0; kb < MR; kb++) {
        if (32 * kb >= n) break;
        const int kend = min(32, n - 32 * kb);
        for (int kk = 0; kk < kend; kk++) {
            const int k = 32 * kb + kk;
            const V bk = __shfl_sync(0xffffffffu, br[kb], kk);
#pragma unroll
            for (int m = kb; m < MR; m++) {
                const int i = lane + 32 * m;
                if (i > k && i < n) br[m] -= (V)M[i + (size_t)n * k] * bk;
            }
        }
    }
#pragma unroll
    for (int kb = MR - 1; kb >= 0; kb--) {
        if (32 * kb >= n) continue;
        const int kend = min(32, n - 32 * kb);
        for (int kk = kend - 1; kk >= 0; kk--) {
            const int k = 32 * kb + kk;
            if (lane == kk) br[kb] /= (V)M[k + (size_t)n * k];
            const V bk = __shfl_sync(0xffffffffu, br[kb], kk);
#pragma unroll
            for (int m = 0; m <= kb; m++) {
                const int i = lane + 32 * m;
                if (i < k) br[m] -= (V)M[i + (size_t)n * k] * bk;
            }
        }
    }
#pragma unroll
    for (int m = 0; m < MR; m++)
        if (lane + 32 * m < n) b[lane + 32 * m] = br[m];
    __syncwarp();
}

// The same factorisation by a team of TW warps (TW = 1: warp_lu itself).
// Warp w owns the columns j = w (mod TW): it swaps their rows, applies the
// trailing update to them and, for its own column k, runs the pivot search
// (the first row of largest modulus, as before) and forms the multipliers.
// Two barriers per step: the pivot row is published, the multipliers are.
// Every element sees the operations of warp_lu in the same order, so the
// factors are the same.  Rows are spread over the lanes (at most MR per
// lane, the multipliers held in registers: n <= 32 MR).
constexpr int SE_MAX_ROWS = 8;   // c_dim <= 256
template <typename T, int TW, int MR>
__device__ bool team_lu(int n, T *M, int *piv, int tid, double *red_v, int *red_i) {
    if constexpr (TW == 1) {
        return warp_lu<T>(n, M, piv, tid);
    } else {
        const int lane = tid & 31, w = tid >> 5;
        bool ok = true;
        for (int k = 0; k < n; k++) {
            const bool own_k = (k % TW) == w;
            if (own_k) {
                T best = (T)-1;
                int bi = n;
                for (int i = k + lane; i < n; i += 32) {
                    T v = fabs(M[i + (size_t)n * k]);
                    if (v > best) { best = v; bi = i; }
                }
                for (int o = 16; o >= 1; o >>= 1) {
                    T ob = __shfl_xor_sync(0xffffffffu, best, o);
                    int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                    if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
                }
                if (bi >= n) bi = k;  // NaN column: keep the diagonal
                if (lane == 0) {
                    red_v[0] = (double)best;
                    red_i[0] = bi;
                    piv[k] = bi;
                }
            }
            __syncthreads();   // the pivot row is published (and the last step's updates are done)
            const T best = (T)red_v[0];
            const int bi = red_i[0];
            if (!(best > (T)0)) ok = false;
            if (bi != k)
                for (int j = w + TW * lane; j < n; j += 32 * TW) {
                    T t = M[k + (size_t)n * j];
                    M[k + (size_t)n * j] = M[bi + (size_t)n * j];
                    M[bi + (size_t)n * j] = t;
                }
            if (own_k) {
                __syncwarp();
                const T d = M[k + (size_t)n * k];
                const T r = (d != (T)0) ? (T)1 / d : (T)0;
                for (int i = k + 1 + lane; i < n; i += 32) M[i + (size_t)n * k] *= r;
            }
            __syncthreads();   // the multipliers are published
            T l[MR];
#pragma unroll
            for (int m = 0; m < MR; m++) {
                const int i = k + 1 + lane + 32 * m;
                l[m] = (i < n) ? M[i + (size_t)n * k] : (T)0;
            }
            int j = k + 1 + ((w - (k + 1)) % TW + TW) % TW;   // this warp's first column after k
            for (; j < n; j += TW) {
                const T mkj = M[k + (size_t)n * j];
#pragma unroll
                for (int m = 0; m < MR; m++) {
                    const int i = k + 1 + lane + 32 * m;
                    if (i < n && l[m] != (T)0) M[i + (size_t)n * j] -= l[m] * mkj;
                }
            }
        }
        __syncthreads();
        return ok;
    }
}

// Dynamic shared memory per team of the LU form (the inverses': GaussMem):
//   feat [n_feat] double | x [n] double | LU32 [n*n] float | d32 [n] float
//   | scale [n] float | piv [n] int
// The FP64 matrix is kept as its entries only, row by row (a fifth of the
// 74 x 74 systems, a third of the 34 x 34: collisions couple the K = 0
// components of all levels, radiation only neighbouring levels): assembly, row
// scaling and the refinement's residuals run over them.  Here they sit in a
// per-team slot of global memory, followed by the dense matrix of the FP64
// fallback; the inverses, which need no dense copy, keep the entries in shared
// memory.
constexpr int NF = 7;  // features per transition
constexpr int SE_GAUSS_DIM = 96;   // largest system inverted,
constexpr int SE_WARP_DIM = 32;    // and by one warp in registers

__host__ __device__ inline size_t se_warp_bytes(int n, int n_feat) {
    size_t b = 0;
    b += sizeof(double) * ((size_t)n_feat + (size_t)n);
    b += sizeof(float) * ((size_t)n * n + 2 * (size_t)n);
    b += sizeof(int) * (size_t)n;
    return (b + 15) & ~(size_t)15;
}

// ---- FP32 inverse by Gauss-Jordan elimination ------------------------------
//
// Step k turns column k of the remaining system into the inverse's: with p the
// pivot row (of largest modulus to 16 bits among the rows not yet used, the
// first of those; rows stay where they are), d = 1 / a_pk and s_j = a_pj d
// (s_k = d),
//     a_ij <- a_ij - a_ik s_j  (a_ik <- -a_ik d),   a_pj <- s_j.
// After the n steps row p_k of a yields x_k from z_j = r_(p_j): a correction of
// the refinement is one product with a, of independent fused multiply-adds,
// where triangular solves are two chains of n dependent steps (they were 43 %
// of the 74 x 74 systems' time, at 320 cycles a step).
//
// The matrix lives in registers: row i in lane i % 32 (register m = i / 32),
// column j in warp j % TW (slot c = j / TW).  The pivot column's slot must be
// a compile-time register, so the slots turn: after every ROT columns of this
// warp the array moves down by ROT, the used columns going to the end of the
// slots in use.  The pivot row goes through shared memory once a step.  A step
// is a chain (search, reciprocal, row, update) of a few hundred cycles: every
// slot is worked on without a test (branches a group of slots made it twice as
// long), so the instances hold the next larger number of slots.
// Measured, LU -> this (with the assembly in order of terms and the work of
// the temperature once a node): 8,192 systems of 74 unknowns 2.29 -> 0.85 ms,
// 8,192 of 39 1.51 -> 0.43 ms, 1,024 of 14 72 -> 26 us.  Of the 74 x 74
// systems' time some two thirds are the elimination (issue slots; with its 60
// multiply-adds a warp and step in packed pairs 0.92 -> 0.84 ms at the time), the rest
// FP64 work.
//
// Every form below (one warp or four, registers or shared memory) does the
// same operations per element, so that their inverses are the same.

// The pivot row of a column over the rows not done (warp-wide), and the
// reciprocal of its element (0, and not ok, where it is 0, denormal or NaN).
template <int MR>
__device__ __forceinline__ int pivot_row(const float (&col)[MR], unsigned done, int lane, float *recip, bool *ok) {
    unsigned key = 0;
    float v = 0.f;
#pragma unroll
    for (int m = 0; m < MR; m++) {
        const unsigned bits = __float_as_uint(col[m]) & 0x7fffffffu;
        // ordered by modulus, then the first row; a NaN below every number
        const unsigned q = (bits > 0x7f800000u ? 0u : bits & ~127u) | (127u - (unsigned)(lane + 32 * m));
        if (!(done >> m & 1) && q > key) { key = q; v = col[m]; }
    }
    const unsigned top = __reduce_max_sync(0xffffffffu, key);
    const bool good = (key & ~127u) >= 0x00800000u;
    const float d = __shfl_sync(0xffffffffu, good ? rcp_approx(v) : 0.f, (127 - (int)(top & 127u)) & 31);
    if (top < 0x00800000u) *ok = false;
    *recip = d;
    return 127 - (int)(top & 127u);
}

// One step's work of a warp on its slots: the pivot row's lane stages the
// scaled row and clears it (its update, with the multiplier -1, leaves the
// scaled row), then every lane updates its rows.  own_slot holds the pivot
// column, if this warp does (zero by then).
// The row's register is chosen by a branch per register; the markers keep the
// compiler from merging the branches into one that indexes the registers at
// run time, which would put the matrix into local memory.
template <int M, int MR, int NC>
__device__ __forceinline__ void stage_row_of(float (&a)[NC][MR], float (&l)[MR], int pm, float d, int own_slot,
                                             float *row, unsigned &done) {
    if (pm == M) {
        asm volatile("// pivot row in register %0" ::"n"(M));
#pragma unroll
        for (int g = 0; g < NC; g += 4) {
            float4 s = make_float4(a[g][M] * d, a[g + 1][M] * d, a[g + 2][M] * d, a[g + 3][M] * d);
            if (g == 0) {
                if (own_slot == 0) s.x = d;
                if (own_slot == 1) s.y = d;
                if (own_slot == 2) s.z = d;
                if (own_slot == 3) s.w = d;
            }
            *reinterpret_cast<float4 *>(row + g) = s;
            a[g][M] = a[g + 1][M] = a[g + 2][M] = a[g + 3][M] = 0.f;
        }
        l[M] = -1.f;
        done |= 1u << M;
        asm volatile("// staged %0" ::"n"(M));
    }
}
template <int MR, int NC>
__device__ __forceinline__ void stage_row(float (&a)[NC][MR], float (&l)[MR], int p, float d, int own_slot,
                                          float *row, int lane, unsigned &done) {
    if (lane != (p & 31)) return;
    stage_row_of<0, MR, NC>(a, l, p >> 5, d, own_slot, row, done);
    if constexpr (MR > 1) stage_row_of<1, MR, NC>(a, l, p >> 5, d, own_slot, row, done);
    if constexpr (MR > 2) stage_row_of<2, MR, NC>(a, l, p >> 5, d, own_slot, row, done);
}
template <int MR, int NC>
__device__ __forceinline__ void update_group(float (&a)[NC][MR], const float (&l)[MR], const float *row, int g) {
    const float4 s = *reinterpret_cast<const float4 *>(row + g);
#pragma unroll
    for (int m = 0; m < MR; m++) {   // (packed pairs: one issue slot for two multiply-adds)
        const float2 ml = make_float2(-l[m], -l[m]);
        const float2 p = __ffma2_rn(ml, make_float2(s.x, s.y), make_float2(a[g][m], a[g + 1][m]));
        const float2 q = __ffma2_rn(ml, make_float2(s.z, s.w), make_float2(a[g + 2][m], a[g + 3][m]));
        a[g][m] = p.x;
        a[g + 1][m] = p.y;
        a[g + 2][m] = q.x;
        a[g + 3][m] = q.y;
    }
}
// slots [0, na) turn by R (na a multiple of R)
template <int MR, int NC, int R>
__device__ __forceinline__ void turn_slots(float (&a)[NC][MR], int na) {
    float t[R][MR];
#pragma unroll
    for (int q = 0; q < R; q++)
#pragma unroll
        for (int m = 0; m < MR; m++) t[q][m] = a[q][m];
#pragma unroll
    for (int c = 0; c < NC; c += R)
#pragma unroll
        for (int q = 0; q < R; q++)
#pragma unroll
            for (int m = 0; m < MR; m++) {
                const float next = c + R + q < NC ? a[(c + R + q) % NC][m] : 0.f;
                a[c + q][m] = c + R == na ? t[q][m] : next;
            }
}

// Shared memory of a team (see se_gauss_bytes).
struct GaussMem {
    float *row;    // [8 nq] staged pivot rows, two per warp
    float *z;      // [4 nq] permuted residual
    double *feat, *x, *val;
    float *valf;   // [nnz + 1] scaled entries, 0
    float *scl;    // [n]
    float *part;   // [4 n] partial products
    float *lcol;   // [2][n32] published pivot columns
    float *pd;     // [2][4] pivot row, 1 / pivot, ok
    int *rmax, *kof;
    float *dense;  // [n n] the inverse of the shared-memory form
};
// columns a warp of four holds in an instance (a quarter of them all), which
// sizes its staged rows
template <int TW, int NC>
constexpr int gauss_quads = NC == 0 ? SE_GAUSS_DIM / 4 : NC * TW / 4;
__host__ __device__ inline size_t se_gauss_bytes(int n, int n_feat, int nnz, int nq, bool dense) {
    size_t b = sizeof(float) * 12 * (size_t)nq;
    b += sizeof(double) * ((size_t)n_feat + (size_t)n + (size_t)nnz);
    b += sizeof(float) * ((size_t)nnz + 1 + 7 * (size_t)n + 2 * (size_t)((n + 31) & ~31) + 8);
    if (dense) b += sizeof(float) * (size_t)n * n;
    return (b + 15) & ~(size_t)15;
}
__device__ __forceinline__ GaussMem gauss_mem(unsigned char *base, int n, int n_feat, int nnz, int nq) {
    GaussMem g;
    g.row = (float *)base;
    g.z = g.row + 8 * nq;
    g.feat = (double *)(g.z + 4 * nq);
    g.x = g.feat + n_feat;
    g.val = g.x + n;
    g.valf = (float *)(g.val + nnz);
    g.scl = g.valf + nnz + 1;
    g.part = g.scl + n;
    g.lcol = g.part + 4 * n;
    g.pd = g.lcol + 2 * ((n + 31) & ~31);
    g.rmax = (int *)(g.pd + 8);
    g.kof = g.rmax + n;
    g.dense = (float *)(g.kof + n);
    return g;
}

// The elimination in registers; kof[p] = k.  False where a pivot was 0 or NaN.
template <int TW, int MR, int NC>
__device__ __forceinline__ bool gauss_registers(int n, float (&a)[NC][MR], const GaussMem &g, int lane, int w) {
    constexpr int nq = gauss_quads<TW, NC>;
    unsigned done = 0;
#pragma unroll
    for (int m = 0; m < MR; m++)
        if (lane + 32 * m >= n) done |= 1u << m;
    bool ok = true;
    if constexpr (TW == 1) {
        const int na = (n + 3) & ~3;
        float *buf = g.row;
        for (int k0 = 0; k0 < n; k0 += 4) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int k = k0 + q;
                if (k < n) {
                    float l[MR], d;
                    const int p = pivot_row<MR>(a[q], done, lane, &d, &ok);
#pragma unroll
                    for (int m = 0; m < MR; m++) { l[m] = a[q][m]; a[q][m] = 0.f; }
                    float *row = buf + (k & 1) * 4 * nq;
                    if (lane == (p & 31)) g.kof[p] = k;
                    stage_row<MR, NC>(a, l, p, d, q, row, lane, done);
                    __syncwarp();
#pragma unroll
                    for (int c = 0; c < NC; c += 4) update_group<MR, NC>(a, l, row, c);
                }
            }
            turn_slots<MR, NC, 4>(a, na);
        }
        __syncwarp();
    } else {
        const int na = (n + TW - 1) / TW, n32 = (n + 31) & ~31;
        auto publish = [&](const float (&col)[MR], int b) {
            float d;
            bool good = true;
            const int p = pivot_row<MR>(col, done, lane, &d, &good);
#pragma unroll
            for (int m = 0; m < MR; m++)
                if (32 * m < n32) g.lcol[b * n32 + lane + 32 * m] = col[m];
            if (lane == 0) {
                g.pd[4 * b] = __int_as_float(p);
                g.pd[4 * b + 1] = d;
                g.pd[4 * b + 2] = good ? 1.f : 0.f;
            }
        };
        if (w == 0) publish(a[0], 0);
        for (int c0 = 0; c0 < na; c0++) {
            for (int q = 0; q < TW; q++) {
                const int k = TW * c0 + q;
                if (k >= n) break;
                // the pivot column of step k is published; the other buffer's
                // readers (step k - 1) are done
                __syncthreads();
                const int b = k & 1;
                const int p = __float_as_int(g.pd[4 * b]);
                const float d = g.pd[4 * b + 1];
                if (g.pd[4 * b + 2] == 0.f) ok = false;
                float l[MR];
#pragma unroll
                for (int m = 0; m < MR; m++) l[m] = (32 * m < n32) ? g.lcol[b * n32 + lane + 32 * m] : 0.f;
                if (w == q)
#pragma unroll
                    for (int m = 0; m < MR; m++) a[0][m] = 0.f;
                float *row = g.row + (2 * w + b) * nq;
                if (w == 0 && lane == 0) g.kof[p] = k;
                stage_row<MR, NC>(a, l, p, d, w == q ? 0 : -1, row, lane, done);
                __syncwarp();
                update_group<MR, NC>(a, l, row, 0);
                // the next pivot column first, so that its search overlaps the
                // other warps' updates
                if (k + 1 < n && w == (q + 1) % TW) {
                    float col[MR];
#pragma unroll
                    for (int m = 0; m < MR; m++) col[m] = (q == TW - 1) ? a[1][m] : a[0][m];
                    publish(col, b ^ 1);
                }
#pragma unroll
                for (int c = 4; c < NC; c += 4) update_group<MR, NC>(a, l, row, c);
            }
            turn_slots<MR, NC, 1>(a, na);
        }
        __syncthreads();
    }
    return ok;
}

// The elimination in shared memory, one warp (systems its registers cannot
// hold).  a is column-major; row [4 quads] stages the pivot row.
template <int MR>
__device__ bool gauss_shared(int n, float *a, float *row, int *kof, int lane) {
    unsigned done = 0;
#pragma unroll
    for (int m = 0; m < MR; m++)
        if (lane + 32 * m >= n) done |= 1u << m;
    bool ok = true;
    for (int k = 0; k < n; k++) {
        float l[MR], d;
#pragma unroll
        for (int m = 0; m < MR; m++) {
            const int i = lane + 32 * m;
            l[m] = (i < n) ? a[i + n * k] : 0.f;
            if (i < n) a[i + n * k] = 0.f;
        }
        const int p = pivot_row<MR>(l, done, lane, &d, &ok);
        if (lane == (p & 31)) {
            kof[p] = k;
            done |= 1u << (p >> 5);
        }
        __syncwarp();
        for (int j = lane; j < n; j += 32) {
            row[j] = (j == k) ? d : a[p + n * j] * d;
            a[p + n * j] = 0.f;
        }
#pragma unroll
        for (int m = 0; m < MR; m++)
            if (lane + 32 * m == p) l[m] = -1.f;
        __syncwarp();
#pragma unroll
        for (int m = 0; m < MR; m++) {
            float *ai = a + lane + 32 * m;
            if (lane + 32 * m >= n) break;
            int j = 0;
            for (; j + 3 < n; j += 4) {
                const float a0 = ai[n * j], a1 = ai[n * (j + 1)], a2 = ai[n * (j + 2)], a3 = ai[n * (j + 3)];
                const float4 s = *reinterpret_cast<const float4 *>(row + j);
                ai[n * j] = fmaf(-l[m], s.x, a0);
                ai[n * (j + 1)] = fmaf(-l[m], s.y, a1);
                ai[n * (j + 2)] = fmaf(-l[m], s.z, a2);
                ai[n * (j + 3)] = fmaf(-l[m], s.w, a3);
            }
            for (; j < n; j++) ai[n * j] = fmaf(-l[m], row[j], ai[n * j]);
        }
        __syncwarp();
    }
    return ok;
}

// A team of TW warps per node.  TW = 1: every warp of the block is a team;
// TW > 1: the block is one team.
// BATCH: the work items are (model, node) pairs of many models (SEBatch); each
// team copies its current model's argument block into shared memory, and the
// dynamic shared memory per team fits the largest model.
// Otherwise the nodes of the one model a0.
// NC >= 0: the inverse by Gauss-Jordan elimination, in registers (NC slots of
// MR rows a lane) or, NC = 0, in shared memory.  NC = -1: LU factors of up to
// 32 MR rows in shared memory, the triangular solves on the team's first warp.
// Blocks per SM: what the matrix's registers leave room for.
template <int TW, int MR, int NC>
constexpr int se_min_blocks() {
    return NC < 0 ? (TW == 1 ? 3 : 24 / TW) : TW == 1 ? 3 : MR * NC > 64 ? 4 : MR * NC > 32 ? 5 : 8;
}
template <int TW, bool BATCH, int MR, int NC>
__global__ void __launch_bounds__(TW == 1 ? 256 : 32 * TW, se_min_blocks<TW, MR, NC>()) k_solve_se(SEArgs a0, SEBatch bw) {
    static_assert(TW == 1 || NC != 0, "the shared-memory elimination is one warp's");
    constexpr bool GAUSS = NC >= 0;
    constexpr int nq = GAUSS ? gauss_quads<TW, NC> : 0;
    constexpr int TS = 32 * TW;   // threads per team
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ SEArgs margs[BATCH && TW == 1 ? 8 : 1];
    __shared__ double red_v[TW];  // cross-warp reductions of a team
    __shared__ int red_i[TW];
    __shared__ unsigned red_k[2 * TW];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int tid = (TW == 1) ? lane : (int)threadIdx.x;    // thread within the team
    const int teams = (TW == 1) ? (int)(blockDim.x >> 5) : 1;
    const int team = (TW == 1) ? wib : 0;
    auto tsync = [&]() {
        if constexpr (TW == 1) __syncwarp();
        else __syncthreads();
    };
    // the largest of two keys each over the team
    auto team_max2 = [&](unsigned &k0, unsigned &k1) {
        k0 = __reduce_max_sync(0xffffffffu, k0);
        k1 = __reduce_max_sync(0xffffffffu, k1);
        if constexpr (TW > 1) {
            if (lane == 0) { red_k[2 * wib] = k0; red_k[2 * wib + 1] = k1; }
            __syncthreads();
#pragma unroll
            for (int q = 0; q < TW; q++) {
                k0 = max(k0, red_k[2 * q]);
                k1 = max(k1, red_k[2 * q + 1]);
            }
        }
    };
    const long long n_items = BATCH ? bw.n_items : (long long)a0.bulk;
    const size_t wbytes = BATCH   ? bw.team_bytes
                          : GAUSS ? se_gauss_bytes(a0.c_dim, a0.n_feat, a0.nnz, nq, NC == 0)
                                  : se_warp_bytes(a0.c_dim, a0.n_feat);
    unsigned char *base = smem + wbytes * team;
    double *const slot = (BATCH ? bw.a64 : a0.a64) +
                         (size_t)((long long)blockIdx.x * teams + team) * (BATCH ? bw.a64_stride : a0.a64_stride);
    int cur_model = -1;

    // (nodes go to the blocks in turn, so that few nodes spread over the SMs)
    for (long long item = (long long)team * gridDim.x + blockIdx.x; item < n_items; item += (long long)gridDim.x * teams) {
        int node;
        if (BATCH) {
            const int2 wi = bw.items[item];
            if (wi.x != cur_model) {
                tsync();
                const int *src = reinterpret_cast<const int *>(bw.models + wi.x);
                int *dst = reinterpret_cast<int *>(&margs[team]);
                for (int k = tid; k < (int)(sizeof(SEArgs) / sizeof(int)); k += TS) dst[k] = src[k];
                tsync();
                cur_model = wi.x;
            }
            node = wi.y;
        } else {
            node = (int)item;
        }
        const SEArgs &a = BATCH ? margs[team] : a0;
        const int n = a.c_dim;
        const GaussMem gm = GAUSS ? gauss_mem(base, n, a.n_feat, a.nnz, nq) : GaussMem{};
        double *feat = GAUSS ? gm.feat : (double *)base;
        double *x = GAUSS ? gm.x : feat + (size_t)a.n_feat;
        double *val = GAUSS ? gm.val : slot;
        float *LU = (float *)(x + n);
        float *d32 = LU + (size_t)n * n;
        float *scl = GAUSS ? gm.scl : d32 + n;
        int *piv = GAUSS ? gm.kof : (int *)(scl + n);
        // a pass of the iterated node loop with failed walks: the last good
        // pass's populations stay (asked once a node: before the loop it cost the
        // 74 x 74 systems' registers, 0.84 -> 0.88 ms)
        if (!BATCH && a.skip && *a.skip) return;
        if (!(a.ab[node] > 0.0)) {  // main_para.f90:213 (pops and alignments stay 0)
            if (!BATCH) {
                for (int c2 = tid; c2 < 2 * a.nlev; c2 += TS) a.pops[(size_t)node + (size_t)a.N * c2] = 0.0;
                for (int l = tid; l < a.L; l += TS) a.jj20[(size_t)node + (size_t)a.N * l] = 0.0;
            }
            continue;
        }
        const double T = a.tkin[node], nH2 = a.h2[node];
        // ---- features (make_AC miscellaneous.f90:331-390) ----
        // What depends on the temperature alone once per node: an FP64
        // instruction of a warp takes the SM 16 cycles.
        // Temperature interpolation (first bracket; below the table the first
        // bracket extrapolates, as the reference's loop does)
        int ib = 0;   // the first i >= 1 with col_temps[i] > T, 0: none
        for (int i0 = 1; i0 < a.c_temp && !ib; i0 += 32) {
            const unsigned above = __ballot_sync(0xffffffffu, i0 + lane < a.c_temp && a.col_temps[i0 + lane] > T);
            if (above) ib = i0 + __ffs(above) - 1;
        }
        double ddT = 0.0;
        if (ib) ddT = (T - a.col_temps[ib - 1]) / (a.col_temps[ib] - a.col_temps[ib - 1]);
        const bool below = a.c_temp > 0 && T <= a.col_temps[0];
        const double rT = 1.0 / T;
        if constexpr (GAUSS)
            for (int i = tid; i < n; i += TS) gm.rmax[i] = 0;
        for (int t = tid; t < a.n_trans; t += TS) {
            const int rr = a.tr_rad[t], cc = a.tr_col[t];
            const double B21 = a.tr_B21[t], A21 = a.tr_A[t];
            double f0 = 0.0, f1 = 0.0, f5 = 0.0, f6 = A21, C21 = 0.0;
            if (rr >= 0) {
                f0 = B21 * a.J0[(size_t)node * a.L + rr];
                f1 = B21 * a.J2[(size_t)node * a.L + rr];
                f5 = a.JE ? B21 * a.JE[(size_t)node * a.L + rr] : f0;
                if (a.LS) f6 = A21 * (1.0 - a.LS[(size_t)node * a.L + rr]);
            }
            if (cc >= 0) {
                const int nT = a.c_temp;
                double cr = 0.0;
                for (int p = 0; p < a.c_par; p++) {
                    const double *Ct = a.Cji + (size_t)nT * (cc + (size_t)a.c_num * p);
                    double v = below ? Ct[0] : 0.0;
                    if (ib) v = Ct[ib - 1] + ddT * (Ct[ib] - Ct[ib - 1]);
                    cr += (a.c_par == 2 ? (p == 0 ? 0.25 : 0.75) : 1.0) * v;
                }
                C21 = cr * nH2 * 1e-6;
            }
            // -h nu / k T: the product with 1 / T, one step of the remainder
            const double hn = -HK * a.tr_nu[t];
            double e = hn * rT;
            const double rem = fma(-e, T, hn);
            if (rem - rem == 0.0) e = fma(rem, rT, e);
            double *f = feat + NF * (size_t)t;
            f[0] = f0;
            f[1] = f1;
            f[2] = A21;
            f[3] = C21;
            f[4] = C21 * exp(e);
            f[5] = f5;
            f[6] = f6;
        }
        if (a.depol) {
            // make_depolarization_temp: every bracket with col_temps(i) > T
            // overwrites D0 (the loop has no exit), so the last bracket
            // decides below the table's top; at or above it the reference
            // leaves D0 unset (0 here)
            const int nT = a.c_temp;
            const double *ct = a.col_temps;
            for (int d = tid; d < a.n_dep; d += TS) {
                const double *tab = a.dep_tab + (size_t)nT * d;
                double v = 0.0;
                if (T <= ct[0]) v = tab[0];
                if (nT >= 2 && ct[nT - 1] > T) {
                    const double ddT = (T - ct[nT - 2]) / (ct[nT - 1] - ct[nT - 2]);
                    v = tab[nT - 2] + ddT * (tab[nT - 1] - tab[nT - 2]);
                }
                v = v * nH2 * 1e-6;
                feat[NF * (size_t)a.n_trans + d] = v;
                if (a.depol == 2) feat[NF * (size_t)a.n_trans + a.n_dep + d] = v;
            }
        }
        if constexpr (!GAUSS)
            if (!a.fp64_only)
                for (int i = tid; i < n * n; i += TS) LU[i] = 0.f;
        tsync();
        // ---- assembly (setup_stateq), row 1 replaced by the normalisation
        // (em_coefs.f90:158-164): the entries with the most terms first, so
        // that the lanes of a warp have equally many; four records per thread
        // in flight; each entry's terms summed in program order
        for (int e0 = tid; e0 < a.nnz; e0 += 4 * TS) {
            int4 rec[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int e = e0 + u * TS;
                rec[u] = (e < a.nnz) ? a.sp_rec[e] : make_int4(-1, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (rec[u].x < 0) continue;
                double v = 0.0;
                if (rec[u].w >= 0) v = a.norm_val[rec[u].w];
                else {
                    const int q1 = rec[u].y + (int)((unsigned)rec[u].z >> 16);
                    int q = rec[u].y;
                    for (; q + 3 < q1; q += 4) {
                        const double c0 = a.term_c[q], c1 = a.term_c[q + 1], c2 = a.term_c[q + 2], c3 = a.term_c[q + 3];
                        const int f0 = a.term_f[q], f1 = a.term_f[q + 1], f2 = a.term_f[q + 2], f3 = a.term_f[q + 3];
                        v = fma(c0, feat[f0], v);
                        v = fma(c1, feat[f1], v);
                        v = fma(c2, feat[f2], v);
                        v = fma(c3, feat[f3], v);
                    }
                    for (; q < q1; q++) v = fma(a.term_c[q], feat[a.term_f[q]], v);
                }
                val[rec[u].z & 0xffff] = v;
                if constexpr (GAUSS)
                    if (v == v) atomicMax(&gm.rmax[rec[u].x & 0xffff], __double2hiint(v) & 0x7fffffff);
            }
        }
        tsync();
        int st = 0;
        bool ok = false, conv = false;
        if constexpr (GAUSS) {
            // ---- FP32 inverse of the matrix, its rows scaled by powers of two
            // to a largest modulus in [1, 2) ----
            float m[NC > 0 ? NC : 1][MR];
            if (!a.fp64_only) {
                for (int i = tid; i < n; i += TS) {
                    const int e = gm.rmax[i] >> 20;
                    scl[i] = e == 0 ? 1.f : e >= 2046 ? 0.f : (float)__hiloint2double((2046 - e) << 20, 0);
                }
                for (int q = tid; q < a.nnz; q += TS) {
                    const int4 rec = a.sp_rec[q];
                    const int e = gm.rmax[rec.x & 0xffff] >> 20, dst = rec.z & 0xffff;
                    const double sc = e == 0 ? 1.0 : e >= 2046 ? 0.0 : __hiloint2double((2046 - e) << 20, 0);
                    gm.valf[dst] = (float)(val[dst] * sc);
                }
                if (tid == 0) gm.valf[a.nnz] = 0.f;
                for (int i = tid; i < 4 * nq; i += TS) gm.z[i] = 0.f;
                tsync();
                if constexpr (NC > 0) {
#pragma unroll
                    for (int c = 0; c < NC; c++) {
                        const int j = (TW == 1 ? 0 : wib) + TW * c;
#pragma unroll
                        for (int u = 0; u < MR; u++) {
                            const int i = lane + 32 * u;
                            m[c][u] = (i < n && j < n) ? gm.valf[a.sp_map[i + n * j]] : 0.f;
                        }
                    }
                    ok = gauss_registers<TW, MR, NC>(n, m, gm, lane, TW == 1 ? 0 : wib);
                } else {
                    for (int i = lane; i < n * n; i += 32) gm.dense[i] = gm.valf[a.sp_map[i]];
                    __syncwarp();
                    ok = gauss_shared<MR>(n, gm.dense, gm.row, gm.kof, lane);
                }
            }
            if (ok) {
                for (int i = tid; i < n; i += TS) x[i] = 0.0;
                double dprev = 1e300;
                for (int it = 0; it < 10; it++) {
                    // r = e_1 - A x (FP64; x = 0 at first), at its pivot's place
                    for (int i = tid; i < n; i += TS) {
                        double s = (i == 0) ? 1.0 : 0.0;
                        if (it) {
                            double s1 = 0.0;   // two chains of dependent FP64 sums
                            int q = a.sp_off[i];
                            const int q1 = a.sp_off[i + 1];
                            for (; q + 1 < q1; q += 2) {
                                s -= val[q] * x[a.sp_col[q]];
                                s1 -= val[q + 1] * x[a.sp_col[q + 1]];
                            }
                            if (q < q1) s -= val[q] * x[a.sp_col[q]];
                            s += s1;
                        }
                        const int k = gm.kof[i];
                        const int zi = (NC > 0 && TW > 1) ? (k % TW) * nq + k / TW : k;
                        gm.z[zi] = (float)(s * (double)scl[i]);
                    }
                    tsync();
                    // the correction: row i of the inverse gives x[kof[i]]; its
                    // terms in four sums, by column j % 4
                    float cor[MR];
                    if constexpr (NC > 0 && TW == 1) {
#pragma unroll
                        for (int u = 0; u < MR; u++) cor[u] = 0.f;
                        float p4[MR][4] = {};
#pragma unroll
                        for (int c = 0; c < NC; c += 4) {
                            const float4 zz = *reinterpret_cast<const float4 *>(gm.z + c);
#pragma unroll
                            for (int u = 0; u < MR; u++) {
                                p4[u][0] = fmaf(m[c][u], zz.x, p4[u][0]);
                                p4[u][1] = fmaf(m[c + 1][u], zz.y, p4[u][1]);
                                p4[u][2] = fmaf(m[c + 2][u], zz.z, p4[u][2]);
                                p4[u][3] = fmaf(m[c + 3][u], zz.w, p4[u][3]);
                            }
                        }
#pragma unroll
                        for (int u = 0; u < MR; u++) cor[u] = (p4[u][0] + p4[u][1]) + (p4[u][2] + p4[u][3]);
                    } else if constexpr (NC > 0) {
                        float acc[MR] = {};
                        const float *zw = gm.z + wib * nq;
#pragma unroll
                        for (int c = 0; c < NC; c += 4) {
                            const float4 zz = *reinterpret_cast<const float4 *>(zw + c);
#pragma unroll
                            for (int u = 0; u < MR; u++) {
                                acc[u] = fmaf(m[c][u], zz.x, acc[u]);
                                acc[u] = fmaf(m[c + 1][u], zz.y, acc[u]);
                                acc[u] = fmaf(m[c + 2][u], zz.z, acc[u]);
                                acc[u] = fmaf(m[c + 3][u], zz.w, acc[u]);
                            }
                        }
#pragma unroll
                        for (int u = 0; u < MR; u++)
                            if (lane + 32 * u < n) gm.part[wib * n + lane + 32 * u] = acc[u];
                        __syncthreads();
                    } else {
#pragma unroll
                        for (int u = 0; u < MR; u++) {
                            const int i = lane + 32 * u;
                            float p0 = 0.f, p1 = 0.f, p2 = 0.f, p3 = 0.f;
                            if (i < n) {
                                int j = 0;
                                for (; j + 3 < n; j += 4) {
                                    p0 = fmaf(gm.dense[i + n * j], gm.z[j], p0);
                                    p1 = fmaf(gm.dense[i + n * (j + 1)], gm.z[j + 1], p1);
                                    p2 = fmaf(gm.dense[i + n * (j + 2)], gm.z[j + 2], p2);
                                    p3 = fmaf(gm.dense[i + n * (j + 3)], gm.z[j + 3], p3);
                                }
                                if (j < n) p0 = fmaf(gm.dense[i + n * j], gm.z[j], p0);
                                if (j + 1 < n) p1 = fmaf(gm.dense[i + n * (j + 1)], gm.z[j + 1], p1);
                                if (j + 2 < n) p2 = fmaf(gm.dense[i + n * (j + 2)], gm.z[j + 2], p2);
                            }
                            cor[u] = (p0 + p1) + (p2 + p3);
                        }
                    }
                    unsigned kd = 0, kx = 0;   // largest |correction| (FP32) and |x| (upper word)
                    auto apply = [&](int i, float d) {
                        const int k = gm.kof[i];
                        const double xv = x[k] + (double)d;
                        x[k] = xv;
                        kd = max(kd, __float_as_uint(fabsf(d)));
                        kx = max(kx, (unsigned)__double2hiint(xv) & 0x7fffffffu);
                    };
                    if constexpr (TW == 1) {
#pragma unroll
                        for (int u = 0; u < MR; u++)
                            if (lane + 32 * u < n) apply(lane + 32 * u, cor[u]);
                    } else {
                        for (int i = tid; i < n; i += TS)
                            apply(i, (gm.part[i] + gm.part[n + i]) + (gm.part[2 * n + i] + gm.part[3 * n + i]));
                    }
                    team_max2(kd, kx);
                    if (TW == 1) __syncwarp();
                    if (kd >= 0x7f800000u || kx >= 0x7ff00000u) break;  // infinite or NaN
                    const double dm = (double)__uint_as_float(kd), xmax = __hiloint2double((int)kx, 0);
                    // converged: the correction is at the level FP64 residuals can
                    // resolve (~cond(SA) * eps), or it stopped shrinking there.  (The
                    // norms are compared only: |x| by its upper word, the correction as
                    // the FP32 number it is.)
                    if (dm <= 2e-14 * xmax) { conv = true; break; }
                    if (it >= 2 && dm <= 1e-12 * xmax && dm > 0.5 * dprev) { conv = true; break; }
                    dprev = dm;
                }
            }
        } else {
            // ---- FP32 LU of the row-scaled matrix (skipped in FP64 mode) ----
            if (!a.fp64_only) {
                for (int i = tid; i < n; i += TS) {
                    double m = 0.0;
                    for (int q = a.sp_off[i]; q < a.sp_off[i + 1]; q++) m = fmax(m, fabs(val[q]));
                    const float sc = (m > 0.0) ? (float)(1.0 / m) : 1.f;
                    scl[i] = sc;
                    for (int q = a.sp_off[i]; q < a.sp_off[i + 1]; q++)
                        LU[i + (size_t)n * a.sp_col[q]] = (float)(val[q] * (double)sc);
                }
                tsync();
                ok = team_lu<float, TW, MR>(n, LU, piv, tid, red_v, red_i);
            }
            if (ok) {
                for (int i = tid; i < n; i += TS) x[i] = 0.0;
                tsync();
                double dprev = 1e300;
                for (int it = 0; it < 10; it++) {
                    // r = e_1 - A x (FP64)
                    for (int i = tid; i < n; i += TS) {
                        double s = (i == 0) ? 1.0 : 0.0, s1 = 0.0;   // two chains of dependent FP64 sums
                        int q = a.sp_off[i];
                        const int q1 = a.sp_off[i + 1];
                        for (; q + 1 < q1; q += 2) {
                            s -= val[q] * x[a.sp_col[q]];
                            s1 -= val[q + 1] * x[a.sp_col[q + 1]];
                        }
                        if (q < q1) s -= val[q] * x[a.sp_col[q]];
                        d32[i] = (float)((s + s1) * (double)scl[i]);
                    }
                    tsync();
                    if (TW == 1 || wib == 0) warp_lu_solve<float, float, MR>(n, LU, piv, d32, lane);
                    tsync();
                    unsigned kd = 0, kx = 0;   // largest |correction| (FP32) and |x| (upper word)
                    for (int i = tid; i < n; i += TS) {
                        const double xv = x[i] + (double)d32[i];
                        x[i] = xv;
                        kd = max(kd, __float_as_uint(fabsf(d32[i])));
                        kx = max(kx, (unsigned)__double2hiint(xv) & 0x7fffffffu);
                    }
                    team_max2(kd, kx);
                    if (TW == 1) __syncwarp();
                    if (kd >= 0x7f800000u || kx >= 0x7ff00000u) break;  // infinite or NaN
                    const double dm = (double)__uint_as_float(kd), xmax = __hiloint2double((int)kx, 0);
                    if (dm <= 2e-14 * xmax) { conv = true; break; }
                    if (it >= 2 && dm <= 1e-12 * xmax && dm > 0.5 * dprev) { conv = true; break; }
                    dprev = dm;
                }
            }
        }
        if (!conv) {
            // FP64 LU on the device, dense
            double *M = slot + a.nnz;
            for (int i = tid; i < n * n; i += TS) M[i] = 0.0;
            tsync();
            for (int q = tid; q < a.nnz; q += TS) {
                const int4 rec = a.sp_rec[q];
                M[(rec.x & 0xffff) + (size_t)n * (rec.x >> 16)] = val[rec.z & 0xffff];
            }
            tsync();
            st |= ok ? PORTAL_NODE_REFINE : 0;
            bool ok64 = team_lu<double, TW, MR>(n, M, piv, tid, red_v, red_i);
            if (!ok64) {
                st |= PORTAL_NODE_SINGULAR;
            } else {
                for (int i = tid; i < n; i += TS) x[i] = (i == 0) ? 1.0 : 0.0;
                tsync();
                if (TW == 1 || wib == 0) warp_lu_solve<double, double, MR>(n, M, piv, x, lane);
                tsync();
                st |= PORTAL_NODE_REFINE;
            }
        }
        tsync();
        // ---- packing (main_sub.f90:112-137): a NaN population zeroes both ----
        for (int l = tid; l < a.nlev; l += TS) {
            const int p0 = a.pack[2 * l], p1 = a.pack[2 * l + 1];
            const bool solved = !(st & PORTAL_NODE_SINGULAR);
            double v0 = (p0 >= 0 && solved) ? x[p0] : 0.0, v1 = (p1 >= 0 && solved) ? x[p1] : 0.0;
            if (v0 != v0) v0 = v1 = 0.0;
            a.pops[(size_t)node + (size_t)a.N * (2 * l)] = v0;
            a.pops[(size_t)node + (size_t)a.N * (2 * l + 1)] = v1;
        }
        if (a.rates) {
            // extra_info rates (em_coefs.f90:188-198): per component i and kind
            // k (spontaneous, radiative, collisional), sum_j |M_k(i,j)| rho_j,
            // M_k the part of setup_stateq's matrix from A, from B J, from C
            // (pop_eqs.f90:424-426, 510-512, 558-559, 599-645); the unsplit
            // field's values (f0, f2) stand for f5, f6.  Each sum in ascending
            // column order, as the reference's; the three kinds' sums together over
            // the team's threads (4,000 systems of 33 unknowns with rates 0.73 ms;
            // kind by kind, 95 of 128 threads idle, 1.55, one warp a node 1.48).
            double *r3 = slot + a.nnz;   // (the FP64 fallback is done with it)
            for (int q3 = tid; q3 < 3 * n; q3 += TS) {
                const int k = q3 / n, i = q3 - k * n;
                double acc = 0.0;
                if (!(st & PORTAL_NODE_SINGULAR))
                    for (int q = a.row_off[i]; q < a.row_off[i + 1]; q++) {
                        const int e = a.row_ent[q];
                        double v = 0.0;
                        for (int t = a.ent_off[e]; t < a.ent_off[e + 1]; t++) {
                            const int tf = a.term_f[t];
                            if (tf >= NF * a.n_trans) {
                                // depolarisation: C_mat where col_dep is assigned; the
                                // carried copies (mode 2) are in Amat only
                                if (k == 2 && tf < NF * a.n_trans + a.n_dep) v += a.term_c[t] * feat[tf];
                                continue;
                            }
                            const int f = tf % NF, base = tf - f;
                            const int kind = (f == 2 || f == 6) ? 0 : (f == 3 || f == 4) ? 2 : 1;
                            if (kind != k) continue;
                            const int fu = (f == 5) ? 0 : (f == 6) ? 2 : f;
                            v += a.term_c[t] * feat[base + fu];
                        }
                        acc += fabs(v) * x[a.ent_pos[e] / n];
                    }
                r3[q3] = acc;
            }
            tsync();
            // packing as the populations (main_sub.f90:116-135): K = 2
            // components of J = 0 levels are 0; a NaN population zeroes the
            // K = 2 rate entry (twice, as in the reference)
            for (int q3 = tid; q3 < 6 * a.nlev; q3 += TS) {
                const int k = q3 / (2 * a.nlev), c2 = q3 - k * 2 * a.nlev;
                const int pidx = a.pack[c2];
                double v = (pidx >= 0) ? r3[k * n + pidx] : 0.0;
                if (c2 & 1) {
                    const double p0 = x[a.pack[c2 - 1]];
                    if (p0 != p0) v = 0.0;
                }
                a.rates[(size_t)node + (size_t)a.N * (k + 3 * (size_t)c2)] = v;
            }
        }
        if (a.jj20)
            for (int l = tid; l < a.L; l += TS)
                a.jj20[(size_t)node + (size_t)a.N * l] =
                    a.J2[(size_t)node * a.L + l] / a.J0[(size_t)node * a.L + l];
        if (tid == 0) {
            a.status[node] |= st;
            if (st & PORTAL_NODE_SINGULAR) atomicAdd(a.nfail, 1);
        }
        tsync();
    }
    if (!BATCH && !(a0.skip && *a0.skip)) {
        // the boundary nodes' rows are 0
        const int nb = a0.N - a0.bulk, cols = 2 * a0.nlev + a0.L;
        const long long total = (long long)nb * cols;
        for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < total;
             q += (long long)gridDim.x * blockDim.x) {
            const int col = (int)(q / nb), i = a0.bulk + (int)(q % nb);
            if (col < 2 * a0.nlev) a0.pops[(size_t)i + (size_t)a0.N * col] = 0.0;
            else a0.jj20[(size_t)i + (size_t)a0.N * (col - 2 * a0.nlev)] = 0.0;
        }
    }
}

// ---- host: the program ---------------------------------------------------

struct Program {
    int c_dim = 0, n_trans = 0, n_dep = 0;
    std::vector<int> count_array, tr_lo, tr_up, tr_rad, tr_col;
    std::vector<double> tr_nu, tr_A, tr_B21;
    std::vector<int> ent_off, ent_pos, term_f, pack, row_off, row_ent;
    std::vector<double> term_c;
    std::vector<double> dep_tab;   // (c_temp, n_dep) depolarisation coefficients
};

// de_polarization depol.f90:242-317 (Morris 1985 Eq. B11, the D^(K) of
// L&L04 Eq. 7.102) for level i (J = i - 1, the reference's assumption) and
// rank K at collision temperature l:
//   (2J+1)^2 sum_{m=1..2J} (-1)^m (2m+1) (J J m; 0 0 0)^2
//            ({J J m; J J 0} - {J J m; J J K}) C_j0(l, m)
// with C_j0(:, m) the first partner's rate of the collisional transition
// from level 1 to level m, 0 for m = 1 (the reference never sets it) and
// for m beyond the levels (the reference reads past its array there).
double depol_coefficient(const portal_ctx *c, int i, int K, int l) {
    const int j = i - 1, nT = c->c_temp;
    const double lj2 = std::pow(2.0 * j + 1.0, 2.0);
    double s = 0.0;
    for (int m = 1; m <= 2 * j; m++) {
        double cj = 0.0;
        if (m <= c->nlev)
            for (int q = 0; q < c->c_num; q++)
                if (c->c_trans[2 * q] == 1 && c->c_trans[2 * q + 1] == m) cj = c->Cji[l + (size_t)nT * q];
        const double fac = std::pow(-1.0, m) * (2.0 * m + 1.0);
        const double w1 = wigner3j(2 * j, 2 * j, 2 * m, 0, 0, 0);
        const double w2 = wigner6j(2 * j, 2 * j, 2 * m, 2 * j, 2 * j, 0);
        const double w3 = wigner6j(2 * j, 2 * j, 2 * m, 2 * j, 2 * j, 2 * K);
        s = s + lj2 * fac * w1 * w1 * (w2 - w3) * cj;
    }
    return s;
}

void build_program(const portal_ctx *c, int kmax, Program &P) {
    const int nlev = c->nlev;
    const std::vector<int> &J = c->j_lev;
    // setup_count_array miscellaneous.f90:206-239
    P.count_array.assign(nlev, 0);
    int cnt = 0;
    for (int i = 0; i < nlev; i++) {
        P.count_array[i] = cnt;
        for (int k = 0; k <= std::min(2 * J[i], kmax); k += 2) cnt++;
    }
    P.c_dim = cnt;
    // all_transitions miscellaneous.f90:394-460
    std::vector<int> T(nlev * nlev, 0);
    auto mark = [&](int a, int b) {
        if (c->e_levs[b] > c->e_levs[a]) T[a * nlev + b] = 1;
        else T[b * nlev + a] = 1;
    };
    for (int i = 0; i < c->r_num; i++) mark(c->r_trans[2 * i] - 1, c->r_trans[2 * i + 1] - 1);
    for (int i = 0; i < c->c_num; i++) mark(c->c_trans[2 * i] - 1, c->c_trans[2 * i + 1] - 1);
    for (int i = 0; i < nlev; i++)
        for (int j = 0; j < nlev; j++)
            if (T[i * nlev + j]) { P.tr_lo.push_back(i); P.tr_up.push_back(j); }
    P.n_trans = (int)P.tr_lo.size();
    // make_AC's matching (first radiative / collisional entry with the same
    // (lower, upper) ordering)
    for (int t = 0; t < P.n_trans; t++) {
        int lo = P.tr_lo[t], up = P.tr_up[t], rr = -1, cc = -1;
        for (int j = 0; j < c->r_num; j++)
            if (c->r_trans[2 * j] - 1 == lo && c->r_trans[2 * j + 1] - 1 == up) { rr = j; break; }
        for (int j = 0; j < c->c_num; j++)
            if (c->c_trans[2 * j] - 1 == lo && c->c_trans[2 * j + 1] - 1 == up) { cc = j; break; }
        double nu = c->e_levs[up] - c->e_levs[lo];
        double A = rr >= 0 ? c->A[rr] : 0.0;
        P.tr_rad.push_back(rr);
        P.tr_col.push_back(cc);
        P.tr_nu.push_back(nu);
        P.tr_A.push_back(A);
        P.tr_B21.push_back(A_TO_B * A / std::pow(nu, 3.0));
    }
    // coupling-constant cache
    std::map<std::tuple<int, int, int, int, int>, std::pair<double, double>> cache;
    auto cc_get = [&](int which, int j, int k, int j2, int k2) {
        auto key = std::make_tuple(which, j, k, j2, k2);
        auto it = cache.find(key);
        if (it != cache.end()) return it->second;
        double a0, a2;
        coupling_constants(which, j, k, j2, k2, &a0, &a2);
        return cache[key] = std::make_pair(a0, a2);
    };
    const int n = P.c_dim;
    std::vector<int> k_of(n, 0);  // K of each component
    for (int i = 0; i < nlev; i++)
        for (int k = 0; k <= std::min(2 * J[i], kmax); k += 2) k_of[P.count_array[i] + k / 2] = k;
    std::map<int, std::vector<std::pair<int, double>>> ent;  // pos -> terms
    // depolarisation rates: one per (level, K = 2 .. min(2J, kmax))
    std::vector<int> dep_id(nlev, -1);
    P.n_dep = 0;
    if (c->depol) {
        for (int i = 0; i < nlev; i++) {
            dep_id[i] = P.n_dep;
            P.n_dep += std::min(2 * J[i], kmax) / 2;
        }
        P.dep_tab.assign((size_t)c->c_temp * P.n_dep, 0.0);
        for (int i = 0; i < nlev; i++)
            for (int K = 2; K <= std::min(2 * J[i], kmax); K += 2)
                for (int l = 0; l < c->c_temp; l++)
                    P.dep_tab[(size_t)l + (size_t)c->c_temp * (dep_id[i] + K / 2 - 1)] =
                        depol_coefficient(c, i + 1, K, l);
    }
    int cur_dep = -1;  // the (level, K) col_dep holds (the reference's loop order)
    auto add = [&](int c1, int c2, int t, int f, double coef) {
        auto &v = ent[c1 + n * c2];
        // couplings between K = 0 components take the split field (f5, f6)
        const bool k00 = (k_of[c1] == 0 && k_of[c2] == 0);
        const int ff = (k00 && f == 0) ? 5 : (k00 && f == 2) ? 6 : f;
        if (coef != 0.0) v.push_back({NF * t + ff, coef});
    };
    auto touch = [&](int c1, int c2) { ent[c1 + n * c2]; };
    for (int i1 = 0; i1 < nlev; i1++) {
        std::vector<int> up, dn;  // transition ids in the reference's order
        for (int i2 = 0; i2 < nlev; i2++)
            for (int q = 0; q < P.n_trans; q++) {
                if (P.tr_lo[q] == i1 && P.tr_up[q] == i2) up.push_back(q);
                if (P.tr_lo[q] == i2 && P.tr_up[q] == i1) dn.push_back(q);
            }
        const int j1 = J[i1];
        const double g1 = 2.0 * j1 + 1.0;
        const int k1m = std::min(2 * j1, kmax);
        for (int q : up) {  // pop_eqs.f90:467-515
            int i2 = P.tr_up[q], j2 = J[i2];
            double g2 = 2.0 * j2 + 1.0;
            int c1 = P.count_array[i1];
            for (int k1 = 0; k1 <= k1m; k1 += 2, c1++) {
                int c2 = P.count_array[i2];
                for (int k2 = 0; k2 <= std::min(2 * j2, kmax); k2 += 2, c2++) {
                    auto ts = cc_get(1, j1, k1, j2, k2);
                    auto te = cc_get(2, j1, k1, j2, k2);
                    touch(c1, c2);
                    add(c1, c2, q, 0, ts.first);
                    add(c1, c2, q, 1, ts.second);
                    add(c1, c2, q, 2, te.first);
                    if (k1 == k2 && k1 == 0) add(c1, c2, q, 3, std::sqrt(g2 / g1));
                }
            }
        }
        for (int q : dn) {  // pop_eqs.f90:518-562
            int i2 = P.tr_lo[q], j2 = J[i2];
            double g2 = 2.0 * j2 + 1.0;
            int c1 = P.count_array[i1];
            for (int k1 = 0; k1 <= k1m; k1 += 2, c1++) {
                int c2 = P.count_array[i2];
                for (int k2 = 0; k2 <= std::min(2 * j2, kmax); k2 += 2, c2++) {
                    auto ta = cc_get(0, j1, k1, j2, k2);
                    touch(c1, c2);
                    add(c1, c2, q, 0, (g1 / g2) * ta.first);
                    add(c1, c2, q, 1, (g1 / g2) * ta.second);
                    if (k1 == k2 && k1 == 0) add(c1, c2, q, 4, std::sqrt(g2 / g1) * (g1 / g2));
                }
            }
        }
        // diagonal block pop_eqs.f90:564-650
        int c1 = P.count_array[i1];
        for (int k1 = 0; k1 <= k1m; k1 += 2, c1++) {
            int c2 = P.count_array[i1];
            for (int k2 = 0; k2 <= k1m; k2 += 2, c2++) {
                touch(c1, c2);
                // col_dep (pop_eqs.f90:642-648), read after the rates below in
                // the reference; a term's position in the entry's sum does not
                // change the FP64 assembly beyond rounding
                if (c->depol) {
                    if (k1 == k2 && k1 >= 2) {
                        cur_dep = dep_id[i1] + k1 / 2 - 1;
                        ent[c1 + n * c2].push_back({NF * P.n_trans + cur_dep, -1.0});
                    } else if (c->depol == 2 && cur_dep >= 0) {
                        ent[c1 + n * c2].push_back({NF * P.n_trans + P.n_dep + cur_dep, -1.0});
                    }
                }
                for (int q : up) {
                    int j3 = J[P.tr_up[q]];
                    double g3 = 2.0 * j3 + 1.0;
                    auto ra = cc_get(3, j1, k1, j3, k2);
                    add(c1, c2, q, 0, -(g3 / g1) * ra.first);
                    add(c1, c2, q, 1, -(g3 / g1) * ra.second);
                    if (k1 == k2) add(c1, c2, q, 4, -(g3 / g1));
                }
                for (int q : dn) {
                    int j3 = J[P.tr_lo[q]];
                    auto rs = cc_get(4, j1, k1, j3, k2);
                    add(c1, c2, q, 0, -rs.first);
                    add(c1, c2, q, 1, -rs.second);
                    if (k1 == k2) {
                        add(c1, c2, q, 2, -1.0);
                        add(c1, c2, q, 3, -1.0);
                    }
                }
            }
        }
    }
    P.ent_off.assign(1, 0);
    P.ent_pos.clear(); P.term_f.clear(); P.term_c.clear();
    for (auto &kv : ent) {
        P.ent_pos.push_back(kv.first);
        for (auto &tc : kv.second) { P.term_f.push_back(tc.first); P.term_c.push_back(tc.second); }
        P.ent_off.push_back((int)P.term_f.size());
    }
    // the entries of each row in ascending column order (ent is keyed by
    // c1 + n c2: column-major)
    P.row_off.assign(n + 1, 0);
    for (int pos : P.ent_pos) P.row_off[pos % n + 1]++;
    for (int i = 0; i < n; i++) P.row_off[i + 1] += P.row_off[i];
    P.row_ent.assign(P.ent_pos.size(), 0);
    {
        std::vector<int> fill(P.row_off.begin(), P.row_off.end() - 1);
        for (int e = 0; e < (int)P.ent_pos.size(); e++) P.row_ent[fill[P.ent_pos[e] % n]++] = e;
    }
    // packing main_sub.f90:112-129: the alignment of a J != 0 level is the
    // component after its rho^0_0.  With kmax = 0 there is none, and the
    // reference then reads the next level's rho^0_0 (and, for the last
    // level, past the end of rhovec); the first is kept, the read past the
    // end gives 0 here.
    P.pack.assign(2 * nlev, -1);
    for (int i = 0; i < nlev; i++) {
        P.pack[2 * i] = P.count_array[i];
        if (J[i] != 0 && P.count_array[i] + 1 < P.c_dim) P.pack[2 * i + 1] = P.count_array[i] + 1;
    }
}

}  // namespace

namespace portal {

int prepare_se(portal_ctx *c, int kmax) {
    if (c->se_kmax == kmax && c->se_built) return PORTAL_OK;
    if (c->depol)
        for (int i = 0; i < c->nlev; i++)
            if (c->j_lev[i] != i)
                return set_err(c, PORTAL_ERR_ARG, "depolarising collisions need j_lev(i) = i - 1 "
                                                  "(de_polarization's assumption, depol.f90:283)");
    Program P;
    build_program(c, kmax, P);
    // pack ints: tr_rad | tr_col | ent_off | ent_pos | term_f | norm_col | pack | col? ;
    std::vector<int> I;
    std::vector<double> D;
    auto putI = [&](const std::vector<int> &v) { size_t o = I.size(); I.insert(I.end(), v.begin(), v.end()); return o; };
    auto putD = [&](const std::vector<double> &v) { size_t o = D.size(); D.insert(D.end(), v.begin(), v.end()); return o; };
    std::vector<double> norm_val(c->nlev);
    for (int i = 0; i < c->nlev; i++) norm_val[i] = std::sqrt(2.0 * c->j_lev[i] + 1.0);
    size_t o_rad = putI(P.tr_rad), o_col = putI(P.tr_col), o_eoff = putI(P.ent_off),
           o_epos = putI(P.ent_pos), o_tf = putI(P.term_f), o_nc = putI(P.count_array),
           o_pack = putI(P.pack), o_roff = putI(P.row_off), o_rent = putI(P.row_ent);
    // the matrix's entries row by row in ascending column order: row offsets
    // and columns; row 1 is the normalisation's
    struct Rec { int pos, first, count, norm; };
    std::vector<Rec> recs;
    std::vector<int> sp_off(1, 0), sp_col;
    for (int i = 0; i < P.c_dim; i++) {
        if (i == 0) {
            for (int l = 0; l < c->nlev; l++) {
                recs.push_back({P.count_array[l] << 16, 0, 0, l});
                sp_col.push_back(P.count_array[l]);
            }
        } else {
            for (int q = P.row_off[i]; q < P.row_off[i + 1]; q++) {
                const int e = P.row_ent[q];
                if (P.ent_off[e + 1] == P.ent_off[e]) continue;
                const int col = P.ent_pos[e] / P.c_dim;
                recs.push_back({i | col << 16, P.ent_off[e], P.ent_off[e + 1] - P.ent_off[e], -1});
                sp_col.push_back(col);
            }
        }
        sp_off.push_back((int)sp_col.size());
    }
    // the assembly's records (row | column << 16, first term, terms << 16 |
    // entry, -1 or the normalisation's level), most terms first; 16-byte
    // aligned for one load each
    std::vector<int> ord(recs.size()), sp_rec;
    for (size_t e = 0; e < ord.size(); e++) ord[e] = (int)e;
    std::stable_sort(ord.begin(), ord.end(), [&](int p, int q) { return recs[p].count > recs[q].count; });
    for (int e : ord)
        sp_rec.insert(sp_rec.end(), {recs[e].pos, recs[e].first, (int)((unsigned)recs[e].count << 16 | (unsigned)e), recs[e].norm});
    // the entry at every place of the matrix (column-major; the one past the
    // last where there is none), for the systems inverted
    std::vector<int> sp_map;
    if (P.c_dim <= SE_GAUSS_DIM) {
        std::vector<unsigned short> at(((size_t)P.c_dim * P.c_dim + 1) & ~(size_t)1, (unsigned short)recs.size());
        for (size_t e = 0; e < recs.size(); e++) at[(recs[e].pos & 0xffff) + (size_t)P.c_dim * (recs[e].pos >> 16)] = (unsigned short)e;
        sp_map.resize(at.size() / 2);
        std::memcpy(sp_map.data(), at.data(), at.size() * sizeof(unsigned short));
    }
    const size_t o_soff = putI(sp_off), o_scol = putI(sp_col), o_map = putI(sp_map);
    while (I.size() % 4) I.push_back(0);
    const size_t o_asm = putI(sp_rec);
    size_t o_nu = putD(P.tr_nu), o_A = putD(P.tr_A), o_B = putD(P.tr_B21), o_tc = putD(P.term_c),
           o_nv = putD(norm_val), o_ct = putD(c->col_temps), o_C = putD(c->Cji), o_dep = putD(P.dep_tab);
    c->se_built = false;   // (a growing buffer loses the program it held)
    if (c->se_ints.reserve(I.size()) || c->se_dbls.reserve(D.size()))
        return set_err(c, PORTAL_ERR_NOMEM, "SE program");
    PCHECK(c, cudaMemcpyAsync(c->se_ints.p, I.data(), I.size() * sizeof(int), cudaMemcpyHostToDevice, c->stream));
    PCHECK(c, cudaMemcpyAsync(c->se_dbls.p, D.data(), D.size() * sizeof(double), cudaMemcpyHostToDevice, c->stream));
    PCHECK(c, cudaStreamSynchronize(c->stream));
    c->se_kmax = kmax;
    c->se_built = true;
    c->c_dim = P.c_dim;
    c->n_trans = P.n_trans;
    c->count_array = P.count_array;
    // remember offsets in the context (packed into se_off)
    c->se_ni = (int)P.ent_pos.size();
    c->se_offs[0] = o_rad; c->se_offs[1] = o_col; c->se_offs[2] = o_eoff; c->se_offs[3] = o_epos;
    c->se_offs[4] = o_tf; c->se_offs[5] = o_nc; c->se_offs[6] = o_pack;
    c->se_offs[7] = o_nu; c->se_offs[8] = o_A; c->se_offs[9] = o_B; c->se_offs[10] = o_tc;
    c->se_offs[11] = o_nv; c->se_offs[12] = o_ct; c->se_offs[13] = o_C;
    c->se_offs[14] = o_roff; c->se_offs[15] = o_rent; c->se_offs[16] = o_dep; c->se_offs[17] = o_asm;
    c->se_offs[18] = o_soff; c->se_offs[19] = o_scol; c->se_offs[20] = o_map;
    c->se_nnz = (int)sp_col.size();
    c->n_dep = P.n_dep;
    c->n_feat = NF * P.n_trans + (c->depol == 2 ? 2 : 1) * P.n_dep;
    return PORTAL_OK;
}

// Validates kmax, builds the SE program of the molecule (once per kmax),
// sizes the outputs and fills the kernel's argument block.
int se_prepare(portal_ctx *c, int kmax, SEArgs *out, size_t *warp_bytes) {
    if (!c->have_cloud || !c->have_mol) return set_err(c, PORTAL_ERR_STATE, "no cloud or molecule");
    if (kmax < 2 || (kmax & 1))
        return set_err(c, PORTAL_ERR_ARG, "kmax must be even and >= 2 (trace_node packs rho^2_0)");
    int rc = prepare_se(c, kmax);
    if (rc) return rc;
    const int n = c->c_dim;
    const size_t wb = se_warp_bytes(n, c->n_feat);
    if (wb > 200 * 1024 || n > 32 * SE_MAX_ROWS)
        return set_err(c, PORTAL_ERR_ARG, "SE system too large for shared memory");
    if (c->reserve_pops() || c->jj20.reserve((size_t)c->N * c->r_num))
        return set_err(c, PORTAL_ERR_NOMEM, "SE outputs");
    SEArgs a;
    a.N = c->N; a.bulk = c->bulk; a.c_dim = n; a.n_trans = c->n_trans; a.nlev = c->nlev; a.L = c->r_num;
    a.c_temp = c->c_temp; a.c_num = c->c_num; a.c_par = c->c_par; a.nent = c->se_ni;
    a.n_feat = c->n_feat; a.n_dep = c->n_dep; a.depol = c->depol;
    a.J0 = c->J0.p; a.J2 = c->J2.p; a.h2 = c->h2.p; a.tkin = c->tkin.p; a.ab = c->active_ab();
    a.JE = c->ali_valid ? c->JE.p : nullptr;
    a.LS = c->ali_valid ? c->LS.p : nullptr;
    const int *I = c->se_ints.p;
    const double *D = c->se_dbls.p;
    a.tr_rad = I + c->se_offs[0]; a.tr_col = I + c->se_offs[1]; a.ent_off = I + c->se_offs[2];
    a.ent_pos = I + c->se_offs[3]; a.term_f = I + c->se_offs[4]; a.norm_col = I + c->se_offs[5];
    a.pack = I + c->se_offs[6];
    a.tr_nu = D + c->se_offs[7]; a.tr_A = D + c->se_offs[8]; a.tr_B21 = D + c->se_offs[9];
    a.term_c = D + c->se_offs[10]; a.norm_val = D + c->se_offs[11]; a.col_temps = D + c->se_offs[12];
    a.Cji = D + c->se_offs[13];
    a.row_off = I + c->se_offs[14]; a.row_ent = I + c->se_offs[15];
    a.sp_rec = reinterpret_cast<const int4 *>(I + c->se_offs[17]);
    a.sp_off = I + c->se_offs[18]; a.sp_col = I + c->se_offs[19];
    a.sp_map = reinterpret_cast<const unsigned short *>(I + c->se_offs[20]);
    a.nnz = c->se_nnz;
    a.dep_tab = c->n_dep ? D + c->se_offs[16] : nullptr;
    a.pops = c->pops.p; a.jj20 = c->jj20.p; a.status = c->status.p;
    a.rates = nullptr;
    a.nfail = (int *)(c->counters.p + 2);
    a.skip = nullptr;
    // PORTAL_SE_FP64=1: every system factorised in FP64 (the refinement's
    // fallback path), flagged PORTAL_NODE_REFINE
    {
        const char *e = getenv("PORTAL_SE_FP64");
        a.fp64_only = (e && e[0] == '1') ? 1 : 0;
    }
    *out = a;
    if (warp_bytes) *warp_bytes = wb;
    return PORTAL_OK;
}

// The per-pass device work before the solve: the failure count.
// Stream-ordered only (capturable).
int se_pass(portal_ctx *c, cudaStream_t s) {
    PCHECK(c, cudaMemsetAsync(c->counters.p + 2, 0, sizeof(unsigned long long), s));
    return PORTAL_OK;
}
// ... and, before a batched solve, zeroed outputs (its items are the bulk
// nodes; the single-model kernel writes the other rows itself)
int se_batch_pass(portal_ctx *c, cudaStream_t s) {
    PCHECK(c, cudaMemsetAsync(c->pops.p, 0, (size_t)c->N * 2 * c->nlev * sizeof(double), s));
    PCHECK(c, cudaMemsetAsync(c->jj20.p, 0, (size_t)c->N * c->r_num * sizeof(double), s));
    return se_pass(c, s);
}

// (the rates' 3 n sums take the dense matrix's place)
size_t se_matrix_doubles(const portal_ctx *c) { return (size_t)c->se_nnz + (size_t)c->c_dim * std::max(c->c_dim, 3); }

// Whether the prepared system is inverted, and the inversion's shared memory
// per warp.  The limit is on the largest form, the same for every launch.
bool se_gauss(const portal_ctx *c) {
    return c->c_dim <= SE_GAUSS_DIM && se_gauss_bytes(c->c_dim, c->n_feat, c->se_nnz, SE_GAUSS_DIM / 4, true) <= 200 * 1024;
}
size_t se_gauss_team_bytes(const portal_ctx *c) {
    return se_gauss_bytes(c->c_dim, c->n_feat, c->se_nnz, SE_GAUSS_DIM / 4, false);
}

// The batched kernel's instance for the batch's largest system, and its warps
// per node.
static const void *se_batch_kernel(int max_dim, bool gauss) {
    return !gauss                   ? (const void *)k_solve_se<1, true, SE_MAX_ROWS, -1>
           : max_dim <= SE_WARP_DIM ? (const void *)k_solve_se<1, true, 1, SE_WARP_DIM>
           : max_dim <= 48          ? (const void *)k_solve_se<4, true, 2, 12>
                                    : (const void *)k_solve_se<4, true, 3, 24>;
}
int se_batch_team(int max_dim, bool gauss) { return gauss && max_dim > SE_WARP_DIM ? 4 : 1; }

int se_batch_blocks_per_sm(int warps_per_block, size_t team_bytes, int max_dim, bool gauss, int *blocks) {
    const size_t smem = team_bytes * (warps_per_block / se_batch_team(max_dim, gauss));
    const void *k = se_batch_kernel(max_dim, gauss);
    *blocks = 0;
    if (allow_dyn_smem(k) != cudaSuccess) return PORTAL_ERR_CUDA;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k, 32 * warps_per_block, smem) == cudaSuccess
               ? PORTAL_OK
               : PORTAL_ERR_CUDA;
}

// (the kernel's dynamic shared memory limit must have been set by
// se_batch_blocks_per_sm)
int se_batch_launch(cudaStream_t s, int grid, int warps_per_block, const SEBatch &bw) {
    const size_t smem = bw.team_bytes * (warps_per_block / se_batch_team(bw.max_dim, bw.gauss));
    SEArgs a0{};
    SEBatch b = bw;
    void *args[] = {&a0, &b};
    if (cudaLaunchKernel(se_batch_kernel(bw.max_dim, bw.gauss), dim3(grid), dim3(32 * warps_per_block), args, smem,
                         s) != cudaSuccess)
        return PORTAL_ERR_CUDA;
    return cudaGetLastError() == cudaSuccess ? PORTAL_OK : PORTAL_ERR_CUDA;
}

// Warps per node: one up to SE_WARP_DIM unknowns, a team of four above
// (PORTAL_SE_TEAM=1|4 overrides).  The barrier a step costs a team more than
// the columns save it while one warp's registers hold them: 1,024 systems of
// 14 unknowns 26 us by one warp, 37 by a team; 1,700 of 19 43 and 66 us; 4,096
// of 31 133 and 172.  Beyond its registers one warp works in shared memory:
// 8,192 of 39 0.88 ms, a team 0.43; of 74 3.5 and 0.85.
inline int se_team_warps(int n) {
    const char *e = getenv("PORTAL_SE_TEAM");
    if (e) {
        const int v = atoi(e);
        if (v == 1 || v == 4) return v;
    }
    return n > SE_WARP_DIM ? 4 : 1;
}

// TW = 1: blocks of up to 8 independent warps; TW > 1: one team per block.
// One FP64 matrix slot per team of the grid.
template <int TW, int MR, int NC>
int launch_se(portal_ctx *c, SEArgs &a) {
    auto kern = k_solve_se<TW, false, MR, NC>;
    const size_t wb = NC >= 0 ? se_gauss_bytes(a.c_dim, a.n_feat, a.nnz, gauss_quads<TW, NC>, NC == 0) : se_warp_bytes(a.c_dim, a.n_feat);
    const int teams = (TW == 1) ? (int)std::min<size_t>(8, (200 * 1024) / wb) : 1;
    const size_t smem = wb * teams;
    PCHECK(c, allow_dyn_smem((const void *)kern));
    int nb = 0;
    PCHECK(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, 32 * TW * teams, smem));
    const int grid = c->sm_count * std::max(1, nb);
    if (c->se_a64.reserve((size_t)grid * teams * a.a64_stride))
        return set_err(c, PORTAL_ERR_NOMEM, "SE matrix scratch");
    a.a64 = c->se_a64.p;
    timer_start(c, T_SE);
    kern<<<grid, 32 * TW * teams, smem, c->stream>>>(a, SEBatch{});
    timer_stop(c, T_SE);
    PCHECK(c, cudaGetLastError());
    return PORTAL_OK;
}

// Enqueues the solve: results in c->pops, c->jj20, c->rates, c->status; the
// number of singular systems in c->counters[2], zeroed here or, after a
// radiation field enqueued before (fresh), with its counters.  fresh: nothing
// is solved where that field has failed walks.
static int try_solve_se(portal_ctx *c, int kmax, bool rates, bool fresh) {
    SEArgs a;
    int rc = se_prepare(c, kmax, &a, nullptr);
    if (rc) return rc;
    if (rates) {
        const size_t nr = (size_t)c->N * 3 * 2 * c->nlev;
        if (c->rates.reserve(nr)) return set_err(c, PORTAL_ERR_NOMEM, "rates output");
        PCHECK(c, cudaMemsetAsync(c->rates.p, 0, nr * sizeof(double), c->stream));
        a.rates = c->rates.p;
    }
    if (fresh) a.skip = c->counters.p + RF_FAILED;
    else if ((rc = se_pass(c, c->stream))) return rc;
    a.a64_stride = se_matrix_doubles(c);
    const int n = c->c_dim;
    if (se_team_warps(n) == 4)
        rc = !se_gauss(c) ? launch_se<4, SE_MAX_ROWS, -1>(c, a)
             : n <= 48    ? launch_se<4, 2, 12>(c, a)
             : n <= 80    ? launch_se<4, 3, 20>(c, a)
                          : launch_se<4, 3, 24>(c, a);
    else
        rc = !se_gauss(c)       ? launch_se<1, SE_MAX_ROWS, -1>(c, a)
             : n <= 16          ? launch_se<1, 1, 16>(c, a)
             : n <= 24          ? launch_se<1, 1, 24>(c, a)
             : n <= SE_WARP_DIM ? launch_se<1, 1, SE_WARP_DIM>(c, a)
                                : launch_se<1, 3, 0>(c, a);
    return rc;
}

int enqueue_solve_se(portal_ctx *c, int kmax, bool rates, bool fresh) {
    int rc = try_solve_se(c, kmax, rates, fresh);
    if (rc == PORTAL_ERR_NOMEM && c->vray.p) {   // the rays' sums of the field, summed once its kernels are done
        PCHECK(c, cudaStreamSynchronize(c->stream));
        c->release_ray_items();
        rc = try_solve_se(c, kmax, rates, fresh);
    }
    return rc;
}

}  // namespace portal

extern "C" int portal_solve_se(portal_ctx *c, int kmax, const double *J0, const double *J2,
                               double *pol_pops, double *rates, double *JJ_20, int *status) {
    if (!c) return PORTAL_ERR_ARG;
    if (!c->have_cloud || !c->have_mol) return set_err(c, PORTAL_ERR_STATE, "no cloud or molecule");
    cudaSetDevice(c->device);
    const size_t LN = (size_t)c->r_num * c->N;
    if ((J0 == nullptr) != (J2 == nullptr))
        return set_err(c, PORTAL_ERR_ARG, "portal_solve_se: pass both J0 and J2 or neither");
    if (J0) {
        if (c->J0.reserve(LN) || c->J2.reserve(LN)) return set_err(c, PORTAL_ERR_NOMEM, "J buffers");
        PCHECK(c, cudaMemcpyAsync(c->J0.p, J0, LN * sizeof(double), cudaMemcpyHostToDevice, c->stream));
        PCHECK(c, cudaMemcpyAsync(c->J2.p, J2, LN * sizeof(double), cudaMemcpyHostToDevice, c->stream));
        PCHECK(c, cudaMemsetAsync(c->status.p, 0, (size_t)c->N * sizeof(int), c->stream));
        c->j_valid = true;
        c->ali_valid = false;  // a field from the host carries no split
    } else if (!c->j_valid) {
        return set_err(c, PORTAL_ERR_STATE, "portal_solve_se: no device-resident radiation field");
    }
    timers_reset(c);
    const HostSpan out[3] = {{pol_pops, (size_t)c->N * 2 * c->nlev * sizeof(double)}, {JJ_20, LN * sizeof(double)},
                             {rates, (size_t)c->N * 6 * c->nlev * sizeof(double)}};
    if (int rc = portal::enqueue_solve_se(c, kmax, rates != nullptr, false)) return rc;
    map_pages(out, 3);   // the caller's result arrays, while the kernel runs
    // every copy behind the kernel, one wait for all
    if (pol_pops)
        PCHECK(c, cudaMemcpyAsync(pol_pops, c->pops.p, (size_t)c->N * 2 * c->nlev * sizeof(double),
                                  cudaMemcpyDeviceToHost, c->stream));
    if (JJ_20)
        PCHECK(c, cudaMemcpyAsync(JJ_20, c->jj20.p, LN * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    if (status)
        PCHECK(c, cudaMemcpyAsync(status, c->status.p, (size_t)c->N * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    if (rates)
        PCHECK(c, cudaMemcpyAsync(rates, c->rates.p, (size_t)c->N * 3 * 2 * c->nlev * sizeof(double),
                                  cudaMemcpyDeviceToHost, c->stream));
    int nsing = 0;
    PCHECK(c, cudaMemcpyAsync(&nsing, c->counters.p + 2, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    PCHECK(c, cudaStreamSynchronize(c->stream));
    timer_collect(c, T_SE);
    c->pops_valid = true;
    if (nsing) return set_err(c, PORTAL_ERR_SINGULAR, std::to_string(nsing) + " singular SE systems");
    return PORTAL_OK;
}

extern "C" int portal_set_depolarization(portal_ctx *c, int mode) {
    if (!c) return PORTAL_ERR_ARG;
    if (mode < 0 || mode > 2) return set_err(c, PORTAL_ERR_ARG, "portal_set_depolarization: mode 0, 1 or 2");
    if (mode != c->depol) {
        c->depol = mode;
        c->se_kmax = -1;  // rebuild the SE program
    }
    return PORTAL_OK;
}
