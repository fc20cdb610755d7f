// Learned warm start for the Lambda iteration: a small MLP trained on the
// GPU with the library's own kernels (no reference counterpart).
//
// Network: n_in -> width (SiLU) -> ... (depth hidden layers) -> n_out
// (linear).  Parameters are FP32 master copies; every GEMM rounds its
// operands to BF16 (weights and activations) and accumulates in FP32 on the
// tensor cores: the forward products with tcgen05, the backward ones, whose
// operands are transposed, with mma.sync m16n8k16.  Inputs and targets are
// standardised with statistics stored in the model.  Networks of layers up to
// 256 wide run as whole-network kernels (k_mlp_rows, k_mlp_grads); wider ones
// layer by layer (k_gemm_tc where a layer fits, k_gemm).
//
// GEMM kernel: C(M,N) = A(M,K) B(K,N) with 64x64 block tiles, 4 warps of
// 32x32, K steps of 32 staged in shared memory as BF16 (K-contiguous rows,
// padded), and fused epilogues:
//   forward hidden   Z = C + b, H = silu(Z)     (Z kept for the backward)
//   forward output   Y = C + b
//   backward dX      dZ_prev = C * silu'(Z_prev)
//   backward dW      G = C
// The operand layouts are template flags: A K-contiguous (row-major M x K)
// or M-contiguous; B K-contiguous (stored N x K) or N-contiguous.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include "common.cuh"
#include "umma.cuh"

using namespace portal;

namespace {

enum Epi { EPI_STORE = 0, EPI_BIAS = 1, EPI_BIAS_SILU = 2, EPI_DSILU = 3 };

struct EpiArgs {
    int kind, ldc;
    float *C;          // output (G, Y, H or dZ)
    float *Z;          // pre-activation out (EPI_BIAS_SILU) or in (EPI_DSILU)
    const float *bias;
};

// (x = 1 + e^-z >= 1; from 2^125 on the sigmoid is subnormal or 0)
__device__ __forceinline__ float sigm(float z) {
    const float x = 1.f + __expf(-z);
    return x < 0x1p125f ? recip_rn(x) : rcp_approx(x);
}

template <bool AK, bool BK>
__global__ void __launch_bounds__(128) k_gemm(int M, int N, int K, const float *__restrict__ A, int lda,
                                              const float *__restrict__ B, int ldb, EpiArgs e) {
    __shared__ __align__(16) __nv_bfloat16 As[64][40];
    __shared__ __align__(16) __nv_bfloat16 Bs[64][40];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int wm = w >> 1, wn = w & 1, g = lane >> 2, t = lane & 3;
    const int m0 = blockIdx.y * 64, n0 = blockIdx.x * 64;
    float acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int q = 0; q < 4; q++) acc[i][j][q] = 0.f;
    for (int k0 = 0; k0 < K; k0 += 32) {
        for (int i = tid; i < 64 * 32; i += 128) {
            int r, kk;
            if (AK) { r = i >> 5; kk = i & 31; } else { kk = i >> 6; r = i & 63; }
            const int gm = m0 + r, gk = k0 + kk;
            float v = 0.f;
            if (gm < M && gk < K) v = AK ? A[(size_t)gm * lda + gk] : A[(size_t)gk * lda + gm];
            As[r][kk] = __float2bfloat16(v);
        }
        for (int i = tid; i < 64 * 32; i += 128) {
            int c, kk;
            if (BK) { c = i >> 5; kk = i & 31; } else { kk = i >> 6; c = i & 63; }
            const int gn = n0 + c, gk = k0 + kk;
            float v = 0.f;
            if (gn < N && gk < K) v = BK ? B[(size_t)gn * ldb + gk] : B[(size_t)gk * ldb + gn];
            Bs[c][kk] = __float2bfloat16(v);
        }
        __syncthreads();
#pragma unroll
        for (int ks = 0; ks < 32; ks += 16) {
            uint32_t af[2][4], bfr[4][2];
#pragma unroll
            for (int mi = 0; mi < 2; mi++) {
                const int rb = wm * 32 + mi * 16;
                af[mi][0] = *(const uint32_t *)&As[rb + g][ks + 2 * t];
                af[mi][1] = *(const uint32_t *)&As[rb + g + 8][ks + 2 * t];
                af[mi][2] = *(const uint32_t *)&As[rb + g][ks + 2 * t + 8];
                af[mi][3] = *(const uint32_t *)&As[rb + g + 8][ks + 2 * t + 8];
            }
#pragma unroll
            for (int ni = 0; ni < 4; ni++) {
                const int cb = wn * 32 + ni * 8;
                bfr[ni][0] = *(const uint32_t *)&Bs[cb + g][ks + 2 * t];
                bfr[ni][1] = *(const uint32_t *)&Bs[cb + g][ks + 2 * t + 8];
            }
#pragma unroll
            for (int mi = 0; mi < 2; mi++)
#pragma unroll
                for (int ni = 0; ni < 4; ni++)
                    asm volatile(
                        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
                        "{%8,%9}, {%0,%1,%2,%3};\n"
                        : "+f"(acc[mi][ni][0]), "+f"(acc[mi][ni][1]), "+f"(acc[mi][ni][2]), "+f"(acc[mi][ni][3])
                        : "r"(af[mi][0]), "r"(af[mi][1]), "r"(af[mi][2]), "r"(af[mi][3]), "r"(bfr[ni][0]),
                          "r"(bfr[ni][1]));
        }
        __syncthreads();
    }
#pragma unroll
    for (int mi = 0; mi < 2; mi++)
#pragma unroll
        for (int ni = 0; ni < 4; ni++)
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int r = m0 + wm * 32 + mi * 16 + g + ((q & 2) ? 8 : 0);
                const int c = n0 + wn * 32 + ni * 8 + 2 * t + (q & 1);
                if (r >= M || c >= N) continue;
                const float v = acc[mi][ni][q];
                const size_t o = (size_t)r * e.ldc + c;
                switch (e.kind) {
                case EPI_STORE: e.C[o] = v; break;
                case EPI_BIAS: e.C[o] = v + e.bias[c]; break;
                case EPI_BIAS_SILU: {
                    const float z = v + e.bias[c];
                    e.Z[o] = z;
                    e.C[o] = z * sigm(z);
                    break;
                }
                case EPI_DSILU: {
                    const float z = e.Z[o], s = sigm(z);
                    e.C[o] = v * s * (1.f + z * (1.f - s));
                    break;
                }
                }
            }
}

// ---- the forward GEMMs on the 5th-generation tensor cores ------------------
// C(M, N) = A(M, K) W(N, K)^T with the fused epilogues above, for K, N <= 256.
// Persistent CTAs of 4 warps (one per SM, the grid at most the SM count):
// each converts all of W to BF16 in shared memory once, then for each of its
// 128-row tiles of A converts the rows to BF16 beside it, one thread issues
// the Kp/16 MMAs of shape 128 x Np x 16 into an FP32 accumulator in tensor
// memory and commits them to an mbarrier, and each warp reads its 32 rows
// back with tcgen05.ld for the epilogue.  Shared-memory operands use the
// canonical no-swizzle K-major layout: 8-row x 16-byte core matrices,
// K-adjacent ones 128 B apart, row groups Kp/8 x 128 B apart (K and N
// zero-padded to multiples of 16).  Waits are bounded: a timeout sets *err,
// the CTA stops and still frees its tensor memory.
constexpr int TC_M = 128;

// the A tile's region doubles as the epilogue's transpose buffer (4 KB per
// warp of 512 threads) once a tile's MMAs are complete
constexpr int TC_EPI_BYTES = 16 * 32 * 32 * 4;
__host__ __device__ inline size_t tc_a_bytes(int Kp) {
    return (size_t)TC_M * Kp * 2 > (size_t)TC_EPI_BYTES ? (size_t)TC_M * Kp * 2 : (size_t)TC_EPI_BYTES;
}
__host__ __device__ inline size_t tc_smem_bytes(int Np, int Kp) {
    return tc_a_bytes(Kp) + (size_t)Np * Kp * 2 + 16;
}

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&h);
}

// rows [r0, r0 + rows) of the row-major src (ld floats per row, K valid
// columns, nrow_valid valid rows) into the canonical BF16 tile; each thread
// first loads TC_U chunks (two float4 each) and then converts them, so that
// many loads are in flight per thread
constexpr int TC_THREADS = 512;
constexpr int TC_U = 4;

__device__ __forceinline__ void tc_load8(const float *p, bool valid, int nk, float *v) {
    if (valid && nk >= 8 && ((reinterpret_cast<uintptr_t>(p) & 15) == 0)) {
        const float4 x = __ldg(reinterpret_cast<const float4 *>(p));
        const float4 y = __ldg(reinterpret_cast<const float4 *>(p) + 1);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
        v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
    } else {
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = (valid && j < nk) ? p[j] : 0.f;
    }
}

__device__ __forceinline__ void tc_stage(unsigned char *tile, int rows, int Kp, const float *__restrict__ src,
                                         int r0, int nrow_valid, int K, int ld, int tid) {
    const int kc = Kp / 8;
    const uint32_t sbo = (uint32_t)kc * 128;
    const int total = rows * kc;
    for (int base = tid; base < total; base += TC_THREADS * TC_U) {
        float v[TC_U][8];
#pragma unroll
        for (int u = 0; u < TC_U; u++) {
            const int i = base + u * TC_THREADS;
            const int r = i / kc, c = i - r * kc;
            tc_load8(src + (size_t)(r0 + r) * ld + c * 8, i < total && r < nrow_valid, K - c * 8, v[u]);
        }
#pragma unroll
        for (int u = 0; u < TC_U; u++) {
            const int i = base + u * TC_THREADS;
            if (i >= total) break;
            const int r = i / kc, c = i - r * kc;
            uint4 q;
            q.x = pack_bf16x2(v[u][0], v[u][1]);
            q.y = pack_bf16x2(v[u][2], v[u][3]);
            q.z = pack_bf16x2(v[u][4], v[u][5]);
            q.w = pack_bf16x2(v[u][6], v[u][7]);
            *reinterpret_cast<uint4 *>(tile + (size_t)(r >> 3) * sbo + (size_t)c * 128 + (size_t)(r & 7) * 16) = q;
        }
    }
}

__global__ void __launch_bounds__(TC_THREADS, 1) k_gemm_tc(int M, int N, int K, int Np, int Kp, uint32_t tcols,
                                                           const float *__restrict__ A, const float *__restrict__ W,
                                                           EpiArgs e, int *err) {
    extern __shared__ __align__(1024) unsigned char tsm[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    unsigned char *As = tsm;
    unsigned char *Bs = tsm + tc_a_bytes(Kp);
    uint64_t *bar = reinterpret_cast<uint64_t *>(Bs + (size_t)Np * Kp * 2);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(bar + 1);
    float *T = reinterpret_cast<float *>(As) + (size_t)warp * 32 * 32;  // this warp's 32 x 32 transpose buffer
    tc_stage(Bs, Np, Kp, W, 0, N, K, K, tid);
    if (warp == 0) umma::tmem_alloc(tslot, tcols);
    if (tid == 0) {
        umma::mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t taddr = *tslot;
    const uint32_t idesc = umma::idesc_bf16_f32(TC_M, Np);
    const uint32_t sbo = (uint32_t)(Kp / 8) * 128;
    const int ntiles = (M + TC_M - 1) / TC_M;
    // epilogue split: warp w reads the lane quarter w % 4 (tcgen05.ld's rule)
    // and every (TC_THREADS / 128)-th 32-column chunk from chunk w / 4
    const int quarter = warp & 3, cgroup = warp >> 2, ngroups = TC_THREADS / 128;
    int iter = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x, iter++) {
        const int m0 = t * TC_M;
        tc_stage(As, TC_M, Kp, A, m0, min(TC_M, M - m0), K, K, tid);
        umma::fence_proxy_async();
        umma::fence_before_sync();
        __syncthreads();   // A staged; the previous tile's accumulator reads are done
        umma::fence_after_sync();
        if (tid == 0) {
            const uint32_t a0 = umma::smem_addr(As), b0 = umma::smem_addr(Bs);
            for (int ks = 0; ks < Kp / 16; ks++)
                umma::mma_bf16(taddr, umma::smem_desc(a0 + ks * 256, 128, sbo),
                               umma::smem_desc(b0 + ks * 256, 128, sbo), idesc, ks > 0);
            umma::mma_commit(bar);
        }
        bool done = false;
        for (int it = 0; it < (1 << 24) && !done; it++) done = umma::mbar_try_wait(bar, (uint32_t)(iter & 1));
        ok = __syncthreads_and(done);
        umma::fence_after_sync();
        if (!ok) {
            if (tid == 0) atomicExch(err, 1);
            break;
        }
        // epilogue: thread t of the warp holds row (rbase + t), columns c0..c0+31;
        // through the warp's transpose buffer (XOR-swizzled, no bank
        // conflicts) each store instruction then writes 32 consecutive
        // columns of one row
        const int rbase = m0 + quarter * 32;
        for (int c0 = cgroup * 32; c0 < Np; c0 += 32 * ngroups) {
            float v[32];
            umma::tmem_ld32(taddr + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0, v);
            const int cl = c0 + lane;                  // the column this lane stores
            const float bl = (e.kind != EPI_STORE && cl < N) ? e.bias[cl] : 0.f;
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 32; j++) T[lane * 32 + (j ^ lane)] = v[j];
            __syncwarp();
            for (int pass = 0; pass < (e.kind == EPI_BIAS_SILU ? 2 : 1); pass++) {
                float *dst = (pass == 0 && e.kind == EPI_BIAS_SILU) ? e.Z : e.C;
                for (int r = 0; r < 32; r++) {
                    const int row = rbase + r;
                    if (row >= M) break;
                    if (cl < N) {
                        const float z = T[r * 32 + (lane ^ r)] + bl;
                        dst[(size_t)row * e.ldc + cl] = (e.kind == EPI_BIAS_SILU && pass == 1) ? z * sigm(z) : z;
                    }
                }
            }
        }
        __syncthreads();   // the transpose buffers share the A tile's memory: all warps are done with them
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(taddr, tcols);
}

// ---- whole-network kernels -------------------------------------------------
// Networks whose layers are all at most 256 wide (the warm start's: 8 -> 256 x
// 3 -> 40) run the forward pass, and in training the loss and the chain of dZ,
// as one kernel per batch: a CTA keeps its rows' activations in shared memory
// as BF16 and streams each layer's weights (a packed BF16 image, canonical
// no-swizzle K-major layout) from L2 by bulk copies that overlap the previous
// layer's epilogue.  The transposed product D = W H^T is formed: out-features
// on the 128 tensor-memory lanes, the CTA's NB rows on the columns, so that
// all warps share the epilogue at any NB.  Layer by layer, each GEMM wrote and
// re-read its FP32 activations, four CTAs per training step converted all of
// W, and a step of 19 launches took 640 us (512 rows; now 2 launches, 35 us,
// the serial latency of 32 CTAs through seven dependent products); every sum
// keeps its order (K in steps of 16, FP32 accumulators, BF16 rounding points
// unchanged).
constexpr int FU_MAX = 256;        // widest layer
constexpr int FU_THREADS = 512;
constexpr int FU_MAX_LAYERS = 17;  // depth <= 16 hidden layers and the output layer

struct FusedNet {
    int n_layers, n_in, n_out;
    int fin[FU_MAX_LAYERS], fout[FU_MAX_LAYERS];       // as given
    int kp[FU_MAX_LAYERS], np[FU_MAX_LAYERS];          // padded to 16
    unsigned pk[FU_MAX_LAYERS];                        // byte offset of the layer's packed weights
    unsigned woff[FU_MAX_LAYERS], boff[FU_MAX_LAYERS]; // in the flat parameters
    int wbuf;                                          // bytes of shared memory for one layer's weights
};
// per-batch buffers of a training step (rows padded to 32)
struct FusedBatch {
    float *Z[FU_MAX_LAYERS];              // (rows, fout) pre-activations of the hidden layers
    float *dZ[FU_MAX_LAYERS];             // (rows, fout)
    __nv_bfloat16 *H[FU_MAX_LAYERS];      // (rows, kp): layer l's input rounded to BF16
    __nv_bfloat16 *dZb[FU_MAX_LAYERS];    // (rows, np)
    double *loss;                         // one partial sum per CTA
};

// byte offset of element (r, k) in a canonical tile of kp columns
__device__ __forceinline__ uint32_t tile_at(int r, int k, int kp) {
    return (uint32_t)(r >> 3) * (uint32_t)(kp * 16) + (uint32_t)(k >> 3) * 128u + (uint32_t)(r & 7) * 16u +
           (uint32_t)(k & 7) * 2u;
}

// packed BF16 weights of every layer from the FP32 parameters (zero padding)
__global__ void k_pack_weights(FusedNet net, const float *__restrict__ p, unsigned char *__restrict__ pk) {
    const int l = blockIdx.y, kc = net.kp[l] / 8, total = net.np[l] * kc;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int n = i / kc, c = i - n * kc;
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int k = 8 * c + j;
            v[j] = (n < net.fout[l] && k < net.fin[l]) ? p[net.woff[l] + (size_t)n * net.fin[l] + k] : 0.f;
        }
        *reinterpret_cast<uint4 *>(pk + net.pk[l] + tile_at(n, 8 * c, net.kp[l])) =
            make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]),
                       pack_bf16x2(v[6], v[7]));
    }
}

// bounded wait for a barrier's phase, all threads of the CTA: false when the
// limit runs out (uniform)
__device__ __forceinline__ bool cta_wait(uint64_t *bar, uint32_t phase) {
    bool done = false;
    for (int it = 0; it < (1 << 24) && !done; it++) done = umma::mbar_try_wait(bar, phase);
    return __syncthreads_and(done);
}

// NB rows per CTA.  TRAIN: also the loss, its gradient and the chain of dZ;
// else raw-unit predictions into Y.
// X: (.., n_in) rows, row i of the batch at idx[i] (or i); st: standardisation
// statistics applied to X (and T), null when they are standardised already.
template <int NB, bool TRAIN>
__global__ void __launch_bounds__(FU_THREADS, 1)
    k_mlp_rows(FusedNet net, int B, const int *__restrict__ idx, const float *__restrict__ X,
               const float *__restrict__ T, const float *__restrict__ st, const float *__restrict__ params,
               const unsigned char *__restrict__ pk, float *__restrict__ Y, FusedBatch fb, float scale, int *err) {
    // an epilogue unit: 32 features x UR rows per warp
    constexpr int TH = FU_THREADS, WARPS = TH / 32, UR = NB == 16 ? 8 : NB == 32 ? 16 : 32, CC = NB / UR;
    extern __shared__ __align__(1024) unsigned char fsm[];
    unsigned char *Ws = fsm, *As = fsm + net.wbuf;
    uint64_t *bar_w = reinterpret_cast<uint64_t *>(As + (size_t)NB * FU_MAX * 2);
    uint64_t *bar_m = bar_w + 1;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(bar_w + 2);
    double *lred = reinterpret_cast<double *>(bar_w + 3);   // WARPS partial losses
    float *Ts = reinterpret_cast<float *>(lred + 16);       // TRAIN: the rows' standardised targets
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row0 = blockIdx.x * NB;
    uint32_t ph_w = 0, ph_m = 0;
    constexpr uint32_t TCOLS = 2 * NB;
    if (warp == 0) umma::tmem_alloc(tslot, TCOLS);
    if (tid == 0) {
        umma::mbar_init(bar_w, 1);
        umma::mbar_init(bar_m, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // one thread: layer l's packed weights into Ws (the buffer must be free)
    auto load_w = [&](int l) {
        const uint32_t bytes = (uint32_t)net.np[l] * net.kp[l] * 2;
        umma::mbar_expect_tx(bar_w, bytes);
        for (uint32_t o = 0; o < bytes; o += 16384)
            umma::bulk_load(Ws + o, pk + net.pk[l] + o, min(16384u, bytes - o), bar_w);
    };
    if (tid == 0) load_w(0);
    // the CTA's input rows, standardised, as BF16
    const float *mx = st, *sx = st ? st + net.n_in : nullptr, *my = st ? st + 2 * net.n_in : nullptr,
                *sy = st ? my + net.n_out : nullptr;
    {
        const int kp = net.kp[0], kc = kp / 2;   // a pair of features per thread
        for (int i = tid; i < NB * kc; i += TH) {
            const int r = i / kc, k = 2 * (i - r * kc), row = row0 + r;
            float v[2] = {0.f, 0.f};
            if (row < B) {
                const float *src = X + (size_t)(idx ? idx[row] : row) * net.n_in;
#pragma unroll
                for (int j = 0; j < 2; j++)
                    if (k + j < net.n_in) v[j] = st ? (src[k + j] - mx[k + j]) / sx[k + j] : src[k + j];
            }
            const uint32_t w = pack_bf16x2(v[0], v[1]);
            *reinterpret_cast<uint32_t *>(As + tile_at(r, k, kp)) = w;
            if (TRAIN) *reinterpret_cast<uint32_t *>(fb.H[0] + (size_t)row * kp + k) = w;
        }
        if (TRAIN)
            for (int i = tid; i < NB * net.n_out; i += TH) {
                const int r = i / net.n_out, f = i - r * net.n_out, row = row0 + r;
                float t0 = (row < B) ? T[(size_t)(idx ? idx[row] : row) * net.n_out + f] : 0.f;
                if (st) t0 = (t0 - my[f]) / sy[f];
                Ts[i] = t0;
            }
    }
    const uint32_t taddr = *tslot;
    const int quarter = warp & 3;
    bool ok = true;
    double loss = 0.0;
    for (int l = 0; l < net.n_layers && ok; l++) {
        const bool last = l == net.n_layers - 1;
        const int kp = net.kp[l], tiles = (net.fout[l] + 127) / 128;
        umma::fence_proxy_async();   // the activations are in shared memory
        umma::fence_before_sync();
        ok = cta_wait(bar_w, ph_w);   // (a barrier of the CTA too)
        ph_w ^= 1;
        if (!ok) break;
        umma::fence_after_sync();
        if (tid == 0) {
            const uint32_t idesc = umma::idesc_bf16_f32(128, NB), sbo = (uint32_t)kp * 16;
            const uint32_t a0 = umma::smem_addr(Ws), b0 = umma::smem_addr(As);
            for (int t = 0; t < tiles; t++)
                for (int ks = 0; ks < kp / 16; ks++)
                    umma::mma_bf16(taddr + t * NB, umma::smem_desc(a0 + t * 16 * sbo + ks * 256, 128, sbo),
                                   umma::smem_desc(b0 + ks * 256, 128, sbo), idesc, ks > 0);
            umma::mma_commit(bar_m);
        }
        ok = cta_wait(bar_m, ph_m);
        ph_m ^= 1;
        if (!ok) break;
        umma::fence_after_sync();
        if (!last && tid == 0) {   // Ws and As are free: the next layer's weights under this epilogue
            umma::fence_proxy_async();
            load_w(l + 1);
        }
        const float *bias = params + net.boff[l];
        const int kpn = last ? net.np[l] : net.kp[l + 1];   // columns of the tile written next
        for (int u = warp >> 2; u < tiles * CC; u += WARPS / 4) {
            const int t = u / CC, cc = u - t * CC;
            const int f = t * 128 + quarter * 32 + lane;    // this thread's feature
            if (t * 128 + quarter * 32 >= kpn) continue;   // whole warp past the layer
            float v[UR];
            const uint32_t tc = taddr + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(t * NB + cc * UR);
            if constexpr (UR == 8) umma::tmem_ld8(tc, v);
            else if constexpr (UR == 16) umma::tmem_ld16(tc, v);
            else umma::tmem_ld32(tc, v);
            const bool on = f < net.fout[l];
            const float b = on ? bias[f] : 0.f;
            const int r0 = cc * UR;
            if (!last) {
                float *Z = TRAIN ? fb.Z[l] : nullptr;
#pragma unroll
                for (int j = 0; j < UR; j++) {
                    const float z = v[j] + b;
                    if (TRAIN && on) Z[(size_t)(row0 + r0 + j) * net.fout[l] + f] = z;
                    v[j] = on ? z * sigm(z) : 0.f;
                }
            } else if (!TRAIN) {
                if (on) {
                    const float s = sy[f], m = my[f];
#pragma unroll
                    for (int j = 0; j < UR; j++)
                        if (row0 + r0 + j < B) Y[(size_t)(row0 + r0 + j) * net.n_out + f] = fmaf(v[j] + b, s, m);
                }
                continue;
            } else {
                float *dZ = fb.dZ[l];
                float sq[UR];
#pragma unroll
                for (int j = 0; j < UR; j++) {
                    const int row = row0 + r0 + j;
                    float d = 0.f;
                    sq[j] = 0.f;
                    if (on && row < B) {
                        d = (v[j] + b) - Ts[(r0 + j) * net.n_out + f];
                        sq[j] = d * d * scale;
                        d = 2.f * d * scale;
                    }
                    if (on) dZ[(size_t)row * net.n_out + f] = d;
                    v[j] = d;
                }
                // the thread's squares in an FP32 tree, the threads' sums in FP64
#pragma unroll
                for (int h = UR / 2; h >= 1; h >>= 1)
#pragma unroll
                    for (int j = 0; j < h; j++) sq[j] += sq[j + h];
                loss += (double)sq[0];
            }
            // the next tile as BF16: neighbouring features pair up, the even lane
            // stores row j's pair, the odd one row j + 1's
            __nv_bfloat16 *G = !TRAIN ? nullptr : last ? fb.dZb[l] : fb.H[l + 1];
            const unsigned mask = (kpn - (t * 128 + quarter * 32) >= 32) ? 0xffffffffu : 0xffffu;
            if ((mask >> lane) & 1u) {
#pragma unroll
                for (int j = 0; j < UR; j += 2) {
                    const float got = __shfl_xor_sync(mask, (lane & 1) ? v[j] : v[j + 1], 1);
                    const int r = r0 + j + (lane & 1);
                    const uint32_t w = (lane & 1) ? pack_bf16x2(got, v[j + 1]) : pack_bf16x2(v[j], got);
                    *reinterpret_cast<uint32_t *>(As + tile_at(r, f & ~1, kpn)) = w;
                    if (TRAIN) *reinterpret_cast<uint32_t *>(G + (size_t)(row0 + r) * kpn + (f & ~1)) = w;
                }
            }
        }
        umma::fence_before_sync();
    }
    if constexpr (TRAIN) {
        // the loss: one FP64 partial per CTA, warps in order
        for (int o = 16; o >= 1; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
        if (lane == 0) lred[warp] = loss;
        __syncthreads();
        if (tid == 0) {
            double s = 0.0;
            for (int w = 0; w < WARPS; w++) s += lred[w];
            fb.loss[blockIdx.x] = s;
        }
        // dZ of layer l-1: (dZ_l W_l) silu'(Z), on mma.sync: rows x inputs, K =
        // outputs; W_l is in Ws as its canonical tile, whose 8 x 8 core matrices
        // ldmatrix reads transposed
        constexpr int MT = NB / 16;   // tiles of 16 rows
        const int g = lane >> 2, t = lane & 3;
        for (int l = net.n_layers - 1; l > 0 && ok; l--) {
            if (l < net.n_layers - 1) {   // (the forward left the last layer's weights)
                ok = cta_wait(bar_w, ph_w);
                ph_w ^= 1;
                if (!ok) break;
            }
            const int kpa = net.np[l], kpw = net.kp[l];   // dZ tile (rows x outputs), W tile (outputs x inputs)
            const int n0 = warp * 16;
            // silu'(Z) needs Z at this thread's outputs: loaded ahead of the products
            const float *Z = fb.Z[l - 1];
            const int nin = net.fin[l];
            float zv[MT][2][4];
#pragma unroll
            for (int i = 0; i < MT; i++)
#pragma unroll
                for (int j = 0; j < 2; j++)
#pragma unroll
                    for (int h = 0; h < 4; h++) {
                        const int r = 16 * i + g + 8 * (h >> 1), c = n0 + 8 * j + 2 * t + (h & 1);
                        zv[i][j][h] = (c < nin) ? Z[(size_t)(row0 + r) * nin + c] : 0.f;
                    }
            float acc[MT][2][4];
#pragma unroll
            for (int i = 0; i < MT; i++)
#pragma unroll
                for (int j = 0; j < 2; j++)
#pragma unroll
                    for (int q = 0; q < 4; q++) acc[i][j][q] = 0.f;
            if (n0 < kpw)
#pragma unroll 4
                for (int k0 = 0; k0 < kpa; k0 += 16) {
                    uint32_t a[MT][4], q[4];
#pragma unroll
                    for (int i = 0; i < MT; i++)
                        umma::ldmatrix4(a[i], As + tile_at(16 * i + (lane & 15), k0 + 8 * (lane >> 4), kpa));
                    umma::ldmatrix4_trans(q, Ws + tile_at(k0 + (lane & 15), n0 + 8 * (lane >> 4), kpw));
#pragma unroll
                    for (int i = 0; i < MT; i++)
#pragma unroll
                        for (int j = 0; j < 2; j++) {
                            const uint32_t b[2] = {q[2 * j], q[2 * j + 1]};
                            umma::mma_sync_bf16(acc[i][j], a[i], b);
                        }
                }
            umma::fence_proxy_async();
            __syncthreads();   // every warp has read dZ_l and W_l
            if (l > 1 && tid == 0) load_w(l - 1);
            float *dZ = fb.dZ[l - 1];
#pragma unroll
            for (int i = 0; i < MT; i++)
#pragma unroll
                for (int j = 0; j < 2; j++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int r = 16 * i + g + 8 * h, c = n0 + 8 * j + 2 * t;
                        if (c >= kpw) continue;
                        float o[2];
#pragma unroll
                        for (int q = 0; q < 2; q++) {
                            const float z = zv[i][j][2 * h + q], s = sigm(z);
                            o[q] = (c + q < nin) ? acc[i][j][2 * h + q] * s * (1.f + z * (1.f - s)) : 0.f;
                            if (c + q < nin) dZ[(size_t)(row0 + r) * nin + c + q] = o[q];
                        }
                        const uint32_t w = pack_bf16x2(o[0], o[1]);
                        *reinterpret_cast<uint32_t *>(As + tile_at(r, c, kpw)) = w;
                        *reinterpret_cast<uint32_t *>(fb.dZb[l - 1] + (size_t)(row0 + r) * kpw + c) = w;
                    }
            __syncthreads();
        }
    }
    if (!ok && tid == 0) atomicExch(err, 1);
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(taddr, TCOLS);
}

// dW = dZ^T Hin of every layer on mma.sync (32 outputs x 64 inputs per CTA of
// four warps, K = the batch's rows in chunks of 64 staged by cp.async), and
// the bias gradients (32 columns per CTA, rows summed in order); then Adam on
// the CTA's own parameters and their packed BF16 copy, or the gradient itself.
// Latency-bound (a CTA's products take a microsecond): four chunks in flight.
// Block 0 also adds the batch's loss to the epoch's.
constexpr int DW_K = 64, DW_STAGES = 4;
constexpr int DW_LA = 40, DW_LB = 72;   // row strides (BF16): 80 and 144 bytes, ldmatrix without bank conflicts
constexpr size_t DW_SMEM = (size_t)DW_STAGES * DW_K * (DW_LA + DW_LB) * 2;
struct AdamArgs {
    float *p, *m, *v;
    unsigned char *pk;
    float lr, b1, b2, eps, c1, c2;
};
// one parameter: (p, m, v) updated with its gradient.  The products fuse as in
// k_adam's expressions: while m / sqrt(v) is near +-1, the first steps amplify
// a last bit of m into a visible change of p.
__device__ __forceinline__ void adam(const AdamArgs &a, float gi, float &p, float &m, float &v) {
    m = fmaf(1.f - a.b1, gi, __fmul_rn(a.b1, m));
    v = fmaf(__fmul_rn(1.f - a.b2, gi), gi, __fmul_rn(a.b2, v));
    p = __fsub_rn(p, a.lr * (m / a.c1) / (sqrtf(v / a.c2) + a.eps));
}
template <bool ADAM>
__global__ void __launch_bounds__(128) k_mlp_grads(FusedNet net, int rows, FusedBatch fb, float *__restrict__ grads,
                                                   AdamArgs ad, int n_loss, double *loss_acc) {
    constexpr int LA = DW_LA, LB = DW_LB;
    extern __shared__ __align__(16) unsigned char gsm[];
    __nv_bfloat16 *sA = reinterpret_cast<__nv_bfloat16 *>(gsm), *sB = sA + DW_STAGES * DW_K * LA;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (blockIdx.x == 0 && tid == 0 && loss_acc) {
        double s = 0.0;
        for (int i = 0; i < n_loss; i++) s += fb.loss[i];
        *loss_acc += s;
    }
    // this CTA's layer and tile: per layer its weight tiles, then its bias strips
    int b = blockIdx.x, l = 0, mt = 0, nt = 0;
    bool bias = false;
    for (;; l++) {
        const int tm = (net.fout[l] + 31) / 32, tn = (net.fin[l] + 63) / 64;
        if (b < tm * tn) { mt = b / tn; nt = b - mt * tn; break; }
        b -= tm * tn;
        if (b < tm) { mt = b; bias = true; break; }
        b -= tm;
    }
    const int nout = net.fout[l], nin = net.fin[l], chunks = (rows + DW_K - 1) / DW_K;
    if (bias) {
        // warps 1-3 stage 64 rows x 32 columns at a time, warp 0 adds them in row order
        constexpr int ST = (int)(DW_SMEM / (DW_K * 32 * 4));
        float *ring = reinterpret_cast<float *>(gsm);
        float sum = 0.f;
        const int c = mt * 32 + lane;
        const size_t i = net.boff[l] + c;
        float p = 0.f, m = 0.f, v = 0.f;
        if (ADAM && warp == 0 && c < nout) { p = ad.p[i]; m = ad.m[i]; v = ad.v[i]; }
        auto stage = [&](int ch) {
            if (warp > 0 && ch < chunks) {
                float *s = ring + (ch % ST) * DW_K * 32 + lane;
                const float *src = fb.dZ[l] + (size_t)ch * DW_K * nout + c;
                const int n = min(DW_K, rows - ch * DW_K);
                for (int r = warp - 1; r < n; r += 3)
                    if (c < nout) umma::cp_async4(s + r * 32, src + (size_t)r * nout);
            }
            umma::cp_async_commit();
        };
        for (int ch = 0; ch < ST - 1; ch++) stage(ch);
        for (int ch = 0; ch < chunks; ch++) {
            umma::cp_async_wait<ST - 2>();
            __syncthreads();
            stage(ch + ST - 1);
            if (warp == 0) {
                const float *s = ring + (ch % ST) * DW_K * 32 + lane;
                const int n = min(DW_K, rows - ch * DW_K);
                if (n == DW_K) {
#pragma unroll
                    for (int r = 0; r < DW_K; r++) sum += s[r * 32];
                } else {
                    for (int r = 0; r < n; r++) sum += s[r * 32];
                }
            }
        }
        umma::cp_async_wait<0>();
        if (warp == 0 && c < nout) {
            if (ADAM) {
                adam(ad, sum, p, m, v);
                ad.p[i] = p; ad.m[i] = m; ad.v[i] = v;
            } else {
                grads[i] = sum;
            }
        }
        return;
    }
    const int lda = net.np[l], ldb = net.kp[l], m0 = mt * 32, n0 = nt * 64;
    const __nv_bfloat16 *A = fb.dZb[l], *Bm = fb.H[l];
    // this thread's 16-byte pieces of a chunk (12 to a row: 4 of A, 8 of B)
    constexpr int PC = DW_K * 12 / 128;
    const __nv_bfloat16 *src[PC];
    int dst[PC], prow[PC];
    size_t step[PC];
#pragma unroll
    for (int k = 0; k < PC; k++) {
        const int i = tid + 128 * k, r = i / 12, q = i - r * 12;
        const bool isA = q < 4;
        const int c = isA ? m0 + 8 * q : n0 + 8 * (q - 4), ld = isA ? lda : ldb;
        src[k] = (isA ? A : Bm) + (size_t)r * ld + c;
        step[k] = (size_t)DW_K * ld;
        dst[k] = isA ? r * LA + 8 * q : DW_STAGES * DW_K * LA + r * LB + 8 * (q - 4);
        prow[k] = c < ld ? r : 1 << 30;   // columns past the tensor: zeros
    }
    auto stage = [&](int ch) {
        const int buf = ch % DW_STAGES;
        if (ch < chunks)
#pragma unroll
            for (int k = 0; k < PC; k++) {
                __nv_bfloat16 *d = sA + dst[k] + buf * DW_K * (dst[k] < DW_STAGES * DW_K * LA ? LA : LB);
                if (prow[k] < rows - ch * DW_K) umma::cp_async16(d, src[k] + ch * step[k]);
                else *reinterpret_cast<uint4 *>(d) = make_uint4(0u, 0u, 0u, 0u);
            }
        umma::cp_async_commit();
    };
    const int wm = (warp >> 1) * 16, wn = (warp & 1) * 32, g = lane >> 2, t = lane & 3;
    float acc[4][4];
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
        for (int q = 0; q < 4; q++) acc[j][q] = 0.f;
    for (int ch = 0; ch < DW_STAGES - 1; ch++) stage(ch);
    // the parameters and moments of this thread's outputs, all loaded before
    // any is stored (one by one, a load waited for each update: 10 of 21 us)
    float p[4][4], mo[4][4], ve[4][4];
    auto at = [&](int j, int h) {
        return net.woff[l] + (size_t)(m0 + wm + g + 8 * (h >> 1)) * nin + n0 + wn + 8 * j + 2 * t + (h & 1);
    };
    auto inside = [&](int j, int h) {
        return m0 + wm + g + 8 * (h >> 1) < nout && n0 + wn + 8 * j + 2 * t + (h & 1) < nin;
    };
    if (ADAM)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int h = 0; h < 4; h++)
                if (inside(j, h)) {
                    p[j][h] = ad.p[at(j, h)];
                    mo[j][h] = ad.m[at(j, h)];
                    ve[j][h] = ad.v[at(j, h)];
                } else {
                    p[j][h] = mo[j][h] = ve[j][h] = 0.f;
                }
    for (int ch = 0; ch < chunks; ch++) {
        umma::cp_async_wait<DW_STAGES - 2>();
        __syncthreads();   // chunk ch has arrived; every warp is done with the one the next stage overwrites
        stage(ch + DW_STAGES - 1);
        const __nv_bfloat16 *a0 = sA + (ch % DW_STAGES) * DW_K * LA, *b0 = sB + (ch % DW_STAGES) * DW_K * LB;
        const int kn = min(DW_K, ((rows - ch * DW_K) + 15) / 16 * 16);
        for (int k0 = 0; k0 < kn; k0 += 16) {
            // A fragments from [k][m]: matrices (m 0-7, k 0-7), (m 8-15, k 0-7), (m 0-7, k 8-15), (m 8-15, k 8-15)
            uint32_t a[4], q[2][4];
            umma::ldmatrix4_trans(a, a0 + (k0 + (lane & 7) + 8 * (lane >> 4)) * LA + wm + 8 * ((lane >> 3) & 1));
#pragma unroll
            for (int h = 0; h < 2; h++)
                umma::ldmatrix4_trans(q[h], b0 + (k0 + (lane & 15)) * LB + wn + 16 * h + 8 * (lane >> 4));
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint32_t bb[2] = {q[j >> 1][2 * (j & 1)], q[j >> 1][2 * (j & 1) + 1]};
                umma::mma_sync_bf16(acc[j], a, bb);
            }
        }
    }
    umma::cp_async_wait<0>();
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
        for (int h = 0; h < 4; h++) {
            if (!inside(j, h)) continue;
            if (ADAM) {
                adam(ad, acc[j][h], p[j][h], mo[j][h], ve[j][h]);
                ad.p[at(j, h)] = p[j][h];
                ad.m[at(j, h)] = mo[j][h];
                ad.v[at(j, h)] = ve[j][h];
            } else {
                grads[at(j, h)] = acc[j][h];
            }
        }
    if (ADAM)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int h = 0; h < 4; h += 2)   // (padding columns are 0)
                if (inside(j, h))
                    *reinterpret_cast<uint32_t *>(ad.pk + net.pk[l] +
                                                  tile_at(m0 + wm + g + 4 * h, n0 + wn + 8 * j + 2 * t, net.kp[l])) =
                        pack_bf16x2(p[j][h], inside(j, h + 1) ? p[j][h + 1] : 0.f);
}

// column sums of dZ (B x n) -> db (n): deterministic, one thread per column
__global__ void k_colsum(int B, int n, const float *__restrict__ dZ, float *__restrict__ db) {
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    float s = 0.f;
    for (int r = 0; r < B; r++) s += dZ[(size_t)r * n + c];
    db[c] = s;
}

// gather a minibatch and standardise: Xb = (X[idx] - mx)/sx, Tb = (Y[idx] - my)/sy
__global__ void k_gather(int B, int nin, int nout, const int *__restrict__ idx, const float *__restrict__ X,
                         const float *__restrict__ Y, const float *__restrict__ st, float *__restrict__ Xb,
                         float *__restrict__ Tb) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= B) return;
    const int s = idx[i];
    const float *mx = st, *sx = st + nin, *my = st + 2 * nin, *sy = st + 2 * nin + nout;
    for (int k = 0; k < nin; k++) Xb[(size_t)i * nin + k] = (X[(size_t)s * nin + k] - mx[k]) / sx[k];
    if (Y)
        for (int k = 0; k < nout; k++) Tb[(size_t)i * nout + k] = (Y[(size_t)s * nout + k] - my[k]) / sy[k];
}

// MSE loss and its gradient on standardised targets; loss partials per block
__global__ void k_mse(int n, const float *__restrict__ Yp, const float *__restrict__ T, float scale,
                      float *__restrict__ dY, float *__restrict__ part) {
    __shared__ float red[256];
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    float l = 0.f;
    if (i < n) {
        const float d = Yp[i] - T[i];
        dY[i] = 2.f * d * scale;
        l = d * d * scale;
    }
    red[threadIdx.x] = l;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

// the epoch's loss on the device: one minibatch's block partial sums added,
// in block order, to a running FP64 total (read once per epoch instead of a
// stream synchronisation per minibatch)
__global__ void k_loss_accum(int nb, const float *__restrict__ part, double *__restrict__ acc) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        double s = 0.0;
        for (int b = 0; b < nb; b++) s += part[b];
        *acc += s;
    }
}

__global__ void k_adam(int n, float *__restrict__ p, const float *__restrict__ gr, float *__restrict__ m,
                       float *__restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = gr[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// de-standardise predictions
__global__ void k_unstd(int B, int nout, const float *__restrict__ st_y, float *__restrict__ Y) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= B * nout) return;
    const int k = i % nout;
    Y[i] = Y[i] * st_y[nout + k] + st_y[k];
}

}  // namespace

struct portal_mlp {
    int device = 0;
    cudaStream_t stream = nullptr;
    int n_in = 0, width = 0, depth = 0, n_out = 0, n_layers = 0;
    std::vector<int> fin, fout;
    std::vector<size_t> woff, boff;
    size_t n_params = 0;
    DevBuf<float> params, grads, adam_m, adam_v, stats;
    DevBuf<float> act;   // activations / pre-activations for one batch
    DevBuf<float> xbuf, ybuf, part;
    DevBuf<double> lossacc;  // the running loss of a training epoch
    DevBuf<int> idx;
    // whole-network kernels (layers up to FU_MAX wide)
    bool fused = false, packed = false;  // packed: pk holds the current parameters
    FusedNet net;
    DevBuf<unsigned char> pk;            // packed BF16 weights
    DevBuf<unsigned char> fbuf;          // buffers of a training batch (FusedBatch)
    FusedBatch fb;
    int fcap = 0;                        // rows fb holds
    DevBuf<float> train_x, train_y;      // a training call's rows and
    DevBuf<int> train_perm;              // their order, kept for the next call
    DevBuf<int> tc_err;  // set by a tensor-core GEMM whose completion wait timed out
    int cap_batch = 0;
    long long step = 0;
    std::string err;
};

namespace {

int mlp_fail(portal_mlp *m, int code, const std::string &msg) {
    if (m) m->err = msg;
    return code;
}

#define MCHECK(m, call)                                                                  \
    do {                                                                                 \
        cudaError_t _e = (call);                                                         \
        if (_e != cudaSuccess) {                                                         \
            cudaGetLastError(); /* reported here, not by the next call's launch check */ \
            return mlp_fail((m), PORTAL_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(_e)); \
        }                                                                                \
    } while (0)

// after a stream synchronize: did a tensor-core GEMM give up waiting?
int tc_status(portal_mlp *m) {
    int e = 0;
    if (cudaMemcpy(&e, m->tc_err.p, sizeof e, cudaMemcpyDeviceToHost) != cudaSuccess)
        return mlp_fail(m, PORTAL_ERR_CUDA, "tensor-core status read");
    if (e) return mlp_fail(m, PORTAL_ERR_CUDA, "a tensor-core GEMM timed out waiting for its MMAs");
    return PORTAL_OK;
}

template <bool AK, bool BK>
void gemm(cudaStream_t s, int M, int N, int K, const float *A, int lda, const float *B, int ldb, EpiArgs e) {
    dim3 grid((N + 63) / 64, (M + 63) / 64);
    k_gemm<AK, BK><<<grid, 128, 0, s>>>(M, N, K, A, lda, B, ldb, e);
}

// A(M,K) row-major times W(N,K)^T on the tensor cores (N, K <= 256)
bool gemm_tc_fits(int N, int K) { return N >= 1 && K >= 1 && N <= 256 && K <= 256; }
void gemm_tc(cudaStream_t s, int M, int N, int K, const float *A, const float *W, EpiArgs e, int *err) {
    const int Np = (N + 15) / 16 * 16, Kp = (K + 15) / 16 * 16;
    uint32_t tcols = 32;
    while ((int)tcols < Np) tcols <<= 1;
    const size_t smem = tc_smem_bytes(Np, Kp);
    allow_dyn_smem((const void *)k_gemm_tc);
    static int nsm = 0;
    if (!nsm) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        if (nsm < 1) nsm = 1;
    }
    const int ntiles = (M + TC_M - 1) / TC_M;
    k_gemm_tc<<<std::min(ntiles, nsm), TC_THREADS, smem, s>>>(M, N, K, Np, Kp, tcols, A, W, e, err);
}

// activation workspace layout for a batch of B rows:
//   X (B x n_in) | per layer l: Z_l, H_l (B x fout[l]) | dA, dB (B x max width)
struct Work {
    float *X, *dA, *dB;
    std::vector<float *> Z, H;
};

size_t work_floats(const portal_mlp *m, int B) {
    size_t n = (size_t)B * m->n_in;
    for (int l = 0; l < m->n_layers; l++) n += 2 * (size_t)B * m->fout[l];
    int wmax = std::max(m->width, m->n_out);
    n += 2 * (size_t)B * wmax;
    return n;
}

int ensure_batch(portal_mlp *m, int B) {
    if (B <= m->cap_batch) return PORTAL_OK;
    m->cap_batch = 0;   // (buffers that grow are freed first)
    if (m->act.reserve(work_floats(m, B)) || m->xbuf.reserve((size_t)B * m->n_in) ||
        m->ybuf.reserve((size_t)B * m->n_out) || m->idx.reserve(B) || m->part.reserve((size_t)B * m->n_out / 256 + 2))
        return mlp_fail(m, PORTAL_ERR_NOMEM, "MLP workspace");
    m->cap_batch = B;
    return PORTAL_OK;
}

Work layout(portal_mlp *m, int B) {
    Work w;
    float *p = m->act.p;
    w.X = p;
    p += (size_t)B * m->n_in;
    for (int l = 0; l < m->n_layers; l++) {
        w.Z.push_back(p);
        p += (size_t)B * m->fout[l];
        w.H.push_back(p);
        p += (size_t)B * m->fout[l];
    }
    const int wmax = std::max(m->width, m->n_out);
    w.dA = p;
    p += (size_t)B * wmax;
    w.dB = p;
    return w;
}

// forward of standardised inputs already in w.X; the output layer's result
// goes to w.H.back()
void forward(portal_mlp *m, int B, Work &w) {
    const float *in = w.X;
    int nin = m->n_in;
    for (int l = 0; l < m->n_layers; l++) {
        const bool last = (l == m->n_layers - 1);
        EpiArgs e{last ? EPI_BIAS : EPI_BIAS_SILU, m->fout[l], w.H[l], w.Z[l], m->params.p + m->boff[l]};
        if (gemm_tc_fits(m->fout[l], nin))
            gemm_tc(m->stream, B, m->fout[l], nin, in, m->params.p + m->woff[l], e, m->tc_err.p);
        else
            gemm<true, true>(m->stream, B, m->fout[l], nin, in, nin, m->params.p + m->woff[l], nin, e);
        in = w.H[l];
        nin = m->fout[l];
    }
}

// backward from dY in w.dA (B x n_out); gradients into m->grads
void backward(portal_mlp *m, int B, Work &w) {
    float *dZ = w.dA, *dPrev = w.dB;
    for (int l = m->n_layers - 1; l >= 0; l--) {
        const int nin = m->fin[l], nout = m->fout[l];
        const float *Hin = (l == 0) ? w.X : w.H[l - 1];
        // dW = dZ^T Hin : (nout x B)(B x nin)
        EpiArgs eg{EPI_STORE, nin, m->grads.p + m->woff[l], nullptr, nullptr};
        gemm<false, false>(m->stream, nout, nin, B, dZ, nout, Hin, nin, eg);
        k_colsum<<<(nout + 127) / 128, 128, 0, m->stream>>>(B, nout, dZ, m->grads.p + m->boff[l]);
        if (l > 0) {
            // dZ_prev = (dZ W) * silu'(Z_prev)
            EpiArgs ed{EPI_DSILU, nin, dPrev, w.Z[l - 1], nullptr};
            gemm<true, false>(m->stream, B, nin, nout, dZ, nout, m->params.p + m->woff[l], nin, ed);
            std::swap(dZ, dPrev);
        }
    }
}

// ---- whole-network path: set-up and launches ----
bool fused_fits(const portal_mlp *m) {
    for (int l = 0; l < m->n_layers; l++)
        if (m->fin[l] > FU_MAX || m->fout[l] > FU_MAX) return false;
    return m->n_layers <= FU_MAX_LAYERS;
}

void fused_setup(portal_mlp *m) {
    FusedNet &n = m->net;
    n.n_layers = m->n_layers; n.n_in = m->n_in; n.n_out = m->n_out;
    n.wbuf = 0;
    unsigned off = 0;
    for (int l = 0; l < m->n_layers; l++) {
        n.fin[l] = m->fin[l]; n.fout[l] = m->fout[l];
        n.kp[l] = (m->fin[l] + 15) / 16 * 16;
        n.np[l] = (m->fout[l] + 15) / 16 * 16;
        n.woff[l] = (unsigned)m->woff[l]; n.boff[l] = (unsigned)m->boff[l];
        n.pk[l] = off;
        off += (unsigned)n.np[l] * n.kp[l] * 2;
        // the MMA reads whole tiles of 128 outputs
        n.wbuf = std::max(n.wbuf, (n.np[l] + 127) / 128 * 128 * n.kp[l] * 2);
    }
}

// rows per CTA of a training step: few, as the step is one CTA's serial chain
// while every CTA has an SM of its own (8 -> 256 x 3 -> 40, one batch an epoch
// with its wait and both launches: 32 to 512 rows 60-62 us, with 32 rows a CTA
// 65-75; 2,048 rows 78 and 82).  From about 4,096 rows on, where the CTAs come
// in several waves, 32 would be the better (118 and 107 us; 16,384 rows 364 and
// 324); the warm start's batches are of 512.
constexpr int TRAIN_NB = 16;
template <int NB, bool TRAIN>
int launch_rows(portal_mlp *m, int B, const int *idx, const float *X, const float *T, const float *st, float *Y,
                float scale) {
    const size_t smem = m->net.wbuf + (size_t)NB * FU_MAX * 2 + 3 * 8 + 16 * 8 + (TRAIN ? sizeof(float) * NB * m->n_out : 0);
    auto k = k_mlp_rows<NB, TRAIN>;
    MCHECK(m, allow_dyn_smem((const void *)k));
    k<<<(B + NB - 1) / NB, FU_THREADS, smem, m->stream>>>(m->net, B, idx, X, T, st, m->params.p, m->pk.p, Y,
                                                                   m->fb, scale, m->tc_err.p);
    MCHECK(m, cudaGetLastError());
    return PORTAL_OK;
}

// the packed weights of the current parameters
int fused_pack(portal_mlp *m) {
    if (m->packed) return PORTAL_OK;
    const FusedNet &n = m->net;
    if (m->pk.reserve(n.pk[n.n_layers - 1] + (size_t)n.np[n.n_layers - 1] * n.kp[n.n_layers - 1] * 2))
        return mlp_fail(m, PORTAL_ERR_NOMEM, "packed weights");
    k_pack_weights<<<dim3(32, n.n_layers), 256, 0, m->stream>>>(n, m->params.p, m->pk.p);
    MCHECK(m, cudaGetLastError());
    m->packed = true;
    return PORTAL_OK;
}

// predictions of B device rows; fewer rows per CTA while every CTA has an SM
// of its own (a CTA's time grows with its rows)
int fused_predict(portal_mlp *m, const float *dX, int B, float *dY, int sms) {
    if (int rc = fused_pack(m)) return rc;
    if (B <= 32 * sms) return launch_rows<32, false>(m, B, nullptr, dX, nullptr, m->stats.p, dY, 0.f);
    if (B <= 64 * sms) return launch_rows<64, false>(m, B, nullptr, dX, nullptr, m->stats.p, dY, 0.f);
    return launch_rows<128, false>(m, B, nullptr, dX, nullptr, m->stats.p, dY, 0.f);
}

int fused_reserve(portal_mlp *m, int B) {
    const int rows = (B + 31) / 32 * 32;
    if (rows <= m->fcap) return PORTAL_OK;
    const FusedNet &n = m->net;
    size_t off = 0;
    auto take = [&](size_t bytes) { const size_t o = off; off += (bytes + 255) & ~(size_t)255; return o; };
    size_t oZ[FU_MAX_LAYERS], odZ[FU_MAX_LAYERS], oH[FU_MAX_LAYERS], odb[FU_MAX_LAYERS];
    for (int l = 0; l < n.n_layers; l++) {
        oZ[l] = take(sizeof(float) * (size_t)rows * n.fout[l]);
        odZ[l] = take(sizeof(float) * (size_t)rows * n.fout[l]);
        oH[l] = take(2 * (size_t)rows * n.kp[l]);
        odb[l] = take(2 * (size_t)rows * n.np[l]);
    }
    const size_t oL = take(sizeof(double) * (size_t)(rows / TRAIN_NB));
    m->fcap = 0;
    if (m->fbuf.reserve(off)) return mlp_fail(m, PORTAL_ERR_NOMEM, "MLP workspace");
    for (int l = 0; l < n.n_layers; l++) {
        m->fb.Z[l] = reinterpret_cast<float *>(m->fbuf.p + oZ[l]);
        m->fb.dZ[l] = reinterpret_cast<float *>(m->fbuf.p + odZ[l]);
        m->fb.H[l] = reinterpret_cast<__nv_bfloat16 *>(m->fbuf.p + oH[l]);
        m->fb.dZb[l] = reinterpret_cast<__nv_bfloat16 *>(m->fbuf.p + odb[l]);
    }
    m->fb.loss = reinterpret_cast<double *>(m->fbuf.p + oL);
    m->fcap = rows;
    return PORTAL_OK;
}

// forward, loss and dZ chain of a batch, then its gradients (grads) or an
// Adam step (ad)
int fused_step(portal_mlp *m, int B, const int *idx, const float *X, const float *T, const float *st, float *grads,
               const AdamArgs *ad, double *loss_acc) {
    if (int rc = fused_pack(m)) return rc;
    if (int rc = launch_rows<TRAIN_NB, true>(m, B, idx, X, T, st, nullptr, 1.f / (float)(B * m->n_out))) return rc;
    int blocks = 0;
    for (int l = 0; l < m->n_layers; l++) {
        const int tm = (m->fout[l] + 31) / 32;
        blocks += tm * ((m->fin[l] + 63) / 64) + tm;
    }
    const int n_loss = (B + TRAIN_NB - 1) / TRAIN_NB;
    MCHECK(m, allow_dyn_smem(ad ? (const void *)k_mlp_grads<true> : (const void *)k_mlp_grads<false>));
    if (ad)
        k_mlp_grads<true><<<blocks, 128, DW_SMEM, m->stream>>>(m->net, B, m->fb, nullptr, *ad, n_loss, loss_acc);
    else
        k_mlp_grads<false><<<blocks, 128, DW_SMEM, m->stream>>>(m->net, B, m->fb, grads, AdamArgs{}, n_loss, loss_acc);
    MCHECK(m, cudaGetLastError());
    return PORTAL_OK;
}

}  // namespace

extern "C" int portal_mlp_create(portal_mlp **out, int device, int n_in, int width, int depth, int n_out,
                                 unsigned long long seed) {
    if (!out || n_in < 1 || width < 1 || depth < 1 || n_out < 1 || width > 4096 || depth > 16)
        return PORTAL_ERR_ARG;
    *out = nullptr;
    if (cudaSetDevice(device) != cudaSuccess) return PORTAL_ERR_NODEVICE;
    portal_mlp *m = new portal_mlp();
    m->device = device;
    m->n_in = n_in; m->width = width; m->depth = depth; m->n_out = n_out;
    m->n_layers = depth + 1;
    size_t off = 0;
    for (int l = 0; l < m->n_layers; l++) {
        const int fi = (l == 0) ? n_in : width, fo = (l == m->n_layers - 1) ? n_out : width;
        m->fin.push_back(fi);
        m->fout.push_back(fo);
        m->woff.push_back(off);
        off += (size_t)fi * fo;
        m->boff.push_back(off);
        off += fo;
    }
    m->n_params = off;
    if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess ||
        m->params.reserve(off) || m->grads.reserve(off) || m->adam_m.reserve(off) || m->adam_v.reserve(off) ||
        m->stats.reserve(2 * (size_t)(n_in + n_out)) || m->tc_err.reserve(1)) {
        delete m;
        return PORTAL_ERR_NOMEM;
    }
    cudaMemset(m->tc_err.p, 0, sizeof(int));
    m->fused = fused_fits(m);
    if (m->fused) fused_setup(m);
    // He-uniform weights, zero biases, identity standardisation
    std::mt19937_64 rng(seed);
    std::vector<float> h(off, 0.f);
    for (int l = 0; l < m->n_layers; l++) {
        const float bound = std::sqrt(6.f / (float)m->fin[l]);
        std::uniform_real_distribution<float> u(-bound, bound);
        for (size_t i = 0; i < (size_t)m->fin[l] * m->fout[l]; i++) h[m->woff[l] + i] = u(rng);
    }
    std::vector<float> st(2 * (size_t)(n_in + n_out), 0.f);
    for (int k = 0; k < n_in; k++) st[n_in + k] = 1.f;
    for (int k = 0; k < n_out; k++) st[2 * n_in + n_out + k] = 1.f;
    cudaMemcpy(m->params.p, h.data(), off * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemcpy(m->stats.p, st.data(), st.size() * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemset(m->adam_m.p, 0, off * sizeof(float));
    cudaMemset(m->adam_v.p, 0, off * sizeof(float));
    *out = m;
    return PORTAL_OK;
}

extern "C" int portal_mlp_destroy(portal_mlp *m) {
    if (!m) return PORTAL_OK;
    cudaSetDevice(m->device);
    if (m->stream) {
        cudaStreamSynchronize(m->stream);
        cudaStreamDestroy(m->stream);
    }
    delete m;
    return PORTAL_OK;
}

extern "C" const char *portal_mlp_last_error(const portal_mlp *m) { return m ? m->err.c_str() : ""; }

extern "C" long long portal_mlp_num_params(const portal_mlp *m) { return m ? (long long)m->n_params : 0; }

extern "C" int portal_mlp_get_params(const portal_mlp *m, float *params, float *stats) {
    if (!m) return PORTAL_ERR_ARG;
    cudaSetDevice(m->device);
    if (params && cudaMemcpy(params, m->params.p, m->n_params * sizeof(float), cudaMemcpyDeviceToHost)) return PORTAL_ERR_CUDA;
    if (stats && cudaMemcpy(stats, m->stats.p, 2 * (size_t)(m->n_in + m->n_out) * sizeof(float),
                            cudaMemcpyDeviceToHost)) return PORTAL_ERR_CUDA;
    return PORTAL_OK;
}

extern "C" int portal_mlp_set_params(portal_mlp *m, const float *params, const float *stats) {
    if (!m) return PORTAL_ERR_ARG;
    cudaSetDevice(m->device);
    if (params) m->packed = false;
    if (params && cudaMemcpy(m->params.p, params, m->n_params * sizeof(float), cudaMemcpyHostToDevice)) return PORTAL_ERR_CUDA;
    if (stats && cudaMemcpy(m->stats.p, stats, 2 * (size_t)(m->n_in + m->n_out) * sizeof(float),
                            cudaMemcpyHostToDevice)) return PORTAL_ERR_CUDA;
    return PORTAL_OK;
}

// one forward + backward on standardised (X, T) given on the host: loss and
// the flat gradient (same layout as the parameters)
extern "C" int portal_mlp_gradients(portal_mlp *m, const float *X, const float *T, int B, float *grads,
                                    float *loss) {
    if (!m || !X || !T || B < 1) return PORTAL_ERR_ARG;
    cudaSetDevice(m->device);
    if (m->fused && !fused_reserve(m, B)) {   // (layer by layer where its buffers do not fit)
        int rc = PORTAL_OK;
        if (m->xbuf.reserve((size_t)B * m->n_in) || m->ybuf.reserve((size_t)B * m->n_out))
            return mlp_fail(m, PORTAL_ERR_NOMEM, "MLP workspace");
        MCHECK(m, cudaMemcpyAsync(m->xbuf.p, X, (size_t)B * m->n_in * sizeof(float), cudaMemcpyHostToDevice, m->stream));
        MCHECK(m, cudaMemcpyAsync(m->ybuf.p, T, (size_t)B * m->n_out * sizeof(float), cudaMemcpyHostToDevice, m->stream));
        if ((rc = fused_step(m, B, nullptr, m->xbuf.p, m->ybuf.p, nullptr, m->grads.p, nullptr, nullptr))) return rc;
        std::vector<double> parts((B + TRAIN_NB - 1) / TRAIN_NB);
        MCHECK(m, cudaMemcpyAsync(parts.data(), m->fb.loss, parts.size() * sizeof(double), cudaMemcpyDeviceToHost, m->stream));
        if (grads)
            MCHECK(m, cudaMemcpyAsync(grads, m->grads.p, m->n_params * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
        MCHECK(m, cudaStreamSynchronize(m->stream));
        if ((rc = tc_status(m))) return rc;
        double s = 0.0;
        for (double p : parts) s += p;
        if (loss) *loss = (float)s;
        return PORTAL_OK;
    }
    int rc = ensure_batch(m, B);
    if (rc) return rc;
    Work w = layout(m, B);
    MCHECK(m, cudaMemcpyAsync(w.X, X, (size_t)B * m->n_in * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    MCHECK(m, cudaMemcpyAsync(m->ybuf.p, T, (size_t)B * m->n_out * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    forward(m, B, w);
    const int n = B * m->n_out, nb = (n + 255) / 256;
    k_mse<<<nb, 256, 0, m->stream>>>(n, w.H.back(), m->ybuf.p, 1.f / (float)n, w.dA, m->part.p);
    backward(m, B, w);
    MCHECK(m, cudaGetLastError());
    std::vector<float> parts(nb);
    MCHECK(m, cudaMemcpyAsync(parts.data(), m->part.p, nb * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    if (grads)
        MCHECK(m, cudaMemcpyAsync(grads, m->grads.p, m->n_params * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    MCHECK(m, cudaStreamSynchronize(m->stream));
    if (int rc2 = tc_status(m)) return rc2;
    if (loss) {
        double s = 0.0;
        for (float p : parts) s += p;
        *loss = (float)s;
    }
    return PORTAL_OK;
}

// Train on (X, Y) (host, raw units): the standardisation statistics are taken
// from this data set, then `epochs` passes of shuffled minibatches with Adam.
extern "C" int portal_mlp_train(portal_mlp *m, const float *X, const float *Y, int M, int epochs, int batch,
                                float lr, unsigned long long seed, float *loss_per_epoch) {
    if (!m || !X || !Y || M < 1 || epochs < 1 || batch < 1) return PORTAL_ERR_ARG;
    cudaSetDevice(m->device);
    const int nin = m->n_in, nout = m->n_out;
    // statistics (FP64 on the host)
    std::vector<float> st(2 * (size_t)(nin + nout));
    // (row by row: a column's sums run over the rows in order, and the columns
    // of a row are next to each other in memory)
    auto column_stats = [M](const float *A, int n, float *mean, float *dev) {
        std::vector<double> s(n, 0.0), s2(n, 0.0);
        for (int i = 0; i < M; i++)
            for (int k = 0; k < n; k++) {
                const double v = A[(size_t)i * n + k];
                s[k] += v;
                s2[k] += v * v;
            }
        for (int k = 0; k < n; k++) {
            const double mu = s[k] / M;
            mean[k] = (float)mu;
            dev[k] = (float)std::sqrt(std::max(s2[k] / M - mu * mu, 1e-12));
        }
    };
    column_stats(X, nin, st.data(), st.data() + nin);
    column_stats(Y, nout, st.data() + 2 * nin, st.data() + 2 * nin + nout);
    MCHECK(m, cudaMemcpyAsync(m->stats.p, st.data(), st.size() * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    DevBuf<float> &dX = m->train_x, &dY = m->train_y;
    // the rows are kept for the next call up to KEEP_BYTES
    struct KeepSmall {
        portal_mlp *m;
        ~KeepSmall() {
            if (sizeof(float) * (m->train_x.n + m->train_y.n) + sizeof(int) * m->train_perm.n <= KEEP_BYTES) return;
            cudaStreamSynchronize(m->stream);
            m->train_x.release();
            m->train_y.release();
            m->train_perm.release();
        }
    } keep{m};
    if (dX.reserve((size_t)M * nin) || dY.reserve((size_t)M * nout)) return mlp_fail(m, PORTAL_ERR_NOMEM, "MLP data");
    MCHECK(m, cudaMemcpyAsync(dX.p, X, (size_t)M * nin * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    MCHECK(m, cudaMemcpyAsync(dY.p, Y, (size_t)M * nout * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    const int B = std::min(batch, M);
    // (layer by layer where the whole-network kernels' buffers do not fit)
    const bool fused = m->fused && !fused_reserve(m, B);
    int rc = fused ? fused_pack(m) : ensure_batch(m, B);
    if (rc) return rc;
    Work w;
    if (!fused) {
        w = layout(m, B);
        m->packed = false;   // (k_adam updates the parameters alone)
    }
    std::mt19937_64 rng(seed);
    std::vector<int> perm(M);
    for (int i = 0; i < M; i++) perm[i] = i;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    DevBuf<int> &pidx = m->train_perm;
    if (pidx.reserve(M)) return mlp_fail(m, PORTAL_ERR_NOMEM, "MLP permutation");
    std::shuffle(perm.begin(), perm.end(), rng);
    for (int ep = 0; ep < epochs; ep++) {
        int nbatch = 0;
        MCHECK(m, cudaMemcpyAsync(pidx.p, perm.data(), (size_t)M * sizeof(int), cudaMemcpyHostToDevice, m->stream));
        if (loss_per_epoch) {
            if (m->lossacc.reserve(1)) return mlp_fail(m, PORTAL_ERR_NOMEM, "loss accumulator");
            MCHECK(m, cudaMemsetAsync(m->lossacc.p, 0, sizeof(double), m->stream));
        }
        MCHECK(m, cudaStreamSynchronize(m->stream));  // perm is rewritten next epoch
        for (int b0 = 0; fused && b0 + B <= M; b0 += B, nbatch++) {
            m->step++;
            const AdamArgs ad{m->params.p, m->adam_m.p, m->adam_v.p, m->pk.p, lr, b1, b2, eps,
                              1.f - std::pow(b1, (float)m->step), 1.f - std::pow(b2, (float)m->step)};
            if ((rc = fused_step(m, B, pidx.p + b0, dX.p, dY.p, m->stats.p, nullptr, &ad,
                                 loss_per_epoch ? m->lossacc.p : nullptr)))
                return rc;
        }
        for (int b0 = 0; !fused && b0 + B <= M; b0 += B) {
            k_gather<<<(B + 127) / 128, 128, 0, m->stream>>>(B, nin, nout, pidx.p + b0, dX.p, dY.p, m->stats.p, w.X,
                                                             m->ybuf.p);
            forward(m, B, w);
            const int n = B * nout, nb = (n + 255) / 256;
            k_mse<<<nb, 256, 0, m->stream>>>(n, w.H.back(), m->ybuf.p, 1.f / (float)n, w.dA, m->part.p);
            backward(m, B, w);
            m->step++;
            const float c1 = 1.f - std::pow(b1, (float)m->step), c2 = 1.f - std::pow(b2, (float)m->step);
            k_adam<<<(int)((m->n_params + 255) / 256), 256, 0, m->stream>>>((int)m->n_params, m->params.p, m->grads.p,
                                                                          m->adam_m.p, m->adam_v.p, lr, b1, b2,
                                                                          eps, c1, c2);
            if (loss_per_epoch) k_loss_accum<<<1, 32, 0, m->stream>>>(nb, m->part.p, m->lossacc.p);
            nbatch++;
        }
        MCHECK(m, cudaGetLastError());
        if (ep + 1 < epochs) std::shuffle(perm.begin(), perm.end(), rng);   // the next epoch's, while this one runs
        if (loss_per_epoch) {
            double eloss = 0.0;
            MCHECK(m, cudaMemcpyAsync(&eloss, m->lossacc.p, sizeof(double), cudaMemcpyDeviceToHost, m->stream));
            MCHECK(m, cudaStreamSynchronize(m->stream));
            loss_per_epoch[ep] = (float)(eloss / std::max(nbatch, 1));
        }
    }
    MCHECK(m, cudaStreamSynchronize(m->stream));
    return tc_status(m);
}

// Predict raw-unit outputs for raw inputs X (host or device pointers as
// flagged).  B rows.
extern "C" int portal_mlp_predict(portal_mlp *m, const float *X, int B, float *Y) {
    if (!m || !X || !Y || B < 1) return PORTAL_ERR_ARG;
    cudaSetDevice(m->device);
    const int chunk = 65536;
    if (m->fused) {
        const int n = std::min(B, chunk);
        if (m->xbuf.reserve((size_t)n * m->n_in) || m->ybuf.reserve((size_t)n * m->n_out))
            return mlp_fail(m, PORTAL_ERR_NOMEM, "MLP predict");
        int sms = 0;
        MCHECK(m, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m->device));
        for (int b0 = 0; b0 < B; b0 += chunk) {
            const int nb = std::min(chunk, B - b0);
            MCHECK(m, cudaMemcpyAsync(m->xbuf.p, X + (size_t)b0 * m->n_in, (size_t)nb * m->n_in * sizeof(float),
                                      cudaMemcpyHostToDevice, m->stream));
            if (int rc = fused_predict(m, m->xbuf.p, nb, m->ybuf.p, sms)) return rc;
            MCHECK(m, cudaMemcpyAsync(Y + (size_t)b0 * m->n_out, m->ybuf.p, (size_t)nb * m->n_out * sizeof(float),
                                      cudaMemcpyDeviceToHost, m->stream));
            MCHECK(m, cudaStreamSynchronize(m->stream));
        }
        return tc_status(m);
    }
    int rc = ensure_batch(m, std::min(B, chunk));
    if (rc) return rc;
    DevBuf<float> dXr;
    if (dXr.reserve((size_t)std::min(B, chunk) * m->n_in)) return mlp_fail(m, PORTAL_ERR_NOMEM, "MLP predict");
    DevBuf<int> iota;
    std::vector<int> h(std::min(B, chunk));
    for (size_t i = 0; i < h.size(); i++) h[i] = (int)i;
    if (iota.reserve(h.size())) return mlp_fail(m, PORTAL_ERR_NOMEM, "MLP predict");
    MCHECK(m, cudaMemcpyAsync(iota.p, h.data(), h.size() * sizeof(int), cudaMemcpyHostToDevice, m->stream));
    for (int b0 = 0; b0 < B; b0 += chunk) {
        const int nb = std::min(chunk, B - b0);
        Work w = layout(m, nb);
        MCHECK(m, cudaMemcpyAsync(dXr.p, X + (size_t)b0 * m->n_in, (size_t)nb * m->n_in * sizeof(float),
                                  cudaMemcpyHostToDevice, m->stream));
        k_gather<<<(nb + 127) / 128, 128, 0, m->stream>>>(nb, m->n_in, m->n_out, iota.p, dXr.p, nullptr, m->stats.p,
                                                          w.X, nullptr);
        forward(m, nb, w);
        k_unstd<<<(nb * m->n_out + 255) / 256, 256, 0, m->stream>>>(nb, m->n_out, m->stats.p + 2 * m->n_in,
                                                                   w.H.back());
        MCHECK(m, cudaMemcpyAsync(Y + (size_t)b0 * m->n_out, w.H.back(), (size_t)nb * m->n_out * sizeof(float),
                                  cudaMemcpyDeviceToHost, m->stream));
        MCHECK(m, cudaStreamSynchronize(m->stream));
    }
    MCHECK(m, cudaGetLastError());
    return tc_status(m);
}
