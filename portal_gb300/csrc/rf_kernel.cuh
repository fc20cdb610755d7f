// The radiation-field kernel (the template shared by the single-model calls
// in rf.cu and the batched launch in rf_batch.cu) and the line-table kernel.
// See rf.cu for the algorithm.
#pragma once

#include <type_traits>

#include <cmath>

#include <algorithm>

#include "internal.cuh"

using namespace portal;

namespace {

constexpr float LOG2E_F = 1.4426950408889634f;
// sqrt(log2 e): a profile argument q scaled by it gives exp(-q^2) = 2^(-q'^2),
// one ex2 of q'^2 with the sign folded into the instruction
constexpr float SQL2E_F = 1.2011224087864498f;
// line-centre optical depth (log2 units) below which every channel of a cell
// takes the Taylor form: x = A g <= A with the profile g = ex2(-q'^2) <= 1
// (ex2 of a non-positive argument does not exceed 1: checked over every float
// of [-1/16, 0]), below the switch OM_TAYLOR_X of one_minus_exp with 0.5 % to
// spare
constexpr float OM_THIN_A = 0.0625f;
// Face crossings closer than this (in units of r_max) are not taken.  The
// reference uses 1e-10 (miscellaneous.f90:1048) against FP64 noise ~1e-16;
// the FP32 walk's noise in t is ~1e-9, and a crossing shorter than 2e-8 is
// 0.02 trace steps, i.e. it contributes nint(...) = 0 steps either way.
constexpr float FACE_EPS = 2e-8f;

struct LineConst {
    double nu, A, B, kd, glo, gup, bb_cmb;
    int lo, up;
};
constexpr int MAX_LINES = 64;

// Compensated (Kahan) FP32 sum: J of one node is a sum of a few hundred ray
// contributions; the compensation keeps it to ~1e-7 of the sum of magnitudes
// without the FP64 pipe.  The terms are passed as explicitly rounded products
// (__fmul_rn at the call sites) and summed with explicit roundings: a
// multiply the compiler fuses into the first subtraction in one kernel
// variant and not in another would make the result depend on the line
// grouping of the variant.
struct KahanF {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float x) {
        const float y = __fsub_rn(x, c);
        const float t = __fadd_rn(s, y);
        c = __fsub_rn(__fsub_rn(t, s), y);
        s = t;
    }
    __device__ __forceinline__ double value() const { return (double)s - (double)c; }
};

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// A node's frame, the part of the ray set-up that all its rays share: b(3), x
// = b x g / |b x g| (3), x x b (3), its position p(3), |p|^2 - 1 as
// pos_quadratic forms it.  One thread per bulk node (the FP64 pipe takes a
// warp's instruction in 16 cycles whether one lane or all use it: formed by
// one lane per item, the frames took a tenth of a 4,096-point pass).
constexpr int FRAME_N = 13;
__device__ __forceinline__ void node_frame(int node, const double *__restrict__ bvec, const double *__restrict__ pos,
                                           double gx, double gy, double gz, double *__restrict__ frames) {
    // find_dir miscellaneous.f90:48-82:
    // dir = R(b,ph) R(x,th) b = cos th b + sin th (cos ph (x x b) + sin ph x)
    const double bx = bvec[3 * (size_t)node], by = bvec[3 * (size_t)node + 1], bz = bvec[3 * (size_t)node + 2];
    double xx = by * gz - bz * gy, xy = bz * gx - bx * gz, xz = bx * gy - by * gx;
    const double xn = sqrt(xx * xx + xy * xy + xz * xz);
    xx /= xn; xy /= xn; xz /= xn;
    const double px = pos[3 * (size_t)node], py = pos[3 * (size_t)node + 1], pz = pos[3 * (size_t)node + 2];
    const double np = __dsqrt_rn(dsum3sq(px, py, pz));
    double *f = frames + FRAME_N * (size_t)node;
    f[0] = bx; f[1] = by; f[2] = bz; f[3] = xx; f[4] = xy; f[5] = xz;
    f[6] = xy * bz - xz * by; f[7] = xz * bx - xx * bz; f[8] = xx * by - xy * bx;
    f[9] = px; f[10] = py; f[11] = pz; f[12] = __dsub_rn(__dmul_rn(np, np), 1.0);
}

// sphere_exit for a direction of unit length up to rounding, with c = |p|^2 -
// 1 given: the same values with a third of the FP64 instructions.  With s =
// |d|^2 = 1 + e, e a few ulp, sqrt(s) = 1 + e/2 - e^2/8 lies just below 1 +
// e/2, which is a double or halfway between two: rounding 1 + e/2 downwards
// rounds sqrt(s) correctly.  The quotient by 2 a = 2 (1 + h), h a few ulp, is
// q - q (h - h^2) with q = n/2, rounded once (h^2 decides where q - q h lies
// halfway between two doubles: rays that leave a node on the sphere at once
// have an n of few bits); and of the two roots only the one taken is divided.
__device__ __forceinline__ double sphere_exit_unit(double px, double py, double pz, double c, double dx, double dy,
                                                   double dz) {
    const double s = dsum3sq(dx, dy, dz), e = __dsub_rn(s, 1.0);
    const bool unit = fabs(e) < 0x1p-40;
    const double nd = unit ? __dadd_rd(1.0, __dmul_rn(0.5, e)) : __dsqrt_rn(s);
    const double a = __dmul_rn(nd, nd);
    const double b = __dmul_rn(2.0, ddot3(px, py, pz, dx, dy, dz));
    const double dis = __dsub_rn(__dmul_rn(b, b), __dmul_rn(__dmul_rn(4.0, a), c));
    if (!(dis > 0.0)) return 0.0;
    const double sq = __dsqrt_rn(dis);
    const double n2 = __dsub_rn(-b, sq), n = (n2 > 0.0) ? n2 : __dadd_rn(-b, sq);
    if (!unit) return __ddiv_rn(n, __dmul_rn(2.0, a));
    const double q = __dmul_rn(0.5, n), h = __dsub_rn(a, 1.0);
    return __fma_rn(-q, __fma_rn(-h, h, h), q);
}

constexpr int RF_MAX_GROUP = 10;          // lines per group without dust
constexpr int RF_MAX_GROUP_DUST = 5;      // with dust (a wider body costs more in registers than it gains)

// The line table's layout: a node's row holds its lines as the cells are staged,
// group by group in packs of two lines, (A, A', S, S') and, with dust, (Ad,
// Ad', Jd, Jd'): one 16-byte load a pack where (A, S, Ad, Jd) per line took
// two of 8, half of the bytes unused.  (Field kernels: 65,536 points x 9 lines
// 309 -> 305 ms, 8,192 x 19 76.6 -> 75.2, 4,096 x 4 1.69 -> 1.67, 6,001 x 7 with
// dust 4.83 -> 4.72.)
struct TabShape {
    int nlg, npk, dust, width;   // width: float4 per node
};
__host__ __device__ inline TabShape tab_shape(int L, int max_group, bool dust) {
    TabShape t;
    const int cap = (dust && max_group > RF_MAX_GROUP_DUST) ? RF_MAX_GROUP_DUST : max_group;
    const int groups = (L + cap - 1) / cap;
    t.nlg = (L + groups - 1) / groups;
    t.npk = (t.nlg + 1) / 2;
    t.dust = dust;
    t.width = groups * (dust ? 2 : 1) * t.npk;
    return t;
}

// Line table and zeroed fields, one thread per (node, line), and -- the blocks
// after its own -- the node frames and what else a pass starts from zero, one
// thread per node.  (One launch instead of nine: at 1,700 nodes the memsets
// were two thirds of the 38 us before the walk.)
__global__ void k_line_table(int N, int L, double dxp, const LineConst *__restrict__ lines,
                             const double *__restrict__ levp, int nlev, const double *__restrict__ b,
                             const double *__restrict__ dustp, const double *__restrict__ tdust,
                             float4 *__restrict__ ltab, TabShape ts, RFArgs a, int table_blocks) {
    if ((int)blockIdx.x >= table_blocks) {
        const int node = (int)((blockIdx.x - table_blocks) * blockDim.x + threadIdx.x);
        if (node < 8) a.counters[node] = 0;
        if (node < N) {
            a.status[node] = 0;
            a.segs[node] = 0;
#pragma unroll
            for (int k = 0; k < 6; k++) a.kmom[(size_t)k * N + node] = 0.f;
        }
        if (node < a.bulk) node_frame(node, a.bvec, a.pos, a.gx, a.gy, a.gz, a.frames);
        return;
    }
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)N * L) return;
    int n = (int)(t / L), l = (int)(t - (long long)n * L);
    a.J0[t] = a.J2[t] = 0.0;
    if (a.JE) a.JE[t] = a.LS[t] = 0.0;
    const LineConst lc = lines[l];
    double p1 = levp[(size_t)nlev * n + lc.lo];
    double p2 = levp[(size_t)nlev * n + lc.up];
    // ray_in inverse_rt.f90:263-266, 293-294, 298-301
    double c1 = 2.2102191e-42 * lc.nu;
    double c2 = 5.272859e-35 * lc.nu;
    double cnu = 299792458.0 / lc.nu;
    double kv = c1 * lc.B * (p1 - lc.glo * p2 / lc.gup);
    double ev = c2 * lc.A * p2;
    double phif = cnu / (1.7724538509055160273 * b[n]) * dxp;
    double Ad = lc.kd * dustp[n] * dxp;
    double Td = tdust[n];
    double Ibb = 0.0;
    if (Td != 0.0) {  // black_body miscellaneous.f90:263-285
        double c2b = 4.79924e-11 / Td;
        Ibb = 1.4744995e-50 * lc.nu * lc.nu * lc.nu / (exp(c2b * lc.nu) - 1.0);
    }
    // optical depth per trace step at unit profile, line source function
    // ev/kv and, with dust, dust optical depth per step, dust emissivity per
    // step: the source function is stored as the FP64 ratio, not the
    // emissivity, so a weak line's S keeps full FP32 precision where kv and ev
    // alone would be FP32 denormals
    const float A = (float)(kv * phif), S = (float)(kv != 0.0 ? ev / kv : 0.0);
    const int g = l / ts.nlg, i0 = l - g * ts.nlg;
    // (an odd group's last pack and a last group's padding repeat the line)
    const int i1 = (l == L - 1 || i0 == ts.nlg - 1) ? 2 * ts.npk : i0 + 1;
    float *row = reinterpret_cast<float *>(ltab + (size_t)n * ts.width);
    for (int i = i0; i < i1; i++) {
        float *p = row + 4 * ((ts.dust ? 2 : 1) * (g * ts.npk + i / 2)) + (i & 1);
        p[0] = A;
        p[2] = S;
        if (ts.dust) {
            p[4] = (float)Ad;
            p[6] = (float)(Ad * Ibb);
        }
    }
}

constexpr double PI_D = 3.141592653589793;  // acos(-1.d0)

// star_all (miscellaneous.f90:1139-1226, circle_points :1228-1265) for ray
// i of a node outside the star: (cos th, ph) of the ray in the field frame
// and its quadrature weight.  sk as in RayBatchStar; f the node frame b (0-2),
// x = b x g / |b x g| (3-5), x x b (6-8).  The first n_star rays cover the
// star's cone (one ray: the reference's x(1:2) = cos(1), i.e. 1 rad off the
// star direction; fewer than ten: a circle at th_star / 2; more: Vogel's
// spiral), the others nth bands of ceiling(nph sin th) rays from th_star to
// pi about the star direction.  Each direction, built about the star
// direction with find_dir (gauge g), is re-expressed by find_angles in the
// field frame (miscellaneous.f90:86-134).
// Returns the direction's (cos th, sin th, cos ph, sin ph) in the field
// frame as inverse_rt rebuilds it (find_dir of acos(mu), ph) and stores the
// weights (w, w c_in / sqrt 2) in *wts.  Out of line: the default path
// keeps the kernel's own code.
// a ray direction in the field frame: (cos th, sin th, cos ph, sin ph)
struct RayDir {
    double ct, st, cp, sp;
};
__device__ __noinline__ RayDir star_ray(const double *sk, int n_star, int i, int nth, int nph, double gx,
                                         double gy, double gz, const double *f, float2 *wts) {
    double x1 = 1.0, x2 = 0.0, w = 0.0;
    if (i < n_star) {
        const double ths = sk[3], dth = sk[4];
        if (n_star == 1) {
            x1 = cos(1.0);
            x2 = cos(1.0);
            w = 2.0 * PI_D * dth;
        } else if (n_star < 10) {
            const double wph = 2.0 * PI_D / n_star;
            x1 = cos(ths / 2.0);
            x2 = i * wph;
            w = wph * dth;
        } else {
            x1 = cos(ths * sqrt(1.0 * (i + 1) / n_star));
            x2 = (i + 1) * (PI_D * (3.0 - sqrt(5.0)));
            w = dth * 2.0 * PI_D / n_star;
        }
        w = w / (4.0 * PI_D);
    } else {
        const double dr = sk[5], thi = sk[6];
        int j = i - n_star, b = 1, np = 1;
        double th = thi;
        for (; b <= nth; b++) {
            th = (b - 1) * dr + thi;
            np = (int)ceil(nph * sin(th));
            if (j < np) break;
            j -= np;
        }
        if (b <= nth) {
            double wth;
            if (b == 1) wth = cos(sk[3]) - cos((b - 0.5) * dr + thi);
            else if (b == nth) wth = cos((b - 1.5) * dr + thi) + 1.0;
            else wth = cos((b - 1.5) * dr + thi) - cos((b - 0.5) * dr + thi);
            const double wph = 2.0 * PI_D / np;
            x1 = cos(th);
            x2 = j * wph;
            w = wth * wph / (4.0 * PI_D);
        }
    }
    // find_dir about k: x_k = k x g / |k x g|, d = cos t k + sin t (cos x2 (x_k x k) + sin x2 x_k)
    const double kx = sk[0], ky = sk[1], kz = sk[2];
    double ux = ky * gz - kz * gy, uy = kz * gx - kx * gz, uz = kx * gy - ky * gx;
    const double un = sqrt(ux * ux + uy * uy + uz * uz);
    ux /= un; uy /= un; uz /= un;
    const double vx = uy * kz - uz * ky, vy = uz * kx - ux * kz, vz = ux * ky - uy * kx;
    const double t = acos(x1), ct = cos(t), st = sin(t), cp = cos(x2), sp = sin(x2);
    const double dx = ct * kx + st * (cp * vx + sp * ux);
    const double dy = ct * ky + st * (cp * vy + sp * uy);
    const double dz = ct * kz + st * (cp * vz + sp * uz);
    // find_angles in the field frame
    const double bd = f[0] * dx + f[1] * dy + f[2] * dz;
    const double thb = (bd > 1.0) ? 0.0 : (bd < -1.0) ? PI_D : acos(bd);
    const double cx = f[1] * dz - f[2] * dy, cy = f[2] * dx - f[0] * dz, cz = f[0] * dy - f[1] * dx;
    const double mub = cos(thb);
    const double phb = atan2(f[3] * dx + f[4] * dy + f[5] * dz, f[3] * cx + f[4] * cy + f[5] * cz);
    *wts = make_float2((float)w, (float)(w * ((3.0 * mub * mub - 1.0) / 2.0) / sqrt(2.0)));
    const double th = acos(mub);
    return RayDir{cos(th), sin(th), cos(phb), sin(phb)};
}

// trace_node's star geometry (main_sub.f90:56-66) and star_all's ray counts
// for the node at p: fills sk and sn of the warp's RayBatchStar.
__device__ __noinline__ void star_node(double *sk, int *sn, double xs, double ys, double zs, double Rs, int nth,
                                       int nph, double px, double py, double pz) {
    const double kx = xs - px, ky = ys - py, kz = zs - pz;
    const double d = sqrt(kx * kx + ky * ky + kz * kz);
    const double q = Rs / d;
    const double dOm = PI_D * (q * q);
    sk[0] = kx / d; sk[1] = ky / d; sk[2] = kz / d;
    const double dth = dOm / (2.0 * PI_D);
    const double ths = acos(1 - dth);
    const double dOm_max = 4.0 * PI_D / (nth * nph);
    const int ns = (int)ceil(dOm / dOm_max);
    const double dr = (PI_D - ths) / nth, thi = ths + dr / 2.0;
    sk[3] = ths; sk[4] = dth; sk[5] = dr; sk[6] = thi;
    int nv = ns;
    for (int b = 1; b <= nth; b++) nv += (int)ceil(nph * sin((b - 1) * dr + thi));
    sn[0] = ns;
    // the reference stops when the rays exceed nth nph (miscellaneous.f90:1203-1206)
    sn[1] = (ns > nth * nph || nv > nth * nph) ? -1 : nv;
}

// check_neigh_fast's star test (miscellaneous.f90:1056-1069) from the node
// at p along d: the star's surface, when the ray meets it first, ends it.
__device__ __noinline__ double star_exit(double sexit, double px, double py, double pz, double dx, double dy,
                                         double dz, double xs, double ys, double zs, double Rs) {
    const double ex = px - xs, ey = py - ys, ez = pz - zs;
    const double qa = dx * dx + dy * dy + dz * dz;
    const double qb = 2.0 * (ex * dx + ey * dy + ez * dz);
    const double qc = (ex * ex + ey * ey + ez * ez) - Rs * Rs;
    const double dis = qb * qb - 4.0 * qa * qc;
    if (dis > 0.0) {
        double r1 = (-qb + sqrt(dis)) / (2.0 * qa);
        const double r2 = (-qb - sqrt(dis)) / (2.0 * qa);
        if (r2 > 0.0) r1 = r2;
        if (r1 > 0.0 && r1 < sexit) return r1;
    }
    return sexit;
}

// Per-warp state of the node being processed and its current batch of (up
// to) 32 rays.
struct RayBatch {
    double frame[FRAME_N];
    float4 dir[32];      // (d_x, d_y, d_z, v_node . d) per ray
    float2 wts[32];      // (w, w c_in / sqrt 2) per ray
    int K[32];           // segments per ray
    int st0[32];         // trace steps in the node's own cell
    float km[6];         // the node's second moment of line 1
};
// The batched kernel's: also the per-node ray sets of star mode.
struct RayBatchStar : RayBatch {
    double sk[7];        // star direction k(3), th_star, dth_star, dth_rest, th_i
    int sn[2];           // star rays, all rays of the node (-1: more than nth nph)
    unsigned smask;      // star rays of the batch
};
constexpr int RF_RAYS_BYTES = (sizeof(RayBatchStar) + 15) & ~15;   // at the start of the warp's shared memory

// ---- shape of a launch: line groups and the warp's shared-memory layout ----
// Lines are integrated in groups of nlg (the group's intensities of one pass
// over the channels live in registers).  A pass covers two slots of 32
// channels (the last one, when the slot count is odd, a single slot); the
// intensities of the passes not running wait in shared memory between two
// chunks of 32 cells.  Lines are handled in packs of two on the packed FP32x2
// pipe (the last line of an odd group packs its two channel slots instead).
struct RFShape {
    int L, nlg, groups, npk, nslot, rt, split;
    int rec_ld, om_ld;                    // row strides: float4 per cell, float per cell
    int o_rec, o_qd, o_om, o_I, o_part, o_v, o_acc, o_row, o_bb, bytes;   // byte offsets in the warp's block
};
// The remainder channel: 2 nvel + 1 channels with nvel a multiple of 16 are
// whole slots and one channel more, which the lanes-over-lines pass takes (no
// dust, at most 32 lines); any other count is padded to whole slots.
__host__ __device__ inline int rf_remainder(int nch, bool dust, int max_lines) {
    const int k = nch / 32;
    return (!dust && max_lines <= 32 && nch % 32 == 1 && (k == 1 || k == 2 || k == 4 || k == 8)) ? 1 : 0;
}

__host__ __device__ inline RFShape rf_shape(int L, int max_group, int nch, bool dust, int rt, bool split,
                                                    int rows = 1) {
    RFShape s;
    const TabShape t = tab_shape(L, max_group, dust);
    s.L = L;
    s.groups = t.width / ((dust ? 2 : 1) * t.npk);
    s.nlg = t.nlg;
    s.npk = t.npk;
    s.rt = rt;
    s.split = split;
    s.nslot = (nch - rt + 31) / 32;
    s.rec_ld = (dust ? 2 * s.npk : s.npk) | 1;
    s.om_ld = s.nlg | 1;
    const int nq = split ? 3 : 1;
    int o = RF_RAYS_BYTES;
    s.o_rec = o; o += 32 * s.rec_ld * 16;
    s.o_qd = o; o += 32 * 16;
    s.o_I = o; o += ((s.nslot / 2) * s.nlg + (s.nslot & 1) * s.npk) * 32 * 8;
    s.o_part = o; o += nq * s.npk * 32 * 8;
    s.o_row = o; o += rows * s.groups * (dust ? 2 : 1) * s.npk * 16;
    s.o_bb = o; o += 2 * s.groups * 2 * s.npk * 4;
    s.o_om = o; o += rt ? 32 * s.om_ld * 4 : 0;
    s.o_v = o; o += nq * 32 * L * 4;
    s.o_acc = o; o += (split ? 8 : 4) * L * 4;
    s.bytes = (o + 15) & ~15;
    return s;
}

// Index of record k of a ray in its warp's walk scratch: blocks of 32
// records, the 32 rays' blocks side by side, so that a warp's live part of
// the scratch is a few consecutive kilobytes (not 32 streams n_depth records
// apart) and a chunk of 32 cells is read from two such blocks at most.
__device__ __forceinline__ int walk_at(int k, int ray) { return ((k >> 5) << 10) + (ray << 5) + (k & 31); }

// f(std::integral_constant<int, k>) for the run-time count k of the group's
// trailing packs that take the Taylor form alone
template <int NPK, int K = 0, typename F>
__device__ __forceinline__ void with_thin_packs(int k, F &f) {
    if constexpr (K < NPK) {
        if (k == K) f(std::integral_constant<int, K>{});
        else with_thin_packs<NPK, K + 1>(k, f);
    } else {
        f(std::integral_constant<int, NPK>{});
    }
}

// I' = I + (1 - e^-tau)(S - I) for two updates on the packed pipe, x = tau
// log2 e >= 0 (lines with kv <= 0 and padding lines carry A = S = 0).  The
// Taylor value is overwritten by 1 - e where x reaches the switch: a compare
// and a predicated subtraction per element, one issue slot less than forming
// 1 - e for both and selecting (the same value: one_minus_exp2).
// thin is a compile-time constant once the pack loops are unrolled.
__device__ __forceinline__ void transfer2(bool thin, float2 &I, float2 A2, float2 S2, float2 g2) {
    const float2 x = __fmul2_rn(A2, g2);
    float2 om = om_taylor2(x);
    if (!thin) {
        const float e0 = ex2(-x.x), e1 = ex2(-x.y);
        asm("{\n .reg .pred p;\n setp.ge.f32 p, %1, %3;\n @p sub.rn.f32 %0, %4, %2;\n}"
            : "+f"(om.x) : "f"(x.x), "f"(e0), "f"(OM_TAYLOR_X), "f"(1.f));
        asm("{\n .reg .pred p;\n setp.ge.f32 p, %1, %3;\n @p sub.rn.f32 %0, %4, %2;\n}"
            : "+f"(om.y) : "f"(x.y), "f"(e1), "f"(OM_TAYLOR_X), "f"(1.f));
    }
    I = __ffma2_rn(om, __ffma2_rn(I, make_float2(-1.f, -1.f), S2), I);
}
__device__ __forceinline__ void transfer1(bool thin, float &I, float A, float S, float g) {
    const float x = A * g;
    const float om = thin ? om_taylor(x) : one_minus_exp(x, ex2(-x));
    I = fmaf(om, S - I, I);
}

// With dust: tau = (kv phi + alpha) dx n, S = (ev phi + j) / (kv phi + alpha),
// and ray_in's gate tau > 1e-30 (inverse_rt.f90:308).  fast: the quotient
// without the division's slow path (quot_rn; the numerator scaled by 2^60, so
// that nothing in it is subnormal), for chunks whose staged values are inside
// its range -- a slow-path branch per division kept the updates from
// overlapping.
struct DustPack {
    float2 A, E, Ad, Jd;
};
__device__ __forceinline__ void transfer2_dust(bool thin, bool fast, float2 &I, const DustPack &c, float2 g2) {
    const float2 tau = __ffma2_rn(c.A, g2, c.Ad), num = __ffma2_rn(c.E, g2, c.Jd);
    float2 S;
    if (fast) {
        const float2 n2 = __fmul2_rn(num, make_float2(0x1p60f, 0x1p60f)), m = __fmul2_rn(tau, make_float2(-1.f, -1.f));
        const float2 r0 = make_float2(rcp_approx(tau.x), rcp_approx(tau.y));
        const float2 r = __ffma2_rn(r0, __ffma2_rn(m, r0, make_float2(1.f, 1.f)), r0);
        const float2 q = __fmul2_rn(n2, r);
        S = __fmul2_rn(__ffma2_rn(r, __ffma2_rn(m, q, n2), q), make_float2(0x1p-60f, 0x1p-60f));
    } else {
        S = make_float2(num.x / tau.x, num.y / tau.y);
    }
    const float2 x = __fmul2_rn(tau, make_float2(LOG2E_F, LOG2E_F));
    float2 om = om_taylor2(x);
    if (!thin) {   // (x < 0 fails the gate below)
        const float e0 = ex2(-x.x), e1 = ex2(-x.y);
        asm("{\n .reg .pred p;\n setp.ge.f32 p, %1, %3;\n @p sub.rn.f32 %0, %4, %2;\n}"
            : "+f"(om.x) : "f"(x.x), "f"(e0), "f"(OM_TAYLOR_X), "f"(1.f));
        asm("{\n .reg .pred p;\n setp.ge.f32 p, %1, %3;\n @p sub.rn.f32 %0, %4, %2;\n}"
            : "+f"(om.y) : "f"(x.y), "f"(e1), "f"(OM_TAYLOR_X), "f"(1.f));
    }
    const float2 d = __ffma2_rn(I, make_float2(-1.f, -1.f), S);
    asm("{\n .reg .pred p;\n setp.gt.f32 p, %1, %4;\n @p fma.rn.f32 %0, %2, %3, %0;\n}"
        : "+f"(I.x) : "f"(tau.x), "f"(om.x), "f"(d.x), "f"(1e-30f));
    asm("{\n .reg .pred p;\n setp.gt.f32 p, %1, %4;\n @p fma.rn.f32 %0, %2, %3, %0;\n}"
        : "+f"(I.y) : "f"(tau.y), "f"(om.y), "f"(d.y), "f"(1e-30f));
}
// the staged values of a cell and line inside the range of the fast quotient
// (|tau| <= |A| + |Ad|, |numerator| <= |E| + |Jd|; a NaN fails)
__device__ __forceinline__ bool dust_in_range(float4 v) {
    return fabsf(v.x) + fabsf(v.z) < 0x1p90f && fabsf(v.y) + fabsf(v.w) < 0x1p-34f;
}

// Sums of N per-lane values over the warp, value l's sum on every lane whose
// low bits name it (sum_line).  Each butterfly step halves the values a lane
// carries while there are two or more left; every sum adds the same partners
// in the same order as N separate butterflies over 16, 8, 4, 2, 1 would.
template <int N>
__device__ __forceinline__ float sum_lines(const float (&v)[N], int o, int lane) {
    if constexpr (N == 1) {
        float x = v[0];
        for (; o >= 1; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        return x;
    } else {
        constexpr int H = (N + 1) / 2;
        float w[H];
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < H; i++) {
            const float b = (2 * i + 1 < N) ? v[2 * i + 1 < N ? 2 * i + 1 : 0] : 0.f;
            const float keep = up ? b : v[2 * i], send = up ? v[2 * i] : b;
            w[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
        return sum_lines<H>(w, o >> 1, lane);
    }
}
template <int N>
__device__ __forceinline__ int sum_line(int lane) {
    int l = 0, bit = 0;
    for (int n = N, o = 16; n > 1; n = (n + 1) / 2, o >>= 1, bit++)
        if (lane & o) l |= 1 << bit;
    return l;
}

// Everything of one warp in shared memory.
struct WarpMem {
    unsigned char *p;
    __device__ __forceinline__ float4 *rec(const RFShape &s) const { return (float4 *)(p + s.o_rec); }
    __device__ __forceinline__ float4 *qd(const RFShape &s) const { return (float4 *)(p + s.o_qd); }
    __device__ __forceinline__ float *om(const RFShape &s) const { return (float *)(p + s.o_om); }
    __device__ __forceinline__ float2 *I(const RFShape &s) const { return (float2 *)(p + s.o_I); }
    __device__ __forceinline__ float2 *part(const RFShape &s) const { return (float2 *)(p + s.o_part); }
    __device__ __forceinline__ float4 *row(const RFShape &s) const { return (float4 *)(p + s.o_row); }
    __device__ __forceinline__ float *bb(const RFShape &s) const { return (float *)(p + s.o_bb); }
    __device__ __forceinline__ float *v(const RFShape &s) const { return (float *)(p + s.o_v); }
    __device__ __forceinline__ float *acc(const RFShape &s) const { return (float *)(p + s.o_acc); }
};

// One pass over NSL channel slots (from slot s0) of a chunk of nc cells for
// the line group g: tk of the group's trailing packs take the Taylor form
// alone (with dust: all or none), fast: transfer2_dust's.  first: the intensities start from the background bb;
// last: the central cell and the weighted channel sums follow, else the
// intensities go back to shared memory.
template <int NLG, int NSL, bool DUST, bool SPLIT>
__device__ __forceinline__ void channel_pass(const RFShape &sh, const WarpMem &m, const float2 *chtab, int nch,
                                             int nvel, int lane, int g, int s0, int nc, int tk, bool fast, bool first,
                                             bool last, const float *bb, const float4 *row0, float fst0) {
    constexpr int NP = NLG / 2, ODD = NLG & 1, NPK = NP + ODD;
    const bool split = SPLIT && sh.split;
    float2 I[NSL][NP > 0 ? NP : 1], Io;   // Io: the odd line's slots
    float2 *sv = m.I(sh) + (size_t)(s0 / 2) * NLG * 32 + lane;
    if (first) {
#pragma unroll
        for (int k = 0; k < NP; k++)
#pragma unroll
            for (int s = 0; s < NSL; s++) I[s][k] = make_float2(bb[2 * k], bb[2 * k + 1]);
        if (ODD) Io = make_float2(bb[NLG - 1], bb[NLG - 1]);
    } else {
#pragma unroll
        for (int s = 0; s < NSL; s++)
#pragma unroll
            for (int k = 0; k < NP; k++) I[s][k] = sv[(s * NP + k) * 32];
        if (ODD) Io = sv[NSL * NP * 32];
    }
    const float4 *rec = m.rec(sh), *qd = m.qd(sh);
    const float2 ch2 = make_float2((float)(lane + 32 * s0 - nvel), (float)(lane + 32 * (s0 + 1) - nvel));
    auto run = [&](auto tag, auto fast_tag) {
        constexpr int TK = decltype(tag)::value;
        constexpr bool FAST = decltype(fast_tag)::value;
        // Gaussian profile of a cell at the lane's channels, exp(-q^2) = 2^(-q'^2)
        // with q' = q sqrt(log2 e) (staged scaled)
        auto profile = [&](int u, float (&gs)[2]) {
            const float4 q4 = qd[u];
            if (NSL == 2) {
                const float2 q = __ffma2_rn(make_float2(q4.z, q4.w), ch2, make_float2(q4.x, q4.y));
                const float2 t = __fmul2_rn(q, q);
                gs[0] = ex2(-t.x);
                gs[1] = ex2(-t.y);
            } else {
                const float q = fmaf(q4.z, ch2.x, q4.x);
                gs[0] = gs[1] = ex2(-(q * q));
            }
        };
        auto cell = [&](int u, const float (&gs)[2]) {
            const float4 *r = rec + u * sh.rec_ld;
#pragma unroll
            for (int k = 0; k < NP; k++) {
                if constexpr (DUST) {
                    const float4 v = r[2 * k], w = r[2 * k + 1];
                    const DustPack c{make_float2(v.x, v.y), make_float2(v.z, v.w), make_float2(w.x, w.y),
                                     make_float2(w.z, w.w)};
#pragma unroll
                    for (int s = 0; s < NSL; s++)
                        transfer2_dust(TK > 0, FAST, I[s][k], c, make_float2(gs[s], gs[s]));
                    continue;
                }
                const float4 v = r[k];
#pragma unroll
                for (int s = 0; s < NSL; s++)
                    transfer2(k >= NPK - TK, I[s][k], make_float2(v.x, v.y), make_float2(v.z, v.w),
                              make_float2(gs[s], gs[s]));
            }
            if (ODD && DUST) {
                const float4 v = r[2 * NP], w = r[2 * NP + 1];
                const DustPack c{make_float2(v.x, v.y), make_float2(v.z, v.w), make_float2(w.x, w.y),
                                 make_float2(w.z, w.w)};
                transfer2_dust(TK > 0, FAST, Io, c, make_float2(gs[0], gs[1]));
            } else if (ODD) {
                const float4 v = r[NP];
                if (NSL == 2)
                    transfer2(TK >= 1, Io, make_float2(v.x, v.y), make_float2(v.z, v.w), make_float2(gs[0], gs[1]));
                else
                    transfer1(TK >= 1, Io.x, v.x, v.z, gs[0]);
            }
        };
        // enough independent updates in flight per iteration: narrow groups
        // run several cells at once (their weights do not depend on each other)
        constexpr int U = DUST ? 1 : NSL * NLG >= 10 ? 1 : NSL * NLG >= 5 ? 2 : 4;
#pragma unroll U
        for (int u = 0; u < nc; u++) {
            float gs[2];
            profile(u, gs);
            cell(u, gs);
        }
    };
    if constexpr (DUST) {
        if (!fast) run(std::integral_constant<int, 0>{}, std::false_type{});
        else if (tk == NPK) run(std::integral_constant<int, 1>{}, std::true_type{});
        else run(std::integral_constant<int, 0>{}, std::true_type{});
    } else {
        auto plain = [&](auto tag) { run(tag, std::false_type{}); };
        // (a pass of one slot is a small part of its cell's work: two classes,
        // as every further body costs instruction fetch)
        if constexpr (NSL == 2) with_thin_packs<NPK>(tk, plain);
        else if (tk == NPK) plain(std::integral_constant<int, NPK>{});
        else plain(std::integral_constant<int, 0>{});
    }
    if (!last) {
#pragma unroll
        for (int s = 0; s < NSL; s++)
#pragma unroll
            for (int k = 0; k < NP; k++) sv[(s * NP + k) * 32] = I[s][k];
        if (ODD) sv[NSL * NP * 32] = Io;
        return;
    }
    // central cell (inverse_rt.f90:320-339): no gate, profile at the node's own
    // b, then the weighted channel sum, slot by slot
    float2 *part = m.part(sh) + lane;
    const float4 *row = row0 + g * (DUST ? 2 : 1) * NPK;
    const int np32 = sh.npk * 32;
    // the intensity after the cell; om and Ie: what L* and J_eff sum
    auto weigh = [&](float2 &I2, int k, float2 g0, float2 &om, float2 &Ie) {
        if constexpr (DUST) {
            const float4 v = row[2 * k], w = row[2 * k + 1];
            const float A[2] = {v.x, v.y}, Sl[2] = {v.z, v.w}, al[2] = {w.x, w.y}, Jd[2] = {w.z, w.w};
            const float gg[2] = {g0.x, g0.y}, Iv[2] = {I2.x, I2.y};
            float o[2], omv[2], Iev[2];
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const float kap = fmaf(A[q], gg[q], al[q]);
                const float tau = kap * fst0;
                const float Sv = fmaf(Sl[q] * A[q], gg[q], Jd[q]) / kap;
                const float x = tau * LOG2E_F;
                const float w1 = one_minus_exp(x, ex2(-x));
                o[q] = fmaf(w1, Sv - Iv[q], Iv[q]);
                omv[q] = Iev[q] = 0.f;
                if (split) {
                    const float lf = A[q] * gg[q] / kap;   // line share of the opacity
                    const float Sd = Jd[q] / kap;          // dust emission share of S
                    Iev[q] = fmaf(w1, Sd - Iv[q], Iv[q]);
                    omv[q] = lf * w1;
                }
            }
            om = make_float2(omv[0], omv[1]);
            Ie = make_float2(Iev[0], Iev[1]);
            return make_float2(o[0], o[1]);
        }
        const float4 v = row[k];
        const float2 x = __fmul2_rn(__fmul2_rn(__fmul2_rn(make_float2(v.x, v.y), g0), make_float2(fst0, fst0)),
                                    make_float2(LOG2E_F, LOG2E_F));
        om = one_minus_exp2(x, ex2(-x.x), ex2(-x.y));
        const float2 mI = __fmul2_rn(I2, make_float2(-1.f, -1.f));
        Ie = __ffma2_rn(om, mI, I2);
        return __ffma2_rn(om, __fadd2_rn(make_float2(v.z, v.w), mI), I2);
    };
#pragma unroll
    for (int s = 0; s < NSL; s++) {
        const int ch = lane + 32 * (s0 + s);
        const bool valid = ch < nch - sh.rt;
        const float2 ct = chtab[valid ? ch : 0];
        const float2 g0 = make_float2(ct.x, ct.x), w2 = make_float2(ct.y, ct.y);
#pragma unroll
        for (int k = 0; k < NP; k++) {
            float2 om, Ie;
            const float2 o = weigh(I[s][k], k, g0, om, Ie);
            if (valid) part[k * 32] = __ffma2_rn(w2, o, part[k * 32]);
            if (split && valid) {
                part[np32 + k * 32] = __ffma2_rn(w2, Ie, part[np32 + k * 32]);
                part[2 * np32 + k * 32] = __ffma2_rn(w2, om, part[2 * np32 + k * 32]);
            }
        }
    }
    if (ODD) {
        const int ch = lane + 32 * s0;
        const bool v0 = ch < nch - sh.rt, v1 = NSL == 2 && ch + 32 < nch - sh.rt;
        const float2 c0 = chtab[v0 ? ch : 0], c1 = chtab[v1 ? ch + 32 : 0];
        float2 om, Ie;
        const float2 o = weigh(Io, NP, make_float2(c0.x, c1.x), om, Ie);
        auto add = [&](float2 *q, float2 y) {
            if (v0) q->x = fmaf(c0.y, y.x, q->x);
            if (v1) q->x = fmaf(c1.y, y.y, q->x);
        };
        add(part + NP * 32, o);
        if (split) {
            add(part + np32 + NP * 32, Ie);
            add(part + 2 * np32 + NP * 32, om);
        }
    }
}

// The nodes of a batch of rays: one, or (FLAT) two, the second's from ray
// `split` on, with its line row behind the first's.
struct BatchNodes {
    float dqfac[2];
    int split;
};

// The channel integration of a warp's batch of nr walked rays: per ray and
// line the weighted channel sum at the node (v), with split also those of
// J_eff and L*.  One chunk of up to 32 cells at a time is staged in shared
// memory (lane = cell); then lanes run over channels, pass by pass.
template <int NLG, bool DUST, bool STAR, int SLOTS, bool SPLIT, bool FLAT>
__device__ __forceinline__ void integrate_batch(const RFArgs &a, const RFShape &shape, const WarpMem &m,
                                                const RayBatch &B, unsigned smask, const float2 *chtab,
                                                const int2 *walk, int nr, const BatchNodes &bn, int lane) {
    const unsigned FULL = 0xffffffffu;
    // (copies: the batched kernel has both in shared memory, where every store
    // to it would have them read again: six clouds in a batch 23.2 -> 22.6 ms)
    const RFShape sh = shape;
    const float4 *const cellv = a.cellv, *const ltab = a.ltab;
    const bool split = SPLIT && sh.split;
    constexpr int NP = NLG / 2, ODD = NLG & 1, NPK = NP + ODD;
    const int L = a.L, nch = a.nch, nvel = a.nvel;
    float4 *rec = m.rec(sh) + lane * sh.rec_ld;
    const int width = sh.groups * (DUST ? 2 : 1) * NPK;   // the line table's
    // walk records of a chunk (lane = cell), the next chunk's -- of this ray,
    // the next line group or the next ray -- loaded while one is integrated
    int2 wcp = make_int2(0, 0);
    {
        const int h = B.K[0] - 1;
        if (lane < min(32, h)) wcp = walk[walk_at(h - lane, 0)];
    }
    for (int rr = 0; rr < nr; rr++) {
        const int Kr = B.K[rr];
        const float4 d4 = B.dir[rr];
        const bool second = FLAT && rr >= bn.split;
        const float dqfac = second ? bn.dqfac[1] : bn.dqfac[0];
        const float4 *row0 = m.row(sh) + (second ? sh.groups * (DUST ? 2 : 1) * NPK : 0);
        const float fst0 = (float)B.st0[rr];
        const float *bb0 = m.bb(sh) + ((STAR && ((smask >> rr) & 1u)) ? sh.groups * 2 * NPK : 0);
        for (int g = 0; g < sh.groups; g++) {
            const int l0 = g * NLG;
            const float *bb = bb0 + g * 2 * NPK;
            // the remainder channel of this lane's line (lane = line of the group)
            float Irem = (sh.rt && lane < NLG) ? bb[lane] : 0.f;
            {
                float2 *part = m.part(sh) + lane;
                for (int k = 0; k < (split ? 3 : 1) * NPK; k++) part[k * 32] = make_float2(0.f, 0.f);
            }
            for (int hi = Kr - 1, first = 1;; hi -= 32, first = 0) {
                const int nc = max(0, min(32, hi));
                const bool last = hi <= 32;
                const int2 wc = wcp;
                {
                    int nh, nrr = rr;
                    if (!last) nh = hi - 32;
                    else if (g + 1 < sh.groups) nh = Kr - 1;
                    else if (rr + 1 < nr) { nrr = rr + 1; nh = B.K[rr + 1] - 1; }
                    else nh = 0;
                    if (lane < min(32, nh)) wcp = walk[walk_at(nh - lane, nrr)];
                }
                __syncwarp();
                unsigned thin = (1u << NPK) - 1u;   // the packs thin in this cell
                bool in_range = true;               // dust: the fast quotient serves this cell
                if (lane < nc) {
                    const float4 cv = cellv[wc.x];
                    const float4 *lt = ltab + (size_t)wc.x * width + g * (DUST ? 2 : 1) * NPK;
                    const float fst = (float)wc.y;
                    const float vp = fmaf(cv.z, d4.z, fmaf(cv.y, d4.y, __fmul_rn(cv.x, d4.x)));
                    const float ib = SQL2E_F * (1.f / cv.w);
                    const float2 qdl = make_float2((d4.w - vp) * ib, dqfac * ib);
                    m.qd(sh)[lane] = make_float4(qdl.x, qdl.x, qdl.y, qdl.y);
                    if constexpr (DUST) {
                        float4 p[2 * NPK], v[2 * NPK];
#pragma unroll
                        for (int k = 0; k < 2 * NPK; k++) p[k] = lt[k];
#pragma unroll
                        for (int l = 0; l < NLG; l++) {
                            const float4 q = p[l & ~1], r = p[l | 1];
                            const float4 t = (l & 1) ? make_float4(q.y, q.w, r.y, r.w) : make_float4(q.x, q.z, r.x, r.z);
                            v[l] = make_float4(t.x * fst, t.y * t.x * fst, t.z * fst, t.w * fst);
                            in_range = in_range && dust_in_range(v[l]);
                            // |tau| <= |A| + |Ad|: the Taylor form in every channel
                            if (!((fabsf(v[l].x) + fabsf(v[l].z)) * LOG2E_F < OM_THIN_A)) thin &= ~(1u << (l / 2));
                        }
                        if (ODD) v[NLG] = v[NLG - 1];
#pragma unroll
                        for (int k = 0; k < NPK; k++) {
                            const float4 t = v[2 * k], w = v[2 * k + 1];
                            rec[2 * k] = make_float4(t.x, w.x, t.y, w.y);
                            rec[2 * k + 1] = make_float4(t.z, w.z, t.w, w.w);
                        }
                    } else {
                        // optical depth at unit profile in log2 units (ex2 takes
                        // it as is) and the source function.  A cell line with kv
                        // <= 0 fails ray_in's gate tau > 1e-30 in every channel
                        // (inverse_rt.f90:308): A = S = 0 leaves I unchanged exactly;
                        // 0 < tau < 2^-54 rounds to a zero weight as in FP64, so
                        // the gate needs no test.  (The padding lines of a last group
                        // repeat its last line; nothing reads their sums.)
                        float4 v[NPK];   // (A, A', S, S')
#pragma unroll
                        for (int k = 0; k < NPK; k++) v[k] = lt[k];
#pragma unroll
                        for (int k = 0; k < NPK; k++) {
                            const bool on0 = v[k].x > 0.f, on1 = v[k].y > 0.f;
                            v[k].x = on0 ? v[k].x * fst * LOG2E_F : 0.f;
                            v[k].y = on1 ? v[k].y * fst * LOG2E_F : 0.f;
                            v[k].z = on0 ? v[k].z : 0.f;
                            v[k].w = on1 ? v[k].w : 0.f;
                            if (!(v[k].x < OM_THIN_A) || !(v[k].y < OM_THIN_A)) thin &= ~(1u << k);
                            rec[k] = v[k];
                        }
                        if (sh.rt) {
                            // the remainder channel's transfer weight of this
                            // cell for the group's lines
                            const float q = fmaf(qdl.y, (float)(nch - 1 - nvel), qdl.x);
                            const float gr = ex2(-(q * q));
                            float *om = m.om(sh) + lane * sh.om_ld;
#pragma unroll
                            for (int k = 0; k < NP; k++) {
                                const float2 x = __fmul2_rn(make_float2(v[k].x, v[k].y), make_float2(gr, gr));
                                const float2 w = one_minus_exp2(x, ex2(-x.x), ex2(-x.y));
                                om[2 * k] = w.x;
                                om[2 * k + 1] = w.y;
                            }
                            if (ODD) {
                                const float x = v[NP].x * gr;
                                om[NLG - 1] = one_minus_exp(x, ex2(-x));
                            }
                        }
                    }
                }
                // Packs whose lines' line-centre optical depth is below OM_THIN_A
                // in every cell of the chunk take the Taylor form of 1 - e^-tau
                // alone in every channel: the full update would pick exactly that
                // value.  Decided per chunk, uniform over the warp, for the
                // group's trailing packs (a rotor's higher lines are the thinner).
                const int tk = __clz(~(__reduce_and_sync(FULL, thin) << (32 - NPK)));
                const bool fast = DUST && __all_sync(FULL, in_range);
                __syncwarp();
                if (!DUST && sh.rt && lane < NLG) {
                    const float *om = m.om(sh) + lane;
                    const float *S = reinterpret_cast<const float *>(m.rec(sh) + (lane >> 1)) + 2 + (lane & 1);
#pragma unroll 4
                    for (int u = 0; u < nc; u++) Irem = fmaf(om[u * sh.om_ld], S[u * sh.rec_ld * 4] - Irem, Irem);
                }
                int s0 = 0;
                if constexpr (SLOTS != 1)
                    for (; s0 + 1 < sh.nslot; s0 += 2)
                        channel_pass<NLG, 2, DUST, SPLIT>(sh, m, chtab, nch, nvel, lane, g, s0, nc, tk, fast, first,
                                                          last, bb, row0, fst0);
                if constexpr (SLOTS != 2)
                    if (s0 < sh.nslot)
                        channel_pass<NLG, 1, DUST, SPLIT>(sh, m, chtab, nch, nvel, lane, g, s0, nc, tk, fast, first,
                                                          last, bb, row0, fst0);
                if (last) break;
            }
            // the channel sums over the lanes, the remainder channel's share
            // added last
            const int line = l0 + sum_line<NLG>(lane);
            for (int q = 0; q < (split ? 3 : 1); q++) {
                const float2 *part = m.part(sh) + q * NPK * 32 + lane;
                float v[NLG];
#pragma unroll
                    for (int k = 0; k < NP; k++) {
                        const float2 p = part[k * 32];
                        v[2 * k] = p.x;
                        v[2 * k + 1] = p.y;
                    }
                if (ODD) v[NLG - 1] = part[NP * 32].x;
                const float t = sum_lines<NLG>(v, 16, lane);
                float *dst = m.v(sh) + (q * 32 + rr) * L;
                if (line < min(l0 + NLG, L)) dst[line] = t;
                if (!DUST && sh.rt) {
                    __syncwarp();
                    if (lane < NLG && l0 + lane < L) {
                        const float *row = reinterpret_cast<const float *>(row0 + g * NPK + (lane >> 1)) + (lane & 1);
                        const float2 ct = chtab[nch - 1];
                        const float x = row[0] * ct.x * fst0 * LOG2E_F;
                        const float om = one_minus_exp(x, ex2(-x));
                        const float r = (q == 0) ? fmaf(om, row[2] - Irem, Irem) : (q == 1) ? fmaf(om, -Irem, Irem) : om;
                        dst[l0 + lane] = __fadd_rn(dst[l0 + lane], __fmul_rn(ct.y, r));
                    }
                }
            }
        }
    }
    __syncwarp();
}

// integrate_batch for a run-time group width (the batched kernel: models of
// any line count in one launch)
template <int NLG, bool DUST, int SLOTS, bool SPLIT>
__device__ __noinline__ void integrate_any_width(const RFArgs &a, const RFShape &sh, const WarpMem &m, const RayBatch &B,
                                        unsigned smask, const float2 *chtab, const int2 *walk, int nr,
                                        const BatchNodes &bn, int lane) {
    integrate_batch<NLG, DUST, true, SLOTS, SPLIT, false>(a, sh, m, B, smask, chtab, walk, nr, bn, lane);
}

// FP32 sums over rays, in ray order.
struct NodeSum {
    KahanF j0, j2, je, ls;
    __device__ __forceinline__ void add(float2 w, float v) {
        j0.add(__fmul_rn(w.x, v));
        j2.add(__fmul_rn(w.y, v));
    }
    __device__ __forceinline__ void add_split(float w, float ve, float vl) {
        je.add(__fmul_rn(w, ve));
        ls.add(__fmul_rn(w, vl));
    }
};
// second moment of line 1's field, sum w I n n (xx yy zz xy xz yz), whose
// traceless part is J^2_Q in any frame: one ray's term of component k
__device__ __forceinline__ float moment_add(float km, int k, float w, float v, float4 d) {
    const float wv = __fmul_rn(w, v);
    const float p = (k == 0 || k == 3 || k == 4) ? d.x : (k == 2) ? d.z : d.y;
    const float q = (k == 0) ? d.x : (k == 1 || k == 3) ? d.y : d.z;
    return fmaf(wv * p, q, km);
}

// NLG: lines per group (0: the model's own, BATCH only).
// SLOTS: 1 for layouts of one slot, 2 for an even number, 0 for any; SPLIT:
// with the split field (when the launch asks for it).  What a layout cannot
// need is left out: the size of the cell loops' code decides how well they
// fetch (65,536 points x 129 channels without the one-slot pass and the split
// sums: 318 -> 310 ms; 2,500 points x 33 channels without the two-slot pass:
// 0.498 -> 0.455).
// BATCH: the work items are (model, node) pairs of many models (RFBatch);
// each warp copies the argument block of its current model into shared
// memory.  Otherwise the nodes of the one model a0.
// FLAT: small clouds have too few nodes to fill the GPU with a warp per node.
// The items are 32, 16 or 8 consecutive rays of all nodes' rays in a row (of
// two nodes at most) and store the rays' per-line channel sums, which
// k_rf_finish adds up in ray order afterwards (the same sums in the same
// order).  Cut across the nodes the walk's lanes are full: as ranges of one
// node's rays, 2,500 points of 44 directions had to be cut into eights to
// balance, which walk with 8 lanes of 32 (0.512 -> 0.480 ms a pass).
// What bounds it there (4,096 points, 4 lines, 65 channels): the load/store
// unit, 70 % of its cycles (the walk's scattered 16-byte loads and the staged
// cells), and issue, 71 %; the FMA pipe 51 %.
template <int NLG, bool DUST, bool BATCH, int SLOTS, bool SPLIT, bool FLAT = false>
__global__ void __launch_bounds__(256, (NLG >= 1 && NLG <= 4) ? 3 : 2) k_radiation_field(RFArgs a0, RFBatch bw, RFShape sh0) {
    static_assert(!(BATCH && FLAT), "batched items are whole nodes");
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const long long gw = (long long)blockIdx.x * (blockDim.x >> 5) + wib;
    const int n_depth = BATCH ? bw.n_depth : a0.n_depth;
    int2 *const walk = (BATCH ? bw.walk : a0.walk) + (size_t)gw * 1024 * (size_t)((n_depth + 31) / 32);
    using RB = typename std::conditional<BATCH, RayBatchStar, RayBatch>::type;
    __shared__ RFArgs margs[BATCH ? RF_BATCH_WARPS : 1];
    __shared__ RFShape mshape[BATCH ? RF_BATCH_WARPS : 1];
    extern __shared__ __align__(16) unsigned char dyn[];
    // per channel: the central cell's profile exp(-q0^2) and the channel weight
    const int nch = BATCH ? bw.nch : a0.nch;
    float2 *chtab = reinterpret_cast<float2 *>(dyn);
    const float *chq = BATCH ? bw.chq : a0.chq, *chw = BATCH ? bw.chw : a0.chw;
    for (int i = threadIdx.x; i < nch; i += blockDim.x) {
        const float q0c = chq[i];
        chtab[i] = make_float2(ex2(-q0c * q0c * LOG2E_F), chw[i]);
    }
    WarpMem m;
    m.p = dyn + ((nch * sizeof(float2) + 15) & ~(size_t)15) + (size_t)wib * (BATCH ? bw.warp_bytes : sh0.bytes);
    RB &B = *reinterpret_cast<RB *>(m.p);
    auto fill_bb = [&](const RFArgs &a, const RFShape &sh) {
        float *bb = m.bb(sh);
        const int per = 2 * sh.npk, n = sh.groups * per;
        for (int i = lane; i < n; i += 32) {
            const int l = (i / per) * sh.nlg + i % per;
            const bool on = i % per < sh.nlg && l < sh.L;
            bb[i] = on ? a.bb[l] : 0.f;
            bb[n + i] = (BATCH && on) ? a.bbs[l] : 0.f;
        }
    };
    if (!BATCH) fill_bb(a0, sh0);
    __syncthreads();

    unsigned long long nseg = 0;
    int cur_model = -1;
    for (;;) {
        int node = 0;
        long long ray0 = 0;   // FLAT: the item's first ray,
        int item_rays = 0;    // and rays
        if (BATCH) {
            long long item = 0;
            if (lane == 0) item = (long long)atomicAdd(&bw.queue[0], 1ULL);
            item = __shfl_sync(FULL, item, 0);
            if (item >= bw.n_items) break;
            const int2 wi = bw.items[item];
            if (wi.x != cur_model) {
                __syncwarp();
                const int *src = reinterpret_cast<const int *>(bw.models + wi.x);
                int *dst = reinterpret_cast<int *>(&margs[wib]);
                for (int k = lane; k < (int)(sizeof(RFArgs) / sizeof(int)); k += 32) dst[k] = src[k];
                __syncwarp();
                if (lane == 0) mshape[wib] = rf_shape(margs[wib].L, bw.max_group, nch, DUST, bw.rt, bw.split);
                __syncwarp();
                fill_bb(margs[wib], mshape[wib]);
                cur_model = wi.x;
            }
            node = wi.y;
        } else {
            long long item = 0;
            if (lane == 0) item = (long long)atomicAdd(&a0.counters[0], 1ULL);
            item = __shfl_sync(FULL, item, 0);
            if constexpr (FLAT) {
                const long long i16 = item - a0.items32, i8 = i16 - a0.items16, all = (long long)a0.bulk * a0.ndir;
                item_rays = i16 < 0 ? 32 : i8 < 0 ? 16 : 8;
                ray0 = i16 < 0 ? 32 * item : 32LL * a0.items32 + (i8 < 0 ? 16 * i16 : 16LL * a0.items16 + 8 * i8);
                if (ray0 >= all) break;
                item_rays = (int)min((long long)item_rays, all - ray0);
                node = (int)(ray0 / a0.ndir);
            } else {
                if (item >= a0.bulk) break;
                node = (int)item;
            }
        }
        const RFArgs &a = BATCH ? margs[wib] : a0;
        const RFShape &sh = BATCH ? mshape[wib] : sh0;
        int st = 0;
        int node_seg = 0;   // the item's ray segments (sum of node_count over its rays)
        BatchNodes bn;
        bn.split = FLAT ? (int)min(32LL, (long long)(node + 1) * a.ndir - ray0) : 32;
        if (FLAT || a.ab[node] > 0.0) {
            if (!FLAT) {
                if (lane < FRAME_N) B.frame[lane] = a.frames[FRAME_N * (size_t)node + lane];
                if (lane < 6) B.km[lane] = 0.f;
                __syncwarp();
            }
            if constexpr (BATCH) {
                if (lane == 0) {
                    if (a.star) {
                        star_node(B.sk, B.sn, a.xs, a.ys, a.zs, a.Rs, a.nth, a.nph, B.frame[9], B.frame[10],
                                  B.frame[11]);
                    } else {
                        B.sn[0] = 0;
                        B.sn[1] = a.ndir;
                    }
                }
            }
            // the node's own line row
            for (int second = 0; second < (FLAT && bn.split < item_rays ? 2 : 1); second++) {
                const int width = sh.groups * (DUST ? 2 : 1) * sh.npk;
                const float4 *lt = a.ltab + (size_t)(node + second) * width;
                for (int i = lane; i < width; i += 32) m.row(sh)[second * width + i] = lt[i];
            }
            if (!FLAT)
                for (int i = lane; i < ((SPLIT && sh.split) ? 8 : 4) * sh.L; i += 32) m.acc(sh)[i] = 0.f;
            __syncwarp();
            int n_rays = a.ndir;
            if constexpr (BATCH) {
                n_rays = B.sn[1];
                if (n_rays < 0) st |= PORTAL_NODE_STAR;
            }
            // the ray's node (FLAT: of this lane's ray)
            const int node_l = FLAT ? min(node + (lane >= bn.split), a.bulk - 1) : node;
            const float4 cvn = a.cellv[node_l];
            if constexpr (FLAT) {
                const float q = 2.f * cvn.w / (float)a.nvel;
                bn.dqfac[0] = __shfl_sync(FULL, q, 0);
                bn.dqfac[1] = __shfl_sync(FULL, q, 31);
                n_rays = item_rays;
            } else {
                bn.dqfac[0] = bn.dqfac[1] = 2.f * cvn.w / (float)a.nvel;
            }
            for (int k0 = 0; st == 0 && k0 < n_rays; k0 += 32) {
                const int nr = min(32, n_rays - k0);
                // ---- (1)+(2) set-up and walk, one lane per ray ----
                int K = 0;
                bool over = false;
                bool sray = false;
                unsigned smask = 0u;
                if constexpr (BATCH) {
                    sray = a.star && lane < nr && k0 + lane < B.sn[0];
                    smask = __ballot_sync(FULL, sray);
                }
                if (FLAT && lane < nr) {
                    B.dir[lane] = make_float4(0.f, 0.f, 0.f, 0.f);
                    B.st0[lane] = B.K[lane] = 0;
                }
                if (lane < nr && (!FLAT || a.ab[node_l] > 0.0)) {
                    const double *f = FLAT ? a.frames + FRAME_N * (size_t)node_l : B.frame;
                    double mu, sth, cph, sph;
                    bool tab = true;
                    if constexpr (BATCH) {
                        if (a.star) {
                            const RayDir r = star_ray(B.sk, B.sn[0], k0 + lane, a.nth, a.nph, a.gx, a.gy, a.gz, f,
                                                      &B.wts[lane]);
                            mu = r.ct; sth = r.st; cph = r.cp; sph = r.sp;
                            tab = false;
                        }
                    }
                    if (tab) {
                        const double *dr =
                            a.dirs + 6 * (FLAT ? (size_t)(ray0 + lane - (long long)node_l * a.ndir) : (size_t)(k0 + lane));
                        mu = dr[0]; sth = dr[1]; cph = dr[2]; sph = dr[3];
                        B.wts[lane] = make_float2((float)dr[4], (float)dr[5]);
                    }
                    const double dx = mu * f[0] + sth * (cph * f[6] + sph * f[3]);
                    const double dy = mu * f[1] + sth * (cph * f[7] + sph * f[4]);
                    const double dz = mu * f[2] + sth * (cph * f[8] + sph * f[5]);
                    double sexit = sphere_exit_unit(f[9], f[10], f[11], f[12], dx, dy, dz);
                    if constexpr (BATCH) {
                        if (sray) sexit = star_exit(sexit, f[9], f[10], f[11], dx, dy, dz, a.xs, a.ys, a.zs, a.Rs);
                    }
                    const float fdx = (float)dx, fdy = (float)dy, fdz = (float)dz;
                    B.dir[lane] = make_float4(fdx, fdy, fdz, cvn.x * fdx + cvn.y * fdy + cvn.z * fdz);
                    // distance left to the sphere exit as an unevaluated float pair
                    // (rh + rl), decremented exactly by each step
                    float rh = (float)sexit, rl = (float)(sexit - (double)rh);
                    float rx = 0.f, ry = 0.f, rz = 0.f;
                    const bool step_ok = a.dx32 > 1e-20f && a.dx32 < 1e20f;   // quot_rn's range
                    int wg = a.wstart[node_l];
                    for (;;) {
                        // the cell's block of the walk tables: its header, the first 12
                        // edges and where their neighbours' blocks start, all in
                        // flight at once (scattered L2 reads: the walk is their
                        // latency, one round trip per step this way, five or six
                        // when offsets, edges and ids were read one after the other)
                        const int2 hd = a.whead[wg];   // (degree, node)
                        const float4 *we = a.wedge + 4 * (size_t)wg;
                        const int4 *wn = reinterpret_cast<const int4 *>(a.wnext) + wg;
                        float4 e[12];
                        int4 t[3];
#pragma unroll
                        for (int i = 0; i < 12; i++) e[i] = we[i];
#pragma unroll
                        for (int i = 0; i < 3; i++) t[i] = wn[i];
                        const float tsph = rh + rl;
                        // check_neigh_fast's scan: best starts at the sphere exit, a
                        // neighbour replaces it when FACE_EPS < t <= best (so among equal
                        // t the later neighbour wins).  t = num/den compared by cross
                        // multiplication (den > 0).
                        float bnum = tsph, bden = 1.f;
                        int bj = -1, bw = 0;
                        auto face = [&](int j, float4 e, int next) {
                            const float den = e.x * fdx + e.y * fdy + e.z * fdz;
                            const float num = e.w - (e.x * rx + e.y * ry + e.z * rz);
                            if (j < hd.x && den > 0.f && num > FACE_EPS * den && num * bden <= bnum * den) {
                                bnum = num;
                                bden = den;
                                bj = j;
                                bw = next;
                            }
                        };
#pragma unroll
                        for (int i = 0; i < 12; i++) {
                            const int4 q = t[i / 4];
                            face(i, e[i], (i & 3) == 0 ? q.x : (i & 3) == 1 ? q.y : (i & 3) == 2 ? q.z : q.w);
                        }
                        for (int j = 12; j < hd.x; j += 4) {
                            float4 e4[4];
#pragma unroll
                            for (int i = 0; i < 4; i++) e4[i] = we[j + i];
                            const int4 q = wn[j >> 2];
                            face(j, e4[0], q.x);
                            face(j + 1, e4[1], q.y);
                            face(j + 2, e4[2], q.z);
                            face(j + 3, e4[3], q.w);
                        }
                        // (0 < bnum <= 2 bden, both lengths of the cloud's geometry)
                        const float delta = (bj < 0) ? tsph : quot_rn(bnum, bden);
                        if (K >= n_depth) { over = true; break; }
                        const int steps = (int)roundf(step_ok ? quot_rn(delta, a.dx32) : delta / a.dx32);   // nint(delta_x/dx)
                        walk[walk_at(K, lane)] = make_int2(hd.y, steps);
                        if (K == 0) B.st0[lane] = steps;
                        K++;
                        if (bj < 0) break;
                        const float4 eb = we[bj];
                        {   // (rh, rl) -= delta: two-sum, then renormalise
                            const float t = rh - delta;
                            const float bv = t - rh;
                            const float err = (rh - (t - bv)) - (delta + bv);
                            const float lo = rl + err;
                            rh = t + lo;
                            rl = lo - (rh - t);
                        }
                        rx = fmaf(delta, fdx, rx) - eb.x;
                        ry = fmaf(delta, fdy, ry) - eb.y;
                        rz = fmaf(delta, fdz, rz) - eb.z;
                        wg = bw;
                    }
                    B.K[lane] = K;
                }
                if constexpr (FLAT) {   // (a walk past n_depth: its node's field is not used)
                    if (over) B.K[lane] = 0;
                    if (lane < nr) a.iseg[ray0 + lane] = over ? -1 : K;
                } else {
                    if (__any_sync(FULL, over)) { st |= PORTAL_NODE_DEPTH; break; }
                    node_seg += __reduce_add_sync(FULL, lane < nr ? K : 0);
                }
                __syncwarp();

                // ---- (3)+(4) channel integration of the batch's rays ----
                if constexpr (NLG > 0) {
                    integrate_batch<NLG, DUST, BATCH, SLOTS, SPLIT, FLAT>(a, sh, m, B, smask, chtab, walk, nr, bn, lane);
                } else {
                    switch (sh.nlg) {
#define RF_WIDTH(n)                                                                                        \
    case n: integrate_any_width<n, DUST, SLOTS, SPLIT>(a, sh, m, B, smask, chtab, walk, nr, bn, lane); break;
                        RF_WIDTH(1) RF_WIDTH(2) RF_WIDTH(3) RF_WIDTH(4)
                    default:
                        if constexpr (DUST) {
                            integrate_any_width<5, DUST, SLOTS, SPLIT>(a, sh, m, B, smask, chtab, walk, nr, bn, lane);
                        } else {
                            switch (sh.nlg) {
                                RF_WIDTH(5) RF_WIDTH(6) RF_WIDTH(7) RF_WIDTH(8) RF_WIDTH(9)
                            default: integrate_any_width<10, DUST, SLOTS, SPLIT>(a, sh, m, B, smask, chtab, walk, nr, bn, lane);
                            }
                        }
                    }
#undef RF_WIDTH
                }
                const float *v = m.v(sh);
                const int L = sh.L;
                if constexpr (FLAT) {   // the rays' channel sums and directions for k_rf_finish
                    const size_t plane = (size_t)a.bulk * a.ndir * L;
                    for (int q = 0; q < ((SPLIT && sh.split) ? 3 : 1); q++)
                        for (int i = lane; i < nr * L; i += 32) a.vray[q * plane + ray0 * L + i] = v[q * 32 * L + i];
                    if (lane < nr) a.dray[ray0 + lane] = B.dir[lane];
                } else {
                    for (int l = lane; l < L; l += 32) {
                        float *acc = m.acc(sh) + l;
                        NodeSum s;
                        s.j0.s = acc[0]; s.j0.c = acc[L]; s.j2.s = acc[2 * L]; s.j2.c = acc[3 * L];
                        for (int r = 0; r < nr; r++) s.add(B.wts[r], v[r * L + l]);
                        acc[0] = s.j0.s; acc[L] = s.j0.c; acc[2 * L] = s.j2.s; acc[3 * L] = s.j2.c;
                        if ((SPLIT && sh.split)) {
                            s.je.s = acc[4 * L]; s.je.c = acc[5 * L]; s.ls.s = acc[6 * L]; s.ls.c = acc[7 * L];
                            for (int r = 0; r < nr; r++)
                                s.add_split(B.wts[r].x, v[(32 + r) * L + l], v[(64 + r) * L + l]);
                            acc[4 * L] = s.je.s; acc[5 * L] = s.je.c; acc[6 * L] = s.ls.s; acc[7 * L] = s.ls.c;
                        }
                    }
                    if (lane < 6) {
                        float km = B.km[lane];
                        for (int r = 0; r < nr; r++) km = moment_add(km, lane, B.wts[r].x, v[r * L], B.dir[r]);
                        B.km[lane] = km;
                    }
                }
                __syncwarp();
            }
        }
        if constexpr (!FLAT) {
            const int L = a.L;
            const bool on = st == 0 && a.ab[node] > 0.0;
            const float *acc = m.acc(sh);
            auto value = [&](int q, int l) { return on ? (double)acc[2 * q * L + l] - (double)acc[(2 * q + 1) * L + l] : 0.0; };
            for (int l = lane; l < L; l += 32) {
                a.J0[(size_t)node * L + l] = value(0, l);
                a.J2[(size_t)node * L + l] = value(1, l);
                if ((SPLIT && sh.split)) {
                    a.JE[(size_t)node * L + l] = value(2, l);
                    a.LS[(size_t)node * L + l] = value(3, l);
                }
            }
            if (lane == 0) {
                a.status[node] = st;
                if (st) atomicAdd(&a.counters[RF_FAILED], 1ULL);
                if (a.segs) a.segs[node] = node_seg;
                if (a.kmom)
                    for (int k = 0; k < 6; k++) a.kmom[(size_t)k * a.N + node] = on ? B.km[k] : 0.f;
            }
        }
        nseg += (unsigned long long)node_seg;
        __syncwarp();
    }
    // segment count (every lane holds the same count; k_rf_finish counts rays' items)
    if (lane == 0 && !FLAT) atomicAdd(BATCH ? &bw.queue[1] : &a0.counters[1], nseg);
}


}  // namespace
