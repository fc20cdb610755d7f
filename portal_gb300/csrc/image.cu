// Stokes image of one inclination: the pixel mode of finish_portal.x.
//
// Reference: para_finish.f90:170-185 (line data), :222-240 (population
// read-back), :354-448 (pixel grid and the three OpenMP loops);
// rotate_all_save miscellaneous.f90:844-907; comp_emcoefs em_coefs.f90:1-113;
// trace_out_raytrace raytrace.f90:58-177 with check_neigh
// miscellaneous.f90:1-46; ray_in_raytrace raytrace.f90:179-323 with
// polarize_prop :1-56 and rot_stokes / rot_stokes_back
// miscellaneous.f90:463-551.
//
// Kernels:
//   k_im_nodes   per node: the inclination rotation (FP64) and the
//                population read-back, then per (node, line) the emission /
//                absorption coefficients, stored as per-trace-step factors at
//                the profile peak (float4), plus per-node Stokes-rotation
//                constants.
//   k_im_dust    per (node, line): the dust's Planck function.
//   k_im_march   one lane per pixel: the start node (argmin of the FP64
//                distance, lowest index on ties) and the fixed-step march
//                along +z.  The step at which a neighbour becomes nearer is
//                predicted from the bisector-plane crossings: FP32 with
//                rounding bounds picks the few neighbours that can cross
//                next, FP64 places their crossings.  The photon's z is
//                advanced to just before it by the reference's own sequence of
//                FP64 additions (computed in exact jumps, add_steps), and
//                check_neigh is replayed exactly (FP64, strict <, list order)
//                from there and at the exit -- over the neighbours that can
//                come within 1e-12 of the current node's squared distance,
//                the others being unable to win -- so the recorded (node,
//                step) list is the reference's.  Bound by the FP64 pipe (16
//                cycles a warp instruction; 70 % busy): 1.26 ms for 257 x 257
//                pixels of a 32,768-point sphere.
//   k_im_stokes, k_im_stokes_tail   per (pixel, line), lanes over velocity
//                channels (whole slots of 32, cell records staged in shared
//                memory 32 at a time) or, for the few channels left over,
//                lanes over pixels: the polarized propagation in the
//                numerically stable form o11 = (phi(p)+phi(m))/2, o12 =
//                -(phi(p)-phi(m))/2, e ch = (E_p+E_m)/2, e sh = (E_p-E_m)/2
//                with p, m = tau_I -/+ tau_Q, E = exp(-.), phi(x) =
//                (1-e^-x)/x, algebraically identical to raytrace.f90:41-53;
//                the optical depth summed with compensation.  Bound by
//                instruction issue (FMA pipe 62 %): 1.32 ms for the 128 whole
//                channels of that cube, 0.04 ms for the last one.
//   k_im_dust, k_im_dust_maps   the dust's Planck function per (node, line)
//                and the channel-independent dust terms per (pixel, line),
//                FP64.
// March and integration in one kernel, 32 pixels to a warp or block, took
// 10.2 ms and (marching warp beside three waiting ones) 4.06 ms on that cube;
// apart 2.62 ms.
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"

namespace portal {
double wigner6j(int tj1, int tj2, int tj3, int tj4, int tj5, int tj6);
}
using namespace portal;

namespace {

struct ImLine {
    double nu0, A, kd, w1, w2, fas, bb_cmb, bb_star;
    int lo, up, j1, j2;  // 0-based levels
};
constexpr int IM_MAX_LINES = 16;

struct ImNodeArgs {
    int N, bulk, nlev, nlines;
    double R[9];              // R_tot column-major
    double tdx;               // tx * dx
    const double *xyz, *vel, *bvec, *b, *tdust, *levp, *pops_in;
    const int *j_lev;
    const ImLine *lines;      // (nlines) the context's own: contexts may run on several threads
    double *xyz_r;            // (3,N) rotated positions
    double *nrm2;             // (N) |X|^2 of the rotated positions (the march's predictions)
    float4 *cellv;            // (vz, 1/b, cos 2alpha, sin 2alpha)
    float4 *cellb;            // (mu2, cos 2phi, sin 2phi, dust rho)
    float4 *coef;             // (nlines, N): eta_I, eta_Q, eps_I, eps_Q per step / (b sqrt(pi)) / peak
};

__global__ void k_im_nodes(ImNodeArgs a) {
    int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= a.N) return;
    // rotate_all_save: x' = R_tot x for positions, velocities, field
    double x[3], v[3], bb[3];
    for (int j = 0; j < 3; j++) {
        double sx = 0.0, sv = 0.0, sb = 0.0;
        for (int k = 0; k < 3; k++) {
            // uncontracted, as the reference's sums (the per-node mode starts
            // its rays at these positions)
            sv = __dadd_rn(sv, __dmul_rn(a.R[j + 3 * k], a.vel[3 * (size_t)n + k]));
            sb = __dadd_rn(sb, __dmul_rn(a.R[j + 3 * k], a.bvec[3 * (size_t)n + k]));
            sx = __dadd_rn(sx, __dmul_rn(a.R[j + 3 * k], a.xyz[3 * (size_t)n + k]));
        }
        x[j] = sx; v[j] = sv; bb[j] = sb;
    }
    for (int j = 0; j < 3; j++) a.xyz_r[3 * (size_t)n + j] = x[j];
    a.nrm2[n] = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
    // rot_stokes: alpha = acos(chi_y), negative when chi_x > 0
    const double cn = sqrt(bb[0] * bb[0] + bb[1] * bb[1]);
    const double chx = bb[0] / cn, chy = bb[1] / cn;
    double al = acos(chy);
    if (chx > 0.0) al = -al;
    // dust angle raytrace.f90:281-285: phi = acos(b_y/|b_xy|), negative when b_x < 0
    double ph = acos(bb[1] / sqrt(bb[0] * bb[0] + bb[1] * bb[1]));
    if (bb[0] < 0.0) ph = -ph;
    a.cellv[n] = make_float4((float)v[2], (float)(1.0 / a.b[n]), (float)cos(2.0 * al), (float)sin(2.0 * al));
    a.cellb[n] = make_float4((float)(1.0 - bb[2] * bb[2]), (float)cos(2.0 * ph), (float)sin(2.0 * ph), 0.f);
    // population read-back para_finish.f90:226-239 and comp_emcoefs for the
    // bulk nodes with a non-zero first population (:418)
    const int N = a.N, nlev = a.nlev;
    auto lp = [&](int l) { return a.levp[(size_t)nlev * n + l]; };
    auto sg = [&](int l) { return sqrt(2.0 * a.j_lev[l] + 1.0); };
    auto pp0 = [&](int l) {  // rho^0_0 of level l after read-back
        return lp(l) / sg(l);
    };
    auto pp2 = [&](int l) {  // rho^2_0 after read-back
        const double r0 = a.pops_in[(size_t)n + (size_t)N * (2 * l)];
        const double r2 = a.pops_in[(size_t)n + (size_t)N * (2 * l + 1)];
        if (l == 0) return r2;  // level 1's alignment keeps the value read
        return (r2 / r0) * lp(l) / sg(l);
    };
    const double th = acos(bb[2]);
    const double ct = cos(th), st = sin(th);
    const double tki = (3.0 * ct * ct - 1.0) / (2.0 * sqrt(2.0));
    const double tkq = -3.0 * st * st / (2.0 * sqrt(2.0));
    const double spi_b = 1.7724538509055160273 * a.b[n];
    for (int j = 0; j < a.nlines; j++) {
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        if (n < a.bulk && pp0(0) != 0.0) {
            const ImLine L = a.lines[j];
            const double r1_0 = pp0(L.lo), r2_0 = pp0(L.up);
            const double r1_2 = pp2(L.lo), r2_2 = pp2(L.up);
            const double g1 = 2.0 * L.j1 + 1.0, g2 = 2.0 * L.j2 + 1.0;
            const double wjj2_1 = L.fas * sqrt(3.0 * g1) * L.w1;
            const double wjj2_2 = L.fas * sqrt(3.0 * g2) * L.w2;
            const double na_I = 1.0 + wjj2_1 * (r1_2 / r1_0) * tki;
            const double na_Q = wjj2_1 * (r1_2 / r1_0) * tkq;
            const double ns_I = 1.0 + wjj2_2 * (r2_2 / r2_0) * tki;
            const double ns_Q = wjj2_2 * (r2_2 / r2_0) * tkq;
            const double b_to_a = L.nu0 * L.nu0 * L.nu0 / 6.781962e49;
            const double Bji = L.A / b_to_a;
            const double hv = 5.273e-35 * L.nu0;
            const double eI = hv * L.A * ns_I * sqrt(g2) * r2_0;
            const double eQ = hv * L.A * ns_Q * sqrt(g2) * r2_0;
            const double nI = hv * (g2 / g1) * Bji * (sqrt(g1) * r1_0 * na_I - sqrt(g2) * r2_0 * ns_I * g1 / g2);
            const double nQ = hv * (g2 / g1) * Bji * (sqrt(g1) * r1_0 * na_Q - sqrt(g2) * r2_0 * ns_Q * g1 / g2);
            // eta = cnu * v_corr * pol, v_corr = exp(-(dv/b)^2)/(b sqrt(pi)); per
            // trace step: * tx dx (raytrace.f90:221, 239, 250-258)
            const double cnu = (double)2.99792e8f / L.nu0;
            const double f = cnu / spi_b * a.tdx;
            // eta_Q exactly 0 (no alignment, sin(theta) = 0, or a line whose
            // w^(2) vanish) makes polarize_prop's eta_I/eta_Q * sinh(0) a NaN
            // (raytrace.f90:41-53): carried as a NaN coefficient, so I, Q, U
            // turn NaN wherever the reference's do, tau stays finite
            o = make_float4((float)(nI * f), nQ == 0.0 ? __int_as_float(0x7fc00000) : (float)(nQ * f),
                            (float)(eI * f), (float)(eQ * f));
        }
        a.coef[(size_t)j * N + n] = o;
    }
}

struct ImArgs {
    int N, npx, im_pix, nlines, nvel, nch, n_depth;
    int mode, nrays;         // 0: pixel grid, nrays = npx^2; 1: one ray per bulk node
    int star;                // star mode: rays starting on the star's disc start at its front
    int dust;                // the cloud has dust
    double Rs, sx, sy, sz;   // R_star / tx and the rotated star position
    double im_size, dx, inv_dx, tdx, alpha, dvel, v0;
    float R[9];              // the rotation (column-major), for directions in the unrotated frame
    const double *xyz;       // rotated (3,N)
    const double *nrm2;      // |X|^2 per node
    const int *off, *idx;    // neighbour CSR
    const float4 *edge;      // (e, |e|^2/2) per directed edge, unrotated
    const float4 *cellv, *cellb, *coef;
    const ImLine *lines;     // (nlines)
    const double *dust_p, *ibb;   // dust density; Planck function of the dust (nlines, N)
    int ray0, rays;          // this launch's rays [ray0, ray0 + rays), of nrays
    int2 *walk;              // march lists, per batch of 32 rays of the launch: 32 x n_depth
    int *cnt;                // per ray of the launch: records, -1 the start lies outside, -2 n_depth overflow
    unsigned char *on_star;  // per ray of the launch: it starts on the star
    int *status;
    float *out[8];           // (npx, npx, nch, nlines) or (nrays, nch, nlines) each, or null
};

__device__ __forceinline__ float phi1(float x) {  // (1 - e^-x)/x, stable near 0
    if (fabsf(x) < 0.1f)
        return 1.f + x * (-0.5f + x * (1.f / 6.f + x * (-1.f / 24.f + x * (1.f / 120.f + x * (-1.f / 720.f)))));
    return (1.f - expf(-x)) / x;
}

// Exponent of the lowest set bit of a double (v = m 2^e with m odd); a large
// value for 0, which constrains nothing.
__device__ __forceinline__ int lsb_exp(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffULL;
    if (b == 0ULL) return 1 << 20;
    int ex = (int)(b >> 52);
    unsigned long long m = b & 0xfffffffffffffULL;
    if (ex) {
        m |= 1ULL << 52;
        ex -= 1075;
    } else {
        ex = -1074;
    }
    return ex + __ffsll((long long)m) - 1;
}

// n successive FP64 additions z = z + dx, bit for bit, in O(binades) steps.
// While every partial sum z + j dx is representable -- all of them are
// multiples of g = min(lsb(z), lsb(dx)), so each is exact as long as its
// magnitude stays below L = g 2^53 -- the additions are exact and their
// result is the single correctly rounded fma(m, dx, z) (m dx itself is exact:
// dx is the REAL*4 step, a 24-bit mantissa, and m < 2^29).  Only a sum that
// enters a binade whose spacing exceeds g can round; that one addition is
// made as the reference makes it, after which z lies on the coarser grid.
// (The quotient only places m, two short of the limit: a product with 1/dx
// serves.)
__device__ double add_steps(double z, long long n, double dx, double inv_dx, int e_dx) {
    while (n > 0) {
        const int eg = min(lsb_exp(z), e_dx);
        const double L = __longlong_as_double((long long)(min(eg + 53, 1022) + 1023) << 52);
        long long m = (long long)floor((L - z) * inv_dx) - 2;  // z + m dx < L, with margin
        if (m > n) m = n;
        if (m > 0) {
            z = __fma_rn((double)m, dx, z);
            n -= m;
        }
        if (n > 0) {
            z = __dadd_rn(z, dx);
            n--;
        }
    }
    return z;
}

__device__ double black_body(double T, double nu) {
    if (T == 0.0) return 0.0;
    return 1.4744995e-50 * nu * nu * nu / (exp(4.79924e-11 / T * nu) - 1.0);
}

// the dust's Planck function per (line, node)
__global__ void k_im_dust(int N, int nlines, const ImLine *__restrict__ lines, const double *__restrict__ tdust,
                          double *__restrict__ ibb) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)N * nlines) return;
    ibb[t] = black_body(tdust[t % N], lines[t / N].nu0);
}

// Index of record k of ray r (of its batch of 32) in the batch's march list:
// blocks of 32 records, the rays' blocks side by side.
__device__ __forceinline__ int march_at(int k, int r) { return ((k >> 5) << 10) + (r << 5) + (k & 31); }
__device__ __forceinline__ const int2 *march_list(const ImArgs &a, int i) {
    return a.walk + (size_t)(i >> 5) * 1024 * (size_t)((a.n_depth + 31) / 32);
}
// Work index w -> the reference's pixel p = a npx + b (para_finish.f90:
// 369-376) with a = w mod npx: consecutive work items step along the cube's
// first (fastest) index (mode 1: w is the node).
__device__ __forceinline__ int ray_of(const ImArgs &a, int w) {
    return (a.mode == 1) ? w : (w % a.npx) * a.npx + w / a.npx;
}
// where channel ch of line j of ray p goes in the output arrays
__device__ __forceinline__ size_t cube_at(const ImArgs &a, int p, int ch, int j) {
    if (a.mode == 1) return (size_t)p + (size_t)a.nrays * ((size_t)ch + (size_t)a.nch * j);
    const int ia = p / a.npx, ib = p % a.npx;
    return (size_t)ia + (size_t)a.npx * ((size_t)ib + (size_t)a.npx * ((size_t)ch + (size_t)a.nch * j));
}

constexpr double IM_NEAR = 1e-12;  // squared distances closer than this are compared in FP64 at every step

// The start node (raytrace.f90:126-134 scans all nodes; strict <, so the
// lowest index wins) and its distance.  The same argmin by greedy descent on
// the Delaunay graph: a node that is not the nearest has a neighbour at most
// as far (the segment to the point leaves its Voronoi cell through a face
// shared with that neighbour), so descending in (distance, index) order ends
// at the nearest node with the lowest index, from any start.  The descent
// runs in FP32 on the edge records (nearer by e.r > |e|^2/2); FP64 distances,
// computed exactly as the reference's norm2, decide between the last node and
// the neighbours that FP32 cannot tell from it.
__device__ int start_node(const ImArgs &a, double x, double y, double z0, double *best_out) {
    int c = 0;
    auto dist = [&](int i) {
        return __dsqrt_rn(dsum3sq(x - a.xyz[3 * (size_t)i], y - a.xyz[3 * (size_t)i + 1],
                                  z0 - a.xyz[3 * (size_t)i + 2]));
    };
    auto offset = [&](int i, float &rx, float &ry, float &rz) {   // point - node, unrotated frame
        const float ux = (float)(x - a.xyz[3 * (size_t)i]), uy = (float)(y - a.xyz[3 * (size_t)i + 1]),
                    uz = (float)(z0 - a.xyz[3 * (size_t)i + 2]);
        rx = a.R[0] * ux + a.R[1] * uy + a.R[2] * uz;
        ry = a.R[3] * ux + a.R[4] * uy + a.R[5] * uz;
        rz = a.R[6] * ux + a.R[7] * uy + a.R[8] * uz;
    };
    double best = 0.0;
    float rx, ry, rz;
    offset(c, rx, ry, rz);
    bool fine = false;
    for (int hop = 0; hop < 2 * a.N; hop++) {
        const int o = a.off[c], deg = a.off[c + 1] - o;
        float g = 0.f;
        int bj = -1;
        unsigned long long close = 0ULL;   // (first 64) neighbours not certainly farther
        const float r2 = rx * rx + ry * ry + rz * rz;
        for (int j0 = 0; j0 < deg; j0 += 8) {
            float4 e8[8];
#pragma unroll
            for (int i = 0; i < 8; i++) e8[i] = a.edge[o + min(j0 + i, deg - 1)];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float4 e = e8[i];
                const float gain = e.x * rx + e.y * ry + e.z * rz - e.w, tol = 1e-6f * (2.f * e.w + r2);
                if (j0 + i >= deg) continue;
                if (gain > tol + g) {
                    g = gain - tol;
                    bj = j0 + i;
                }
                if (j0 + i < 64 && gain > -tol) close |= 1ULL << (j0 + i);
            }
        }
        if (!fine && bj >= 0) {
            c = a.idx[o + bj];
            offset(c, rx, ry, rz);
            continue;
        }
        // FP64: (distance, index) order over the neighbours in doubt
        if (!fine) best = dist(c);
        fine = true;
        int nbest = c;
        double dbest = best;
        auto probe = [&](int j) {
            const int nb = a.idx[o + j];
            const double d = dist(nb);
            if (d < dbest || (d == dbest && nb < nbest)) { dbest = d; nbest = nb; }
        };
        for (unsigned long long m = close; m; m &= m - 1ULL) probe(__ffsll((long long)m) - 1);
        for (int j = 64; j < deg; j++) probe(j);
        if (nbest == c) break;
        c = nbest;
        best = dbest;
        offset(c, rx, ry, rz);
    }
    *best_out = best;
    return c;
}

// The fixed-step march of one ray along +z (trace_out_raytrace): records
// (node, step) at every change of the nearest node and at the exit.
// Returns the record count; *st: 1 more than n_depth records, 3 the start
// point is outside the unit sphere.
__device__ int march(const ImArgs &a, int ray, int lane, int2 *dl, int *st_out, int *fs_out, int e_dx) {
    const int p = ray;
    double x, y;
    if (a.mode == 1) {  // the node's rotated sky position (para_finish.f90:296)
        x = a.xyz[3 * (size_t)p];
        y = a.xyz[3 * (size_t)p + 1];
    } else {
        const int ia = p / a.npx - a.im_pix, ib = p % a.npx - a.im_pix;
        x = ia * a.im_size / a.im_pix;
        y = ib * a.im_size / a.im_pix;
    }
    // the oracle's FP64 arithmetic, without FMA contraction, throughout the march
    const double zs0 = -1.0 * __dsqrt_rn(__dsub_rn(__dsub_rn(1.0, __dmul_rn(x, x)), __dmul_rn(y, y)));
    double z0 = zs0;
    if (a.star) {  // raytrace.f90:103-115: on the star's disc, start at its front
        const double xc = __dsub_rn(x, a.sx), yc = __dsub_rn(y, a.sy);
        if (__dsqrt_rn(__dadd_rn(__dmul_rn(xc, xc), __dmul_rn(yc, yc))) < a.Rs) {
            z0 = __dadd_rn(a.sz, a.Rs);
            *fs_out = 1;
        }
    }
    double best;
    int c = start_node(a, x, y, z0, &best);
    if (!(best < 10.0)) {  // start point outside the unit sphere (NaN; rsave = 10)
        *st_out = 3;
        return 0;
    }
    double z = z0;
    int k = 0, nc = 0;
    const double zexit = -zs0, z_inside = zexit - 4.0 * a.dx;   // between -zexit and here no step can exit
    const float nx = a.R[2], ny = a.R[5], nz = a.R[8];   // the ray's direction, unrotated frame
    for (;;) {
        // Where the nearest node can change next: in FP32 on the edge records,
        // with bounds on their rounding.  Half the difference of the squared
        // distances to neighbour j and to c at a distance s ahead is num - s
        // den, num = |e|^2/2 - e.r and den = e.n; |num| is off by less than B =
        // 1e-6 (|e|^2 + |r|^2), den by less than D = 4e-7 |e|.  So a crossing
        // lies before s_up = min (num + B)/(den - D), and only neighbours with
        // num - B - s (den + D) <= IM_NEAR up to s = s_up + window can win
        // check_neigh's strict comparison there; FP64 then looks at those alone.
        const double cx = a.xyz[3 * (size_t)c], cy = a.xyz[3 * (size_t)c + 1], cz = a.xyz[3 * (size_t)c + 2];
        const int o = a.off[c], deg = a.off[c + 1] - o;
        const float ux = (float)(x - cx), uy = (float)(y - cy), uz = (float)(z - cz);
        const float rx = a.R[0] * ux + a.R[1] * uy + a.R[2] * uz;
        const float ry = a.R[3] * ux + a.R[4] * uy + a.R[5] * uz;
        const float rz = a.R[6] * ux + a.R[7] * uy + a.R[8] * uz;
        const float r2 = rx * rx + ry * ry + rz * rz;
        const double WIN = 6.0 * a.dx;
        const float win = 8.f * (float)a.dx;
        unsigned long long cand = 0ULL;   // of the first 64 neighbours
        float un = fmaxf((float)(zexit - z), 0.f) + win, ud = 1.f;   // s_up
        for (int j0 = 0; j0 < deg; j0 += 8) {
            float4 e8[8];
#pragma unroll
            for (int i = 0; i < 8; i++) e8[i] = a.edge[o + min(j0 + i, deg - 1)];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float4 e = e8[i];
                if (j0 + i >= deg) continue;
                const float num = e.w - (e.x * rx + e.y * ry + e.z * rz), den = e.x * nx + e.y * ny + e.z * nz;
                const float B = 1e-6f * (2.f * e.w + r2), D = 4e-7f * sqrtf(2.f * e.w);
                const float hn = fmaxf(num + B, 0.f), hd = den - D;
                if (hd > 0.f && hn * ud < un * hd) {
                    un = hn;
                    ud = hd;
                }
                // (s_up only falls further in this loop: the set is a superset)
                if (j0 + i < 64 && (num - B - 1e-12f) * ud <= (den + D) * (un + win * ud)) cand |= 1ULL << (j0 + i);
                if (j0 + i < 64 && num - B <= 1e-12f) cand |= 1ULL << (j0 + i);
            }
        }
        // the FP64 crossings of the candidates: the steps before kt are those at
        // which every neighbour is farther than c by IM_NEAR or more, which
        // exceeds the FP64 rounding of both squared distances (~1e-15)
        double tn = zexit, td = 1.0;
        bool now = false;
        const double cc = a.nrm2[c];
        auto cross = [&](int j) {
            const int nb = a.idx[o + j];
            const double gx = a.xyz[3 * (size_t)nb], gy = a.xyz[3 * (size_t)nb + 1], gz = a.xyz[3 * (size_t)nb + 2];
            // |P-X_n|^2 - |P-X_c|^2 = A - 2 z dzn along the ray
            const double d2 = 2.0 * (gz - cz);
            const double A = a.nrm2[nb] - cc - 2.0 * x * (gx - cx) - 2.0 * y * (gy - cy) - IM_NEAR;
            if (A - z * d2 < 0.0) now = true;   // already (nearly) nearer: replay now
            else if (d2 > 0.0 && A * td < tn * d2) {
                tn = A;
                td = d2;
            }
        };
        {
            const float s_lim = un / ud + win;
            unsigned long long keep = 0ULL;
            for (unsigned long long m = cand; m; m &= m - 1ULL) {
                const int j = __ffsll((long long)m) - 1;
                const float4 e = a.edge[o + j];
                const float num = e.w - (e.x * rx + e.y * ry + e.z * rz), den = e.x * nx + e.y * ny + e.z * nz;
                const float B = 1e-6f * (2.f * e.w + r2), D = 4e-7f * sqrtf(2.f * e.w);
                if (num - B - 1e-12f > 0.f && num - B - 1e-12f > s_lim * (den + D)) continue;
                keep |= 1ULL << j;
                cross(j);
            }
            cand = keep;
            for (int j = 64; j < deg; j++) cross(j);
        }
        // (the quotient from an FP32 reciprocal and one Newton step: to 1e-13, it
        // only places the replay)
        const double rtd = (double)(1.f / (float)td), q0 = tn * rtd;
        const double zt = now ? z : q0 + (tn - q0 * td) * rtd;
        const double z_lim = fmin(zt, zexit) + WIN;
        if (!now) {
            // z after k steps is z0 + k dx to ~1e-12, far within the 1e-6 of a step
            // left here; the exit is replayed from three steps before
            const long long kt = min((long long)floor((zt - z0) * a.inv_dx - 1e-6),
                                     (long long)floor((zexit - z0) * a.inv_dx) - 3);
            if ((long long)k < kt) {  // the reference's own additions, in jumps
                z = add_steps(z, kt - k, a.dx, a.inv_dx, e_dx);
                k = (int)kt;
            }
        }
        // exact replay of trace_out_raytrace's loop until c changes or the ray exits
        bool done = false, changed = false;
        while (!done && !changed) {
            z = z + a.dx;
            k++;
            // norm2(X_phot) > 1: the rounded root of s exceeds 1 when s exceeds 1 + 2^-52
            if (!(z > zs0 && z < z_inside) && dsum3sq(x, y, z) > 1.0 + 0x1p-52) {
                if (nc >= a.n_depth) { *st_out = 1; return nc; }
                dl[march_at(nc++, lane)] = make_int2(c, k);
                done = true;
            }
            // check_neigh miscellaneous.f90:1-46, in list order: the candidates
            // while z <= z_lim (and every neighbour past the 64th), else all
            double d0 = dsum3sq(x - cx, y - cy, z - cz);
            int nn = c;
            auto probe = [&](int j) {
                const int nb = a.idx[o + j];
                const double ex = x - a.xyz[3 * (size_t)nb], ey = y - a.xyz[3 * (size_t)nb + 1],
                             ez = z - a.xyz[3 * (size_t)nb + 2];
                const double dd = dsum3sq(ex, ey, ez);
                if (dd < d0) { d0 = dd; nn = nb; }
            };
            if (z <= z_lim) {
                for (unsigned long long m = cand; m; m &= m - 1ULL) probe(__ffsll((long long)m) - 1);
                for (int j = 64; j < deg; j++) probe(j);
            } else {
                for (int j = 0; j < deg; j++) probe(j);
            }
            if (nn != c) {
                if (nc >= a.n_depth) { *st_out = 1; return nc; }
                dl[march_at(nc++, lane)] = make_int2(nn, k);
                c = nn;
                changed = true;
            }
        }
        if (done) break;
    }
    return nc;
}

// The marches of the launch's rays, one lane per ray, `per` rays to a warp:
// with few rays a full warp's serial chain (the longest of its 32 marches) is
// the launch's time, and more warps of fewer rays run beside each other.
__global__ void __launch_bounds__(64) k_im_march(ImArgs a, int per) {
    const int i = (blockIdx.x * 2 + (threadIdx.x >> 5)) * per + (threadIdx.x & 31);
    if ((int)(threadIdx.x & 31) >= per || i >= a.rays) return;
    const int p = ray_of(a, a.ray0 + i);
    int st = 0, fs = 0;
    const int nc = march(a, p, i & 31, const_cast<int2 *>(march_list(a, i)), &st, &fs, lsb_exp(a.dx));
    a.cnt[i] = st == 0 ? nc : st == 3 ? -1 : -2;
    a.on_star[i] = (unsigned char)fs;
    if (a.status) a.status[p] = st;
}

// The dust maps (raytrace.f90:268-290, finish :301-317): independent of the
// channel, FP64, one thread per (ray, line).
__global__ void __launch_bounds__(64) k_im_dust_maps(ImArgs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
    if (i >= a.rays) return;
    const ImLine L = a.lines[j];
    const int ncr = a.cnt[i];
    const int2 *dl = march_list(a, i);
    const double Iin = a.on_star[i] ? L.bb_star : L.bb_cmb;
    double Id = Iin, sig0 = 0.0, sig2 = 0.0, Qd = 0.0, Ud = 0.0, taud = 0.0;
    for (int k = 0; a.dust && k + 1 < ncr; k++) {
        const int2 e0 = dl[march_at(k, i & 31)];
        const int cell = e0.x, dk = dl[march_at(k + 1, i & 31)].y - e0.y;
        const double tau_d = L.kd * a.dust_p[cell] * (a.tdx * (double)dk);
        if (tau_d > 1e-30) {
            const float4 cb = a.cellb[cell];
            const double Ibb = a.ibb[(size_t)j * a.N + cell];
            const double ed = exp(-tau_d);
            const double mu2 = cb.x;
            const double sI = 0.5 * a.alpha * (mu2 - 2.0 / 3.0), sQ = a.alpha * mu2;
            Id = Id * ed + Ibb * (1 - ed);
            sig0 = sig0 * ed + Ibb * (1 - ed);
            sig2 = sig2 * ed + sI * Ibb * (1 - ed);
            Qd = Qd * ed + sQ * Ibb * (1 - ed) * cb.y;
            Ud = Ud * ed + sQ * Ibb * (1 - ed) * cb.z;
            taud = taud + tau_d;
        }
    }
    double Idf = Id - L.bb_cmb, Qdf = 0.0, Udf = 0.0, tdf = 0.0;
    if (Idf != 0.0) {
        Qdf = Idf * Qd / (sig0 - sig2);
        Udf = Idf * Ud / (sig0 - sig2);
        tdf = taud;
    }
    const bool bad = ncr < 0;
    const float v[4] = {bad ? NAN : (float)Idf, bad ? NAN : (float)Qdf, bad ? NAN : (float)Udf, bad ? NAN : (float)tdf};
    const int p = ray_of(a, a.ray0 + i);
    for (int ch = 0; ch < a.nch; ch++) {
        const size_t o = cube_at(a, p, ch, j);
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (a.out[4 + q]) a.out[4 + q][o] = v[q];
    }
}

// Stokes state of one (ray, line, channel) along its march.
struct Stokes {
    float I, Q, U, tau, tauc;
    __device__ __forceinline__ void start(float Iin) { I = Iin; Q = 0.f; U = 0.f; tau = 0.f; tauc = 0.f; }
    // a cell: cv (v_z, 1/b, cos 2 alpha, sin 2 alpha), cf the line's
    // coefficients, fdk trace steps, vobs the channel's velocity
    __device__ __forceinline__ void cell(float4 cv, float4 cf, float fdk, float vobs) {
        const float q = (vobs - cv.x) * cv.y;
        const float vc = expf(-q * q) * fdk;
        const float ta = cf.x * vc, tq = cf.y * vc, ei = cf.z * vc, eq = cf.w * vc;
        if (ta > 1e-30f) {  // raytrace.f90:260
            // rot_stokes into the node frame
            const float Qn = Q * cv.z + U * cv.w;
            const float Un = U * cv.z - Q * cv.w;
            const float pm = ta - tq, pp = ta + tq;
            const float Ep = expf(-pm), Em = expf(-pp);
            const float fp = phi1(pm), fm = phi1(pp);
            const float o11 = 0.5f * (fp + fm), o12 = -0.5f * (fp - fm);
            const float ech = 0.5f * (Ep + Em), esh = 0.5f * (Ep - Em);
            const float In = o11 * ei + o12 * eq + (ech * I - esh * Qn);
            const float Qo = o12 * ei + o11 * eq + (-esh * I + ech * Qn);
            const float Uo = Un * expf(-ta);
            I = In;
            // rot_stokes_back
            Q = Qo * cv.z - Uo * cv.w;
            U = Uo * cv.z + Qo * cv.w;
            // compensated tau sum
            const float yk = ta - tauc;
            const float tk = tau + yk;
            tauc = (tk - tau) - yk;
            tau = tk;
        } else if (cv.z != cv.z) {
            // the reference rotates Q, U into the node frame and back at
            // every cell; a field along the line of sight has no frame
            // (NaN angle), which makes them NaN there too
            Q = cv.z;
            U = cv.z;
        }
    }
    __device__ __forceinline__ void store(const ImArgs &a, int p, int ch, int j, bool bad) const {
        const size_t o = cube_at(a, p, ch, j);
        const float v[4] = {bad ? NAN : (float)((double)I - a.lines[j].bb_cmb), bad ? NAN : Q, bad ? NAN : U,
                            bad ? NAN : tau};
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (a.out[q]) a.out[q][o] = v[q];
    }
};
__device__ __forceinline__ float channel_velocity(const ImArgs &a, int ch) {
    return (float)((ch - a.nvel) * a.dvel + a.v0);
}

// Whole slots of 32 channels: a warp takes NS slots (from slot s0) of one
// line of one ray, lanes over channels, the cells' records staged 32 at a
// time.  The rays of a block of warps are neighbours in the image, so the
// stores of a channel fill sectors.
constexpr int IM_WARPS = 8;
template <int NS>
__global__ void __launch_bounds__(32 * IM_WARPS) k_im_stokes(ImArgs a, int s0) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ float4 s_cv[IM_WARPS][32], s_cf[IM_WARPS][32];
    __shared__ float s_dk[IM_WARPS][32];
    const int i = blockIdx.x * IM_WARPS + warp, j = blockIdx.y;
    if (i >= a.rays) return;
    const int cnt = a.cnt[i], ncr = max(cnt, 0);
    const int2 *dl = march_list(a, i);
    const float Iin = (float)(a.on_star[i] ? a.lines[j].bb_star : a.lines[j].bb_cmb);  // I_in (raytrace.f90:97-115)
    Stokes st[NS];
    float vobs[NS];
#pragma unroll
    for (int s = 0; s < NS; s++) {
        st[s].start(Iin);
        vobs[s] = channel_velocity(a, min(lane + 32 * (s0 + s), a.nch - 1));
    }
    for (int k0 = 0; k0 + 1 < ncr; k0 += 32) {
        const int n = min(32, ncr - 1 - k0);
        __syncwarp();
        if (lane < n) {
            const int2 e0 = dl[march_at(k0 + lane, i & 31)];
            const int k1 = dl[march_at(k0 + lane + 1, i & 31)].y;
            s_cv[warp][lane] = a.cellv[e0.x];
            s_cf[warp][lane] = a.coef[(size_t)j * a.N + e0.x];
            s_dk[warp][lane] = (float)(k1 - e0.y);
        }
        __syncwarp();
        for (int k = 0; k < n; k++) {
            const float4 cv = s_cv[warp][k], cf = s_cf[warp][k];
            const float fdk = s_dk[warp][k];
#pragma unroll
            for (int s = 0; s < NS; s++) st[s].cell(cv, cf, fdk, vobs[s]);
        }
    }
    const int p = ray_of(a, a.ray0 + i);
#pragma unroll
    for (int s = 0; s < NS; s++) {
        const int ch = lane + 32 * (s0 + s);
        if (ch < a.nch) st[s].store(a, p, ch, j, cnt < 0);
    }
}

// The channels past the whole slots (ch0 on), lanes over rays: a thread takes
// up to 4 of one line of one ray.  One such channel would otherwise cost a
// slot of 32 lanes (the reference's 2 nvel + 1 channels always leave some).
__global__ void __launch_bounds__(64) k_im_stokes_tail(ImArgs a, int ch0) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, c0 = ch0 + 4 * blockIdx.z;
    if (i >= a.rays) return;
    const int cnt = a.cnt[i], n = min(4, a.nch - c0);
    const int2 *dl = march_list(a, i);
    const float Iin = (float)(a.on_star[i] ? a.lines[j].bb_star : a.lines[j].bb_cmb);
    Stokes st[4];
    float vobs[4];
#pragma unroll
    for (int s = 0; s < 4; s++) {
        st[s].start(Iin);
        vobs[s] = channel_velocity(a, min(c0 + s, a.nch - 1));
    }
    int2 e0 = (cnt > 0) ? dl[march_at(0, i & 31)] : make_int2(0, 0);
    for (int k = 0; k + 1 < cnt; k++) {
        const int2 e1 = dl[march_at(k + 1, i & 31)];
        const float4 cv = a.cellv[e0.x], cf = a.coef[(size_t)j * a.N + e0.x];
        const float fdk = (float)(e1.y - e0.y);
#pragma unroll
        for (int s = 0; s < 4; s++)
            if (s < n) st[s].cell(cv, cf, fdk, vobs[s]);
        e0 = e1;
    }
    const int p = ray_of(a, a.ray0 + i);
#pragma unroll
    for (int s = 0; s < 4; s++)
        if (s < n) st[s].store(a, p, c0 + s, j, cnt < 0);
}
// Leftover channels up to this many go to the tail kernel, more to a padded
// slot.
constexpr int IM_TAIL = 16;

}  // namespace

// mode 0: the pixel grid (2 im_pix + 1)^2; mode 1: one ray per bulk node
static int image_call(portal_ctx *c, const double *pol_pops, int nlines, const int *l1, const int *l2,
                      double th_inc, double ph_az, int nvel, double dvel, double v0, int mode, int im_pix,
                      double im_size, double alpha, double dx, int n_depth_rt, double *xy, float *const *dout,
                      int *status) {
    const char *fn = mode ? "portal_image_nodes" : "portal_image";
    if (!c->have_cloud || !c->have_mol) return set_err(c, PORTAL_ERR_STATE, "no cloud or molecule");
    if (nlines < 1 || nlines > IM_MAX_LINES || !l1 || !l2 || nvel < 0 || 2 * nvel + 1 > 288 ||
        im_pix < 1 || !(im_size > 0.0) || !(dx > 0.0) || n_depth_rt < 1)
        return set_err(c, PORTAL_ERR_ARG, std::string(fn) + ": bad arguments");
    if (mode == 0 && im_size * im_size * 2.0 >= 1.0)
        return set_err(c, PORTAL_ERR_ARG, "portal_image: im_size must keep the image corners inside "
                                          "the unit sphere (im_size < 1/sqrt(2))");
    if (!pol_pops && !c->have_pops())
        return set_err(c, PORTAL_ERR_STATE, std::string(fn) + ": no pol_pops (pass them or run portal_solve_se)");
    cudaSetDevice(c->device);
    timers_reset(c);
    const int N = c->N, nlev = c->nlev, nch = 2 * nvel + 1, npx = 2 * im_pix + 1;
    const int nrays = mode ? c->bulk : npx * npx;
    // line data (para_finish.f90:173-185): every line takes the frequency of the
    // last (l1, l2) pair, as the whole-array assignment there does
    ImLine h[IM_MAX_LINES];
    for (int i = 0; i < nlines; i++) {
        if (l1[i] < 1 || l1[i] > nlev || l2[i] < 1 || l2[i] > nlev)
            return set_err(c, PORTAL_ERR_ARG, std::string(fn) + ": line level out of range");
        if (mode && l1[i] > c->r_num)
            return set_err(c, PORTAL_ERR_ARG, "portal_image_nodes: t_Aji(l1) needs l1 <= the number of "
                                              "radiative transitions");
    }
    const double nu_last = c->e_levs[l2[nlines - 1] - 1] - c->e_levs[l1[nlines - 1] - 1];
    for (int i = 0; i < nlines; i++) {
        ImLine &L = h[i];
        L.nu0 = nu_last;
        L.A = 0.0; L.kd = 0.0;
        for (int r = 0; r < c->r_num; r++)
            if (l2[i] == c->r_trans[2 * r + 1] && l1[i] == c->r_trans[2 * r]) {
                L.A = c->A[r]; L.kd = c->kd_v[r];
                break;
            }
        if (mode) L.A = c->A[l1[i] - 1];  // para_finish.f90:303 passes t_Aji(l1(j))
        L.lo = l1[i] - 1; L.up = l2[i] - 1;
        L.j1 = c->j_lev[L.lo]; L.j2 = c->j_lev[L.up];
        L.w1 = wigner6j(2, 2, 4, 2 * L.j1, 2 * L.j1, 2 * L.j2);
        L.w2 = wigner6j(2, 2, 4, 2 * L.j2, 2 * L.j2, 2 * L.j1);
        L.fas = ((1 + L.j1 + L.j2) % 2 == 0) ? 1.0 : -1.0;
        L.bb_cmb = 1.4744995e-50 * std::pow(nu_last, 3.0) *
                   std::pow(std::exp(4.79924e-11 / 2.73 * nu_last) - 1.0, -1.0);
        L.bb_star = (c->star_mode && c->T_star > 0.0)
                        ? 1.4744995e-50 * std::pow(nu_last, 3.0) *
                              std::pow(std::exp(4.79924e-11 / c->T_star * nu_last) - 1.0, -1.0)
                        : 0.0;
    }
    if (c->im_lines.reserve(sizeof(ImLine) * IM_MAX_LINES)) return set_err(c, PORTAL_ERR_NOMEM, "image lines");
    const ImLine *lines = reinterpret_cast<const ImLine *>(c->im_lines.p);
    PCHECK(c, cudaMemcpyAsync(c->im_lines.p, h, sizeof(ImLine) * nlines, cudaMemcpyHostToDevice, c->stream));
    // rotation R_tot = R_z(ph_az) R_x(th_inc) (rotmat miscellaneous.f90:146-181)
    auto rotmat = [](const double *nv, double th, double *R) {
        double ct = std::cos(th), oc = 1.0 - ct, s = std::sin(th);
        for (int i = 0; i < 3; i++) R[i + 3 * i] = ct + oc * nv[i] * nv[i];
        R[0 + 3 * 1] = nv[0] * nv[1] * oc - nv[2] * s; R[1 + 3 * 0] = nv[1] * nv[0] * oc + nv[2] * s;
        R[0 + 3 * 2] = nv[0] * nv[2] * oc + nv[1] * s; R[2 + 3 * 0] = nv[2] * nv[0] * oc - nv[1] * s;
        R[1 + 3 * 2] = nv[1] * nv[2] * oc - nv[0] * s; R[2 + 3 * 1] = nv[2] * nv[1] * oc + nv[0] * s;
    };
    const double xv[3] = {1, 0, 0}, zv[3] = {0, 0, 1};
    double Rth[9], Rph[9];
    rotmat(xv, th_inc, Rth);
    rotmat(zv, ph_az, Rph);
    ImNodeArgs na;
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) {
            double s = 0.0;
            for (int k = 0; k < 3; k++) s += Rph[i + 3 * k] * Rth[k + 3 * j];
            na.R[i + 3 * j] = s;
        }
    // device buffers
    DevBuf<double> &xyz_r = c->im_xyz, &pops_d = c->im_pops, &nrm2 = c->im_nrm2, &ibb = c->im_ibb;
    DevBuf<int> &jl = c->im_jl, &stat = c->im_stat, &cnt = c->im_cnt;
    DevBuf<float4> &cellv = c->im_cellv, &cellb = c->im_cellb, &coef = c->im_coef;
    DevBuf<float> &outd = c->im_out;
    DevBuf<unsigned char> &on_star = c->im_star;
    // the cubes are kept for the next call up to KEEP_BYTES
    struct KeepSmall {
        DevBuf<float> &b;
        ~KeepSmall() {
            if (b.n * sizeof(float) > KEEP_BYTES) b.release();
        }
    } keep{outd};
    const size_t cube = (size_t)nrays * nch * nlines;
    if (xyz_r.reserve(3 * (size_t)N) || nrm2.reserve(N) || cellv.reserve(N) || cellb.reserve(N) ||
        coef.reserve((size_t)nlines * N) || jl.reserve(nlev) || stat.reserve((size_t)(nrays > 0 ? nrays : 1)))
        return set_err(c, PORTAL_ERR_NOMEM, "image buffers");
    const double *pops_src = c->pops.p;
    if (pol_pops) {
        if (pops_d.reserve((size_t)N * 2 * nlev)) return set_err(c, PORTAL_ERR_NOMEM, "pol_pops");
        PCHECK(c, cudaMemcpyAsync(pops_d.p, pol_pops, (size_t)N * 2 * nlev * sizeof(double),
                                  cudaMemcpyHostToDevice, c->stream));
        pops_src = pops_d.p;
    }
    PCHECK(c, cudaMemcpyAsync(jl.p, c->j_lev.data(), nlev * sizeof(int), cudaMemcpyHostToDevice, c->stream));
    na.N = N; na.bulk = c->bulk; na.nlev = nlev; na.nlines = nlines; na.tdx = c->tx * dx;
    na.xyz = c->pos64.p; na.vel = c->vel64.p; na.bvec = c->bvec64.p; na.b = c->b64.p;
    na.tdust = c->tdust.p; na.levp = c->levp.p; na.pops_in = pops_src; na.j_lev = jl.p; na.lines = lines;
    na.xyz_r = xyz_r.p; na.nrm2 = nrm2.p; na.cellv = cellv.p; na.cellb = cellb.p; na.coef = coef.p;
    timer_start(c, T_EMCOEF);
    k_im_nodes<<<(N + 127) / 128, 128, 0, c->stream>>>(na);
    timer_stop(c, T_EMCOEF);
    PCHECK(c, cudaGetLastError());
    if (c->has_dust) {
        if (ibb.reserve((size_t)nlines * N)) return set_err(c, PORTAL_ERR_NOMEM, "dust emission");
        const long long tot = (long long)nlines * N;
        k_im_dust<<<(unsigned)((tot + 127) / 128), 128, 0, c->stream>>>(N, nlines, lines, c->tdust.p, ibb.p);
        PCHECK(c, cudaGetLastError());
    }
    // outputs on the device
    int nout = 0;
    for (int q = 0; q < 8; q++) nout += dout[q] ? 1 : 0;
    if (outd.reserve(cube * (nout ? nout : 1))) return set_err(c, PORTAL_ERR_NOMEM, "image outputs");
    ImArgs ia;
    ia.N = N; ia.npx = npx; ia.im_pix = im_pix; ia.nlines = nlines; ia.nvel = nvel; ia.nch = nch;
    ia.mode = mode; ia.nrays = nrays;
    // star mode: R_star / tx (para_finish.f90:187) and the star's position rotated with the
    // nodes (rotate_all_save miscellaneous.f90:899-904), used unscaled as the reference does
    ia.star = c->star_mode;
    ia.Rs = c->star_mode ? c->R_star() : 0.0;
    {
        double sp[3] = {0.0, 0.0, 0.0};
        for (int j = 0; j < 3; j++)
            for (int k = 0; k < 3; k++) sp[j] = sp[j] + na.R[j + 3 * k] * c->X_star[k];
        ia.sx = sp[0]; ia.sy = sp[1]; ia.sz = sp[2];
    }
    ia.n_depth = n_depth_rt; ia.im_size = im_size; ia.dx = dx; ia.tdx = c->tx * dx; ia.alpha = alpha; ia.dvel = dvel; ia.v0 = v0;
    ia.xyz = xyz_r.p; ia.nrm2 = nrm2.p; ia.off = c->nb_off.p; ia.idx = c->nb_idx.p; ia.cellv = cellv.p; ia.cellb = cellb.p;
    ia.lines = lines; ia.coef = coef.p; ia.dust_p = c->dustp.p; ia.ibb = ibb.p; ia.dust = c->has_dust; ia.status = stat.p;
    ia.edge = c->edge.p; ia.inv_dx = 1.0 / dx;
    for (int i = 0; i < 9; i++) ia.R[i] = (float)na.R[i];
    {
        int q2 = 0;
        for (int q = 0; q < 8; q++) ia.out[q] = dout[q] ? outd.p + cube * (q2++) : nullptr;
    }
    // Rays per launch: as many as keep the march lists (n_depth_rt records per
    // ray) within 6 GB, fewer where the device cannot hold that.
    const size_t list = 1024 * (size_t)((n_depth_rt + 31) / 32);   // int2 records per batch of 32 rays
    long long batches = std::max(1, (nrays + 31) / 32);
    batches = std::min(batches, std::max<long long>(c->sm_count, (long long)(6e9 / (list * sizeof(int2)))));
    while (c->walk.reserve(batches * list) != cudaSuccess) {
        if ((batches /= 2) < 1) return set_err(c, PORTAL_ERR_NOMEM, "image walk scratch");
    }
    if (cnt.reserve(32 * batches) || on_star.reserve(32 * batches))
        return set_err(c, PORTAL_ERR_NOMEM, "image walk scratch");
    ia.walk = c->walk.p;
    ia.cnt = cnt.p;
    ia.on_star = on_star.p;
    const bool stokes = dout[0] || dout[1] || dout[2] || dout[3], dustmaps = dout[4] || dout[5] || dout[6] || dout[7];
    const int left = nch % 32, tail = left <= IM_TAIL ? left : 0, slots = (nch - tail + 31) / 32;
    timer_start(c, T_IMWALK);
    for (ia.ray0 = 0; ia.ray0 < nrays; ia.ray0 += ia.rays) {
        ia.rays = (int)std::min<long long>(nrays - ia.ray0, 32 * batches);
        // rays per marching warp: fewer while that leaves at most 8 warps per SM
        // (3,000 rays: 0.49 ms with 32 a warp, 0.36 with 4; 9,001: 0.97 with
        // 32, 0.88 with 8; beyond that the FP64 pipe is full and whole warps win:
        // 66,049 rays 2.6 ms with 32, 3.1 with 16)
        int per = 32;
        while (per > 4 && ia.rays / (per / 2) <= 8 * c->sm_count) per /= 2;
        k_im_march<<<(ia.rays + 2 * per - 1) / (2 * per), 64, 0, c->stream>>>(ia, per);
        if (dustmaps) k_im_dust_maps<<<dim3((ia.rays + 63) / 64, nlines), 64, 0, c->stream>>>(ia);
        const dim3 grid((ia.rays + IM_WARPS - 1) / IM_WARPS, nlines);
        for (int s0 = 0; stokes && s0 < slots; s0 += 4) switch (std::min(4, slots - s0)) {
            case 1: k_im_stokes<1><<<grid, 32 * IM_WARPS, 0, c->stream>>>(ia, s0); break;
            case 2: k_im_stokes<2><<<grid, 32 * IM_WARPS, 0, c->stream>>>(ia, s0); break;
            case 3: k_im_stokes<3><<<grid, 32 * IM_WARPS, 0, c->stream>>>(ia, s0); break;
            default: k_im_stokes<4><<<grid, 32 * IM_WARPS, 0, c->stream>>>(ia, s0);
            }
        if (stokes && tail)
            k_im_stokes_tail<<<dim3((ia.rays + 63) / 64, nlines, (tail + 3) / 4), 64, 0, c->stream>>>(ia, nch - tail);
    }
    timer_stop(c, T_IMWALK);
    PCHECK(c, cudaGetLastError());
    HostSpan spans[9];
    for (int q = 0; q < 8; q++) spans[q] = {dout[q], cube * sizeof(float)};
    spans[8] = {xy, 2 * (size_t)nrays * sizeof(double)};
    map_pages(spans, 9);   // while the kernels run
    for (int q = 0; q < 8; q++)
        if (dout[q])
            PCHECK(c, cudaMemcpyAsync(dout[q], ia.out[q], cube * sizeof(float), cudaMemcpyDeviceToHost, c->stream));
    std::vector<int> sth((size_t)nrays);
    std::vector<double> xyz_h;
    if (xy) {
        xyz_h.resize(3 * (size_t)N);
        PCHECK(c, cudaMemcpyAsync(xyz_h.data(), xyz_r.p, xyz_h.size() * sizeof(double), cudaMemcpyDeviceToHost,
                                  c->stream));
    }
    PCHECK(c, cudaMemcpyAsync(sth.data(), stat.p, sth.size() * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    PCHECK(c, cudaStreamSynchronize(c->stream));
    timer_collect(c, T_EMCOEF);
    timer_collect(c, T_IMWALK);
    if (status) std::copy(sth.begin(), sth.end(), status);
    if (xy)  // the rows of inc%02d-xy.dat (para_finish.f90:269-271)
        for (int n = 0; n < nrays; n++) {
            xy[2 * (size_t)n] = c->tx * xyz_h[3 * (size_t)n];
            xy[2 * (size_t)n + 1] = c->tx * xyz_h[3 * (size_t)n + 1];
        }
    for (size_t i = 0; i < sth.size(); i++)
        if (sth[i] == 1)
            return set_err(c, PORTAL_ERR_DEPTH, std::string("node_count > n_depth_rt for ") +
                                                    (mode ? "node " : "pixel ") + std::to_string(i + 1));
    return PORTAL_OK;
}

extern "C" int portal_image(portal_ctx *c, const double *pol_pops, int nlines, const int *l1,
                            const int *l2, double th_inc, double ph_az, int nvel, double dvel,
                            double v0, int im_pix, double im_size, double alpha, double dx,
                            int n_depth_rt, float *I, float *Q, float *U, float *tau, float *dust_I,
                            float *dust_Q, float *dust_U, float *dust_tau, int *status) {
    if (!c) return PORTAL_ERR_ARG;
    float *const out[8] = {I, Q, U, tau, dust_I, dust_Q, dust_U, dust_tau};
    return image_call(c, pol_pops, nlines, l1, l2, th_inc, ph_az, nvel, dvel, v0, 0, im_pix, im_size, alpha, dx,
                      n_depth_rt, nullptr, out, status);
}

extern "C" int portal_image_nodes(portal_ctx *c, const double *pol_pops, int nlines, const int *l1,
                                  const int *l2, double th_inc, double ph_az, int nvel, double dvel,
                                  double v0, double alpha, double dx, int n_depth_rt, double *xy, float *I,
                                  float *Q, float *U, float *tau, float *dust_I, float *dust_Q, float *dust_U,
                                  float *dust_tau, int *status) {
    if (!c) return PORTAL_ERR_ARG;
    float *const out[8] = {I, Q, U, tau, dust_I, dust_Q, dust_U, dust_tau};
    return image_call(c, pol_pops, nlines, l1, l2, th_inc, ph_az, nvel, dvel, v0, 1, 1, 0.5, alpha, dx,
                      n_depth_rt, xy, out, status);
}
