// Radiation field of every node: the inverse_rt loop of main_portal.x.
//
// Reference: main_para.f90:210-257 -> trace_node main_sub.f90:82-84 ->
// inverse_rt inverse_rt.f90:1-137, trace_out :139-214 (with
// check_neigh_fast miscellaneous.f90:1017-1076, pos_quadratic :1078-1098),
// ray_in :217-344, find_dir miscellaneous.f90:48-82.
//
// Kernels:
//   k_line_table   per (node, line): the opacity / emissivity factors that
//                  ray_in rebuilds for every (direction, channel, cell):
//                  A = kv * c/nu / (sqrt(pi) b) * tx*dx   (optical depth per
//                  trace step per unit Gaussian profile value), E the same
//                  for the emissivity, and the dust terms.  HBM-bound, tiny.
//   k_radiation_field  one warp per node (persistent warps, node queue) or,
//                  for small clouds, per range of rays, whose sums
//                  k_rf_finish adds per node; the directions of
//                  legendre_all in batches of 32 rays:
//                   (1) FP64 set-up, one lane per ray: the direction
//                       (find_dir's rotation in closed form) and the
//                       sphere-exit distance (pos_quadratic from the node,
//                       as trace_out's first step computes it);
//                   (2) the Voronoi walk, one lane per ray, 32 rays in
//                       flight per warp.  The photon is kept relative to the
//                       current node, so the face crossing
//                       t = (|e|^2/2 - e.r) / (e.d) is formed from the
//                       FP64-derived edge vectors without cancellation
//                       against absolute coordinates; the neighbour scan
//                       keeps check_neigh_fast's sequential tie rule.  The
//                       (cell, steps) list of each ray goes to a per-warp
//                       scratch slice in global memory (L2-resident);
//                   (3) the channel integration inward over the walk, lanes
//                       over channels, lines looped in registers, cell
//                       records staged in shared memory 32 cells at a time;
//                   (4) the profile-weighted channel sum (warp reduction)
//                       and the compensated accumulation of J^0_0, J^2_0
//                       over directions (fixed order: deterministic).
//                  On request it also splits J^0_0 = J_eff + L* S_line at
//                  the central cell: J_eff the field without the node's own
//                  line emission, L* = dJ^0_0/dS_line the diagonal of the
//                  Lambda operator (what the node's own cell contributes per
//                  unit source function) -- the inputs of the preconditioned
//                  SE of the accelerated Lambda iteration.
#include <cmath>
#include <cstdlib>

#include "rf_kernel.cuh"

using namespace portal;


namespace {

// upload per-line constants of the molecule into the context
int upload_lines(portal_ctx *c) {
    if (c->r_num > MAX_LINES)
        return set_err(c, PORTAL_ERR_ARG, "more than 64 radiative lines are not supported");
    std::vector<LineConst> h(c->r_num);
    std::vector<float> bb(c->r_num);
    for (int k = 0; k < c->r_num; k++) {
        int lo = c->r_trans[2 * k] - 1, up = c->r_trans[2 * k + 1] - 1;
        h[k].nu = c->nu[k];
        h[k].A = c->A[k];
        h[k].B = c->Bij[k];
        h[k].kd = c->kd_v[k];
        h[k].glo = 2.0 * c->j_lev[lo] + 1.0;
        h[k].gup = 2.0 * c->j_lev[up] + 1.0;
        // black_body(2.73, nu) miscellaneous.f90:263-285
        h[k].bb_cmb = 1.4744995e-50 * std::pow(c->nu[k], 3.0) *
                      std::pow(std::exp(4.79924e-11 / 2.73 * c->nu[k]) - 1.0, -1.0);
        h[k].lo = lo;
        h[k].up = up;
        bb[k] = (float)h[k].bb_cmb;
    }
    if (c->linebuf.reserve(sizeof(LineConst) * c->r_num) || c->bbcmb.reserve(c->r_num) ||
        c->bbstar.reserve(c->r_num))
        return set_err(c, PORTAL_ERR_NOMEM, "line constants");
    // star rays start from black_body(T_star) (inverse_rt.f90:113-115)
    std::vector<float> bs(c->r_num, 0.f);
    if (c->star_mode && c->T_star > 0.0)
        for (int k = 0; k < c->r_num; k++)
            bs[k] = (float)(1.4744995e-50 * std::pow(c->nu[k], 3.0) *
                            std::pow(std::exp(4.79924e-11 / c->T_star * c->nu[k]) - 1.0, -1.0));
    PCHECK(c, cudaMemcpyAsync(c->bbstar.p, bs.data(), sizeof(float) * c->r_num, cudaMemcpyHostToDevice,
                              c->stream));
    PCHECK(c, cudaMemcpyAsync(c->linebuf.p, h.data(), sizeof(LineConst) * c->r_num, cudaMemcpyHostToDevice,
                              c->stream));
    PCHECK(c, cudaMemcpyAsync(c->bbcmb.p, bb.data(), sizeof(float) * c->r_num, cudaMemcpyHostToDevice,
                              c->stream));
    return PORTAL_OK;
}

// Warps per block of the radiation-field kernel: 4, or PORTAL_RF_WARPS (4..8).
inline int rf_warps() {
    const char *e = getenv("PORTAL_RF_WARPS");
    const int v = e ? atoi(e) : 4;
    return (v >= 4 && v <= 8) ? v : 4;
}

// The widest line group: lines are split into the fewest groups of at most
// this many, of equal width.  PORTAL_RF_LINE_GROUP=3|4|5|10 overrides.
inline int max_line_group() {
    const char *e = getenv("PORTAL_RF_LINE_GROUP");
    if (e) {
        const int v = atoi(e);
        if (v == 3 || v == 4 || v == 5 || v == 10) return v;
    }
    return RF_MAX_GROUP;
}

// Items of rays: sums the rays' channel sums of every node in ray order (one
// warp per node, lane = line), as the whole-node items do.
__global__ void __launch_bounds__(128) k_rf_finish(RFArgs a, int split) {
    const int lane = threadIdx.x & 31;
    const int node = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
    if (node >= a.bulk) return;
    int st = 0, seg = 0;
    for (int r0 = 0; r0 < a.ndir; r0 += 32) {
        const int s = (r0 + lane < a.ndir) ? a.iseg[(size_t)node * a.ndir + r0 + lane] : 0;
        if (__any_sync(0xffffffffu, s < 0)) {   // the walks stop at these rays, as the whole-node loop does
            st = PORTAL_NODE_DEPTH;
            break;
        }
        seg += __reduce_add_sync(0xffffffffu, s);
    }
    const bool on = st == 0 && a.ab[node] > 0.0;
    const int L = a.L;
    const size_t ray0 = (size_t)node * a.ndir, plane = (size_t)a.bulk * a.ndir * L;
    float km = 0.f;
    for (int l = lane; l - lane < L; l += 32) {
        NodeSum s;
        const int line = min(l, L - 1);
        for (int r0 = 0; on && r0 < a.ndir; r0 += 32) {
            const int nr = min(32, a.ndir - r0);
            const double *dr = a.dirs + 6 * (size_t)(r0 + min(lane, nr - 1));
            const float w = (float)dr[4], w2 = (float)dr[5];
            const float *v = a.vray + (ray0 + r0) * L + line;
#pragma unroll 8
            for (int r = 0; r < nr; r++) {
                const float2 wt = make_float2(__shfl_sync(0xffffffffu, w, r), __shfl_sync(0xffffffffu, w2, r));
                s.add(wt, v[(size_t)r * L]);
                if (split) s.add_split(wt.x, v[plane + (size_t)r * L], v[2 * plane + (size_t)r * L]);
            }
            if (l == lane && lane < 6) {
                const float *v0 = a.vray + (ray0 + r0) * L;
                for (int r = 0; r < nr; r++)
                    km = moment_add(km, lane, (float)a.dirs[6 * (size_t)(r0 + r) + 4], v0[(size_t)r * L],
                                    a.dray[ray0 + r0 + r]);
            }
        }
        if (l >= L) continue;
        a.J0[(size_t)node * L + l] = on ? s.j0.value() : 0.0;
        a.J2[(size_t)node * L + l] = on ? s.j2.value() : 0.0;
        if (split) {
            a.JE[(size_t)node * L + l] = on ? s.je.value() : 0.0;
            a.LS[(size_t)node * L + l] = on ? s.ls.value() : 0.0;
        }
    }
    if (a.kmom && lane < 6) a.kmom[(size_t)lane * a.N + node] = on ? km : 0.f;
    if (lane == 0) {
        a.status[node] = st;
        if (st) atomicAdd(&a.counters[RF_FAILED], 1ULL);
        if (a.segs) a.segs[node] = seg;
        atomicAdd(&a.counters[1], (unsigned long long)seg);
    }
}

// Whether the items are rays, not nodes, and how many of 32, 16 and 8 rays:
// full walks first, shorter ones behind, so that the last items to finish do
// not leave the GPU idle; 16 rays a resident warp in sixteens, 4 in eights
// (measured from 0 to 32 and 2 to 16 of each: 1,024 points 0.148 ms (0.216
// with thirty-twos to the end), 4,096 points 1.69 (1.73), 6,001 with dust 4.85
// (5.10), 34 passes over 2,500 16.3 (16.3; in eights alone 20.2)).  No more
// than a node's rays, so that an item has two nodes at most.  From 16 nodes a
// resident warp on the nodes themselves balance.
bool ray_items(RFArgs &a, bool split, long long resident) {
    if (a.bulk >= 16 * resident || a.ndir <= 8) return false;
    const long long rays = (long long)a.bulk * a.ndir;
    if ((double)rays * (a.L * (split ? 3 : 1) * 4 + 20) > 2e9) return false;   // scratch limit
    const long long eights = std::min(rays, 4 * resident), sixteens = std::min(rays - eights, 16 * resident);
    a.items32 = a.ndir >= 32 ? (int)((rays - eights - sixteens) / 32) : 0;
    a.items16 = a.ndir >= 16 ? (int)((rays - eights - 32LL * a.items32) / 16) : 0;
    return true;
}

bool reserve_ray_items(portal_ctx *c, size_t rays, int values) {
    if (!c->vray.reserve(rays * values) && !c->dray.reserve(rays) && !c->iseg.reserve(rays)) return true;
    c->release_ray_items();
    return false;
}

template <bool FLAT>
const void *rf_kernel(const RFShape &sh, bool dust, bool split) {
    const int slots = sh.nslot == 1 ? 1 : sh.nslot % 2 == 0 ? 2 : 0;
    return dust         ? rf_kernel_dust<FLAT>(sh.nlg, slots)
           : slots == 1 ? rf_kernel_one<FLAT>(sh.nlg, split)
           : slots == 0 ? rf_kernel_any<FLAT>(sh.nlg)
           : split      ? rf_kernel_even_split<FLAT>(sh.nlg)
                        : rf_kernel_even<FLAT>(sh.nlg);
}

int launch_rf(portal_ctx *c, RFArgs &a, int n_depth) {
    const bool dust = c->has_dust, split = a.JE != nullptr;
    const int rt = rf_remainder(a.nch, dust, a.L);
    const size_t table = (a.nch * sizeof(float2) + 15) & ~(size_t)15;
    RFShape sh = rf_shape(a.L, max_line_group(), a.nch, dust, rt, split);
    const void *kern = nullptr;
    int wpb = 0, nb = 0;
    size_t dyn = 0;
    auto set_up = [&](bool flat) -> int {
        sh = rf_shape(a.L, max_line_group(), a.nch, dust, rt, split, flat ? 2 : 1);
        kern = flat ? rf_kernel<true>(sh, dust, split) : rf_kernel<false>(sh, dust, split);
        wpb = rf_warps();
        while (wpb > 1 && table + (size_t)wpb * sh.bytes > 200 * 1024) wpb--;   // many lines and channels
        dyn = table + (size_t)wpb * sh.bytes;
        PCHECK(c, allow_dyn_smem(kern));
        PCHECK(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, 32 * wpb, dyn));
        if (nb < 1) nb = 1;
        // where the device cannot hold the walk scratch of all blocks: without
        // the rays' sums of a call before, then fewer blocks per SM
        while (c->walk.reserve((size_t)nb * c->sm_count * wpb * rf_walk_records(n_depth)) != cudaSuccess) {
            if (c->vray.p) c->release_ray_items();
            else if (--nb < 1) return set_err(c, PORTAL_ERR_NOMEM, "walk scratch allocation failed");
        }
        return PORTAL_OK;
    };
    // about the warps resident: what the registers (the kernel's launch bounds)
    // and shared memory leave room for
    const long long fit = std::max<long long>(1, (224LL * 1024) / (sh.bytes + (long long)table / 4));
    bool flat = ray_items(a, split, c->sm_count * std::min(fit, sh.nlg <= 4 ? 24LL : 16LL));
    if (int rc = set_up(flat)) return rc;
    if (flat && !reserve_ray_items(c, (size_t)a.bulk * a.ndir, a.L * (split ? 3 : 1))) {
        flat = false;   // whole nodes need no rays' sums
        if (int rc = set_up(flat)) return rc;
    }
    const int grid = nb * c->sm_count;
    a.walk = c->walk.p;
    if (flat) {
        a.vray = c->vray.p; a.dray = c->dray.p; a.iseg = c->iseg.p;
    }
    timer_start(c, T_RF);
    RFBatch none{};
    void *args[] = {&a, &none, &sh};
    PCHECK(c, cudaLaunchKernel(kern, dim3(grid), dim3(32 * wpb), args, dyn, c->stream));
    if (flat && a.bulk > 0) k_rf_finish<<<(a.bulk + 3) / 4, 128, 0, c->stream>>>(a, split);
    timer_stop(c, T_RF);
    PCHECK(c, cudaGetLastError());
    return PORTAL_OK;
}

// Star mode: the node loop through the batched kernel with one model.  Its
// instantiations carry the per-node star ray sets (star_all); the
// single-model kernel leaves that code out, which keeps its registers for the
// integration (1 % faster on the benchmark sphere).
int launch_rf_star(portal_ctx *c, RFArgs &a, int n_depth) {
    RFBatch bw{};
    rf_batch_shape(&bw, &a.L, 1, a.nch, c->has_dust, max_line_group(), a.JE != nullptr);
    int nb = 0;
    if (rf_batch_blocks_per_sm(bw, c->has_dust, &nb))
        return set_err(c, PORTAL_ERR_CUDA, "star mode: occupancy query failed");
    if (nb < 1) nb = 1;
    const int grid = nb * c->sm_count;
    if (c->walk.reserve((size_t)grid * RF_BATCH_WARPS * rf_walk_records(n_depth)) != cudaSuccess)
        return set_err(c, PORTAL_ERR_NOMEM, "walk scratch allocation failed");
    if (c->star_items_n != c->bulk) c->star_items_n = -1;   // (a growing buffer loses its items)
    if (c->star_model.reserve(sizeof(RFArgs)) || c->star_items.reserve(c->bulk > 0 ? c->bulk : 1))
        return set_err(c, PORTAL_ERR_NOMEM, "star-mode work items");
    if (c->star_items_n != c->bulk) {
        std::vector<int2> it((size_t)c->bulk);
        for (int n = 0; n < c->bulk; n++) it[n] = make_int2(0, n);
        PCHECK(c, cudaMemcpyAsync(c->star_items.p, it.data(), it.size() * sizeof(int2), cudaMemcpyHostToDevice,
                                  c->stream));
        PCHECK(c, cudaStreamSynchronize(c->stream));
        c->star_items_n = c->bulk;
    }
    a.walk = c->walk.p;
    PCHECK(c, cudaMemcpyAsync(c->star_model.p, &a, sizeof(RFArgs), cudaMemcpyHostToDevice, c->stream));
    bw.models = reinterpret_cast<const RFArgs *>(c->star_model.p);
    bw.items = c->star_items.p;
    bw.n_items = c->bulk;
    bw.queue = c->counters.p;  // [0] next item, [1] segments, as the single-model kernel's counters
    bw.walk = c->walk.p;
    bw.n_depth = n_depth;
    bw.chq = a.chq;
    bw.chw = a.chw;
    timer_start(c, T_RF);
    const int rc = rf_batch_launch(c->stream, grid, c->has_dust, bw);
    timer_stop(c, T_RF);
    if (rc) return set_err(c, rc, std::string("star mode: ") + cudaGetErrorString(cudaGetLastError()));
    // the argument block is read by the kernel: keep it until the stream passes here
    PCHECK(c, cudaStreamSynchronize(c->stream));
    return PORTAL_OK;
}

int dispatch_rf(portal_ctx *c, RFArgs &a, int n_depth) {
    return a.star ? launch_rf_star(c, a, n_depth) : launch_rf(c, a, n_depth);
}

}  // namespace

namespace portal {

// float4 per node of the widest line table any launch asks for
static size_t ltab_width(int L) {
    int w = 0;
    for (int group : {3, 4, 5, RF_MAX_GROUP})
        for (bool dust : {false, true}) w = std::max(w, tab_shape(L, group, dust).width);
    return (size_t)w;
}

size_t rf_walk_records(int n_depth) { return (size_t)1024 * (size_t)((n_depth + 31) / 32); }

// Validates the call, uploads the molecule's line constants and the
// direction / channel tables, sizes the outputs and fills the kernel's
// argument block (walk scratch and counters are the launcher's).
int rf_prepare(portal_ctx *c, int nth, int nph, int nvel, const double *gvec, double dx, int n_depth,
               bool split, RFArgs *out) {
    if (!c->have_cloud || !c->have_mol) return set_err(c, PORTAL_ERR_STATE, "no cloud or molecule");
    if (c->nlev != (int)c->j_lev.size())
        return set_err(c, PORTAL_ERR_STATE, "cloud and molecule disagree on nlev");
    if (nth < 1 || nph < 1 || nvel < 1 || n_depth < 1 || !gvec || !(dx > 0.0) || 2 * nvel + 1 > 288)
        return set_err(c, PORTAL_ERR_ARG, "portal_radiation_field: bad nth/nph/nvel/n_depth/dx "
                                          "(at most 288 channels)");
    cudaSetDevice(c->device);
    const int L = c->r_num, N = c->N;
    const int nch = 2 * nvel + 1;
    // line constants, direction table (legendre_all) and channel tables: kept
    // until the molecule, the star, the angles or the channels change (the
    // quadrature's knots are found in long double, which this machine has in
    // software: 0.1 ms of each call)
    const bool new_lines = !c->lines_ready, new_dirs = nth != c->tab_nth || nph != c->tab_nph,
               new_ch = nvel != c->tab_nvel;
    if (new_lines) {
        if (int rc = upload_lines(c)) return rc;
    }
    std::vector<double> dt;
    std::vector<float> ct;
    int ndir = c->tab_ndir;
    if (new_dirs) {
        std::vector<double> xth;
        ndir = legendre_all(nth, nph, xth);
        dt.resize(6 * (size_t)ndir);
        for (int k = 0; k < ndir; k++) {
            double mu = xth[3 * k], ph = xth[3 * k + 1], w = xth[3 * k + 2];
            double th = std::acos(mu);
            double c_in = (3.0 * mu * mu - 1.0) / 2.0;
            dt[6 * k + 0] = std::cos(th);
            dt[6 * k + 1] = std::sin(th);
            dt[6 * k + 2] = std::cos(ph);
            dt[6 * k + 3] = std::sin(ph);
            dt[6 * k + 4] = w;
            dt[6 * k + 5] = w * c_in / std::sqrt(2.0);
        }
    }
    if (new_ch) {
        ct.resize(2 * (size_t)nch);
        const double spi = std::sqrt(std::acos(-1.0));
        for (int i = 0; i < nch; i++) {
            int nv = i - nvel;
            double q0 = 2.0 * nv / nvel;
            ct[i] = (float)q0;
            // phi_v0 * d_v = exp(-q0^2)/(sqrt(pi) b) * 2 b / nvel
            ct[nch + i] = (float)(std::exp(-q0 * q0) * 2.0 / (spi * nvel));
        }
    }
    // what is replaced is not kept: a growing buffer loses its contents, and a
    // call that fails further down must not leave them marked as held
    if (new_dirs) c->tab_nth = 0;
    if (new_ch) c->tab_nvel = 0;
    if (c->dirtab.reserve(6 * (size_t)ndir) || c->chtab.reserve(2 * (size_t)nch) ||
        c->ltab.reserve((size_t)N * ltab_width(L)) || c->J0.reserve((size_t)L * N) || c->J2.reserve((size_t)L * N) ||
        c->nodeseg.reserve((size_t)N) || c->frames.reserve(FRAME_N * (size_t)N) || c->kmom.reserve((size_t)6 * N))
        return set_err(c, PORTAL_ERR_NOMEM, "radiation-field buffers");
    if (split && (c->JE.reserve((size_t)L * N) || c->LS.reserve((size_t)L * N)))
        return set_err(c, PORTAL_ERR_NOMEM, "split-field buffers");
    if (new_dirs)
        PCHECK(c, cudaMemcpyAsync(c->dirtab.p, dt.data(), dt.size() * sizeof(double), cudaMemcpyHostToDevice,
                                  c->stream));
    if (new_ch)
        PCHECK(c, cudaMemcpyAsync(c->chtab.p, ct.data(), ct.size() * sizeof(float), cudaMemcpyHostToDevice,
                                  c->stream));
    // the host vectors go out of scope: the copies must have happened
    if (new_lines || new_dirs || new_ch) PCHECK(c, cudaStreamSynchronize(c->stream));
    c->tab_nth = nth; c->tab_nph = nph; c->tab_ndir = ndir; c->tab_nvel = nvel;
    c->lines_ready = true;
    RFArgs a;
    a.N = N; a.bulk = c->bulk; a.L = L; a.nvel = nvel; a.nch = nch; a.ndir = ndir; a.n_depth = n_depth;
    a.dx32 = (float)dx;
    a.pos = c->pos64.p; a.bvec = c->bvec64.p; a.ab = c->ab.p; a.cellv = c->cellv.p;
    a.wstart = c->wstart; a.whead = c->whead.p; a.wedge = c->wedge.p; a.wnext = c->wnext.p; a.ltab = c->ltab.p;
    a.dirs = c->dirtab.p; a.chq = c->chtab.p; a.chw = c->chtab.p + nch; a.bb = c->bbcmb.p;
    a.gx = gvec[0]; a.gy = gvec[1]; a.gz = gvec[2];
    a.ab = c->active_ab();
    a.star = c->star_mode; a.nth = nth; a.nph = nph;
    a.xs = c->X_star[0]; a.ys = c->X_star[1]; a.zs = c->X_star[2];
    a.Rs = c->star_mode ? c->R_star() : 0.0;
    a.bbs = c->bbstar.p;
    a.J0 = c->J0.p; a.J2 = c->J2.p; a.status = c->status.p; a.counters = c->counters.p;
    a.segs = c->nodeseg.p;
    a.kmom = c->kmom.p;
    a.JE = split ? c->JE.p : nullptr;
    a.LS = split ? c->LS.p : nullptr;
    a.walk = nullptr;
    a.frames = c->frames.p;
    a.items32 = a.items16 = 0;
    a.vray = nullptr; a.dray = nullptr; a.iseg = nullptr;
    // the line table's transfer step (main_para.f90:135 dx times r_max)
    c->rf_dxp = c->tx * dx;
    *out = a;
    return PORTAL_OK;
}

// The per-pass device work before the walk: zeroed outputs and counters, node
// frames and the line table from the current populations.  Stream-ordered only (capturable).
// max_group (0: the model's own launch) and dust: the launch the table is for.
int rf_pass(portal_ctx *c, const RFArgs &a, int max_group, bool dust, cudaStream_t s) {
    const int L = c->r_num, N = c->N;
    const long long tot = (long long)N * L;
    const int table_blocks = (int)((tot + 255) / 256);
    k_line_table<<<table_blocks + (std::max(N, 8) + 255) / 256, 256, 0, s>>>(
        N, L, c->rf_dxp, reinterpret_cast<const LineConst *>(c->linebuf.p), c->levp.p, c->nlev, c->b64.p,
        c->dustp.p, c->tdust.p, c->ltab.p, tab_shape(L, max_group ? max_group : max_line_group(), dust), a,
        table_blocks);
    PCHECK(c, cudaGetLastError());
    return PORTAL_OK;
}

// Enqueues the line table and the radiation field; J stays in c->J0/J2 (and
// the split field in c->JE/LS when `split`), the pass's counters in
// c->counters ([1] segments).
int enqueue_radiation_field(portal_ctx *c, int nth, int nph, int nvel, const double *gvec, double dx, int n_depth,
                            bool split) {
    RFArgs a;
    int rc = rf_prepare(c, nth, nph, nvel, gvec, dx, n_depth, split, &a);
    if (rc) return rc;
    c->j_valid = c->ali_valid = false;   // (the pass starts by clearing the field)
    timer_start(c, T_LINETAB);
    if ((rc = rf_pass(c, a, 0, c->has_dust, c->stream))) return rc;
    timer_stop(c, T_LINETAB);
    return dispatch_rf(c, a, n_depth);
}

// The error of a pass with failed nodes: a walk past n_depth or a star ray set
// past nth*nph is an error, as the reference stops there.
int failed_nodes(portal_ctx *c) {
    std::vector<int> st((size_t)c->N);
    PCHECK(c, cudaMemcpyAsync(st.data(), c->status.p, st.size() * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    PCHECK(c, cudaStreamSynchronize(c->stream));
    int nf = 0, first = -1, bits = 0;
    for (int i = 0; i < c->N; i++)
        if (st[i] & (PORTAL_NODE_DEPTH | PORTAL_NODE_STAR)) {
            if (first < 0) first = i;
            bits |= st[i];
            nf++;
        }
    if (!nf) return PORTAL_OK;
    return set_err(c, (bits & PORTAL_NODE_DEPTH) ? PORTAL_ERR_DEPTH : PORTAL_ERR_ARG,
                   std::string((bits & PORTAL_NODE_DEPTH) ? "node_count > n_depth" : "star rays > nth*nph") + " for " +
                       std::to_string(nf) + " node(s), the first node " + std::to_string(first + 1));
}

}  // namespace portal

namespace {

int radiation_field_call(portal_ctx *c, int nth, int nph, int nvel, const double *gvec, double dx,
                         int n_depth, double *J0, double *J2, double *JE, double *LS, bool split, int *status,
                         long long *n_segments) {
    if (!c) return PORTAL_ERR_ARG;
    timers_reset(c);
    const RayItems give_back(c);
    const size_t LN = (size_t)c->r_num * c->N;
    if (int rc = portal::enqueue_radiation_field(c, nth, nph, nvel, gvec, dx, n_depth, split)) return rc;
    const HostSpan out[4] = {{J0, LN * sizeof(double)}, {J2, LN * sizeof(double)}, {JE, LN * sizeof(double)},
                             {LS, LN * sizeof(double)}};
    map_pages(out, 4);   // the caller's result arrays, while the kernel runs
    // every copy behind the kernels, one wait for all
    if (J0) PCHECK(c, cudaMemcpyAsync(J0, c->J0.p, LN * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    if (J2) PCHECK(c, cudaMemcpyAsync(J2, c->J2.p, LN * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    if (split && JE) PCHECK(c, cudaMemcpyAsync(JE, c->JE.p, LN * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    if (split && LS) PCHECK(c, cudaMemcpyAsync(LS, c->LS.p, LN * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    std::vector<int> st_host;
    int *st = status;
    if (!st) { st_host.resize(c->N); st = st_host.data(); }
    PCHECK(c, cudaMemcpyAsync(st, c->status.p, (size_t)c->N * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    unsigned long long cnt[2];
    PCHECK(c, cudaMemcpyAsync(cnt, c->counters.p, sizeof cnt, cudaMemcpyDeviceToHost, c->stream));
    PCHECK(c, cudaStreamSynchronize(c->stream));
    timer_collect(c, T_LINETAB);
    timer_collect(c, T_RF);
    if (n_segments) *n_segments = (long long)cnt[1];
    c->j_valid = true;
    c->ali_valid = split;
    for (int i = 0; i < c->N; i++) {
        if (st[i] & PORTAL_NODE_DEPTH)
            return set_err(c, PORTAL_ERR_DEPTH, "node_count > n_depth for node " + std::to_string(i + 1));
        if (st[i] & PORTAL_NODE_STAR)
            return set_err(c, PORTAL_ERR_ARG, "star mode: the star's rays exceed nth*nph for node " +
                                                  std::to_string(i + 1) + " (a node this close to the star "
                                                                          "stops the reference too)");
    }
    return PORTAL_OK;
}

}  // namespace

extern "C" int portal_radiation_field(portal_ctx *c, int nth, int nph, int nvel, const double *gvec,
                                      double dx, int n_depth, double *J0, double *J2, int *status,
                                      long long *n_segments) {
    return radiation_field_call(c, nth, nph, nvel, gvec, dx, n_depth, J0, J2, nullptr, nullptr, false, status,
                                n_segments);
}

extern "C" int portal_radiation_field_split(portal_ctx *c, int nth, int nph, int nvel, const double *gvec,
                                            double dx, int n_depth, double *J0, double *J2, double *J_eff,
                                            double *L_star, int *status, long long *n_segments) {
    return radiation_field_call(c, nth, nph, nvel, gvec, dx, n_depth, J0, J2, J_eff, L_star, true, status,
                                n_segments);
}

extern "C" int portal_node_segments(portal_ctx *c, int *segments) {
    if (!c || !segments) return PORTAL_ERR_ARG;
    if (!c->j_valid || !c->nodeseg.p) return set_err(c, PORTAL_ERR_STATE, "no radiation field computed");
    PCHECK(c, cudaMemcpyAsync(segments, c->nodeseg.p, (size_t)c->N * sizeof(int), cudaMemcpyDeviceToHost,
                              c->stream));
    PCHECK(c, cudaStreamSynchronize(c->stream));
    return PORTAL_OK;
}

extern "C" int portal_field_moments(portal_ctx *c, double *moments) {
    if (!c || !moments) return PORTAL_ERR_ARG;
    if (!c->j_valid || !c->kmom.p) return set_err(c, PORTAL_ERR_STATE, "no radiation field computed");
    std::vector<float> h((size_t)6 * c->N);
    PCHECK(c, cudaMemcpyAsync(h.data(), c->kmom.p, h.size() * sizeof(float), cudaMemcpyDeviceToHost, c->stream));
    PCHECK(c, cudaStreamSynchronize(c->stream));
    for (int n = 0; n < c->N; n++)
        for (int k = 0; k < 6; k++) moments[6 * (size_t)n + k] = (double)h[(size_t)k * c->N + n];
    return PORTAL_OK;
}
