// FP64 engine kernels.
//
// Same pipeline as the FP32 engine, but with absolute FP64 positions in [0, L) and every
// floating-point operation in the order the reference's FP64 half-step engine performs it
// (naive_dpd_engine_half_step.hpp, dpd_maths_core_half_step.hpp).  This translation unit is
// compiled with -fmad=false, so no multiply-add is fused; with the canonical cell order
// (ascending bead id inside a cell) each bead's force is summed in the reference's order and
// the trajectory is bit-identical to the reference's.
//
// State per bead (sorted): pos = (x, y, z, hash as the low bits of w), vel = (v, 0),
// frc = (f, 0).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>

#include "../../include/pdpd_gpu.h"
#include "pdpd_cells.cuh"
#include "pdpd_walk.cuh"

namespace pdpd {
namespace {

constexpr int MAX_PAIR = 256;

struct WorldCache {
    WorldDev w;
    uint32_t world;
};

__device__ __forceinline__ uint32_t hash_of(const Vec4d &p)
{
    return (uint32_t)__double_as_longlong(p.w);
}

__device__ __forceinline__ void load_world(const KArgs &a, uint32_t world, WorldCache &wc,
                                           Vec2d *s_pair)
{
    if (wc.world != world) {
        __syncthreads();
        if (threadIdx.x == 0) {
            wc.w = a.worlds[world];
            wc.world = world;
        }
        __syncthreads();
        const uint32_t np = wc.w.n_types * wc.w.n_types;
        const Vec2d *pair = (const Vec2d *)a.pair;
        for (uint32_t i = threadIdx.x; i < np && i < MAX_PAIR; i += blockDim.x)
            s_pair[i] = pair[wc.w.param_base + i];
        __syncthreads();
    }
}

// update_pos (dpd_maths_core_half_step.hpp:22-49): x' = (x + v dt) + f (dt dt / 2), with the
// reference's single periodic wrap.  Returns the global cell of x'.  The comparisons are made
// on the bits (non-negative doubles order as their bits do): an FP64 comparison costs as much
// as an FP64 addition, which is what the force pass is bound by.
__device__ __forceinline__ uint32_t advance_position64(const WorldDev &w, double dt, double hdt2,
                                                       double x[3], const double v[3],
                                                       const double f[3], uint32_t &err)
{
    int c[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const double L = w.Ld[d];
        const long long Lb = __double_as_longlong(L);
        double xn = x[d] + v[d] * dt + f[d] * hdt2;
        const long long b = __double_as_longlong(xn);
        if (b < 0 && (b << 1) != 0) {  // xn < 0 (or a NaN, caught below)
            xn += L;
            if (xn == L) xn = 0;
        } else if (b >= Lb) {  // xn >= L (or a NaN)
            xn -= L;
        }
        const long long e = __double_as_longlong(xn);
        if (!((e >= 0 && e < Lb) || (e << 1) == 0)) {  // moved more than a box, or non-finite
            err |= ERR_OUT_OF_BOX;
            xn = 0.0;
        }
        x[d] = xn;
        c[d] = (int)xn;  // = floor: xn >= 0
    }
    return w.cell_base + ((uint32_t)c[0] * (uint32_t)w.L[1] + (uint32_t)c[1]) * (uint32_t)w.L[2] +
           (uint32_t)c[2];
}

// calc_distance_from_to (naive_dpd_engine_half_step.hpp:198-209).
__device__ __forceinline__ void distance_from_to(const WorldDev &w, const double base[3],
                                                 const double other[3], double res[3])
{
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const double len = (double)w.L[i];
        const double dx = other[i] - base[i];
        const int wrap_neg = dx > len * 0.5;
        const int wrap_pos = dx < -len * 0.5;
        res[i] = dx + (double)(wrap_pos - wrap_neg) * len;
    }
}

__device__ __forceinline__ void load_x(const Vec4d *__restrict__ pos, uint32_t slot, double x[3])
{
    const Vec4d p = pos[slot];
    x[0] = p.x;
    x[1] = p.y;
    x[2] = p.z;
}

// Bond forces, one thread per Hookean bond or angle bond, from the positions pos of the beads'
// slots (slot_of_id): each evaluated once, exactly as
// update_hookean_bond / update_angle_bond (naive_dpd_engine_half_step.hpp:426-483) and
// calc_angle_force (dpd_maths_core_half_step.hpp:177-229) do, and stored with the sign it is
// added with at the CSR row of each of its beads (row_of): the force kernel adds a bead's rows in
// order after the pair forces (F - t == F + (-t) in IEEE arithmetic), which is the reference's
// order of additions to the bead's force.  (A thread per bead, evaluating each of its terms,
// took 76 us for the 64^3 box: 2.4 times the terms, and warps that mix both kinds.)
__device__ __forceinline__ void store_term64(const KArgs &a, uint32_t row, double x, double y, double z)
{
    ((Vec4d *)a.bterm)[a.row_of[row]] = Vec4d{x, y, z, 0.0};
}

__device__ __forceinline__ void hookean64(const KArgs &a, const Vec4d *pos, const WorldDev &w, uint32_t k,
                                          uint32_t head, uint32_t tail, uint32_t &err)
{
    const Vec4d prm = ((const Vec4d *)a.bond_params)[k];
    double xh[3], xt[3], dx[3];
    load_x(pos, a.slot_of_id[head], xh);
    load_x(pos, a.slot_of_id[tail], xt);
    distance_from_to(w, xh, xt, dx);
    const double dr = sqrt(dx[0] * dx[0] + dx[1] * dx[1] + dx[2] * dx[2]);
    if (dr > 2.0) err |= ERR_BOND_SNAPPED;
    const double dr0 = prm.y - dr;
    const double hookean_force = prm.x * dr0;
    const double s = hookean_force / dr;
    const double f[3] = {dx[0] * s, dx[1] * s, dx[2] * s};
    store_term64(a, 2 * k, -f[0], -f[1], -f[2]);
    store_term64(a, 2 * k + 1, f[0], f[1], f[2]);
}

__device__ __forceinline__ void angle64(const KArgs &a, const Vec4d *pos, const WorldDev &w, uint32_t g,
                                        const uint32_t *hmt)
{
    const Vec4d prm = ((const Vec4d *)a.bond_params)[a.n_bonds + g];
    double xh[3], xm[3], xt[3];
    load_x(pos, a.slot_of_id[hmt[0]], xh);
    load_x(pos, a.slot_of_id[hmt[1]], xm);
    load_x(pos, a.slot_of_id[hmt[2]], xt);
    double first[3], second[3];
    distance_from_to(w, xh, xm, first);
    distance_from_to(w, xm, xt, second);
    const double r01 = sqrt(first[0] * first[0] + first[1] * first[1] + first[2] * first[2]);
    const double r12 = sqrt(second[0] * second[0] + second[1] * second[1] + second[2] * second[2]);
    const double kappa = prm.x, cos_theta0 = prm.y, sin_theta0 = prm.z;
    double hf[3] = {0, 0, 0}, tf[3] = {0, 0, 0}, mf[3] = {0, 0, 0};
    const double mag_product = r01 * r12;
    if (mag_product > 0.0001) {
        const double b1_mag_sq = r01 * r01;
        const double b2_mag_sq = r12 * r12;
        const double b1_dot_b2 = first[0] * second[0] + first[1] * second[1] + first[2] * second[2];
        const double p1 = b1_dot_b2 / b1_mag_sq;
        const double p2 = b1_dot_b2 / b2_mag_sq;
        const double cos_phi_sq = p1 * p2;
        double force_mag = kappa / mag_product;
        if (fabs(b1_dot_b2) > 0.000001 && sin_theta0 > 0) {
            const double inv_prefactor = 1.0 / sqrt(1.0 / cos_phi_sq - 1.0);
            force_mag = force_mag * (cos_theta0 - sin_theta0 * inv_prefactor);
        }
#pragma unroll
        for (int d = 0; d < 3; d++) {
            hf[d] = (first[d] * p1 - second[d]) * force_mag;
            tf[d] = (first[d] - second[d] * p2) * force_mag;
            mf[d] = -(hf[d] + tf[d]);
        }
    }
    const uint32_t row = 2 * a.n_bonds + 3 * g;
    store_term64(a, row, hf[0], hf[1], hf[2]);
    store_term64(a, row + 1, mf[0], mf[1], mf[2]);
    store_term64(a, row + 2, tf[0], tf[1], tf[2]);
}

constexpr int LIST_MAX = 32;

// make_relative_cell_pos (naive_dpd_engine_half_step.hpp:181-196) for one direction:
// neighbour cell and the periodic shift of its beads (+L, -L or +0.0: the values the
// reference's (is_right - is_left) * L takes, chosen without arithmetic).
__device__ __forceinline__ uint32_t neighbour64(const WorldDev &w, const int c[3], const int dir[3],
                                                const double Ld[3], double delta[3])
{
    int op[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const int raw = c[i] + dir[i];
        const int is_left = raw < 0;
        const int is_right = raw == w.L[i];
        op[i] = raw + (is_left - is_right) * w.L[i];
        delta[i] = is_right ? Ld[i] : (is_left ? -Ld[i] : 0.0);
    }
    return w.cell_base + ((uint32_t)op[0] * (uint32_t)w.L[1] + (uint32_t)op[1]) * (uint32_t)w.L[2] +
           (uint32_t)op[2];
}

// calc_force's terms of one in-range pair (dpd_maths_core_half_step.hpp:69-157, kappa = 0,
// r0 = 0.5), each operation in the reference's order: the force pass adds e * scaled, and the
// pair log (k_pair_log64) records the terms the reference's ForceLogging logs.
struct PairTerms64 {
    double e[3], wr, sqrt_gammap, u, con, diss, rand_scale, rand, scaled;
};

__device__ __forceinline__ PairTerms64 pair_terms64(double dx0, double dx1, double dx2, double dr,
                                                    const Vec2d pp, const Vec4d &vh, const Vec4d &vj,
                                                    uint32_t hh, uint32_t hj, uint32_t th_lo,
                                                    uint32_t th_hi, double scale_inv_sqrt_dt)
{
    PairTerms64 q;
    const double inv_dr = 1.0 / dr;
    const double dv0 = vh.x - vj.x, dv1 = vh.y - vj.y, dv2 = vh.z - vj.z;
    q.wr = 1.0 - dr;
    q.con = pp.x * q.wr;
    q.e[0] = dx0 * inv_dr;
    q.e[1] = dx1 * inv_dr;
    q.e[2] = dx2 * inv_dr;
    const double rdotv = q.e[0] * dv0 + q.e[1] * dv1 + q.e[2] * dv2;
    q.sqrt_gammap = pp.y * q.wr;
    q.diss = -q.sqrt_gammap * q.sqrt_gammap * rdotv;
    q.u = (double)hash_u(th_lo, th_hi, hh, hj);
    q.rand_scale = q.sqrt_gammap * scale_inv_sqrt_dt;
    q.rand = q.rand_scale * q.u;
    // (the reference also adds kappa (r0 - dr) with kappa = 0: a zero, which changes no sum)
    q.scaled = q.con + q.diss + q.rand;
    return q;
}

// Phase 2: the reference's pair filter and calc_force (dpd_maths_core_half_step.hpp:69-157,
// kappa = 0, r0 = 0.5) for the listed candidates, in list order, each operation in the
// reference's order.  The list holds every neighbour that can be in range (the walk's
// prefilter is conservative); the exact FP64 test here keeps dr2 < 1 and dr2 >= 1e-18
// (naive_dpd_engine_half_step.hpp:404-411), so the terms added are the reference's.
__device__ __forceinline__ void list_forces64(const Vec4d *__restrict__ pos,
                                              const Vec4d *__restrict__ vel,
                                              const uint32_t *__restrict__ s_j,
                                              const uint8_t *__restrict__ s_dir, int col, int n,
                                              const WorldDev &w, const int c[3], const double Ld[3],
                                              const double xh[3], const Vec4d &vh, uint32_t hh,
                                              uint32_t ti, const Vec2d *__restrict__ pair,
                                              const Vec2d *__restrict__ cp, uint32_t hc,
                                              const uint32_t *__restrict__ cellg,
                                              uint32_t th_lo, uint32_t th_hi,
                                              double scale_inv_sqrt_dt, double F[3])
{
    const uint32_t nt = w.n_types;
    const uint32_t n2 = nt * nt;
    const double min2 = (double)min_dist_sqr_f();
    for (int k = 0; k < n; k++) {
        const uint32_t j = s_j[k * TILE_BEADS + col];
        const uint32_t d = s_dir[k * TILE_BEADS + col];
        const int dir[3] = {(int)(d & 3u) - 1, (int)((d >> 2) & 3u) - 1, (int)((d >> 4) & 3u) - 1};
        double delta[3];
        neighbour64(w, c, dir, Ld, delta);
        const Vec4d pj = pos[j];
        const double obx = pj.x + delta[0], oby = pj.y + delta[1], obz = pj.z + delta[2];
        const double dx0 = xh[0] - obx, dx1 = xh[1] - oby, dx2 = xh[2] - obz;
        const double dr2 = dx0 * dx0 + dx1 * dx1 + dx2 * dx2;
        if (dr2 >= 1 || dr2 < min2) continue;
        const Vec4d vj = vel[j];
        const double dr = sqrt(dr2);
        const uint32_t hj = hash_of(pj);
        const uint32_t pk = ti * nt + min(hj >> 28, nt - 1u);
        Vec2d pp = pair[pk];
        if (cp) {  // spatial strengths: mean of the two beads' cell values (half_merge.hpp:570-583)
            const Vec2d h = cp[(size_t)hc * n2 + pk], o = cp[(size_t)(cellg[j] - w.cell_base) * n2 + pk];
            pp.x = (h.x + o.x) * 0.5;
            pp.y = (h.y + o.y) * 0.5;
        }
        const PairTerms64 q = pair_terms64(dx0, dx1, dx2, dr, pp, vh, vj, hh, hj, th_lo, th_hi, scale_inv_sqrt_dt);
        F[0] = F[0] + q.e[0] * q.scaled;
        F[1] = F[1] + q.e[1] * q.scaled;
        F[2] = F[2] + q.e[2] * q.scaled;
    }
}

// The home bead's data the list evaluation needs.
struct Home64 {
    double x[3];
    Vec4d v;
    uint32_t hash, ti, hc;
    int c[3];
};

__device__ __forceinline__ Home64 home64(const KArgs &a, const WorldDev &w, uint32_t s)
{
    Home64 h;
    const Vec4d p = ((const Vec4d *)a.posA)[s];
    h.x[0] = p.x;
    h.x[1] = p.y;
    h.x[2] = p.z;
    h.v = ((const Vec4d *)a.velA)[s];
    h.hash = hash_of(p);
    h.ti = min(h.hash >> 28, w.n_types - 1u);
    h.hc = a.cellg[s] - w.cell_base;
    decode_cell(h.hc, w.L, h.c[0], h.c[1], h.c[2]);
    return h;
}

__device__ __forceinline__ void eval_list64(const KArgs &a, const WorldDev &w, const Vec2d *s_pair,
                                            const uint32_t *s_j, const uint8_t *s_dir, int col, int n,
                                            const Home64 &h, uint32_t th_lo, uint32_t th_hi, double F[3])
{
    const double Ld[3] = {(double)w.L[0], (double)w.L[1], (double)w.L[2]};
    const Vec2d *cp = w.spatial ? (const Vec2d *)a.cellpair + w.cellpair_base : nullptr;
    list_forces64((const Vec4d *)a.posA, (const Vec4d *)a.velA, s_j, s_dir, col, n, w, h.c, Ld, h.x, h.v,
                  h.hash, h.ti, s_pair, cp, h.hc, a.cellg, th_lo, th_hi, w.scale_inv_sqrt_dt, F);
}

// The neighbour walk of one bead: for each of the 27 directions in (-1..1)^3 order, for each
// bead of that cell in id order (the reference's update_cell_forces order,
// naive_dpd_engine_half_step.hpp:358-424), candidates are appended to the bead's list
// (column threadIdx.x); a full list is evaluated into F on the spot.  Returns the entries
// left in the list.
//
// The walk itself does no FP64 arithmetic (the GPU's FP64 pipe is the kernel's bound): it
// tests the beads' FP32 cell offsets (posf, x - floor(x) rounded to FP32, error <= 2^-25)
// against a squared distance of 1.0001, and list_forces64 applies the exact FP64 test.  The
// FP32 separation of two offsets differs from the exact one by < 3e-7 per axis, so its
// square differs by < 4e-6 for pairs in range: no neighbour with dr2 < 1 is dropped, and the
// list's in-range entries, in order, are the reference's.  Rows and cells whose nearest face
// is >= 1.0001 away (FP32 gaps of the same offsets) hold no neighbour in range.
__device__ __forceinline__ int walk64(const KArgs &a, const WorldDev &w, const Vec2d *s_pair,
                                      uint32_t *s_j, uint8_t *s_dir, int cap, uint32_t th_lo,
                                      uint32_t th_hi, const Home64 &h, const float4 oh, double F[3])
{
    const float4 *__restrict__ posf = a.posf;
    const uint32_t *__restrict__ start = a.start;
    const float PRUNE = 1.0001f;
    int n = 0;
    int dir[3];
    for (dir[0] = -1; dir[0] <= 1; dir[0]++) {
        const float gx = slab_gap(oh.x, dir[0]);
        const float ax = oh.x - (float)dir[0];
        for (dir[1] = -1; dir[1] <= 1; dir[1]++) {
            const float gy = slab_gap(oh.y, dir[1]);
            const float gxy = gx * gx + gy * gy;
            if (gxy >= PRUNE) continue;
            const float ay = oh.y - (float)dir[1];
            for (dir[2] = -1; dir[2] <= 1; dir[2]++) {
                const float gz = slab_gap(oh.z, dir[2]);
                if (gxy + gz * gz >= PRUNE) continue;
                const float az = oh.z - (float)dir[2];
                int op[3];
#pragma unroll
                for (int i = 0; i < 3; i++) op[i] = wrap_index(h.c[i] + dir[i], w.L[i]);
                const uint32_t nc = w.cell_base + ((uint32_t)op[0] * (uint32_t)w.L[1] + (uint32_t)op[1]) * (uint32_t)w.L[2] + (uint32_t)op[2];
                const uint32_t j1 = start[nc + 1];
                const uint8_t dpk = (uint8_t)((dir[0] + 1) | ((dir[1] + 1) << 2) | ((dir[2] + 1) << 4));
                for (uint32_t j = start[nc]; j < j1; j++) {
                    const float4 q = posf[j];
                    const float ex = ax - q.x, ey = ay - q.y, ez = az - q.z;
                    if (ex * ex + ey * ey + ez * ez >= PRUNE) continue;
                    if (n == cap) {
                        eval_list64(a, w, s_pair, s_j, s_dir, threadIdx.x, n, h, th_lo, th_hi, F);
                        n = 0;
                    }
                    s_j[n * TILE_BEADS + threadIdx.x] = j;
                    s_dir[n * TILE_BEADS + threadIdx.x] = dpk;
                    n++;
                }
            }
        }
    }
    return n;
}

// Pair log (pdpd_log_pair_terms): for each sorted slot whose bead is in the sorted id list
// sel, every in-range pair of the 27-direction walk in the reference's order
// (naive_dpd_engine_half_step.hpp:300-424), with calc_force's terms as the reference's
// ForceLogging records them (dpd_maths_core_half_step.hpp:131-153).  Count pass (out null):
// counts[k] = pairs of sel[k]; write pass: the records of sel[k] at out + offs[k].
__global__ void k_pair_log64(KArgs a, const uint32_t *__restrict__ sel, uint32_t n_sel,
                             const uint32_t *__restrict__ offs, uint32_t *__restrict__ counts,
                             PairLogRec *__restrict__ out)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= a.n_beads) return;
    const uint32_t id = a.ids[s];
    uint32_t lo = 0, hi = n_sel;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) / 2;
        if (sel[mid] < id) lo = mid + 1; else hi = mid;
    }
    if (lo == n_sel || sel[lo] != id) return;
    const uint32_t k = lo;
    uint32_t wl = 0, wh = a.n_worlds;
    while (wh - wl > 1) {
        const uint32_t mid = (wl + wh) / 2;
        if (a.worlds[mid].bead_base <= id) wl = mid; else wh = mid;
    }
    const WorldDev &w = a.worlds[wl];
    const Home64 h = home64(a, w, s);
    const uint64_t th = t_hash((uint32_t)w.t, w.seed);
    const uint32_t th_lo = (uint32_t)th, th_hi = (uint32_t)(th >> 32);
    const double Ld[3] = {(double)w.L[0], (double)w.L[1], (double)w.L[2]};
    const Vec2d *pair = (const Vec2d *)a.pair + w.param_base;
    const Vec2d *cp = w.spatial ? (const Vec2d *)a.cellpair + w.cellpair_base : nullptr;
    const Vec4d *pos = (const Vec4d *)a.posA, *vel = (const Vec4d *)a.velA;
    const uint32_t nt = w.n_types, n2 = nt * nt;
    const double min2 = (double)min_dist_sqr_f();
    uint32_t n = 0;
    int dir[3];
    for (dir[0] = -1; dir[0] <= 1; dir[0]++)
        for (dir[1] = -1; dir[1] <= 1; dir[1]++)
            for (dir[2] = -1; dir[2] <= 1; dir[2]++) {
                double delta[3];
                const uint32_t nc = neighbour64(w, h.c, dir, Ld, delta);
                for (uint32_t j = a.start[nc]; j < a.start[nc + 1]; j++) {
                    const Vec4d pj = pos[j];
                    const double obx = pj.x + delta[0], oby = pj.y + delta[1], obz = pj.z + delta[2];
                    const double dx0 = h.x[0] - obx, dx1 = h.x[1] - oby, dx2 = h.x[2] - obz;
                    const double dr2 = dx0 * dx0 + dx1 * dx1 + dx2 * dx2;
                    if (dr2 >= 1 || dr2 < min2) continue;
                    if (out) {
                        const Vec4d vj = vel[j];
                        const double dr = sqrt(dr2);
                        const uint32_t hj = hash_of(pj);
                        const uint32_t pk = h.ti * nt + min(hj >> 28, nt - 1u);
                        Vec2d pp = pair[pk];
                        if (cp) {
                            const Vec2d hv = cp[(size_t)h.hc * n2 + pk], ov = cp[(size_t)(a.cellg[j] - w.cell_base) * n2 + pk];
                            pp.x = (hv.x + ov.x) * 0.5;
                            pp.y = (hv.y + ov.y) * 0.5;
                        }
                        const PairTerms64 q =
                            pair_terms64(dx0, dx1, dx2, dr, pp, h.v, vj, h.hash, hj, th_lo, th_hi, w.scale_inv_sqrt_dt);
                        PairLogRec &r = out[offs[k] + n];
                        r.t = w.t;
                        r.home_id = id;
                        r.other_id = a.ids[j];
                        r.home_hash = h.hash;
                        r.other_hash = hj;
                        r.dx[0] = dx0;
                        r.dx[1] = dx1;
                        r.dx[2] = dx2;
                        r.dr = dr;
                        r.inv_root_dt = w.scale_inv_sqrt_dt;
                        r.gammap = q.sqrt_gammap * q.sqrt_gammap;
                        r.rng = q.u;
                        r.con = q.con;
                        r.diss = q.diss;
                        r.rng_scale = q.rand_scale;
                        r.rand = q.rand;
                        const double dpd_force = q.con + q.diss + q.rand;
                        for (int d = 0; d < 3; d++) r.f[d] = q.e[d] * dpd_force;
                    }
                    n++;
                }
            }
    if (!out) counts[k] = n;
}

// Lists of a tile, re-dealt to threads by length (see k_force64).
struct Balance64 {
    uint32_t hist[LIST_MAX + 2];
    uint8_t n[TILE_BEADS];
    uint8_t perm[TILE_BEADS];
    double f[3][TILE_BEADS];
};

// Thread k's bond or angle bond.
__device__ __forceinline__ void bonds64(const KArgs &a, const Vec4d *pos, uint32_t k, bool angle)
{
    if (k >= (angle ? a.n_angles : a.n_bonds)) return;
    const uint32_t *ids = angle ? a.bond_list + 2 * (size_t)a.n_bonds + 3 * (size_t)k : a.bond_list + 2 * (size_t)k;
    // (only polymer beads have bond forces, and their slots kept by id)
    if ((a.hash[ids[0]] | a.hash[ids[1]] | (angle ? a.hash[ids[2]] : 0u)) & (1u << 27)) return;
    const uint32_t id = ids[0];
    uint32_t lo = 0, hi = a.n_worlds;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (a.worlds[mid].bead_base <= id) lo = mid; else hi = mid;
    }
    const WorldDev &w = a.worlds[lo];
    uint32_t err = 0;
    if (angle) angle64(a, pos, w, k, ids);
    else hookean64(a, pos, w, k, ids[0], ids[1], err);
    if (err) atomicOr(&a.worlds[lo].err, err);
}

// The cells' prefix sum (blocks [0, nb)) and, without pair lists (whose kernel takes them else),
// the Hookean bonds (the next bb) and the angle bonds, from the advanced, not yet re-sorted state
// (slot_of_id is that of the sorted state it came from).
template <bool ONE_PASS>
__global__ void __launch_bounds__(SCAN_THREADS) k_cells64(KArgs a, uint32_t nb, uint32_t bb, int tick)
{
    step_kernel_begin();
    if (blockIdx.x < nb) {
        scan_cells<ONE_PASS>(a, tick);
        return;
    }
    const bool angle = blockIdx.x - nb >= bb;
    bonds64(a, (const Vec4d *)a.posB, (blockIdx.x - nb - (angle ? bb : 0u)) * SCAN_THREADS + threadIdx.x, angle);
}

// Bonds, update_mom and either the final write or the next update_pos with its cell count, for
// one bead whose pair forces are in F.
template <int FINAL>
__device__ __forceinline__ void integrate64(const KArgs &a, const WorldDev &w, uint32_t world, uint32_t s,
                                            double F[3])
{
    const double dt = w.dt, hdt = w.hdt, hdt2 = w.hdt2;
    uint32_t err = 0;
    const Vec4d ph = ((const Vec4d *)a.posA)[s];
    const Vec4d vh = ((const Vec4d *)a.velA)[s];
    const uint32_t hh = hash_of(ph);
    double x[3] = {ph.x, ph.y, ph.z};
    const uint32_t id = a.ids[s];
    if (!(hh & (1u << 27))) {  // polymer bead: its bond terms, in CSR order
        const Vec4d *bt = (const Vec4d *)a.bterm;
#pragma unroll 1
        for (uint32_t r = a.bond_row[id]; r < a.bond_row[id + 1]; r++) {
            const Vec4d t = bt[r];
            F[0] = F[0] + t.x;
            F[1] = F[1] + t.y;
            F[2] = F[2] + t.z;
        }
    }
    // update_mom: v += f * half(dt); a stationary type's v and f are cleared instead
    // (naive_dpd_engine_half_merge.hpp:387-394), so the next update_pos leaves it in place
    double v[3] = {vh.x + F[0] * hdt, vh.y + F[1] * hdt, vh.z + F[2] * hdt};
    if ((w.stationary >> (hh >> 28)) & 1u) {
        v[0] = v[1] = v[2] = 0.0;
        F[0] = F[1] = F[2] = 0.0;
    }
    if (FINAL) {
        Vec4d vo = {v[0], v[1], v[2], id_word64(id)};
        Vec4d fo = {F[0], F[1], F[2], 0.0};
        ((Vec4d *)a.velB)[s] = vo;
        ((Vec4d *)a.frc)[s] = fo;
        if (!(isfinite(v[0]) && isfinite(v[1]) && isfinite(v[2]))) err |= ERR_NONFINITE;
    } else {
        const uint32_t key = advance_position64(w, dt, hdt2, x, v, F, err);
        cell_arrive(a, key, id);
        Vec4d po = {x[0], x[1], x[2], ph.w};
        Vec4d vo = {v[0] + F[0] * hdt, v[1] + F[1] * hdt, v[2] + F[2] * hdt, id_word64(id)};
        ((Vec4d *)a.posB)[s] = po;
        ((Vec4d *)a.velB)[s] = vo;
        a.key[s] = key;
    }
    if (err) atomicOr(&a.worlds[world].err, err);
}

#include "pdpd_fp64_pairs.cuh"

// Force pass without pair lists (pdpd_fp64_pairs.cuh), of a tile of TILE_BEADS sorted beads, one
// thread per bead:
//   1. each thread walks its bead's neighbours into its list;
//   2. the lists are counting-sorted by length and thread t evaluates list perm[t], so the
//      lanes of a warp evaluate lists of about the same length (the FP64 pipe executes an
//      instruction for the whole warp whatever its active lanes); every list is still
//      summed by one thread in its own order, so the result is the same;
//   3. each thread adds its bead's bond terms (bonds64) in CSR order, then update_mom and
//      either the final write or the next update_pos with its cell count.
template <int FINAL>
__global__ void __launch_bounds__(TILE_BEADS) k_force64(KArgs a)
{
    __shared__ Vec2d s_pair[MAX_PAIR];
    __shared__ uint32_t s_j[LIST_MAX * TILE_BEADS];
    __shared__ uint8_t s_dir[LIST_MAX * TILE_BEADS];
    __shared__ WorldCache wc;
    __shared__ Balance64 B;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) wc.world = 0xffffffffu;
    __syncthreads();
    const int cap = (a.list_capacity > 0 && a.list_capacity < LIST_MAX) ? a.list_capacity : LIST_MAX;
    for (uint32_t tile = blockIdx.x; tile < a.n_tiles; tile += gridDim.x) {
        const Tile tl = a.tiles[tile];
        load_world(a, tl.world, wc, s_pair);
        const WorldDev &w = wc.w;
        const uint32_t s = tl.slot_begin + tid;
        const bool act = s < tl.slot_end;
        const uint64_t th = t_hash((uint32_t)w.t, w.seed);
        const uint32_t th_lo = (uint32_t)th, th_hi = (uint32_t)(th >> 32);
        double F[3] = {0.0, 0.0, 0.0};
        int n = 0;
        if (act) {
            const Home64 h = home64(a, w, s);
            n = walk64(a, w, s_pair, s_j, s_dir, cap, th_lo, th_hi, h, a.posf[s], F);
        }
        if (tid < LIST_MAX + 2) B.hist[tid] = 0u;
        B.n[tid] = (uint8_t)n;
        B.f[0][tid] = F[0];
        B.f[1][tid] = F[1];
        B.f[2][tid] = F[2];
        __syncthreads();
        const uint32_t rank = atomicAdd(&B.hist[n], 1u);  // n <= LIST_MAX
        __syncthreads();
        if (warp == 0) {  // exclusive prefix of the LIST_MAX + 1 bins
            const uint32_t v = B.hist[lane];
            uint32_t inc = v;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, off);
                if (lane >= off) inc += y;
            }
            B.hist[lane] = inc - v;
            if (lane == 31) B.hist[32] = inc;
        }
        __syncthreads();
        B.perm[B.hist[n] + rank] = (uint8_t)tid;
        __syncthreads();
        {
            const int o = B.perm[tid];
            const int no = B.n[o];
            if (no > 0) {
                const Home64 h = home64(a, w, tl.slot_begin + (uint32_t)o);
                double G[3] = {B.f[0][o], B.f[1][o], B.f[2][o]};
                eval_list64(a, w, s_pair, s_j, s_dir, o, no, h, th_lo, th_hi, G);
                B.f[0][o] = G[0];
                B.f[1][o] = G[1];
                B.f[2][o] = G[2];
            }
        }
        __syncthreads();
        if (act) {
            F[0] = B.f[0][tid];
            F[1] = B.f[1][tid];
            F[2] = B.f[2][tid];
            integrate64<FINAL>(a, w, tl.world, s, F);
        }
        __syncthreads();  // the lists and B are reused by the next tile
    }
}

__global__ void __launch_bounds__(TILE_BEADS) k_begin64(KArgs a)
{
    step_kernel_begin();
    for (uint32_t tile = blockIdx.x; tile < a.n_tiles; tile += gridDim.x) {
        const Tile tl = a.tiles[tile];
        const uint32_t s = tl.slot_begin + threadIdx.x;
        if (s >= tl.slot_end) continue;
        const WorldDev &w = a.worlds[tl.world];
        const double dt = w.dt, hdt = w.hdt, hdt2 = w.hdt2;
        uint32_t err = 0;
        const Vec4d ph = ((const Vec4d *)a.posA)[s];
        const Vec4d vh = ((const Vec4d *)a.velA)[s];
        const Vec4d fh = ((const Vec4d *)a.frc)[s];
        double x[3] = {ph.x, ph.y, ph.z};
        // a stationary type is not moved and keeps its v (naive_dpd_engine_half_merge.hpp:329-333)
        const bool st = (w.stationary >> (hash_of(ph) >> 28)) & 1u;
        const double v[3] = {st ? 0.0 : vh.x, st ? 0.0 : vh.y, st ? 0.0 : vh.z};
        const double F[3] = {st ? 0.0 : fh.x, st ? 0.0 : fh.y, st ? 0.0 : fh.z};
        const uint32_t key = advance_position64(w, dt, hdt2, x, v, F, err);
        const uint32_t id = a.ids[s];
        cell_arrive(a, key, id);
        Vec4d po = {x[0], x[1], x[2], ph.w};
        Vec4d vo = st ? Vec4d{vh.x, vh.y, vh.z, id_word64(id)}
                      : Vec4d{v[0] + F[0] * hdt, v[1] + F[1] * hdt, v[2] + F[2] * hdt, id_word64(id)};
        ((Vec4d *)a.posB)[s] = po;
        ((Vec4d *)a.velB)[s] = vo;
        a.key[s] = key;
        if (err) atomicOr(&a.worlds[tl.world].err, err);
    }
}

__global__ void k_bin64(KArgs a, const uint32_t *__restrict__ hash_in)
{
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= a.n_beads) return;
    uint32_t lo = 0, hi = a.n_worlds;
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) / 2;
        if (a.worlds[mid].bead_base <= g) lo = mid; else hi = mid;
    }
    const WorldDev &w = a.worlds[lo];
    // rows of 9 doubles, or field-major blocks (x, v, f) of staging_n beads each
    const size_t stride = a.staging_fields ? 3 : 9, field = a.staging_fields ? 3 * (size_t)a.staging_n : 3;
    const double *st = a.staging + stride * g;
    int c[3];
    double x[3];
    uint32_t err = 0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        double xd = st[d];
        if (!(xd >= 0.0 && xd < (double)w.L[d])) {
            err |= ERR_OUT_OF_BOX;
            xd = 0.0;
        }
        x[d] = xd;
        c[d] = (int)floor(xd);
    }
    if (err) atomicOr(&a.worlds[lo].err, err);
    const uint32_t key = w.cell_base + ((uint32_t)c[0] * (uint32_t)w.L[1] + (uint32_t)c[1]) * (uint32_t)w.L[2] + (uint32_t)c[2];
    cell_arrive(a, key, g);
    Vec4d po = {x[0], x[1], x[2], __longlong_as_double((long long)hash_in[g])};
    Vec4d vo = {st[field], st[field + 1], st[field + 2], id_word64(g)};
    Vec4d fo = {st[2 * field], st[2 * field + 1], st[2 * field + 2], 0.0};
    ((Vec4d *)a.posB)[g] = po;
    ((Vec4d *)a.velB)[g] = vo;
    ((Vec4d *)a.frcB)[g] = fo;
    a.key[g] = key;
}

__global__ void k_finish64(KArgs a)
{
    step_kernel_begin();
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < a.n_beads) ((Vec4d *)a.velA)[s] = ((const Vec4d *)a.velB)[s];
    if (blockIdx.x == 0)
        for (uint32_t w = threadIdx.x; w < a.n_worlds; w += blockDim.x) a.worlds[w].t += 1;
}

}  // namespace

int launch_bin64(const KArgs &a, const uint32_t *hash_in, cudaStream_t s)
{
    if (a.n_beads == 0) return 0;
    k_bin64<<<(a.n_beads + 255) / 256, 256, 0, s>>>(a, hash_in);
    return 1;
}

int launch_begin64(const KArgs &a, cudaStream_t s)
{
    launch_step_kernel(k_begin64, (uint32_t)a.grid_blocks, TILE_BEADS, 0, s, a);
    return 1;
}

int launch_pair_log64(const KArgs &a, const uint32_t *sel, uint32_t n_sel, const uint32_t *offs,
                      uint32_t *counts, PairLogRec *out, cudaStream_t s)
{
    if (a.n_beads == 0 || n_sel == 0) return 0;
    k_pair_log64<<<(a.n_beads + 127) / 128, 128, 0, s>>>(a, sel, n_sel, offs, counts, out);
    return 1;
}

int launch_cells64(const KArgs &a, int tick, int bonds, cudaStream_t s)
{
    const uint32_t nb = scan_blocks(a.n_cells);
    const uint32_t bb = bonds && !a.list ? (a.n_bonds + SCAN_THREADS - 1) / SCAN_THREADS : 0u;
    const uint32_t ab = bonds && !a.list ? (a.n_angles + SCAN_THREADS - 1) / SCAN_THREADS : 0u;
    if (scan_one_pass(a.n_cells)) launch_step_kernel(k_cells64<true>, nb + bb + ab, SCAN_THREADS, 0, s, a, nb, bb, tick);
    else launch_step_kernel(k_cells64<false>, nb + bb + ab, SCAN_THREADS, 0, s, a, nb, bb, tick);
    return 1;
}

// Entries of the list kernel's queue: bricks, then chunks of bonds and of angles.
static uint32_t list64_work(const KArgs &a)
{
    return a.n_bricks + (a.n_bonds + BOND64_CHUNK - 1) / BOND64_CHUNK + (a.n_angles + BOND64_CHUNK - 1) / BOND64_CHUNK;
}

int launch_force64(const KArgs &a, int final_step, cudaStream_t s)
{
    if (a.list) {  // each pair once
        const List64Layout L = list64_layout(a.brick_hc_max, a.brick_maxb);
        const uint32_t bb = (a.n_bonds + BOND64_CHUNK - 1) / BOND64_CHUNK;
        const uint32_t work = list64_work(a);
        const uint32_t grid = std::max<uint32_t>(1, std::min<uint32_t>((uint32_t)a.brick_grid, work));
        // (a list that was not made is not read: the error reaches the caller)
        if (launch_step_kernel(a.brick_planes == 3 ? k_list64<3> : k_list64<1>, grid, LIST64_THREADS,
                               a.brick_smem, s, a, L,
                               bb, work) != cudaSuccess)
            return 0;
        const uint32_t pb = (a.pair_cap + PAIRS64_THREADS - 1) / PAIRS64_THREADS;
        launch_step_kernel(k_pairs64, std::min<uint32_t>((uint32_t)a.pair_blocks, std::max(1u, pb)), PAIRS64_THREADS, 0, s, a);
        const uint32_t parts = a.n_tiles * (TILE_BEADS / SUM64_BEADS);
        if (a.n_tiles == 0) return 2;
        if (final_step) launch_step_kernel(k_sum64<1>, parts, SUM64_THREADS, 0, s, a);
        else launch_step_kernel(k_sum64<0>, parts, SUM64_THREADS, 0, s, a);
        return 3;
    }
    // Launched when the kernel in front has finished: its few blocks then spread evenly over the SMs,
    // whose FP64 pipe they share (spread_smem; 24^3 of density 3, step, 264 us crowded, 184 spread by
    // shared memory, 173 so; 16^3 of density 8 7,070, 3,220, 3,170).
    if (final_step)
        k_force64<1><<<a.grid_blocks, TILE_BEADS, 0, s>>>(a);
    else
        k_force64<0><<<a.grid_blocks, TILE_BEADS, 0, s>>>(a);
    return 1;
}

// Largest staged-bead capacity of a k_list64 brick with two blocks per SM.
uint32_t list64_maxb_limit(uint32_t hc_max)
{
    int dev = 0, smem_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess)
        return 2046u;
    const int budget = smem_sm / 2 - 1024 - (int)list64_layout(hc_max, 0).bytes - 128;
    return (uint32_t)std::max(64, std::min((int)FULL_MAX_STAGED, budget / (int)LIST64_BEAD_BYTES)) & ~1u;
}

int list64_setup(const KArgs &a, int sm_count, int *grid, uint32_t *smem)
{
    const auto k = a.brick_planes == 3 ? k_list64<3> : k_list64<1>;
    const int bytes = (int)list64_layout(a.brick_hc_max, a.brick_maxb).bytes;
    int nb = 0;
    cudaError_t e = allow_dynamic_smem((const void *)k);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, LIST64_THREADS, bytes);
    if (e != cudaSuccess) return (int)e;
    if (nb < 1) return (int)cudaErrorInvalidConfiguration;
    *grid = nb * sm_count;
    *smem = std::max((uint32_t)bytes, spread_smem(std::min((uint32_t)*grid, list64_work(a)), nb, sm_count));
    return 0;
}

int launch_finish64(const KArgs &a, cudaStream_t s)
{
    launch_step_kernel(k_finish64, (a.n_beads + 255) / 256 + 1, 256, 0, s, a);
    return 1;
}

}  // namespace pdpd

// =======================================================================================
// Allocation-free stepping (pdpd_step_noalloc).
//
// Some callers cannot allocate device memory: code running while a CUDA stream is being
// captured into a graph (cudaMalloc is not a capturable operation), or a host framework
// that owns every device allocation through its own pool and forbids side allocations.
// For them, pdpd_step_noalloc advances one small bond-free world with the FP64 integrator
// on device arrays the caller owns, and keeps its own scratch -- the cell counts, cell
// starts, arrival ranks and the canonical bead order of the counting sort -- in the
// file-scope array g_noalloc_scratch below instead of allocating it.  Every GPU that loads
// the library holds this array (about 2 MB) until the process exits.  All calls share
// it: calls that overlap on the GPU (on different streams, or from different host threads
// without ordering) race on it and corrupt each other's cell lists.
//
// The arithmetic is the engine's FP64 path: update_pos, counting sort with beads in id
// order inside each cell, pair forces in the reference's direction order, update_mom,
// compiled without fused multiply-add -- so the result equals pdpd_run's bit for bit.
// =======================================================================================

namespace pdpd {
namespace {

constexpr uint32_t NA_MAX_BEADS = 65536;
constexpr uint32_t NA_MAX_CELLS = 32768;

struct NaScratch {
    uint32_t err;
    uint32_t cnt[NA_MAX_CELLS];
    uint32_t start[NA_MAX_CELLS + 1];
    uint2 keyrank[NA_MAX_BEADS];
    uint32_t tmp[NA_MAX_BEADS];
    float4 pos[NA_MAX_BEADS];  // in cell order: offset in the cell (x - floor(x) in FP32), bead id
};

struct NaParams {
    int32_t L[3];
    uint32_t n;
    uint32_t n_cells;
    uint32_t nt;
    double dt;
    double scale_inv_sqrt_dt;
    uint64_t seed;
    int64_t t;
    double pair[256][2];  // a_ij, sqrt(gamma_ij)
};

}  // namespace
}  // namespace pdpd

static __device__ __align__(256) unsigned char g_noalloc_scratch[sizeof(pdpd::NaScratch)];

namespace pdpd {
namespace {

// Before a call's first step: zeroes the cell counts (each step's scan leaves them zero) and the
// error word, so that a bead lost in any step of the call is reported at its end.
__global__ void k_na_clear(NaScratch *S, uint32_t n_cells)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n_cells) S->cnt[i] = 0u;
    if (i == 0) S->err = 0u;
}

// update_pos (dpd_maths_core_half_step.hpp:22-49) and the bead's new cell and arrival rank; before
// it (mom) the update_mom (:51-61) of the step before, the same bead's.
__global__ void k_na_update_pos(NaParams p, NaScratch *S, double *x, double *v, double *f, int mom)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const double dt = p.dt, hdt = dt * 0.5, hdt2 = (dt * dt) * 0.5;
    int c[3];
    for (int d = 0; d < 3; d++) {
        const double L = (double)p.L[d];
        const double fd = f[3 * i + d];
        double vd = v[3 * i + d];
        if (mom) vd = vd + fd * hdt;
        double xn = x[3 * i + d] + vd * dt + fd * hdt2;
        if (xn < 0) {
            xn += L;
            if (xn == L) xn = 0;
        } else if (xn >= L) {
            xn -= L;
        }
        if (!(xn >= 0.0 && xn < L)) {
            atomicOr(&S->err, (uint32_t)ERR_OUT_OF_BOX);
            xn = 0.0;
        }
        x[3 * i + d] = xn;
        c[d] = (int)floor(xn);
        v[3 * i + d] = vd + fd * hdt;
    }
    const uint32_t key = ((uint32_t)c[0] * (uint32_t)p.L[1] + (uint32_t)c[1]) * (uint32_t)p.L[2] + (uint32_t)c[2];
    const uint32_t rank = atomicAdd(&S->cnt[key], 1u);
    S->keyrank[i] = make_uint2(key, rank);
}

// Exclusive scan of the cell counts in one block of 1024 threads.
__global__ void __launch_bounds__(1024) k_na_scan(NaScratch *S, uint32_t n_cells, uint32_t n)
{
    __shared__ uint32_t wsum[32];
    const uint32_t per = (n_cells + 1023) / 1024;
    const uint32_t b = threadIdx.x * per, e = min(n_cells, b + per);
    uint32_t tsum = 0;
    for (uint32_t k = b; k < e; k++) tsum += S->cnt[k];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = tsum;
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= off) inc += y;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    uint32_t run = inc - tsum;
    for (int k = 0; k < warp; k++) run += wsum[k];
    for (uint32_t k = b; k < e; k++) {
        S->start[k] = run;
        run += S->cnt[k];
        S->cnt[k] = 0u;
    }
    if (threadIdx.x == 0) S->start[n_cells] = n;
}

__global__ void k_na_place(NaScratch *S, uint32_t n)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint2 kr = S->keyrank[i];
    S->tmp[S->start[kr.x] + kr.y] = i;
}

// Canonical cell order: beads of a cell in ascending id, as the reference's cell lists.
__global__ void k_na_canon(NaScratch *S, uint32_t n, const double *__restrict__ x)
{
    const uint32_t d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= n) return;
    const uint32_t i = S->tmp[d];
    const uint32_t key = S->keyrank[i].x;
    const uint32_t b = S->start[key], e = S->start[key + 1];
    uint32_t rank = 0;
    for (uint32_t k = b; k < e; k++) rank += S->tmp[k] < i ? 1u : 0u;
    float o[3];
    for (int k = 0; k < 3; k++) o[k] = (float)(x[3 * i + k] - floor(x[3 * i + k]));
    S->pos[b + rank] = make_float4(o[0], o[1], o[2], __uint_as_float(i));
}

// One pair's term on bead i from bead j in direction dir (0..26, z fastest) of cell c: the
// reference's separation, pair test and calc_force (naive_dpd_engine_half_step.hpp:181-196,
// 404-411, dpd_maths_core_half_step.hpp:69-157); false when out of range.
__device__ __forceinline__ bool na_pair(const NaParams &p, const double (*pair)[2], const double *__restrict__ x,
                                        const double *__restrict__ v, const uint32_t *__restrict__ hash, uint32_t i,
                                        uint32_t j, const int c[3], uint32_t dir, uint32_t th_lo, uint32_t th_hi,
                                        double t[3])
{
    const int d[3] = {(int)(dir / 9) - 1, (int)(dir / 3 % 3) - 1, (int)(dir % 3) - 1};
    double dx[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int raw = c[k] + d[k];
        const double delta = raw == p.L[k] ? (double)p.L[k] : (raw < 0 ? -(double)p.L[k] : 0.0);
        dx[k] = x[3 * i + k] - (x[3 * j + k] + delta);
    }
    const double dr2 = dx[0] * dx[0] + dx[1] * dx[1] + dx[2] * dx[2];
    if (dr2 >= 1 || dr2 < (double)min_dist_sqr_f()) return false;
    const Vec4d vi = {v[3 * i], v[3 * i + 1], v[3 * i + 2], 0.0}, vj = {v[3 * j], v[3 * j + 1], v[3 * j + 2], 0.0};
    const uint32_t hi = hash[i], hj = hash[j];
    const uint32_t pk = min(hi >> 28, p.nt - 1u) * p.nt + min(hj >> 28, p.nt - 1u);
    const PairTerms64 q = pair_terms64(dx[0], dx[1], dx[2], sqrt(dr2), Vec2d{pair[pk][0], pair[pk][1]}, vi, vj, hi, hj,
                                       th_lo, th_hi, p.scale_inv_sqrt_dt);
    for (int k = 0; k < 3; k++) t[k] = q.e[k] * q.scaled;
    return true;
}

// The cell of bead i.
__device__ __forceinline__ void na_cell_of(const NaParams &p, const NaScratch *S, uint32_t i, int c[3])
{
    const uint32_t key = S->keyrank[i].x, yz = (uint32_t)p.L[1] * (uint32_t)p.L[2];
    c[0] = (int)(key / yz);
    c[1] = (int)(key / (uint32_t)p.L[2] % (uint32_t)p.L[1]);
    c[2] = (int)(key % (uint32_t)p.L[2]);
}

// The cell in direction d of cell c.
__device__ __forceinline__ uint32_t na_neighbour(const NaParams &p, const int c[3], const int d[3])
{
    int op[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int raw = c[k] + d[k];
        op[k] = raw < 0 ? raw + p.L[k] : (raw == p.L[k] ? 0 : raw);
    }
    return ((uint32_t)op[0] * (uint32_t)p.L[1] + (uint32_t)op[1]) * (uint32_t)p.L[2] + (uint32_t)op[2];
}

// Visit the beads of direction (dx, dy, dz)'s cell that can be in range of the bead at offset o in
// cell c: the conservative FP32 test of the engine's lists (walk_global64).
template <class Visit>
__device__ __forceinline__ void na_cell(const NaParams &p, const NaScratch *S, const int c[3], const float4 o,
                                        uint32_t dir, Visit visit)
{
    const int d[3] = {(int)(dir / 9) - 1, (int)(dir / 3 % 3) - 1, (int)(dir % 3) - 1};
    const float gx = slab_gap(o.x, d[0]), gy = slab_gap(o.y, d[1]), gz = slab_gap(o.z, d[2]);
    if (gx * gx + gy * gy + gz * gz >= WALK_R2) return;
    const float ax = o.x - (float)d[0], ay = o.y - (float)d[1], az = o.z - (float)d[2];
    const uint32_t nc = na_neighbour(p, c, d), k1 = S->start[nc + 1];
    for (uint32_t k = S->start[nc]; k < k1; k++) {
        const float4 q = S->pos[k];
        const float ex = ax - q.x, ey = ay - q.y, ez = az - q.z;
        if (ex * ex + ey * ey + ez * ez < WALK_R2) visit(__float_as_uint(q.w));
    }
}

// Pair forces of NA_BEADS beads, consecutive in cell order.  Eight lanes of a bead walk its 9
// neighbour rows into lists (a row each, the first lane also the last row); the block's
// candidates are then evaluated flat, a thread each, and a thread per bead and axis adds a
// bead's terms in walk order, the reference's.  One thread per bead did all of this for itself,
// a serial chain of FP64 latencies on 48 blocks: 458 us for the 16^3 box against 34 us.
constexpr int NA_BEADS = 16, NA_LANES = 8, NA_THREADS = NA_BEADS * NA_LANES, NA_ROWS = 9;
constexpr uint32_t NA_ROW_CAP = 24, NA_TERMS = 512;

// A bead among so many that a row of its candidates does not fit: its eight lanes go through the
// cells together, in order, eight candidates at a time, and evaluate the candidates so far whenever
// the bead's list (the room of all its rows) is full.  (By the first lane alone, one pair after
// the other: 10^3 box of density 20, step 3,530 us against 490; 8^3 of density 60 14,700 and 3,640.)
// (It reads its bead anew, so that the kernel keeps nothing for it through its other work.)
__device__ __noinline__ void na_long_bead(const NaParams &p, const double (*pair)[2], const NaScratch *S,
                                          const double *__restrict__ x, const double *__restrict__ v,
                                          const uint32_t *__restrict__ hash, uint32_t h, uint32_t th_lo, uint32_t th_hi,
                                          uint32_t *list, double (*terms)[NA_TERMS], double *__restrict__ f)
{
    constexpr uint32_t CAP = NA_ROWS * NA_ROW_CAP, CHUNK = NA_TERMS / NA_BEADS;
    const int b = threadIdx.x / NA_LANES, sub = threadIdx.x % NA_LANES;
    const uint32_t shift = threadIdx.x & 31u & ~(NA_LANES - 1u), lanes = ((1u << NA_LANES) - 1u) << shift;
    const float4 o = S->pos[h];
    const uint32_t i = __float_as_uint(o.w);
    int c[3];
    na_cell_of(p, S, i, c);
    uint32_t n = 0;
    double F = 0.0;  // of axis `sub`
    auto evaluate = [&]() {
        __syncwarp(lanes);
        for (uint32_t e0 = 0; e0 < n; e0 += CHUNK) {
            const uint32_t m = min(n - e0, CHUNK);
            for (uint32_t e = sub; e < m; e += NA_LANES) {
                const uint32_t ent = list[e0 + e];
                double t[3] = {0.0, 0.0, 0.0};
                na_pair(p, pair, x, v, hash, i, ent & 0xffffu, c, ent >> 16, th_lo, th_hi, t);
                for (int k = 0; k < 3; k++) terms[k][b * CHUNK + e] = t[k];
            }
            __syncwarp(lanes);
            if (sub < 3)
                for (uint32_t e = 0; e < m; e++) F = F + terms[sub][b * CHUNK + e];
            __syncwarp(lanes);
        }
        n = 0;
    };
    for (uint32_t dir = 0; dir < 27; dir++) {
        const int d[3] = {(int)(dir / 9) - 1, (int)(dir / 3 % 3) - 1, (int)(dir % 3) - 1};
        const float gx = slab_gap(o.x, d[0]), gy = slab_gap(o.y, d[1]), gz = slab_gap(o.z, d[2]);
        if (gx * gx + gy * gy + gz * gz >= WALK_R2) continue;
        const uint32_t nc = na_neighbour(p, c, d), k1 = S->start[nc + 1];
        const float ax = o.x - (float)d[0], ay = o.y - (float)d[1], az = o.z - (float)d[2];
        for (uint32_t k0 = S->start[nc]; k0 < k1; k0 += NA_LANES) {
            uint32_t j = 0;
            bool in = false;
            if (k0 + sub < k1) {
                const float4 q = S->pos[k0 + sub];
                const float ex = ax - q.x, ey = ay - q.y, ez = az - q.z;
                j = __float_as_uint(q.w);
                in = ex * ex + ey * ey + ez * ez < WALK_R2 && !(j == i && dir == 13);
            }
            const uint32_t hits = __ballot_sync(lanes, in) >> shift;
            if (in) list[n + __popc(hits & ((1u << sub) - 1u))] = j | dir << 16;
            n += __popc(hits);
            if (n > CAP - NA_LANES) evaluate();
        }
    }
    evaluate();
    if (sub < 3) f[3 * i + sub] = F;
}

__global__ void __launch_bounds__(NA_THREADS) k_na_forces(const __grid_constant__ NaParams p, const NaScratch *S,
                                                          const double *__restrict__ x, const double *__restrict__ v,
                                                          double *__restrict__ f, const uint32_t *__restrict__ hash)
{
    __shared__ double s_pair[256][2];
    __shared__ double s_t[3][NA_TERMS];
    __shared__ uint32_t s_row[NA_BEADS * NA_ROWS][NA_ROW_CAP];  // bead, direction << 16
    __shared__ uint32_t s_pre[NA_BEADS * NA_ROWS + 1];          // entry counts, then their prefix
    __shared__ uint32_t s_id[NA_BEADS];
    __shared__ int s_c[NA_BEADS][3];
    __shared__ uint32_t s_long[NA_BEADS];  // a row of this bead does not fit
    const int tid = threadIdx.x, b = tid / NA_LANES, sub = tid % NA_LANES;
    for (uint32_t k = tid; k < p.nt * p.nt; k += NA_THREADS) {
        s_pair[k][0] = p.pair[k][0];
        s_pair[k][1] = p.pair[k][1];
    }
    if (tid < NA_BEADS) s_long[tid] = 0u;
    __syncthreads();
    const uint32_t h = blockIdx.x * NA_BEADS + b;
    const bool act = h < p.n;
    uint32_t i = 0;
    int c[3] = {0, 0, 0};
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    if (act) {
        o = S->pos[h];
        i = __float_as_uint(o.w);
        na_cell_of(p, S, i, c);
        if (sub == 0) {
            s_id[b] = i;
            for (int k = 0; k < 3; k++) s_c[b][k] = c[k];
        }
    }
    for (int row = sub; row < NA_ROWS; row += NA_LANES) {
        uint32_t n = 0, *out = s_row[b * NA_ROWS + row];
        for (uint32_t dz = 0; act && dz < 3; dz++)
            na_cell(p, S, c, o, 3 * row + dz, [&](uint32_t j) {
                if (j == i && row == 4 && dz == 1) return;
                if (n < NA_ROW_CAP) out[n] = j | (3 * row + dz) << 16;
                n++;
            });
        if (n > NA_ROW_CAP) {
            s_long[b] = 1u;
            n = 0;
        }
        s_pre[b * NA_ROWS + row] = n;
    }
    __syncthreads();
    if (tid < 32) {  // exclusive prefix of the rows' counts
        uint32_t carry = 0;
        for (int r0 = 0; r0 < NA_BEADS * NA_ROWS; r0 += 32) {
            const int r = r0 + tid;
            const uint32_t n = r < NA_BEADS * NA_ROWS ? s_pre[r] : 0u;
            uint32_t inc = n;
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, off);
                if (tid >= off) inc += y;
            }
            if (r < NA_BEADS * NA_ROWS) s_pre[r] = carry + inc - n;
            carry += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (tid == 0) s_pre[NA_BEADS * NA_ROWS] = carry;
    }
    __syncthreads();
    const uint64_t th = t_hash((uint32_t)p.t, p.seed);
    const uint32_t th_lo = (uint32_t)th, th_hi = (uint32_t)(th >> 32);
    const uint32_t total = s_pre[NA_BEADS * NA_ROWS];
    const int sb = tid % NA_BEADS, axis = tid / NA_BEADS;  // the summing threads' bead and axis
    const uint32_t b0 = s_pre[sb * NA_ROWS], b1 = s_pre[(sb + 1) * NA_ROWS];
    double F = 0.0;
    for (uint32_t c0 = 0; c0 < total; c0 += NA_TERMS) {
        const uint32_t c1 = min(total, c0 + NA_TERMS);
        for (uint32_t e = c0 + tid; e < c1; e += NA_THREADS) {
            uint32_t r = 0;  // the entry's row: the last with s_pre[r] <= e
            for (uint32_t step = 128; step > 0; step >>= 1)
                if (r + step < NA_BEADS * NA_ROWS && s_pre[r + step] <= e) r += step;
            const uint32_t ent = s_row[r][e - s_pre[r]], eb = r / NA_ROWS;
            double t[3] = {0.0, 0.0, 0.0};
            na_pair(p, s_pair, x, v, hash, s_id[eb], ent & 0xffffu, s_c[eb], ent >> 16, th_lo, th_hi, t);
            for (int k = 0; k < 3; k++) s_t[k][e - c0] = t[k];
        }
        __syncthreads();
        if (axis < 3)
            for (uint32_t e = max(b0, c0); e < min(b1, c1); e++) F = F + s_t[axis][e - c0];
        __syncthreads();
    }
    if (axis < 3 && blockIdx.x * NA_BEADS + sb < p.n && !s_long[sb]) f[3 * s_id[sb] + axis] = F;
    if (h < p.n && s_long[b]) na_long_bead(p, s_pair, S, x, v, hash, h, th_lo, th_hi, s_row[b * NA_ROWS], s_t, f);
}

// update_mom (dpd_maths_core_half_step.hpp:51-61).
__global__ void k_na_update_mom(NaParams p, double *v, const double *f)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const double hdt = p.dt * 0.5;
    for (int d = 0; d < 3; d++) v[3 * i + d] = v[3 * i + d] + f[3 * i + d] * hdt;
}

constexpr int NA_MAX_DEVICES = 64;
std::mutex g_na_mutex;
void *g_na_scratch[NA_MAX_DEVICES];

}  // namespace
}  // namespace pdpd

extern "C" int pdpd_step_noalloc(const pdpd_world *w, double *d_x, double *d_v, double *d_f,
                                 const uint32_t *d_hash, uint32_t n_steps, void *stream)
{
    using namespace pdpd;
    auto fail = [](int code, const char *msg) {
        set_thread_error(msg);
        return code;
    };
    if (!w) return fail(PDPD_E_INVALID, "pdpd_step_noalloc: no world");
    if (w->n_bonds || w->n_angles)
        return fail(PDPD_E_UNSUPPORTED, "pdpd_step_noalloc: worlds with bonds are not supported");
    if (w->n_bead_types == 0 || w->n_bead_types > 16 || !w->conservative || !w->dissipative)
        return fail(PDPD_E_INVALID, "pdpd_step_noalloc: 1..16 bead types with interaction matrices required");
    if (w->stationary)
        for (uint32_t k = 0; k < w->n_bead_types; k++)
            if (w->stationary[k]) return fail(PDPD_E_UNSUPPORTED, "Engine does not support stationary bead types.");
    if (w->cell_conservative || w->cell_dissipative)
        return fail(PDPD_E_UNSUPPORTED, "The allocation-free entry point does not support per-cell strengths.");
    if (!(w->dt > 0 && w->dt < 1)) return fail(PDPD_E_INVALID, "pdpd_step_noalloc: dt must be in (0, 1)");
    uint64_t cells = 1;
    for (int k = 0; k < 3; k++) {
        if (w->box[k] < 2) return fail(PDPD_E_INVALID, "Distance in each direction must be at least 2");
        cells *= (uint64_t)w->box[k];
    }
    if (w->n_beads > NA_MAX_BEADS || cells > NA_MAX_CELLS)
        return fail(PDPD_E_NOMEM, "pdpd_step_noalloc: at most 65536 beads and 32768 cells (the fixed scratch size)");
    if (n_steps == 0 || w->n_beads == 0) return PDPD_OK;
    if (!d_x || !d_v || !d_f || !d_hash) return fail(PDPD_E_INVALID, "pdpd_step_noalloc: missing device array");

    int dev = 0;
    cudaError_t ce = cudaGetDevice(&dev);
    if (ce != cudaSuccess || dev < 0 || dev >= NA_MAX_DEVICES)
        return fail(PDPD_E_CUDA, "pdpd_step_noalloc: no current CUDA device");
    void *scratch = nullptr;
    {
        // First call on a device: look up the device address of the scratch array.
        std::lock_guard<std::mutex> lock(g_na_mutex);
        if (!g_na_scratch[dev]) {
            ce = cudaGetSymbolAddress(&g_na_scratch[dev], g_noalloc_scratch);
            if (ce != cudaSuccess) {
                g_na_scratch[dev] = nullptr;
                return fail(PDPD_E_CUDA, "pdpd_step_noalloc: cudaGetSymbolAddress failed");
            }
        }
        scratch = g_na_scratch[dev];
    }
    NaScratch *S = (NaScratch *)scratch;
    cudaStream_t s = (cudaStream_t)stream;
    NaParams p;
    memset(&p, 0, sizeof p);
    for (int k = 0; k < 3; k++) p.L[k] = w->box[k];
    p.n = w->n_beads;
    p.n_cells = (uint32_t)cells;
    p.nt = w->n_bead_types;
    p.dt = w->dt;
    p.scale_inv_sqrt_dt = sqrt(24 * 1.0 / w->dt);
    p.seed = w->seed;
    for (uint32_t k = 0; k < p.nt * p.nt; k++) {
        p.pair[k][0] = w->conservative[k];
        p.pair[k][1] = sqrt(w->dissipative[k]);
    }
    const uint32_t gb = (p.n + 255) / 256, gc = (p.n_cells + 255) / 256;
    k_na_clear<<<gc, 256, 0, s>>>(S, p.n_cells);
    for (uint32_t step = 0; step < n_steps; step++) {
        p.t = w->t + (int64_t)step;
        k_na_update_pos<<<gb, 256, 0, s>>>(p, S, d_x, d_v, d_f, step > 0 ? 1 : 0);
        k_na_scan<<<1, 1024, 0, s>>>(S, p.n_cells, p.n);
        k_na_place<<<gb, 256, 0, s>>>(S, p.n);
        k_na_canon<<<gb, 256, 0, s>>>(S, p.n, d_x);
        k_na_forces<<<(p.n + NA_BEADS - 1) / NA_BEADS, NA_THREADS, 0, s>>>(p, S, d_x, d_v, d_f, d_hash);
    }
    k_na_update_mom<<<gb, 256, 0, s>>>(p, d_v, d_f);
    uint32_t err = 0;
    ce = cudaGetLastError();
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(&err, &S->err, sizeof err, cudaMemcpyDeviceToHost, s);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(s);
    if (ce != cudaSuccess) return fail(PDPD_E_CUDA, cudaGetErrorString(ce));
    if (err) return fail(PDPD_E_BEAD_LOST, "pdpd_step_noalloc: a bead left the box or became non-finite");
    return PDPD_OK;
}
