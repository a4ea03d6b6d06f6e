// FP64 pair forces, each pair evaluated once.  Included inside pdpd_fp64.cu's anonymous
// namespace.
//
// GB300 runs FP64 at 2 lanes per clock per SM, an FP64 instruction takes its pipe for the whole
// warp whatever its active lanes, and a pair force is ~50 FP64 instructions: the force pass is
// bound by the number of FP64 warp instructions.  A pair term is exactly antisymmetric when no
// periodic shift enters it (x_i - x_j, e, v_i - v_j change sign, everything else is the same to
// the bit), so it is computed once, by the bead of the lower slot, and the other bead adds
// its negation; a pair across the box's faces (the reference shifts the neighbour, which rounds
// differently from either side) and the pairs of a world with unsymmetric strengths are
// evaluated from both sides.  Every bead adds its terms in its own walk's order, so its force
// is the reference's to the bit.  Three kernels:
//   k_list64   each bead's candidates in walk order (list) and, of these, the pairs it evaluates
//              itself (pair_i, pair_j): FP32 walk over a staged brick (pdpd_walk.cuh), no FP64 work;
//   k_pairs64  one thread per pair: full warps of FP64 work, whatever the beads' counts; it also
//              enters the pair in the other bead's list;
//   k_sum64    each bead adds its terms in order, then bonds and integration.
// 64^3 polymer box, force pass with bonds: 1.78 ms with each bead evaluating all its pairs
// (k_force64), 0.83 ms so (lists and bonds 0.16, pairs 0.44 at 84% of the FP64 pipe, sums 0.21).
// (Pairs evaluated by the listing blocks themselves, to have the FP64 pipe busy meanwhile: 0.82
// ms, and 0.092 -> 0.105 at 27^3: two blocks per SM do not keep both halves going.)
// k_force64 stays for batches the lists have no memory for or too many beads for (a list
// entry holds a slot in 25 bits).

// A list entry is one of: L64_OWN | q, the bead evaluates pair q; the slot of a lower bead (25
// bits), which evaluates the pair; and, once that has happened, L64_OTHER | q in its place.
constexpr uint32_t L64_SLOT = (1u << 25) - 1u;
constexpr uint32_t L64_OWN = 1u << 31, L64_OTHER = 1u << 30, L64_PAIR = L64_OTHER - 1u;
constexpr uint32_t L64_BOTH = 1u << 31;  // pair_j: the pair is evaluated from both sides
constexpr uint32_t L64_NONE = 0xffffffffu;

// Evaluated from both sides: bead j reached across the box's faces, or unsymmetric strengths.
// Else the bead of the lower slot evaluates the pair.
__device__ __forceinline__ bool both_sides(const WorldDev &w, uint32_t code)
{
    return (code & 0x80000000u) || w.asym;
}

// The candidates of a bead from global memory, in walk order (a bead of a brick too full to
// stage, or with too many candidates for its segments): visit(slot, dir, image) with the
// direction packed 2 bits per axis as d + 1.  The same conservative test as the staged walk's.
template <class Visit>
__device__ __forceinline__ void walk_global64(const KArgs &a, const WorldDev &w, uint32_t s, const int c[3],
                                              const float4 oh, Visit visit)
{
    for (int dx = -1; dx <= 1; dx++)
        for (int dy = -1; dy <= 1; dy++)
            for (int dz = -1; dz <= 1; dz++) {
                const float gx = slab_gap(oh.x, dx), gy = slab_gap(oh.y, dy), gz = slab_gap(oh.z, dz);
                if (gx * gx + gy * gy + gz * gz >= WALK_R2) continue;
                const int raw[3] = {c[0] + dx, c[1] + dy, c[2] + dz};
                int op[3];
                bool image = false;
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    op[k] = wrap_index(raw[k], w.L[k]);
                    image |= op[k] != raw[k];
                }
                const uint32_t nc = w.cell_base + ((uint32_t)op[0] * (uint32_t)w.L[1] + (uint32_t)op[1]) * (uint32_t)w.L[2] + (uint32_t)op[2];
                const float ax = oh.x - (float)dx, ay = oh.y - (float)dy, az = oh.z - (float)dz;
                const uint32_t dir = (uint32_t)(dx + 1) | ((uint32_t)(dy + 1) << 2) | ((uint32_t)(dz + 1) << 4);
                const uint32_t j1 = a.start[nc + 1];
                for (uint32_t j = a.start[nc]; j < j1; j++) {
                    const float4 q = a.posf[j];
                    const float ex = ax - q.x, ey = ay - q.y, ez = az - q.z;
                    if (ex * ex + ey * ey + ez * ez >= WALK_R2 || (j == s && dir == 21u)) continue;
                    visit(j, dir, image);
                }
            }
}

struct List64Header {
    WorldDev w;
    uint32_t home_rows[65];
    uint32_t total, next;
    uint16_t halo_row[64];
};

// Shared memory of k_list64: header, hstart, hslot, row bases, then per staged bead offsets
// (xy), z in brick coordinates (zf) and {slot, halo cell code} (sc), and the walk segments.
struct List64Layout {
    uint32_t hc_max, maxb, off_hstart, off_hslot, off_rowbase, off_xy, off_zf, off_sc, off_segs, bytes;
};

constexpr uint32_t LIST64_BEAD_BYTES = 20;
constexpr int LIST64_THREADS = 512;
// Walk segments per thread: a bead whose segments do not fit takes the slow global walk (at 9, one for
// each row, 0.1% of the beads of a box of density 3, and 35 of 50 us of the kernel at 27^3)
constexpr int LIST64_SEGS = 18;

__host__ __device__ inline List64Layout list64_layout(uint32_t hc_max, uint32_t maxb)
{
    List64Layout L{};
    L.hc_max = hc_max;
    L.maxb = maxb;
    maxb = (maxb + 3) & ~3u;
    uint32_t off = (uint32_t)((sizeof(List64Header) + 15) & ~size_t(15));
    auto take = [&](uint32_t bytes) {
        const uint32_t at = off;
        off = (off + bytes + 15) & ~15u;
        return at;
    };
    L.off_hstart = take(3 * hc_max);
    L.off_hslot = take(4 * hc_max);
    L.off_rowbase = take(4 * (hc_max / 3));
    L.off_xy = take(8 * maxb);
    L.off_zf = take(4 * maxb);
    L.off_sc = take(8 * maxb);
    L.off_segs = take(4 * (LIST64_SEGS + 1) * LIST64_THREADS);
    L.bytes = off;
    return L;
}

// Candidate lists of the beads of a brick, one thread per home bead.  A warp takes room for its
// beads' entries and pairs from two cursors (a block at a time, a 16th of the atomics, is no
// faster: 164 us against 161 for the 64^3 box); where there is none left, its beads are marked
// (lrec.x) and k_sum64 evaluates all their pairs itself.  The order in which warps take room
// changes where a list lies, not what is in it.  Bound by instruction issue; no FP64 work.
//
// The queue's entries after the bricks are chunks of the bond forces: FP64 work, which the pipe
// has nothing else of meanwhile, in a few warps (64^3 polymer box: 25 us in the prefix sum's
// launch).
//
// PLANES = 3, in the smallest batches (small_shape): three lanes per bead, one per plane of
// neighbour rows, whose parts of the list follow each other.  (8^3 water, step: 31.5 ->
// 28.5 us; 16^3 43.6 -> 41.7, 24^3 74.2 -> 72.5.)
constexpr uint32_t BOND64_CHUNK = 128;
template <int PLANES>
__global__ void __launch_bounds__(LIST64_THREADS, 2) k_list64(KArgs a, List64Layout lay, uint32_t bb, uint32_t work)
{
    constexpr int T = LIST64_THREADS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    List64Header &H = *reinterpret_cast<List64Header *>(smem_raw);
    uint16_t *hstart = reinterpret_cast<uint16_t *>(smem_raw + lay.off_hstart);
    uint32_t *hslot = reinterpret_cast<uint32_t *>(smem_raw + lay.off_hslot);
    uint32_t *rowbase = reinterpret_cast<uint32_t *>(smem_raw + lay.off_rowbase);
    float *xy = reinterpret_cast<float *>(smem_raw + lay.off_xy);
    float *zf = reinterpret_cast<float *>(smem_raw + lay.off_zf);
    uint2 *sc = reinterpret_cast<uint2 *>(smem_raw + lay.off_sc);
    const int tid = threadIdx.x, lane = tid & 31;
    uint32_t *segs = reinterpret_cast<uint32_t *>(smem_raw + lay.off_segs) + tid;
    const int cap = (a.list_capacity > 0 && a.list_capacity < LIST64_SEGS) ? max(3, a.list_capacity) : LIST64_SEGS;
    uint32_t world = L64_NONE;
    Brick first{};
    if (blockIdx.x < a.n_bricks) {  // (what no step changes is read before the wait)
        first = a.bricks[blockIdx.x];
        if (tid == 0) H.w = a.worlds[first.world];
        world = first.world;
    }
    step_kernel_wait();
    __syncthreads();
    for (uint32_t bi = blockIdx.x; bi < work;) {
        if (bi >= a.n_bricks) {  // Hookean bonds, then angle bonds
            const uint32_t c = bi - a.n_bricks;
            const bool angle = c >= bb;
            if (tid < BOND64_CHUNK)
                bonds64(a, (const Vec4d *)a.posA, (c - (angle ? bb : 0u)) * BOND64_CHUNK + tid, angle);
            __syncthreads();
            if (tid == 0) H.next = gridDim.x + atomicAdd(a.brick_next, 1u);
            __syncthreads();
            bi = H.next;
            continue;
        }
        const Brick br = bi == blockIdx.x ? first : a.bricks[bi];
        if (br.world != world) {
            if (tid == 0) H.w = a.worlds[br.world];
            world = br.world;
            __syncthreads();
        }
        const WorldDev &w = H.w;
        const int HY = br.by + 2, HZ = br.bz + 2;
        uint32_t total = 0, n_home = 0;
        brick_stage_rows<T>(a, w, br, a.posf, H.home_rows, H.halo_row, &H.total, hstart, hslot, rowbase, xy, zf, lay.maxb, total,
                            n_home, [&](uint32_t j, uint32_t slot, const float4 &, uint32_t code) {
                                sc[j] = make_uint2(slot, code);
                            });
        const bool staged = total <= lay.maxb;
        constexpr uint32_t WARP_BEADS = PLANES == 3 ? 10u : 32u;
        for (uint32_t t0 = (tid >> 5) * WARP_BEADS; t0 < n_home; t0 += (T / 32) * WARP_BEADS) {
            const int plane = PLANES == 3 ? lane % 3 : 0;
            const uint32_t t = t0 + (PLANES == 3 ? lane / 3 : lane);
            const int r = home_row_near(H.home_rows, br.bx * br.by, t0, t);
            const bool act = t < n_home && (PLANES == 1 || lane < 30);
            uint32_t s = 0, code = 0;
            uint32_t n = 0, own = 0;
            bool dense = !staged;
            int c[3] = {0, 0, 0};
            if (act) {
                const int row = H.halo_row[r];
                const uint32_t k = t - H.home_rows[r];
                s = hslot[row * HZ + 1] + k;
                if (staged) {
                    const uint32_t si = hstart[row * (HZ + 1) + 1] + k;
                    const float *q = xy + 2 * si - (si & 1u);
                    code = sc[si].y;
                    n = (uint32_t)walk_rows<T, PLANES>((const ulonglong2 *)xy, (const uint64_t *)zf, segs, cap, hstart, HY,
                                                       HZ + 1, code, si, q[0], q[2], a.posf[s].z,
                                                       [&](int) { dense = true; }, plane);
                    if (!dense) {
                        SegReader<T> seg(segs);
                        for (uint32_t e = 0; e < n; e++) {
                            const uint2 o = sc[seg.next()];
                            own += both_sides(w, o.y) || o.x > s;
                        }
                    }
                }
            }
            if (PLANES == 3) {  // a bead of whose lanes one has too many is left to the first
                const uint32_t any = __ballot_sync(0xffffffffu, dense) >> (lane - plane) & 7u;
                dense = any != 0u;
                if (dense && plane != 0) n = own = 0;
            }
            if (act) {
                if (dense && plane == 0) {
                    n = own = 0;
                    decode_cell(a.cellg[s] - w.cell_base, w.L, c[0], c[1], c[2]);
                    walk_global64(a, w, s, c, a.posf[s], [&](uint32_t j, uint32_t, bool image) {
                        n++;
                        own += both_sides(w, image ? 0x80000000u : 0u) || j > s;
                    });
                }
            }
            // room for the warp's entries and pairs
            uint32_t n_inc = n, own_inc = own;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, n_inc, off), z = __shfl_up_sync(0xffffffffu, own_inc, off);
                if (lane >= off) {
                    n_inc += y;
                    own_inc += z;
                }
            }
            unsigned long long first = 0, pfirst = 0;
            if (lane == 31) {
                first = atomicAdd(a.list_cursor, (unsigned long long)n_inc);
                pfirst = atomicAdd(a.list_cursor + 1, (unsigned long long)own_inc);
            }
            const uint32_t n_all = __shfl_sync(0xffffffffu, n_inc, 31), own_all = __shfl_sync(0xffffffffu, own_inc, 31);
            first = __shfl_sync(0xffffffffu, first, 31);
            pfirst = __shfl_sync(0xffffffffu, pfirst, 31);
            if (first + n_all > a.list_cap || pfirst + own_all > a.pair_cap) {
                // no room left: what the warp took of the pairs' holds none
                for (unsigned long long q = pfirst + lane; q < pfirst + own_all && q < a.pair_cap; q += 32)
                    a.pair_i[q] = L64_NONE;
                if (act && plane == 0) a.lrec[s] = make_uint2(L64_NONE, 0u);
                continue;
            }
            const uint32_t at = (uint32_t)first + n_inc - n;
            uint32_t q = (uint32_t)pfirst + own_inc - own;
            uint32_t all = n;
            if (PLANES == 3) all += __shfl_down_sync(0xffffffffu, n, 1) + __shfl_down_sync(0xffffffffu, n, 2);
            if (!act) continue;
            uint32_t *list = a.list + at;
            if (plane == 0) a.lrec[s] = make_uint2(at, all);
            if (PLANES == 3 && dense && plane != 0) continue;
            auto emit = [&](uint32_t j, uint32_t dir, bool both) {
                if (both || j > s) {
                    *list++ = L64_OWN | q;
                    a.pair_i[q] = s;
                    a.pair_j[q++] = j | (dir << 25) | (both ? L64_BOTH : 0u);
                } else {
                    *list++ = j;
                }
            };
            if (dense) {
                walk_global64(a, w, s, c, a.posf[s], [&](uint32_t j, uint32_t dir, bool image) {
                    emit(j, dir, both_sides(w, image ? 0x80000000u : 0u));
                });
            } else {
                SegReader<T> seg(segs);
                for (uint32_t e = 0; e < n; e++) {
                    const uint2 o = sc[seg.next()];
                    const uint32_t d = (o.y & 0x00ffffffu) + 0x00010101u - (code & 0x00ffffffu);  // d + 1 per byte
                    emit(o.x, (d & 3u) | ((d >> 6) & 0xcu) | ((d >> 12) & 0x30u), both_sides(w, o.y));
                }
            }
        }
        __syncthreads();
        if (tid == 0) H.next = gridDim.x + atomicAdd(a.brick_next, 1u);
        __syncthreads();
        bi = H.next;
    }
}

// One pair's term on bead i (calc_force through pair_terms64), from bead j in direction dir
// (2 bits per axis, d + 1): the reference's separation and pair test
// (naive_dpd_engine_half_step.hpp:181-196, 404-411); false when out of range.  shifted: j may lie
// across the box's faces.
__device__ __forceinline__ bool pair_term64(const KArgs &a, const WorldDev &w, uint32_t i, uint32_t j, uint32_t dir,
                                            bool shifted, uint32_t th_lo, uint32_t th_hi, double t[3])
{
    const Vec4d pi = ((const Vec4d *)a.posA)[i];
    Vec4d pj = ((const Vec4d *)a.posA)[j];
    if (shifted) {
        int c[3];
        decode_cell(a.cellg[i] - w.cell_base, w.L, c[0], c[1], c[2]);
        const int d[3] = {(int)(dir & 3u) - 1, (int)((dir >> 2) & 3u) - 1, (int)((dir >> 4) & 3u) - 1};
        const double Ld[3] = {(double)w.L[0], (double)w.L[1], (double)w.L[2]};
        double delta[3];
        neighbour64(w, c, d, Ld, delta);
        pj.x += delta[0];
        pj.y += delta[1];
        pj.z += delta[2];
    }
    const double dx0 = pi.x - pj.x, dx1 = pi.y - pj.y, dx2 = pi.z - pj.z;
    const double dr2 = dx0 * dx0 + dx1 * dx1 + dx2 * dx2;
    // dr2 < 1 and dr2 >= min2 on the bits (dr2 is not negative: an integer comparison, not an FP64 one)
    const long long bits = __double_as_longlong(dr2);
    if (bits >= 0x3ff0000000000000ll || bits < __double_as_longlong((double)min_dist_sqr_f())) return false;
    const Vec4d vi = ((const Vec4d *)a.velA)[i], vj = ((const Vec4d *)a.velA)[j];
    const uint32_t hi = hash_of(pi), hj = hash_of(pj);
    const uint32_t n2 = w.n_types * w.n_types;
    const uint32_t pk = min(hi >> 28, w.n_types - 1u) * w.n_types + min(hj >> 28, w.n_types - 1u);
    Vec2d pp = ((const Vec2d *)a.pair)[w.param_base + pk];
    if (w.spatial) {  // mean of the two beads' cell values (naive_dpd_engine_half_merge.hpp:570-583)
        const Vec2d *cp = (const Vec2d *)a.cellpair + w.cellpair_base;
        const Vec2d h = cp[(size_t)(a.cellg[i] - w.cell_base) * n2 + pk], o = cp[(size_t)(a.cellg[j] - w.cell_base) * n2 + pk];
        pp.x = (h.x + o.x) * 0.5;
        pp.y = (h.y + o.y) * 0.5;
    }
    const PairTerms64 q = pair_terms64(dx0, dx1, dx2, sqrt(dr2), pp, vi, vj, hi, hj, th_lo, th_hi, w.scale_inv_sqrt_dt);
    t[0] = q.e[0] * q.scaled;
    t[1] = q.e[1] * q.scaled;
    t[2] = q.e[2] * q.scaled;
    return true;
}

// The pair terms, one thread per pair: bound by the FP64 pipe.  A pair out of range (the lists
// are conservative) gets a zero term: adding it changes nothing.  The thread also enters the pair
// in the other bead's list, in the place of its slot (not there: out of range from that
// side); these look-ups wait on memory while other warps have the pipe.
constexpr int PAIRS64_THREADS = 64;
__global__ void __launch_bounds__(PAIRS64_THREADS) k_pairs64(KArgs a)
{
    step_kernel_wait();
    const unsigned long long n_all = a.list_cursor[1];
    const uint32_t n = (uint32_t)min(n_all, (unsigned long long)a.pair_cap);
    uint32_t world = L64_NONE, th_lo = 0, th_hi = 0;
    for (uint32_t q = blockIdx.x * PAIRS64_THREADS + threadIdx.x; q < n; q += gridDim.x * PAIRS64_THREADS) {
        const uint32_t i = a.pair_i[q], e = a.pair_j[q], j = e & L64_SLOT;
        if (i == L64_NONE) continue;
        uint32_t lo = 0, hi = a.n_worlds;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) / 2;
            if (a.worlds[mid].bead_base <= i) lo = mid; else hi = mid;
        }
        const WorldDev &w = a.worlds[lo];
        if (lo != world) {
            const uint64_t th = t_hash((uint32_t)w.t, w.seed);
            th_lo = (uint32_t)th;
            th_hi = (uint32_t)(th >> 32);
            world = lo;
        }
        if (!(e & L64_BOTH)) {
            const uint2 o = a.lrec[j];
            for (uint32_t k = 0; k < o.y; k += 4) {  // (four at a time: their loads overlap)
                uint32_t y[4], at = L64_NONE;
#pragma unroll
                for (uint32_t u = 0; u < 4; u++) y[u] = a.list[o.x + min(k + u, o.y - 1u)];
#pragma unroll
                for (uint32_t u = 0; u < 4; u++)
                    if (y[u] == i) at = o.x + min(k + u, o.y - 1u);
                if (at != L64_NONE) {
                    a.list[at] = L64_OTHER | q;
                    break;
                }
            }
        }
        double t[3] = {0.0, 0.0, 0.0};
        pair_term64(a, w, i, j, (e >> 25) & 63u, (e & L64_BOTH) != 0u, th_lo, th_hi, t);
        double *out = a.term + 3 * (size_t)q;
        out[0] = t[0];
        out[1] = t[1];
        out[2] = t[2];
    }
}

// All pair terms of a bead without a list, added in walk order.
__device__ __noinline__ void bead_forces64(const KArgs &a, const WorldDev &w, uint32_t s, uint32_t th_lo,
                                           uint32_t th_hi, double F[3])
{
    int c[3];
    decode_cell(a.cellg[s] - w.cell_base, w.L, c[0], c[1], c[2]);
    walk_global64(a, w, s, c, a.posf[s], [&](uint32_t j, uint32_t dir, bool) {
        double t[3];
        if (!pair_term64(a, w, s, j, dir, true, th_lo, th_hi, t)) return;
        F[0] = F[0] + t[0];
        F[1] = F[1] + t[1];
        F[2] = F[2] + t[2];
    });
}

// A pair's term on bead s when the other bead has no list.
__device__ __noinline__ void single_term64(const KArgs &a, const WorldDev &w, uint32_t s, uint32_t other,
                                           double t[3])
{
    const uint64_t th = t_hash((uint32_t)w.t, w.seed);
    pair_term64(a, w, s, other, 21u, false, (uint32_t)th, (uint32_t)(th >> 32), t);
}

// Sum and integration of 32 sorted beads of one world (a part of a tile).  The beads' entries are
// taken flat, one thread each, and their terms brought into shared memory with the sign they are
// added with; then a thread per bead and axis adds them in order, and a thread per bead
// integrates.
constexpr int SUM64_THREADS = 128, SUM64_BEADS = 32, SUM64_ENTRIES = 512;
template <int FINAL>
__global__ void __launch_bounds__(SUM64_THREADS, 12) k_sum64(KArgs a)
{
    step_kernel_wait();
    constexpr int PARTS = TILE_BEADS / SUM64_BEADS;
    __shared__ double s_t[3][SUM64_ENTRIES];
    __shared__ uint32_t s_pre[SUM64_BEADS + 1], s_at[SUM64_BEADS];
    __shared__ double s_f[3][SUM64_BEADS];
    const int tid = threadIdx.x, lane = tid & 31, axis = tid >> 5;
    const Tile tl = a.tiles[blockIdx.x / PARTS];
    const uint32_t s0 = tl.slot_begin + (blockIdx.x % PARTS) * SUM64_BEADS;
    if (s0 >= tl.slot_end) return;  // (block-uniform)
    const WorldDev &w = a.worlds[tl.world];
    const uint32_t s = s0 + lane;
    const bool act = s < tl.slot_end;
    bool no_list = false;
    if (tid < 32) {  // exclusive prefix of the beads' entry counts
        const uint2 rec = act ? a.lrec[s] : make_uint2(0u, 0u);
        no_list = rec.x == L64_NONE;
        uint32_t inc = rec.y;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, off);
            if (lane >= off) inc += y;
        }
        s_pre[lane] = inc - rec.y;
        s_at[lane] = rec.x;
        if (lane == 31) s_pre[32] = inc;
    }
    __syncthreads();
    const uint32_t total = s_pre[32], b0 = s_pre[lane], b1 = s_pre[lane + 1];
    double F = 0.0;
    for (uint32_t c0 = 0; c0 < total; c0 += SUM64_ENTRIES) {
        const uint32_t c1 = min(total, c0 + SUM64_ENTRIES);
#pragma unroll 4
        for (uint32_t e = c0 + tid; e < c1; e += SUM64_THREADS) {
            int b = 0;  // the entry's bead: the last with s_pre[b] <= e
#pragma unroll
            for (int step = 16; step > 0; step >>= 1)
                if (s_pre[b + step] <= e) b += step;
            const uint32_t ent = a.list[s_at[b] + (e - s_pre[b])];
            double t[3] = {0.0, 0.0, 0.0};
            if (ent & (L64_OWN | L64_OTHER)) {
                const double *in = a.term + 3 * (size_t)(ent & L64_PAIR);
                const int sign = (int)((ent & L64_OTHER) << 1);
#pragma unroll
                for (int d = 0; d < 3; d++)  // (the sign flipped on the bits: a negation is an FP64 instruction)
                    t[d] = __hiloint2double(__double2hiint(in[d]) ^ sign, __double2loint(in[d]));
            } else if (a.lrec[ent].x == L64_NONE) {
                single_term64(a, w, s0 + b, ent, t);
            }
#pragma unroll
            for (int d = 0; d < 3; d++) s_t[d][e - c0] = t[d];
        }
        __syncthreads();
        if (axis < 3) {
            const uint32_t e1 = min(b1, c1);
#pragma unroll 1
            for (uint32_t e = max(b0, c0); e < e1; e++) F = F + s_t[axis][e - c0];
        }
        __syncthreads();
    }
    if (axis < 3) s_f[axis][lane] = F;
    __syncthreads();
    if (tid < 32 && act) {
        double G[3] = {s_f[0][lane], s_f[1][lane], s_f[2][lane]};
        if (no_list) {
            const uint64_t th = t_hash((uint32_t)w.t, w.seed);
            bead_forces64(a, w, s, (uint32_t)th, (uint32_t)(th >> 32), G);
        }
        integrate64<FINAL>(a, w, tl.world, s, G);
    }
}
