// GPU planner for one native GEMM call: block tile shape and split-K.
//
// Replaces the reference's CPU planner (core/matrix_matrix/planner.zig):
// desiredThreadCount :88 / rowTaskCount :170 / runPlannedTasks :296 split C
// into at most 64 disjoint column/row tasks for host threads.  On the GPU the
// equivalent decision is how many CTAs cover C (tile shape) and, when C has
// too few tiles to fill the 148 SMs, how far to split K; dgemm_tile_route then
// says which kernel runs the planned tiles.  Host code only.
#include <algorithm>

#include "kernels.h"

namespace zb {

GemmPlan plan_native_gemm(int m, int n, int k, int elem_bytes, int sm_count) {
    GemmPlan p;
    p.sm_count = sm_count;
    // n == 1 or m == 1: matrix-vector kernels, K split only while the outputs
    // alone leave SMs idle.
    if (n == 1 || m == 1) {
        p.tile = TILE_GEMV;
        p.splits = gemv_split_count(n == 1 ? m : n, k);
        return p;
    }
    // At most 16 columns (rows) of C: 128 x 16 (16 x 128) FP64 tiles or the
    // FP32 narrow kernel, K split while the output tiles leave SMs idle.
    if ((n <= 16 && m >= 512) || (m <= 16 && n >= 512)) {
        p.tile = n <= 16 ? TILE_NARROW_N : TILE_NARROW_M;
        p.splits = narrow_split_count(m, n, k, sm_count);
        return p;
    }
    // FP64 with fewer 128 x 128 tiles than half the SMs and a short K (<= 1024,
    // too short for split-K to fill the machine with 256-deep slices): 64 x 64
    // tiles (4 warps), K split into slices down to 64 deep until about two CTAs
    // per SM are resident (small products, the coupling GEMMs of blocked TRSM;
    // one CTA per SM measured 5-20 % slower at 512-1024 x 512 x 512-1024, three
    // or four no better than two).  Longer K keeps the 128 x 128 tiles and
    // their split-K below.
    if (elem_bytes == 8 && k <= 1024 && 2L * ((m + 127) / 128) * ((n + 127) / 128) < sm_count) {
        p.tile = TILE_64x64;
        const long tiles = (long)((m + 63) / 64) * ((n + 63) / 64);
        if (tiles < 2L * sm_count && k >= 128) {
            long s = 2L * sm_count / std::max<long>(tiles, 1);
            s = std::min<long>(s, k / 64);
            s = std::min<long>(s, 64);
            if (s >= 2) p.splits = (int)s;
        }
        return p;
    }
    // Narrow-N, tall-M shapes (e.g. 131072 x 64 x 64) are HBM-bound: a 64-wide
    // tile avoids computing (and staging) a half-empty 128-wide tile.
    if (elem_bytes == 8 && n <= 64 && m >= 1024) p.tile = TILE_128x64;
    const int bn = (p.tile == TILE_128x64) ? 64 : 128;
    const long tiles = (long)((m + 127) / 128) * ((n + bn - 1) / bn);
    // Fewer tiles than SMs: split K (each slice at least 256 deep) so that
    // about one wave of CTAs covers the machine; the partials cost one
    // (splits + 2) m n element pass.
    p.splits = 1;
    if (tiles < sm_count && k >= 512) {
        long s = sm_count / std::max<long>(tiles, 1);
        s = std::min<long>(s, k / 256);
        s = std::min<long>(s, 64);
        if (s >= 2) p.splits = (int)s;
    }
    return p;
}

int dgemm_tma_k_chunk(int k, int splits) {
    splits = std::max(1, splits);
    const int c = (k + splits - 1) / splits;
    return (c + kDgemmTmaSlice - 1) / kDgemmTmaSlice * kDgemmTmaSlice;
}

namespace {

constexpr long kMaxGridY = 65535;  // the tile kernels put column tiles on grid.y

// Cluster size with which a planned product runs on the 64 x 64 warp-specialised tiles
// instead (dgemm_ws, which needs none of the plan's workspace); 0: it does not.
int ws_cluster(int m, int n, int k, int tri, bool tma, const GemmPlan& plan) {
    if (!plan.automatic) return 0;
    const long sms = plan.sm_count;
    const long t64 = (long)((m + 63) / 64) * ((n + 63) / 64);
    if (plan.tile == TILE_64x64) {
        // about one 64 x 64 tile per SM (99 .. 148 tiles on 148 SMs), which is where the plan has
        // two K ranges: two CTAs of a cluster per tile.  Fewer tiles keep the cp.async tiles,
        // which split K further and reduce through L2 (81 tiles, three ranges against a cluster
        // of two: 576 x 576 x 1024 34.5 against 44.9 us, and two ranges round worse than three;
        // clusters of 4 and 8 lost too: 384 x 384 x 1024 21.0 / 15.5 us, 256 x 256 x 1024 15.3 /
        // 9.3).  110 tiles, 640 x 704 x 512: 26.3 us on the cluster, 29.1 through the workspace.
        return plan.splits == 2 && k >= 256 && tma ? 2 : 0;
    }
    if (plan.tile != TILE_128x128 || plan.splits > 1 || k < 256) return 0;
    // 64-wide column tiles run out of grid.y at half the columns of 128-wide ones
    if ((n + 63L) / 64 > kMaxGridY) return 0;
    // both tile sizes run in rounds of one tile per SM; a 128 x 128 round at 0.955 of the
    // pipe, a 64 x 64 one (a quarter of the work) at 0.90 (2048^3: 559 / 517 us, 3000^3 TT
    // 1689 / 1628, 1536^3, one round of 128 x 128 tiles, 212 / 229)
    const long m1 = (m + 127) / 128, n1 = (n + 127) / 128, m6 = (m + 63) / 64;
    const long live1 = tri ? m1 * (m1 + 1) / 2 : m1 * n1, live6 = tri ? m6 * (m6 + 1) / 2 : t64;
    const double r128 = 4.0 * ((live1 + sms - 1) / sms) / 0.955;
    double r64 = ((live6 + sms - 1) / sms) / 0.90;
    // a triangle's CTAs without a tile leave at once, and the others land unevenly: 0.6 to 1.4
    // tiles over the average load of an SM, and never under 3.2 (order 2876, k 1335: 377 us on
    // 128 x 128 tiles, 413 on these; order 2200: 376 / 267; order 1700, lower: 193 / 206)
    if (tri) r64 = std::max((double)live6 / sms + 1.2, 3.2) / 0.90;
    return r64 < 0.98 * r128 && tma ? 1 : 0;
}

// CTAs of `c`-clusters that run with an SM each.  A cluster lives inside one GPC, so up to
// c - 1 SMs of every GPC stay free: on 148 SMs 15 clusters of eight run side by side, 33 of
// four and 74 of two; the 16th, 34th, ... share SMs with the others, and their launch takes
// twice as long as the SM count suggests.
long cluster_ctas(int c, long sms) { return c > 2 ? sms - 7 * c / 2 : sms; }

// Cluster size with which a planned small product runs on the 64 x 64 cluster tiles
// (dgemm_cluster_kernel: one launch, none of the plan's workspace); 0: it does not.
// Never fewer K ranges than the plan, which splits down to 64-deep slices (256 x 256 x 1024 in
// 16 ranges 9.6 us, a cluster of 8 15.1).  Microseconds on the device, plan / cluster of four.
int small_cluster(int m, int n, int k, const GemmPlan& plan) {
    const long t64 = (long)((m + 63) / 64) * ((n + 63) / 64), sms = plan.sm_count;
    if (!plan.automatic || plan.tile != TILE_64x64 || plan.splits < 2) return 0;
    if (k > 256 && plan.splits != 4) return 0;
    // an SM for each CTA (up to 33 tiles): saves the second launch (33 tiles, k = 192: 8.5 / 6.7;
    // 16 tiles, k = 256: 6.6 / 6.8, and 11.4 / 9.3 a call)
    if (4 * t64 <= cluster_ctas(4, sms)) return 4;
    // more than two CTAs for an SM: the last clusters run alone (72 tiles, k = 512: 0.75 x)
    if (4 * t64 > sms + cluster_ctas(4, sms)) return 0;
    // two CTAs on an SM: where the plan's ranges are twice as long (k = 160: 1.05 - 1.2 x) or
    // share SMs too (50 tiles, k = 192: 1.26 x; 34 - 37 tiles, k = 192 .. 319, where they have an
    // SM each: 0.78 - 0.99 x; 40 - 59 tiles with four ranges, k = 257 .. 319: 0.77 - 1.04 x)
    if (k <= 256) return plan.splits == 2 || plan.splits * t64 > sms ? 4 : 0;
    // 60 to 70 tiles, which the plan gives four ranges whatever K: 1.02 - 1.08 x up to k = 768,
    // 0.95 - 1.01 x at 1024
    return 2 * sms / t64 == 4 && k <= 768 ? 4 : 0;
}

}  // namespace

DgemmRoute dgemm_tile_route(int m, int n, int k, int tri, bool tma, const GemmPlan& plan) {
    DgemmRoute r;
    const int splits = std::max(1, plan.splits);
    if (const int c = ws_cluster(m, n, k, tri, tma, plan)) {
        r.kernel = DGEMM_WS_64;
        r.cluster = c;
        return r;
    }
    if (const int c = small_cluster(m, n, k, plan)) {
        r.kernel = DGEMM_CLUSTER_64;
        r.cluster = c;
        return r;
    }
    if (plan.tile == TILE_128x128 && tma) {
        r.kernel = DGEMM_TMA_128;
        r.k_chunk = dgemm_tma_k_chunk(k, splits);
        r.ranges = (k + r.k_chunk - 1) / r.k_chunk;
        if (r.ranges == 2 && plan.automatic) {
            r.cluster = 2;
            r.ranges = 1;
        }
        return r;
    }
    r.kernel = DGEMM_TILES;
    r.k_chunk = ((k + splits - 1) / splits + kDgemmSlice - 1) / kDgemmSlice * kDgemmSlice;
    r.ranges = (k + r.k_chunk - 1) / r.k_chunk;
    return r;
}

// The largest cluster with at most one CTA per SM and 16-deep ranges, where its CTAs then have
// less to do than the plan's: (K / c) x 64 columns against (K / splits) x 128 (1024^3: c = 1
// against two K ranges, 65 against 61 us, keeps the plan; 300 x 300 x 4000, c = 8 against 15:
// 36.9 / 37.1; 256 x 256 x 262144, c = 8 against 37, keeps it).  Clusters that share SMs have
// half the rate: they need shorter ranges than the plan's (18 tiles, c = 8: k = 1500, five
// ranges, 1.5 x; 2048, eight, 0.97; 4000, fifteen, 0.64.  36 tiles, c = 4: k = 511 2.9 x, 1500,
// five ranges, 0.91).
SgemmRoute sgemm_tile_route(int m, int n, int k, const GemmPlan& plan) {
    SgemmRoute r;
    const int splits = std::max(1, plan.splits);
    const long t = (long)((m + 127) / 128) * ((n + 63) / 64);
    for (int c = 8; c >= 1; c /= 2)
        if (c * t <= plan.sm_count && (c == 1 || k >= 16 * c)) {
            const bool alone = c * t <= cluster_ctas(c, plan.sm_count);
            r.cluster = (alone ? 2 * c : c) > splits ? c : 0;
            r.halves = r.cluster && c < splits;
            break;
        }
    return r;
}

}  // namespace zb
