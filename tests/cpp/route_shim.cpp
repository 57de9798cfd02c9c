// C entry points over the planner's routing rules (host code, linked with csrc/planner.cpp).
#include "kernels.h"

namespace zb {
// of the matrix-vector and narrow kernels, whose shapes are not asked for here
int gemv_split_count(int, int) { return 1; }
int narrow_split_count(int, int, int, int) { return 1; }
}  // namespace zb

// out: tile, planned splits, kernel, cluster, ranges, k_chunk
extern "C" void dgemm_route(int m, int n, int k, int tri, int tma, int automatic, int sms, int* out) {
    zb::GemmPlan p = zb::plan_native_gemm(m, n, k, 8, sms);
    p.automatic = automatic != 0;
    const zb::DgemmRoute r = zb::dgemm_tile_route(m, n, k, tri, tma != 0, p);
    const int v[6] = {p.tile, p.splits, r.kernel, r.cluster, r.ranges, r.k_chunk};
    for (int i = 0; i < 6; ++i) out[i] = v[i];
}

// out: planned splits, cluster, halves
extern "C" void sgemm_route(int m, int n, int k, int sms, int* out) {
    const zb::GemmPlan p = zb::plan_native_gemm(m, n, k, 4, sms);
    const zb::SgemmRoute r = zb::sgemm_tile_route(m, n, k, p);
    out[0] = p.splits, out[1] = r.cluster, out[2] = r.halves;
}
