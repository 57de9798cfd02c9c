// Native FP64 GEMM on 64 x 64 tiles, warp-specialised, K split inside a cluster (sm_100a).
//
//   C = alpha * op(A) * op(B) + beta * C     (column-major, any lda / ldb / ldc)
//
// The contraction of gemm_f64.cu / gemm_f64_tma.cu (the reference's packed-SIMD
// body, kernels/shared/matrix_matrix/packed_simd.zig:306) for TMA-describable
// operands whose 128 x 128 tiles fill the last wave of SMs badly.  Bound: the
// FP64 tensor pipe.  A quarter-size tile deals the work in quarter-size steps:
// 2048^3 is 1.73 waves of 128 x 128 tiles (two take the time) but 6.92 rounds
// of 64 x 64 tiles, 559 -> 517 us; DMMA pipe 91 % of active cycles.
//
// One producer warp feeds 16-deep K slices by TMA into a four-slice ring (64 KB),
// four math warps (2 x 2 of 32 x 32) run DMMA on them, three CTAs per SM: an
// mma.sync m16n8k8 .f64 holds its warp's issue for the 64 cycles it occupies
// the sub-partition's pipe, so a warp's fragment loads and barrier polls are
// only hidden by other warps' products, and three CTAs in different phases hide
// them better than one CTA's warps in step (64 x 64 x 4096 on one CTA per SM
// runs at 0.71 of the pipe, three CTAs at 0.91).
//
// With about one tile per SM, K is split over a cluster of two CTAs: each leaves its
// partial tile in shared memory and sums half of the columns of both through
// distributed shared memory, in rank order (deterministic); no workspace and no
// second launch (1024 x 512 x 1024, beta 1: 49.5 -> 45.0 us against cp.async
// tiles with a reduction kernel; 1000 x 500 x 300: 20.3 -> 18.3).
#include "bounded_wait.cuh"
#include "common.cuh"
#include "kernels.h"
#include "ozaki.h"

namespace zb {
namespace {

constexpr int kWM = 64, kWN = 64, kWK = 16, kWStages = 4;
constexpr int kWMathWarps = 4;                      // 2 x 2 warps of 32 x 32
constexpr int kWThreads = (kWMathWarps + 1) * 32;   // + a producer warp (one TMA thread)
constexpr int kWOpBytes = kWM * kWK * 8;            // 8 KB per operand and stage
constexpr int kWStageBytes = 2 * kWOpBytes;
constexpr int kWPitch = kWM + 2;                    // partial tile [column][row]
constexpr size_t kWSmem = 1024 + (size_t)kWStages * kWStageBytes + 128;
static_assert(kWN * kWPitch * 8 <= kWStages * kWStageBytes, "the partial tile reuses the ring");
constexpr unsigned long long kWWaitNs = 4000000000ull;

struct WsParams {
    int M, N, K, k_chunk, tri;
    double alpha, beta;
    double* C;
    long ldc;
    int* report;
    unsigned long long wait_ns;
};

// Byte offsets of an element in the two tile orientations (128-byte rows, the
// 16-byte chunk index XORed with the row index mod 8, as TMA's 128-byte swizzle).
//   MN-major: four boxes of 16 k-rows x 16 elements; K-major: 64 rows x 16 k.
ZB_DEVICE uint32_t ws_mn_off(int mn, int k) {
    return (uint32_t)((mn >> 4) * 2048 + k * 128 + ((((mn & 15) >> 1) ^ (k & 7)) << 4) + ((mn & 1) << 3));
}
ZB_DEVICE uint32_t ws_k_off(int mn, int k) {
    return (uint32_t)(mn * 128 + (((k >> 1) ^ (mn & 7)) << 4) + ((k & 1) << 3));
}

ZB_DEVICE void ld_cluster_f64x2(uint32_t addr, double& x, double& y) {
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];\n" : "=d"(x), "=d"(y) : "r"(addr) : "memory");
}
ZB_DEVICE int ld_cluster_s32(uint32_t addr) {
    int v;
    asm volatile("ld.shared::cluster.s32 %0, [%1];\n" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
template <bool A_MN, bool B_K>
__global__ void __launch_bounds__(kWThreads, 3)
dgemm_ws_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                const __grid_constant__ WsParams P) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + kWStages * kWStageBytes);
    uint64_t* empty = full + kWStages;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(empty + kWStages);

    const int m0 = blockIdx.x * kWM, n0 = blockIdx.y * kWN;
    // triangle mode: the whole cluster leaves a tile that holds no element of the stored triangle
    if ((P.tri == 1 && m0 > n0 + kWN - 1) || (P.tri == 2 && m0 + kWM - 1 < n0)) return;
    const int splits = gridDim.z, rank = blockIdx.z;  // the cluster spans gridDim.z
    const int kb = rank * P.k_chunk;
    const int ke = min(P.K, kb + P.k_chunk);
    const int KT = max(0, (ke - kb + kWK - 1) / kWK);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kWStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kWMathWarps);
        }
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == kWMathWarps && lane == 0) {
        prefetch_tmap(&tmA);
        prefetch_tmap(&tmB);
    }
    __syncthreads();
    // launched during the tail of the kernel before it (which may write A, B or C)
    grid_dependency_wait();
    const WaitCtl W{abort_flag, nullptr, P.report, P.wait_ns};

    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    const int g = lane >> 2, t = lane & 3;
    double acc[2][4][4];
    if (warp >= kWMathWarps) {
        // ---------------------------------------------------------- producer
        if (lane == 0) {
            bool ok = true;
            int s = 0;
            uint32_t ph = 0;
            Issued issued;
            for (int kt = 0; kt < KT; ++kt) {
                if (!(ok = wait_phase(&empty[s], ph ^ 1u, W, WAIT_PRODUCER_EMPTY_A))) break;
                const uint32_t sa = smem_u32(smem + s * kWStageBytes), sb = sa + kWOpBytes;
                const int k0 = kb + kt * kWK;
                mbar_arrive_expect_tx(&full[s], kWStageBytes);
                if (A_MN) {
#pragma unroll
                    for (int b = 0; b < kWM / 16; ++b) tma_load_2d(sa + b * 2048, &tmA, &full[s], m0 + 16 * b, k0);
                } else {
                    tma_load_2d(sa, &tmA, &full[s], k0, m0);
                }
                if (B_K) {
                    tma_load_2d(sb, &tmB, &full[s], k0, n0);
                } else {
#pragma unroll
                    for (int b = 0; b < kWN / 16; ++b) tma_load_2d(sb + b * 2048, &tmB, &full[s], n0 + 16 * b, k0);
                }
                issued.note(s, ph);
                if (++s == kWStages) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            // aborted: the bytes of every issued copy land before shared memory is reused
            if (!ok) issued.drain(full, kWStages, P.wait_ns);
        }
    } else {
        // -------------------------------------------------------- math warps
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int v = 0; v < 4; ++v) acc[i][j][v] = 0.0;
        // fragment offsets as in dgemm_tma_kernel: MMA row r = g + 8 v reads physical row
        // 2 g + v, k index kappa physical k 2 (kappa mod 4) + kappa / 4, and for a K-major
        // op(B) column n physical column (n >> 1) | ((n & 1) << 2)
        uint32_t a_off[2][2], b_off[4][2];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int v = 0; v < 2; ++v)
                a_off[i][v] = A_MN ? ws_mn_off(wm + 16 * i + 2 * g, 2 * t + v) : ws_k_off(wm + 16 * i + 2 * g + v, 2 * t);
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int v = 0; v < 2; ++v)
                b_off[j][v] = kWOpBytes + (B_K ? ws_k_off(wn + 8 * j + ((g >> 1) | ((g & 1) << 2)), 2 * t)
                                               : ws_mn_off(wn + 8 * j + g, 2 * t + v));
        int s = 0;
        uint32_t ph = 0;
        for (int kt = 0; kt < KT; ++kt) {
            if (!wait_phase(&full[s], ph, W, WAIT_MMA_FULL_A)) break;
            const uint8_t* st = smem + s * kWStageBytes;
#pragma unroll
            for (int ks = 0; ks < kWK; ks += 8) {
                const uint32_t mn_step = ks * 128, k_xor = (ks >> 1) << 4;
                double af[2][4], bf[4][2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    if (A_MN) {
                        const double2 p0 = *reinterpret_cast<const double2*>(st + a_off[i][0] + mn_step);
                        const double2 p1 = *reinterpret_cast<const double2*>(st + a_off[i][1] + mn_step);
                        af[i][0] = p0.x, af[i][1] = p0.y, af[i][2] = p1.x, af[i][3] = p1.y;
                    } else {
                        const double2 p0 = *reinterpret_cast<const double2*>(st + (a_off[i][0] ^ k_xor));
                        const double2 p1 = *reinterpret_cast<const double2*>(st + (a_off[i][1] ^ k_xor));
                        af[i][0] = p0.x, af[i][2] = p0.y, af[i][1] = p1.x, af[i][3] = p1.y;
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (B_K) {
                        const double2 q = *reinterpret_cast<const double2*>(st + (b_off[j][0] ^ k_xor));
                        bf[j][0] = q.x, bf[j][1] = q.y;
                    } else {
                        bf[j][0] = *reinterpret_cast<const double*>(st + b_off[j][0] + mn_step);
                        bf[j][1] = *reinterpret_cast<const double*>(st + b_off[j][1] + mn_step);
                    }
                }
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) dmma_16x8x8(acc[i][j], af[i], bf[j]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[s]);
            if (++s == kWStages) {
                s = 0;
                ph ^= 1u;
            }
        }
    }
    __syncthreads();  // every slice consumed, no copy in flight: the ring becomes the partial tile

    double* T = reinterpret_cast<double*>(smem);
    if (warp < kWMathWarps) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const int r = wm + 16 * i + 2 * g + (v >> 1);
                    const int c = wn + 8 * j + (B_K ? t + 4 * (v & 1) : 2 * t + (v & 1));
                    T[c * kWPitch + r] = acc[i][j][v];
                }
    }
    if (splits > 1)
        cluster_sync();
    else
        __syncthreads();
    // CTA `rank` sums its columns of the tile over the ranks, in rank order, and writes
    // them; nothing is written when a wait of any rank ran out
    bool ok = true;
    if (splits == 1) {
        ok = !*abort_flag;
    } else {
        const uint32_t flag = smem_u32(const_cast<int*>(abort_flag));
        for (int z = 0; z < splits; ++z) ok = ok && ld_cluster_s32(mapa_shared(flag, z)) == 0;
    }
    const int cols = kWN / splits, c_first = rank * cols;
    for (int q = threadIdx.x; ok && q < cols * (kWM / 2); q += kWThreads) {
        const int r = (q % (kWM / 2)) * 2, c = c_first + q / (kWM / 2);
        const int row = m0 + r, col = n0 + c;
        if (row >= P.M || col >= P.N) continue;
        double* cp = P.C + (long)col * P.ldc + row;
        const bool in0 = P.tri == 0 || (P.tri == 1 ? row <= col : row >= col);
        const bool in1 = row + 1 < P.M && (P.tri == 0 || (P.tri == 1 ? row + 1 <= col : row + 1 >= col));
        double c0 = 0.0, c1 = 0.0;
        if (P.beta != 0.0) {
            if (in0) c0 = cp[0];
            if (in1) c1 = cp[1];
        }
        double x0 = 0.0, x1 = 0.0;
        if (splits == 1) {
            x0 = T[c * kWPitch + r];
            x1 = T[c * kWPitch + r + 1];
        } else {
            const uint32_t at = smem_u32(T + c * kWPitch + r);
            for (int z = 0; z < splits; ++z) {
                double y0, y1;
                ld_cluster_f64x2(mapa_shared(at, z), y0, y1);
                x0 += y0;
                x1 += y1;
            }
        }
        x0 *= P.alpha;
        x1 *= P.alpha;
        if (P.beta != 0.0) {
            x0 = fma(P.beta, c0, x0);
            x1 = fma(P.beta, c1, x1);
        }
        if (in0) cp[0] = x0;
        if (in1) cp[1] = x1;
    }
    if (splits > 1) cluster_sync();  // no CTA leaves while its partial tile may be read
}

template <bool A_MN, bool B_K>
cudaError_t launch_ws(const CUtensorMap& ma, const CUtensorMap& mb, const WsParams& P, int splits, cudaStream_t st) {
    auto kern = dgemm_ws_kernel<A_MN, B_K>;
    cudaError_t e = ensure_dynamic_smem(kern, (int)kWSmem);
    if (e != cudaSuccess) return e;
    const dim3 grid((P.M + kWM - 1) / kWM, (P.N + kWN - 1) / kWN, splits);
    prof_begin(st);
    e = launch_dependent_cluster(kern, grid, dim3(kWThreads), kWSmem, st, dim3(1, 1, splits), ma, mb, P);
    count_launch();
    prof_end(st);
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace

cudaError_t dgemm_ws(const GemmArgsF64& g, int splits, cudaStream_t st) {
    const bool a_mn = g.transa == 'N', b_k = g.transb == 'N';
    if (splits != 1 && splits != 2) return cudaErrorInvalidValue;
    CUtensorMap ma, mb;
    cudaError_t e = a_mn ? make_f64_map(&ma, g.a, g.m, g.k, g.lda, kWK) : make_f64_map(&ma, g.a, g.k, g.m, g.lda, kWM);
    if (e != cudaSuccess) return e;
    e = b_k ? make_f64_map(&mb, g.b, g.k, g.n, g.ldb, kWN) : make_f64_map(&mb, g.b, g.n, g.k, g.ldb, kWK);
    if (e != cudaSuccess) return e;
    WsParams P{g.m, g.n, g.k, 0, g.tri, g.alpha, g.beta, g.c, g.ldc, nullptr, kWWaitNs};
    P.k_chunk = ((g.k + splits - 1) / splits + kWK - 1) / kWK * kWK;
    if ((e = wait_report_word(&P.report)) != cudaSuccess) return e;
    if (a_mn && b_k) return launch_ws<true, true>(ma, mb, P, splits, st);
    if (a_mn) return launch_ws<true, false>(ma, mb, P, splits, st);
    if (b_k) return launch_ws<false, true>(ma, mb, P, splits, st);
    return launch_ws<false, false>(ma, mb, P, splits, st);
}

}  // namespace zb
