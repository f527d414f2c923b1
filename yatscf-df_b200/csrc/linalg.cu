// Dense FP64 building blocks for the SCF: a tiled DGEMM, inverse square
// roots from eigenpairs (TinySCF.c:58-76, build_DF_tensor.c:205-237), and the
// pivoted Cholesky of the initial guess (TinySCF.c:282-322, LAPACK dpstf2
// semantics). The eigensolver itself is in eigh.cu.
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstdint>
#include <cstdlib>
#include <map>
#include <mutex>

#include <utility>
#include <vector>

#include "fork.h"
#include "tiles.cuh"
#include "tune.h"
#include "tscf_internal.h"
#include "umma.cuh"

namespace tscf {

std::atomic<long long> g_launches{0}, g_bulk_gemms{0};

// the pools of fork.h outlive static destruction
std::mutex &Fork::lock()
{
    static std::mutex *m = new std::mutex;
    return *m;
}
std::vector<Fork::Set *> &Fork::pool(int dev)
{
    static auto *p = new std::map<int, std::vector<Set *>>;
    return (*p)[dev];
}

// ------------------------------------------------------------------ DGEMM
// Five tile shapes: FFMA 64x64 (default), 32x32 (more blocks for small
// matrices) and 128x64 (more reuse for large ones) (dgemm_tile), and 128x128
// and 64x64 on the FP64 tensor cores (dgemm_tile_dmma, dgemm_tile_dmma64). The
// autotuner picks one per call shape the first time the shape is met outside
// a stream capture; they sum over k in the same order. A sixth, K split over
// warps (k_dgemm_dmma32ks), rounds differently and goes by a rule (ksplit_order).
template <bool TA, bool TB, int BM, int BN>
__global__ void __launch_bounds__(256) k_dgemm(int m, int n, int k, double alpha, const double *__restrict__ A, int lda,
                                               const double *__restrict__ B, int ldb, double beta, double *C, int ldc)
{
    dgemm_tile<TA, TB, BM, BN>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, blockIdx.y * BM, blockIdx.x * BN);
}

template <int BM, int BN>
static void dgemm_shape(bool ta, bool tb, int m, int n, int k, double alpha, const double *A, int lda,
                        const double *B, int ldb, double beta, double *C, int ldc, cudaStream_t s)
{
    dim3 grid((n + BN - 1) / BN, (m + BM - 1) / BM);
    g_launches++;
    if (!ta && !tb) k_dgemm<false, false, BM, BN><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    else if (!ta && tb) k_dgemm<false, true, BM, BN><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    else if (ta && !tb) k_dgemm<true, false, BM, BN><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    else k_dgemm<true, true, BM, BN><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
}

template <bool TA, bool TB>
__global__ void __launch_bounds__(256, 1) k_dgemm_dmma(int m, int n, int k, double alpha, const double *__restrict__ A,
                                                       int lda, const double *__restrict__ B, int ldb, double beta,
                                                       double *C, int ldc)
{
    dgemm_tile_dmma<TA, TB>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, blockIdx.y * 128, blockIdx.x * 128);
}

static bool dgemm_bulk_fits(bool ta, bool tb, int m, int n, int k, const double *A, int lda, const double *B, int ldb,
                            double beta, const double *C, int ldc);
static bool dgemm_bulk(int m, int n, int k, double alpha, const double *A, int lda, const double *B, int ldb, double *C,
                       int ldc, cudaStream_t s);

static void dgemm_dmma(bool ta, bool tb, int m, int n, int k, double alpha, const double *A, int lda, const double *B,
                       int ldb, double beta, double *C, int ldc, cudaStream_t s)
{
    if (dgemm_bulk_fits(ta, tb, m, n, k, A, lda, B, ldb, beta, C, ldc) && dgemm_bulk(m, n, k, alpha, A, lda, B, ldb, C, ldc, s))
        return;
    dim3 grid((n + 127) / 128, (m + 127) / 128);
    g_launches++;
    if (!ta && !tb) k_dgemm_dmma<false, false><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    else if (!ta && tb) k_dgemm_dmma<false, true><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    else if (ta && !tb) k_dgemm_dmma<true, false><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    else k_dgemm_dmma<true, true><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
}

// ---- the same product for large A B with row-major operands in whole 16-byte
// units: 168 x 96 tiles over 12 warps of 56 x 24 in a persistent CTA per SM,
// fed by a producer warp (the fourth warp of one SM quarter, which leaves each
// 128 registers). Lane 0 of it loads 32-wide K chunks by TMA, two chunks ahead,
// behind mbarriers, so the other warps issue nothing but fragment reads and
// DMMAs and never wait for one another. Neighbouring CTAs take the tiles of one
// row block, so A comes from HBM once and B stays in L2. Each output is one FMA
// chain over k, as in every other tile but the K-split one: the same bits.
// DMMA rate bounds it: C40H82's DF tensor (122,420 x 3870 x 3870) takes 105 ms,
// 34.9 TF/s or 94% of that rate, against 133 ms on the 128 x 128 tile above. With
// one untiled bulk copy per row (256 B of A, 768 B of B) instead of tensor boxes
// it took 145 ms.
// Shared memory: boxes of 16 doubles (128 B) a row in the 128-byte swizzle, two of
// 168 rows of A, six of 32 rows of B. Fragment row fr is tile row perm(fr), and
// fragment column fr is column colperm(fr) of a 16-column box, such that the 16
// lanes of a half-warp read 16 different bank pairs.
constexpr int BG_WM = 3, BG_NX = 7, BG_WN = 4, BG_NY = 3;
constexpr int BG_M = BG_WM * BG_NX * 8, BG_N = BG_WN * BG_NY * 8, BG_K = 32;
constexpr int BG_WARPS = BG_WM * BG_WN, BG_THREADS = (BG_WARPS + 1) * 32, BG_STAGES = 3;
constexpr int BG_ABOX = BG_M * 16, BG_BBOX = BG_K * 16;   // doubles
constexpr int BG_STAGE = BG_K / 16 * BG_ABOX + BG_N / 16 * BG_BBOX;
constexpr size_t BG_SMEM = sizeof(double) * BG_STAGES * BG_STAGE + 1024;
constexpr long long BG_WAIT = 2000000000LL;   // clock cycles a barrier wait may take (~1 s)
static_assert(BG_SMEM + 64 <= 227 * 1024 && BG_M <= 256, "bulk GEMM stages exceed shared memory");
static_assert(BG_ABOX % 128 == 0 && BG_BBOX % 128 == 0, "swizzled boxes start at multiples of 1024 bytes");

__global__ void __launch_bounds__(BG_THREADS, 1)
    k_dgemm_bulk(const __grid_constant__ CUtensorMap mA, const __grid_constant__ CUtensorMap mB, int m, int n, int k,
                 double alpha, double *__restrict__ C, int ldc, int ntn, int ntiles, int *gave_up)
{
    extern __shared__ __align__(1024) unsigned char bg_raw[];
    double *bgsm = (double *) (((uintptr_t) bg_raw + 1023) & ~(uintptr_t) 1023);
    __shared__ uint64_t full[BG_STAGES], empty[BG_STAGES];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int q = 0; q < BG_STAGES; q++) {
            umma::mbar_init(&full[q], 1);
            umma::mbar_init(&empty[q], BG_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async;" ::: "memory");
    }
    __syncthreads();
    int st = 0, phase = 0;
    if (warp == BG_WARPS) {   // ---- producer
        if (lane != 0) return;
        bool first = true;    // the first BG_STAGES chunks find their stage empty
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
            const int m0 = t / ntn * BG_M, n0 = t % ntn * BG_N;
            for (int k0 = 0; k0 < k; k0 += BG_K) {
                if (!first && !umma::mbar_wait_bounded(&empty[st], phase ^ 1, gave_up, 41, BG_WAIT)) {
                    for (int q = 0; q < BG_STAGES; q++) {   // its copies in flight, oldest first
                        umma::mbar_wait_bounded(&full[st], phase ^ 1, gave_up, 42, BG_WAIT);
                        if (++st == BG_STAGES) {
                            st = 0;
                            phase ^= 1;
                        }
                    }
                    return;
                }
                double *As = bgsm + (size_t) st * BG_STAGE, *Bs = As + BG_K / 16 * BG_ABOX;
                umma::mbar_expect_tx(&full[st], (unsigned) (sizeof(double) * BG_STAGE));
#pragma unroll
                for (int q = 0; q < BG_K / 16; q++) umma::tma_load_2d(As + q * BG_ABOX, &mA, &full[st], k0 + 16 * q, m0);
#pragma unroll
                for (int q = 0; q < BG_N / 16; q++) umma::tma_load_2d(Bs + q * BG_BBOX, &mB, &full[st], n0 + 16 * q, k0);
                if (++st == BG_STAGES) {
                    st = 0;
                    phase ^= 1;
                    first = false;
                }
            }
        }
        return;
    }
    const int wm = (warp / BG_WN) * BG_NX * 8, f0 = (warp % BG_WN) * BG_NY;   // f0: first 8-column fragment
    const int fr = lane >> 2, fc = lane & 3, perm = (2 * fr & 7) | (fr >> 2);
    // element (r, kk) of A's box: 16 r + 2 ((kk / 2) ^ (r & 7)) + kk % 2; B's (kk, c) alike
    const int oa = (wm + perm) * 16 + (((fc >> 1) ^ perm) << 1) + (fc & 1);
    int ob[BG_NY];
#pragma unroll
    for (int y = 0; y < BG_NY; y++) {
        const int f = f0 + y, chunk = ((f & 1) << 1) | ((fr & 2) << 1) | (fr >> 2);
        ob[y] = (f >> 1) * BG_BBOX + fc * 16 + ((chunk ^ fc) << 1) + (fr & 1);
    }
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int m0 = t / ntn * BG_M, n0 = t % ntn * BG_N;
        double acc[BG_NX][BG_NY][2];
#pragma unroll
        for (int x = 0; x < BG_NX; x++)
#pragma unroll
            for (int y = 0; y < BG_NY; y++) acc[x][y][0] = acc[x][y][1] = 0.0;
        for (int k0 = 0; k0 < k; k0 += BG_K) {
            if (!umma::mbar_wait_bounded(&full[st], phase, gave_up, 43, BG_WAIT)) return;
            const double *As = bgsm + (size_t) st * BG_STAGE, *Bs = As + BG_K / 16 * BG_ABOX;
#pragma unroll
            for (int k4 = 0; k4 < BG_K; k4 += 4) {   // zeros behind k, m and n
                double a[BG_NX], b[BG_NY];
                const double *ap = As + k4 / 16 * BG_ABOX + (oa ^ (k4 % 16));
#pragma unroll
                for (int x = 0; x < BG_NX; x++) a[x] = ap[128 * x];
#pragma unroll
                for (int y = 0; y < BG_NY; y++) b[y] = Bs[(ob[y] ^ (2 * (k4 & 4))) + 16 * k4];
#pragma unroll
                for (int x = 0; x < BG_NX; x++)
#pragma unroll
                    for (int y = 0; y < BG_NY; y++) dmma_8x8x4(acc[x][y][0], acc[x][y][1], a[x], b[y]);
            }
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(&empty[st]);
            if (++st == BG_STAGES) {
                st = 0;
                phase ^= 1;
            }
        }
#pragma unroll
        for (int x = 0; x < BG_NX; x++) {
            const int gi = m0 + wm + 8 * x + perm;
#pragma unroll
            for (int y = 0; y < BG_NY; y++) {
                const int f = f0 + y, gj = n0 + (f >> 1) * 16 + 4 * (f & 1) + 8 * (fc & 1) + 2 * (fc >> 1);
                if (gi < m && gj < n)
                    *reinterpret_cast<double2 *>(C + (size_t) gi * ldc + gj) =
                        make_double2(alpha * acc[x][y][0], alpha * acc[x][y][1]);
            }
        }
    }
}

// Whether k_dgemm_bulk takes the product: 16-byte units throughout, C written
// only, and its waves of 168 x 96 tiles at 94% of the DMMA rate cost less than
// those of 128 x 128 tiles at 75%. Measured, bulk against 128 x 128 (ms):
// 1010^3 0.144 / 0.186, 1680^3 0.460 / 0.588, 1950^3 0.526 / 0.685, 3072^3
// 2.04 / 2.12, 3870^3 3.58 / 4.66, 33600 x 960 x 960 1.81 / 2.52, 3870 x 3870 x 64
// 0.087 / 0.127; where its last wave is nearly empty (2688^3, 3.03 waves)
// 1.43 / 1.40, which the rule leaves to the 128 x 128 tile.
static bool dgemm_bulk_fits(bool ta, bool tb, int m, int n, int k, const double *A, int lda, const double *B, int ldb,
                            double beta, const double *C, int ldc)
{
    if (ta || tb || beta != 0.0 || k < BG_K || ((lda | ldb | ldc | n | k) & 1)) return false;
    if (((uintptr_t) A | (uintptr_t) B | (uintptr_t) C) & 15) return false;
    const long long nsm = num_sms();
    const long long tiles = (long long) ((m + BG_M - 1) / BG_M) * ((n + BG_N - 1) / BG_N);
    const long long old = (long long) ((m + 127) / 128) * ((n + 127) / 128);
    const double waves = (double) ((tiles + nsm - 1) / nsm), old_waves = (double) ((old + nsm - 1) / nsm);
    return tiles < (1LL << 31) && waves * (BG_M * BG_N) / 0.94 < old_waves * (128 * 128) / 0.75;
}

static bool dgemm_bulk(int m, int n, int k, double alpha, const double *A, int lda, const double *B, int ldb, double *C,
                       int ldc, cudaStream_t s)
{
    CUtensorMap mA, mB;
    if (!wait_word() || !umma::make_map_2d(&mA, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, A, m, k, lda, 16, BG_M) ||
        !umma::make_map_2d(&mB, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, B, k, n, ldb, 16, BG_K))
        return false;
    if (cudaFuncSetAttribute(k_dgemm_bulk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) BG_SMEM) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    const int ntn = (n + BG_N - 1) / BG_N, ntiles = ntn * ((m + BG_M - 1) / BG_M);
    k_dgemm_bulk<<<std::min(ntiles, num_sms()), BG_THREADS, BG_SMEM, s>>>(mA, mB, m, n, k, alpha, C, ldc, ntn, ntiles,
                                                                               wait_word());
    g_launches++;
    g_bulk_gemms++;
    return true;
}

template <bool TA, bool TB>
__global__ void __launch_bounds__(128) k_dgemm_dmma64(int m, int n, int k, double alpha, const double *__restrict__ A,
                                                      int lda, const double *__restrict__ B, int ldb, double beta,
                                                      double *C, int ldc)
{
    dgemm_tile_dmma64<TA, TB>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, blockIdx.y * 64, blockIdx.x * 64);
}

static void dgemm_dmma64(bool ta, bool tb, int m, int n, int k, double alpha, const double *A, int lda,
                         const double *B, int ldb, double beta, double *C, int ldc, cudaStream_t s)
{
    dim3 grid((n + 63) / 64, (m + 63) / 64);
    g_launches++;
    if (!ta && !tb) k_dgemm_dmma64<false, false><<<grid, 128, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    else if (!ta && tb) k_dgemm_dmma64<false, true><<<grid, 128, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    else if (ta && !tb) k_dgemm_dmma64<true, false><<<grid, 128, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    else k_dgemm_dmma64<true, true><<<grid, 128, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
}

// ---- 32 x 32 output tile per 256 threads on the FP64 tensor cores, the K
// range split over the 8 warps: for the tall-skinny and small products of the
// density refinement, DIIS and orbital alignment (n x n_occ outputs, n_occ^2
// outputs with K = n), where the 64/128 tiles leave most SMs idle and a
// single warp per tile would run the whole K loop alone. Each 64-wide K chunk
// is prefetched into registers while the previous one is multiplied (warp w
// takes chunk rows 8w..8w+7); the eight partial tiles are summed through
// shared memory in a fixed order.
constexpr int KS_T = 32, KS_K = 64, KS_LD = KS_K + 4;

template <bool TA, bool TB>
__global__ void __launch_bounds__(256) k_dgemm_dmma32ks(int m, int n, int k, double alpha,
                                                        const double *__restrict__ A, int lda,
                                                        const double *__restrict__ B, int ldb, double beta,
                                                        double *C, int ldc)
{
    __shared__ double sm[2 * KS_T * KS_LD];   // As[32][68], Bs[32][68]; then the partial-tile slots
    double *As = sm, *Bs = sm + KS_T * KS_LD;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int fr = lane >> 2, fc = lane & 3;
    const int m0 = blockIdx.y * KS_T, n0 = blockIdx.x * KS_T;
    double acc[4][4][2];
#pragma unroll
    for (int x = 0; x < 4; x++)
#pragma unroll
        for (int y = 0; y < 4; y++) acc[x][y][0] = acc[x][y][1] = 0.0;
    double pa[8], pb[8];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const int l = tid + 256 * r;
            int row, kk;
            if (!TA) { row = l / KS_K; kk = l % KS_K; } else { kk = l / KS_T; row = l % KS_T; }
            const int gi = m0 + row, gk = k0 + kk;
            pa[r] = (gi < m && gk < k) ? (TA ? A[(size_t) gk * lda + gi] : A[(size_t) gi * lda + gk]) : 0.0;
            int col;
            if (!TB) { kk = l / KS_T; col = l % KS_T; } else { col = l / KS_K; kk = l % KS_K; }
            const int gj = n0 + col, gk2 = k0 + kk;
            pb[r] = (gj < n && gk2 < k) ? (TB ? B[(size_t) gj * ldb + gk2] : B[(size_t) gk2 * ldb + gj]) : 0.0;
        }
    };
    fetch(0);
    for (int k0 = 0; k0 < k; k0 += KS_K) {
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const int l = tid + 256 * r;
            if (!TA) As[(l / KS_K) * KS_LD + l % KS_K] = pa[r];
            else As[(l % KS_T) * KS_LD + l / KS_T] = pa[r];
            if (!TB) Bs[(l % KS_T) * KS_LD + l / KS_T] = pb[r];
            else Bs[(l / KS_K) * KS_LD + l % KS_K] = pb[r];
        }
        __syncthreads();
        if (k0 + KS_K < k) fetch(k0 + KS_K);
#pragma unroll
        for (int k4 = 0; k4 < 8; k4 += 4) {
            const int kc = 8 * warp + k4 + fc;
            double a[4], b[4];
#pragma unroll
            for (int x = 0; x < 4; x++) a[x] = As[(8 * x + fr) * KS_LD + kc];
#pragma unroll
            for (int y = 0; y < 4; y++) b[y] = Bs[(8 * y + fr) * KS_LD + kc];
#pragma unroll
            for (int x = 0; x < 4; x++)
#pragma unroll
                for (int y = 0; y < 4; y++) dmma_8x8x4(acc[x][y][0], acc[x][y][1], a[x], b[y]);
        }
        __syncthreads();
    }
    // warps 4-7 into 0-3, then 2-3 into 0-1, then 1 into 0 (slots of 32 x 32 per warp)
    double *red = sm;
    for (int half = 4; half >= 1; half >>= 1) {
        if (warp >= half && warp < 2 * half) {
#pragma unroll
            for (int x = 0; x < 4; x++)
#pragma unroll
                for (int y = 0; y < 4; y++)
#pragma unroll
                    for (int h = 0; h < 2; h++) red[(warp - half) * 1024 + ((x * 4 + y) * 2 + h) * 32 + lane] = acc[x][y][h];
        }
        __syncthreads();
        if (warp < half) {
#pragma unroll
            for (int x = 0; x < 4; x++)
#pragma unroll
                for (int y = 0; y < 4; y++)
#pragma unroll
                    for (int h = 0; h < 2; h++) acc[x][y][h] += red[warp * 1024 + ((x * 4 + y) * 2 + h) * 32 + lane];
        }
        __syncthreads();
    }
    if (warp != 0) return;
#pragma unroll
    for (int x = 0; x < 4; x++) {
        const int gi = m0 + 8 * x + fr;
        if (gi >= m) continue;
#pragma unroll
        for (int y = 0; y < 4; y++) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int gj = n0 + 8 * y + 2 * fc + h;
                if (gj >= n) continue;
                double *c = C + (size_t) gi * ldc + gj;
                *c = (beta == 0.0) ? alpha * acc[x][y][h] : alpha * acc[x][y][h] + beta * *c;
            }
        }
    }
}

static void dgemm_dmma32ks(bool ta, bool tb, int m, int n, int k, double alpha, const double *A, int lda,
                           const double *B, int ldb, double beta, double *C, int ldc, cudaStream_t s)
{
    dim3 grid((n + KS_T - 1) / KS_T, (m + KS_T - 1) / KS_T);
    g_launches++;
    if (!ta && !tb) k_dgemm_dmma32ks<false, false><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    else if (!ta && tb) k_dgemm_dmma32ks<false, true><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    else if (ta && !tb) k_dgemm_dmma32ks<true, false><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    else k_dgemm_dmma32ks<true, true><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
}

static void dgemm_variant(int v, bool ta, bool tb, int m, int n, int k, double alpha, const double *A, int lda,
                          const double *B, int ldb, double beta, double *C, int ldc, cudaStream_t s)
{
    if (v == 5) dgemm_dmma32ks(ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
    else if (v == 4) dgemm_dmma64(ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
    else if (v == 3) dgemm_dmma(ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
    else if (v == 1) dgemm_shape<32, 32>(ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
    else if (v == 2) dgemm_shape<128, 64>(ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
    else dgemm_shape<64, 64>(ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
}

// ------------------------------------------------------------------ small products
// C = alpha op(A) op(B) for products too small to be worth tuning (m n k < 2e6):
// one output per thread in 16 x 16 tiles, K in chunks of 64 that are loaded one
// chunk ahead. They are latency-bound, and the 64 x 64 tile gives one of them
// a handful of CTAs with 16 outputs per thread and a barrier pair every 16 steps: a
// 60 x 60 x 60 product took 9.1 us, now 3.0 us. Each output is the same chain of
// multiply-adds over k, bit for bit.
constexpr int SM_T = 16, SM_K = 64;
template <bool TA, bool TB>
__global__ void __launch_bounds__(256) k_dgemm_small(int m, int n, int k, double alpha, const double *__restrict__ A,
                                                     int lda, const double *__restrict__ B, int ldb, double *C, int ldc)
{
    __shared__ double As[2][SM_K][SM_T + 1], Bs[2][SM_K][SM_T + 1];
    constexpr int NL = SM_K * SM_T / 256;
    const int tid = threadIdx.x, tx = tid % SM_T, ty = tid / SM_T;
    const int m0 = blockIdx.y * SM_T, n0 = blockIdx.x * SM_T;
    double ra[NL], rb[NL];
    auto load = [&](int k0) {
#pragma unroll
        for (int r = 0; r < NL; r++) {
            const int l = tid + 256 * r;
            const int ak = TA ? l / SM_T : l % SM_K, ar = TA ? l % SM_T : l / SM_K;
            const int bk = TB ? l % SM_K : l / SM_T, bc = TB ? l / SM_K : l % SM_T;
            const int gi = m0 + ar, gj = n0 + bc;
            ra[r] = (gi < m && k0 + ak < k) ? (TA ? A[(size_t) (k0 + ak) * lda + gi] : A[(size_t) gi * lda + k0 + ak]) : 0.0;
            rb[r] = (gj < n && k0 + bk < k) ? (TB ? B[(size_t) gj * ldb + k0 + bk] : B[(size_t) (k0 + bk) * ldb + gj]) : 0.0;
        }
    };
    load(0);
    double acc = 0.0;
    for (int k0 = 0, buf = 0; k0 < k; k0 += SM_K, buf ^= 1) {
#pragma unroll
        for (int r = 0; r < NL; r++) {
            const int l = tid + 256 * r;
            As[buf][TA ? l / SM_T : l % SM_K][TA ? l % SM_T : l / SM_K] = ra[r];
            Bs[buf][TB ? l % SM_K : l / SM_T][TB ? l / SM_K : l % SM_T] = rb[r];
        }
        __syncthreads();   // the other buffer's readers have passed the barrier of the chunk before
        if (k0 + SM_K < k) load(k0 + SM_K);
        const int kn = min(SM_K, k - k0);
        int kk = 0;
        for (; kk + 8 <= kn; kk += 8) {
#pragma unroll
            for (int q = 0; q < 8; q++) acc = fma(As[buf][kk + q][ty], Bs[buf][kk + q][tx], acc);
        }
        for (; kk < kn; kk++) acc = fma(As[buf][kk][ty], Bs[buf][kk][tx], acc);
    }
    if (m0 + ty < m && n0 + tx < n) C[(size_t) (m0 + ty) * ldc + n0 + tx] = alpha * acc;
}

static void dgemm_small(bool ta, bool tb, int m, int n, int k, double alpha, const double *A, int lda, const double *B,
                        int ldb, double *C, int ldc, cudaStream_t s)
{
    const dim3 grid((n + SM_T - 1) / SM_T, (m + SM_T - 1) / SM_T);
    g_launches++;
    if (!ta && !tb) k_dgemm_small<false, false><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, C, ldc);
    else if (!ta && tb) k_dgemm_small<false, true><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, C, ldc);
    else if (ta && !tb) k_dgemm_small<true, false><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, C, ldc);
    else k_dgemm_small<true, true><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, C, ldc);
}

// ------------------------------------------------------------------ Newton-Schulz iterations of small matrices
// The whole iteration of an o x o matrix in one CTA, matrices in shared memory
// (row pitch NS padded to 4, zeros in the padding): the occupied dimension of a
// small molecule makes each product a few us of latency, and launching three
// kernels per step cost more than the step (a water cluster's SCF iteration had
// 37 + 32 such launches per molecule and refinement step). 4 x 4 outputs per
// thread; each output is one chain of multiply-adds over k in order, as in
// dgemm's small products: the same bits.
constexpr int NS_THREADS = 512;
constexpr int NS_MAX = 84;   // 4 matrices of 84 x 84 doubles in 227 KB

// C = op(A) B over o terms; op(A)(i, k) = TA ? A[k][i] : A[i][k]; C must not be A or B.
template <bool TA>
__device__ __forceinline__ void ns_product(const double *A, const double *B, double *C, int o, int ld)
{
    const int nt = ld / 4;
    for (int t = threadIdx.x; t < nt * nt; t += NS_THREADS) {
        const int i0 = t / nt * 4, j0 = t % nt * 4;
        double acc[4][4] = {};
#pragma unroll 4
        for (int k = 0; k < o; k++) {
            double a[4];
            if (TA) {
                const double2 u = *reinterpret_cast<const double2 *>(A + k * ld + i0);
                const double2 v = *reinterpret_cast<const double2 *>(A + k * ld + i0 + 2);
                a[0] = u.x, a[1] = u.y, a[2] = v.x, a[3] = v.y;
            } else {
#pragma unroll
                for (int x = 0; x < 4; x++) a[x] = A[(i0 + x) * ld + k];
            }
            const double2 b0 = *reinterpret_cast<const double2 *>(B + k * ld + j0);
            const double2 b1 = *reinterpret_cast<const double2 *>(B + k * ld + j0 + 2);
#pragma unroll
            for (int x = 0; x < 4; x++) {
                acc[x][0] = fma(a[x], b0.x, acc[x][0]);
                acc[x][1] = fma(a[x], b0.y, acc[x][1]);
                acc[x][2] = fma(a[x], b1.x, acc[x][2]);
                acc[x][3] = fma(a[x], b1.y, acc[x][3]);
            }
        }
#pragma unroll
        for (int x = 0; x < 4; x++) {
            *reinterpret_cast<double2 *>(C + (i0 + x) * ld + j0) = make_double2(acc[x][0], acc[x][1]);
            *reinterpret_cast<double2 *>(C + (i0 + x) * ld + j0 + 2) = make_double2(acc[x][2], acc[x][3]);
        }
    }
    __syncthreads();
}
// M <- 1.5 I - 0.5 M (the padding stays zero)
__device__ __forceinline__ void ns_flip(double *M, int o, int ld)
{
    for (int l = threadIdx.x; l < o * o; l += NS_THREADS) {
        const int i = l / o, j = l - i * o;
        M[i * ld + j] = (i == j ? 1.5 : 0.0) - 0.5 * M[i * ld + j];
    }
    __syncthreads();
}
__device__ __forceinline__ void ns_load(const double *g, double *M, int o, int ld)
{
    for (int l = threadIdx.x; l < ld * ld; l += NS_THREADS) {
        const int i = l / ld, j = l - i * ld;
        M[l] = (i < o && j < o) ? g[(size_t) i * o + j] : 0.0;
    }
}
__device__ __forceinline__ void ns_store(const double *M, double *g, int o, int ld)
{
    for (int l = threadIdx.x; l < o * o; l += NS_THREADS) g[l] = M[l / o * ld + l % o];
}

// iters steps X <- X (1.5 I - 0.5 X^T X); X in place, Y = X^T X of the result.
__global__ void __launch_bounds__(NS_THREADS) k_ns_polar(double *gX, double *gY, int o, int iters)
{
    extern __shared__ __align__(16) double ns[];
    const int ld = (o + 3) & ~3;
    double *X = ns, *Y = ns + ld * ld, *M = Y + ld * ld;
    ns_load(gX, X, o, ld);
    __syncthreads();
    for (int it = 0; it < iters; it++) {
        ns_product<true>(X, X, Y, o, ld);
        ns_flip(Y, o, ld);
        ns_product<false>(X, Y, M, o, ld);
        double *t = X;
        X = M;
        M = t;
    }
    ns_product<true>(X, X, Y, o, ld);
    ns_store(X, gX, o, ld);
    ns_store(Y, gY, o, ld);
}

// Z = M^-1/2 by iters coupled steps T = 1.5 I - 0.5 Z Y, Y <- Y T, Z <- T Z from Y = M, Z = I.
__global__ void __launch_bounds__(NS_THREADS) k_ns_inv_sqrt(const double *gM, double *gZ, int o, int iters)
{
    extern __shared__ __align__(16) double ns[];
    const int ld = (o + 3) & ~3;
    double *Y = ns, *Z = Y + ld * ld, *T = Z + ld * ld, *W = T + ld * ld;
    ns_load(gM, Y, o, ld);
    for (int l = threadIdx.x; l < ld * ld; l += NS_THREADS) Z[l] = (l / ld == l % ld && l / ld < o) ? 1.0 : 0.0;
    __syncthreads();
    for (int it = 0; it < iters; it++) {
        ns_product<false>(Z, Y, T, o, ld);
        ns_flip(T, o, ld);
        ns_product<false>(Y, T, W, o, ld);
        double *t = Y;
        Y = W;
        W = t;
        ns_product<false>(T, Z, W, o, ld);
        t = Z;
        Z = W;
        W = t;
    }
    ns_store(Z, gZ, o, ld);
}

static size_t ns_smem(int o, int mats)
{
    const size_t ld = (o + 3) & ~3;
    return sizeof(double) * mats * ld * ld;
}

bool ns_fits(int o) { return o >= 1 && o <= NS_MAX; }

// The limit is a kernel's, not a launch's: every caller sets the largest size's, or a thread with a
// smaller molecule could lower it under another thread's launch.
template <class F>
static int ns_limit(F kernel, int mats)
{
    TSCF_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) ns_smem(NS_MAX, mats)));
    return OK;
}

int ns_polar(double *d_X, double *d_Y, int o, int iters, cudaStream_t s)
{
    if (const int rc = ns_limit(k_ns_polar, 3)) return rc;
    k_ns_polar<<<1, NS_THREADS, ns_smem(o, 3), s>>>(d_X, d_Y, o, iters);
    g_launches++;
    return cuda_launch_rc("polar factor");
}

int ns_inv_sqrt(const double *d_M, double *d_Z, int o, int iters, cudaStream_t s)
{
    if (const int rc = ns_limit(k_ns_inv_sqrt, 4)) return rc;
    k_ns_inv_sqrt<<<1, NS_THREADS, ns_smem(o, 4), s>>>(d_M, d_Z, o, iters);
    g_launches++;
    return cuda_launch_rc("inverse square root");
}

// Whether a tuned product goes to the K-split tile. Every other tile sums over k
// in one chain, so they may be timed against one another; the K-split tile rounds
// differently, and the accelerated solve turns 1e-16 in X, or in a refinement
// product, into 1e-9 of its density. Timed against the others it won or lost by a
// coin toss near the line (1010^3 with A transposed: 0.147 ms both; 585 x 93 x 93:
// 9.7 us both), so C40H82's density differed by 2-5e-9 from process to process.
// The line lies where its advantage ends, at 6 (A transposed), 4 (B transposed)
// or 5 of its CTAs an SM; times of the K-split tile over the best other one: A
// transposed 760^3 0.67, 910^3 0.92 (841 CTAs), 935^3 1.01 (900), 1152^3 1.09;
// plain 760^3 0.93, 835^3 0.98 (729), 885^3 1.09 (784); B transposed
// 760 x 760 x 121 0.88 (576), 835 x 835 x 133 1.08 (729), with a long K
// 835 x 835 x 266 0.96 (729), 885 x 885 x 282 1.02 (784). At the other end few CTAs
// with one K chunk and a half have nothing to split: 400 x 80 x 80 1.26,
// 510 x 81 x 81 1.12, 500 x 100 x 100 0.90.
static bool ksplit_order(bool ta, bool tb, int m, int n, int k)
{
    const long long tiles = (long long) ((m + KS_T - 1) / KS_T) * ((n + KS_T - 1) / KS_T);
    if (k < 100 && tiles < 64) return false;
    const int per = ta ? 6 : (!tb || k >= 256) ? 5 : 4;
    return tiles <= (long long) per * num_sms();
}

void dgemm(bool ta, bool tb, int m, int n, int k, double alpha, const double *A, int lda, const double *B, int ldb,
           double beta, double *C, int ldc, cudaStream_t s)
{
    if (m <= 0 || n <= 0) return;
    char key[96];
    snprintf(key, sizeof(key), "dgemm:%d%d:%dx%dx%d", (int) ta, (int) tb, m, n, k);
    int v = tune_lookup(key);
    if (v < 0) {
        v = 0;
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        cudaStreamIsCapturing(s, &cs);
        // tune only where re-running is harmless: C overwritten (beta = 0) and
        // not read by the product
        const char *c0 = (const char *) C, *c1 = c0 + sizeof(double) * ((size_t) (m - 1) * ldc + n);
        auto disjoint = [&](const double *X, size_t elems) {
            const char *x0 = (const char *) X, *x1 = x0 + sizeof(double) * elems;
            return x1 <= c0 || c1 <= x0;
        };
        const size_t ea = ta ? (size_t) k * lda : (size_t) m * lda, eb = tb ? (size_t) n * ldb : (size_t) k * ldb;
        if (tune_enabled() && cs == cudaStreamCaptureStatusNone && beta == 0.0 && disjoint(A, ea) && disjoint(B, eb) &&
            (double) m * n * k >= 2e6) {
            if (ksplit_order(ta, tb, m, n, k)) {
                tune_fix(key, 5);
                dgemm_variant(5, ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
                return;
            }
            v = tune_run(key, {0, 1, 2, 3, 4}, [&](int c) { dgemm_variant(c, ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s); }, s);
            return;
        }
        if (beta == 0.0 && (double) m * n * k < 2e6) {
            dgemm_small(ta, tb, m, n, k, alpha, A, lda, B, ldb, C, ldc, s);
            return;
        }
    }
    dgemm_variant(v, ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
}

// Tile shape from the call shape alone, for the many distinct shapes of the
// eigensolver's panel updates (tuning each one would cost more than it saves):
// the K-split tile for outputs of few 64 x 64 tiles with a long K, the 128 x 128 DMMA tile
// for large outputs, the 64 x 64 DMMA tile otherwise.
void dgemm_untuned(bool ta, bool tb, int m, int n, int k, double alpha, const double *A, int lda, const double *B,
                   int ldb, double beta, double *C, int ldc, cudaStream_t s)
{
    if (m <= 0 || n <= 0) return;
    int v = 4;
    const double tiles64 = std::ceil(m / 64.0) * std::ceil(n / 64.0);
    const double nsm = num_sms();
    if (k >= 256 && tiles64 < 2.0 * nsm) v = 5;
    else if ((double) m * n >= 4.0 * nsm * 128 * 128) v = 3;
    dgemm_variant(v, ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
}

// SM count of the current device (cached for the first 64 ordinals).
int num_sms()
{
    static std::atomic<int> cached[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    const bool cacheable = dev >= 0 && dev < 64;
    if (cacheable && cached[dev].load(std::memory_order_relaxed) > 0) return cached[dev].load(std::memory_order_relaxed);
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    if (v <= 0) v = 1;
    if (cacheable) cached[dev].store(v, std::memory_order_relaxed);
    return v;
}

int cuda_launch_rc(const char *what)
{
    const cudaError_t err = cudaPeekAtLastError();
    if (err == cudaSuccess) return OK;
    fprintf(stderr, "[tinyscf] CUDA error in %s: %s\n", what, cudaGetErrorString(err));
    return ERR_CUDA;
}

// ---------------------------------------------------------------- bounded waits
int *wait_word()
{
    static int *const word = [] {
        int *p = nullptr;
        if (cudaHostAlloc(&p, 64, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
            cudaGetLastError();
            return (int *) nullptr;
        }
        *p = 0;
        return p;
    }();
    return word;
}

static std::mutex g_wait_mu;
static unsigned g_wait_reports = 0;   // times the word was found set
static int g_wait_code = 0;           // and what it held the last time

static int take_locked()
{
    volatile int *w = wait_word();
    const int code = w ? *w : 0;
    if (code) {
        *w = 0;
        g_wait_code = code;
        g_wait_reports++;
    }
    return code;
}

int waits_take()
{
    std::lock_guard<std::mutex> lk(g_wait_mu);
    return take_locked();
}

unsigned waits_mark()
{
    std::lock_guard<std::mutex> lk(g_wait_mu);
    return g_wait_reports;
}

int waits_check(unsigned &mark, const char *what)
{
    std::lock_guard<std::mutex> lk(g_wait_mu);
    take_locked();
    if (g_wait_reports == mark) return OK;
    mark = g_wait_reports;
    fprintf(stderr, "[tinyscf] %s: a bounded wait timed out (code %d)\n", what, g_wait_code);
    return ERR_CUDA;
}

__global__ void k_wait_probe(long long cycles, int *gave_up)
{
    __shared__ uint64_t bar;
    umma::mbar_init(&bar, 1);
    umma::mbar_wait_bounded(&bar, 0, gave_up, 71, cycles);
}

int wait_probe(long long cycles, cudaStream_t s)
{
    if (cycles < 0 || !wait_word()) return ERR_INPUT;
    k_wait_probe<<<1, 1, 0, s>>>(cycles, wait_word());
    g_launches++;
    return cudaStreamSynchronize(s) == cudaSuccess ? OK : ERR_CUDA;
}

// ---------------------------------------------------------------- device memory
// The engine's large buffers come from the device's stream-ordered memory
// pool, kept reserved (release threshold: unlimited), so that freeing an
// engine hands its memory to the next one without unmapping and remapping;
// TINYSCF_MEMPOOL=0 uses cudaMalloc / cudaFree instead. The choice is made
// once per process. TinySCF_trim_memory returns the pool's unused memory.
static bool pool_mode()
{
    static const bool on = [] {
        const char *v = getenv("TINYSCF_MEMPOOL");
        return !(v && v[0] == '0');
    }();
    return on;
}

int dev_malloc(void **p, size_t bytes, cudaStream_t s)
{
    *p = nullptr;
    if (bytes == 0) bytes = 16;
    if (pool_mode()) {
        static std::mutex mu;
        static bool configured[64] = {};
        int dev = 0;
        cudaGetDevice(&dev);
        {
            std::lock_guard<std::mutex> lk(mu);
            if (dev >= 0 && dev < 64 && !configured[dev]) {
                cudaMemPool_t pool;
                if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
                    uint64_t thr = UINT64_MAX;
                    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr);
                }
                configured[dev] = true;
            }
        }
        if (cudaMallocAsync(p, bytes, s) != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess) {
            cudaGetLastError();
            *p = nullptr;
            return ERR_ALLOC;
        }
        return OK;
    }
    if (cudaMalloc(p, bytes) != cudaSuccess) {
        cudaGetLastError();
        *p = nullptr;
        return ERR_ALLOC;
    }
    return OK;
}

void dev_free(void *p, cudaStream_t s)
{
    if (!p) return;
    if (pool_mode()) cudaFreeAsync(p, s);
    else cudaFree(p);
}

int dev_trim(int device)
{
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, device) != cudaSuccess) return ERR_CUDA;
    if (cudaDeviceSynchronize() != cudaSuccess) return ERR_CUDA;
    return cudaMemPoolTrimTo(pool, 0) == cudaSuccess ? OK : ERR_CUDA;
}

__global__ void k_scale_rows_invsqrt(const double *w, const double *V, double *out, int n)
{
    size_t idx = (size_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t) n * n) return;
    int k = (int) (idx / n);
    out[idx] = V[idx] / sqrt(w[k]);
}

void inv_sqrt_from_eig(const double *d_w, const double *d_V, double *d_X, double *d_tmp, int n, cudaStream_t s)
{
    size_t nn = (size_t) n * n;
    g_launches++;
    k_scale_rows_invsqrt<<<(unsigned) ((nn + 255) / 256), 256, 0, s>>>(d_w, d_V, d_tmp, n);
    // X = V^T diag(w^-1/2) V
    dgemm(true, false, n, n, n, 1.0, d_V, n, d_tmp, n, 0.0, d_X, n, s);
}

// ------------------------------------------------------------------ pivoted Cholesky
// One 1024-thread block runs LAPACK dpstf2 (UPLO = 'L') step for step on the
// logical matrix A(i,j) = A[i*n + j]: left-looking column updates, diagonal
// candidates A(i,i) - sum_k A(i,k)^2 accumulated in work[], first-maximum
// pivot, the same row/column swaps, stop when the pivot <= tol.
struct ValIdx {
    double v;
    int i;
};
__device__ __forceinline__ ValIdx better(ValIdx a, ValIdx b)
{
    if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
    return a;
}

__device__ ValIdx block_argmax(ValIdx x, ValIdx *sh)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        ValIdx y;
        y.v = __shfl_down_sync(0xffffffff, x.v, o);
        y.i = __shfl_down_sync(0xffffffff, x.i, o);
        x = better(x, y);
    }
    if (lane == 0) sh[wid] = x;
    __syncthreads();
    if (wid == 0) {
        x = (lane < (int) (blockDim.x >> 5)) ? sh[lane] : ValIdx{-DBL_MAX, 0x7fffffff};
        for (int o = 16; o > 0; o >>= 1) {
            ValIdx y;
            y.v = __shfl_down_sync(0xffffffff, x.v, o);
            y.i = __shfl_down_sync(0xffffffff, x.i, o);
            x = better(x, y);
        }
        if (lane == 0) sh[0] = x;
    }
    __syncthreads();
    ValIdx r = sh[0];
    __syncthreads();
    return r;
}

// blkp (nullptr: one block): the block of every position, permuted with the
// pivots. A is block diagonal in these blocks (the SAD density: one block per
// atom), so column j of the factor is nonzero only in the rows of the pivot's
// block and every product with another block's entry is an exact zero: the
// rows of other blocks are skipped and their squared-norm sums left alone,
// which changes no bit of the result (adding +-0 is exact) but makes each
// step cost the pivot search instead of an (n - j) x j update.
__global__ void __launch_bounds__(1024) k_pstf2(double *A, int n, double tol, int *piv, int *rank_out, double *work,
                                                int *blkp)
{
    __shared__ ValIdx sh[32];
    __shared__ int s_stop;
    double *dot = work, *cand = work + n;
#define AA(i, j) A[(size_t) (i) * n + (j)]
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        dot[i] = 0.0;
        piv[i] = i;
    }
    __syncthreads();
    // j = 0: pivot on the largest diagonal element
    ValIdx best{-DBL_MAX, 0x7fffffff};
    for (int i = threadIdx.x; i < n; i += blockDim.x) best = better(best, ValIdx{AA(i, i), i});
    best = block_argmax(best, sh);
    double ajj = best.v;
    int pvt = best.i;
    if (threadIdx.x == 0) s_stop = (ajj <= 0.0 || isnan(ajj)) ? 1 : 0;
    __syncthreads();
    if (s_stop) {
        if (threadIdx.x == 0) *rank_out = 0;
        return;
    }
    int rank = n;
    for (int j = 0; j < n; j++) {
        if (j > 0) {
            ValIdx b{-DBL_MAX, 0x7fffffff};
            const int bprev = blkp ? blkp[j - 1] : 0;
            for (int i = j + threadIdx.x; i < n; i += blockDim.x) {
                if (!blkp || blkp[i] == bprev) {
                    double a = AA(i, j - 1);
                    dot[i] += a * a;
                }
                double c = AA(i, i) - dot[i];
                cand[i] = c;
                b = better(b, ValIdx{c, i});
            }
            b = block_argmax(b, sh);
            pvt = b.i;
            ajj = b.v;
            if (ajj <= tol || isnan(ajj)) {
                if (threadIdx.x == 0) AA(j, j) = ajj;
                rank = j;
                break;
            }
        }
        if (j != pvt) {
            __syncthreads();
            if (threadIdx.x == 0) {
                AA(pvt, pvt) = AA(j, j);
                double t = dot[j]; dot[j] = dot[pvt]; dot[pvt] = t;
                int p = piv[pvt]; piv[pvt] = piv[j]; piv[j] = p;
                if (blkp) {
                    const int q = blkp[pvt]; blkp[pvt] = blkp[j]; blkp[j] = q;
                }
            }
            for (int c = threadIdx.x; c < j; c += blockDim.x) {          // rows j and pvt, columns 0..j-1
                double t = AA(j, c); AA(j, c) = AA(pvt, c); AA(pvt, c) = t;
            }
            for (int r = pvt + 1 + threadIdx.x; r < n; r += blockDim.x) { // columns j and pvt below pvt
                double t = AA(r, j); AA(r, j) = AA(r, pvt); AA(r, pvt) = t;
            }
            for (int r = j + 1 + threadIdx.x; r < pvt; r += blockDim.x) { // column j (rows j+1..pvt-1) vs row pvt
                double t = AA(r, j); AA(r, j) = AA(pvt, r); AA(pvt, r) = t;
            }
            __syncthreads();
        }
        ajj = sqrt(ajj);
        if (threadIdx.x == 0) AA(j, j) = ajj;
        __syncthreads();
        // A(j+1:n, j) = (A(j+1:n, j) - A(j+1:n, 0:j) A(j, 0:j)^T) / ajj : one warp per row
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
        const double rinv = 1.0 / ajj;
        const int bj = blkp ? blkp[j] : 0;
        for (int r = j + 1 + wid; r < n; r += nw) {
            if (blkp && blkp[r] != bj) continue;   // zero column entry: (0 - 0) / ajj stays +0
            double s = 0.0;
            for (int c = lane; c < j; c += 32)
                if (!blkp || blkp[c] == bj) s += AA(r, c) * AA(j, c);
            for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffff, s, o);
            if (lane == 0) AA(r, j) = (AA(r, j) - s) * rinv;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) *rank_out = rank;
#undef AA
}

void pivoted_cholesky(double *d_A, int n, double tol, int *d_piv, int *d_rank, double *d_work, cudaStream_t s,
                      const int *d_blk, int *d_blk_work)
{
    g_launches++;
    int *blkp = nullptr;
    if (d_blk && d_blk_work) {
        cudaMemcpyAsync(d_blk_work, d_blk, sizeof(int) * n, cudaMemcpyDeviceToDevice, s);
        blkp = d_blk_work;
    }
    k_pstf2<<<1, 1024, 0, s>>>(d_A, n, tol, d_piv, d_rank, d_work, blkp);
}

__global__ void k_d2cocc(const double *chol, const int *rank_p, double *C, int nbf, int nocc)
{
    size_t idx = (size_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t) nbf * nocc) return;
    int i = (int) (idx / nocc), j = (int) (idx % nocc);
    int rank = *rank_p;
    double v = (j < nbf) ? chol[(size_t) i * nbf + j] : 0.0;
    if (rank < nocc && j >= rank) v = 0.0;
    if (i < nocc && j >= i) v = 0.0;
    C[idx] = v;
}

void d2cocc_copy(const double *d_chol, const int *d_rank, double *d_Cocc, int nbf, int nocc, cudaStream_t s)
{
    size_t n = (size_t) nbf * nocc;
    g_launches++;
    k_d2cocc<<<(unsigned) ((n + 255) / 256), 256, 0, s>>>(d_chol, d_rank, d_Cocc, nbf, nocc);
}

// ------------------------------------------------------------------ elementwise
__global__ void k_fill(double *d, double v, size_t n)
{
    size_t i = (size_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) d[i] = v;
}
void fill(double *d, double v, size_t n, cudaStream_t s)
{
    if (n) g_launches++;
    if (n) k_fill<<<(unsigned) ((n + 255) / 256), 256, 0, s>>>(d, v, n);
}
__global__ void k_scale_copy(const double *a, double *b, double f, size_t n)
{
    size_t i = (size_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) b[i] = f * a[i];
}
void scale_copy(const double *src, double *dst, double a, size_t n, cudaStream_t s)
{
    if (n) g_launches++;
    if (n) k_scale_copy<<<(unsigned) ((n + 255) / 256), 256, 0, s>>>(src, dst, a, n);
}

}  // namespace tscf
