// Coulomb (J), exchange (K) and Fock assembly on sm_100a, FP64.
//
// J (build_Fock.c:37-130) is two bandwidth-bound passes over the DF tensor:
//   t(P)   = sum_{i<=j in CSR} (2 - d_ij) D_ij B(ij,P)        (row-streamed GEMV)
//   J_ij   = B(ij,:) . t                                       (one warp per pair)
// K (build_Fock.c:244-347) is the occupied half-transform
//   T(i,s,P) = sum_{j in row i} Cocc(j,s) B(ij,P)               (gather GEMM per row i)
// followed by K = T T^T over the flattened (s,P) index (upper tiles, split-K).
// The DF tensor is stored once per unordered pair (B_u); every ordered CSR
// entry of the reference (bf_pair_j / bf_mask_displs) maps to its row.
#include <algorithm>
#include <cmath>
#include <cstdio>

#include "tiles.cuh"
#include "tscf_internal.h"
#include "umma.cuh"

namespace tscf {

// ------------------------------------------------------------------ J
__global__ void k_j_weights(const int *up_i, const int *up_j, const double *D, double *w, int nup, int nbf)
{
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nup) return;
    int i = up_i[k], j = up_j[k];
    w[k] = (i == j ? 1.0 : 2.0) * D[(size_t) i * nbf + j];
}

// Each block streams a contiguous range of upper rows and keeps its partial
// t(P) for every column in registers (jt_rows).
template <typename BT, int COLS>
__global__ void __launch_bounds__(JT_THREADS) k_j_tpart(const BT *__restrict__ B, const int *__restrict__ up_u,
                                                        const double *__restrict__ w, int nup, int naux, int rows_per_blk,
                                                        double *__restrict__ part)
{
    const int r0 = blockIdx.x * rows_per_blk, r1 = min(nup, r0 + rows_per_blk);
    jt_rows<BT, COLS>(B, up_u, w, naux, r0, r1, part + (size_t) blockIdx.x * naux);
}

// The FP32 copy of B with an even naux (jt_rows_f2: float2 column pairs, two
// rows per step, the same sums as jt_rows<float> bit for bit).
__global__ void __launch_bounds__(JT_THREADS) k_j_tpart_f2(const float *__restrict__ B, const int *__restrict__ up_u,
                                                           const double *__restrict__ w, int nup, int naux,
                                                           int rows_per_blk, double *__restrict__ part)
{
    const int r0 = blockIdx.x * rows_per_blk, r1 = min(nup, r0 + rows_per_blk);
    jt_rows_f2(B, up_u, w, naux, r0, r1, part + (size_t) blockIdx.x * naux);
}

// t(P) = sum over the blocks' partial rows, in block order (jt_reduce_col).
__global__ void k_j_treduce(const double *part, int nblk, int naux, double *t)
{
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= naux) return;
    t[p] = jt_reduce_col(part, nblk, naux, p);
}

template <typename BT>
__global__ void __launch_bounds__(256) k_j_rows(const BT *__restrict__ B, const int *up_i, const int *up_j,
                                                const int *up_u, const double *__restrict__ t, int nup, int naux,
                                                int nbf, double *J)
{
    extern __shared__ double ts[];
    for (int p = threadIdx.x; p < naux; p += blockDim.x) ts[p] = t[p];
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int nw = blockDim.x >> 5;
    for (int k = blockIdx.x * nw + wid; k < nup; k += gridDim.x * nw) {
        const BT *row = B + (size_t) up_u[k] * naux;
        double s = 0.0;
        for (int p = lane; p < naux; p += 32) s = fma((double) __ldg(row + p), ts[p], s);
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffff, s, o);
        if (lane == 0) {
            int i = up_i[k], j = up_j[k];
            J[(size_t) i * nbf + j] = s;
            J[(size_t) j * nbf + i] = s;
        }
    }
}

int build_J_part_blocks(const FockPlan &p)
{
    int nb = 2 * num_sms();
    if (p.nup < nb) nb = p.nup > 0 ? p.nup : 1;
    return nb;
}

template <typename BT>
static void build_J_t(const FockPlan &p, const BT *B, const double *d_D, double *d_J, double *d_t, double *d_part,
                      int nblk, double *d_w, cudaStream_t s)
{
    g_launches += 4;
    k_j_weights<<<(p.nup + 255) / 256, 256, 0, s>>>(p.up_i, p.up_j, d_D, d_w, p.nup, p.nbf);
    int rows_per_blk = (p.nup + nblk - 1) / nblk;
    if (sizeof(BT) == sizeof(float) && jt_pairs_ok((const float *) B, p.naux))
        k_j_tpart_f2<<<nblk, JT_THREADS, 0, s>>>((const float *) B, p.up_u, d_w, p.nup, p.naux, rows_per_blk,
                                                 d_part);
    else if (p.naux <= 8 * JT_THREADS)
        k_j_tpart<BT, 8><<<nblk, JT_THREADS, 0, s>>>(B, p.up_u, d_w, p.nup, p.naux, rows_per_blk, d_part);
    else
        k_j_tpart<BT, JT_COLS><<<nblk, JT_THREADS, 0, s>>>(B, p.up_u, d_w, p.nup, p.naux, rows_per_blk, d_part);
    k_j_treduce<<<(p.naux + 63) / 64, 64, 0, s>>>(d_part, nblk, p.naux, d_t);
    int blocks = num_sms() * 4;
    const size_t shm = sizeof(double) * p.naux;   // t(P) staged in shared memory
    if (shm > 48 * 1024)   // the largest naux's: a limit is the kernel's, other threads launch it too
        cudaFuncSetAttribute(k_j_rows<BT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sizeof(double) * MAX_NAUX);
    k_j_rows<BT><<<blocks, 256, shm, s>>>(B, p.up_i, p.up_j, p.up_u, d_t, p.nup, p.naux, p.nbf, d_J);
}

void build_J(const FockPlan &p, const double *d_D, double *d_J, double *d_t, double *d_part, int nblk, double *d_w,
             cudaStream_t s)
{
    build_J_t<double>(p, p.B, d_D, d_J, d_t, d_part, nblk, d_w, s);
}

void build_J_f32(const FockPlan &p, const float *B32, const double *d_D, double *d_J, double *d_t, double *d_part,
                 int nblk, double *d_w, cudaStream_t s)
{
    build_J_t<float>(p, B32, d_D, d_J, d_t, d_part, nblk, d_w, s);
}

__global__ void k_to_f32(const double *in, float *out, size_t n)
{
    for (size_t i = (size_t) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t) gridDim.x * blockDim.x)
        out[i] = (float) in[i];
}

void convert_f32(const double *in, float *out, size_t n, cudaStream_t s)
{
    g_launches++;
    k_to_f32<<<num_sms() * 8, 256, 0, s>>>(in, out, n);
}

// ------------------------------------------------------------------ K, FP64
// T[i][s][P]: block tile 64 (s) x 64 (P), K-step 16 rows of CSR row i.
__global__ void __launch_bounds__(256) k_halftransform(const double *__restrict__ B, const double *__restrict__ C,
                                                       const int *__restrict__ csr_j, const int *__restrict__ csr_u,
                                                       const int *__restrict__ displs, int nocc, int naux,
                                                       double *__restrict__ T)
{
    half_tile(B, C, csr_j, csr_u, displs, nocc, naux, T, blockIdx.z, blockIdx.y * KT_M, blockIdx.x * KT_N);
}

__global__ void __launch_bounds__(256, 1) k_halftransform_wide(const double *__restrict__ B, const double *__restrict__ C,
                                                               const int *__restrict__ csr_j,
                                                               const int *__restrict__ csr_u,
                                                               const int *__restrict__ displs, int nocc, int naux,
                                                               double *__restrict__ T)
{
    half_tile_wide(B, C, csr_j, csr_u, displs, nocc, naux, T, blockIdx.z, blockIdx.y * KH_S, blockIdx.x * KH_P);
}

__global__ void __launch_bounds__(256, 1) k_halftransform_dmma(const double *__restrict__ B, const double *__restrict__ C,
                                                               const int *__restrict__ csr_j,
                                                               const int *__restrict__ csr_u,
                                                               const int *__restrict__ displs, int nocc, int naux,
                                                               double *__restrict__ T)
{
    half_tile_dmma(B, C, csr_j, csr_u, displs, nocc, naux, T, blockIdx.z, blockIdx.y * KH_S, blockIdx.x * KH_P);
}

// ---- K half-transform on the FP64 tensor cores, persistent and pipelined.
// CTA b takes the items b, b + grid, ... (item = row i, S occupied columns
// s0.., PW aux columns p0.., with the occupied tiles of one (i, p0) adjacent so
// the gathered DF rows are reused from L2). The CSR chunks of 16 partner rows
// (the K steps) of its items form one stream that cp.async copies KH_STAGES - 1
// steps ahead of the DMMA tiles: the gathers of the next chunks, the tile math
// and the write-out of a finished item overlap. Each step's row indices are
// read one step earlier still, so no copy waits on an index load; the
// fragments of the next four k are read before the DMMAs of the current four.
//
// Bound by the FP64 tensor cores, so the tile's S is fitted to n_occ: WS x WP
// warps of 8 NX x 32 outputs, S = 8 WS NX the multiple of 8, 16 or 24 that holds
// n_occ (up to 168, more in several tiles). With a fixed S = 64 C20H42's 81
// occupied orbitals were 128 columns of work (2.55 ms, now 1.82 ms), 13 waters'
// 65 were 128 (0.83 ms, now 0.53 ms). Summation order: k ascending in
// every output, as one chain of multiply-adds (what DMMA does, bit for bit).
constexpr int KH_STAGES = 4;
constexpr int KH_SMAX = 168;

__device__ __forceinline__ void cp_async8(double *dst, const double *src, int bytes)
{
    const unsigned d = (unsigned) __cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

struct KhCursor {
    int item, i, s0, p0, r0, r_end, step, nsteps;
};

template <int WS, int NX, int WP, int NY>
struct KhTile {
    static constexpr int S = WS * NX * 8, P = WP * NY * 8, THREADS = WS * WP * 32;
    static constexpr int AS = S + 4, BS = P + 4;   // strides = 4 or 12 (mod 16) doubles: conflict-free fragments
    static constexpr int STAGE = KT_K * (AS + BS);
    static constexpr size_t SMEM = sizeof(double) * KH_STAGES * STAGE;
};

template <int S, int P>
__device__ __forceinline__ void kh_set(KhCursor &c, int item, int n_items, int stiles, int ptiles,
                                       const int *__restrict__ displs)
{
    c.item = item;
    if (item >= n_items) return;
    const int per_row = stiles * ptiles;
    c.i = item / per_row;
    const int rem = item - c.i * per_row;
    c.p0 = (rem / stiles) * P;
    c.s0 = (rem % stiles) * S;
    c.r0 = displs[c.i];
    c.r_end = displs[c.i + 1];
    c.step = 0;
    c.nsteps = max(1, (c.r_end - c.r0 + KT_K - 1) / KT_K);   // a row without partners still writes its zeros
}

template <int S, int P>
__device__ __forceinline__ void kh_next(KhCursor &c, int n_items, int stiles, int ptiles,
                                        const int *__restrict__ displs)
{
    if (c.item >= n_items) return;
    if (++c.step < c.nsteps) c.r0 += KT_K;
    else kh_set<S, P>(c, c.item + gridDim.x, n_items, stiles, ptiles, displs);
}

// For an odd naux (rows start at any 8 bytes): every thread copies its share.
template <int WS, int NX, int WP, int NY>
__global__ void __launch_bounds__(KhTile<WS, NX, WP, NY>::THREADS, 1)
    k_halftransform_pipe(const double *__restrict__ B, const double *__restrict__ C, const int *__restrict__ csr_j,
                         const int *__restrict__ csr_u, const int *__restrict__ displs, int nocc, int naux,
                         double *__restrict__ T, int n_items, int stiles, int ptiles, unsigned long long *rowmax)
{
    using K = KhTile<WS, NX, WP, NY>;
    constexpr int S = K::S, PW = K::P, NT = K::THREADS;
    extern __shared__ __align__(16) double khsm[];
    constexpr int NBC = KT_K * PW, NB = (NBC + NT - 1) / NT;   // B copies per step, per thread
    constexpr int NAC = KT_K * S, NA = (NAC + NT - 1) / NT;            // Cocc copies per step, per thread
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ws = (warp / WP) * NX * 8, wp = (warp % WP) * NY * 8;
    const int fr = lane >> 2, fc = lane & 3;
    int iu[NB], ij[NA];
    KhCursor P, Q;   // P: the next step to copy; Q: the step the tiles consume
    kh_set<S, PW>(P, blockIdx.x, n_items, stiles, ptiles, displs);
    Q = P;
    auto load_idx = [&]() {   // row indices of P's step (-1: past the row, zero fill)
#pragma unroll
        for (int q = 0; q < NB; q++) {
            const int c = tid + NT * q;
            const int r = P.r0 + c / PW;
            iu[q] = (c < NBC && P.item < n_items && r < P.r_end) ? csr_u[r] : -1;
        }
#pragma unroll
        for (int q = 0; q < NA; q++) {
            const int c = tid + NT * q;
            const int r = P.r0 + c / S;
            ij[q] = (c < NAC && P.item < n_items && r < P.r_end) ? csr_j[r] : -1;
        }
    };
    auto issue = [&](int buf) {   // copies of P's step into stage buffer buf, one commit group
        double *As = khsm + (size_t) buf * K::STAGE, *Bs = As + KT_K * K::AS;
        if (P.item < n_items) {
#pragma unroll
            for (int q = 0; q < NB; q++) {
                const int c = tid + NT * q;
                if (NBC % NT == 0 || c < NBC) {
                    const int kk = c / PW, cc = c % PW;
                    const int pg = P.p0 + cc;
                    const bool ok = iu[q] >= 0 && pg < naux;
                    const double *src = ok ? B + (size_t) iu[q] * naux + pg : B;
                    cp_async8(&Bs[kk * K::BS + cc], src, ok ? 8 : 0);
                }
            }
#pragma unroll
            for (int q = 0; q < NA; q++) {
                const int c = tid + NT * q;
                if (NAC % NT == 0 || c < NAC) {
                    const int kk = c / S, cc = c % S, sg = P.s0 + cc;
                    const bool ok = ij[q] >= 0 && sg < nocc;
                    cp_async8(&As[kk * K::AS + cc], ok ? C + (size_t) ij[q] * nocc + sg : C, ok ? 8 : 0);
                }
            }
        }
        cp_async_commit();
    };
    for (int st = 0; st < KH_STAGES - 1; st++) {
        load_idx();
        issue(st);
        kh_next<S, PW>(P, n_items, stiles, ptiles, displs);
    }
    load_idx();
    double acc[NX][NY][2];
#pragma unroll
    for (int x = 0; x < NX; x++)
#pragma unroll
        for (int y = 0; y < NY; y++) acc[x][y][0] = acc[x][y][1] = 0.0;
    for (int g = 0; Q.item < n_items; g++) {
        cp_async_wait<KH_STAGES - 2>();   // this thread's copies of step g have landed
        __syncthreads();                  // everyone's have, and step g - 1's buffer is free
        const double *As = khsm + (size_t) (g % KH_STAGES) * K::STAGE + fc * K::AS + ws + fr;
        const double *Bs = khsm + (size_t) (g % KH_STAGES) * K::STAGE + KT_K * K::AS + fc * K::BS + wp + fr;
        double a[2][NX], b[2][NY];
        auto frag = [&](int w, int k4) {
#pragma unroll
            for (int x = 0; x < NX; x++) a[w][x] = As[k4 * K::AS + 8 * x];
#pragma unroll
            for (int y = 0; y < NY; y++) b[w][y] = Bs[k4 * K::BS + 8 * y];
        };
        frag(0, 0);
#pragma unroll
        for (int k4 = 0; k4 < KT_K; k4 += 4) {
            const int w = (k4 / 4) & 1;
            if (k4 + 4 < KT_K) frag(w ^ 1, k4 + 4);
#pragma unroll
            for (int x = 0; x < NX; x++)
#pragma unroll
                for (int y = 0; y < NY; y++) dmma_8x8x4(acc[x][y][0], acc[x][y][1], a[w][x], b[w][y]);
            if (k4 == 0) {   // the next copies go out behind the first DMMAs
                issue((g + KH_STAGES - 1) % KH_STAGES);
                kh_next<S, PW>(P, n_items, stiles, ptiles, displs);
                load_idx();
            }
        }
        if (++Q.step == Q.nsteps) {   // item done: write its tile, start the next
            double amax = 0.0;        // max |T| of the tile (padding entries are zero)
#pragma unroll
            for (int x = 0; x < NX; x++) {
                const int sg = Q.s0 + ws + 8 * x + fr;
                double *row = T + ((size_t) Q.i * nocc + (sg < nocc ? sg : 0)) * naux;
#pragma unroll
                for (int y = 0; y < NY; y++) {
                    const int pg = Q.p0 + wp + 8 * y + 2 * fc;
                    if (sg < nocc && pg < naux) row[pg] = acc[x][y][0];
                    if (sg < nocc && pg + 1 < naux) row[pg + 1] = acc[x][y][1];
                    amax = fmax(amax, fmax(fabs(acc[x][y][0]), fabs(acc[x][y][1])));
                    acc[x][y][0] = acc[x][y][1] = 0.0;
                }
            }
            if (rowmax) {   // row maxima for the integer-tensor-core K (non-negative: bit order = value order)
                for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffff, amax, o));
                if (lane == 0 && amax > 0.0) atomicMax(rowmax + Q.i, (unsigned long long) __double_as_longlong(amax));
            }
            kh_set<S, PW>(Q, Q.item + gridDim.x, n_items, stiles, ptiles, displs);
        }
    }
    cp_async_wait<0>();
}

// ---- the same tiles with a producer warp (even naux): it keeps bulk copies of
// the chunks' rows in flight (one instruction a row, 16-byte aligned because
// naux and the padded row pitch of Cocc are even) behind mbarriers, so the other
// warps only read fragments and issue DMMAs, and drift apart by up to the
// pipeline's depth: nothing but the chunk they wait for stops them. With all warps
// issuing the copies between block barriers the tensor cores idled 30% of the
// time (C40H82 13.4 ms, now 10.1 ms; C20H42 1.82 ms, now 1.40 ms). The copies in one
// of the tiles' warps instead cost more than they saved (13.7 ms). The SM quarter
// that holds the producer as its fourth warp gives each 128 registers, which
// bounds the tile of 12 warps (56 x 24 a warp).
constexpr long long KH_WAIT = 2000000000LL;   // clock cycles a barrier wait may take (~1 s)

__device__ __forceinline__ void bulk_row(double *dst, const double *src, unsigned bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     umma::smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(umma::smem_u32(bar))
                 : "memory");
}

template <int WS, int NX, int WP, int NY>
struct KhBulk : KhTile<WS, NX, WP, NY> {
    using K = KhTile<WS, NX, WP, NY>;
    static constexpr int WARPS = WS * WP, THREADS = (WARPS + 1) * 32;
    static constexpr int FIT = (int) ((220 << 10) / (sizeof(double) * K::STAGE));
    static constexpr int STAGES = FIT < 6 ? FIT : 6;
    static constexpr size_t SMEM = sizeof(double) * STAGES * K::STAGE;
};

// Cocc in rows of cp doubles (zeros behind n_occ), then a block of zeros for the rows behind a chunk's last.
__global__ void k_pad_cocc(const double *__restrict__ C, double *__restrict__ Cp, int nbf, int nocc, int cp, int zeros)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nbf * cp + zeros) return;
    const int i = k / cp, s = k - i * cp;
    Cp[k] = (i < nbf && s < nocc) ? C[(size_t) i * nocc + s] : 0.0;
}

template <int WS, int NX, int WP, int NY>
__global__ void __launch_bounds__(KhBulk<WS, NX, WP, NY>::THREADS, 1)
    k_halftransform_bulk(const double *__restrict__ B, const double *__restrict__ Cp, int cp, const double *zeros,
                         const int *__restrict__ csr_j, const int *__restrict__ csr_u, const int *__restrict__ displs,
                         int nocc, int naux, double *__restrict__ T, int n_items, int stiles, int ptiles,
                         unsigned long long *rowmax, int *gave_up)
{
    using K = KhBulk<WS, NX, WP, NY>;
    constexpr int S = K::S, PW = K::P, ST = K::STAGES;
    extern __shared__ __align__(16) double khsm[];
    __shared__ uint64_t full[ST], empty[ST];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int k = 0; k < ST; k++) {
            umma::mbar_init(&full[k], 1);
            umma::mbar_init(&empty[k], K::WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async;" ::: "memory");
    }
    __syncthreads();
    KhCursor Q;
    kh_set<S, PW>(Q, blockIdx.x, n_items, stiles, ptiles, displs);
    if (warp == K::WARPS) {   // ---- producer: lanes 0..15 copy the chunk's DF rows, lanes 16..31 its rows of Cocc
        const int kk = lane & 15;
        const bool isB = lane < 16;
        int idx = -1;
        auto fetch = [&]() {
            const int r = Q.r0 + kk;
            idx = (Q.item < n_items && r < Q.r_end) ? (isB ? csr_u[r] : csr_j[r]) : -1;
        };
        fetch();
        for (int g = 0; Q.item < n_items; g++) {
            const int st = g % ST;
            if (g >= ST && !umma::mbar_wait_bounded(&empty[st], ((g / ST) - 1) & 1, gave_up, 31, KH_WAIT)) {
                for (int k = g - ST; k < g; k++)   // its copies in flight
                    umma::mbar_wait_bounded(&full[k % ST], (k / ST) & 1, gave_up, 32, KH_WAIT);
                return;
            }
            double *As = khsm + (size_t) st * K::STAGE, *Bs = As + KT_K * K::AS;
            const unsigned nb = (unsigned) min(PW, naux - Q.p0) * 8u, na = S * 8u;
            if (lane == 0) umma::mbar_expect_tx(&full[st], KT_K * (nb + na));
            __syncwarp();
            if (isB) bulk_row(Bs + kk * K::BS, idx >= 0 ? B + (size_t) idx * naux + Q.p0 : zeros, nb, &full[st]);
            else bulk_row(As + kk * K::AS, idx >= 0 ? Cp + (size_t) idx * cp + Q.s0 : zeros, na, &full[st]);
            kh_next<S, PW>(Q, n_items, stiles, ptiles, displs);
            fetch();
        }
        return;
    }
    const int ws = (warp / WP) * NX * 8, wp = (warp % WP) * NY * 8;
    const int fr = lane >> 2, fc = lane & 3;
    double acc[NX][NY][2];
#pragma unroll
    for (int x = 0; x < NX; x++)
#pragma unroll
        for (int y = 0; y < NY; y++) acc[x][y][0] = acc[x][y][1] = 0.0;
    int st = 0, phase = 0;
    while (Q.item < n_items) {
        if (!umma::mbar_wait_bounded(&full[st], phase, gave_up, 33, KH_WAIT)) return;
        const double *As = khsm + (size_t) st * K::STAGE + fc * K::AS + ws + fr;
        const double *Bs = khsm + (size_t) st * K::STAGE + KT_K * K::AS + fc * K::BS + wp + fr;
#pragma unroll
        for (int k4 = 0; k4 < KT_K; k4 += 4) {
            double a[NX], b[NY];
#pragma unroll
            for (int x = 0; x < NX; x++) a[x] = As[k4 * K::AS + 8 * x];
#pragma unroll
            for (int y = 0; y < NY; y++) b[y] = Bs[k4 * K::BS + 8 * y];
#pragma unroll
            for (int x = 0; x < NX; x++)
#pragma unroll
                for (int y = 0; y < NY; y++) dmma_8x8x4(acc[x][y][0], acc[x][y][1], a[x], b[y]);
        }
        __syncwarp();
        if (lane == 0) umma::mbar_arrive(&empty[st]);
        if (++st == ST) {
            st = 0;
            phase ^= 1;
        }
        if (++Q.step < Q.nsteps) continue;
        double amax = 0.0;   // item done: write its tile, start the next
#pragma unroll
        for (int x = 0; x < NX; x++) {
            const int sg = Q.s0 + ws + 8 * x + fr;
            double *row = T + ((size_t) Q.i * nocc + (sg < nocc ? sg : 0)) * naux;
#pragma unroll
            for (int y = 0; y < NY; y++) {
                const int pg = Q.p0 + wp + 8 * y + 2 * fc;
                if (sg < nocc && pg < naux) {
                    *reinterpret_cast<double2 *>(row + pg) = make_double2(acc[x][y][0], acc[x][y][1]);
                    amax = fmax(amax, fmax(fabs(acc[x][y][0]), fabs(acc[x][y][1])));
                }
                acc[x][y][0] = acc[x][y][1] = 0.0;
            }
        }
        if (rowmax) {
            for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffff, amax, o));
            if (lane == 0 && amax > 0.0) atomicMax(rowmax + Q.i, (unsigned long long) __double_as_longlong(amax));
        }
        kh_set<S, PW>(Q, Q.item + gridDim.x, n_items, stiles, ptiles, displs);
    }
}

// Doubles of FockPlan::Cpad for nbf x nocc: rows padded to whole tiles, and a block of zeros.
size_t half_pad_elems(int nbf, int nocc)
{
    const size_t tiles = (nocc + KH_SMAX - 1) / KH_SMAX;
    return (size_t) nbf * (nocc + 32 * tiles) + 512;
}

template <int WS, int NX, int WP, int NY>
static void launch_half(const FockPlan &p, const double *C, double *T, unsigned long long *rowmax, cudaStream_t s)
{
    using K = KhTile<WS, NX, WP, NY>;
    using KB = KhBulk<WS, NX, WP, NY>;
    const int stiles = (p.nocc + K::S - 1) / K::S, ptiles = (p.naux + K::P - 1) / K::P;
    const long long items = (long long) p.nbf * stiles * ptiles;
    auto grid = [&](auto kernel, int threads, size_t smem) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
        int per = 1;   // the small tiles fit several times on an SM
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem);
        return (int) std::min<long long>(items, (long long) num_sms() * std::max(per, 1));
    };
    if (p.naux % 2 == 0 && p.Cpad && wait_word()) {
        const int cp = stiles * K::S, zeros = std::max(K::S, K::P);
        const int n = p.nbf * cp + zeros;
        k_pad_cocc<<<(n + 255) / 256, 256, 0, s>>>(C, p.Cpad, p.nbf, p.nocc, cp, zeros);
        g_launches++;
        const int g = grid(k_halftransform_bulk<WS, NX, WP, NY>, KB::THREADS, KB::SMEM);
        k_halftransform_bulk<WS, NX, WP, NY><<<g, KB::THREADS, KB::SMEM, s>>>(
            p.B, p.Cpad, cp, p.Cpad + (size_t) p.nbf * cp, p.csr_j, p.csr_u, p.csr_displs, p.nocc, p.naux, T,
            (int) items, stiles, ptiles, rowmax, wait_word());
    } else {
        const int g = grid(k_halftransform_pipe<WS, NX, WP, NY>, K::THREADS, K::SMEM);
        k_halftransform_pipe<WS, NX, WP, NY><<<g, K::THREADS, K::SMEM, s>>>(p.B, C, p.csr_j, p.csr_u, p.csr_displs, p.nocc,
                                                                        p.naux, T, (int) items, stiles, ptiles, rowmax);
    }
}

// The tile for the occupied part o (n_occ in equal parts of at most 168): the
// fewest padded orbitals within the registers, 4 warps or a multiple (each SM
// quarter has its own FP64 tensor pipe: 9 warps of 56 x 32 took 13.0 ms on C40H82).
//   o <= 56:  one row of warps, 8 o' x 32 outputs a warp; 128 or 256 aux columns
//   o <= 88:  one row, 24 aux columns a warp, 192 in all; or two rows, 128 columns
//   o <= 128: two rows, 128 columns
//   o <= 168: three rows, 12 warps: 96 columns without, or 128 with spilled registers
// Where two are named the autotuner times both.
static void half_pipe(const FockPlan &p, const double *C, double *T, unsigned long long *rowmax, cudaStream_t s, bool wide)
{
    const int tiles = (p.nocc + KH_SMAX - 1) / KH_SMAX, o = (p.nocc + tiles - 1) / tiles;
#define TSCF_HALF(WS, NX, WP, NY)                       \
    case NX:                                            \
        launch_half<WS, NX, WP, NY>(p, C, T, rowmax, s); \
        return;
    if (o <= 56 && !wide) {
        switch ((o + 7) / 8) {
            TSCF_HALF(1, 1, 4, 4) TSCF_HALF(1, 2, 4, 4) TSCF_HALF(1, 3, 4, 4) TSCF_HALF(1, 4, 4, 4)
            TSCF_HALF(1, 5, 4, 4) TSCF_HALF(1, 6, 4, 4) TSCF_HALF(1, 7, 4, 4)
        }
    } else if (o <= 56) {
        switch ((o + 7) / 8) {
            TSCF_HALF(1, 1, 8, 4) TSCF_HALF(1, 2, 8, 4) TSCF_HALF(1, 3, 8, 4) TSCF_HALF(1, 4, 8, 4)
            TSCF_HALF(1, 5, 8, 4) TSCF_HALF(1, 6, 8, 4) TSCF_HALF(1, 7, 8, 4)
        }
    } else if (o <= 88 && wide) {
        switch ((o + 7) / 8) {
            TSCF_HALF(1, 8, 8, 3) TSCF_HALF(1, 9, 8, 3) TSCF_HALF(1, 10, 8, 3) TSCF_HALF(1, 11, 8, 3)
        }
    } else if (o <= 128) {
        switch ((o + 15) / 16) {
            TSCF_HALF(2, 4, 4, 4) TSCF_HALF(2, 5, 4, 4) TSCF_HALF(2, 6, 4, 4) TSCF_HALF(2, 7, 4, 4)
            TSCF_HALF(2, 8, 4, 4)
        }
    } else if (!wide) {
        switch ((o + 23) / 24) { TSCF_HALF(3, 6, 4, 3) TSCF_HALF(3, 7, 4, 3) }
    } else {
        switch ((o + 23) / 24) { TSCF_HALF(3, 6, 4, 4) TSCF_HALF(3, 7, 4, 4) }
    }
#undef TSCF_HALF
}

// K partial tiles: upper tile pairs (bi <= bj) of 64x64, split over the
// flattened Q = nocc*naux index. Kpart[split][i][j].
__global__ void __launch_bounds__(256) k_syrk_part(const double *__restrict__ T, int nbf, long long Q, long long qchunk,
                                                   const int2 *__restrict__ tiles, double *__restrict__ Kpart)
{
    const int2 tl = tiles[blockIdx.x];
    const int split = blockIdx.y;
    const long long q_beg = (long long) split * qchunk, q_end = min(Q, q_beg + qchunk);
    syrk_tile(T, nbf, Q, q_beg, q_end, tl.x * KT_M, tl.y * KT_N, Kpart + (size_t) split * nbf * nbf);
}

__global__ void __launch_bounds__(256, 1) k_syrk_part128(const double *__restrict__ T, int nbf, long long Q,
                                                         long long qchunk, const int2 *__restrict__ tiles,
                                                         double *__restrict__ Kpart)
{
    const int2 tl = tiles[blockIdx.x];
    const int split = blockIdx.y;
    const long long q_beg = (long long) split * qchunk, q_end = min(Q, q_beg + qchunk);
    syrk_tile128(T, nbf, Q, q_beg, q_end, tl.x * KB_T, tl.y * KB_T, Kpart + (size_t) split * nbf * nbf);
}

__global__ void __launch_bounds__(256, 1) k_syrk_dmma(const double *__restrict__ T, int nbf, long long Q,
                                                      long long qchunk, const int2 *__restrict__ tiles,
                                                      double *__restrict__ Kpart)
{
    const int2 tl = tiles[blockIdx.x];
    const int split = blockIdx.y;
    const long long q_beg = (long long) split * qchunk, q_end = min(Q, q_beg + qchunk);
    syrk_tile_dmma(T, nbf, Q, q_beg, q_end, tl.x * KB_T, tl.y * KB_T, Kpart + (size_t) split * nbf * nbf);
}

// K[i][j] = K[j][i] = sum_split Kpart[split][i][j] for i <= j (TinySCF keeps
// the upper triangle and mirrors it, build_Fock.c:369-379).
__global__ void k_syrk_reduce(const double *Kpart, int nsplit, int nbf, double *K)
{
    size_t idx = (size_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t) nbf * nbf) return;
    int i = (int) (idx / nbf), j = (int) (idx % nbf);
    if (i > j) return;
    double s = 0.0;
    for (int k = 0; k < nsplit; k++) s += Kpart[(size_t) k * nbf * nbf + idx];
    K[idx] = s;
    K[(size_t) j * nbf + i] = s;
}

size_t build_K_part_elems(const FockPlan &p, int ksplit) { return (size_t) ksplit * p.nbf * p.nbf; }

void build_K_halftransform(const FockPlan &p, const double *d_Cocc, double *d_T, cudaStream_t s, int wide,
                           unsigned long long *d_rowmax)
{
    if (p.nbf <= 0 || p.nocc <= 0 || p.naux <= 0) return;   // T is empty: no grid to launch
    g_launches++;
    if (wide >= 3) {
        if (d_rowmax) cudaMemsetAsync(d_rowmax, 0, sizeof(unsigned long long) * p.nbf, s);
        half_pipe(p, d_Cocc, d_T, d_rowmax, s, wide == 4);
    } else if (wide) {
        dim3 g1((p.naux + KH_P - 1) / KH_P, (p.nocc + KH_S - 1) / KH_S, p.nbf);
        if (wide == 2)
            k_halftransform_dmma<<<g1, 256, 0, s>>>(p.B, d_Cocc, p.csr_j, p.csr_u, p.csr_displs, p.nocc, p.naux, d_T);
        else
            k_halftransform_wide<<<g1, 256, 0, s>>>(p.B, d_Cocc, p.csr_j, p.csr_u, p.csr_displs, p.nocc, p.naux, d_T);
    } else {
        dim3 g1((p.naux + KT_N - 1) / KT_N, (p.nocc + KT_M - 1) / KT_M, p.nbf);
        k_halftransform<<<g1, 256, 0, s>>>(p.B, d_Cocc, p.csr_j, p.csr_u, p.csr_displs, p.nocc, p.naux, d_T);
    }
}

void build_K_syrk(const FockPlan &p, const double *d_T, double *d_K, double *d_Kpart, int ksplit, const int2 *d_tiles,
                  cudaStream_t s, int tile)
{
    const int tdim = tile == KSYRK_DMMA ? KB_T : tile;
    const int nt = (p.nbf + tdim - 1) / tdim;
    const int ntiles = nt * (nt + 1) / 2;
    const long long Q = (long long) p.nocc * p.naux;
    long long qchunk = (Q + ksplit - 1) / ksplit;
    qchunk = (qchunk + KT_K - 1) / KT_K * KT_K;
    dim3 g2(ntiles, ksplit);
    g_launches += 2;
    if (tile == KSYRK_DMMA) k_syrk_dmma<<<g2, 256, 0, s>>>(d_T, p.nbf, Q, qchunk, d_tiles, d_Kpart);
    else if (tile == KB_T) k_syrk_part128<<<g2, 256, 0, s>>>(d_T, p.nbf, Q, qchunk, d_tiles, d_Kpart);
    else k_syrk_part<<<g2, 256, 0, s>>>(d_T, p.nbf, Q, qchunk, d_tiles, d_Kpart);
    size_t nn = (size_t) p.nbf * p.nbf;
    k_syrk_reduce<<<(unsigned) ((nn + 255) / 256), 256, 0, s>>>(d_Kpart, ksplit, p.nbf, d_K);
}

// ------------------------------------------------------------------ F and energy
__global__ void k_fock_energy(const double *H, const double *J, const double *K, const double *D, double *F,
                              double *epart, size_t n)
{
    double e = fock_energy_range(H, J, K, D, F, (size_t) blockIdx.x * blockDim.x + threadIdx.x, n,
                                 (size_t) gridDim.x * blockDim.x);
    e = block_sum(e);
    if (threadIdx.x == 0) epart[blockIdx.x] = e;
}

void build_F_energy(const double *d_H, const double *d_J, const double *d_K, const double *d_D, double *d_F,
                    double *d_epart, int n, cudaStream_t s)
{
    g_launches++;
    k_fock_energy<<<ENERGY_BLOCKS, 256, 0, s>>>(d_H, d_J, d_K, d_D, d_F, d_epart, (size_t) n * n);
}

}  // namespace tscf
