// FP64 symmetric eigensolver of the SCF: X = S^-1/2 (TinySCF.c:58-76), the
// DF metric's (P|Q)^-1/2 (build_DF_tensor.c:205-237) and the orthogonalised
// Fock eigensolve (build_density.c:37-69), where the reference calls
// LAPACKE_dsyev. Three stages, all on the device:
//
//  1. Householder tridiagonalisation Q^T A Q = T (LAPACK dsytrd/dlatrd's
//     recurrence). Panels of TRD_NB columns: one cooperative kernel per panel
//     runs the column steps -- update the column with the panel's earlier
//     reflectors, form the reflector, the symmetric matrix-vector product with
//     the trailing matrix (not yet updated for the panel), the panel
//     corrections -- separated by grid barriers; then two GEMMs apply the
//     rank-2*TRD_NB update to the trailing matrix.
//  2. Divide and conquer on T (Cuppen): T is torn by rank-one updates down to
//     1 x 1 pieces; each merge of two solved halves deflates small and close
//     components (LAPACK dlaed2's tests, Givens rotations for close pairs),
//     finds the roots of the secular equation by bisection on the offset from
//     the nearer pole, recomputes z from the roots (Gu-Eisenstat, so that the
//     eigenvectors come out orthogonal) and multiplies the halves' vectors by
//     the merge's vectors. All merges of one tree level run in the same launches.
//  3. Back-transformation with the compact WY form of each panel
//     (H_p..H_(p+nb-1) = I - V T V^T), three GEMMs per panel.
//
// Every grid barrier spins a bounded number of times; a barrier that runs out
// sets the process's wait word (waits_check reports it) and every CTA returns.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <vector>

#include <cooperative_groups.h>

#include "tiles.cuh"
#include "tscf_internal.h"

namespace tscf {

std::atomic<long long> g_eig_launches{0};

namespace {

constexpr int TRD_THREADS = 512;
constexpr int TRD_NB = 32;        // columns per panel
constexpr int TRD_SEG = 256;     // columns per item of the symmetric matrix-vector product
constexpr int GR_KS = 8;          // row slices of the reflector blocks' Gram matrices
constexpr int BT_NB = 128;        // reflectors per block of the back-transformation
constexpr int DC_CHUNK = 256;     // items per CTA of the thread-per-item D&C kernels
constexpr int DC_WCHUNK = 8;      // items per CTA of the warp-per-item D&C kernels (256 threads)
constexpr long long kBarrierSpins = 1LL << 22;   // acquire polls before a barrier gives up (~ 2 s)

__device__ __forceinline__ double warp_sum_bcast(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffff, v, o);
    return __shfl_sync(0xffffffff, v, 0);
}

__device__ __forceinline__ double warp_prod_bcast(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v *= __shfl_down_sync(0xffffffff, v, o);
    return __shfl_sync(0xffffffff, v, 0);
}

// Sum over the block in a fixed order (warp trees, then warp 0 over the
// warps); the result is returned to every thread.
template <int NT>
__device__ __forceinline__ double block_sum_all(double v, double *sh)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffff, v, o);
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    if (wid == 0) {
        double x = lane < NT / 32 ? sh[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffff, x, o);
        if (lane == 0) sh[32] = x;
    }
    __syncthreads();
    const double r = sh[32];
    __syncthreads();
    return r;
}

template <int NT>
__device__ __forceinline__ double block_max_all(double v, double *sh)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffff, v, o));
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    if (wid == 0) {
        double x = lane < NT / 32 ? sh[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x = fmax(x, __shfl_down_sync(0xffffffff, x, o));
        if (lane == 0) sh[32] = x;
    }
    __syncthreads();
    const double r = sh[32];
    __syncthreads();
    return r;
}

// Grid barrier for a cooperative launch (all CTAs co-resident): a 64-bit
// ticket counter that only grows (zeroed before each solve). Thread 0 of each
// CTA arrives with a release add and spins with acquire loads until the
// counter reaches the end of its episode (the next multiple of nblk). The
// wait is bounded: a CTA whose wait runs out sets the error flag and returns
// false, and the caller returns; CTAs still waiting for it run out in turn.
__device__ __forceinline__ unsigned long long atom_add_release(unsigned long long *p, unsigned long long v)
{
    unsigned long long old;
    asm volatile("atom.add.release.gpu.u64 %0, [%1], %2;" : "=l"(old) : "l"(p), "l"(v) : "memory");
    return old;
}

__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.acquire.gpu.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ bool grid_barrier(unsigned long long *bar, int *err, unsigned nblk)
{
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned long long ticket = atom_add_release(bar, 1ull);
        const unsigned long long target = (ticket / nblk + 1) * nblk;
        long long spins = 0;
        bool ok = true;
        while (ld_acquire(bar) < target) {
            if (++spins > kBarrierSpins) {
                *(volatile int *) err = 51;
                ok = false;
                break;
            }
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// ------------------------------------------------------------------ tridiagonalisation
// Storage: reflector j is row j of VT (v_j[j+1] = 1, zero before); within a
// panel, PVW rows 0..NB-1 hold the panel's v and rows NB..2NB-1 its w, PWV the
// same two halves swapped, so that the trailing update A22 -= V W^T + W V^T is
// one GEMM PVW^T PWV with K = 2 NB, and every in-panel access to v or w runs
// along a row (coalesced).
struct TrdArgs {
    double *A;      // n x n work matrix (trailing part updated after each panel)
    double *VT;     // n x n reflectors as rows
    double *PVW, *PWV;   // 2 TRD_NB x n each
    double *d, *e, *tau;
    double *col;
    double *y;      // [segment][row] partial sums of A v
    double *part;   // [G] norms | [2 TRD_NB][G] panel dots | [G] w.v
    unsigned long long *bar;
    int *err;
    int n, p, cols, G;
};

__global__ void __launch_bounds__(TRD_THREADS, 1) k_sytrd_panel(TrdArgs a)
{
    extern __shared__ double sv[];   // v of the current column, by absolute row
    __shared__ double s_a2[TRD_NB], s_wv[TRD_NB], s_vv[TRD_NB], s_vj[TRD_NB], s_wj[TRD_NB];
    __shared__ double s_red[33];
    __shared__ double s_dot[TRD_THREADS / 32][2 * TRD_NB];
    __shared__ double s_tau, s_scal, s_beta;
    const int n = a.n, p = a.p, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int gtid = blockIdx.x * TRD_THREADS + tid, GT = a.G * TRD_THREADS;
    const int gw = blockIdx.x * (TRD_THREADS / 32) + wid, GW = a.G * (TRD_THREADS / 32);
    // Row r of the matrix belongs to the 8-lane group r for the whole panel
    // (G * TRD_THREADS / 8 >= n); lane l8 of the group keeps the row's entries
    // of panel columns l8, l8 + 8, l8 + 16, l8 + 24 of V and W in registers.
    const int l8 = lane & 7, r = gtid >> 3;
    const bool own = r < n;
    constexpr int NQ = TRD_NB / 8;
    double pv[NQ], pw[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) pv[q] = pw[q] = 0.0;
    const int nseg = (n + TRD_SEG - 1) / TRD_SEG;
    double *part_n = a.part, *part_d = a.part + a.G, *part_w = part_d + (size_t) a.G * 2 * TRD_NB;
    const double *A = a.A;
    // row p of the symmetric matrix: column p of the first step
    double arow = (own && r >= p && l8 == 0) ? A[(size_t) p * n + r] : 0.0;
    for (int c = 0; c < a.cols; c++) {
        const int j = p + c;
        // ---- phase 1: column j of the panel-corrected matrix, rows j..n-1 (s_vj, s_wj: row j's V and W)
        double v = 0.0;
        if (own && r >= j) {
            v = arow;
#pragma unroll
            for (int q = 0; q < NQ; q++) {
                const int cc = l8 + 8 * q;
                if (cc < c) v -= pv[q] * s_wj[cc] + pw[q] * s_vj[cc];
            }
        }
        v += __shfl_xor_sync(0xffffffff, v, 1);
        v += __shfl_xor_sync(0xffffffff, v, 2);
        v += __shfl_xor_sync(0xffffffff, v, 4);
        double ss = 0.0;
        if (own && r >= j && l8 == 0) {
            a.col[r] = v;
            if (r >= j + 2) ss = v * v;
        }
        ss = block_sum_all<TRD_THREADS>(ss, s_red);
        if (tid == 0) part_n[blockIdx.x] = ss;
        // items (row rr, segment sg) of phase 2's y = A v, over rows j+1..n-1 and the segments holding
        // columns j+1..n-1; A does not change within the panel, so a warp's first item is loaded here
        const int s0 = (j + 1) / TRD_SEG, ns = nseg - s0, nitems = (n - j - 1) * ns;
        double av[TRD_SEG / 32];
        auto load_item = [&](int it) {
            const int rr = j + 1 + it / ns, sg = s0 + it % ns;
            const double *row = A + (size_t) rr * n + sg * TRD_SEG + lane;
#pragma unroll
            for (int k = 0; k < TRD_SEG / 32; k++) {
                const int c2 = sg * TRD_SEG + lane + 32 * k;
                av[k] = (it < nitems && c2 > j && c2 < n) ? row[32 * k] : 0.0;
            }
        };
        if (j < n - 1) load_item(gw);
        if (!grid_barrier(a.bar, a.err, a.G)) return;
        if (j == n - 1) {
            if (gtid == 0) a.d[j] = a.col[j];
            break;
        }
        // ---- phase 2: reflector (every CTA forms the same one), v, y = A v by segments, panel dots
        for (int rr = j + 1 + tid; rr < n; rr += TRD_THREADS) sv[rr] = a.col[rr];   // issued with part_n's loads
        if (wid == 0) {
            double s = 0.0;
            for (int b = lane; b < a.G; b += 32) s += part_n[b];
            s = warp_sum_bcast(s);
            if (lane == 0) {
                const double alpha = a.col[j + 1];
                if (s == 0.0) {
                    s_tau = 0.0;
                    s_beta = alpha;
                    s_scal = 0.0;
                } else {
                    const double nrm = sqrt(alpha * alpha + s);
                    const double beta = alpha >= 0.0 ? -nrm : nrm;
                    s_tau = (beta - alpha) / beta;
                    s_beta = beta;
                    s_scal = 1.0 / (alpha - beta);
                }
            }
        }
        __syncthreads();
        const double tau = s_tau, scal = s_scal;
        for (int rr = j + 1 + tid; rr < n; rr += TRD_THREADS) sv[rr] = (rr == j + 1) ? 1.0 : sv[rr] * scal;
        __syncthreads();
        if (gtid == 0) {
            a.d[j] = a.col[j];
            a.e[j] = s_beta;
            a.tau[j] = tau;
        }
        for (int rr = j + 1 + gtid; rr < n; rr += GT) {
            const double vr = sv[rr];
            a.VT[(size_t) j * n + rr] = vr;
            a.PVW[(size_t) c * n + rr] = vr;
            a.PWV[(size_t) (TRD_NB + c) * n + rr] = vr;
        }
        const double vr_own = (own && r > j) ? sv[r] : 0.0;
        if (l8 == (c & 7)) {   // this row's entry of the new reflector (static register indexing)
#pragma unroll
            for (int q = 0; q < NQ; q++)
                if (q == (c >> 3)) pv[q] = vr_own;
        }
        {
            // the next item's loads are issued before this one's sum, which is a chain of shuffles: at n = 3870
            // (26 items a warp in the first columns) the panels took 85 ms without, now 72 ms; 4.7 ms of the panels
            // above 600 rows at n = 1010 (1 or 2 items) did not change
            for (int it = gw; it < nitems; it += GW) {
                const int rr = j + 1 + it / ns, sg = s0 + it % ns;
                double acc[TRD_SEG / 32];
#pragma unroll
                for (int k = 0; k < TRD_SEG / 32; k++) {
                    const int c2 = sg * TRD_SEG + lane + 32 * k;
                    acc[k] = (c2 > j && c2 < n) ? av[k] * sv[c2] : 0.0;
                }
                load_item(it + GW);
                static_assert(TRD_SEG == 256, "the pairwise sum below is written for 8 values per lane");
                const double y = warp_sum_bcast(((acc[0] + acc[4]) + (acc[2] + acc[6])) +
                                                ((acc[1] + acc[5]) + (acc[3] + acc[7])));
                if (lane == 0) a.y[(size_t) sg * n + rr] = y;
            }
        }
        if (c > 0) {
            // panel dots W^T v and V^T v over this CTA's rows, from the registers: groups of a warp
            // (lanes with equal l8) summed by shuffles, then the warps in shared memory
            double dw[NQ], dv[NQ];
#pragma unroll
            for (int q = 0; q < NQ; q++) {
                dw[q] = pw[q] * vr_own;
                dv[q] = pv[q] * vr_own;
                dw[q] += __shfl_xor_sync(0xffffffff, dw[q], 8);
                dw[q] += __shfl_xor_sync(0xffffffff, dw[q], 16);
                dv[q] += __shfl_xor_sync(0xffffffff, dv[q], 8);
                dv[q] += __shfl_xor_sync(0xffffffff, dv[q], 16);
            }
            if (lane < 8) {
#pragma unroll
                for (int q = 0; q < NQ; q++) {
                    s_dot[wid][lane + 8 * q] = dw[q];
                    s_dot[wid][TRD_NB + lane + 8 * q] = dv[q];
                }
            }
            __syncthreads();
            if (tid < 2 * TRD_NB) {
                double sacc = 0.0;
                for (int w = 0; w < TRD_THREADS / 32; w++) sacc += s_dot[w][tid];
                part_d[(size_t) tid * a.G + blockIdx.x] = sacc;
            }
        }
        if (!grid_barrier(a.bar, a.err, a.G)) return;
        // ---- phase 3: w = tau (y - V (W^T v) - W (V^T v)) for this row, partial w.v
        double ypart = 0.0;
        if (own && r > j)
            for (int sg = s0 + l8; sg < nseg; sg += 8) ypart += a.y[(size_t) sg * n + r];
        for (int cc = wid; cc < c; cc += TRD_THREADS / 32) {
            double sw = 0.0, sx = 0.0;
            for (int b = lane; b < a.G; b += 32) {
                sw += part_d[(size_t) cc * a.G + b];
                sx += part_d[(size_t) (TRD_NB + cc) * a.G + b];
            }
            sw = warp_sum_bcast(sw);
            sx = warp_sum_bcast(sx);
            if (lane == 0) {
                s_wv[cc] = sw;
                s_vv[cc] = sx;
            }
        }
        // the next column's row of A (issued here, used after the next two barriers)
        const bool nxt = c + 1 < a.cols;
        arow = (nxt && own && r >= j + 1 && l8 == 0) ? A[(size_t) (j + 1) * n + r] : 0.0;
        __syncthreads();
        double t = ypart;
        if (own && r > j) {
#pragma unroll
            for (int q = 0; q < NQ; q++) {
                const int cc = l8 + 8 * q;
                if (cc < c) t -= pv[q] * s_wv[cc] + pw[q] * s_vv[cc];
            }
        }
        t += __shfl_xor_sync(0xffffffff, t, 1);
        t += __shfl_xor_sync(0xffffffff, t, 2);
        t += __shfl_xor_sync(0xffffffff, t, 4);
        const double w = (own && r > j) ? tau * t : 0.0;
        if (l8 == (c & 7)) {
#pragma unroll
            for (int q = 0; q < NQ; q++)
                if (q == (c >> 3)) pw[q] = w;
        }
        double wd = 0.0;
        if (own && r > j && l8 == 0) {
            a.PWV[(size_t) c * n + r] = w;   // before its a2 v term; row j+1's entry is read by every CTA
            wd = w * vr_own;
        }
        wd = block_sum_all<TRD_THREADS>(wd, s_red);
        if (tid == 0) part_w[blockIdx.x] = wd;
        if (!grid_barrier(a.bar, a.err, a.G)) return;
        // ---- phase 4: a2 = -tau/2 (w.v), w += a2 v; row j+1's V and W for the next column
        if (wid == 0) {
            double s = 0.0;
            for (int b = lane; b < a.G; b += 32) s += part_w[b];
            s = warp_sum_bcast(s);
            if (lane == 0) s_a2[c] = -0.5 * tau * s;
        } else if (nxt && wid == 1 && lane <= c) {
            s_vj[lane] = a.PVW[(size_t) lane * n + j + 1];
            s_wj[lane] = a.PWV[(size_t) lane * n + j + 1];   // before a2 v; completed below
        }
        __syncthreads();
        if (l8 == (c & 7)) {
#pragma unroll
            for (int q = 0; q < NQ; q++)
                if (q == (c >> 3)) pw[q] += s_a2[c] * pv[q];
        }
        if (nxt && tid <= c) s_wj[tid] += s_a2[tid] * s_vj[tid];   // global W holds the values before a2 v
        __syncthreads();
    }
    // final W of this panel's rows, into both stacked panels for the trailing update
    if (own && r >= p + a.cols) {
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const int cc = l8 + 8 * q;
            if (cc < a.cols) {
                a.PWV[(size_t) cc * n + r] = pw[q];
                a.PVW[(size_t) (TRD_NB + cc) * n + r] = pw[q];
            }
        }
    }
}

// The same panel for n <= TRC_MAX_N in one thread-block cluster. CTA g owns
// rows 64 g .. 64 g + 63, as CTA g of k_sytrd_panel does; the rows of the
// symmetric product are dealt to the CTAs cyclically. The steps' column, norm
// and dot partials, products and the next row of V and W go to the shared
// memory of the CTAs that read them (remote stores), followed by a hardware
// cluster barrier: three barriers a column and no round trips through L2, where
// the grid's barriers and gathers take 9.7 us a column however small n is: here
// 5.6 us at n = 260 and 3.3 us at n = 24. A CTA's rows of the trailing matrix
// stay in shared memory for the panel, which bounds the panels that run here
// (trc_in_smem).
// What is left is the chain of dependent FP64 operations of a column step, so
// sums that others wait for are short trees of adds over shared values instead
// of shuffles. Every sum has the order of k_sytrd_panel (8 lanes a row, 4 rows a
// warp, 16 warps a CTA, then CTAs in lane order; levels that only add zeros are
// left out): the results are the same bit for bit.
constexpr int TRC_MAX_N = 1024;             // 16 CTAs of 64 rows
constexpr size_t TRC_SMEM_ROWS = 190 << 10; // most bytes of trailing-matrix rows kept per CTA
constexpr int TRC_W = TRD_THREADS / 32;     // warps per CTA

// Address of a shared variable in CTA `rank` of the cluster, and a store to it.
__device__ __forceinline__ unsigned cl_addr(const void *p, int rank)
{
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((unsigned) __cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void cl_store(unsigned addr, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}

// Sum of v[k] over the warp for each k < K (K a power of two, at most 32), in the
// pairing of a shfl_down tree from 16 to 1: while values are left to split, lanes
// keep one half of them and hand over the other, so K sums take ~K shuffles
// instead of 5 K. The sum of value k lands in lane trc_lane<K>(k).
template <int K>
__device__ __forceinline__ int trc_lane(int k)
{
    int lane = 0, half = K / 2;
    for (int o = 16; half > 0; o >>= 1, half >>= 1)
        if (k & half) lane |= o;
    return lane;
}
template <int K>
__device__ __forceinline__ double warp_sums(double (&v)[K], int lane)
{
#pragma unroll
    for (int o = 16, half = K / 2; o > 0; o >>= 1, half >>= 1) {
        if (half > 0) {
            const bool up = lane & o;
#pragma unroll
            for (int k = 0; k < half; k++) {
                const double give = up ? v[k] : v[k + half], keep = up ? v[k + half] : v[k];
                v[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        }
    }
    return v[0];
}

// x[0] + ... + x[15] (stride st) in the pairing of a shfl_down tree.
__device__ __forceinline__ double tree16(const double *x, int st)
{
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = x[k * st] + x[(k + 8) * st];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < o; k++) v[k] += v[k + o];
    return v[0];
}

constexpr int TRC_LD = TRC_W + 1;   // row pitch of the warp partials: lanes read them a row apart
// Sum of the warp partials x[cta][warp] of the whole cluster, in every lane.
__device__ __forceinline__ double cluster_sum(const double (*x)[TRC_LD], int CS, int lane)
{
    double v = lane < CS ? tree16(x[lane], 1) : 0.0;
    for (int o = 8; o > 0; o >>= 1)
        if (o < CS) v += __shfl_xor_sync(0xffffffffu, v, o);
    return __shfl_sync(0xffffffffu, v, 0);
}

// doubles of the column buffer: whole segments
__host__ __device__ constexpr int trc_col(int n) { return (n + TRD_SEG - 1) / TRD_SEG * TRD_SEG; }

template <int NSEG>
__global__ void __launch_bounds__(TRD_THREADS, 1) k_sytrd_cluster(TrdArgs a)
{
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) double dyn[];
    __shared__ double s_wv[TRD_NB], s_vv[TRD_NB], s_row[2 * TRD_NB], s_dot[TRC_W][2 * TRD_NB];
    __shared__ double s_tau[TRD_NB], s_e[TRD_NB], s_d[TRD_NB], s_scal, s_a2;
    // written by the CTAs of the cluster
    __shared__ double g_w[16][TRC_LD], g_dot[16][2 * TRD_NB], g_row[2 * TRD_NB], g_y[NSEG][64];
    cg::cluster_group cl = cg::this_cluster();
    auto sync_all = [&]() {
        if (a.G == 1) __syncthreads();
        else cl.sync();
    };
    const int n = a.n, p = a.p, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int CS = a.G, me = blockIdx.x, rbase = 64 * me;
    double *g_col = dyn, *sA = dyn + trc_col(n);   // the column; this CTA's rows of the trailing matrix
    const int l8 = lane & 7, r = rbase + (tid >> 3);
    const bool own = r < n;
    const int wrow = rbase + 4 * wid;      // first of this warp's four rows
    constexpr int NQ = TRD_NB / 8;
    double pv[NQ], pw[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) pv[q] = pw[q] = 0.0;
    const double *A = a.A;
    // rows p + me, p + me + CS, ... of the trailing matrix are this CTA's
    const int c0 = p & ~31, ld = n - c0;   // columns c0..n-1 are kept: whole 32-column blocks from the panel's on
    for (int k = wid; p + me + k * CS < n; k += TRC_W) {
        const double *src = A + (size_t) (p + me + k * CS) * n + c0;
        for (int c = lane; c < ld; c += 32) sA[k * ld + c] = src[c];
    }
    for (int l = tid; l < 16 * TRC_LD; l += TRD_THREADS) (&g_w[0][0])[l] = 0.0;
    for (int l = tid; l < trc_col(n); l += TRD_THREADS) g_col[l] = 0.0;
    if (tid < 2 * TRD_NB) g_row[tid] = s_row[tid] = 0.0;
    for (int l = tid; l < TRC_W * 2 * TRD_NB; l += TRD_THREADS) (&s_dot[0][0])[l] = 0.0;
    if (tid < TRD_NB) s_wv[tid] = s_vv[tid] = 0.0;
    const unsigned to_col[2] = {cl_addr(g_col + r, min(l8, CS - 1)), cl_addr(g_col + r, min(l8 + 8, CS - 1))};
    const unsigned to_w = cl_addr(&g_w[me][wid], min(lane, CS - 1));
    double arow = (own && r >= p) ? A[(size_t) p * n + r] : 0.0;
    double a2 = 0.0;                       // of the previous column
    sync_all();   // every CTA runs, its partials zeroed, before the first remote store
    for (int c = 0; c < a.cols; c++) {
        const int j = p + c;
        // ---- phase 1: column j of the panel-corrected matrix, rows j..n-1 (g_row: row j's V and W; W's
        // entry of the last column still lacks its a2 v)
        if (wrow < n && wrow + 3 >= j) {
            double v = l8 == 0 ? arow : 0.0;
#pragma unroll
            for (int q = 0; q < NQ; q++) {   // columns behind c - 1 hold zeros
                const int cc = l8 + 8 * q;
                const double vj = g_row[cc], w0 = g_row[TRD_NB + cc];
                const double wj = cc == c - 1 ? w0 + a2 * vj : w0;
                v -= pv[q] * wj + pw[q] * vj;
            }
            v += __shfl_xor_sync(0xffffffff, v, 1);
            v += __shfl_xor_sync(0xffffffff, v, 2);
            v += __shfl_xor_sync(0xffffffff, v, 4);
            if (own && r >= j) {
                if (l8 < CS) cl_store(to_col[0], v);
                if (l8 + 8 < CS) cl_store(to_col[1], v);
            }
        }
        sync_all();
        if (j == n - 1) {
            if (tid == 0) s_d[c] = g_col[j];
            break;
        }
        // ---- phase 2: the reflector (every CTA forms the same one), y = A v, panel dots
        if (wid == 0) {
            // |x|^2 of rows j+2.. in the groups' order: 4 rows, 16 of those, then the 64-row groups in lane order
            constexpr int H = 2 * NSEG;   // lanes 0-15: group 2 h, lanes 16-31: group 2 h + 1
            double part[H];
#pragma unroll
            for (int h = 0; h < H; h++) {
                const int rr = 128 * h + 4 * lane;   // the buffer is zero behind the column
                const double2 u = *reinterpret_cast<const double2 *>(g_col + rr);
                const double2 v = *reinterpret_cast<const double2 *>(g_col + rr + 2);
                const double x0 = rr >= j + 2 ? __dmul_rn(u.x, u.x) : 0.0, x1 = rr + 1 >= j + 2 ? __dmul_rn(u.y, u.y) : 0.0;
                const double x2 = rr + 2 >= j + 2 ? __dmul_rn(v.x, v.x) : 0.0;
                const double x3 = rr + 3 >= j + 2 ? __dmul_rn(v.y, v.y) : 0.0;
                part[h] = (x0 + x2) + (x1 + x3);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1)
#pragma unroll
                for (int h = 0; h < H; h++) part[h] += __shfl_xor_sync(0xffffffffu, part[h], o);
            // the tree over groups 0..15 (zeros behind the last): groups g and g + 8, then + 4, + 2, + 1
            double s = 0.0;
#pragma unroll
            for (int half = 1; half >= 0; half--) {   // even groups first, then the odd ones
                double g[8];
#pragma unroll
                for (int h = 0; h < 8; h++) g[h] = h < H ? __shfl_sync(0xffffffffu, part[h < H ? h : 0], 16 * (1 - half)) : 0.0;
                const double x = ((g[0] + g[4]) + (g[2] + g[6])) + ((g[1] + g[5]) + (g[3] + g[7]));
                s = half ? x : s + x;
            }
            const double alpha = g_col[j + 1];
            double tau, beta, scal;
            if (s == 0.0) {
                tau = 0.0;
                beta = alpha;
                scal = 0.0;
            } else {
                const double nrm = sqrt(alpha * alpha + s);
                beta = alpha >= 0.0 ? -nrm : nrm;
                tau = (beta - alpha) / beta;
                scal = 1.0 / (alpha - beta);
            }
            if (lane == 0) {
                s_tau[c] = tau;
                s_scal = scal;
                s_d[c] = g_col[j];
                s_e[c] = beta;
            }
        }
        __syncthreads();
        const double tau = s_tau[c], scal = s_scal;
        const double vr_own = (own && r > j) ? (r == j + 1 ? 1.0 : g_col[r] * scal) : 0.0;
        if (l8 == (c & 7)) {
#pragma unroll
            for (int q = 0; q < NQ; q++)
                if (q == (c >> 3)) pv[q] = vr_own;
        }
        if (c > 0 && rbase < n) {
            // panel dots W^T v and V^T v of this CTA's rows: 4 rows a warp by shuffles, then the warps in order;
            // the last two warps add them up while the others go on to the product
            const int w0 = max(0, (j + 1 - rbase) >> 2), w1 = min(TRC_W, (n - rbase + 3) >> 2);   // warps with rows > j
            if (wid == w0 - 1) s_dot[wid][lane] = s_dot[wid][lane + 32] = 0.0;   // its last row is done
            if (wid >= w0 && wid < w1) {
                // lanes without bit 8 keep W^T v, with it V^T v; without bit 16 columns 0..15, with it 16..31
                const bool hi8 = lane & 8, hi16 = lane & 16;
                double d[NQ];
#pragma unroll
                for (int q = 0; q < NQ; q++) {
                    const double dw = __dmul_rn(pw[q], vr_own), dv = __dmul_rn(pv[q], vr_own);
                    d[q] = (hi8 ? dv : dw) + __shfl_xor_sync(0xffffffff, hi8 ? dw : dv, 8);
                }
                static_assert(NQ == 4, "two columns per lane after the second exchange");
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const double x = (hi16 ? d[q + 2] : d[q]) + __shfl_xor_sync(0xffffffff, hi16 ? d[q] : d[q + 2], 16);
                    s_dot[wid][(hi8 ? TRD_NB : 0) + l8 + 8 * (q + (hi16 ? 2 : 0))] = x;
                }
            }
            if (wid < TRC_W - 2) {
                asm volatile("bar.arrive 1, %0;" ::"n"(TRD_THREADS) : "memory");
            } else {
                asm volatile("bar.sync 1, %0;" ::"n"(TRD_THREADS) : "memory");
                const int k = tid & 63;
                double sacc = 0.0, x[TRC_W];
#pragma unroll
                for (int w = 0; w < TRC_W; w++) x[w] = s_dot[w][k];   // idle warps hold zeros
#pragma unroll
                for (int w = 0; w < TRC_W; w++) sacc += x[w];
                for (int q = 0; q < CS; q++) cl_store(cl_addr(&g_dot[me][k], q), sacc);
            }
        }
        {
            // rows p + me + CS (wid + 16 k), k = 0..3, by segments of TRD_SEG columns
            constexpr int K = NSEG == 3 ? 16 : 4 * NSEG;   // sums of this warp: (segment, k), padded to a power of two
            const int s0 = (j + 1) / TRD_SEG;
            double sum[K];
#pragma unroll
            for (int k = 0; k < K; k++) sum[k] = 0.0;
            // rows are dealt in order, so the last row of a warp tells whether it has one behind row j
            const int most = (n - 1 - p - me) / CS;   // last local row of this CTA
            const int last = n - 1 - p < me || most < wid ? -1 : p + me + CS * (most - ((most - wid) & (TRC_W - 1)));
            const bool any = last > j;
#pragma unroll
            for (int sg = 0; sg < NSEG; sg++) {
                if (sg < s0 || !any) continue;
                double vs[TRD_SEG / 32];
                unsigned on = 0;   // this lane's columns j+1..n-1
#pragma unroll
                for (int x = 0; x < TRD_SEG / 32; x++) {
                    const int c2 = sg * TRD_SEG + lane + 32 * x;
                    vs[x] = c2 == j + 1 ? 1.0 : g_col[c2] * scal;
                    on |= (unsigned) (c2 > j && c2 < n) << x;
                }
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int kk = wid + TRC_W * k, rr = p + me + CS * kk;
                    if (rr <= j || rr >= n) continue;
                    const double *row = sA + kk * ld - c0 + sg * TRD_SEG + lane;
                    double acc[TRD_SEG / 32];
#pragma unroll
                    for (int x = 0; x < TRD_SEG / 32; x++)
                        acc[x] = (on >> x) & 1 ? __dmul_rn(row[32 * x], vs[x]) : 0.0;
                    sum[sg * 4 + k] = ((acc[0] + acc[4]) + (acc[2] + acc[6])) + ((acc[1] + acc[5]) + (acc[3] + acc[7]));
                }
            }
            if (any) {   // uniform over the warp
                const double y = warp_sums<K>(sum, lane);
#pragma unroll
                for (int k = 0; k < 4 * NSEG; k++) {
                    const int rr = p + me + CS * (wid + TRC_W * (k & 3));
                    if (lane == trc_lane<K>(k) && rr > j && rr < n)
                        cl_store(cl_addr(&g_y[k >> 2][rr & 63], rr >> 6), y);
                }
            }
        }
        sync_all();
        // ---- phase 3: w = tau (y - V (W^T v) - W (V^T v)) for this row, partial w.v
        double ypart = 0.0;
        const int s0 = (j + 1) / TRD_SEG;
        if (own && r > j)
            for (int sg = s0 + l8; sg < NSEG; sg += 8) ypart += g_y[sg][r - rbase];
        if (tid < 64 && (tid & 31) < c) {
            double x = 0.0;
            if (CS > 8) {
                double y[16];
#pragma unroll
                for (int q = 0; q < 16; q++) y[q] = q < CS && 64 * q < n ? g_dot[q][tid] : 0.0;
                x = tree16(y, 1);
            } else {
                double y[8];
#pragma unroll
                for (int q = 0; q < 8; q++) y[q] = q < CS && 64 * q < n ? g_dot[q][tid] : 0.0;
                x = ((y[0] + y[4]) + (y[2] + y[6])) + ((y[1] + y[5]) + (y[3] + y[7]));
            }
            (tid < 32 ? s_wv : s_vv)[tid & 31] = x;
        }
        const bool nxt = c + 1 < a.cols;
        arow = (nxt && own && r >= j + 1) ? A[(size_t) (j + 1) * n + r] : 0.0;
        __syncthreads();
        if (wrow < n && wrow + 3 > j) {
            double t = ypart;
#pragma unroll
            for (int q = 0; q < NQ; q++) {
                // column c itself: W's entry is still zero, V's meets a zero sum
                const int cc = l8 + 8 * q;
                t -= pv[q] * s_wv[cc] + pw[q] * s_vv[cc];
            }
            t += __shfl_xor_sync(0xffffffff, t, 1);
            t += __shfl_xor_sync(0xffffffff, t, 2);
            t += __shfl_xor_sync(0xffffffff, t, 4);
            const double w = (own && r > j) ? tau * t : 0.0;
            if (l8 == (c & 7)) {
#pragma unroll
                for (int q = 0; q < NQ; q++)
                    if (q == (c >> 3)) pw[q] = w;
            }
            if (nxt && r == j + 1) {   // row j+1's V and W for everyone (W of column c before its a2 v)
#pragma unroll
                for (int q = 0; q < NQ; q++) {
                    s_row[l8 + 8 * q] = pv[q];
                    s_row[TRD_NB + l8 + 8 * q] = pw[q];
                }
            }
            double wd = __dmul_rn(w, vr_own);   // the same in a row's 8 lanes
            wd += __shfl_xor_sync(0xffffffff, wd, 16);
            wd += __shfl_xor_sync(0xffffffff, wd, 8);
            if (lane < CS) cl_store(to_w, wd);
        } else if (wrow < n && wrow + 3 == j) {   // these rows are done
            if (lane < CS) cl_store(to_w, 0.0);
        }
        if (nxt && me == (j + 1) / 64) {
            __syncthreads();
            const double x = s_row[tid & 63];
            for (int q = tid >> 6; q < CS; q += TRD_THREADS / 64) cl_store(cl_addr(&g_row[tid & 63], q), x);
        }
        sync_all();
        // ---- phase 4: a2 = -tau/2 (w.v), w += a2 v
        if (wid == 0) {
            const double x = -0.5 * tau * cluster_sum(g_w, CS, lane);
            if (lane == 0) s_a2 = x;
        }
        __syncthreads();
        a2 = s_a2;
        if (l8 == (c & 7)) {
#pragma unroll
            for (int q = 0; q < NQ; q++)
                if (q == (c >> 3)) pw[q] += a2 * pv[q];
        }
    }
    __syncthreads();   // s_d of the last column: written by thread 0, read below by the column's own thread
    // the reflectors, and the final W of the rows behind the panel, into both stacked panels (nothing is written
    // to global memory inside the loop: a barrier's release would wait for it)
    if (own) {
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const int cc = l8 + 8 * q;
            if (cc < a.cols && r > p + cc) {
                a.VT[(size_t) (p + cc) * n + r] = pv[q];
                a.PVW[(size_t) cc * n + r] = pv[q];
                a.PWV[(size_t) (TRD_NB + cc) * n + r] = pv[q];
            }
            if (cc < a.cols && r >= p + a.cols) {
                a.PWV[(size_t) cc * n + r] = pw[q];
                a.PVW[(size_t) (TRD_NB + cc) * n + r] = pw[q];
            }
        }
    }
    if (me == 0 && tid < a.cols) {
        a.d[p + tid] = s_d[tid];
        if (p + tid < n - 1) {
            a.e[p + tid] = s_e[tid];
            a.tau[p + tid] = s_tau[tid];
        }
    }
    sync_all();   // no CTA leaves while another may still write to it
}

// CTAs of the cluster: every 64 rows need an owner; up to 16, about 24 rows of the product each.
int trc_ctas(int n) { return n <= 64 ? 1 : std::min(16, std::max((n + 63) / 64, (n + 23) / 24)); }
// Bytes of a CTA's rows of the trailing matrix of size m (with the panel's leading partial column block).
size_t trc_rows_bytes(int n, int m) { return sizeof(double) * (size_t) ((m + trc_ctas(n) - 1) / trc_ctas(n)) * (m + 31); }
// The panels that run in a cluster: those whose trailing rows fit in its shared memory (616 rows on 16 CTAs).
// Larger ones would stream A from L2 into 16 SMs: 16.6 us a column at 1010 rows against 10.4 us on the whole chip.
bool trc_in_smem(int n, int m) { return trc_rows_bytes(n, m) <= TRC_SMEM_ROWS; }
size_t trc_smem(int n, int m) { return sizeof(double) * (size_t) trc_col(n) + trc_rows_bytes(n, m); }

const void *trc_kernel(int n)
{
    switch ((n + TRD_SEG - 1) / TRD_SEG) {
    case 1: return (const void *) k_sytrd_cluster<1>;
    case 2: return (const void *) k_sytrd_cluster<2>;
    case 3: return (const void *) k_sytrd_cluster<3>;
    default: return (const void *) k_sytrd_cluster<4>;
    }
}

// Launch configuration of the cluster panel with m trailing rows; attr must outlive it.
cudaLaunchConfig_t trc_config(int n, int m, cudaStream_t s, cudaLaunchAttribute *attr)
{
    const unsigned cs = trc_ctas(n);
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = cs;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cs);
    cfg.blockDim = dim3(TRD_THREADS);
    cfg.dynamicSmemBytes = trc_smem(n, m);
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// Whether the device takes the cluster panel for n rows.
bool trc_usable(int n)
{
    if (n > TRC_MAX_N) return false;
    const void *k = trc_kernel(n);
    const int most = (int) (sizeof(double) * trc_col(n) + TRC_SMEM_ROWS);
    if (cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t cfg = trc_config(n, n, 0, &attr);
    cfg.dynamicSmemBytes = most;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, k, &cfg) != cudaSuccess || clusters < 1) {
        cudaGetLastError();
        return false;
    }
    return true;
}

// Partial Gram matrices V_B^T V_B of the reflector blocks (the reflectors of
// block B are rows p0..p0+bb-1 of VT, zero before column p0 + 1): CTA (B,
// 32 x 32 tile, slice ks of the columns) writes its slice's sum to Gp[B][ks].
__global__ void __launch_bounds__(256) k_wy_gram(const double *VT, double *Gp, int n, int nref)
{
    __shared__ double As[32][65], Bs[32][65];
    const int B = blockIdx.x, tile = blockIdx.y, ks = blockIdx.z;
    const int p0 = B * BT_NB, bb = min(BT_NB, nref - p0);
    const int ta = tile / (BT_NB / 32), tb = tile % (BT_NB / 32);
    const int K0 = p0 + 1, K = n - K0, kper = (K + GR_KS - 1) / GR_KS;
    const int k0 = K0 + ks * kper, k1 = min(n, k0 + kper);
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    double acc[2][2] = {};
    for (int kc = k0; kc < k1; kc += 64) {
        for (int l = threadIdx.x; l < 32 * 64; l += 256) {
            const int rr = l / 64, kk = l % 64, k = kc + kk;
            const int ra = ta * 32 + rr, rb = tb * 32 + rr;
            As[rr][kk] = (ra < bb && k < k1) ? VT[(size_t) (p0 + ra) * n + k] : 0.0;
            Bs[rr][kk] = (rb < bb && k < k1) ? VT[(size_t) (p0 + rb) * n + k] : 0.0;
        }
        __syncthreads();
#pragma unroll 8
        for (int kk = 0; kk < 64; kk++) {
            const double a0 = As[ty][kk], a1 = As[ty + 16][kk], b0 = Bs[tx][kk], b1 = Bs[tx + 16][kk];
            acc[0][0] += a0 * b0;
            acc[0][1] += a0 * b1;
            acc[1][0] += a1 * b0;
            acc[1][1] += a1 * b1;
        }
        __syncthreads();
    }
    double *G = Gp + (size_t) (B * GR_KS + ks) * BT_NB * BT_NB;
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int jj = 0; jj < 2; jj++) G[(size_t) (ta * 32 + ty + 16 * i) * BT_NB + tb * 32 + tx + 16 * jj] = acc[i][jj];
}

// T of the compact WY form of each block of BT_NB reflectors:
// H_p0 ... H_(p0+bb-1) = I - V T V^T, T upper triangular (LAPACK dlarft,
// forward, columnwise), from the block's Gram matrix (the sum of its
// GR_KS slices). One CTA per block, one warp per four rows of T: row i needs
// only its own entries, T(i, c) = -tau_c sum_(l = i..c-1) T(i, l) G(l, c), so a
// warp runs along its row and adds T(i, l) G(l, c) to every later column c (lane
// c % 32) as soon as T(i, l) is known. The sums run over l in the order of the
// column-by-column form, which one thread per row ran as a serial chain of
// bb^2 / 2 dependent multiply-adds: 280 us per call, whatever n, now 50 us
// (most of it the Gram slices' sum).
constexpr int TF_THREADS = 1024, TF_ROWS = BT_NB / (TF_THREADS / 32);
__global__ void __launch_bounds__(TF_THREADS) k_wy_tfactor(const double *Gp, const double *tau, double *Tf, int nref)
{
    extern __shared__ double tsm[];        // the Gram matrix, BT_NB x BT_NB
    constexpr int NC = BT_NB / 32;
    const int B = blockIdx.x, p0 = B * BT_NB, bb = min(BT_NB, nref - p0), tid = threadIdx.x, lane = tid & 31;
    const double *G = Gp + (size_t) B * GR_KS * BT_NB * BT_NB;
    for (int l = tid; l < BT_NB * BT_NB; l += TF_THREADS) {
        double g = 0.0;
#pragma unroll
        for (int ks = 0; ks < GR_KS; ks++) g += G[(size_t) ks * BT_NB * BT_NB + l];
        tsm[l] = g;
    }
    double tc[NC];
#pragma unroll
    for (int q = 0; q < NC; q++) tc[q] = lane + 32 * q < bb ? tau[p0 + lane + 32 * q] : 0.0;
    __syncthreads();
    double acc[TF_ROWS][NC], t[TF_ROWS][NC];
    const int i0 = tid >> 5;               // rows i0, i0 + 32, ...
#pragma unroll
    for (int x = 0; x < TF_ROWS; x++)
#pragma unroll
        for (int q = 0; q < NC; q++) acc[x][q] = t[x][q] = 0.0;
#pragma unroll
    for (int lq = 0; lq < NC; lq++) {
        for (int ll = 0; ll < 32; ll++) {
            const int l = 32 * lq + ll;
            if (l < i0) continue;
            if (l >= bb) break;
            double g[NC];
#pragma unroll
            for (int q = lq; q < NC; q++) g[q] = tsm[l * BT_NB + lane + 32 * q];
#pragma unroll
            for (int x = 0; x < TF_ROWS; x++) {
                const int i = i0 + 32 * x;
                if (l < i) continue;
                // lane ll holds column l: its sum is complete
                const double mine = l == i ? tc[lq] : -tc[lq] * acc[x][lq];
                if (lane == ll) t[x][lq] = mine;
                const double tl = __shfl_sync(0xffffffffu, mine, ll);
#pragma unroll
                for (int q = lq; q < NC; q++)
                    if (lane + 32 * q > l) acc[x][q] = fma(tl, g[q], acc[x][q]);
            }
        }
    }
#pragma unroll
    for (int x = 0; x < TF_ROWS; x++)
#pragma unroll
        for (int q = 0; q < NC; q++)
            Tf[(size_t) B * BT_NB * BT_NB + (size_t) (i0 + 32 * x) * BT_NB + lane + 32 * q] = t[x][q];
}

// ------------------------------------------------------------------ divide and conquer
struct DcNodes {
    const int *lo, *mid, *hi;
    double *rho;      // per node, 2 |e[mid-1]|
    int *kcnt, *rcnt; // per node: non-deflated count, rotation count
};

struct DcPos {        // per position of the tridiagonal (node-local arrays start at lo)
    double *lam;      // eigenvalues of the solved pieces (ascending within each piece)
    double *ds;       // sorted, deflation-modified d
    double *dK, *zK;  // non-deflated d and z (compact)
    double *lamb, *tau;  // root j = lamb[j] + tau[j], lamb the nearer pole
    double *zh, *nrm;
    double *lamnew;
    int *perm;        // sorted position -> index into the concatenated children
    int *keep, *defl; // sorted positions kept / deflated (compact)
    int *rowinfo;     // sorted position -> kept index i, or -(deflated index + 1)
    int *colsrc;      // output column -> secular root j (< k) or k + deflated index
    int2 *rot;        // Givens rotations of the close pairs (rows pj, nj, sorted positions)
    double2 *rotcs;   // their (C, S)
};

// Both eigenvector buffers start as the identity: a piece of size one keeps
// its vector in both, so a merge finds it whichever buffer it reads.
__global__ void k_dc_init(const double *d, const double *e, double *lam, double *Qa, double *Qb, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    // every boundary i|i+1 is the split point of exactly one merge: tear both sides
    double v = d[i];
    if (i + 1 < n) v -= fabs(e[i]);
    if (i > 0) v -= fabs(e[i - 1]);
    lam[i] = v;
    Qa[(size_t) i * n + i] = 1.0;
    Qb[(size_t) i * n + i] = 1.0;
}

// The deflation scan of a merge, by one thread: small z components, and close
// pairs that a Givens rotation deflates (LAPACK dlaed2's two tests). sd, sz are
// the sorted d and z (modified by the rotations).
__device__ __forceinline__ void deflation_scan(double *sd, double *sz, int m, double rho, double zmax, double tol,
                                               int *keep, int *defl, int *rowinfo, int2 *rot, double2 *rotcs, int &k,
                                               int &nr)
{
    int nd_ = 0;
    k = nr = 0;
    if (rho * zmax <= tol) {
        for (int s = 0; s < m; s++) {
            rowinfo[s] = -(nd_ + 1);
            defl[nd_++] = s;
        }
    } else {
        int pj = -1;
        for (int s = 0; s < m; s++) {
            if (rho * fabs(sz[s]) <= tol) {
                rowinfo[s] = -(nd_ + 1);
                defl[nd_++] = s;
                continue;
            }
            if (pj < 0) {
                pj = s;
                continue;
            }
            // close pair: |t C S| <= tol with C = z_s / h, S = -z_pj / h, h = hypot(z_s, z_pj)
            const double zp = sz[pj], zs = sz[s], t = sd[s] - sd[pj];
            if (fabs(t * zs * zp) <= tol * (zs * zs + zp * zp)) {
                const double tt = hypot(zs, zp), C = zs / tt, S = -zp / tt;
                sz[s] = tt;
                sz[pj] = 0.0;
                rot[nr] = make_int2(pj, s);
                rotcs[nr] = make_double2(C, S);
                nr++;
                const double dp = sd[pj] * C * C + sd[s] * S * S;
                sd[s] = sd[pj] * S * S + sd[s] * C * C;
                sd[pj] = dp;
                rowinfo[pj] = -(nd_ + 1);
                defl[nd_++] = pj;
                pj = s;
            } else {
                rowinfo[pj] = k;
                keep[k++] = pj;
                pj = s;
            }
        }
        if (pj >= 0) {
            rowinfo[pj] = k;
            keep[k++] = pj;
        }
    }
}

// Sorting of the two halves, z, the tolerance and the deflation scan. One CTA per node.
__global__ void __launch_bounds__(512) k_dc_deflate(DcNodes nd, DcPos ps, const double *Q, const double *e, int n,
                                                    int node0)
{
    extern __shared__ double dsm[];
    __shared__ double s_red[33];
    const int node = node0 + blockIdx.x;
    const int lo = nd.lo[node], mid = nd.mid[node], hi = nd.hi[node];
    const int m = hi - lo, m1 = mid - lo, m2 = hi - mid;
    double *sd = dsm, *sz = dsm + m;
    int *sp = (int *) (dsm + 2 * m);
    const double rho_raw = e[mid - 1];
    const double rho = 2.0 * fabs(rho_raw), sg = rho_raw >= 0.0 ? 1.0 : -1.0;
    const double *L1 = ps.lam + lo, *L2 = ps.lam + mid;
    const double rs2 = 1.0 / sqrt(2.0);
    // every slot holds a valid index even if non-finite values make the merge below collide
    for (int idx = threadIdx.x; idx < m; idx += blockDim.x) {
        sd[idx] = 0.0;
        sz[idx] = 0.0;
        sp[idx] = idx;
    }
    __syncthreads();
    double dmax = 0.0, zmax = 0.0;
    for (int idx = threadIdx.x; idx < m; idx += blockDim.x) {
        double x, zz;
        int pos;
        if (idx < m1) {
            x = L1[idx];
            zz = Q[(size_t) (mid - 1) * n + lo + idx];
            int a = 0, b = m2;   // first L2 >= x
            while (a < b) {
                const int c = (a + b) >> 1;
                if (L2[c] < x) a = c + 1; else b = c;
            }
            pos = idx + a;
        } else {
            const int i2 = idx - m1;
            x = L2[i2];
            zz = sg * Q[(size_t) mid * n + mid + i2];
            int a = 0, b = m1;   // first L1 > x
            while (a < b) {
                const int c = (a + b) >> 1;
                if (L1[c] <= x) a = c + 1; else b = c;
            }
            pos = i2 + a;
        }
        pos = min(max(pos, 0), m - 1);
        zz *= rs2;
        sd[pos] = x;
        sz[pos] = zz;
        sp[pos] = idx;
        dmax = fmax(dmax, fabs(x));
        zmax = fmax(zmax, fabs(zz));
    }
    dmax = block_max_all<512>(dmax, s_red);
    zmax = block_max_all<512>(zmax, s_red);
    const double tol = 8.0 * DBL_EPSILON * fmax(dmax, zmax);
    int *keep = ps.keep + lo, *defl = ps.defl + lo, *rowinfo = ps.rowinfo + lo;
    if (threadIdx.x == 0) {
        int k, nr;
        deflation_scan(sd, sz, m, rho, zmax, tol, keep, defl, rowinfo, ps.rot + lo, ps.rotcs + lo, k, nr);
        nd.kcnt[node] = k;
        nd.rcnt[node] = nr;
        nd.rho[node] = rho;
    }
    __syncthreads();
    const int k = nd.kcnt[node];
    for (int s = threadIdx.x; s < m; s += blockDim.x) {
        ps.ds[lo + s] = sd[s];
        ps.perm[lo + s] = sp[s];
    }
    for (int i = threadIdx.x; i < k; i += blockDim.x) {
        const int s = keep[i];
        ps.dK[lo + i] = sd[s];
        ps.zK[lo + i] = sz[s];
    }
}

// Block tables: entry b = (node, first item) for the items [first, first + chunk) of that node.
__device__ __forceinline__ void secular_parts(const double *sd, const double *sz, int k, int j, double rho,
                                              double dorg, double t, int lane, double &p1, double &dp1, double &p2,
                                              double &dp2)
{
    double a = 0.0, b = 0.0, c = 0.0, d = 0.0;
    for (int i = lane; i < k; i += 32) {
        const double q = sz[i] / ((sd[i] - dorg) - t);
        if (i <= j) {
            a += sz[i] * q;
            b += q * q;
        } else {
            c += sz[i] * q;
            d += q * q;
        }
    }
    double v[4] = {a, b, c, d};   // the sums of four shuffle trees, in 6 shuffles instead of 20
    const double x = warp_sums<4>(v, lane);
    p1 = rho * __shfl_sync(0xffffffffu, x, trc_lane<4>(0));
    dp1 = rho * __shfl_sync(0xffffffffu, x, trc_lane<4>(1));
    p2 = rho * __shfl_sync(0xffffffffu, x, trc_lane<4>(2));
    dp2 = rho * __shfl_sync(0xffffffffu, x, trc_lane<4>(3));
}

// Roots of f(l) = 1 + rho sum_i z_i^2 / (d_i - l) = 0, one warp per root:
// l_j = pole + tau, the pole the nearer of d_j, d_(j+1) (its position is the
// origin of tau, so tau keeps full relative accuracy), tau bracketed by the
// signs of f. Each step fits psi1 + psi2 on either side of the root by
// c + s / (pole - t) matched to value and slope at the current tau (the two
// poles around the root) and takes the model's root inside the bracket;
// a bisection step (geometric while the bracket spans more than a factor 4)
// when it falls outside. Stops when the step is below 2 eps |tau| or the
// bracket closes. At the root the model's step is rounding and often falls on the
// bracket's end, so most roots go through tens of bisections of a wide bracket
// before it closes (50 us per level however few roots). at_noise stops where
// |f| is within the rounding of its own terms instead, which determines the root
// as far as f can (the criterion of LAPACK's dlaed4, whose eps is the unit
// roundoff DBL_EPSILON / 2): 13 us. The bracketed
// stop stays for the eigenbases of the accelerated form and of X and (P|Q)^-1/2,
// whose users amplify the last bits (1e-16 in X moves its density by 1e-9).
// One warp; the root of position j as org, tau (tau relative to sd[org]).
__device__ __forceinline__ void secular_root(const double *sd, const double *sz, int k, int j, double rho, int lane,
                                             bool at_noise, int &org, double &tau)
{
    if (k == 1) {
        org = 0;
        tau = rho * sz[0] * sz[0];
    } else {
        const bool last = j == k - 1;
        double a, b;   // bracket in tau: f(a) < 0 < f(b)
        if (last) {
            double s = 0.0;
            for (int i = lane; i < k; i += 32) s += sz[i] * sz[i];
            org = j;
            a = 0.0;
            b = rho * warp_sum_bcast(s);
        } else {
            const double delta = sd[j + 1] - sd[j];
            double p1, dp1, p2, dp2;
            secular_parts(sd, sz, k, j, rho, sd[j], 0.5 * delta, lane, p1, dp1, p2, dp2);
            if (1.0 + p1 + p2 > 0.0) {
                org = j;
                a = 0.0;
                b = 0.5 * delta;
            } else {
                org = j + 1;
                a = -0.5 * delta;
                b = 0.0;
            }
        }
        const double dorg = sd[org];
        const double del1 = sd[j] - dorg;                       // lower pole, relative
        const double del2 = last ? 0.0 : sd[j + 1] - dorg;      // upper pole, relative
        tau = 0.5 * (a + b);
        for (int it = 0; it < 200; it++) {
            double p1, dp1, p2, dp2;
            secular_parts(sd, sz, k, j, rho, dorg, tau, lane, p1, dp1, p2, dp2);
            const double f = 1.0 + p1 + p2;
            if (f == 0.0) break;
            if (at_noise && fabs(f) <= 0.5 * DBL_EPSILON * (8.0 * (1.0 + fabs(p1) + fabs(p2)) + fabs(tau) * (dp1 + dp2))) break;
            if (f < 0.0) a = tau; else b = tau;
            if (!(b - a > 4.0 * DBL_EPSILON * fmax(fabs(a), fabs(b)))) break;
            // two-pole model: C + s1 / (del1 - x) + s2 / (del2 - x) = 0
            const double e1 = del1 - tau, s1 = dp1 * e1 * e1, c1 = p1 - s1 / e1;
            double x = NAN;
            if (last) {
                const double C = 1.0 + c1 + p2;
                if (C > 0.0) x = del1 + s1 / C;
            } else {
                const double e2 = del2 - tau, s2 = dp2 * e2 * e2, c2 = p2 - s2 / e2;
                const double C = 1.0 + c1 + c2;
                const double qa = C, qb = -(C * (del1 + del2) + s1 + s2), qc = C * del1 * del2 + s1 * del2 + s2 * del1;
                const double disc = qb * qb - 4.0 * qa * qc;
                if (disc >= 0.0) {
                    const double q = -0.5 * (qb + copysign(sqrt(disc), qb));
                    const double r1 = q / qa, r2 = qc / q;
                    const bool in1 = r1 > a && r1 < b, in2 = r2 > a && r2 < b;
                    x = in1 && (!in2 || fabs(r1 - tau) < fabs(r2 - tau)) ? r1 : (in2 ? r2 : NAN);
                }
            }
            if (!(x > a && x < b)) {   // bisection, geometric on the side of the origin while the bracket is wide
                const double lo_ = fmin(fabs(a), fabs(b)), hi_ = fmax(fabs(a), fabs(b));
                const double sg = (a + b) >= 0.0 ? 1.0 : -1.0;
                x = (lo_ > 0.0 && hi_ > 4.0 * lo_ && a * b > 0.0) ? sg * sqrt(lo_ * hi_) : 0.5 * (a + b);
                if (x == 0.0) x = 0.5 * (a + b);
                if (!(x > a && x < b)) break;
            }
            const bool done = fabs(x - tau) <= 2.0 * DBL_EPSILON * fabs(x);
            tau = x;
            if (done) break;
        }
    }
}

__global__ void __launch_bounds__(256) k_dc_secular(DcNodes nd, DcPos ps, const int2 *tab, bool at_noise)
{
    extern __shared__ double dsm[];
    const int2 tb = tab[blockIdx.x];
    const int node = tb.x, lo = nd.lo[node], k = nd.kcnt[node];
    if (tb.y >= k) return;
    double *sd = dsm, *sz = dsm + k;
    for (int i = threadIdx.x; i < k; i += blockDim.x) {
        sd[i] = ps.dK[lo + i];
        sz[i] = ps.zK[lo + i];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, j = tb.y + (threadIdx.x >> 5);
    if (j >= k) return;
    const double rho = nd.rho[node];
    int org;
    double tau;
    secular_root(sd, sz, k, j, rho, lane, at_noise, org, tau);
    if (lane == 0) {
        ps.lamb[lo + j] = sd[org];
        ps.tau[lo + j] = tau;
    }
}

// z recomputed from the roots (Gu-Eisenstat): zh_i^2 = -(d_i - l_i) prod_(j != i) (d_i - l_j) / (d_i - d_j).
__global__ void __launch_bounds__(256) k_dc_zhat(DcNodes nd, DcPos ps, const int2 *tab)
{
    extern __shared__ double dsm[];
    const int2 tb = tab[blockIdx.x];
    const int node = tb.x, lo = nd.lo[node], k = nd.kcnt[node];
    if (tb.y >= k) return;
    double *sd = dsm, *sl = dsm + k, *st = dsm + 2 * k;
    for (int i = threadIdx.x; i < k; i += blockDim.x) {
        sd[i] = ps.dK[lo + i];
        sl[i] = ps.lamb[lo + i];
        st[i] = ps.tau[lo + i];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, i = tb.y + (threadIdx.x >> 5);
    if (i >= k) return;
    const double di = sd[i];
    double pr = 1.0;
    for (int j = lane; j < k; j += 32) {
        const double del = (di - sl[j]) - st[j];
        pr *= (j == i) ? del : del / (di - sd[j]);
    }
    pr = warp_prod_bcast(pr);
    if (lane == 0) ps.zh[lo + i] = copysign(sqrt(fmax(-pr, 0.0)), ps.zK[lo + i]);
}

// Norm of each secular eigenvector u_j(i) = zh_i / (d_i - l_j).
__global__ void __launch_bounds__(256) k_dc_norms(DcNodes nd, DcPos ps, const int2 *tab)
{
    extern __shared__ double dsm[];
    const int2 tb = tab[blockIdx.x];
    const int node = tb.x, lo = nd.lo[node], k = nd.kcnt[node];
    if (tb.y >= k) return;
    double *sd = dsm, *sz = dsm + k;
    for (int i = threadIdx.x; i < k; i += blockDim.x) {
        sd[i] = ps.dK[lo + i];
        sz[i] = ps.zh[lo + i];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, j = tb.y + (threadIdx.x >> 5);
    if (j >= k) return;
    const double lb = ps.lamb[lo + j], tj = ps.tau[lo + j];
    double s = 0.0;
    for (int i = lane; i < k; i += 32) {
        const double u = sz[i] / ((sd[i] - lb) - tj);
        s += u * u;
    }
    s = warp_sum_bcast(s);
    if (lane == 0) ps.nrm[lo + j] = sqrt(s);
}

// Output order of the node's eigenvalues (ascending; ties by source index) by rank counting.
__global__ void __launch_bounds__(DC_CHUNK) k_dc_order(DcNodes nd, DcPos ps, const int2 *tab)
{
    extern __shared__ double dsm[];
    const int2 tb = tab[blockIdx.x];
    const int node = tb.x, lo = nd.lo[node], m = nd.hi[node] - lo, k = nd.kcnt[node];
    double *sv = dsm;
    for (int a = threadIdx.x; a < m; a += blockDim.x)
        sv[a] = (a < k) ? ps.lamb[lo + a] + ps.tau[lo + a] : ps.ds[lo + ps.defl[lo + a - k]];
    __syncthreads();
    const int a = tb.y + threadIdx.x;
    if (a >= m) return;
    const double x = sv[a];
    int r = 0;
    for (int b = 0; b < m; b++) {
        const double y = sv[b];
        r += (y < x || (y == x && b < a)) ? 1 : 0;
    }
    r = min(r, m - 1);
    ps.lamnew[lo + r] = x;
    ps.colsrc[lo + r] = a;
}

// The merge's eigenvector matrix U, one warp per sorted position s (written to
// row perm[s], i.e. in the children's order): column c = secular vector j
// (normalised) or the unit vector of a deflated position.
__global__ void __launch_bounds__(256) k_dc_build(DcNodes nd, DcPos ps, const int2 *tab, double *Us, int n)
{
    const int2 tb = tab[blockIdx.x];
    const int node = tb.x, lo = nd.lo[node], m = nd.hi[node] - lo, k = nd.kcnt[node];
    const int lane = threadIdx.x & 31, s = tb.y + (threadIdx.x >> 5);
    if (s >= m) return;
    const int info = ps.rowinfo[lo + s];
    const double di = info >= 0 ? ps.dK[lo + info] : 0.0, zi = info >= 0 ? ps.zh[lo + info] : 0.0;
    double *row = Us + (size_t) (lo + ps.perm[lo + s]) * n + lo;   // row of the child-order basis
    for (int c = lane; c < m; c += 32) {
        const int src = ps.colsrc[lo + c];
        double v;
        if (src >= 0 && src < k) v = info >= 0 ? zi / ((di - ps.lamb[lo + src]) - ps.tau[lo + src]) / ps.nrm[lo + src] : 0.0;
        else v = (info < 0 && -(info + 1) == src - k) ? 1.0 : 0.0;
        row[c] = v;
    }
}

// Givens rotations of the deflation (on sorted positions, i.e. rows perm[.]
// of U), applied in reverse order; a thread per column.
__global__ void __launch_bounds__(DC_CHUNK) k_dc_rotate(DcNodes nd, DcPos ps, const int2 *tab, double *Us, int n)
{
    const int2 tb = tab[blockIdx.x];
    const int node = tb.x, lo = nd.lo[node], m = nd.hi[node] - lo, nr = nd.rcnt[node];
    const int c = tb.y + threadIdx.x;
    if (nr == 0 || c >= m) return;
    double *U = Us + (size_t) lo * n + lo + c;
    const int *perm = ps.perm + lo;
    for (int r = nr - 1; r >= 0; r--) {
        const int2 pr = ps.rot[lo + r];
        const double2 cs = ps.rotcs[lo + r];
        const size_t ix = (size_t) perm[pr.x] * n, iy = (size_t) perm[pr.y] * n;
        const double x = U[ix], y = U[iy];
        U[ix] = cs.x * x - cs.y * y;
        U[iy] = cs.y * x + cs.x * y;
    }
}

__global__ void k_dc_commit_lam(DcNodes nd, DcPos ps, const int2 *tab)
{
    const int2 tb = tab[blockIdx.x];
    const int node = tb.x, lo = nd.lo[node], m = nd.hi[node] - lo;
    const int a = tb.y + threadIdx.x;
    if (a < m) ps.lam[lo + a] = ps.lamnew[lo + a];
}

// New vectors of a node: [Q1 0; 0 Q2] U, one half at a time (rows of child
// 1 with child 1's block, rows of child 2 with child 2's), read from Qin and
// written to Qout; 64 x 64 tiles on the FP64 tensor cores. Tile entry:
// (node, half, tile row, tile column).
__global__ void __launch_bounds__(128) k_dc_gemm(DcNodes nd, const int4 *tiles, const double *Qin, const double *Us,
                                                 double *Qout, int n)
{
    const int4 t = tiles[blockIdx.x];
    const int node = t.x >> 1, half = t.x & 1;
    const int lo = nd.lo[node], mid = nd.mid[node], hi = nd.hi[node], m = hi - lo;
    const int r0 = half ? mid : lo, mh = half ? hi - mid : mid - lo;
    const double *Ab = Qin + (size_t) r0 * n + r0;
    const double *Bb = Us + (size_t) r0 * n + lo;
    double *Cb = Qout + (size_t) r0 * n + lo;
    dgemm_tile_dmma64<false, false>(mh, m, mh, 1.0, Ab, n, Bb, n, 0.0, Cb, n, t.y * 64, t.z * 64);
}

// A merge of at most DC_SMALL positions in one CTA: the nine steps above in
// shared memory, one launch per tree level instead of nine (the levels below 64
// were 54 of an eigensolve's launches, each a few us for almost no work). Every
// value is formed as in the separate kernels: the same bits.
constexpr int DC_SMALL = 64;
constexpr size_t DC_SMALL_SMEM = sizeof(double) * DC_SMALL * (DC_SMALL + 1 + DC_SMALL / 2 + 1);
__global__ void __launch_bounds__(256) k_dc_merge_small(DcNodes nd, double *lam, const double *e, const double *Qin,
                                                        double *Qout, int n, int node0, bool at_noise)
{
    constexpr int MS = DC_SMALL;
    __shared__ double sd[MS], sz[MS], dK[MS], zK[MS], lamb[MS], tau[MS], zh[MS], nrm[MS], sv[MS], s_red[33];
    __shared__ int sp[MS], keep[MS], defl[MS], rowinfo[MS], colsrc[MS];
    __shared__ int2 rot[MS];
    __shared__ double2 rotcs[MS];
    __shared__ int s_k, s_nr;
    extern __shared__ double dsm[];
    double (*U)[MS + 1] = (double (*)[MS + 1]) dsm;
    double (*Q)[MS / 2 + 1] = (double (*)[MS / 2 + 1]) (dsm + MS * (MS + 1));   // both halves' vectors, row by row
    const int node = node0 + blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int lo = nd.lo[node], mid = nd.mid[node], hi = nd.hi[node];
    const int m = hi - lo, m1 = mid - lo, m2 = hi - mid;
    const double rho_raw = e[mid - 1];
    const double rho = 2.0 * fabs(rho_raw), sg = rho_raw >= 0.0 ? 1.0 : -1.0;
    const double *L1 = lam + lo, *L2 = lam + mid;
    const double rs2 = 1.0 / sqrt(2.0);
    for (int l = tid; l < m * (MS / 2); l += 256) {
        const int i = l / (MS / 2), c = l % (MS / 2), r0 = i < m1 ? lo : mid, mh = i < m1 ? m1 : m2;
        if (c < mh) Q[i][c] = Qin[(size_t) (lo + i) * n + r0 + c];
    }
    for (int idx = tid; idx < m; idx += 256) {
        sd[idx] = 0.0;
        sz[idx] = 0.0;
        sp[idx] = idx;
        colsrc[idx] = 0;
    }
    __syncthreads();
    // sorting of the halves, z, tolerance
    double dmax = 0.0, zmax = 0.0;
    for (int idx = tid; idx < m; idx += 256) {
        double x, zz;
        int pos;
        if (idx < m1) {
            x = L1[idx];
            zz = Q[m1 - 1][idx];
            int a = 0, b = m2;   // first L2 >= x
            while (a < b) {
                const int c = (a + b) >> 1;
                if (L2[c] < x) a = c + 1; else b = c;
            }
            pos = idx + a;
        } else {
            const int i2 = idx - m1;
            x = L2[i2];
            zz = sg * Q[m1][i2];
            int a = 0, b = m1;   // first L1 > x
            while (a < b) {
                const int c = (a + b) >> 1;
                if (L1[c] <= x) a = c + 1; else b = c;
            }
            pos = i2 + a;
        }
        pos = min(max(pos, 0), m - 1);
        zz *= rs2;
        sd[pos] = x;
        sz[pos] = zz;
        sp[pos] = idx;
        dmax = fmax(dmax, fabs(x));
        zmax = fmax(zmax, fabs(zz));
    }
    dmax = block_max_all<256>(dmax, s_red);
    zmax = block_max_all<256>(zmax, s_red);
    const double tol = 8.0 * DBL_EPSILON * fmax(dmax, zmax);
    if (tid == 0) {
        int k, nr;
        deflation_scan(sd, sz, m, rho, zmax, tol, keep, defl, rowinfo, rot, rotcs, k, nr);
        s_k = k;
        s_nr = nr;
    }
    __syncthreads();
    const int k = s_k, nr = s_nr;
    for (int i = tid; i < k; i += 256) {
        dK[i] = sd[keep[i]];
        zK[i] = sz[keep[i]];
    }
    __syncthreads();
    for (int j = wid; j < k; j += 8) {   // roots
        int org;
        double t;
        secular_root(dK, zK, k, j, rho, lane, at_noise, org, t);
        if (lane == 0) {
            lamb[j] = dK[org];
            tau[j] = t;
        }
    }
    __syncthreads();
    for (int i = wid; i < k; i += 8) {   // z from the roots
        const double di = dK[i];
        double pr = 1.0;
        for (int j = lane; j < k; j += 32) {
            const double del = (di - lamb[j]) - tau[j];
            pr *= (j == i) ? del : del / (di - dK[j]);
        }
        pr = warp_prod_bcast(pr);
        if (lane == 0) zh[i] = copysign(sqrt(fmax(-pr, 0.0)), zK[i]);
    }
    __syncthreads();
    for (int j = wid; j < k; j += 8) {   // norms
        const double lb = lamb[j], tj = tau[j];
        double q = 0.0;
        for (int i = lane; i < k; i += 32) {
            const double u = zh[i] / ((dK[i] - lb) - tj);
            q += u * u;
        }
        q = warp_sum_bcast(q);
        if (lane == 0) nrm[j] = sqrt(q);
    }
    for (int a = tid; a < m; a += 256) sv[a] = (a < k) ? lamb[a] + tau[a] : sd[defl[a - k]];
    __syncthreads();
    if (tid < m) {   // output order
        const double x = sv[tid];
        int q = 0;
        for (int b = 0; b < m; b++) {
            const double y = sv[b];
            q += (y < x || (y == x && b < tid)) ? 1 : 0;
        }
        q = min(q, m - 1);
        lam[lo + q] = x;   // every read of the halves' values lies behind a barrier
        colsrc[q] = tid;
    }
    __syncthreads();
    for (int l = tid; l < m * m; l += 256) {   // the merge's vectors, in the children's order
        const int sidx = l / m, c = l - sidx * m;
        const int info = rowinfo[sidx], src = colsrc[c];
        double v;
        if (src < k) v = info >= 0 ? zh[info] / ((dK[info] - lamb[src]) - tau[src]) / nrm[src] : 0.0;
        else v = (info < 0 && -(info + 1) == src - k) ? 1.0 : 0.0;
        U[sp[sidx]][c] = v;
    }
    __syncthreads();
    if (tid < m)
        for (int q = nr - 1; q >= 0; q--) {
            const int ix = sp[rot[q].x], iy = sp[rot[q].y];
            const double2 cs = rotcs[q];
            const double x = U[ix][tid], y = U[iy][tid];
            U[ix][tid] = cs.x * x - cs.y * y;
            U[iy][tid] = cs.y * x + cs.x * y;
        }
    __syncthreads();
    for (int l = tid; l < m * m; l += 256) {   // [Q1 0; 0 Q2] U: one chain of multiply-adds per output, as DMMA
        const int i = l / m, c = l - i * m, b0 = i < m1 ? 0 : m1, mh = i < m1 ? m1 : m2;
        double acc = 0.0;
        for (int q = 0; q < mh; q++) acc = fma(Q[i][q], U[b0 + q][c], acc);
        Qout[(size_t) (lo + i) * n + lo + c] = acc;
    }
}

__global__ void k_transpose(const double *in, double *out, int n)
{
    __shared__ double tile[32][33];
    const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += 8) {
        const int i = by + r, j = bx + threadIdx.x;
        if (i < n && j < n) tile[r][threadIdx.x] = in[(size_t) i * n + j];
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += 8) {
        const int i = bx + r, j = by + threadIdx.x;
        if (i < n && j < n) out[(size_t) i * n + j] = tile[threadIdx.x][r];
    }
}

__global__ void k_copy_scalar_eig(const double *A, double *w, double *V)
{
    w[0] = A[0];
    V[0] = 1.0;
}

// ------------------------------------------------------------------ small Cholesky-QR helpers
// Lower Cholesky factor of a symmetric positive definite o x o matrix, in place
// (row-major, lower triangle), left-looking, one warp per row; a non-positive
// or non-finite pivot sets *fail.
__global__ void __launch_bounds__(1024) k_potrf_lower(double *G, int o, int *fail)
{
    __shared__ double s_piv;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int j = 0; j < o; j++) {
        if (wid == 0) {
            double s = 0.0;
            for (int c = lane; c < j; c += 32) s += G[(size_t) j * o + c] * G[(size_t) j * o + c];
            s = warp_sum_bcast(s);
            if (lane == 0) {
                const double ajj = G[(size_t) j * o + j] - s;
                if (!(ajj > 0.0) || !isfinite(ajj)) *fail = 1;
                const double l = (ajj > 0.0 && isfinite(ajj)) ? sqrt(ajj) : 1.0;
                G[(size_t) j * o + j] = l;
                s_piv = l;
            }
        }
        __syncthreads();
        const double rinv = 1.0 / s_piv;
        for (int r = j + 1 + wid; r < o; r += nw) {
            double s = 0.0;
            for (int c = lane; c < j; c += 32) s += G[(size_t) r * o + c] * G[(size_t) j * o + c];
            s = warp_sum_bcast(s);
            if (lane == 0) G[(size_t) r * o + j] = (G[(size_t) r * o + j] - s) * rinv;
        }
        __syncthreads();
    }
}

// Xc = (L^-1)^T stored row-major (column j of L^-1 in row j of Xc), upper part
// of L^-1 zero; one thread per column of the inverse.
__global__ void k_trtri_lower(const double *L, double *Xc, int o)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= o) return;
    double *x = Xc + (size_t) j * o;
    for (int i = 0; i < j; i++) x[i] = 0.0;
    x[j] = 1.0 / L[(size_t) j * o + j];
    for (int i = j + 1; i < o; i++) {
        double s = 0.0;
        for (int kk = j; kk < i; kk++) s += L[(size_t) i * o + kk] * x[kk];
        x[i] = -s / L[(size_t) i * o + i];
    }
}

// The two of them for o up to CQ_MAX with the factor in shared memory (row
// pitch odd, so a column is read without bank conflicts); every sum keeps its
// order. k_potrf_small: the kernel above on a resident G. k_trtri_small: a warp
// per column of the inverse, which adds L(i, k) x(k) to every later i as soon as
// x(k) is known, instead of a thread per column with a chain of o^2 / 2
// multiply-adds. o = 161: 473 and 420 us, now 373 and 74 us.
constexpr int CQ_MAX = 168, CQ_THREADS = 1024;
__host__ __device__ constexpr int cq_pitch(int o) { return o | 1; }
size_t cq_smem(int o) { return sizeof(double) * (size_t) o * cq_pitch(o); }

__global__ void __launch_bounds__(CQ_THREADS) k_potrf_small(double *G, int o, int *fail)
{
    extern __shared__ double cq[];
    __shared__ double s_piv;
    const int ld = cq_pitch(o), lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    constexpr int NW = CQ_THREADS / 32;
    for (int l = threadIdx.x; l < o * o; l += CQ_THREADS) cq[l / o * ld + l % o] = G[l];
    __syncthreads();
    for (int j = 0; j < o; j++) {
        if (wid == 0) {
            double s = 0.0;
            for (int c = lane; c < j; c += 32) s += cq[j * ld + c] * cq[j * ld + c];
            s = warp_sum_bcast(s);
            if (lane == 0) {
                const double ajj = cq[j * ld + j] - s;
                if (!(ajj > 0.0) || !isfinite(ajj)) *fail = 1;
                const double l = (ajj > 0.0 && isfinite(ajj)) ? sqrt(ajj) : 1.0;
                cq[j * ld + j] = l;
                s_piv = l;
            }
        }
        __syncthreads();
        const double rinv = 1.0 / s_piv;
        for (int r = j + 1 + wid; r < o; r += NW) {
            double s = 0.0;
            for (int c = lane; c < j; c += 32) s += cq[r * ld + c] * cq[j * ld + c];
            s = warp_sum_bcast(s);
            if (lane == 0) cq[r * ld + j] = (cq[r * ld + j] - s) * rinv;
        }
        __syncthreads();
    }
    for (int l = threadIdx.x; l < o * o; l += CQ_THREADS) G[l] = cq[l / o * ld + l % o];
}

__global__ void __launch_bounds__(CQ_THREADS) k_trtri_small(const double *L, double *Xc, int o)
{
    extern __shared__ double cq[];
    constexpr int NQ = (CQ_MAX + 31) / 32;
    const int ld = cq_pitch(o), lane = threadIdx.x & 31, j = blockIdx.x * (CQ_THREADS / 32) + (threadIdx.x >> 5);
    for (int l = threadIdx.x; l < o * o; l += CQ_THREADS) cq[l / o * ld + l % o] = L[l];
    __syncthreads();
    if (j >= o) return;
    double acc[NQ], x[NQ];   // of rows lane + 32 q
#pragma unroll
    for (int q = 0; q < NQ; q++) acc[q] = x[q] = 0.0;
#pragma unroll
    for (int kq = 0; kq < NQ; kq++)
        for (int kl = 0; kl < 32; kl++) {
            const int k = 32 * kq + kl;
            if (k < j) continue;
            if (k >= o) break;
            const double mine = (k == j ? 1.0 : -acc[kq]) / cq[k * ld + k];
            if (lane == kl) x[kq] = mine;
            const double xk = __shfl_sync(0xffffffffu, mine, kl);
#pragma unroll
            for (int q = kq; q < NQ; q++) {
                const int i = lane + 32 * q;
                if (i > k && i < o) acc[q] = fma(cq[i * ld + k], xk, acc[q]);
            }
        }
#pragma unroll
    for (int q = 0; q < NQ; q++)
        if (lane + 32 * q < o) Xc[(size_t) j * o + lane + 32 * q] = x[q];
}

__global__ void k_hash_fill(double *A, size_t n)
{
    size_t i = (size_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    unsigned long long h = (i + 1) * 0x9E3779B97F4A7C15ULL;
    h ^= h >> 31;
    h *= 0xBF58476D1CE4E5B9ULL;
    h ^= h >> 29;
    A[i] = (double) (h >> 11) * (1.0 / 9007199254740992.0) - 0.5;
}

}  // namespace

// ------------------------------------------------------------------ host side
struct Eig {
    int n = 0, G = 1, npanels = 0, nblk = 0;
    bool cluster = false;   // panels in one thread-block cluster (k_sytrd_cluster)
    // tridiagonalisation and back-transformation
    double *A = nullptr, *VT = nullptr, *PVW = nullptr, *PWV = nullptr, *d = nullptr, *e = nullptr, *tau = nullptr,
           *col = nullptr, *y = nullptr, *part = nullptr, *Gb = nullptr, *Tf = nullptr, *Y = nullptr, *Y2 = nullptr;
    unsigned long long *bar = nullptr;
    // divide and conquer: eigenvector buffers of alternate tree levels (Qa reuses A) and the merge's U
    double *Qb = nullptr, *Us = nullptr;
    DcNodes nodes{};
    DcPos pos{};
    int *node_mem = nullptr;
    double *node_rho = nullptr;
    int2 *tab_c = nullptr, *tab_w = nullptr;
    int4 *tiles = nullptr;
    struct Level {
        int depth, node0, nnodes, maxm, c0, nc, w0, nw, t0, nt;
    };
    std::vector<Level> levels;
    // Cholesky-QR of dominant_subspace
    double *Gx = nullptr;
    int go = 0;
    int *acc = nullptr;
    std::vector<void *> allocs;
};

namespace {

template <typename T>
bool ealloc(Eig *e, T **p, size_t count)
{
    void *q = nullptr;
    if (dev_malloc(&q, sizeof(T) * (count ? count : 1), 0) != OK) return false;
    e->allocs.push_back(q);
    *p = (T *) q;
    return true;
}

bool dc_plan(Eig *E)
{
    const int n = E->n;
    struct Node {
        int dep, lo, mid, hi;
    };
    std::vector<Node> nodes;
    std::vector<Node> stack{{0, 0, 0, n}};
    while (!stack.empty()) {
        Node x = stack.back();
        stack.pop_back();
        if (x.hi - x.lo <= 1) continue;
        x.mid = x.lo + (x.hi - x.lo) / 2;
        nodes.push_back(x);
        stack.push_back({x.dep + 1, x.lo, 0, x.mid});
        stack.push_back({x.dep + 1, x.mid, 0, x.hi});
    }
    std::stable_sort(nodes.begin(), nodes.end(), [](const Node &a, const Node &b) { return a.dep > b.dep; });
    std::vector<int> lo, mid, hi;
    std::vector<int2> tc, tw;
    std::vector<int4> tt;
    E->levels.clear();
    size_t i = 0;
    while (i < nodes.size()) {
        Eig::Level L{};
        L.node0 = (int) i;
        L.c0 = (int) tc.size();
        L.w0 = (int) tw.size();
        L.t0 = (int) tt.size();
        const int dep = nodes[i].dep;
        L.depth = dep;
        for (; i < nodes.size() && nodes[i].dep == dep; i++) {
            const int id = (int) i, m = nodes[i].hi - nodes[i].lo;
            lo.push_back(nodes[i].lo);
            mid.push_back(nodes[i].mid);
            hi.push_back(nodes[i].hi);
            L.maxm = std::max(L.maxm, m);
            for (int f = 0; f < m; f += DC_CHUNK) tc.push_back(make_int2(id, f));
            for (int f = 0; f < m; f += DC_WCHUNK) tw.push_back(make_int2(id, f));
            const int ntc = (m + 63) / 64;
            for (int h = 0; h < 2; h++) {
                const int mh = h ? nodes[i].hi - nodes[i].mid : nodes[i].mid - nodes[i].lo;
                for (int a = 0; a < (mh + 63) / 64; a++)
                    for (int b = 0; b < ntc; b++) tt.push_back(make_int4(2 * id + h, a, b, 0));
            }
        }
        L.nnodes = (int) i - L.node0;
        L.nc = (int) tc.size() - L.c0;
        L.nw = (int) tw.size() - L.w0;
        L.nt = (int) tt.size() - L.t0;
        E->levels.push_back(L);
    }
    const size_t nn = nodes.size();
    if (!ealloc(E, &E->node_mem, 5 * nn) || !ealloc(E, &E->node_rho, nn)) return false;
    std::vector<int> packed(5 * nn, 0);
    std::copy(lo.begin(), lo.end(), packed.begin());
    std::copy(mid.begin(), mid.end(), packed.begin() + nn);
    std::copy(hi.begin(), hi.end(), packed.begin() + 2 * nn);
    if (nn && cudaMemcpy(E->node_mem, packed.data(), sizeof(int) * 5 * nn, cudaMemcpyHostToDevice) != cudaSuccess)
        return false;
    E->nodes.lo = E->node_mem;
    E->nodes.mid = E->node_mem + nn;
    E->nodes.hi = E->node_mem + 2 * nn;
    E->nodes.kcnt = E->node_mem + 3 * nn;
    E->nodes.rcnt = E->node_mem + 4 * nn;
    E->nodes.rho = E->node_rho;
    if (!ealloc(E, &E->tab_c, tc.size()) || !ealloc(E, &E->tab_w, tw.size()) || !ealloc(E, &E->tiles, tt.size()))
        return false;
    if (!tc.empty() && cudaMemcpy(E->tab_c, tc.data(), sizeof(int2) * tc.size(), cudaMemcpyHostToDevice) != cudaSuccess)
        return false;
    if (!tw.empty() && cudaMemcpy(E->tab_w, tw.data(), sizeof(int2) * tw.size(), cudaMemcpyHostToDevice) != cudaSuccess)
        return false;
    if (!tt.empty() && cudaMemcpy(E->tiles, tt.data(), sizeof(int4) * tt.size(), cudaMemcpyHostToDevice) != cudaSuccess)
        return false;
    return true;
}

// Opt in to the dynamic shared memory the kernels ask for: the device's
// per-block opt-in maximum less each kernel's static shared memory.
template <typename K>
bool optin_one(K kern, int optin)
{
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, kern) != cudaSuccess) return false;
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                optin - (int) fa.sharedSizeBytes) == cudaSuccess;
}

bool smem_optin()
{
    static int done_dev = -1;
    int dev = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    if (done_dev == dev) return true;
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return false;
    if (!optin_one(k_sytrd_panel, optin) || !optin_one(k_wy_tfactor, optin) || !optin_one(k_dc_deflate, optin) ||
        !optin_one(k_dc_merge_small, optin) || !optin_one(k_potrf_small, optin) || !optin_one(k_trtri_small, optin) || !optin_one(k_dc_secular, optin) ||
        !optin_one(k_dc_zhat, optin) || !optin_one(k_dc_norms, optin) || !optin_one(k_dc_order, optin))
        return false;
    done_dev = dev;
    return true;
}

}  // namespace

Eig *eig_create(int n, cudaStream_t s)
{
    (void) s;
    if (n < 1 || n > EIG_MAX_N) return nullptr;
    if (!smem_optin()) {
        fprintf(stderr, "[tinyscf] eigensolver: shared-memory opt-in failed: %s\n",
                cudaGetErrorString(cudaGetLastError()));
        return nullptr;
    }
    Eig *E = new Eig();
    E->n = n;
    int dev = 0, nsm = 1, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const size_t dyn = sizeof(double) * (size_t) n;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_sytrd_panel, TRD_THREADS, dyn);
    E->G = std::max(1, std::min({nsm * std::max(per, 1), nsm, (n + 7) / 8}));
    if ((long long) E->G * TRD_THREADS / 8 < n) {   // the panel kernel gives every row its own 8 lanes
        fprintf(stderr, "[tinyscf] eigensolver: %d CTAs cannot hold %d rows\n", E->G, n);
        delete E;
        return nullptr;
    }
    E->cluster = trc_usable(n);
    E->npanels = (n + TRD_NB - 1) / TRD_NB;
    E->nblk = (n - 1 + BT_NB - 1) / BT_NB;   // blocks of the n - 1 reflectors
    const size_t nn = (size_t) n * n;
    bool ok = ealloc(E, &E->A, nn) && ealloc(E, &E->VT, nn) && ealloc(E, &E->Qb, nn) && ealloc(E, &E->Us, nn) &&
              ealloc(E, &E->PVW, (size_t) 2 * TRD_NB * n) && ealloc(E, &E->PWV, (size_t) 2 * TRD_NB * n) &&
              ealloc(E, &E->Y, (size_t) n * BT_NB) && ealloc(E, &E->Y2, (size_t) n * BT_NB) && ealloc(E, &E->d, n) &&
              ealloc(E, &E->e, n) && ealloc(E, &E->tau, n) && ealloc(E, &E->col, n) &&
              ealloc(E, &E->y, (size_t) ((n + TRD_SEG - 1) / TRD_SEG) * n) &&
              ealloc(E, &E->part, (size_t) E->G * (2 + 2 * TRD_NB)) &&
              ealloc(E, &E->Gb, (size_t) std::max(E->nblk, 1) * GR_KS * BT_NB * BT_NB) &&
              ealloc(E, &E->Tf, (size_t) std::max(E->nblk, 1) * BT_NB * BT_NB) && ealloc(E, &E->bar, 2) &&
              ealloc(E, &E->acc, 1) && wait_word() != nullptr;
    DcPos &P = E->pos;
    ok = ok && ealloc(E, &P.lam, n) && ealloc(E, &P.ds, n) && ealloc(E, &P.dK, n) && ealloc(E, &P.zK, n) &&
         ealloc(E, &P.lamb, n) && ealloc(E, &P.tau, n) && ealloc(E, &P.zh, n) && ealloc(E, &P.nrm, n) &&
         ealloc(E, &P.lamnew, n) && ealloc(E, &P.perm, n) && ealloc(E, &P.keep, n) && ealloc(E, &P.defl, n) &&
         ealloc(E, &P.rowinfo, n) && ealloc(E, &P.colsrc, n) && ealloc(E, &P.rot, n) && ealloc(E, &P.rotcs, n);
    ok = ok && dc_plan(E);
    if (!ok) {
        fprintf(stderr, "[tinyscf] eigensolver workspace for n = %d: %s\n", n, cudaGetErrorString(cudaGetLastError()));
        eig_destroy(E);
        return nullptr;
    }
    cudaMemset(P.colsrc, 0, sizeof(int) * n);
    cudaMemset(P.perm, 0, sizeof(int) * n);
    cudaMemset(E->bar, 0, sizeof(unsigned long long));
    const cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) {
        fprintf(stderr, "[tinyscf] eigensolver set-up for n = %d: %s\n", n, cudaGetErrorString(err));
        eig_destroy(E);
        return nullptr;
    }
    return E;
}

void eig_destroy(Eig *e)
{
    if (!e) return;
    for (void *p : e->allocs) dev_free(p, 0);
    cudaStreamSynchronize(0);
    delete e;
}

bool eig_small_launches(const Eig *e) { return e->cluster && trc_in_smem(e->n, e->n); }

namespace {

int tridiagonalize(Eig *E, const double *d_A, cudaStream_t s)
{
    const int n = E->n;
    const size_t nn = (size_t) n * n;
    TSCF_CUDA_CHECK(cudaMemcpyAsync(E->A, d_A, sizeof(double) * nn, cudaMemcpyDeviceToDevice, s));
    TSCF_CUDA_CHECK(cudaMemsetAsync(E->VT, 0, sizeof(double) * nn, s));
    TSCF_CUDA_CHECK(cudaMemsetAsync(E->tau, 0, sizeof(double) * n, s));
    TSCF_CUDA_CHECK(cudaMemsetAsync(E->e, 0, sizeof(double) * n, s));
    TSCF_CUDA_CHECK(cudaMemsetAsync(E->bar, 0, sizeof(unsigned long long), s));
    const size_t dyn = sizeof(double) * (size_t) n;
    for (int P = 0; P < E->npanels; P++) {
        TrdArgs a;
        a.A = E->A;
        a.VT = E->VT;
        a.PVW = E->PVW;
        a.PWV = E->PWV;
        a.d = E->d;
        a.e = E->e;
        a.tau = E->tau;
        a.col = E->col;
        a.y = E->y;
        a.part = E->part;
        a.bar = E->bar;
        a.err = wait_word();
        a.n = n;
        a.p = P * TRD_NB;
        a.cols = std::min(TRD_NB, n - a.p);
        a.G = E->G;
        void *args[] = {&a};
        g_launches++;
        g_eig_launches++;
        const int m = n - a.p;
        if (E->cluster && trc_in_smem(n, m)) {
            cudaLaunchAttribute attr;
            const cudaLaunchConfig_t cfg = trc_config(n, m, s, &attr);
            a.G = (int) cfg.gridDim.x;
            TSCF_CUDA_CHECK(cudaLaunchKernelExC(&cfg, trc_kernel(n), args));
        } else {
            TSCF_CUDA_CHECK(cudaLaunchCooperativeKernel((const void *) k_sytrd_panel, dim3(E->G), dim3(TRD_THREADS),
                                                        args, dyn, s));
        }
        const int q = a.p + a.cols, mt = n - q;
        if (mt > 0) {
            // A22 -= V W^T + W V^T = PVW^T PWV over the trailing columns (a full panel: cols = TRD_NB)
            dgemm_untuned(true, false, mt, mt, 2 * TRD_NB, -1.0, E->PVW + q, n, E->PWV + q, n, 1.0,
                          E->A + (size_t) q * n + q, n, s);
            g_eig_launches++;
        }
    }
    return cuda_launch_rc("tridiagonalisation");
}

// Eigenvectors of T into the columns of the returned buffer (E->A or E->Qb).
int divide_conquer(Eig *E, cudaStream_t s, double **out, bool at_noise)
{
    const int n = E->n;
    const size_t nn = (size_t) n * n;
    double *buf[2] = {E->A, E->Qb};   // level of depth L writes buf[L % 2], reads its children from the other
    TSCF_CUDA_CHECK(cudaMemsetAsync(buf[0], 0, sizeof(double) * nn, s));
    TSCF_CUDA_CHECK(cudaMemsetAsync(buf[1], 0, sizeof(double) * nn, s));
    TSCF_CUDA_CHECK(cudaMemsetAsync(E->Us, 0, sizeof(double) * nn, s));
    g_launches++;
    g_eig_launches++;
    k_dc_init<<<(n + 255) / 256, 256, 0, s>>>(E->d, E->e, E->pos.lam, buf[0], buf[1], n);
    for (const auto &L : E->levels) {
        const size_t m = (size_t) L.maxm;
        const double *Qin = buf[(L.depth + 1) % 2];
        double *Qout = buf[L.depth % 2];
        if (L.maxm <= DC_SMALL) {
            k_dc_merge_small<<<L.nnodes, 256, DC_SMALL_SMEM, s>>>(E->nodes, E->pos.lam, E->e, Qin, Qout, n, L.node0, at_noise);
            g_launches++;
            g_eig_launches++;
            continue;
        }
        k_dc_deflate<<<L.nnodes, 512, 20 * m, s>>>(E->nodes, E->pos, Qin, E->e, n, L.node0);
        k_dc_secular<<<L.nw, 256, 16 * m, s>>>(E->nodes, E->pos, E->tab_w + L.w0, at_noise);
        k_dc_zhat<<<L.nw, 256, 24 * m, s>>>(E->nodes, E->pos, E->tab_w + L.w0);
        k_dc_norms<<<L.nw, 256, 16 * m, s>>>(E->nodes, E->pos, E->tab_w + L.w0);
        k_dc_order<<<L.nc, DC_CHUNK, 8 * m, s>>>(E->nodes, E->pos, E->tab_c + L.c0);
        k_dc_build<<<L.nw, 256, 0, s>>>(E->nodes, E->pos, E->tab_w + L.w0, E->Us, n);
        k_dc_rotate<<<L.nc, DC_CHUNK, 0, s>>>(E->nodes, E->pos, E->tab_c + L.c0, E->Us, n);
        k_dc_commit_lam<<<L.nc, DC_CHUNK, 0, s>>>(E->nodes, E->pos, E->tab_c + L.c0);
        k_dc_gemm<<<L.nt, 128, 0, s>>>(E->nodes, E->tiles + L.t0, Qin, E->Us, Qout, n);
        g_launches += 9;
        g_eig_launches += 9;
    }
    *out = buf[0];   // the root has depth 0
    return cuda_launch_rc("divide and conquer");
}

// Vout = Z^T Q^T, Z (the tridiagonal's eigenvectors, columns of Zc), Q the
// product of the reflectors, in blocks of BT_NB reflectors from the last:
// Vout <- Vout - (Vout V) T^T V^T.
int back_transform(Eig *E, const double *Zc, double *d_V, cudaStream_t s)
{
    const int n = E->n, nref = n - 1;
    g_launches += 3;
    g_eig_launches += 3;
    k_wy_gram<<<dim3(E->nblk, (BT_NB / 32) * (BT_NB / 32), GR_KS), 256, 0, s>>>(E->VT, E->Gb, n, nref);
    k_wy_tfactor<<<E->nblk, TF_THREADS, sizeof(double) * BT_NB * BT_NB, s>>>(E->Gb, E->tau, E->Tf, nref);
    k_transpose<<<dim3((n + 31) / 32, (n + 31) / 32), dim3(32, 8), 0, s>>>(Zc, d_V, n);
    for (int B = E->nblk - 1; B >= 0; B--) {
        const int p0 = B * BT_NB, bb = std::min(BT_NB, nref - p0), mv = n - p0 - 1;
        const double *V = E->VT + (size_t) p0 * n + p0 + 1;
        dgemm_untuned(false, true, n, bb, mv, 1.0, d_V + p0 + 1, n, V, n, 0.0, E->Y, BT_NB, s);
        dgemm_untuned(false, true, n, bb, bb, 1.0, E->Y, BT_NB, E->Tf + (size_t) B * BT_NB * BT_NB, BT_NB, 0.0, E->Y2,
                      BT_NB, s);
        dgemm_untuned(false, false, n, mv, bb, -1.0, E->Y2, BT_NB, V, n, 1.0, d_V + p0 + 1, n, s);
        g_eig_launches += 3;
    }
    return cuda_launch_rc("back-transformation");
}

}  // namespace

// Eigenvalues ascending into d_w, eigenvectors as rows of d_V (V[k*n + i] =
// entry i of eigenvector k). d_V may alias d_A.
int eig_run(Eig *E, const double *d_A, double *d_w, double *d_V, cudaStream_t s, bool at_noise)
{
    if (!E) return ERR_STATE;
    const int n = E->n;
    if (n == 1) {
        g_launches++;
        g_eig_launches++;
        k_copy_scalar_eig<<<1, 1, 0, s>>>(d_A, d_w, d_V);
        return cuda_launch_rc("eigensolve (n = 1)");
    }
    RC_(tridiagonalize(E, d_A, s));
    double *Z = nullptr;
    RC_(divide_conquer(E, s, &Z, at_noise));
    RC_(back_transform(E, Z, d_V, s));
    TSCF_CUDA_CHECK(cudaMemcpyAsync(d_w, E->pos.lam, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    return OK;
}

// ------------------------------------------------------------------ dominant subspace
// Rows of U (o x n) become an orthonormal basis of the dominant o-dimensional
// invariant subspace of a symmetric n x n matrix M, by subspace iteration from
// a fixed pseudo-random start: W <- W M, orthonormalised every kOrthoEvery
// products and at the end by Cholesky-QR (G = W W^T = L L^T, W <- L^-1 W,
// with L^-1 from a triangular inverse so the update is one GEMM), the last one
// applied twice for orthogonality to rounding. For a matrix close to a rank-o
// projector (a predicted density in the orthogonal basis) each product
// shrinks the other directions by the ratio of the (o+1)-th to the o-th
// eigenvalue, while the kept directions, with eigenvalues near 1, stay well
// conditioned between orthonormalisations.
namespace {
const int kOrthoEvery = 3;

// W <- L^-1 U for G = U U^T = L L^T (U, W: o x n row-major; G: o x o scratch).
// A failed factorisation sets E->acc on the device.
void chol_qr(Eig *E, const double *U, double *W, double *G, int n, int o, cudaStream_t s)
{
    dgemm(false, true, o, o, n, 1.0, U, n, U, n, 0.0, G, o, s);   // G = U U^T
    if (o <= CQ_MAX) {
        k_potrf_small<<<1, CQ_THREADS, cq_smem(o), s>>>(G, o, E->acc);
        k_trtri_small<<<(o + CQ_THREADS / 32 - 1) / (CQ_THREADS / 32), CQ_THREADS, cq_smem(o), s>>>(G, E->Gx, o);
    } else {
        k_potrf_lower<<<1, 1024, 0, s>>>(G, o, E->acc);
        k_trtri_lower<<<(o + 127) / 128, 128, 0, s>>>(G, E->Gx, o);
    }
    g_launches += 2;
    // row-major Gx is (L^-1)^T, so W = Gx^T U
    dgemm(true, false, o, n, o, 1.0, E->Gx, o, U, n, 0.0, W, n, s);
}
}  // namespace

int dominant_subspace(Eig *E, const double *d_M, double *d_U, double *d_W, double *d_G, int n, int o, int iters,
                      cudaStream_t s)
{
    if (!E || o <= 0 || o > n || iters < 1) return ERR_INPUT;
    if (E->go < o) {
        if (E->Gx) {
            dev_free(E->Gx, s);
            E->allocs.erase(std::find(E->allocs.begin(), E->allocs.end(), (void *) E->Gx));
            E->Gx = nullptr;
        }
        if (!ealloc(E, &E->Gx, (size_t) o * o)) return ERR_ALLOC;
        E->go = o;
    }
    TSCF_CUDA_CHECK(cudaMemsetAsync(E->acc, 0, sizeof(int), s));
    const size_t on = (size_t) o * n;
    double *cur = d_W, *nxt = d_U;   // cur: the basis (or an unorthonormalised product of it)
    k_hash_fill<<<(unsigned) ((on + 255) / 256), 256, 0, s>>>(cur, on);
    g_launches++;
    for (int it = 1; it <= iters; it++) {
        dgemm(false, false, o, n, n, 1.0, cur, n, d_M, n, 0.0, nxt, n, s);   // nxt = cur M (M symmetric)
        if (it % kOrthoEvery == 0 || it == iters) chol_qr(E, nxt, cur, d_G, n, o, s);
        else std::swap(cur, nxt);
    }
    chol_qr(E, cur, nxt, d_G, n, o, s);   // second pass: orthonormal to rounding
    if (nxt != d_U) TSCF_CUDA_CHECK(cudaMemcpyAsync(d_U, nxt, sizeof(double) * on, cudaMemcpyDeviceToDevice, s));
    int acc = 0;
    TSCF_CUDA_CHECK(cudaMemcpyAsync(&acc, E->acc, sizeof(int), cudaMemcpyDeviceToHost, s));
    TSCF_CUDA_CHECK(cudaStreamSynchronize(s));
    return acc == 0 ? OK : ERR_NUMERIC;
}

}  // namespace tscf
