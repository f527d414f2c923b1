// The integral recursions with every index a compile-time constant: Obara-Saika
// vertical recursion, electron transfer restricted to the classes that the
// result needs, and horizontal-recursion leaves. All arrays are indexed by
// constants, so the small classes live in registers and the large ones spill
// to fixed local addresses; the index arithmetic and the component table
// loads of a run-time recursion (most of its instructions) are gone.
#pragma once

#include <utility>

#include "tscf_internal.h"

namespace tscf {
namespace unrolled {

template <int V>
struct Int {
    static constexpr int value = V;
    __host__ __device__ constexpr operator int() const { return V; }
};

template <class F, int... I>
__device__ __forceinline__ void sfor_impl(F &&f, std::integer_sequence<int, I...>)
{
    (f(Int<I>{}), ...);
}
// f(Int<0>{}), ..., f(Int<N-1>{})
template <int N, class F>
__device__ __forceinline__ void sfor(F &&f)
{
    sfor_impl(static_cast<F &&>(f), std::make_integer_sequence<int, N>{});
}

// Component c of level l in lexicographic order (xx, xy, xz, yy, yz, zz).
struct Cart {
    int x, y, z;
    __host__ __device__ constexpr int at(int d) const { return d == 0 ? x : (d == 1 ? y : z); }
    __host__ __device__ constexpr int first() const { return x > 0 ? 0 : (y > 0 ? 1 : 2); }
};
__host__ __device__ constexpr Cart cart(int l, int c)
{
    int n = 0;
    while ((n + 1) * (n + 2) / 2 <= c) n++;
    const int z = c - n * (n + 1) / 2;
    return Cart{l - n, n - z, z};
}
__host__ __device__ constexpr int cpos(Cart q)
{
    const int n = q.y + q.z;
    return n * (n + 1) / 2 + q.z;
}
__host__ __device__ constexpr Cart step(Cart q, int d, int by)
{
    return Cart{q.x + (d == 0 ? by : 0), q.y + (d == 1 ? by : 0), q.z + (d == 2 ? by : 0)};
}
// level and component of cumulative index e
__host__ __device__ constexpr int lev_of(int e)
{
    int l = 0;
    while (ncum(l) <= e) l++;
    return l;
}
__host__ __device__ constexpr Cart cart_cum(int e)
{
    const int l = lev_of(e);
    return cart(l, e - ncum(l - 1));
}
__host__ __device__ constexpr int cum(Cart q) { return ncum(q.x + q.y + q.z - 1) + cpos(q); }

// F_m(T) * pref, m = 0..L; T in [0, BOYS_TMAX): 7-term Taylor expansion of F_L
// about the nearest grid point of the table, downward recursion; beyond:
// asymptotic form.
template <int L>
__device__ __forceinline__ void boys_scaled(const double *table, double T, double pref, double (&F)[L + 1])
{
    if (T >= BOYS_TMAX) {
        double f = 0.5 * pref * sqrt(M_PI / T);
        F[0] = f;
        const double i2t = 0.5 / T;
#pragma unroll
        for (int m = 1; m <= L; m++) {
            f *= (2 * m - 1) * i2t;
            F[m] = f;
        }
        return;
    }
    const int k = __double2int_rn(T * (1.0 / BOYS_DT));
    const double d = k * BOYS_DT - T;
    const double *row = table + k * 16 + L;
    double f = row[6];
    f = row[5] + f * d * (1.0 / 6.0);
    f = row[4] + f * d * (1.0 / 5.0);
    f = row[3] + f * d * (1.0 / 4.0);
    f = row[2] + f * d * (1.0 / 3.0);
    f = row[1] + f * d * (1.0 / 2.0);
    f = row[0] + f * d;
    f *= pref;
    F[L] = f;
    if constexpr (L > 0) {
        const double eT = pref * exp(-T), t2 = 2.0 * T;
#pragma unroll
        for (int m = L - 1; m >= 0; m--) {
            f = (t2 * f + eT) * (1.0 / (2 * m + 1));
            F[m] = f;
        }
    }
}

__host__ __device__ constexpr int vrr_width(int L)
{
    int best = 1;
    for (int l = 0; l <= L; l++) {
        const int v = ncart(l) * (L - l + 1);
        if (v > best) best = v;
    }
    return best;
}

// [e|0] for all |e| <= L into e0[ncum(L)] from the scaled Boys values F:
// [e+1_i]^(m) = PA_i [e]^(m) + WP_i [e]^(m+1) + e_i/(2z) ([e-1_i]^(m) - rz [e-1_i]^(m+1)).
template <int L>
__device__ __forceinline__ void vrr(const double (&F)[L + 1], const double (&PA)[3], const double (&WP)[3],
                                    double inv2z, double rz, double (&e0)[ncum(L)])
{
    constexpr int W = vrr_width(L);
    double lev[3][W];
#pragma unroll
    for (int m = 0; m <= L; m++) lev[0][m] = F[m];
    e0[0] = F[0];
    sfor<L>([&](auto li) {
        constexpr int l = decltype(li)::value + 1, M = L - l;
        sfor<ncart(l)>([&](auto ci) {
            constexpr int c = decltype(ci)::value;
            constexpr Cart q = cart(l, c);
            constexpr int i = q.first(), ai = q.at(i) - 1;
            constexpr Cart u = step(q, i, -1);
            constexpr int c1 = cpos(u) * (M + 2);
            if constexpr (ai > 0) {
                constexpr int c2 = cpos(step(u, i, -1)) * (M + 3);
                const double f = ai * inv2z;
#pragma unroll
                for (int m = 0; m <= M; m++)
                    lev[l % 3][c * (M + 1) + m] =
                        PA[i] * lev[(l + 2) % 3][c1 + m] + WP[i] * lev[(l + 2) % 3][c1 + m + 1] +
                        f * (lev[(l + 1) % 3][c2 + m] - rz * lev[(l + 1) % 3][c2 + m + 1]);
            } else {
#pragma unroll
                for (int m = 0; m <= M; m++)
                    lev[l % 3][c * (M + 1) + m] =
                        PA[i] * lev[(l + 2) % 3][c1 + m] + WP[i] * lev[(l + 2) % 3][c1 + m + 1];
            }
            e0[ncum(l - 1) + c] = lev[l % 3][c * (M + 1)];
        });
    });
}

// Electron transfer from [e|0] to [e|f], f = FLO..FHI, e = ELO..EHI (levels):
//   [e|f+1_i] = cAB_i [e|f] + e_i/(2eta)[e-1_i|f] + f_i/(2eta)[e|f-1_i] - (zeta/eta)[e+1_i|f];
// level k of f is formed only for the e that level FHI needs. Adds scale * [e|f] to
// acc[(e - ncum(ELO-1)) * NF + f - ncum(FLO-1)].
__host__ __device__ constexpr int etr_lo(int elo, int fhi, int k) { return elo - (fhi - k) > 0 ? elo - (fhi - k) : 0; }
__host__ __device__ constexpr int etr_first(int elo, int fhi, int k) { return ncum(etr_lo(elo, fhi, k) - 1); }
__host__ __device__ constexpr int etr_count(int elo, int ehi, int fhi, int k)
{
    return ncum(ehi + fhi - k) - etr_first(elo, fhi, k);
}
__host__ __device__ constexpr int etr_width(int elo, int ehi, int fhi)
{
    int best = 1;
    for (int k = 1; k <= fhi; k++) {
        const int v = etr_count(elo, ehi, fhi, k) * ncart(k);
        if (v > best) best = v;
    }
    return best;
}

template <int ELO, int EHI, int FLO, int FHI>
__device__ __forceinline__ void etr_add(const double (&e0)[ncum(EHI + FHI)], const double (&cAB)[3], double inv2eta,
                                        double zeta_eta, double scale,
                                        double (&acc)[(ncum(EHI) - ncum(ELO - 1)) * (ncum(FHI) - ncum(FLO - 1))])
{
    constexpr int NE = ncum(EHI) - ncum(ELO - 1), NF = ncum(FHI) - ncum(FLO - 1), E0 = ncum(ELO - 1);
    if constexpr (FLO == 0) {
#pragma unroll
        for (int e = 0; e < NE; e++) acc[e * NF] += scale * e0[E0 + e];
    }
    if constexpr (FHI > 0) {
        constexpr int W = etr_width(ELO, EHI, FHI);
        double buf[3][W];   // level k in buf[k % 3], k >= 1; level 0 is e0
        sfor<FHI>([&](auto ki) {
            constexpr int k = decltype(ki)::value + 1;   // the level being formed, from k - 1 and k - 2
            constexpr int first = etr_first(ELO, FHI, k), count = etr_count(ELO, EHI, FHI, k);
            constexpr int first1 = k == 1 ? 0 : etr_first(ELO, FHI, k - 1);
            constexpr int first2 = k <= 2 ? 0 : etr_first(ELO, FHI, k - 2);
            sfor<count>([&](auto ei) {
                constexpr int e = first + decltype(ei)::value;
                constexpr Cart qe = cart_cum(e);
                sfor<ncart(k)>([&](auto gi) {
                    constexpr int g = decltype(gi)::value;
                    constexpr Cart qg = cart(k, g);
                    constexpr int i = qg.first(), hi = qg.at(i) - 1, eid = qe.at(i);
                    constexpr Cart qh = step(qg, i, -1);
                    constexpr int ch = cpos(qh), n1 = ncart(k - 1), eup = cum(step(qe, i, 1));
                    auto lower = [&](int ee) { return k == 1 ? e0[ee] : buf[(k - 1) % 3][(ee - first1) * n1 + ch]; };
                    double v = cAB[i] * lower(e) - zeta_eta * lower(eup);
                    if constexpr (eid > 0) v += eid * inv2eta * lower(cum(step(qe, i, -1)));
                    if constexpr (hi > 0) {
                        constexpr int ch2 = cpos(step(qh, i, -1)), n2 = ncart(k - 2 > 0 ? k - 2 : 0);
                        v += hi * inv2eta * (k == 2 ? e0[e] : buf[(k + 1) % 3][(e - first2) * n2 + ch2]);
                    }
                    buf[k % 3][(e - first) * ncart(k) + g] = v;
                    if constexpr (k >= FLO && e >= E0 && e < E0 + NE)
                        acc[(e - E0) * NF + ncum(k - 1) - ncum(FLO - 1) + g] += scale * v;
                });
            });
        });
    }
}

// Horizontal recursion for lb <= 2: (a b| = sum_k w_k (e_k 0|, AB = A - B; f(k, e_k, w_k) per leaf.
template <int LA, int CA, int LB, int CB, class F>
__device__ __forceinline__ void for_leaves(const double (&AB)[3], F &&f)
{
    static_assert(LB <= 2, "leaves are written out for d shells");
    constexpr Cart a = cart(LA, CA), b = cart(LB, CB);
    if constexpr (LB == 0) {
        f(Int<cum(a)>{}, 1.0);
    } else if constexpr (LB == 1) {
        constexpr int i = b.first();
        f(Int<cum(step(a, i, 1))>{}, 1.0);
        f(Int<cum(a)>{}, AB[i]);
    } else {
        constexpr int i = b.first(), j = step(b, i, -1).first();
        f(Int<cum(step(step(a, i, 1), j, 1))>{}, 1.0);
        f(Int<cum(step(a, i, 1))>{}, AB[j]);
        f(Int<cum(step(a, j, 1))>{}, AB[i]);
        f(Int<cum(a)>{}, AB[i] * AB[j]);
    }
}

// A bra primitive pair: exponent sum, its inverse, centre, prefactor, and b (for the transfer coefficients).
struct PrimPair {
    double z, iz, x, y, zc, k, b;
};

}  // namespace unrolled
}  // namespace tscf
