// Integrals of the classes of total angular momentum L <= 3 by the
// Obara-Saika vertical recursion and the Head-Gordon-Pople horizontal one
// (S. Obara, A. Saika, J. Chem. Phys. 84, 3963 (1986); M. Head-Gordon,
// J. A. Pople, J. Chem. Phys. 89, 5777 (1988)).
//
// What bounds these classes with Rys quadrature is the look-up of the roots:
// 2 n series per primitive quartet, read from shared memory by lanes that
// each need another interval (about 10 wavefronts per 16-byte load, so 280
// cycles of the SM for n = 2 beside some 130 cycles of FP64 work).  Here one
// series gives F_L(x), e^-x the lower orders by the stable downward
// recursion, and the recursion itself takes fewer operations at this L.  The
// horizontal transfers are done once per contracted quartet.
#pragma once
#include "jk_common.cuh"

// F_m(x), m <= 3, from the power series of 10 terms on intervals of width 1/2
// (shared-memory copy; an interval is five 16-byte words, an odd number, so
// that different intervals start in different banks)
struct BoysS {
    static constexpr int WORDS = BOYS_NINT * BOYS_NC;  // doubles of one order
    static constexpr double XMAX = 0.5 * BOYS_NINT;
};
static_assert(BOYS_NC == 10, "rows of five 16-byte words");

template <int M>
__device__ __forceinline__ void boys_table_copy(const double* __restrict__ g, double* __restrict__ tab) {
    const double* src = g + BOYS_OFF + M * BoysS::WORDS;
    for (int e = threadIdx.x; e < BoysS::WORDS; e += blockDim.x) tab[e] = __ldg(src + e);
}

// F[m] = F_m(x) for m = 0 .. M
template <int M>
__device__ __forceinline__ void boys_all(const double* __restrict__ tab, double x, double* F) {
    if (x >= BoysS::XMAX) {
        // e^-x is below 1e-16 of every F_m kept: F_m = (2m - 1)!! sqrt(pi) / (2^(m+1) x^(m+1/2))
        const double rx = rsqrt(x), hx = 0.5 * rx * rx;
        F[0] = 0.88622692545275801365 * rx;
#pragma unroll
        for (int m = 1; m <= M; m++) F[m] = F[m - 1] * ((2 * m - 1) * hx);
        return;
    }
    const int i = (int)(2. * x);
    const double t = fma(4., x, -(double)(2 * i + 1));  // (x - centre) / (1/4)
    const double2* c = reinterpret_cast<const double2*>(tab + i * BOYS_NC);
    double2 p = c[4];
    double v = fma(p.y, t, p.x);
#pragma unroll
    for (int k = 3; k >= 0; k--) {
        p = c[k];
        v = fma(fma(v, t, p.y), t, p.x);
    }
    F[M] = v;
    if constexpr (M > 0) {
        const double ex = exp(-x), x2 = x + x;
#pragma unroll
        for (int m = M; m > 0; m--) F[m - 1] = fma(x2, F[m], ex) * (1. / (2 * m - 1));
    }
}

// index of the Cartesian component (lx, ., lz) of angular momentum l
__host__ __device__ constexpr int cart_index(int l, int lx, int lz) { return (l - lx) * (l - lx + 1) / 2 + lz; }
__host__ __device__ constexpr int cart_pow(int l, int c, int d) {
    return d == 0 ? cart_lx(l, c) : (d == 1 ? cart_ly(l, c) : cart_lz(l, c));
}
// axis along which component c is raised from a lower one, and that one
__host__ __device__ constexpr int cart_axis(int l, int c) { return cart_lx(l, c) > 0 ? 0 : (cart_ly(l, c) > 0 ? 1 : 2); }
__host__ __device__ constexpr int cart_down(int l, int c, int d) {
    return cart_index(l - 1, cart_lx(l, c) - (d == 0), cart_lz(l, c) - (d == 2));
}
// component c with one more power along d
__host__ __device__ constexpr int cart_up(int l, int c, int d) {
    return cart_index(l + 1, cart_lx(l, c) + (d == 0), cart_lz(l, c) + (d == 2));
}

template <class C>
struct JKOS {
    static constexpr int LA = C::LI + C::LJ, LC = C::LK + C::LL, L = LA + LC;
    // (dp|ss) and (fs|ss), all of it on the bra, run slower this way (5.9 against 3.7 ms for the (dp|ss) of
    // (H2O)64 / cc-pVDZ: the [f|s] intermediates spill) and keep the roots
    static constexpr bool USE = L <= 3 && LA < 3;
    static_assert(!USE || (C::LJ <= 1 && C::LL <= 1), "horizontal transfer by one unit");
    // contracted [e0|f0]: e = LI .. LA, f = LK .. LC
    static constexpr int NA = ncart(LA), NC = ncart(LC);
    static constexpr int NE = C::LJ ? ncart(C::LI) + NA : NA, NF = C::LL ? ncart(C::LK) + NC : NC;
    __host__ __device__ static constexpr int oe(int e) { return e == C::LI ? 0 : ncart(C::LI); }
    __host__ __device__ static constexpr int of(int f) { return f == C::LK ? 0 : ncart(C::LK); }

    // adds one primitive quartet; pre = the (ss|ss) prefactor, PA = P - Ri,
    // QC = Q - Rk, PQ = P - Q
    static __device__ __forceinline__ void prim(const double* F, double pre, const JKPrim& p, const double* PA,
                                                const double* QC, const double* PQ, double* E) {
        double T[LA + 1][LC + 1][L + 1][NA][NC];
        const double ra = p.B * p.iAB, rc = p.A * p.iAB;  // rho / A, rho / B
        const double ha = 0.5 * p.iA, hc = 0.5 * p.iB, hac = 0.5 * p.iAB;
        double WP[3], WQ[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            WP[d] = -ra * PQ[d];
            WQ[d] = rc * PQ[d];
        }
#pragma unroll
        for (int m = 0; m <= L; m++) T[0][0][m][0][0] = pre * F[m];
#pragma unroll
        for (int a = 0; a < LA; a++)
#pragma unroll
            for (int m = 0; m < L - a; m++)
#pragma unroll
                for (int t = 0; t < ncart(a + 1); t++) {
                    const int d = cart_axis(a + 1, t), lo = cart_down(a + 1, t, d);
                    double v = PA[d] * T[a][0][m][lo][0] + WP[d] * T[a][0][m + 1][lo][0];
                    if (a > 0) {
                        const int n = cart_pow(a, lo, d);
                        if (n > 0) {
                            const int l2 = cart_down(a, lo, d);
                            v += (n * ha) * (T[a > 0 ? a - 1 : 0][0][m][l2][0] - ra * T[a > 0 ? a - 1 : 0][0][m + 1][l2][0]);
                        }
                    }
                    T[a + 1][0][m][t][0] = v;
                }
#pragma unroll
        for (int c = 0; c < LC; c++)
#pragma unroll
            for (int a = 0; a <= LA; a++)
#pragma unroll
                for (int m = 0; m < LC - c; m++)
#pragma unroll
                    for (int s = 0; s < ncart(c + 1); s++) {
                        const int d = cart_axis(c + 1, s), lo = cart_down(c + 1, s, d);
#pragma unroll
                        for (int t = 0; t < ncart(a); t++) {
                            double v = QC[d] * T[a][c][m][t][lo] + WQ[d] * T[a][c][m + 1][t][lo];
                            if (c > 0) {
                                const int n = cart_pow(c, lo, d);
                                if (n > 0) {
                                    const int l2 = cart_down(c, lo, d);
                                    v += (n * hc) * (T[a][c > 0 ? c - 1 : 0][m][t][l2] -
                                                     rc * T[a][c > 0 ? c - 1 : 0][m + 1][t][l2]);
                                }
                            }
                            if (a > 0) {
                                const int n = cart_pow(a, t, d);
                                if (n > 0)
                                    v += (n * hac) * T[a > 0 ? a - 1 : 0][c][m + 1][cart_down(a, t, d)][lo];
                            }
                            T[a][c + 1][m][t][s] = v;
                        }
                    }
#pragma unroll
        for (int e = C::LI; e <= LA; e++)
#pragma unroll
            for (int f = C::LK; f <= LC; f++)
#pragma unroll
                for (int t = 0; t < ncart(e); t++)
#pragma unroll
                    for (int s = 0; s < ncart(f); s++) E[(oe(e) + t) * NF + of(f) + s] += T[e][f][0][t][s];
    }

    // (ij|kl) from the contracted [e0|f0]
    static __device__ __forceinline__ void transfer(const double* E, const double* AB, const double* CD, double* acc) {
#pragma unroll
        for (int i = 0; i < C::NFI; i++)
#pragma unroll
            for (int j = 0; j < C::NFJ; j++) {
                double B[NF];  // (i j| over the ket components
                if (C::LJ == 0) {
#pragma unroll
                    for (int f = 0; f < NF; f++) B[f] = E[i * NF + f];
                } else {
                    const int up = oe(LA) + cart_up(C::LI, i, j);
#pragma unroll
                    for (int f = 0; f < NF; f++) B[f] = E[up * NF + f] + AB[j] * E[i * NF + f];
                }
#pragma unroll
                for (int k = 0; k < C::NFK; k++)
#pragma unroll
                    for (int l = 0; l < C::NFL; l++)
                        acc[((i * C::NFJ + j) * C::NFK + k) * C::NFL + l] =
                            C::LL == 0 ? B[k] : B[of(LC) + cart_up(C::LK, k, l)] + CD[l] * B[k];
            }
    }
};
