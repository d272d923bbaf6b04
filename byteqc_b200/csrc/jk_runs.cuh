// Run kernels: the J/K kernels of the classes whose quartets fit one thread
// (JKClass::THREAD).
//
// What bounds these classes is not the recursion but the digestion: each
// contracted quartet reads the density at, and adds into K at, all
// (NFI + NFJ)(NFK + NFL) elements of its four K blocks, scattered over
// matrices of tens of MB.  A quartet at a time (the previous shape of these
// kernels) that was 16 scattered sector requests for a (ps|ss) quartet of
// some 150 FP64 operations, and the kernels waited on them.
//
// Work item: a run (up to 32 bra pairs ij that share the shell i, in Schwarz
// order) x a chunk (32 consecutive ket pairs kl of the class, in Schwarz buckets,
// one per lane).  The warp walks the bra pairs of the run; a lane keeps its
// ket pair's data, D_kl, D_ik, D_il and the sums for J_kl, K_ik and K_il
// across the walk (in registers, or in lane-private shared memory where they
// are many), and adds those to global memory once per item.  Per quartet only
// D_jk, D_jl are read and K_jk, K_jl added, j being the shell of the lower
// angular momentum: 4 scattered requests instead of 16 for (ps|ss), 8 instead
// of 56 for (ds|ps).  The bra pair's data is the same for the whole warp and
// lies in one record per pair (a few 16-byte loads).
//
// J_ij is a sum over the lanes.  Where a bra pair has few components (JT) the
// lanes put their terms into a 16 x 32 buffer in shared memory, one row per
// value, and a full buffer is summed by half a row per lane: 3 instructions
// per value instead of the 15 and more of a shuffle tree.
//
// The kernels run at 12 to 20 warps per SM and wait on latency, so the loop
// over the bra pairs touches no memory it could have had before: the run's
// records and D_ij are staged in shared memory when the item starts, and the
// D_jk, D_jl of small classes are asked for before the integrals.
//
// Screening: entry e of a run keeps the kets of Schwarz ranks [lo_e, hi_e) (the
// reference's decisions, from jk_screen_kernel).  A warp loads the bounds of the
// run's entries into its lanes, finds with one ballot the entries that meet
// its chunk, and walks those; a lane outside an entry's range contributes
// zeros.
#pragma once
#include "jk_kernels.cuh"
#include "jk_os.cuh"

#define JK_RUN_THREADS 128
#define JK_RUN_SMEM (110 * 1024)  // shared memory per block for two blocks per SM

// where a lane keeps its sums and its density elements
template <class C>
struct JKRunShape {
    static constexpr int NK = C::NFI * (C::NFK + C::NFL);  // K_ik, K_il elements
    static constexpr int NJ = C::NFK * C::NFL;             // J_kl elements
    static constexpr int NE = NK + NJ;
    static constexpr int NV = C::NFI * C::NFJ;             // J_ij elements
    // Boys table (L <= 3, JKOS) or Rys table; the FP32 tables are smaller
    static constexpr size_t TABW = JKOS<C>::USE ? BoysS::WORDS : RysS<C::NROOTS>::TWORDS;
    static constexpr size_t TAB = (TABW * sizeof(double) + 15) & ~(size_t)15;
    static_assert(RysF<C::NROOTS>::WORDS * sizeof(float) <= TAB || C::NROOTS > JK_F32_ROOTS, "FP32 table");
    static constexpr size_t SLOT = (size_t)NE * JK_RUN_THREADS * sizeof(double);
    static constexpr size_t JBUF = (size_t)JK_RUN_THREADS * 16 * sizeof(double);
    // staged records (12 doubles per entry) and D_ij
    static constexpr size_t STAGE = (size_t)JK_RUN_THREADS * 12 * sizeof(double);
    static constexpr bool DST = NV <= 10;
    static constexpr size_t DIJ = DST ? (size_t)JK_RUN_THREADS * NV * sizeof(double) : 0;
    static constexpr size_t FIX = TAB + STAGE + DIJ;
    // registers up to 15 elements ((ps|ps), (pp|ps)); then shared memory as
    // far as two blocks per SM allow; (fs|fs) adds per quartet
    static constexpr bool KREG = NE <= 15;
    static constexpr bool KSM = !KREG && FIX + SLOT <= JK_RUN_SMEM;
    static constexpr bool DREG = KREG;
    static constexpr bool DSM = KSM && FIX + 2 * SLOT <= JK_RUN_SMEM;
    static constexpr size_t SLOTS = (KSM ? SLOT : 0) + (DSM ? SLOT : 0);
    static constexpr bool JT = NV <= 10 && FIX + SLOTS + JBUF <= JK_RUN_SMEM;
    static constexpr size_t SMEM = FIX + SLOTS + (JT ? JBUF : 0);
    // One root at a time in a rolled loop where the code of all roots, times
    // the passes, does not stay in the instruction cache: unrolled, (fp|ps)
    // (4 passes, 3 roots) waited for instructions most (2.8 of 8.5 stalled
    // warps per issue).  (H2O)32 / def2-TZVP, unrolled and rolled: (fp|ps) 14.9
    // and 11.2 ms, (fs|pp) 7.4 and 5.7, (fs|fs) 4.9 and 3.2; at 2 and 3 passes
    // (dp|ps) 9.7 and 9.7, (pp|pp) 7.1 and 6.3, but on a contracted basis 3.34
    // and 3.63, 1.40 and 1.63.
    static constexpr bool ROLL = C::NPASS >= 4;
    // elements numbered J_kl [0, NJ), K_ik [NJ, ..), K_il
    static constexpr int OIK = NJ, OIL = NJ + C::NFI * C::NFK;
};

// shared memory of a build of n_dm > 1 densities (the sums only if they fit)
template <class C>
__host__ __device__ constexpr size_t jk_run_multi_smem(int n_dm) {
    using S = JKRunShape<C>;
    return S::FIX + n_dm * S::SLOT <= JK_RUN_SMEM ? S::FIX + n_dm * S::SLOT : S::FIX;
}

// Sums of V per-lane values over the warp by recursive halving: at each step
// a lane keeps half of its values and sends the other half to its partner
// (V = 3: 6 shuffles of a double instead of 15).  On return lane L holds the
// total of value jk_wsum_index<VP>(L) in v[0], or a copy of another lane's.
template <int N, int O>
__device__ __forceinline__ void jk_wsum_step(double* v) {
    const int lane = threadIdx.x & 31;
    if constexpr (N > 1) {
        constexpr int H = N / 2;
        const bool up = lane & O;
#pragma unroll
        for (int x = 0; x < H; x++) {
            const double send = up ? v[x] : v[x + H];
            const double keep = up ? v[x + H] : v[x];
            v[x] = keep + __shfl_xor_sync(0xffffffffu, send, O);
        }
        if constexpr (O > 1) jk_wsum_step<H, O / 2>(v);
    } else {
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], O);
        if constexpr (O > 1) jk_wsum_step<1, O / 2>(v);
    }
}

// index of the value that lane holds, -1 for the lanes holding a copy
template <int VP>
__device__ __forceinline__ int jk_wsum_index(int lane) {
    int idx = 0, n = VP, o = 16;
#pragma unroll
    for (int s = 0; s < 5; s++) {
        if (n > 1) {
            n >>= 1;
            if (lane & o) idx += n;
        } else if (lane & o) {
            idx = -1000;
        }
        o >>= 1;
    }
    return idx < 0 ? -1 : idx;
}

// Adds the warp's totals of the NV per-lane values v (value e at out(e)).
template <int NV, class Out>
__device__ __forceinline__ void jk_warp_add(double* v, const Out& out) {
    constexpr int V = NV < 16 ? NV : 16;
    constexpr int VP = V <= 1 ? 1 : V <= 2 ? 2 : V <= 4 ? 4 : V <= 8 ? 8 : 16;
    double t[VP];
#pragma unroll
    for (int e = 0; e < VP; e++) t[e] = e < V ? v[e < V ? e : 0] : 0.;
    jk_wsum_step<VP, 16>(t);
    const int idx = jk_wsum_index<VP>(threadIdx.x & 31);
    if (idx >= 0 && idx < V) out(idx, t[0]);
    if constexpr (NV > 16)
        jk_warp_add<NV - 16>(v + 16, [&](int e, double x) { out(16 + e, x); });
}

// bra primitive pair from its record
__device__ __forceinline__ JKPP jk_bra_pp(const double* __restrict__ rec) {
    const double2* r = reinterpret_cast<const double2*>(rec);
    const double2 u = __ldg(r), v = __ldg(r + 1), w = __ldg(r + 2);
    JKPP p;
    p.a = u.x;
    p.ia = u.y;
    p.e = v.x;
    p.P[0] = v.y;
    p.P[1] = w.x;
    p.P[2] = w.y;
    return p;
}
__device__ __forceinline__ JKPPF jk_bra_ppf(const float* __restrict__ rec) {
    const float4 u = __ldg(reinterpret_cast<const float4*>(rec));
    const float2 v = __ldg(reinterpret_cast<const float2*>(rec) + 2);
    JKPPF p;
    p.a = u.x;
    p.ia = u.y;
    p.e = u.z;
    p.D[0] = u.w;
    p.D[1] = v.x;
    p.D[2] = v.y;
    return p;
}

// One warp's work on one item.  The state of a lane: element e of
// [0, OIK) is J_kl, of [OIK, OIL) K_ik, of [OIL, NE) K_il; the density
// element it is paired with (D_kl, D_ik, D_il) has the same number.  What the
// loop over the bra pairs needs of the segment is copied here: the segment
// itself (in shared memory) would be read again after every atomic.
//
// KROWS: element (a, b) of K goes to a * nao + b, so that the lanes of a warp,
// whose ket shells are consecutive, add side by side; the caller reads V + V^T
// only, or transposes.  Otherwise to a + nao * b, the layout of the C-ABI
// (per-class-pair entries).  A template argument: with the two strides read
// from the segment the builds took 1 to 2 % longer ((ps|ps) 332 bytes of
// spill loads instead of 220); writing a + nao * b in every build, (H2O)64 /
// cc-pVDZ took 146 instead of 95 ms and (H2O)32 / TZVP 288 instead of 256.
template <class C, typename R, bool MULTI, bool KROWS>
struct JKRunItem {
    using S = JKRunShape<C>;
    static constexpr int NFI = C::NFI, NFJ = C::NFJ, NFK = C::NFK, NFL = C::NFL, TS = JK_RUN_THREADS;
    static constexpr bool KREG = S::KREG && !MULTI, DREG = S::DREG && !MULTI, DSM = S::DSM && !MULTI;
    static constexpr bool JT = S::JT && !MULTI;
    static constexpr int NJK = NFJ * NFK, NJL = NFJ * NFL, NV = S::NV;
    static constexpr int EW = NV <= 16 ? 16 / NV : 1;  // bra pairs per J_ij buffer
    static constexpr bool DEARLY = !MULTI && NJK + NJL <= 4;
    static constexpr bool DST = S::DST && !MULTI;
    static constexpr bool F32P = JKF32Prim<C, R>::value;

    const JKSeg& sg;
    const double* tab;
    double *ssum, *sden, *jbuf;  // this thread's shared-memory slots (stride TS), the warp's buffer
    double2* rec;                // the warp's staged records, 6 per entry
    double* sdij;                // and D_ij, NV per entry
    double sum[KREG ? S::NE : 1], den[DREG ? S::NE : 1];
    double kjk[MULTI ? 1 : NJK], kjl[MULTI ? 1 : NJL];
    const double *D, *dpb, *bprim;
    const float* bprimf;
    double *vk, *jpb;
    bool keep, dj, dk, active;
    int ndm, nao, i0, j0, k0, l0, col, prim_kl, npij, npkl, pst_ij, el;
    double norm, ri[3], rj[3], rk[3], rl[3];
    JKPP kp;
    JKPPF kpf;
    double djk[DEARLY ? NJK : 1], djl[DEARLY ? NJL : 1];

    __device__ __forceinline__ const double* drow(int m, int a) const { return D + ((size_t)m * nao + a) * nao; }
    // K element (a, b) of density m at krow(m, a) + kcol(b)
    __device__ __forceinline__ double* krow(int m, int a) const {
        return KROWS ? vk + ((size_t)m * nao + a) * nao : vk + (size_t)m * nao * nao + a;
    }
    __device__ __forceinline__ size_t kcol(int b) const { return KROWS ? b : (size_t)b * nao; }

    // density element paired with element e of the state
    __device__ __forceinline__ double dload(int m, int e) const {
        if (e < S::OIK)
            return sg.dp ? __ldg(sg.dp + sg.pk_kl + m * sg.pk_stride + (size_t)e * sg.pst_kl + col)
                         : __ldg(drow(m, l0 + e % NFL) + k0 + e / NFL);
        if (e < S::OIL) return __ldg(drow(m, i0 + (e - S::OIK) / NFK) + k0 + (e - S::OIK) % NFK);
        return __ldg(drow(m, i0 + (e - S::OIL) / NFL) + l0 + (e - S::OIL) % NFL);
    }
    __device__ __forceinline__ double density(int m, int e) const {
        if constexpr (DREG) return den[e];
        else if constexpr (DSM) return sden[e * TS];
        else return dload(m, e);
    }
    // element e of the state added to the output
    __device__ __forceinline__ void gadd(int m, int e, double v) const {
        if (e < S::OIK) {
            if (sg.jp) atomicAdd(sg.jp + sg.pk_kl + m * sg.pk_stride + (size_t)e * sg.pst_kl + col, v);
            else atomicAdd(sg.vj + (size_t)m * nao * nao + (k0 + e / NFL) + (size_t)nao * (l0 + e % NFL), v);
        } else if (e < S::OIL) {
            atomicAdd(krow(m, i0 + (e - S::OIK) / NFK) + kcol(k0 + (e - S::OIK) % NFK), v);
        } else {
            atomicAdd(krow(m, i0 + (e - S::OIL) / NFL) + kcol(l0 + (e - S::OIL) % NFL), v);
        }
    }
    __device__ __forceinline__ void add(int m, int e, double v) {
        if constexpr (KREG) sum[e] += v;
        else if (keep) ssum[(size_t)(m * S::NE + e) * TS] += v;
        else gadd(m, e, v);
    }
    // J_ij element x of the bra pair of entry `entry` of the run's class
    __device__ __forceinline__ void jadd(int m, int entry, int x, double v) const {
        if (jpb) atomicAdd(jpb + m * sg.pk_stride + (size_t)entry * NV + x, v);
        else atomicAdd(sg.vj + (size_t)m * nao * nao + (i0 + x / NFJ) + (size_t)nao * (j0 + x % NFJ), v);
    }

    // integrals of the quartet for the bra components [CI0, CI0 + NI), summed
    // over primitives and roots into acc
    __device__ __forceinline__ JKPP bra(int p) const {
        if (p) return jk_bra_pp(bprim + (size_t)p * pst_ij * 8);
        const double2 u = rec[6 * el], v = rec[6 * el + 1], w = rec[6 * el + 2];
        return JKPP{u.x, u.y, v.x, {v.y, w.x, w.y}};
    }
    __device__ __forceinline__ JKPPF braf(int p) const {
        if (p) return jk_bra_ppf(bprimf + (size_t)p * pst_ij * 8);
        const float4 u = reinterpret_cast<const float4*>(rec)[6 * el];
        const float2 v = *reinterpret_cast<const float2*>(rec + 6 * el + 1);
        return JKPPF{u.x, u.y, u.z, {u.w, v.x, v.y}};
    }

    template <int CI0, int NI>
    __device__ __forceinline__ void integrals(R* acc) {
        constexpr int NR = C::NROOTS;
#pragma unroll
        for (int e = 0; e < NI * NFJ * NFK * NFL; e++) acc[e] = R(0);
        if constexpr (F32P) {
            const float* tabf = reinterpret_cast<const float*>(tab);
            float dij[3], dkl[3], ac[3];
#pragma unroll
            for (int d = 0; d < 3; d++) {
                dij[d] = (float)(ri[d] - rj[d]);
                dkl[d] = (float)(rk[d] - rl[d]);
                ac[d] = (float)(ri[d] - rk[d]);
            }
            const float normf = (float)norm;
            for (int q = 0; q < npkl; q++) {
                if (npkl > 1) kpf = jk_ppf(sg, prim_kl + q * sg.pst_kl);
                for (int p = 0; p < npij; p++) {
                    const JKPrimF pr = jk_prim_f2(braf(p), kpf, ac);
                    auto root = [&](float s, float w) {
                        float Ix[C::GS], Iy[C::GS], Iz[C::GS];
                        jk_unit_f<C>(pr, s, w, 0, normf, dij, dkl, Ix);
                        jk_unit_f<C>(pr, s, w, 1, normf, dij, dkl, Iy);
                        jk_unit_f<C>(pr, s, w, 2, normf, dij, dkl, Iz);
                        jk_thread_products<C, R, CI0, NI>(acc, Ix, Iy, Iz);
                    };
                    if constexpr (S::ROLL) {
#pragma unroll 1
                        for (int r = 0; r < NR; r++) {
                            float s, w;
                            rys_root_one_f<NR>(tabf, pr.x, r, s, w);
                            root(s, w);
                        }
                    } else {
                        float rs[NR], rw[NR];
                        rys_table_all_f<NR>(tabf, pr.x, rs, rw);
#pragma unroll
                        for (int r = 0; r < NR; r++) root(rs[r], rw[r]);
                    }
                }
            }
        } else if constexpr (JKOS<C>::USE) {
            using OS = JKOS<C>;
            static_assert(CI0 == 0 && NI == NFI && sizeof(R) == 8, "one pass");
            double E[OS::NE * OS::NF];
#pragma unroll
            for (int e = 0; e < OS::NE * OS::NF; e++) E[e] = 0.;
            for (int q = 0; q < npkl; q++) {
                if (npkl > 1) kp = jk_pp(sg, prim_kl + q * sg.pst_kl);
                for (int p = 0; p < npij; p++) {
                    const JKPrim pr = jk_prim2(bra(p), kp);
                    double F[OS::L + 1], PA[3], QC[3], PQ[3];
                    boys_all<OS::L>(tab, pr.x, F);
#pragma unroll
                    for (int d = 0; d < 3; d++) {
                        PA[d] = pr.P[d] - ri[d];
                        QC[d] = pr.Q[d] - rk[d];
                        PQ[d] = pr.P[d] - pr.Q[d];
                    }
                    OS::prim(F, norm * pr.sy, pr, PA, QC, PQ, E);
                }
            }
            const double AB[3] = {ri[0] - rj[0], ri[1] - rj[1], ri[2] - rj[2]};
            const double CD[3] = {rk[0] - rl[0], rk[1] - rl[1], rk[2] - rl[2]};
            OS::transfer(E, AB, CD, acc);
        } else {
            for (int q = 0; q < npkl; q++) {
                if (npkl > 1) kp = jk_pp(sg, prim_kl + q * sg.pst_kl);
                for (int p = 0; p < npij; p++) {
                    const JKPrim pr = jk_prim2(bra(p), kp);
                    auto root = [&](double s, double w) {
                        R Ix[C::GS], Iy[C::GS], Iz[C::GS];
                        jk_unit<C, R>(pr, s, w, 0, norm, ri, rj, rk, rl, Ix);
                        jk_unit<C, R>(pr, s, w, 1, norm, ri, rj, rk, rl, Iy);
                        jk_unit<C, R>(pr, s, w, 2, norm, ri, rj, rk, rl, Iz);
                        jk_thread_products<C, R, CI0, NI>(acc, Ix, Iy, Iz);
                    };
                    if constexpr (S::ROLL) {
#pragma unroll 1
                        for (int r = 0; r < NR; r++) {
                            double s, w;
                            rys_root_one<NR>(tab, pr.x, r, s, w);
                            root(s, w);
                        }
                    } else {
                        double rs[NR], rw[NR];
                        rys_table_all<NR>(tab, pr.x, rs, rw);
#pragma unroll
                        for (int r = 0; r < NR; r++) root(rs[r], rw[r]);
                    }
                }
            }
        }
    }

    __device__ __forceinline__ void load_dj(int m, double* djk, double* djl) const {
#pragma unroll
        for (int j = 0; j < NFJ; j++) {
            const double* row = drow(m, j0 + j);
#pragma unroll
            for (int k = 0; k < NFK; k++) djk[j * NFK + k] = __ldg(row + k0 + k);
#pragma unroll
            for (int l = 0; l < NFL; l++) djl[j * NFL + l] = __ldg(row + l0 + l);
        }
    }

    template <int CI0, int NI>
    __device__ __forceinline__ void pass(int entry) {
        constexpr int NA = NI * NFJ * NFK * NFL, V0 = CI0 * NFJ, NX = NI * NFJ;
        R acc[NA];
        if (active) {
            integrals<CI0, NI>(acc);
        } else {
#pragma unroll
            for (int e = 0; e < NA; e++) acc[e] = R(0);
        }
#define ACC(i, j, k, l) ((double)acc[(((i) * NFJ + (j)) * NFK + (k)) * NFL + (l)])
        for (int m = 0; m < ndm; m++) {
            if (dj) {
                double vij[NX];
#pragma unroll
                for (int e = 0; e < NX; e++) vij[e] = 0.;
#pragma unroll
                for (int e = 0; e < S::NJ; e++) {
                    const double d = density(m, e);
#pragma unroll
                    for (int x = 0; x < NX; x++) vij[x] += ACC(x / NFJ, x % NFJ, e / NFL, e % NFL) * d;
                }
                if constexpr (JT) {
                    double* row = jbuf + (el % EW) * NV * 32 + V0 * 32 + (threadIdx.x & 31);
#pragma unroll
                    for (int x = 0; x < NX; x++) row[x * 32] = vij[x];
                } else {
                    jk_warp_add<NX>(vij, [&](int x, double v) { jadd(m, entry, V0 + x, v); });
                }
            }
            if (!active) continue;
            if (dj) {
                double v[S::NJ];
#pragma unroll
                for (int e = 0; e < S::NJ; e++) v[e] = 0.;
#pragma unroll
                for (int x = 0; x < NX; x++) {
                    double d;
                    if constexpr (DST) d = sdij[el * NV + V0 + x];
                    else d = dpb ? __ldg(dpb + m * sg.pk_stride + (size_t)entry * NV + V0 + x)
                                 : __ldg(drow(m, j0 + x % NFJ) + i0 + CI0 + x / NFJ);
#pragma unroll
                    for (int e = 0; e < S::NJ; e++) v[e] += ACC(x / NFJ, x % NFJ, e / NFL, e % NFL) * d;
                }
#pragma unroll
                for (int e = 0; e < S::NJ; e++) add(m, e, v[e]);
            }
            if (dk) {
                double ljk[DEARLY ? 1 : NJK], ljl[DEARLY ? 1 : NJL];
                if constexpr (!DEARLY) load_dj(m, ljk, ljl);
                const double *djk = DEARLY ? this->djk : ljk, *djl = DEARLY ? this->djl : ljl;
#pragma unroll
                for (int i = 0; i < NI; i++)
#pragma unroll
                    for (int k = 0; k < NFK; k++) {
                        double v = 0;
#pragma unroll
                        for (int e = 0; e < NJL; e++) v += ACC(i, e / NFL, k, e % NFL) * djl[e];
                        add(m, S::OIK + (CI0 + i) * NFK + k, v);
                    }
#pragma unroll
                for (int i = 0; i < NI; i++)
#pragma unroll
                    for (int l = 0; l < NFL; l++) {
                        double v = 0;
#pragma unroll
                        for (int e = 0; e < NJK; e++) v += ACC(i, e / NFK, e % NFK, l) * djk[e];
                        add(m, S::OIL + (CI0 + i) * NFL + l, v);
                    }
                double vjk[NJK], vjl[NJL];
#pragma unroll
                for (int e = 0; e < NJK; e++) vjk[e] = 0.;
#pragma unroll
                for (int e = 0; e < NJL; e++) vjl[e] = 0.;
#pragma unroll
                for (int i = 0; i < NI; i++) {
#pragma unroll
                    for (int l = 0; l < NFL; l++) {
                        const double d = density(m, S::OIL + (CI0 + i) * NFL + l);
#pragma unroll
                        for (int e = 0; e < NJK; e++) vjk[e] += ACC(i, e / NFK, e % NFK, l) * d;
                    }
#pragma unroll
                    for (int k = 0; k < NFK; k++) {
                        const double d = density(m, S::OIK + (CI0 + i) * NFK + k);
#pragma unroll
                        for (int e = 0; e < NJL; e++) vjl[e] += ACC(i, e / NFL, k, e % NFL) * d;
                    }
                }
                if constexpr (MULTI) {
                    flush_j(m, vjk, vjl);
                } else {
#pragma unroll
                    for (int e = 0; e < NJK; e++) kjk[e] += vjk[e];
#pragma unroll
                    for (int e = 0; e < NJL; e++) kjl[e] += vjl[e];
                }
            }
        }
#undef ACC
    }

    __device__ __forceinline__ void flush_j(int m, const double* vjk, const double* vjl) const {
#pragma unroll
        for (int j = 0; j < NFJ; j++) {
            double* row = krow(m, j0 + j);
#pragma unroll
            for (int k = 0; k < NFK; k++) atomicAdd(row + kcol(k0 + k), vjk[j * NFK + k]);
#pragma unroll
            for (int l = 0; l < NFL; l++) atomicAdd(row + kcol(l0 + l), vjl[j * NFL + l]);
        }
    }

    template <int P>
    __device__ __forceinline__ void passes(int entry) {
        constexpr int CI0 = P * C::GI;
        if constexpr (CI0 < NFI) {
            pass<CI0, (CI0 + C::GI < NFI ? C::GI : NFI - CI0)>(entry);
            passes<P + 1>(entry);
        }
    }

    // sums the rows of the J_ij buffer: value v of the window of bra pairs
    // [w EW, w EW + EW) of the run, for those in `done`
    __device__ __forceinline__ void flush_jbuf(int e0, int w, unsigned done) const {
        const int lane = threadIdx.x & 31, v = lane & 15, x = w * EW + v / NV;
        __syncwarp();
        const bool on = v < EW * NV && x < 32 && ((done >> x) & 1);
        double t = 0.;
        if (on) {
            const double* row = jbuf + v * 32 + (lane & 16);
#pragma unroll
            for (int c = 0; c < 16; c++) t += row[c ^ v];
        }
        t += __shfl_xor_sync(0xffffffffu, t, 16);
        if (on && lane < 16) {
            if (jpb) {
                atomicAdd(jpb + (size_t)(e0 + x) * NV + v % NV, t);
            } else {
                const int jj = __double2loint(rec[6 * x + 4].y);
                const int c = v % NV;
                atomicAdd(sg.vj + (i0 + c / NFJ) + (size_t)nao * (jj + c % NFJ), t);
            }
        }
        __syncwarp();
    }

    __device__ __forceinline__ void work(long long item) {
        const int lane = threadIdx.x & 31;
        int run = 0;  // 32-ary search of the item prefix, all lanes probing
        for (int n = sg.nrun; n > 1;) {
            const int step = (n + 31) >> 5;
            const bool ok = lane * step < n && __ldg(sg.ioff + run + lane * step) <= item;
            const int last = __popc(__ballot_sync(0xffffffffu, ok)) - 1;
            run += last * step;
            n = min(step, n - last * step);
        }
        const int e0 = __ldg(sg.run0 + run), ne = __ldg(sg.run0 + run + 1) - e0;
        int elo = 0, ehi = 0, ent = 0;
        if (lane < ne) {
            elo = sg.elo ? __ldg(sg.elo + e0 + lane) : 0;
            ehi = __ldg(sg.ehi + e0 + lane);
            ent = __ldg(sg.ent + e0 + lane);
        }
        const int base =
            sg.elo ? jk_item_base(__reduce_min_sync(0xffffffffu, elo < ehi ? elo : 0x7fffffff), sg.bucket, 32) : 0;
        const int mycol = base + 32 * (int)(item - __ldg(sg.ioff + run)) + lane;
        // Schwarz ranks of the chunk's pairs
        const bool in = mycol < sg.pst_kl;
        const int rank = in ? __ldg(sg.rank + sg.pair_kl0 + mycol) : -1;
        const int rmin = __reduce_min_sync(0xffffffffu, in ? rank : 0x7fffffff),
                  rmax = __reduce_max_sync(0xffffffffu, rank);
        unsigned mask = __ballot_sync(0xffffffffu, elo < ehi && elo <= rmax && ehi > rmin);
        if (mask == 0) return;
        const int ent0 = __shfl_sync(0xffffffffu, ent, 0);
        pst_ij = sg.pst_ij;
        col = min(mycol, sg.pst_kl - 1);
        const int bkl = sg.pair_kl0 + col;
        nao = sg.nao;
        D = sg.dm;
        vk = sg.vk;
        dj = sg.vj != nullptr;
        dk = vk != nullptr;
        dpb = sg.dpb ? sg.dpb + sg.pk_ij : nullptr;
        jpb = sg.jpb ? sg.jpb + sg.pk_ij : nullptr;
        k0 = __ldg(sg.pao + bkl);
        l0 = __ldg(sg.pao + sg.npt + bkl);
        load_pair_centres(sg, bkl, rk, rl);
        {
            const int bij = sg.pair_ij0 + ent0;  // the shell i of the run
            i0 = __ldg(sg.pao + bij);
#pragma unroll
            for (int d = 0; d < 3; d++) ri[d] = __ldg(sg.pgeo + (size_t)d * sg.npt + bij);
        }
        prim_kl = sg.prim_kl0 + col;
        npkl = sg.pnp ? __ldg(sg.pnp + bkl) : sg.nprim_kl;
        if constexpr (F32P) kpf = jk_ppf(sg, prim_kl);
        else kp = jk_pp(sg, prim_kl);
        ndm = MULTI ? sg.n_dm : 1;
        keep = MULTI ? jk_run_multi_smem<C>(ndm) > S::FIX : (S::KREG || S::KSM);
        if constexpr (KREG) {
#pragma unroll
            for (int e = 0; e < S::NE; e++) sum[e] = 0.;
        } else if (keep) {
            for (int e = 0; e < ndm * S::NE; e++) ssum[e * TS] = 0.;
        }
        if constexpr (DREG || DSM) {
#pragma unroll
            for (int e = 0; e < S::NE; e++)
                if (e < S::OIK ? dj : dk) {
                    if constexpr (DREG) den[e] = dload(0, e);
                    else sden[e * TS] = dload(0, e);
                }
        }
        // pair index of the ket in the bra's class, for the ij == kl diagonal
        const int diag = sg.pair_ij0 == sg.pair_kl0 ? mycol : -1;
        const double* bprim0 = sg.bprim + (size_t)e0 * 8;
        const float* bprimf0 = sg.bprimf + (size_t)e0 * 8;
        // stage the run
        __syncwarp();
        if ((mask >> lane) & 1) {
            double2* r = rec + 6 * lane;
            if constexpr (F32P) {
                const float4* f = reinterpret_cast<const float4*>(bprimf0 + lane * 8);
                reinterpret_cast<float4*>(r)[0] = __ldg(f);
                reinterpret_cast<float4*>(r)[1] = __ldg(f + 1);
            } else {
                const double2* f = reinterpret_cast<const double2*>(bprim0 + lane * 8);
                r[0] = __ldg(f);
                r[1] = __ldg(f + 1);
                r[2] = __ldg(f + 2);
            }
            const double2* f = reinterpret_cast<const double2*>(sg.bpair + (size_t)(e0 + lane) * 4);
            r[3] = __ldg(f);
            r[4] = __ldg(f + 1);
            *reinterpret_cast<int4*>(r + 5) = make_int4(elo, ehi, ent, 0);
        }
        if constexpr (DST)
            if (dj) {
                if (dpb) {
                    for (int x = lane; x < ne * NV; x += 32) sdij[x] = __ldg(dpb + (size_t)e0 * NV + x);
                } else if (lane < ne) {
                    const int jj = __ldg(sg.pao + sg.npt + sg.pair_ij0 + ent);
#pragma unroll
                    for (int x = 0; x < NV; x++)
                        sdij[lane * NV + x] = __ldg(drow(0, jj + x % NFJ) + i0 + x / NFJ);
                }
            }
        __syncwarp();
        bool used = false;  // whether this lane had a quartet
        unsigned done = 0;  // bra pairs in the J_ij buffer
        while (mask) {
            el = __ffs(mask) - 1;
            mask &= mask - 1;
            const int4 bound = *reinterpret_cast<const int4*>(rec + 6 * el + 5);
            const double2 pb = rec[6 * el + 4];
            active = rank >= bound.x && rank < bound.y;
            used |= active;
            j0 = __double2loint(pb.y);
            npij = __double2hiint(pb.y);
            if constexpr (DEARLY)
                if (dk) load_dj(0, djk, djl);
            if constexpr (C::LJ > 0) {
                const double2 pa = rec[6 * el + 3];
                rj[0] = pa.x;
                rj[1] = pa.y;
                rj[2] = pb.x;
            } else {
                rj[0] = rj[1] = rj[2] = 0.;
            }
            if constexpr (F32P) bprimf = bprimf0 + el * 8;
            else bprim = bprim0 + el * 8;
            // 2 pi^3 / sqrt(pi), halved on the ij == kl diagonal (g2e.c:41, g2e.cu:1025)
            norm = bound.z == diag ? 0.5 * JK_FAC : JK_FAC;
            if constexpr (!MULTI) {
#pragma unroll
                for (int e = 0; e < NJK; e++) kjk[e] = 0.;
#pragma unroll
                for (int e = 0; e < NJL; e++) kjl[e] = 0.;
            }
            passes<0>(e0 + el);
            if constexpr (!MULTI)
                if (dk && active) flush_j(0, kjk, kjl);
            if constexpr (JT) {
                done |= 1u << el;
                if (dj && (mask == 0 || (__ffs(mask) - 1) / EW != el / EW)) {
                    flush_jbuf(e0, el / EW, done);
                    done = 0;
                }
            }
        }
        if (used && keep) {
            for (int m = 0; m < ndm; m++) {
#pragma unroll
                for (int e = 0; e < S::NE; e++)
                    if (e < S::OIK ? dj : dk) {
                        if constexpr (KREG) gadd(m, e, sum[e]);
                        else gadd(m, e, ssum[(size_t)(m * S::NE + e) * TS]);
                    }
            }
        }
    }
};

// Resident blocks asked of the register allocator.  One more of each in the
// double kernels (6, 5, 4 for 5, 4, 3) spills: (H2O)32 / TZVP 212 instead of 206
// ms, (H2O)64 / cc-pVDZ 143 instead of 112.
template <class C, typename R>
struct JKRunMinBlocks {
    static constexpr int value = sizeof(R) == 4 ? (C::W <= 10 ? 5 : (C::W <= 24 ? 4 : (C::W <= 40 ? 3 : 2)))
                                                : (C::W <= 4 ? 5 : (C::W <= 10 ? 4 : (C::W <= 24 ? 3 : 2)));
};

// The items of one warp.  segt: exclusive item prefix of the segments.
// Static mode (queue null): the warps of the grid take items in turn, so that
// neighbouring warps share the bra pairs of a run in L1.  Persistent mode: a
// warp takes `grab` consecutive items from *queue (zeroed before the launch)
// until they run out.  seg: the warp's copy of the segment it works on.
template <class Item>
__device__ __forceinline__ void jk_run_items(const JKSeg* __restrict__ segs, const long long* __restrict__ segt,
                                             int nseg, long long total, unsigned long long* queue, int grab,
                                             JKSeg& seg, Item& w) {
    const int lane = threadIdx.x & 31;
    const long long nwarps = (long long)gridDim.x * (JK_RUN_THREADS / 32);
    long long sbeg = 0, send = 0;
    for (long long t0 = (long long)blockIdx.x * (JK_RUN_THREADS / 32) + (threadIdx.x >> 5);; t0 += nwarps) {
        long long t = t0, tend = t0 + 1;
        if (queue) {
            unsigned long long g = 0;
            if (lane == 0) g = atomicAdd(queue, (unsigned long long)grab);
            t = (long long)__shfl_sync(0xffffffffu, g, 0);
            tend = min(total, t + grab);
        }
        if (t >= total) break;
        for (; t < tend; t++) {
            if (t >= send || t < sbeg) {
                const int s = jk_find_seg(segt, nseg, t);
                sbeg = segt[s];
                send = segt[s + 1];
                __syncwarp();
                const int* src = reinterpret_cast<const int*>(segs + s);
                int* dst = reinterpret_cast<int*>(&seg);
                for (int x = lane; x < (int)(sizeof(JKSeg) / 4); x += 32) dst[x] = src[x];
                __syncwarp();
            }
            w.work(t - sbeg);
        }
    }
}

template <class C, typename R, bool MULTI, bool KROWS>
__global__ void __launch_bounds__(JK_RUN_THREADS, (JKRunMinBlocks<C, R>::value))
    jk_run_kernel(const JKSeg* __restrict__ segs, const long long* __restrict__ segt, int nseg,
                  unsigned long long* queue, int grab) {
    extern __shared__ __align__(16) double jk_tab[];
    __shared__ JKSeg s_seg[JK_RUN_THREADS / 32];  // the segment each warp works on
    using S = JKRunShape<C>;
    const long long total = segt[nseg];
    const int warp = threadIdx.x >> 5;
    if (!queue && (long long)blockIdx.x * (JK_RUN_THREADS / 32) >= total) return;  // block-uniform
    if (total == 0) return;
    if constexpr (JKF32Prim<C, R>::value) rys_table_copy_f<C::NROOTS>(segs[0].rys, reinterpret_cast<float*>(jk_tab));
    else if constexpr (JKOS<C>::USE) boys_table_copy<JKOS<C>::L>(segs[0].rys, jk_tab);
    else rys_table_copy<C::NROOTS>(segs[0].rys, jk_tab);
    __syncthreads();
    double* stage = jk_tab + S::TAB / sizeof(double);
    double* dij = stage + S::STAGE / sizeof(double);
    double* slots = jk_tab + S::FIX / sizeof(double);
    JKRunItem<C, R, MULTI, KROWS> w{s_seg[warp],
                             jk_tab,
                             slots + threadIdx.x,
                             slots + S::SLOT / sizeof(double) + threadIdx.x,
                             slots + S::SLOTS / sizeof(double) + warp * 16 * 32,
                             reinterpret_cast<double2*>(stage) + warp * 32 * 6,
                             dij + warp * 32 * S::NV};
    jk_run_items(segs, segt, nseg, total, queue, grab, s_seg[warp], w);
}
