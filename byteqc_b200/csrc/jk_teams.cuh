// Team run kernels: the J/K kernels of the classes too large for a thread per
// quartet whose bra component i has a lane of its own (JKClass::TRUN).
//
// A team of T = NFI lanes (6 or 10) works on one ket pair and walks the bra
// pairs of a run, as the lanes of jk_runs.cuh do; TPW = 32 / T teams share a
// warp and the run, and nothing crosses warps, so there is no block barrier.
// Lane ci of a team keeps row ci of K_ik and K_il (complete in the lane) and
// its part of J_kl over the run, and adds them once per run.  Per quartet
// only J_ij (summed over the teams of the warp) and K_jk, K_jl (summed over
// the lanes of the team) leave the warp.
//
// Products: these kernels were bound by shared-memory loads, three per
// product of two multiplications.  The 2D blocks in shared memory now stop
// at the bra transfer (LK + LL + 1 entries per (i, j) instead of
// (LK+1)(LL+1)); a lane loads its rows of one root, does the ket transfer in
// registers (a few FMAs) and forms all its products from registers: 18 loads
// for the 27 components of a (dp|pp) lane and root instead of 81.
#pragma once
#include "jk_runs.cuh"

template <class C, typename R>
struct JKTRunShape {
    static constexpr int T = C::T, TPW = C::TPW, MM = C::MM, NR = C::NROOTS;
    static constexpr int NB = 128 / (int)sizeof(R);  // banks in elements of R
    // strides of a unit's block H[i][j][m]: rows of different i in different
    // banks, an odd stride between the units that the lanes write at once
    static constexpr int SJ = MM + 1;
    static constexpr int pick_si() {
        int best = (C::LJ + 1) * SJ, bw = 1 << 20;
        for (int s = (C::LJ + 1) * SJ; s < (C::LJ + 1) * SJ + NB; s++) {
            int a[8] = {};
            for (int x = 0; x <= C::LI; x++) a[x] = x * s;
            const int w = jk_bank_ways(a, C::LI + 1, NB);
            if (w < bw) {
                bw = w;
                best = s;
            }
        }
        return best;
    }
    static constexpr int SI = pick_si();
    static constexpr int GS = (C::LI * SI + C::LJ * SJ + MM + 1) | 1;
    static constexpr int NJ = C::NFJ * (C::NFK + C::NFL);  // K_jk, K_jl elements
    static constexpr int NKET = C::NFK * C::NFL;
    static constexpr int PS = (NJ > NKET ? NJ : NKET) | 1;  // doubles per lane of the team sums
    static constexpr int GW = (3 * NR * GS * (int)sizeof(R) + 7) / 8;
    static constexpr int WORDS0 = GW > T * PS ? GW : T * PS;
    // team stride in doubles, odd multiple of 2: the teams of a warp in
    // different banks
    static constexpr int WORDS = ((WORDS0 + 1) & ~1) % 4 == 2 ? ((WORDS0 + 1) & ~1) : ((WORDS0 + 1) & ~1) + 2;
    static constexpr bool SMEM_TAB = NR <= 4;
    static constexpr bool F32P = JKF32Prim<C, R>::value;
    static_assert(!F32P || SMEM_TAB, "single-precision roots come from shared memory");
    static constexpr size_t TAB = SMEM_TAB ? ((size_t)RysS<NR>::TWORDS * sizeof(double) + 15) & ~(size_t)15 : 0;
    static constexpr size_t WARP = (size_t)TPW * WORDS * 8 + 32 * 12 * 8;  // team regions, staged records
    static constexpr size_t SMEM = TAB + (JK_RUN_THREADS / 32) * WARP;
};

template <class C, typename R, bool MULTI, bool KROWS>
struct JKTRunItem {
    using S = JKTRunShape<C, R>;
    static constexpr int NFI = C::NFI, NFJ = C::NFJ, NFK = C::NFK, NFL = C::NFL, T = C::T, TPW = C::TPW;
    static constexpr int NR = C::NROOTS, NJK = NFJ * NFK, NJL = NFJ * NFL, NKET = NFK * NFL, MM = C::MM;
    static constexpr int NV = NFI * NFJ;

    const JKSeg& sg;
    const double* tab;
    R* g;          // the team's 2D blocks
    double* part;  // the same memory: per-lane sums of the team
    double2* rec;  // the warp's staged records, 6 per entry
    double kik[NFK], kil[NFL], jkl[NKET];
    const double *D, *dpb, *bprim;
    const float* bprimf;
    double *vk, *jpb;
    bool dj, dk, active, mine;
    int ndm, nao, i0, j0, k0, l0, col, prim_kl, npij, npkl, pst_ij, el, ci, team;
    double norm, ri[3], rj[3], rk[3], rl[3];
    int ox, oy, oz;  // rows of component ci

    __device__ __forceinline__ const double* drow(int m, int a) const { return D + ((size_t)m * nao + a) * nao; }
    // K element (a, b) of density m at krow(m, a) + kcol(b), as in JKRunItem
    __device__ __forceinline__ double* krow(int m, int a) const {
        return KROWS ? vk + ((size_t)m * nao + a) * nao : vk + (size_t)m * nao * nao + a;
    }
    __device__ __forceinline__ size_t kcol(int b) const { return KROWS ? b : (size_t)b * nao; }

    __device__ __forceinline__ double dkl(int m, int e) const {
        return sg.dp ? __ldg(sg.dp + sg.pk_kl + m * sg.pk_stride + (size_t)e * sg.pst_kl + col)
                     : __ldg(drow(m, l0 + e % NFL) + k0 + e / NFL);
    }

    // the 3 NR (axis, root) blocks of one primitive quartet, spread over the team
    __device__ __forceinline__ void build(int p, int q) const {
        if constexpr (S::F32P) {
            JKPPF b;
            if (p) {
                b = jk_bra_ppf(bprimf + (size_t)p * pst_ij * 8);
            } else {
                const float4 u = reinterpret_cast<const float4*>(rec)[6 * el];
                const float2 v = *reinterpret_cast<const float2*>(rec + 6 * el + 1);
                b = JKPPF{u.x, u.y, u.z, {u.w, v.x, v.y}};
            }
            float dij[3], dklv[3], ac[3];
#pragma unroll
            for (int d = 0; d < 3; d++) {
                dij[d] = (float)(ri[d] - rj[d]);
                dklv[d] = (float)(rk[d] - rl[d]);
                ac[d] = (float)(ri[d] - rk[d]);
            }
            const JKPrimF pr = jk_prim_f2(b, jk_ppf(sg, prim_kl + q * sg.pst_kl), ac);
            for (int u = ci; u < 3 * NR; u += T) {
                const int r = u / 3, d = u - 3 * r;
                float s, w;
                rys_root_one_f<NR>(reinterpret_cast<const float*>(tab), pr.x, r, s, w);
                jk_unit_f<C, S::SI, S::SJ, false>(pr, s, w, d, (float)norm, dij, dklv, g + u * S::GS);
            }
        } else {
            JKPP b;
            if (p) {
                b = jk_bra_pp(bprim + (size_t)p * pst_ij * 8);
            } else {
                const double2 u = rec[6 * el], v = rec[6 * el + 1], w = rec[6 * el + 2];
                b = JKPP{u.x, u.y, v.x, {v.y, w.x, w.y}};
            }
            const JKPrim pr = jk_prim2(b, jk_pp(sg, prim_kl + q * sg.pst_kl));
            for (int u = ci; u < 3 * NR; u += T) {
                const int r = u / 3, d = u - 3 * r;
                double s, w;
                if constexpr (S::SMEM_TAB) rys_root_one<NR>(tab, pr.x, r, s, w);
                else rys_root<NR>(tab, pr.x, r, s, w);
                jk_unit<C, R, S::SI, S::SJ, false>(pr, s, w, d, norm, ri, rj, rk, rl, g + u * S::GS);
            }
        }
    }

    // rows H[ix][j][.] of one axis and root -> X[j][k][l] in registers
    __device__ __forceinline__ void rows(const R* h, R dklv, R* X) const {
#pragma unroll
        for (int j = 0; j <= C::LJ; j++) {
            R B[MM + 1];
#pragma unroll
            for (int m = 0; m <= MM; m++) B[m] = h[j * S::SJ + m];
#pragma unroll
            for (int l = 0; l <= C::LL; l++) {
#pragma unroll
                for (int k = 0; k <= C::LK; k++) X[(j * (C::LK + 1) + k) * (C::LL + 1) + l] = B[k];
#pragma unroll
                for (int c = 0; c + l + 1 <= MM; c++) B[c] = B[c + 1] + dklv * B[c];
            }
        }
    }

    __device__ __forceinline__ void products(R* acc) const {
        const R d0 = (R)(rk[0] - rl[0]), d1 = (R)(rk[1] - rl[1]), d2 = (R)(rk[2] - rl[2]);
#pragma unroll
        for (int r = 0; r < NR; r++) {
            constexpr int NX = (C::LJ + 1) * (C::LK + 1) * (C::LL + 1);
            R X[NX], Y[NX], Z[NX];
            rows(g + (3 * r) * S::GS + ox, d0, X);
            rows(g + (3 * r + 1) * S::GS + oy, d1, Y);
            rows(g + (3 * r + 2) * S::GS + oz, d2, Z);
#define AT(f, j, k, l) ((f(C::LJ, j) * (C::LK + 1) + f(C::LK, k)) * (C::LL + 1) + f(C::LL, l))
#pragma unroll
            for (int j = 0; j < NFJ; j++)
#pragma unroll
                for (int k = 0; k < NFK; k++)
#pragma unroll
                    for (int l = 0; l < NFL; l++)
                        acc[(j * NFK + k) * NFL + l] +=
                            X[AT(cart_lx, j, k, l)] * Y[AT(cart_ly, j, k, l)] * Z[AT(cart_lz, j, k, l)];
#undef AT
        }
    }

    // adds the lane's kept sums of density m
    __device__ __forceinline__ void flush(int m) {
        if (dk && mine) {
            double* row = krow(m, i0 + ci);
#pragma unroll
            for (int k = 0; k < NFK; k++) atomicAdd(row + kcol(k0 + k), kik[k]);
#pragma unroll
            for (int l = 0; l < NFL; l++) atomicAdd(row + kcol(l0 + l), kil[l]);
        }
        if (dj) {  // J_kl: sum over the team
            __syncwarp();
            if (team < TPW) {
#pragma unroll
                for (int e = 0; e < NKET; e++) part[ci * S::PS + e] = jkl[e];
            }
            __syncwarp();
            if (mine)
                for (int e = ci; e < NKET; e += T) {
                    double v = 0.;
#pragma unroll
                    for (int t = 0; t < T; t++) v += part[t * S::PS + e];
                    if (sg.jp) atomicAdd(sg.jp + sg.pk_kl + m * sg.pk_stride + (size_t)e * sg.pst_kl + col, v);
                    else atomicAdd(sg.vj + (size_t)m * nao * nao + (k0 + e / NFL) + (size_t)nao * (l0 + e % NFL), v);
                }
            __syncwarp();
        }
    }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int k = 0; k < NFK; k++) kik[k] = 0.;
#pragma unroll
        for (int l = 0; l < NFL; l++) kil[l] = 0.;
#pragma unroll
        for (int e = 0; e < NKET; e++) jkl[e] = 0.;
    }

    __device__ __forceinline__ void digest(const R* acc, int entry) {
#define A1(j, k, l) ((double)acc[((j) * NFK + (k)) * NFL + (l)])
        for (int m = 0; m < ndm; m++) {
            if (dj) {
                double v[NFJ];
#pragma unroll
                for (int j = 0; j < NFJ; j++) v[j] = 0.;
                if (active) {
#pragma unroll
                    for (int e = 0; e < NKET; e++) {
                        const double d = dkl(m, e);
#pragma unroll
                        for (int j = 0; j < NFJ; j++) v[j] += A1(j, e / NFL, e % NFL) * d;
                    }
#pragma unroll
                    for (int j = 0; j < NFJ; j++) {
                        const double d = dpb ? __ldg(dpb + m * sg.pk_stride + (size_t)entry * NV + ci * NFJ + j)
                                             : __ldg(drow(m, j0 + j) + i0 + ci);
#pragma unroll
                        for (int e = 0; e < NKET; e++) jkl[e] += A1(j, e / NFL, e % NFL) * d;
                    }
                }
                // J_ij: lane ci of every team holds row ci; sum over the teams
#pragma unroll
                for (int j = 0; j < NFJ; j++) {
                    double t = v[j];
#pragma unroll
                    for (int x = 1; x < TPW; x++) t += __shfl_down_sync(0xffffffffu, v[j], x * T);
                    if (team == 0) {
                        if (jpb) atomicAdd(jpb + m * sg.pk_stride + (size_t)entry * NV + ci * NFJ + j, t);
                        else atomicAdd(sg.vj + (size_t)m * nao * nao + (i0 + ci) + (size_t)nao * (j0 + j), t);
                    }
                }
            }
            if (dk) {
                if (active) {
                    const double* irow = drow(m, i0 + ci);
                    double pj[NJK];
#pragma unroll
                    for (int e = 0; e < NJK; e++) pj[e] = 0.;
#pragma unroll
                    for (int l = 0; l < NFL; l++) {
                        const double d = __ldg(irow + l0 + l);
#pragma unroll
                        for (int e = 0; e < NJK; e++) pj[e] += A1(e / NFK, e % NFK, l) * d;
                    }
#pragma unroll
                    for (int e = 0; e < NJK; e++) part[ci * S::PS + e] = pj[e];
                    double pl[NJL];
#pragma unroll
                    for (int e = 0; e < NJL; e++) pl[e] = 0.;
#pragma unroll
                    for (int k = 0; k < NFK; k++) {
                        const double d = __ldg(irow + k0 + k);
#pragma unroll
                        for (int e = 0; e < NJL; e++) pl[e] += A1(e / NFL, k, e % NFL) * d;
                    }
#pragma unroll
                    for (int e = 0; e < NJL; e++) part[ci * S::PS + NJK + e] = pl[e];
#pragma unroll
                    for (int j = 0; j < NFJ; j++) {
                        const double* row = drow(m, j0 + j);
#pragma unroll
                        for (int l = 0; l < NFL; l++) {
                            const double d = __ldg(row + l0 + l);
#pragma unroll
                            for (int k = 0; k < NFK; k++) kik[k] += A1(j, k, l) * d;
                        }
#pragma unroll
                        for (int k = 0; k < NFK; k++) {
                            const double d = __ldg(row + k0 + k);
#pragma unroll
                            for (int l = 0; l < NFL; l++) kil[l] += A1(j, k, l) * d;
                        }
                    }
                }
                __syncwarp();
                if (active)
                    for (int e = ci; e < S::NJ; e += T) {
                        double v = 0.;
#pragma unroll
                        for (int t = 0; t < T; t++) v += part[t * S::PS + e];
                        const int x = e - NJK;
                        if (e < NJK) atomicAdd(krow(m, j0 + e / NFK) + kcol(k0 + e % NFK), v);
                        else atomicAdd(krow(m, j0 + x / NFL) + kcol(l0 + x % NFL), v);
                    }
                __syncwarp();
            }
            if constexpr (MULTI) {
                mine = active;
                flush(m);
                clear();
            }
        }
#undef A1
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
            sg.elo ? jk_item_base(__reduce_min_sync(0xffffffffu, elo < ehi ? elo : 0x7fffffff), sg.bucket, TPW) : 0;
        team = lane / T;
        ci = team < TPW ? lane - team * T : 0;
        const int mycol = team < TPW ? base + TPW * (int)(item - __ldg(sg.ioff + run)) + team : -1;
        // Schwarz ranks of the item's ket pairs
        const bool in = mycol >= 0 && mycol < sg.pst_kl;
        const int rank = in ? __ldg(sg.rank + sg.pair_kl0 + mycol) : -1;
        const int rmin = __reduce_min_sync(0xffffffffu, in ? rank : 0x7fffffff),
                  rmax = __reduce_max_sync(0xffffffffu, rank);
        unsigned mask = __ballot_sync(0xffffffffu, elo < ehi && elo <= rmax && ehi > rmin);
        if (mask == 0) return;
        const int ent0 = __shfl_sync(0xffffffffu, ent, 0);
        pst_ij = sg.pst_ij;
        col = max(0, min(mycol, sg.pst_kl - 1));
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
        ox = cart_lx(C::LI, ci) * S::SI;
        oy = cart_ly(C::LI, ci) * S::SI;
        oz = cart_lz(C::LI, ci) * S::SI;
        prim_kl = sg.prim_kl0 + col;
        npkl = sg.pnp ? __ldg(sg.pnp + bkl) : sg.nprim_kl;
        const int qmax = __reduce_max_sync(0xffffffffu, npkl);
        ndm = MULTI ? sg.n_dm : 1;
        clear();
        const int diag = sg.pair_ij0 == sg.pair_kl0 ? mycol : -1;
        const double* bprim0 = sg.bprim + (size_t)e0 * 8;
        const float* bprimf0 = sg.bprimf + (size_t)e0 * 8;
        __syncwarp();
        if ((mask >> lane) & 1) {  // stage the run
            double2* r = rec + 6 * lane;
            if constexpr (S::F32P) {
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
        __syncwarp();
        bool used = false;
        while (mask) {
            el = __ffs(mask) - 1;
            mask &= mask - 1;
            const int4 bound = *reinterpret_cast<const int4*>(rec + 6 * el + 5);
            const double2 pa = rec[6 * el + 3], pb = rec[6 * el + 4];
            active = rank >= bound.x && rank < bound.y;
            used |= active;
            rj[0] = pa.x;
            rj[1] = pa.y;
            rj[2] = pb.x;
            j0 = __double2loint(pb.y);
            npij = __double2hiint(pb.y);
            bprimf = bprimf0 + el * 8;
            bprim = bprim0 + el * 8;
            norm = bound.z == diag ? 0.5 * JK_FAC : JK_FAC;
            R acc[C::NACC];
#pragma unroll
            for (int e = 0; e < C::NACC; e++) acc[e] = R(0);
            for (int q = 0; q < qmax; q++)
                for (int p = 0; p < npij; p++) {
                    const bool on = active && q < npkl;
                    if (on) build(p, q);
                    __syncwarp();
                    if (on) products(acc);
                    __syncwarp();
                }
            digest(acc, e0 + el);
        }
        if constexpr (!MULTI) {
            mine = used;
            flush(0);
        }
    }
};

// segt, queue and grab as in jk_run_kernel; warps work on their own items
template <class C, typename R, bool MULTI, bool KROWS>
__global__ void __launch_bounds__(JK_RUN_THREADS, 2)
    jk_trun_kernel(const JKSeg* __restrict__ segs, const long long* __restrict__ segt, int nseg,
                   unsigned long long* queue, int grab) {
    extern __shared__ __align__(16) double jk_tab[];
    __shared__ JKSeg s_seg[JK_RUN_THREADS / 32];
    using S = JKTRunShape<C, R>;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long total = segt[nseg];
    if (!queue && (long long)blockIdx.x * (JK_RUN_THREADS / 32) >= total) return;  // block-uniform
    if (total == 0) return;
    const double* rys = segs[0].rys;
    if constexpr (S::F32P) rys_table_copy_f<C::NROOTS>(rys, reinterpret_cast<float*>(jk_tab));
    else if constexpr (S::SMEM_TAB) rys_table_copy<C::NROOTS>(rys, jk_tab);
    __syncthreads();
    double* mem = jk_tab + (S::TAB + warp * S::WARP) / sizeof(double);
    const int team = min(lane / C::T, C::TPW - 1);
    double* reg = mem + 32 * 12 + (size_t)team * S::WORDS;
    JKTRunItem<C, R, MULTI, KROWS> w{s_seg[warp], S::SMEM_TAB ? jk_tab : rys, reinterpret_cast<R*>(reg), reg,
                              reinterpret_cast<double2*>(mem)};
    jk_run_items(segs, segt, nseg, total, queue, grab, s_seg[warp], w);
}
