// C-ABI of the J/K engine (declared in include/byteqc_jk.h): basis setup with
// device-side Schwarz screening, the per-call density screen and quartet
// enumeration on the device, the class launches, and the AO transforms.
#include <cublas_v2.h>
#include <math.h>
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <memory>
#include <mutex>
#include <numeric>
#include <string>
#include <vector>

#include "../../include/byteqc_jk.h"
#include "jk_launch.cuh"
#include "jk_internal.h"
#include "jk_pair.cuh"

static int class_index(const jk_basis* b, int cp_ij, int cp_kl);
static int make_plan(jk_basis* b, int nshards, int shard, JKPlan** out);

// primitive-pair screen of the run kernels: exp(-mu r^2) below exp(-60)
// (the default exponent cutoff of libcint's pair data) contributes nothing
#define JK_PRIM_EXPCUT 60.0

// ---------------------------------------------------------------------------
// errors
// ---------------------------------------------------------------------------
static thread_local std::string g_err;

static int set_err(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_err = buf;
    return code;
}

#define CUDA_TRY(x)                                                                               \
    do {                                                                                          \
        cudaError_t e_ = (x);                                                                     \
        if (e_ != cudaSuccess) {                                                                  \
            cudaGetLastError(); /* the check after the next call's launches would find it */      \
            return set_err(JK_ERR_CUDA, "%s: %s", #x, cudaGetErrorString(e_));                    \
        }                                                                                         \
    } while (0)

extern "C" const char* jk_last_error(void) { return g_err.c_str(); }

// ---------------------------------------------------------------------------
// launcher tables
// ---------------------------------------------------------------------------
static JKTables g_tabs;
#define g_tab64 g_tabs.t64
#define g_tab32 g_tabs.t32
static std::once_flag g_tab_once;
static void init_tables() {
    std::call_once(g_tab_once, [] {
        JK_REGISTER_ALL();
        jk_register_generic(&g_tabs);
    });
}


static double common_fac_sp(int l) {
    return l == 0 ? 0.282094791773878143 : (l == 1 ? 0.488602511902919921 : 1.0);
}

// ---------------------------------------------------------------------------
// Schwarz matrix on the device: q[i,j] = sqrt(max_{a in i, b in j} |(ab|ab)|)
// over the Cartesian functions of the pair (the quantity PySCF's
// CVHFsetnr_direct_scf gives the reference, cuobc/scf/hf.py:341).
// One thread per shell pair, bra shell of the larger l.
// ---------------------------------------------------------------------------
template <int LI, int LJ>
__global__ void jk_qcond_kernel(const int* __restrict__ pi, const int* __restrict__ pj, int npairs,
                                const int* __restrict__ atm, const int* __restrict__ bas,
                                const double* __restrict__ env, int nbas, double* __restrict__ q,
                                const double* __restrict__ rys) {
    using C = JKClass<LI, LJ, LI, LJ>;
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npairs) return;
    int ish = pi[p], jsh = pj[p];
    const double* ri = env + atm[bas[ish * BAS_SLOTS + ATOM_OF] * ATM_SLOTS + PTR_COORD];
    const double* rj = env + atm[bas[jsh * BAS_SLOTS + ATOM_OF] * ATM_SLOTS + PTR_COORD];
    int npi = bas[ish * BAS_SLOTS + NPRIM_OF], npj = bas[jsh * BAS_SLOTS + NPRIM_OF];
    const double* ai = env + bas[ish * BAS_SLOTS + PTR_EXP];
    const double* aj = env + bas[jsh * BAS_SLOTS + PTR_EXP];
    const double* ci = env + bas[ish * BAS_SLOTS + PTR_COEFF];
    const double* cj = env + bas[jsh * BAS_SLOTS + PTR_COEFF];
    double fsp = (LI == 0 ? 0.282094791773878143 : (LI == 1 ? 0.488602511902919921 : 1.0)) *
                 (LJ == 0 ? 0.282094791773878143 : (LJ == 1 ? 0.488602511902919921 : 1.0));
    double r2 = 0;
    for (int d = 0; d < 3; d++) r2 += (ri[d] - rj[d]) * (ri[d] - rj[d]);
    double diag[C::NFI * C::NFJ];
#pragma unroll
    for (int e = 0; e < C::NFI * C::NFJ; e++) diag[e] = 0;
    double r_i[3] = {ri[0], ri[1], ri[2]}, r_j[3] = {rj[0], rj[1], rj[2]};
    for (int ip = 0; ip < npi; ip++)
        for (int jp = 0; jp < npj; jp++) {
            double A = ai[ip] + aj[jp];
            double eij = fsp * ci[ip] * cj[jp] * exp(-r2 * ai[ip] * aj[jp] / A);
            double P[3];
            for (int d = 0; d < 3; d++) P[d] = (ai[ip] * ri[d] + aj[jp] * rj[d]) / A;
            for (int kp = 0; kp < npi; kp++)
                for (int lp = 0; lp < npj; lp++) {
                    double B = ai[kp] + aj[lp];
                    double ekl = fsp * ci[kp] * cj[lp] * exp(-r2 * ai[kp] * aj[lp] / B);
                    JKPrim pr;
                    pr.A = A;
                    pr.B = B;
                    pr.AB = A + B;
                    pr.iA = 1. / A;
                    pr.iB = 1. / B;
                    pr.iAB = 1. / pr.AB;
                    for (int d = 0; d < 3; d++) {
                        pr.P[d] = P[d];
                        pr.Q[d] = (ai[kp] * ri[d] + aj[lp] * rj[d]) / B;
                    }
                    double dx = pr.P[0] - pr.Q[0], dy = pr.P[1] - pr.Q[1], dz = pr.P[2] - pr.Q[2];
                    pr.x = A * B / pr.AB * (dx * dx + dy * dy + dz * dz);
                    pr.sy = eij * ekl / (sqrt(pr.AB) * A * B);
                    for (int r = 0; r < C::NROOTS; r++) {
                        double s, w;
                        rys_root<C::NROOTS>(rys, pr.x, r, s, w);
                        double Ix[C::GS], Iy[C::GS], Iz[C::GS];
                        jk_unit<C, double>(pr, s, w, 0, JK_FAC, r_i, r_j, r_i, r_j, Ix);
                        jk_unit<C, double>(pr, s, w, 1, JK_FAC, r_i, r_j, r_i, r_j, Iy);
                        jk_unit<C, double>(pr, s, w, 2, JK_FAC, r_i, r_j, r_i, r_j, Iz);
#pragma unroll
                        for (int a = 0; a < C::NFI; a++)
#pragma unroll
                            for (int b = 0; b < C::NFJ; b++) {
                                int ox = cart_lx(LI, a) * (C::SI + C::SK) + cart_lx(LJ, b) * (C::SJ + 1);
                                int oy = cart_ly(LI, a) * (C::SI + C::SK) + cart_ly(LJ, b) * (C::SJ + 1);
                                int oz = cart_lz(LI, a) * (C::SI + C::SK) + cart_lz(LJ, b) * (C::SJ + 1);
                                diag[a * C::NFJ + b] += Ix[ox] * Iy[oy] * Iz[oz];
                            }
                    }
                }
        }
    double mx = 0;
#pragma unroll
    for (int e = 0; e < C::NFI * C::NFJ; e++) mx = fmax(mx, fabs(diag[e]));
    double v = sqrt(mx);
    q[(size_t)ish * nbas + jsh] = v;
    q[(size_t)jsh * nbas + ish] = v;
}

// Schwarz diagonal of pairs with a shell above f (jk_generic.cu); lmax is
// the larger l of the pairs in the list
void jk_qcond_generic(const int* pi, const int* pj, int n, const int* atm, const int* bas, const double* env,
                      int nbas, double* q, const double* rys, int lmax, cudaStream_t st);

typedef void (*qcond_fn)(const int*, const int*, int, const int*, const int*, const double*, int, double*,
                         const double*, cudaStream_t);
template <int LI, int LJ>
static void qcond_launch(const int* pi, const int* pj, int n, const int* atm, const int* bas, const double* env,
                         int nbas, double* q, const double* rys, cudaStream_t st) {
    if (n > 0) jk_qcond_kernel<LI, LJ><<<(n + 63) / 64, 64, 0, st>>>(pi, pj, n, atm, bas, env, nbas, q, rys);
}
static qcond_fn g_qcond[4][4] = {
    {qcond_launch<0, 0>, nullptr, nullptr, nullptr},
    {qcond_launch<1, 0>, qcond_launch<1, 1>, nullptr, nullptr},
    {qcond_launch<2, 0>, qcond_launch<2, 1>, qcond_launch<2, 2>, nullptr},
    {qcond_launch<3, 0>, qcond_launch<3, 1>, qcond_launch<3, 2>, qcond_launch<3, 3>},
};

// ---------------------------------------------------------------------------
// per-call kernels: density condensation and quartet screening
// ---------------------------------------------------------------------------
// dm_cond[gi, gj] = max over the dms of max |D[p, q]|, p in group gi, q in gj
// (lib.condense('absmax') over the group AO boundaries, cuobc/scf/hf.py:104-107),
// of one molecule (one) or many (tab, blockIdx.z).  A warp per row of D, the
// rows of a group spread over gridDim.x blocks that meet in an atomic maximum
// of the bit patterns (ordered as the non-negative values): one block per
// group pair, as this kernel had, took 3.2 ms of the 220 ms build of (H2O)64 /
// cc-pVDZ (5248 functions in 3 groups).  out starts at zero.
#define JK_DMC_GROUPS 256
__global__ void __launch_bounds__(256) jk_dm_cond_kernel(const JKDmCond one, const JKDmCond* __restrict__ tab) {
    const JKDmCond m = tab ? tab[blockIdx.z] : one;
    const int gi = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (gi >= m.ngroups) return;
    __shared__ unsigned long long smax[JK_DMC_GROUPS];
    const bool sh = m.ngroups <= JK_DMC_GROUPS;
    unsigned long long* gout = reinterpret_cast<unsigned long long*>(m.out) + (size_t)gi * m.ngroups;
    if (sh)
        for (int g = threadIdx.x; g < m.ngroups; g += blockDim.x) smax[g] = 0;
    __syncthreads();
    const int p0 = m.gao[gi], np = m.gao[gi + 1] - p0;
    const long long rows = (long long)np * m.n_dm;
    for (long long r = (long long)blockIdx.x * 8 + warp; r < rows; r += (long long)gridDim.x * 8) {
        const int idm = (int)(r / np), p = p0 + (int)(r - (long long)idm * np);
        const double* row = m.dm + ((size_t)idm * m.nao + p) * m.nao;
        for (int g = 0; g < m.ngroups; g++) {
            double mx = 0;
            for (int q = m.gao[g] + lane; q < m.gao[g + 1]; q += 32) mx = fmax(mx, fabs(row[q]));
            for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            if (lane == 0)
                atomicMax(sh ? smax + g : gout + g, (unsigned long long)__double_as_longlong(mx));
        }
    }
    if (!sh) return;
    __syncthreads();
    for (int g = threadIdx.x; g < m.ngroups; g += blockDim.x)
        if (smax[g]) atomicMax(gout + g, smax[g]);
}

// clears every molecule's counters and condensed density (blockIdx.x = molecule)
__global__ void jk_zero_kernel(const JKDmCond* __restrict__ tab) {
    const JKDmCond m = tab[blockIdx.x];
    for (int e = threadIdx.x; e < m.nzero; e += blockDim.x) m.zero[e] = 0;
}

// max over the six group pairs of a class quartet of the condensed density
__device__ __forceinline__ double jk_cq_sub(const double* c, int ngroups, int gi, int gj, int gk, int gl) {
    return fmax(fmax(fmax(c[gi * ngroups + gj], c[gk * ngroups + gl]), fmax(c[gi * ngroups + gk], c[gj * ngroups + gk])),
                fmax(c[gi * ngroups + gl], c[gj * ngroups + gl]));
}

// Screening of one class quartet, with the reference's decision per
// contracted quartet (cuobc/scf/hf.py:136-145, 567-578 and
// cuobc/lib/gvhf/nr_jk_driver.cu:252-280):
//   skip the class quartet if prescreen and max(dm_cond over its 6 group
//   pairs) < tol; else with scale = nbins / log(min(tol/sub, 0.1)) and
//   s = floor(scale * log_q), keep (ij, kl) iff s_ij + s_kl < nbins (and
//   kl <= ij inside a diagonal class quartet).
// Because log_q is sorted descending inside a class, the kept kl of a row
// form a prefix; its length is found by binary search.  Mixed precision
// (fp32_cutoff > 0): the kept prefix of a row splits again at the bound
// q_ij q_kl sub = fp32_cutoff (unclipped log q); the leading part (larger
// bounds) runs in FP64, the tail in FP32.
struct JKScreen {
    bool skip, mixed, diag;
    double scale, log_thr;
    int nbins;
    __device__ __forceinline__ JKScreen(const JKScreenCQ& cq, double tol, int nb, int prescreen, double fp32_cutoff) {
        const double sub = jk_cq_sub(cq.dm_cond, cq.ngroups, cq.gi, cq.gj, cq.gk, cq.gl);
        skip = prescreen && sub < tol;
        nbins = nb;
        scale = nb / log(fmin(tol / sub, 0.1));
        mixed = fp32_cutoff > 0;
        log_thr = mixed ? log(fp32_cutoff / sub) : 0.;  // q_ij q_kl >= fp32_cutoff / sub
        diag = cq.cp_ij == cq.cp_kl;
    }
    // kept kets of row ij: [0, c64) in FP64, [c64, cnt) in FP32
    __device__ __forceinline__ void row(const JKScreenCQ& cq, int ij, int& c64, int& cnt) const {
        c64 = cnt = 0;
        if (skip) return;
        const int sij = (int)floor(scale * cq.lq_ij[ij]);
        if (sij >= nbins) return;
        const int b = nbins - sij;
        // count kl with floor(scale * lq_kl) < b (non-decreasing in kl)
        int lo = 0, hi = cq.n_kl;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if ((int)floor(scale * cq.lq_kl[mid]) < b) lo = mid + 1; else hi = mid;
        }
        cnt = lo;
        if (diag && cnt > ij + 1) cnt = ij + 1;
        c64 = cnt;
        if (mixed && cnt > 0) {
            // kl with rq_ij + rq_kl >= log_thr (non-increasing in kl)
            const double need = log_thr - cq.rq_ij[ij];
            lo = 0;
            hi = cnt;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (cq.rq_kl[mid] >= need) lo = mid + 1; else hi = mid;
            }
            c64 = lo;
        }
    }
};

// Row classes (team and generic kernels): one block of 256 threads.  qoff counts the FP64 part, qoff32 the FP32 part, whose first
// column per row is klb[ij].
__device__ __forceinline__ void jk_screen_rows(const JKScreenCQ& cq, const JKScreen& sc) {
    __shared__ long long carry, carry32;
    __shared__ long long wsum[32], wsum32[32];
    if (threadIdx.x == 0) {
        carry = carry32 = 0;
        cq.qoff[0] = 0;
        cq.qoff32[0] = 0;
    }
    __syncthreads();
    for (int base = 0; base < cq.n_ij; base += blockDim.x) {
        const int ij = base + threadIdx.x;
        int cnt = 0, c64 = 0;
        if (ij < cq.n_ij) {
            sc.row(cq, ij, c64, cnt);
            cq.klb[ij] = c64;
        }
        long long i64, i32;
        jk_block_scan2(c64, cnt - c64, i64, i32, wsum, wsum32, carry, carry32);
        if (ij < cq.n_ij) {
            cq.qoff[ij + 1] = i64;
            cq.qoff32[ij + 1] = i32;
        }
    }
    if (threadIdx.x == 0) {
        cq.task0[0] = 0;
        cq.task0[1] = carry;
        cq.task032[0] = 0;
        cq.task032[1] = carry32;
    }
}

// Screening of a build, blockIdx.x = class quartet.  Row classes: the first
// block, as above.  Run classes: a warp per run, a lane per entry.
// Writes the entries' bounds, adds up the quartet counts and leaves the
// items of each run in ioff / ioff32 (made a prefix by jk_run_scan_kernel).
__global__ void __launch_bounds__(256) jk_screen_kernel(const JKScreenCQ* __restrict__ cqs, double tol, int nbins,
                                                            int prescreen, double fp32_cutoff) {
    const JKScreenCQ cq = cqs[blockIdx.x];
    if (cq.runs ? (int)(blockIdx.y * 8) >= cq.nrun : blockIdx.y > 0) return;  // block-uniform
    const JKScreen sc(cq, tol, nbins, prescreen, fp32_cutoff);
    if (!cq.runs) {
        jk_screen_rows(cq, sc);
        return;
    }
    const int lane = threadIdx.x & 31;
    long long n64 = 0, n32 = 0;
    for (int run = blockIdx.y * 8 + (threadIdx.x >> 5); run < cq.nrun; run += gridDim.y * 8) {
        const int e0 = cq.run0[run], ne = cq.run0[run + 1] - e0;
        int c64 = 0, cnt = 0;
        if (lane < ne) {
            sc.row(cq, cq.erank[e0 + lane], c64, cnt);
            cq.klb[e0 + lane] = c64;
            cq.kle[e0 + lane] = cnt;
        }
        n64 += c64;
        n32 += cnt - c64;
        const int h64 = __reduce_max_sync(0xffffffffu, c64);
        const int l32 = jk_item_base(__reduce_min_sync(0xffffffffu, c64 < cnt ? c64 : 0x7fffffff), cq.bucket, cq.runs);
        const int h32 = __reduce_max_sync(0xffffffffu, c64 < cnt ? cnt : 0);
        if (lane == 0) {
            cq.ioff[run] = (jk_bucket_end(h64, cq.bucket, cq.n_kl) + cq.runs - 1) / cq.runs;
            cq.ioff32[run] = h32 > 0 ? (jk_bucket_end(h32, cq.bucket, cq.n_kl) - l32 + cq.runs - 1) / cq.runs : 0;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        n64 += __shfl_xor_sync(0xffffffffu, n64, o);
        n32 += __shfl_xor_sync(0xffffffffu, n32, o);
    }
    if (lane == 0 && (n64 | n32)) {
        atomicAdd((unsigned long long*)cq.task0 + 1, (unsigned long long)n64);
        atomicAdd((unsigned long long*)cq.task032 + 1, (unsigned long long)n32);
    }
}

// items per run -> exclusive prefix in place, totals to tot[1] (one block)
__device__ __forceinline__ void jk_run_scan_body(int nrun, long long* ioff, long long* ioff32, long long* tot,
                                                 long long* tot32) {
    __shared__ long long carry, carry32;
    __shared__ long long wsum[32], wsum32[32];
    if (threadIdx.x == 0) carry = carry32 = 0;
    __syncthreads();
    for (int base = 0; base < nrun; base += blockDim.x) {
        const int r = base + threadIdx.x;
        const long long a = r < nrun ? ioff[r] : 0, b = r < nrun && ioff32 ? ioff32[r] : 0;
        long long ia, ib;
        jk_block_scan2(a, b, ia, ib, wsum, wsum32, carry, carry32);
        if (r < nrun) {
            ioff[r] = ia - a;
            if (ioff32) ioff32[r] = ib - b;
        }
    }
    if (threadIdx.x == 0) {
        tot[0] = 0;
        tot[1] = carry;
        if (tot32) {
            tot32[0] = 0;
            tot32[1] = carry32;
        }
    }
}
__global__ void __launch_bounds__(1024) jk_run_scan_kernel(const JKScreenCQ* __restrict__ cqs) {
    const JKScreenCQ cq = cqs[blockIdx.x];
    if (cq.runs) jk_run_scan_body(cq.nrun, cq.ioff, cq.ioff32, cq.itm, cq.itm32);
}

// per-class-pair entries: items of each run from the entries' ket ends
__global__ void jk_run_items_kernel(const __grid_constant__ JKSeg sg, int chunk, long long* __restrict__ ioff) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < sg.nrun; r += gridDim.x * blockDim.x) {
        int h = 0;
        for (int e = sg.run0[r]; e < sg.run0[r + 1]; e++) h = max(h, sg.ehi[e]);
        ioff[r] = (jk_bucket_end(h, sg.bucket, sg.pst_kl) + chunk - 1) / chunk;
    }
}
__global__ void __launch_bounds__(1024) jk_run_scan1_kernel(const __grid_constant__ JKSeg sg, long long* ioff,
                                                            long long* itm, JKSeg* dst) {
    jk_seg_copy(sg, dst);
    jk_run_scan_body(sg.nrun, ioff, nullptr, itm, nullptr);
}

// last index i in [0, n] with off[i] <= t (off non-decreasing, off[0] <= t)
__device__ __forceinline__ int jk_slot(const int* __restrict__ off, int n, int t) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(off + mid) <= t) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// What follows of the uploaded lists per pair (set-up, one thread per pair): the
// geometry, the inverses of the two orders, the entries' ranks and the log q
// clipped at 0.  Uploaded, these were two thirds of the bytes of a set-up.
__global__ void __launch_bounds__(256) jk_pair_tables_kernel(int npair, int ncp, const int* __restrict__ locs,
                                                             const int* __restrict__ bra, const int* __restrict__ ket,
                                                             const int* __restrict__ rank, const int* __restrict__ ent,
                                                             const double* __restrict__ bx, int nbas,
                                                             const int* __restrict__ ao_loc,
                                                             const double* __restrict__ raw, double* __restrict__ lq,
                                                             double* __restrict__ geo, int* __restrict__ pao,
                                                             int* __restrict__ pos, int* __restrict__ inv,
                                                             int* __restrict__ erank) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npair) return;
    const int p0 = __ldg(locs + jk_slot(locs, ncp, p)), x = p - p0, e = ent[p];
    pos[p0 + rank[p]] = x;
    inv[p0 + e] = x;
    erank[p] = rank[p0 + e];
    lq[p] = raw[p] > 0. ? 0. : raw[p];
    const int sh[2] = {bra[p], ket[p]};
    for (int a = 0; a < 2; a++) {
        for (int d = 0; d < 3; d++) geo[(size_t)(3 * a + d) * npair + p] = bx[(size_t)d * nbas + sh[a]];
        pao[(size_t)a * npair + p] = ao_loc[sh[a]];
    }
}

// ... and per primitive pair: 1 / a12, the single-precision copy, and the bra
// records of the run kernels (JKSeg::bprim, bprimf, bpair), gathered in
// run-entry order.  prim: a12 | e12 | x12 | y12 | z12 | 1 / a12, stride n; primitive
// k of position r of class c at plocs[c] + k * (pairs of c) + r.
__global__ void __launch_bounds__(256) jk_prim_tables_kernel(int n, int npair, int ncp, const int* __restrict__ locs,
                                                             const int* __restrict__ plocs, double* __restrict__ prim,
                                                             float* __restrict__ primf, const int* __restrict__ inv,
                                                             const double* __restrict__ geo,
                                                             const int* __restrict__ pao, const int* __restrict__ pnp,
                                                             double* __restrict__ bprim, float* __restrict__ bprimf,
                                                             double* __restrict__ bpair) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const size_t N = n;
    const int c = jk_slot(plocs, ncp, t), q0 = __ldg(plocs + c), p0 = __ldg(locs + c), np = __ldg(locs + c + 1) - p0;
    const int k = (t - q0) / np, p = p0 + (t - q0) - k * np, e = inv[p];
    const double a = prim[t], ia = 1. / a, e12 = prim[N + t];
    prim[5 * N + t] = ia;
    double* d = bprim + ((size_t)q0 + (size_t)k * np + e) * 8;
    float* g = bprimf + ((size_t)q0 + (size_t)k * np + e) * 8;
    d[0] = a;
    d[1] = ia;
    d[2] = e12 * ia;
    primf[t] = g[0] = (float)a;
    primf[N + t] = g[1] = (float)ia;
    primf[2 * N + t] = g[2] = (float)(e12 / a);
    for (int x = 0; x < 3; x++) {
        // the product centre; single precision keeps it relative to the bra
        // shell's, so that the small differences P - R_i keep their precision
        const double P = prim[(2 + x) * N + t];
        d[3 + x] = P;
        primf[(3 + x) * N + t] = g[3 + x] = (float)(P - geo[(size_t)x * npair + p]);
    }
    d[6] = d[7] = 0.;
    g[6] = g[7] = 0.f;
    if (k == 0) {
        double* b = bpair + ((size_t)p0 + e) * 4;
        for (int x = 0; x < 3; x++) b[x] = geo[(size_t)(3 + x) * npair + p];
        b[3] = __hiloint2double(pnp[p], pao[(size_t)npair + p]);
    }
}

// the call's buffers into the segments of a plan
struct JKCall {
    const double* dm;
    double *vj, *vk;
    const double* dp;
    double* jp;
    const double* dpb;
    double* jpb;
    int n_dm;
    double* kt;     // K of the run kernels (JKPackMol::kt), or null: they add into vk
    long long nkt;  // its size
};
// Pair-packed J side.  mode 0: gather the density blocks of every pair into
// dp (element c of pair p of class k at off_k + c*np_k + p, one copy per
// density) and into dpb (entry-major: element c of entry e at off_k +
// e*ncomp_k + c; inv gives a pair's entry); mode 1: add the packed J
// accumulators jp and jpb into vj.  Every (pair, component) is a distinct
// element of D and of vj.
__device__ __forceinline__ void jk_pack_body(const JKPackMol& a, int mode) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < a.total;
         t += (long long)gridDim.x * blockDim.x) {
        int lo = 0, hi = a.ncls - 1;
        while (lo < hi) {
            int mid = (lo + hi + 1) >> 1;
            if (a.cls[mid].off <= t) lo = mid; else hi = mid - 1;
        }
        const JKPackCls k = a.cls[lo];
        const long long local = t - k.off;
        const int comp = (int)(local / k.np), p = (int)(local - (long long)comp * k.np);
        const int x = comp / k.nfj, y = comp - x * k.nfj;
        const int pair = k.pair0 + p;
        const long long tb = k.off + (long long)a.inv[pair] * (k.nfi * k.nfj) + comp;
        const size_t e = (size_t)(a.ao_loc[a.pair2bra[pair]] + x) + (size_t)a.nao * (a.ao_loc[a.pair2ket[pair]] + y);
        for (int m = 0; m < a.n_dm; m++) {
            const size_t mo = (size_t)m * a.nao * a.nao;
            if (mode == 0) {
                const double v = a.dm[mo + e];
                a.dp[m * a.total + t] = v;
                a.dpb[m * a.total + tb] = v;
            } else {
                a.vj[mo + e] += a.jp[m * a.total + t] + a.jpb[m * a.total + tb];
            }
        }
    }
}

// vk[a + nao b] += kt[a nao + b], 32 x 32 tiles through shared memory (256
// threads); atomics, since builds of other handles may add into the same vk
__device__ __forceinline__ void jk_kadd_body(const JKPackMol& a) {
    __shared__ double t[32][33];
    const int n = a.nao, nt = (n + 31) / 32, x = threadIdx.x & 31, y0 = threadIdx.x >> 5;
    const long long tiles = (long long)a.n_dm * nt * nt;
    for (long long b = blockIdx.x; b < tiles; b += gridDim.x) {
        const int m = (int)(b / ((long long)nt * nt)), r = (int)(b - (long long)m * nt * nt);
        const int p0 = r / nt * 32, q0 = r % nt * 32;
        const size_t mo = (size_t)m * n * n;
        for (int y = y0; y < 32; y += 8)
            if (p0 + y < n && q0 + x < n) t[y][x] = a.kt[mo + (size_t)(p0 + y) * n + q0 + x];
        __syncthreads();
        for (int y = y0; y < 32; y += 8)
            if (q0 + y < n && p0 + x < n) atomicAdd(a.vk + mo + (size_t)(q0 + y) * n + p0 + x, t[x][y]);
        __syncthreads();
    }
}

// end of a build: the J accumulators (total > 0) and kt (if any) to the outputs
__global__ void __launch_bounds__(256) jk_finish_kernel(const JKPackMol one) {
    if (one.total > 0) jk_pack_body(one, 1);
    if (one.kt) jk_kadd_body(one);
}

// Start of a build, one launch: the call's buffers into the segments, the
// counters and the J accumulators cleared, the densities packed.
__global__ void __launch_bounds__(256) jk_begin_kernel(JKSeg* __restrict__ s64, JKSeg* __restrict__ s32, int nseg,
                                                       const JKCall c, unsigned long long* __restrict__ zero,
                                                       long long nzero, const JKPackMol pm) {
    const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
    for (long long i = t0; i < 2 * nseg; i += step) {
        JKSeg& s = i < nseg ? s64[i] : s32[i - nseg];
        s.dm = c.dm;
        s.vj = c.vj;
        s.vk = c.kt && s.nrun > 0 ? c.kt : c.vk;
        s.dp = c.dp;
        s.jp = c.jp;
        s.dpb = c.dpb;
        s.jpb = c.jpb;
        s.n_dm = c.n_dm;
    }
    for (long long i = t0; i < nzero; i += step) zero[i] = 0;
    for (long long i = t0; i < c.nkt; i += step) c.kt[i] = 0.;
    if (pm.total > 0) {
        const long long na = 2 * pm.n_dm * pm.total;  // jp and jpb lie together
        for (long long i = t0; i < na; i += step) pm.jp[i] = 0.;
        jk_pack_body(pm, 0);
    }
}

// one molecule per blockIdx.y
__global__ void __launch_bounds__(256) jk_pack_batch_kernel(const JKPackMol* __restrict__ mols, int mode) {
    const JKPackMol m = mols[blockIdx.y];
    if (m.total > 0) jk_pack_body(m, mode);
    if (mode == 1 && m.kt) jk_kadd_body(m);
}

// 2 (V + V^T) of the first nj matrices (J), V + V^T of the others (K), where
// V[i, j] = mem[i + nao j]; out_rm[p, q] = fac (mem[p nao + q] + mem[q nao + p]).
// 32 x 32 tiles, the transposed one through shared memory, so that both reads
// and the write are whole rows (the element-wise kernel before read a column
// per warp).
__global__ void __launch_bounds__(256) jk_symmetrize_kernel(const double* __restrict__ in, double* __restrict__ out,
                                                            int nao, int nmat, int nj) {
    __shared__ double t[32][33];
    const int nt = (nao + 31) / 32, x = threadIdx.x & 31, y0 = threadIdx.x >> 5;
    const long long tiles = (long long)nmat * nt * nt;
    for (long long b = blockIdx.x; b < tiles; b += gridDim.x) {
        const int m = (int)(b / ((long long)nt * nt)), r = (int)(b - (long long)m * nt * nt);
        const int p0 = r / nt * 32, q0 = r % nt * 32;
        const double* v = in + (size_t)m * nao * nao;
        const double fac = m < nj ? 2. : 1.;
        for (int y = y0; y < 32; y += 8)
            if (q0 + y < nao && p0 + x < nao) t[y][x] = v[(size_t)(q0 + y) * nao + p0 + x];
        __syncthreads();
        for (int y = y0; y < 32; y += 8)
            if (p0 + y < nao && q0 + x < nao) {
                const size_t e = (size_t)(p0 + y) * nao + q0 + x;
                out[(size_t)m * nao * nao + e] = fac * (v[e] + t[x][y]);
            }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// basis object
// ---------------------------------------------------------------------------

static void free_basis(jk_basis* b) {
    if (!b) return;
    cudaFree(b->mem_bas);
    cudaFree(b->mem_pair);
    jk_plan_free(b->plan);
    for (auto& p : b->shard_plans) jk_plan_free(p.second);
    for (void* p : b->retired) cudaFree(p);
    cudaFree(b->d_work);
    b->fan.destroy();
    cudaFree(b->d_pk);
    cudaFree(b->d_kt);
    if (b->blas) cublasDestroy(b->blas);
    delete b;
}

// Arrays of one set-up step in one device allocation: a request per array, the
// ones with contents uploaded, small ones together (a basis made some forty
// allocations and thirty copies, about 10 us each, and as many frees).
struct JKArena {
    struct Item {
        void** dst;
        const void* src;
        size_t src_bytes, off;
    };
    std::vector<Item> items;
    size_t total = 0;
    // n elements at *dst, the first nsrc from src (all of them by default)
    template <typename T>
    void add(T** dst, size_t n, const T* src = nullptr, size_t nsrc = (size_t)-1) {
        const size_t k = src ? std::min(n, nsrc) : 0;
        items.push_back({(void**)dst, src, k * sizeof(T), total});
        total += (std::max<size_t>(n, 1) * sizeof(T) + 255) & ~(size_t)255;
    }
    cudaError_t commit(void** mem) {
        cudaError_t e = cudaMalloc(mem, total);
        if (e != cudaSuccess) return e;
        std::vector<char> stage;  // neighbouring small items
        size_t at = 0;
        auto flush = [&] {
            if (!stage.empty())
                e = cudaMemcpyAsync((char*)*mem + at, stage.data(), stage.size(), cudaMemcpyHostToDevice,
                                    cudaStreamLegacy);
            stage.clear();
        };
        for (const Item& it : items) {
            *it.dst = (char*)*mem + it.off;
            if (it.src_bytes == 0 || it.src_bytes > 65536) {
                flush();
                if (e == cudaSuccess && it.src_bytes)
                    e = cudaMemcpyAsync(*it.dst, it.src, it.src_bytes, cudaMemcpyHostToDevice, cudaStreamLegacy);
            } else {
                if (stage.empty()) at = it.off;
                stage.resize(it.off - at + it.src_bytes);
                memcpy(stage.data() + (it.off - at), it.src, it.src_bytes);
            }
            if (e != cudaSuccess) return e;
        }
        flush();
        return e == cudaSuccess ? jk_internal_uploaded() : e;
    }
};

extern "C" int jk_rys_table_uniform(void);
extern "C" const double* jk_rys_coef_host(long long* count);

// Rys coefficient table in global memory, one copy per device, kept until exit
static std::mutex g_rys_mu;
static double* g_rys_dev[64];
static int rys_table_device(const double** out) {
    int dev;
    CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return set_err(JK_ERR_ARG, "device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> lk(g_rys_mu);
    if (!g_rys_dev[dev]) {
        long long n;
        const double* h = jk_rys_coef_host(&n);
        double* d;
        CUDA_TRY(cudaMalloc(&d, sizeof(double) * n));
        cudaError_t e = cudaMemcpy(d, h, sizeof(double) * n, cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = jk_internal_uploaded();
        if (e != cudaSuccess) {
            cudaFree(d);
            CUDA_TRY(e);
        }
        g_rys_dev[dev] = d;
    }
    *out = g_rys_dev[dev];
    return JK_OK;
}

// Schwarz ranks per bucket of a class of n pairs: 16 buckets, of whole chunks
// of 32 (a class up to 512 pairs is sorted inside its chunks only)
static int sort_bucket(int n) { return std::max(32, (n / 16 + 31) / 32 * 32); }

// Run length of a class quartet's bra (an index of JK_RUN_LEN): the longest
// that still gives `items` items per SM before screening; a molecule too small
// for that takes the shortest.  In a build the launches of the classes share the
// device, and 16 per SM do: at 5, 10, 16 and 40 (as it was) (H2O)8 / cc-pVDZ takes
// 1.34, 1.34, 1.41 and 1.58 ms, 37 atoms in 6-31G* 31.4, 31.8, 31.8 and 33.3, (H2O)12 /
// cc-pVDZ with an FP32 part 3.03, 3.02, 3.13 and 3.28, (H2O)9 / cc-pVDZ with one and
// two densities 4.95, 4.69, 4.58 and 4.58: below 16 the last one is slower.  At 160
// (H2O)32 / TZVP takes 263 ms instead of 255.  A per-class-pair call has the device
// to itself and keeps 40.
#define JK_RUN_ITEMS 16
#define JK_RUN_ITEMS_PAIR 40
// Contracted class quartets of at least this many primitive quartets go down to
// single bra pairs in a build too: a lane's chain of two of them is what a small
// molecule waits for.  Six waters in a six-fold contracted minimal basis 5.2 ms a
// quartet per thread, 11.2 with runs of two at least, 6.4 now; 13 atoms in 6-31G*
// 1.10 and 0.86 ms, 13 atoms / TZVP 5.2 and 4.95; 24 molecules in 6-31G* in a batch
// 40.9 and 40.2 ms, but 42.3 with single pairs for every class quartet.
#define JK_RUN_NPQ 64
static int run_level(const jk_basis* b, int cp_ij, int n_kl, int chunk, int levels, int items) {
    for (int v = 0; v < levels - 1; v++)
        if ((long long)b->h_nrun[v][cp_ij] * ((n_kl + chunk - 1) / chunk) >= (long long)items * b->nsm) return v;
    return levels - 1;
}

static int create_impl(const int* atm, int natm, const int* bas, int nbas, const double* env, int nenv,
                       const int* group_off, int ngroups, double cutoff, int diag_block_with_triu, jk_basis* b) {
    init_tables();
    if (!jk_rys_table_uniform()) return set_err(JK_ERR_ARG, "Rys tables must use intervals of width 2");
    {
        int rc = rys_table_device(&b->rys);
        if (rc) return rc;
    }
    CUDA_TRY(cudaGetDevice(&b->device));
    CUDA_TRY(cudaDeviceGetAttribute(&b->nsm, cudaDevAttrMultiProcessorCount, b->device));
    b->natm = natm;
    b->nbas = nbas;
    b->ngroups = ngroups;
    b->cutoff = cutoff;
    b->diag_fac = diag_block_with_triu ? 1.0 : 0.5;
    // shells must be sorted into groups of equal (l, nprim), one contraction each
    b->h_group_off.assign(group_off, group_off + ngroups + 1);
    if (b->h_group_off[0] != 0 || b->h_group_off[ngroups] != nbas)
        return set_err(JK_ERR_ARG, "group offsets must span 0..nbas");
    b->h_ao_loc.resize(nbas + 1);
    b->h_ao_loc[0] = 0;
    for (int i = 0; i < nbas; i++) {
        int l = bas[i * BAS_SLOTS + ANG_OF];
        if (l < 0 || l > JK_LMAX_ALL)
            return set_err(JK_ERR_UNSUPPORTED, "shell %d has l=%d; this engine handles l <= %d", i, l, JK_LMAX_ALL);
        if (bas[i * BAS_SLOTS + NCTR_OF] != 1)
            return set_err(JK_ERR_ARG, "shell %d: generally contracted shells must be split first", i);
        b->h_ao_loc[i + 1] = b->h_ao_loc[i] + (l + 1) * (l + 2) / 2;
    }
    b->nao = b->h_ao_loc[nbas];
    for (int g = 0; g < ngroups; g++) {
        int s0 = group_off[g], s1 = group_off[g + 1];
        if (s1 <= s0) return set_err(JK_ERR_ARG, "empty group %d", g);
        int l = bas[s0 * BAS_SLOTS + ANG_OF], np = bas[s0 * BAS_SLOTS + NPRIM_OF];
        for (int s = s0; s < s1; s++)
            if (bas[s * BAS_SLOTS + ANG_OF] != l || bas[s * BAS_SLOTS + NPRIM_OF] != np)
                return set_err(JK_ERR_ARG, "group %d mixes (l, nprim)", g);
        // groups may come in any l order (the density-fitting basis of
        // int3c concatenates molecule, exponent-0 shell and auxiliary
        // basis); the J/K class launches exist for classes whose bra and
        // ket are ordered by l, others report JK_ERR_UNSUPPORTED at build
        b->h_group_l.push_back(l);
        b->h_group_nprim.push_back(np);
    }
    // device copies of the basis
    std::vector<int> gao(ngroups + 1);
    for (int g = 0; g <= ngroups; g++) gao[g] = b->h_ao_loc[group_off[g]];
    std::vector<double> bx(3 * (size_t)nbas);
    for (int i = 0; i < nbas; i++) {
        const double* r = env + atm[bas[i * BAS_SLOTS + ATOM_OF] * ATM_SLOTS + PTR_COORD];
        bx[i] = r[0];
        bx[nbas + i] = r[1];
        bx[2 * (size_t)nbas + i] = r[2];
    }
    CUDA_TRY(b->fan.init());
    JKArena bas_mem;
    bas_mem.add(&b->d_env, nenv, env);
    bas_mem.add(&b->d_bas_x, bx.size(), bx.data());
    bas_mem.add(&b->d_atm, (size_t)natm * ATM_SLOTS, atm);
    bas_mem.add(&b->d_bas, (size_t)nbas * BAS_SLOTS, bas);
    bas_mem.add(&b->d_ao_loc, b->h_ao_loc.size(), b->h_ao_loc.data());
    bas_mem.add(&b->d_group_ao, gao.size(), gao.data());
    CUDA_TRY(bas_mem.commit(&b->mem_bas));

    // Schwarz matrix on the device, the pairs by their two l, a launch each
    b->h_qcond.resize((size_t)nbas * nbas);
    {
        std::vector<int> pi[JK_LMAX_ALL + 1][JK_LMAX_ALL + 1], pj[JK_LMAX_ALL + 1][JK_LMAX_ALL + 1];
        for (int i = 0; i < nbas; i++)
            for (int j = 0; j <= i; j++) {
                int li = bas[i * BAS_SLOTS + ANG_OF], lj = bas[j * BAS_SLOTS + ANG_OF];
                if (li >= lj) { pi[li][lj].push_back(i); pj[li][lj].push_back(j); }
                else { pi[lj][li].push_back(j); pj[lj][li].push_back(i); }
            }
        double* d_q;
        int *dpi[JK_LMAX_ALL + 1][JK_LMAX_ALL + 1], *dpj[JK_LMAX_ALL + 1][JK_LMAX_ALL + 1];
        JKArena mem;
        mem.add(&d_q, (size_t)nbas * nbas);
        for (int a = 0; a <= JK_LMAX_ALL; a++)
            for (int c = 0; c <= a; c++) {
                if (pi[a][c].empty()) continue;
                mem.add(&dpi[a][c], pi[a][c].size(), pi[a][c].data());
                mem.add(&dpj[a][c], pj[a][c].size(), pj[a][c].data());
            }
        void* tmp = nullptr;
        cudaError_t e = mem.commit(&tmp);
        int k = 0;
        for (int a = JK_LMAX_ALL; a >= 0 && e == cudaSuccess; a--)
            for (int c = a; c >= 0 && e == cudaSuccess; c--) {
                const int n = (int)pi[a][c].size();
                if (!n) continue;
                cudaStream_t st = b->fan.pick(k++);
                if (a <= JK_LMAX)
                    g_qcond[a][c](dpi[a][c], dpj[a][c], n, b->d_atm, b->d_bas, b->d_env, nbas, d_q, b->rys, st);
                else
                    jk_qcond_generic(dpi[a][c], dpj[a][c], n, b->d_atm, b->d_bas, b->d_env, nbas, d_q, b->rys, a, st);
                e = cudaGetLastError();
            }
        for (int x = 0; x < JK_SIDE_STREAMS; x++) {  // also after an error: tmp is freed below
            const cudaError_t es = cudaStreamSynchronize(b->fan.s[x]);
            if (e == cudaSuccess) e = es;
        }
        if (e == cudaSuccess)
            e = cudaMemcpy(b->h_qcond.data(), d_q, sizeof(double) * (size_t)nbas * nbas, cudaMemcpyDeviceToHost);
        cudaFree(tmp);
        CUDA_TRY(e);
    }
    // Schwarz-sorted pair lists per lower-triangular group pair, in the
    // reference's class order (cuobc/scf/hf.py:343-389)
    const std::vector<double>& q = b->h_qcond;
    b->h_pair_locs.push_back(0);
    std::vector<int> obra, oket, orank, opos;  // device order, see below
    {
        struct Cand {
            double q;
            int at;  // place in (bra shell, ket shell) order
        };
        std::vector<Cand> lst;
        std::vector<int> sh_i, sh_j, rank_of, fill;
        for (int gi = 0; gi < ngroups; gi++)
            for (int gj = 0; gj <= gi; gj++) {
                lst.clear();
                sh_i.clear();
                sh_j.clear();
                int p0 = group_off[gi], p1 = group_off[gi + 1], q0 = group_off[gj], q1 = group_off[gj + 1];
                for (int i = p0; i < p1; i++)
                    for (int j = q0; j < q1; j++) {
                        if (gi == gj && !diag_block_with_triu && j > i) continue;
                        double v = q[(size_t)i * nbas + j];
                        if (v > cutoff) {
                            lst.push_back({v, (int)sh_i.size()});
                            sh_i.push_back(i);
                            sh_j.push_back(j);
                        }
                    }
                std::stable_sort(lst.begin(), lst.end(), [](const Cand& x, const Cand& y) { return x.q > y.q; });
                const int np = (int)lst.size(), at0 = b->h_pair_locs.back(), S = sort_bucket(np);
                rank_of.resize(np);
                for (int x = 0; x < np; x++) {
                    const Cand& c = lst[x];
                    rank_of[c.at] = x;
                    b->h_pair2bra.push_back(sh_i[c.at]);
                    b->h_pair2ket.push_back(sh_j[c.at]);
                    double lq = log(c.q);
                    b->h_log_q.push_back(lq > 0 ? 0 : lq);
                    b->h_log_q_raw.push_back(lq);
                }
                // the pairs in shell order, each to the end of its rank's bucket
                fill.assign(np / S + 1, 0);
                obra.resize(at0 + np);
                oket.resize(at0 + np);
                orank.resize(at0 + np);
                opos.resize(at0 + np);
                for (int y = 0; y < np; y++) {
                    const int x = rank_of[y], k = x / S, pos = k * S + fill[k]++;
                    orank[at0 + pos] = x;
                    opos[at0 + x] = pos;
                    obra[at0 + pos] = sh_i[y];
                    oket[at0 + pos] = sh_j[y];
                }
                b->h_cls_gi.push_back(gi);
                b->h_cls_gj.push_back(gj);
                b->h_pair_locs.push_back(at0 + np);
            }
    }
    b->ncp = (int)b->h_cls_gi.size();
    // Device order of a class's pairs: buckets of sort_bucket(pairs)
    // consecutive Schwarz ranks, inside a bucket by (bra shell, ket shell).
    // The lanes of a run kernel's warp hold consecutive pairs, so the D_jk they
    // read and the K_jk they add to lie on a few sectors instead of one each
    // ((ps| pairs of (H2O)64 / cc-pVDZ: 5 sectors per 32 lanes for k and 23
    // for l instead of 30 and 30), for at most one bucket of lanes idle at the
    // end of a row (6 %).  The lists that the C-ABI gives out stay in rank
    // order, as do log q and the screening.
    const size_t npair = b->h_pair2bra.size();
    // primitive-pair data (cuobc/lib/gint/pair_data.c:83-141)
    long long npp = 0;
    b->h_prim_locs.push_back(0);
    for (int c = 0; c < b->ncp; c++) {
        int np12 = b->h_group_nprim[b->h_cls_gi[c]] * b->h_group_nprim[b->h_cls_gj[c]];
        npp += (long long)(b->h_pair_locs[c + 1] - b->h_pair_locs[c]) * np12;
        if (npp > 0x7fffffffLL) return set_err(JK_ERR_ARG, "too many primitive pairs");
        b->h_prim_locs.push_back((int)npp);
    }
    b->nprim_total = npp;
    std::vector<double> prim(5 * (size_t)(npp ? npp : 1));  // 1 / a12 and the rest of the tables: on the device
    double *a12 = prim.data(), *e12 = a12 + npp, *x12 = e12 + npp, *y12 = x12 + npp, *z12 = y12 + npp;
    std::vector<std::pair<int, int>> order;
    b->h_pnp.assign(std::max<size_t>(b->h_pair2bra.size(), 1), 0);
    for (int c = 0; c < b->ncp; c++) {
        // primitive-major within the class: primitive k of pair r at
        // h_prim_locs[c] + k * (pairs in the class) + r
        const int p0 = b->h_pair_locs[c], pst = b->h_pair_locs[c + 1] - p0;
        for (int p = p0; p < p0 + pst; p++) {
            int ish = obra[p], jsh = oket[p];
            int npi = bas[ish * BAS_SLOTS + NPRIM_OF], npj = bas[jsh * BAS_SLOTS + NPRIM_OF];
            int li = bas[ish * BAS_SLOTS + ANG_OF], lj = bas[jsh * BAS_SLOTS + ANG_OF];
            const double* ai = env + bas[ish * BAS_SLOTS + PTR_EXP];
            const double* aj = env + bas[jsh * BAS_SLOTS + PTR_EXP];
            const double* ci = env + bas[ish * BAS_SLOTS + PTR_COEFF];
            const double* cj = env + bas[jsh * BAS_SLOTS + PTR_COEFF];
            const double* ri = env + atm[bas[ish * BAS_SLOTS + ATOM_OF] * ATM_SLOTS + PTR_COORD];
            const double* rj = env + atm[bas[jsh * BAS_SLOTS + ATOM_OF] * ATM_SLOTS + PTR_COORD];
            double norm = common_fac_sp(li) * common_fac_sp(lj);
            double dx = ri[0] - rj[0], dy = ri[1] - rj[1], dz = ri[2] - rj[2];
            double r2 = dx * dx + dy * dy + dz * dz;
            // primitive pairs whose Gaussian-product factor exp(-ai aj/(ai+aj) r^2)
            // is above exp(-JK_PRIM_EXPCUT) first, their count in h_pnp
            // (the run kernels loop over those only; the others carry a
            // factor below 1e-26 and are kept after them for the kernels
            // that loop over all)
            order.clear();
            for (int pass = 0; pass < 2; pass++)
                for (int ip = 0; ip < npi; ip++)
                    for (int jp = 0; jp < npj; jp++) {
                        const bool kept = r2 * ai[ip] * aj[jp] / (ai[ip] + aj[jp]) <= JK_PRIM_EXPCUT;
                        if (kept == (pass == 0)) order.push_back({ip, jp});
                        if (pass == 0 && kept) b->h_pnp[p]++;
                    }
            long long off = b->h_prim_locs[c] + (p - p0);
            for (const auto& pr : order) {
                const int ip = pr.first, jp = pr.second;
                {
                    double aij = ai[ip] + aj[jp];
                    a12[off] = aij;
                    e12[off] = norm * ci[ip] * cj[jp] * exp(-r2 * ai[ip] * aj[jp] / aij);
                    if (ish == jsh) e12[off] *= b->diag_fac;
                    x12[off] = (ai[ip] * ri[0] + aj[jp] * rj[0]) / aij;
                    y12[off] = (ai[ip] * ri[1] + aj[jp] * rj[1]) / aij;
                    z12[off] = (ai[ip] * ri[2] + aj[jp] * rj[2]) / aij;
                }
                off += pst;
            }
        }
    }
    // runs of every class's pairs: the pairs of one first shell, in Schwarz
    // order, cut at each run length
    std::vector<int> ent(npair), run0;
    {
        for (int v = 0; v < JK_RUN_LEVELS_PAIR; v++) {
            b->h_nrun[v].assign(b->ncp, 0);
            b->h_run_off[v].assign(b->ncp, 0);
        }
        // single pairs: run r holds entry r, in every class
        int mx = 0;
        for (int c = 0; c < b->ncp; c++) mx = std::max(mx, b->h_pair_locs[c + 1] - b->h_pair_locs[c]);
        run0.resize(mx + 1);
        std::iota(run0.begin(), run0.end(), 0);
        std::vector<int> at(nbas + 1), end(nbas + 1);
        for (int c = 0; c < b->ncp; c++) {
            const int p0 = b->h_pair_locs[c], np = b->h_pair_locs[c + 1] - p0;
            const int s0 = group_off[b->h_cls_gi[c]], s1 = group_off[b->h_cls_gi[c] + 1];
            int* e = ent.data() + p0;
            // e: positions by first shell (counting sort, ranks ascending in a shell)
            for (int x = s0; x <= s1; x++) at[x] = 0;
            for (int x = 0; x < np; x++) at[b->h_pair2bra[p0 + x] + 1]++;
            for (int x = s0; x < s1; x++) at[x + 1] += at[x];
            for (int x = s0; x <= s1; x++) end[x] = at[x];
            for (int x = 0; x < np; x++) e[at[b->h_pair2bra[p0 + x]]++] = opos[p0 + x];
            b->h_nrun[JK_RUN_LEVELS_PAIR - 1][c] = np;
            for (int v = 0; v < JK_RUN_LEVELS_PAIR - 1; v++) {
                b->h_run_off[v][c] = (int)run0.size();
                for (int x = s0; x < s1; x++)
                    for (int beg = end[x]; beg < end[x + 1]; beg += JK_RUN_LEN[v]) run0.push_back(beg);
                b->h_nrun[v][c] = (int)run0.size() - b->h_run_off[v][c];
                run0.push_back(np);
            }
        }
    }
    // class quartets (cp_ij >= cp_kl), each with its slices of the screening buffers
    std::vector<long long> qoff_at, ioff_at, ent_at;
    for (int cij = 0; cij < b->ncp; cij++)
        for (int ckl = 0; ckl <= cij; ckl++) {
            JKScreenCQ c{};
            c.cp_ij = cij;
            c.cp_kl = ckl;
            c.gi = b->h_cls_gi[cij];
            c.gj = b->h_cls_gj[cij];
            c.gk = b->h_cls_gi[ckl];
            c.gl = b->h_cls_gj[ckl];
            c.pair_ij0 = b->h_pair_locs[cij];
            c.n_ij = b->h_pair_locs[cij + 1] - c.pair_ij0;
            c.pair_kl0 = b->h_pair_locs[ckl];
            c.n_kl = b->h_pair_locs[ckl + 1] - c.pair_kl0;
            if (c.n_ij == 0 || c.n_kl == 0) continue;
            const double npq = (double)b->h_group_nprim[c.gi] * b->h_group_nprim[c.gj] * b->h_group_nprim[c.gk] *
                               b->h_group_nprim[c.gl];
            c.runs = g_tabs.run[class_index(b, cij, ckl)];
            qoff_at.push_back(b->qoff_total);
            ioff_at.push_back(b->ioff_total);
            ent_at.push_back(b->ent_total);
            b->ent_total += c.n_ij;
            if (c.runs) {
                c.level = run_level(b, cij, c.n_kl, c.runs, npq >= JK_RUN_NPQ ? JK_RUN_LEVELS_PAIR : JK_RUN_LEVELS, JK_RUN_ITEMS);
                c.nrun = b->h_nrun[c.level][cij];
                b->ioff_total += 2LL * c.nrun;
            } else {
                b->qoff_total += c.n_ij + 1;
            }
            b->h_cq.push_back(c);
            // unscreened work for shard plans: quartets x primitive
            // quartets x roots x Cartesian components (+ the digestion)
            const int l4[4] = {b->h_group_l[c.gi], b->h_group_l[c.gj], b->h_group_l[c.gk], b->h_group_l[c.gl]};
            double nf = 1.;
            for (int a = 0; a < 4; a++) nf *= (l4[a] + 1) * (l4[a] + 2) / 2;
            const double nq = cij == ckl ? 0.5 * c.n_ij * (c.n_ij + 1.) : (double)c.n_ij * c.n_kl;
            b->h_cq_cost.push_back(nq * (npq * ((l4[0] + l4[1] + l4[2] + l4[3]) / 2 + 1) * nf + 12. * nf));
        }
    b->ncq = (int)b->h_cq.size();
    // pair-packed layout of the J side (jk_build)
    b->h_pack.clear();
    b->pack_total = 0;
    int mx = 1;  // pairs of the largest class
    for (int c = 0; c < b->ncp; c++) {
        JKPackCls k;
        k.off = b->pack_total;
        k.pair0 = b->h_pair_locs[c];
        k.np = b->h_pair_locs[c + 1] - k.pair0;
        const int li = b->h_group_l[b->h_cls_gi[c]], lj = b->h_group_l[b->h_cls_gj[c]];
        k.nfi = (li + 1) * (li + 2) / 2;
        k.nfj = (lj + 1) * (lj + 2) / 2;
        b->pack_total += (long long)k.np * k.nfi * k.nfj;
        b->h_pack.push_back(k);
        mx = std::max(mx, k.np);
    }
    // the buffers a build clears: condensed density, then {0, count} of the
    // quartets and items of both parts
    b->zero_bytes = sizeof(double) * ((size_t)ngroups * ngroups + 8 * (size_t)b->ncq);
    int *d_locs, *d_plocs;
    unsigned long long* zero;
    JKArena mem;
    mem.add(&b->d_prim, 6 * (size_t)npp, prim.data(), 5 * (size_t)npp);
    mem.add(&b->d_log_q_raw, npair, b->h_log_q_raw.data());
    mem.add(&b->d_pair2bra, npair, obra.data());
    mem.add(&b->d_pair2ket, npair, oket.data());
    mem.add(&b->d_rank, npair, orank.data());
    mem.add(&b->d_ent, npair, ent.data());
    mem.add(&b->d_pnp, b->h_pnp.size(), b->h_pnp.data());
    mem.add(&b->d_run0, run0.size(), run0.data());
    mem.add(&b->d_pack, b->h_pack.size(), b->h_pack.data());
    mem.add(&d_locs, b->h_pair_locs.size(), b->h_pair_locs.data());
    mem.add(&d_plocs, b->h_prim_locs.size(), b->h_prim_locs.data());
    mem.add(&b->d_log_q, npair);
    mem.add(&b->d_pos, npair);
    mem.add(&b->d_inv, npair);
    mem.add(&b->d_erank, npair);
    mem.add(&b->d_pgeo, 6 * npair);
    mem.add(&b->d_pao, 2 * npair);
    mem.add(&b->d_primf, 6 * (size_t)npp);
    mem.add(&b->d_bprim, 8 * (size_t)npp);
    mem.add(&b->d_bprimf, 8 * (size_t)npp);
    mem.add(&b->d_bpair, 4 * npair);
    mem.add(&b->d_qoff, (size_t)b->qoff_total);
    mem.add(&b->d_qoff32, (size_t)b->qoff_total);
    mem.add(&b->d_ioff, (size_t)b->ioff_total);
    mem.add(&b->d_klb, (size_t)b->ent_total);
    mem.add(&b->d_kle, (size_t)b->ent_total);
    mem.add(&zero, b->zero_bytes / 8);
    mem.add(&b->d_cq, b->h_cq.size());
    // the per-class-pair entries: row prefixes sized once for the largest
    // class, so those calls never free a buffer a queued kernel still reads
    mem.add(&b->d_task01, 2);
    mem.add(&b->d_seg1, 1);
    mem.add(&b->d_qoff1, (size_t)mx + 1);
    mem.add(&b->d_ehi1, mx);
    b->qoff1_cap = mx + 1;
    CUDA_TRY(mem.commit(&b->mem_pair));
    b->d_zero = zero;
    if (npair) {
        jk_pair_tables_kernel<<<(unsigned)((npair + 255) / 256), 256>>>(
            (int)npair, b->ncp, d_locs, b->d_pair2bra, b->d_pair2ket, b->d_rank, b->d_ent, b->d_bas_x, nbas,
            b->d_ao_loc, b->d_log_q_raw, b->d_log_q, b->d_pgeo, b->d_pao, b->d_pos, b->d_inv, b->d_erank);
        jk_prim_tables_kernel<<<(unsigned)((npp + 255) / 256), 256>>>(
            (int)npp, (int)npair, b->ncp, d_locs, d_plocs, b->d_prim, b->d_primf, b->d_inv, b->d_pgeo, b->d_pao,
            b->d_pnp, b->d_bprim, b->d_bprimf, b->d_bpair);
        CUDA_TRY(cudaGetLastError());
    }
    b->d_dm_cond = (double*)b->d_zero;
    b->d_task0 = (long long*)(b->d_dm_cond + (size_t)ngroups * ngroups);
    b->d_task032 = b->d_task0 + 2 * b->ncq;
    for (int c = 0; c < b->ncq; c++) {
        JKScreenCQ& q = b->h_cq[c];
        q.ngroups = ngroups;
        q.lq_ij = b->d_log_q + q.pair_ij0;
        q.lq_kl = b->d_log_q + q.pair_kl0;
        q.rq_ij = b->d_log_q_raw + q.pair_ij0;
        q.rq_kl = b->d_log_q_raw + q.pair_kl0;
        q.dm_cond = b->d_dm_cond;
        q.qoff = b->d_qoff + qoff_at[c];
        q.qoff32 = b->d_qoff32 + qoff_at[c];
        q.klb = b->d_klb + ent_at[c];
        q.kle = b->d_kle + ent_at[c];
        q.ioff = b->d_ioff + ioff_at[c];
        q.ioff32 = q.ioff + q.nrun;
        q.ent = b->d_ent + q.pair_ij0;
        q.erank = b->d_erank + q.pair_ij0;
        q.bucket = sort_bucket(q.n_kl);
        q.run0 = b->d_run0 + b->h_run_off[q.level][q.cp_ij];
        q.task0 = b->d_task0 + 2 * c;
        q.task032 = b->d_task032 + 2 * c;
        q.itm = b->d_task0 + 4 * b->ncq + 2 * c;
        q.itm32 = b->d_task0 + 6 * b->ncq + 2 * c;
    }
    if (b->ncq)
        CUDA_TRY(cudaMemcpyAsync(b->d_cq, b->h_cq.data(), sizeof(JKScreenCQ) * b->ncq, cudaMemcpyHostToDevice,
                                 cudaStreamLegacy));
    // the class launches of jk_build (bases with classes that no J/K kernel
    // serves, as the density fitting's, do without)
    int rc = make_plan(b, 1, 0, &b->plan);
    if (rc && rc != JK_ERR_UNSUPPORTED) return rc;
    CUDA_TRY(jk_internal_uploaded());
    return JK_OK;
}

extern "C" int jk_basis_create(const int* atm, int natm, const int* bas, int nbas, const double* env, int nenv,
                               const int* group_offsets, int ngroups, double cutoff, int diag_block_with_triu,
                               jk_basis_t** out) {
    if (!atm || !bas || !env || !group_offsets || !out || natm <= 0 || nbas <= 0 || ngroups <= 0)
        return set_err(JK_ERR_ARG, "jk_basis_create: invalid arguments");
    jk_basis* b = new jk_basis();
    int rc = jk_guard([&] {
        return create_impl(atm, natm, bas, nbas, env, nenv, group_offsets, ngroups, cutoff, diag_block_with_triu, b);
    });
    if (rc != JK_OK) {
        free_basis(b);
        *out = nullptr;
        return rc;
    }
    *out = b;
    return JK_OK;
}

extern "C" int jk_basis_destroy(jk_basis_t* b) {
    free_basis(b);
    return JK_OK;
}

extern "C" int jk_basis_info(const jk_basis_t* b, int* info) {
    if (!b || !info) return set_err(JK_ERR_ARG, "jk_basis_info: invalid arguments");
    info[0] = b->nbas;
    info[1] = b->nao;
    info[2] = b->ngroups;
    info[3] = b->ncp;
    info[4] = (int)b->h_pair2bra.size();
    info[5] = (int)b->nprim_total;
    info[6] = b->ncq;
    return JK_OK;
}

extern "C" int jk_basis_pairs(const jk_basis_t* b, int* pair2shls, int* pair_locs, double* log_q, double* q_cond) {
    if (!b) return set_err(JK_ERR_ARG, "jk_basis_pairs: null basis");
    size_t np = b->h_pair2bra.size();
    if (pair2shls) {
        std::copy(b->h_pair2bra.begin(), b->h_pair2bra.end(), pair2shls);
        std::copy(b->h_pair2ket.begin(), b->h_pair2ket.end(), pair2shls + np);
    }
    if (pair_locs) std::copy(b->h_pair_locs.begin(), b->h_pair_locs.end(), pair_locs);
    if (log_q) std::copy(b->h_log_q.begin(), b->h_log_q.end(), log_q);
    if (q_cond) std::copy(b->h_qcond.begin(), b->h_qcond.end(), q_cond);
    return JK_OK;
}

static void fill_seg(const jk_basis* b, int cp_ij, int cp_kl, const long long* qoff, int n_ij, const double* dm,
                     int n_dm, double* vj, double* vk, JKSeg* s) {
    *s = JKSeg{};
    s->rys = b->rys;
    s->qoff = qoff;
    s->n_ij = n_ij;
    s->pair_ij0 = b->h_pair_locs[cp_ij];
    s->pair_kl0 = b->h_pair_locs[cp_kl];
    s->prim_ij0 = b->h_prim_locs[cp_ij];
    s->prim_kl0 = b->h_prim_locs[cp_kl];
    s->nprim_ij = b->h_group_nprim[b->h_cls_gi[cp_ij]] * b->h_group_nprim[b->h_cls_gj[cp_ij]];
    s->nprim_kl = b->h_group_nprim[b->h_cls_gi[cp_kl]] * b->h_group_nprim[b->h_cls_gj[cp_kl]];
    s->pst_ij = b->h_pair_locs[cp_ij + 1] - b->h_pair_locs[cp_ij];
    s->pst_kl = b->h_pair_locs[cp_kl + 1] - b->h_pair_locs[cp_kl];
    s->nao = b->nao;
    s->n_dm = n_dm;
    long long n = b->nprim_total;
    s->a12 = b->d_prim;
    s->e12 = b->d_prim + n;
    s->x12 = b->d_prim + 2 * n;
    s->y12 = b->d_prim + 3 * n;
    s->z12 = b->d_prim + 4 * n;
    s->ia12 = b->d_prim + 5 * n;
    s->pf = b->d_primf;
    s->npf = n;
    s->pgeo = b->d_pgeo;
    s->pnp = b->d_pnp;
    s->rank = b->d_rank;
    s->pos = b->d_pos;
    s->bucket = sort_bucket(s->pst_kl);
    s->bprim = b->d_bprim + 8 * (size_t)s->prim_ij0;
    s->bprimf = b->d_bprimf + 8 * (size_t)s->prim_ij0;
    s->bpair = b->d_bpair + 4 * (size_t)s->pair_ij0;
    s->pao = b->d_pao;
    s->npt = (int)b->h_pair2bra.size();
    s->dm = dm;
    s->vj = vj;
    s->vk = vk;
    s->pk_ij = b->h_pack[cp_ij].off;
    s->pk_kl = b->h_pack[cp_kl].off;
    s->pk_stride = b->pack_total;
    s->ls[0] = b->h_group_l[b->h_cls_gi[cp_ij]];
    s->ls[1] = b->h_group_l[b->h_cls_gj[cp_ij]];
    s->ls[2] = b->h_group_l[b->h_cls_gi[cp_kl]];
    s->ls[3] = b->h_group_l[b->h_cls_gj[cp_kl]];
}

static int class_index(const jk_basis* b, int cp_ij, int cp_kl) {
    int li = b->h_group_l[b->h_cls_gi[cp_ij]], lj = b->h_group_l[b->h_cls_gj[cp_ij]];
    int lk = b->h_group_l[b->h_cls_gi[cp_kl]], ll = b->h_group_l[b->h_cls_gj[cp_kl]];
    return JK_CLASS_INDEX(li, lj, lk, ll);
}

static int shard_plan(const double* cost, int n, int nshards, int* owner) {
    if (n < 0 || nshards < 1 || (n > 0 && (!cost || !owner)))
        return set_err(JK_ERR_ARG, "jk_shard_plan: invalid arguments");
    std::vector<int> ord(n);
    for (int i = 0; i < n; i++) ord[i] = i;
    std::stable_sort(ord.begin(), ord.end(), [&](int a, int c) { return cost[a] > cost[c]; });
    std::vector<double> load(nshards, 0.);
    for (int i : ord) {
        int best = 0;
        for (int r = 1; r < nshards; r++)
            if (load[r] < load[best]) best = r;
        owner[i] = best;
        load[best] += cost[i];
    }
    return JK_OK;
}

extern "C" int jk_shard_plan(const double* cost, int n, int nshards, int* owner) {
    return jk_guard([&] { return shard_plan(cost, n, nshards, owner); });
}

static unsigned dm_cond_blocks(int nao) { return (unsigned)std::min(64, nao / 8 + 1); }

// owner of every class quartet for nshards shards (cached per basis)
static const int* shard_owners(jk_basis* b, int nshards) {
    if (b->cq_owner_n != nshards || (int)b->h_cq_owner.size() != b->ncq) {
        b->h_cq_owner.assign(b->ncq, 0);
        shard_plan(b->h_cq_cost.data(), b->ncq, nshards, b->h_cq_owner.data());
        b->cq_owner_n = nshards;
    }
    return b->h_cq_owner.data();
}

// class launches of one shard of a build
static int make_plan(jk_basis* b, int nshards, int shard, JKPlan** out) {
    std::unique_ptr<JKPlan, void (*)(JKPlan*)> p(new JKPlan(), jk_plan_free);
    const int* owner = nshards > 1 ? shard_owners(b, nshards) : nullptr;
    int rc = JK_OK;
    for (int c = 0; c < b->ncq && !rc; c++)
        if (!owner || owner[c] == shard) rc = jk_plan_add(p.get(), b, 0, c, false);
    if (!rc) rc = jk_plan_finish(p.get(), {b}, {b->h_cq.data()});
    *out = rc ? nullptr : p.release();
    return rc;
}

static bool is_capturing(cudaStream_t st) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return cs != cudaStreamCaptureStatusNone;
}

// a workspace of the basis of at least `need` doubles
static int grow(jk_basis* b, double** p, size_t* cap, size_t need) {
    if (need <= *cap) return JK_OK;
    if (b->captured && *p) b->retired.push_back(*p);
    else cudaFree(*p);
    *p = nullptr;
    *cap = 0;
    CUDA_TRY(cudaMalloc(p, sizeof(double) * need));
    *cap = need;
    return JK_OK;
}

// krows: the caller reads V + V^T of K only, which the run kernels may then
// leave by rows; otherwise vk gets the layout of the C-ABI
static int build(jk_basis* b, const double* dm, int n_dm, double* vj, double* vk, bool krows, const jk_opts_t* opts,
                 void* stream) {
    if (!b || !dm || n_dm <= 0) return set_err(JK_ERR_ARG, "jk_build: invalid arguments");
    if (!vj && !vk) return JK_OK;
    cudaStream_t st = (cudaStream_t)stream;
    double tol = opts ? opts->direct_scf_tol : b->cutoff;
    int nbins = opts && opts->nbins > 0 ? opts->nbins : 10;
    int prescreen = opts ? opts->prescreen : 1;
    const int nshards = opts && opts->nshards > 1 ? opts->nshards : 1;
    const int shard = nshards > 1 ? opts->shard : 0;
    if (nshards > 1 && (shard < 0 || shard >= nshards)) return set_err(JK_ERR_ARG, "jk_build: shard out of range");
    const bool capturing = is_capturing(st);
    b->captured |= capturing;
    // the plan of this split; the first build of a split inside a capture,
    // which cannot make it, launches its class quartets one by one from the
    // tables of the whole build
    if (!b->plan) {  // a class without a kernel
        int rc = make_plan(b, 1, 0, &b->plan);
        if (rc) return rc;
    }
    JKPlan* plan = b->plan;
    const int* singly = nullptr;
    if (nshards > 1) {
        auto it = b->shard_plans.find({nshards, shard});
        if (it != b->shard_plans.end() && it->second) {
            plan = it->second;
        } else if (capturing) {
            singly = shard_owners(b, nshards);
        } else {
            JKPlan*& slot = b->shard_plans[{nshards, shard}];
            if (!slot) {
                int rc = make_plan(b, nshards, shard, &slot);
                if (rc) return rc;
            }
            plan = slot;
        }
    }
    int rc = JK_OK;
    // pair-packed density and J accumulators for the run kernels
    const bool packed = vj && b->pack_total > 0;
    JKCall call{dm, vj, vk, nullptr, nullptr, nullptr, nullptr, n_dm, nullptr, 0};
    JKPackMol pm{};
    const int pk_blocks = (int)std::min<long long>((b->pack_total + 255) / 256, (long long)b->nsm * 8);
    if (packed) {
        rc = grow(b, &b->d_pk, &b->pk_cap, (size_t)4 * n_dm * b->pack_total);
        if (rc) return rc;
        pm = jk_internal_pack_mol(b, dm, n_dm, b->d_pk, b->d_pk + 2 * (size_t)n_dm * b->pack_total, vj);
        call.dp = pm.dp;
        call.jp = pm.jp;
        call.dpb = pm.dpb;
        call.jpb = pm.jpb;
    }
    // K by rows into a buffer of the handle, added transposed at the end; a
    // capture cannot allocate it, and lets the run kernels write vk itself
    bool direct = false;
    if (vk && !krows) {
        const size_t need = (size_t)n_dm * b->nao * b->nao;
        direct = capturing && need > b->kt_cap;
        if (!direct) {
            rc = grow(b, &b->d_kt, &b->kt_cap, need);
            if (rc) return rc;
            call.kt = b->d_kt;
            call.nkt = (long long)need;
        }
    }
    jk_begin_kernel<<<std::max(pk_blocks, 8), 256, 0, st>>>(plan->d_seg[0], plan->d_seg[1], plan->nseg, call,
                                                            (unsigned long long*)b->d_zero,
                                                            (long long)(b->zero_bytes / 8), pm);
    CUDA_TRY(cudaGetLastError());
    const JKDmCond dc{dm, b->d_group_ao, b->d_dm_cond, b->nao, n_dm, b->ngroups, nullptr, 0};
    jk_dm_cond_kernel<<<dim3(dm_cond_blocks(b->nao), b->ngroups), 256, 0, st>>>(dc, nullptr);
    CUDA_TRY(cudaGetLastError());
    if (b->ncq == 0) return JK_OK;
    double fp32_cutoff = opts ? opts->fp32_cutoff : 0.;
    const bool mixed = fp32_cutoff > 0;
    rc = jk_internal_screen(b->d_cq, b->ncq, tol, nbins, prescreen, fp32_cutoff, st);
    if (!rc && !singly) rc = jk_plan_prefix(plan, mixed, st);
    if (rc) return rc;
    // class launches on side streams: 4 of them, 8 with the FP32 parts or for a
    // molecule whose launches leave most of the device idle (8 and 4 streams: one
    // water 186 and 220 us, 13 atoms / TZVP, 3662 pairs, 5.2 and 6.9 ms; from (H2O)8
    // / cc-pVDZ, 6112 pairs, on the two are within 1 %, and 4 are cheaper to fork)
    const int np = mixed ? 2 : 1, ns = mixed || b->h_pair2bra.size() < 4096 ? 8 : 4;
    CUDA_TRY(b->fan.begin(st, ns));
    for (int k = 0; k < (int)plan->keys.size(); k++)
        for (int part = 0; part < np; part++) {
            const JKPlanKey& key = plan->keys[k];
            cudaStream_t side = b->fan.s[(np * k + part) % ns];
            if (!singly) rc = jk_plan_launch(plan, k, part, key.cfg[part], n_dm, b->nsm, side, direct);
            else
                for (int x = 0; x < (int)key.segs.size() && !rc; x++)
                    if (singly[key.segs[x].second] == shard)
                        rc = jk_plan_launch_one(plan, k, x, part, b->h_cq[key.segs[x].second], n_dm, b->nsm, side, direct);
            if (rc) return rc;
        }
    CUDA_TRY(b->fan.end(st, ns));
    if (call.kt) {
        if (!packed) {
            pm.nao = b->nao;
            pm.n_dm = n_dm;
        }
        pm.kt = call.kt;
        pm.vk = vk;
    }
    if (packed || pm.kt) {
        const long long nt = (b->nao + 31) / 32, tiles = pm.kt ? n_dm * nt * nt : 0;
        const int blocks = (int)std::min<long long>(std::max<long long>(tiles, pm.total ? pk_blocks : 1), b->nsm * 8LL);
        jk_finish_kernel<<<blocks, 256, 0, st>>>(pm);
        CUDA_TRY(cudaGetLastError());
    }
    return JK_OK;
}

extern "C" int jk_build(jk_basis_t* b, const double* dm, int n_dm, double* vj, double* vk, const jk_opts_t* opts,
                        void* stream) {
    return jk_guard([&] { return build(b, dm, n_dm, vj, vk, false, opts, stream); });
}

// Row prefix of one class pair's task list from the host bins of the
// per-class-pair entries (nr_jk_driver.cu:252-280, nr_fill_ao_ints.cu:519-545):
// row ij in bin s (ij[s] <= ij < ij[s+1]) keeps c_s = kl[nbins - s] - kl[0]
// columns (none when kl[0] != 0: the reference's bins start at 0), at most
// ij + 1 of them on a diagonal class pair of jk_build_class_pair; rows below
// ij[0] or from ij[nbins] on keep none.  The bins go to the device by value,
// so the entries neither copy nor synchronise.
#define JK_ROWBINS_MAX 64
struct JKRowBins {
    int nbins, diag;
    int ij[JK_ROWBINS_MAX + 1], kl[JK_ROWBINS_MAX + 1];
};

// tasks of rows [0, r)
__host__ __device__ inline long long jk_rowbins_tasks(const JKRowBins& b, long long r) {
    if (b.kl[0] != 0) return 0;
    long long acc = 0;
    for (int s = 0; s < b.nbins; s++) {
        const long long lo = b.ij[s];
        const long long hi = r < b.ij[s + 1] ? r : b.ij[s + 1];
        if (hi <= lo) continue;
        const long long c = b.kl[b.nbins - s] - b.kl[0];
        if (!b.diag) {
            acc += c * (hi - lo);
        } else {
            // rows below c keep row + 1 columns, the others c
            const long long m = lo > (c < hi ? c : hi) ? lo : (c < hi ? c : hi);
            acc += (m * (m + 1) - lo * (lo + 1)) / 2 + c * (hi - m);
        }
    }
    return acc;
}

// columns row r keeps
struct JKRowBinsCols {
    JKRowBins b;
    int n_kl;
    __device__ __forceinline__ int operator()(int r) const {
        if (b.kl[0] != 0) return 0;
        for (int s = 0; s < b.nbins; s++)
            if (r >= b.ij[s] && r < b.ij[s + 1]) {
                const int c = min(b.kl[b.nbins - s], n_kl);
                return b.diag && c > r + 1 ? r + 1 : c;
            }
        return 0;
    }
};

// run classes of many bra pairs: ket end of every entry
__global__ void jk_run_rowbins_kernel(const __grid_constant__ JKRowBinsCols cols, int n_ij,
                                      const int* __restrict__ erank, int* __restrict__ ehi) {
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n_ij; e += gridDim.x * blockDim.x)
        ehi[e] = cols(erank[e]);
}

__device__ __forceinline__ void jk_rowbins_body(const JKRowBins& rb, int n_ij, long long* __restrict__ qoff,
                                                long long* __restrict__ task0) {
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r <= n_ij;
         r += (long long)gridDim.x * blockDim.x)
        qoff[r] = jk_rowbins_tasks(rb, r);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        task0[0] = 0;
        task0[1] = jk_rowbins_tasks(rb, n_ij);
    }
}
__global__ void jk_rowbins_kernel(const JKRowBins rb, int n_ij, long long* __restrict__ qoff,
                                  long long* __restrict__ task0) {
    jk_rowbins_body(rb, n_ij, qoff, task0);
}
// ... and the segment of a J/K call (a row class) to *dst
__global__ void jk_rowbins_seg_kernel(const JKRowBins rb, int n_ij, long long* __restrict__ qoff,
                                      long long* __restrict__ task0, const __grid_constant__ JKSeg sg, JKSeg* dst) {
    if (blockIdx.x == 0) jk_seg_copy(sg, dst);
    jk_rowbins_body(rb, n_ij, qoff, task0);
}

static int row_bins(const int* bins_ij, const int* bins_kl, int nbins, int diag, JKRowBins* rb) {
    if (nbins > JK_ROWBINS_MAX) return set_err(JK_ERR_ARG, "nbins %d above %d", nbins, JK_ROWBINS_MAX);
    rb->nbins = nbins;
    rb->diag = diag;
    for (int s = 0; s <= nbins; s++) {
        rb->ij[s] = bins_ij[s];
        rb->kl[s] = bins_kl[s];
        if (s && (bins_ij[s] < bins_ij[s - 1] || bins_kl[s] < bins_kl[s - 1]))
            return set_err(JK_ERR_ARG, "bins must not decrease");
    }
    return JK_OK;
}

// bins of a per-class-pair call -> the basis's row prefix and task count, on
// `st`, and the segment (if any) to *dst; returns the task count through *tot
static int class_pair_rows(jk_basis* b, const JKRowBins& rb, int n_ij, const JKSeg* seg, JKSeg* dst, cudaStream_t st,
                           long long* tot) {
    if (n_ij + 1 > (int)b->qoff1_cap) return set_err(JK_ERR_ARG, "class pair larger than the basis' classes");
    *tot = jk_rowbins_tasks(rb, n_ij);
    const int blocks = (int)std::min<long long>((n_ij + 256) / 256, (long long)b->nsm * 4);
    if (seg) jk_rowbins_seg_kernel<<<blocks, 256, 0, st>>>(rb, n_ij, b->d_qoff1, b->d_task01, *seg, dst);
    else jk_rowbins_kernel<<<blocks, 256, 0, st>>>(rb, n_ij, b->d_qoff1, b->d_task01);
    CUDA_TRY(cudaGetLastError());
    return JK_OK;
}

extern "C" int jk_class_pair_tasks(const int* bins_ij, const int* bins_kl, int nbins, int n_ij, int diag,
                                   long long* qoff, long long* total) {
    if (!bins_ij || !bins_kl || nbins <= 0 || nbins > JK_ROWBINS_MAX || n_ij < 0 || !total)
        return set_err(JK_ERR_ARG, "jk_class_pair_tasks: invalid arguments");
    JKRowBins rb;
    rb.nbins = nbins;
    rb.diag = diag ? 1 : 0;
    for (int s = 0; s <= nbins; s++) {
        rb.ij[s] = bins_ij[s];
        rb.kl[s] = bins_kl[s];
        if (s && (bins_ij[s] < bins_ij[s - 1] || bins_kl[s] < bins_kl[s - 1]))
            return set_err(JK_ERR_ARG, "bins must not decrease");
    }
    if (qoff)
        for (int r = 0; r <= n_ij; r++) qoff[r] = jk_rowbins_tasks(rb, r);
    *total = jk_rowbins_tasks(rb, n_ij);
    return JK_OK;
}

extern "C" int jk_build_class_pair(jk_basis_t* b, double* vj, double* vk, const double* dm, int nao, int n_dm,
                                   const int* bins_locs_ij, const int* bins_locs_kl, int nbins, int cp_ij,
                                   int cp_kl, void* stream) {
    if (!b || !dm || !bins_locs_ij || !bins_locs_kl || nbins <= 0) return set_err(JK_ERR_ARG, "invalid arguments");
    if (nao != b->nao) return set_err(JK_ERR_ARG, "nao %d does not match the basis (%d)", nao, b->nao);
    if (cp_ij < 0 || cp_ij >= b->ncp || cp_kl < 0 || cp_kl > cp_ij) return set_err(JK_ERR_ARG, "bad class pair");
    if (!vj && !vk) return JK_OK;
    cudaStream_t st = (cudaStream_t)stream;
    int n_ij = b->h_pair_locs[cp_ij + 1] - b->h_pair_locs[cp_ij];
    // kl bin kb pairs with ij in [bins_ij[0], bins_ij[nbins - kb]) (nr_jk_driver.cu:252-280):
    // row ij (in bin sij) keeps kl < bins_kl[nbins - sij]; diagonal classes keep kl <= ij
    jk_launch_fn fn = g_tabs.pair[class_index(b, cp_ij, cp_kl)];
    if (!fn) return set_err(JK_ERR_UNSUPPORTED, "no kernel for this class pair");
    JKRowBins rb;
    int rc = row_bins(bins_locs_ij, bins_locs_kl, nbins, cp_ij == cp_kl, &rb);
    if (rc) return rc;
    if (n_dm <= 0) return JK_OK;  // no densities (the launchers take n_dm <= 1 as one)
    JKSeg seg;
    fill_seg(b, cp_ij, cp_kl, b->d_qoff1, n_ij, dm, n_dm, vj, vk, &seg);
    long long tot = 0;
    const int* erank;
    int chunk;
    if (jk_internal_pair_runs(b, cp_ij, cp_kl, &seg, b->d_ehi1, b->d_qoff1, &erank, &chunk)) {
        const JKRowBinsCols cols{rb, seg.pst_kl};
        if (n_ij == 0 || seg.pst_kl == 0) return JK_OK;
        if (n_ij <= JK_PAIR_PREP_ROWS) {
            jk_pair_prep_kernel<<<1, jk_pair_prep_threads(seg.nrun), 0, st>>>(cols, seg, b->d_seg1, erank, chunk, b->d_ehi1, b->d_qoff1,
                                                    b->d_task01);
            CUDA_TRY(cudaGetLastError());
        } else {
            jk_run_rowbins_kernel<<<(n_ij + 255) / 256, 256, 0, st>>>(cols, n_ij, erank, b->d_ehi1);
            CUDA_TRY(cudaGetLastError());
            rc = jk_internal_run_items(seg, chunk, b->d_task01, b->d_seg1, st);
        }
        tot = (long long)seg.nrun * ((seg.pst_kl + chunk - 1) / chunk);
    } else {
        rc = class_pair_rows(b, rb, n_ij, &seg, b->d_seg1, st, &tot);
    }
    if (rc) return rc;
    return jk_internal_launch(b, cp_ij, cp_kl, b->d_seg1, b->d_task01, tot, n_dm, stream);
}

// ERI tensor of one class pair (jk_generic.cu)
cudaError_t jk_launch_fill(const JKSeg& seg, const long long* task0, long long max_tasks, int nsm, double* eri,
                           const long long* strides, const int* offsets, cudaStream_t st);

extern "C" int jk_fill_int2e(jk_basis_t* b, double* eri, int nao, const int* strides, const int* ao_offsets,
                             const int* bins_locs_ij, const int* bins_locs_kl, int nbins, int cp_ij, int cp_kl,
                             void* stream) {
    if (!b || !eri || !strides || !ao_offsets || !bins_locs_ij || !bins_locs_kl || nbins <= 0)
        return set_err(JK_ERR_ARG, "jk_fill_int2e: invalid arguments");
    if (nao != b->nao) return set_err(JK_ERR_ARG, "nao %d does not match the basis (%d)", nao, b->nao);
    // any two class pairs (the two-centre metric of int3c.get_int2c pairs
    // auxiliary classes in both orders)
    if (cp_ij < 0 || cp_ij >= b->ncp || cp_kl < 0 || cp_kl >= b->ncp) return set_err(JK_ERR_ARG, "bad class pair");
    cudaStream_t st = (cudaStream_t)stream;
    long long s64[4];
    int off[4];
    for (int a = 0; a < 4; a++) {
        s64[a] = strides[a];
        off[a] = ao_offsets[a];
    }
    // The templated kernels exist for classes with the bra class not below the
    // ket class; (ij|kl) = (kl|ij), so the other order runs as the swapped one
    // instead of on the generic kernel (16 of the 24 (ij|P) class pairs of
    // (H2O)8 / cc-pVDZ: 6.2 of its 6.3 ms).  The bins keep the same quartets
    // either way round when both start at pair 0.
    const int *bij = bins_locs_ij, *bkl = bins_locs_kl;
    if (!g_tabs.fill[class_index(b, cp_ij, cp_kl)] && g_tabs.fill[class_index(b, cp_kl, cp_ij)] && bij[0] == 0 &&
        bkl[0] == 0) {
        std::swap(cp_ij, cp_kl);
        std::swap(bij, bkl);
        for (int a = 0; a < 2; a++) {
            std::swap(s64[a], s64[a + 2]);
            std::swap(off[a], off[a + 2]);
        }
    }
    const int n_ij = b->h_pair_locs[cp_ij + 1] - b->h_pair_locs[cp_ij];
    // kl bin kb pairs with ij in [bins_ij[0], bins_ij[nbins - kb]): row ij (in
    // bin sij) keeps kl < bins_kl[nbins - sij] (nr_fill_ao_ints.cu:519-545)
    JKRowBins rb;
    long long tot = 0;
    int rc = row_bins(bij, bkl, nbins, 0, &rb);
    if (!rc) rc = class_pair_rows(b, rb, n_ij, nullptr, nullptr, st, &tot);
    if (rc) return rc;
    JKSeg seg;
    fill_seg(b, cp_ij, cp_kl, b->d_qoff1, n_ij, nullptr, 0, nullptr, nullptr, &seg);
    CUDA_TRY(jk_launch_fill(seg, b->d_task01, tot, b->nsm, eri, s64, off, st));
    return JK_OK;
}

// ---------------------------------------------------------------------------
// Expansion of the dense ERI tensor from its canonical class pairs (entry
// jk_expand_int2e): group(a) >= group(b), group(c) >= group(d), class pair of
// (a, b) >= that of (c, d).  Two passes, each reading and writing whole rows
// of tiles: the eight permuted copies of every block that this replaces moved
// the tensor one strided element at a time (1.0 of the 1.5 ms of GPU time of
// the (H2O)2 / cc-pVDZ tensor, and 168 launches).
// ---------------------------------------------------------------------------
__device__ __forceinline__ int jk_group_of(const int* __restrict__ gao, int ng, int a) {
    int lo = 0, hi = ng - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (gao[mid] <= a) lo = mid; else hi = mid - 1;
    }
    return lo;
}
__device__ __forceinline__ long long jk_class_of(int g, int h) {
    const long long x = max(g, h), y = min(g, h);
    return x * (x + 1) / 2 + y;
}
// pass 1: both orders of (a, b) and of (c, d) where class(ab) >= class(cd);
// block: plane (a, b) (blockIdx.x), a 32 x 32 tile of (c, d) (blockIdx.y)
__global__ void __launch_bounds__(256) jk_expand1_kernel(double* __restrict__ eri, int n, const int* __restrict__ gao,
                                                         int ng) {
    __shared__ double t1[32][33], t2[32][33];
    __shared__ int gc[32], gd[32];
    const int nt = (n + 31) / 32;
    const int a = blockIdx.x / n, b = blockIdx.x - a * n;
    const int c0 = blockIdx.y / nt * 32, d0 = blockIdx.y % nt * 32;
    const int x = threadIdx.x & 31, y0 = threadIdx.x >> 5;
    const int ga = jk_group_of(gao, ng, a), gb = jk_group_of(gao, ng, b);
    const size_t n2 = (size_t)n * n;
    const size_t src = (ga >= gb ? (size_t)a * n + b : (size_t)b * n + a) * n2, dst = ((size_t)a * n + b) * n2;
    if (threadIdx.x < 32) gc[x] = c0 + x < n ? jk_group_of(gao, ng, c0 + x) : 0;
    else if (threadIdx.x < 64) gd[x] = d0 + x < n ? jk_group_of(gao, ng, d0 + x) : 0;
    for (int y = y0; y < 32; y += 8) {
        if (c0 + y < n && d0 + x < n) t1[y][x] = eri[src + (size_t)(c0 + y) * n + d0 + x];
        if (d0 + y < n && c0 + x < n) t2[y][x] = eri[src + (size_t)(d0 + y) * n + c0 + x];
    }
    __syncthreads();
    const long long p = jk_class_of(ga, gb);
    for (int y = y0; y < 32; y += 8) {
        if (c0 + y >= n || d0 + x >= n) continue;
        const bool up = gc[y] >= gd[x];
        if (p < jk_class_of(gc[y], gd[x]) || (ga >= gb && up)) continue;  // pass 2, or canonical itself
        eri[dst + (size_t)(c0 + y) * n + d0 + x] = up ? t1[y][x] : t2[x][y];
    }
}
// pass 2: (ab|cd) = (cd|ab) where class(ab) < class(cd); block: (a, c)
// (blockIdx.x), a 32 x 32 tile of (b, d) (blockIdx.y)
__global__ void __launch_bounds__(256) jk_expand2_kernel(double* __restrict__ eri, int n, const int* __restrict__ gao,
                                                         int ng) {
    __shared__ double t[32][33];
    __shared__ int gb[32], gd[32];
    const int nt = (n + 31) / 32;
    const int a = blockIdx.x / n, c = blockIdx.x - a * n;
    const int b0 = blockIdx.y / nt * 32, d0 = blockIdx.y % nt * 32;
    const int x = threadIdx.x & 31, y0 = threadIdx.x >> 5;
    const int ga = jk_group_of(gao, ng, a), gc = jk_group_of(gao, ng, c);
    const size_t n2 = (size_t)n * n;
    if (threadIdx.x < 32) gb[x] = b0 + x < n ? jk_group_of(gao, ng, b0 + x) : 0;
    else if (threadIdx.x < 64) gd[x] = d0 + x < n ? jk_group_of(gao, ng, d0 + x) : 0;
    __syncthreads();
    for (int y = y0; y < 32; y += 8)  // rows d, columns b
        if (d0 + y < n && b0 + x < n && jk_class_of(ga, gb[x]) < jk_class_of(gc, gd[y]))
            t[y][x] = eri[((size_t)c * n + d0 + y) * n2 + (size_t)a * n + b0 + x];
    __syncthreads();
    for (int y = y0; y < 32; y += 8)  // rows b, columns d
        if (b0 + y < n && d0 + x < n && jk_class_of(ga, gb[y]) < jk_class_of(gc, gd[x]))
            eri[((size_t)a * n + b0 + y) * n2 + (size_t)c * n + d0 + x] = t[x][y];
}

extern "C" int jk_expand_int2e(jk_basis_t* b, double* eri, int nao, void* stream) {
    if (!b || !eri) return set_err(JK_ERR_ARG, "jk_expand_int2e: invalid arguments");
    if (nao != b->nao) return set_err(JK_ERR_ARG, "nao %d does not match the basis (%d)", nao, b->nao);
    if ((long long)nao * nao > 0x7fffffffLL || (nao + 31) / 32 > 255)
        return set_err(JK_ERR_ARG, "jk_expand_int2e: nao %d too large", nao);
    cudaStream_t st = (cudaStream_t)stream;
    const unsigned nt = (nao + 31) / 32;
    const dim3 g(nao * nao, nt * nt);
    jk_expand1_kernel<<<g, 256, 0, st>>>(eri, nao, b->d_group_ao, b->ngroups);
    jk_expand2_kernel<<<g, 256, 0, st>>>(eri, nao, b->d_group_ao, b->ngroups);
    CUDA_TRY(cudaGetLastError());
    return JK_OK;
}

// row-major C[M,N] = alpha op(A) op(B) + beta C through column-major cuBLAS
static cublasStatus_t gemm_rm(cublasHandle_t h, bool ta, bool tb, int M, int N, int K, double alpha,
                              const double* A, int lda, const double* B, int ldb, double beta, double* C, int ldc) {
    return cublasDgemm(h, tb ? CUBLAS_OP_T : CUBLAS_OP_N, ta ? CUBLAS_OP_T : CUBLAS_OP_N, N, M, K, &alpha, B, ldb,
                       A, lda, &beta, C, ldc);
}

#define BLAS_TRY(x)                                                              \
    do {                                                                         \
        cublasStatus_t s_ = (x);                                                 \
        if (s_ != CUBLAS_STATUS_SUCCESS) return set_err(JK_ERR_CUDA, "%s: cublas status %d", #x, (int)s_); \
    } while (0)

extern "C" int jk_get_jk(jk_basis_t* b, const double* coeff, int nao0, const double* dm0, int n_dm, double* vj0,
                         double* vk0, const jk_opts_t* opts, void* stream) {
    if (!b || !coeff || !dm0 || n_dm <= 0 || nao0 <= 0) return set_err(JK_ERR_ARG, "jk_get_jk: invalid arguments");
    cudaStream_t st = (cudaStream_t)stream;
    int nao = b->nao;
    size_t nn = (size_t)nao * nao * n_dm, nt = (size_t)nao * nao0 * n_dm;
    size_t need = 5 * nn + 2 * nt;
    int rc = grow(b, &b->d_work, &b->work_cap, need);
    if (rc) return rc;
    if (!b->blas) BLAS_TRY(cublasCreate(&b->blas));
    BLAS_TRY(cublasSetStream(b->blas, st));
    double* dms = b->d_work;
    double* vjw = dms + nn;
    double* vkw = vjw + nn;
    double* sym = vkw + nn;      // J, then K
    double* tmp = sym + 2 * nn;  // 2 n_dm x (nao x nao0)
    // dms = C D C^T (cuobc/scf/hf.py:73-74)
    for (int m = 0; m < n_dm; m++) {
        const double* D = dm0 + (size_t)m * nao0 * nao0;
        BLAS_TRY(gemm_rm(b->blas, false, false, nao, nao0, nao0, 1.0, coeff, nao0, D, nao0, 0.0, tmp, nao0));
        BLAS_TRY(gemm_rm(b->blas, false, true, nao, nao, nao0, 1.0, tmp, nao0, coeff, nao0, 0.0,
                         dms + (size_t)m * nao * nao, nao));
    }
    if (!vj0 && !vk0) return JK_OK;
    double* v0 = vj0 ? vjw : vkw;  // the outputs lie together
    const size_t nv = vj0 && vk0 ? 2 * nn : nn;
    CUDA_TRY(cudaMemsetAsync(v0, 0, sizeof(double) * nv, st));
    rc = jk_guard([&] { return build(b, dms, n_dm, vj0 ? vjw : nullptr, vk0 ? vkw : nullptr, true, opts, stream); });
    if (rc) return rc;
    // J = 2 C^T (V + V^T) C, K = C^T (V + V^T) C (cuobc/scf/hf.py:171-181):
    // one symmetrisation, one product with C from the right for all matrices
    const int nmat = (int)(nv / nn) * n_dm;
    jk_symmetrize_kernel<<<b->nsm * 4, 256, 0, st>>>(v0, sym, nao, nmat, vj0 ? n_dm : 0);
    CUDA_TRY(cudaGetLastError());
    BLAS_TRY(gemm_rm(b->blas, false, false, nmat * nao, nao0, nao, 1.0, sym, nao, coeff, nao0, 0.0, tmp, nao0));
    for (int m = 0; m < nmat; m++) {
        double* out = vj0 && m < n_dm ? vj0 + (size_t)m * nao0 * nao0
                                      : vk0 + (size_t)(vj0 ? m - n_dm : m) * nao0 * nao0;
        BLAS_TRY(gemm_rm(b->blas, true, false, nao0, nao0, nao, 1.0, coeff, nao0, tmp + (size_t)m * nao * nao0, nao0,
                         0.0, out, nao0));
    }
    return JK_OK;
}

// ---------------------------------------------------------------------------
// introspection for the bench and the tests
// ---------------------------------------------------------------------------
// per class quartet: cp_ij, cp_kl, li, lj, lk, ll, nprim_ij, nprim_kl
extern "C" int jk_basis_cq_info(const jk_basis_t* b, int* out) {
    if (!b || !out) return set_err(JK_ERR_ARG, "jk_basis_cq_info: invalid arguments");
    for (int c = 0; c < b->ncq; c++) {
        const JKScreenCQ& cq = b->h_cq[c];
        int* o = out + 8 * c;
        o[0] = cq.cp_ij;
        o[1] = cq.cp_kl;
        o[2] = b->h_group_l[cq.gi];
        o[3] = b->h_group_l[cq.gj];
        o[4] = b->h_group_l[cq.gk];
        o[5] = b->h_group_l[cq.gl];
        o[6] = b->h_group_nprim[cq.gi] * b->h_group_nprim[cq.gj];
        o[7] = b->h_group_nprim[cq.gk] * b->h_group_nprim[cq.gl];
    }
    return JK_OK;
}

// screened contracted-quartet counts of the last jk_build, per class quartet
extern "C" int jk_last_counts(const jk_basis_t* b, long long* out, void* stream) {
    if (!b || !out) return set_err(JK_ERR_ARG, "jk_last_counts: invalid arguments");
    if (b->ncq == 0) return JK_OK;
    std::vector<long long> t(2 * (size_t)b->ncq), t32(2 * (size_t)b->ncq);
    CUDA_TRY(cudaMemcpyAsync(t.data(), b->d_task0, sizeof(long long) * t.size(), cudaMemcpyDeviceToHost,
                             (cudaStream_t)stream));
    CUDA_TRY(cudaMemcpyAsync(t32.data(), b->d_task032, sizeof(long long) * t32.size(), cudaMemcpyDeviceToHost,
                             (cudaStream_t)stream));
    CUDA_TRY(cudaStreamSynchronize((cudaStream_t)stream));
    // FP64 quartets in out[0..ncq), FP32 quartets (mixed mode) in out[ncq..2 ncq)
    for (int c = 0; c < b->ncq; c++) {
        out[c] = t[2 * c + 1];
        out[b->ncq + c] = t32[2 * c + 1];
    }
    return JK_OK;
}

// FMA-pipe peak: 8 independent FMA chains per thread, whole device
template <typename T>
__global__ void jk_fma_peak_kernel(T* out, int iters) {
    T a[8];
#pragma unroll
    for (int k = 0; k < 8; k++) a[k] = (T)(threadIdx.x * 1e-7 + k);
    const T b = (T)0.9999999, c = (T)1e-7;
    for (int i = 0; i < iters; i++) {
#pragma unroll
        for (int u = 0; u < 16; u++) {
#pragma unroll
            for (int k = 0; k < 8; k++) a[k] = fma(a[k], b, c);
        }
    }
    T s = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) s += a[k];
    if (s == (T)-1) out[0] = s;  // keeps the chains alive
}

extern "C" int jk_fma_peak(int fp32, double* tflops) {
    if (!tflops) return set_err(JK_ERR_ARG, "jk_fma_peak: null output");
    int dev, nsm;
    CUDA_TRY(cudaGetDevice(&dev));
    CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    void* buf;
    CUDA_TRY(cudaMalloc(&buf, 16));
    cudaEvent_t e0, e1;
    CUDA_TRY(cudaEventCreate(&e0));
    CUDA_TRY(cudaEventCreate(&e1));
    const int iters = 4096, threads = 256, blocks = nsm * 8;
    double best = 0;
    for (int rep = 0; rep < 4; rep++) {
        CUDA_TRY(cudaEventRecord(e0));
        if (fp32) jk_fma_peak_kernel<float><<<blocks, threads>>>((float*)buf, iters);
        else jk_fma_peak_kernel<double><<<blocks, threads>>>((double*)buf, iters);
        CUDA_TRY(cudaEventRecord(e1));
        CUDA_TRY(cudaEventSynchronize(e1));
        float ms;
        CUDA_TRY(cudaEventElapsedTime(&ms, e0, e1));
        double flops = 2.0 * 8 * 16 * (double)iters * threads * blocks;
        if (rep > 0 && flops / (ms * 1e-3) / 1e12 > best) best = flops / (ms * 1e-3) / 1e12;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(buf);
    *tflops = best;
    return JK_OK;
}

// device evaluation of the Rys tables and the Boys functions at a batch of
// points, through the functions that the kernels call (modes in byteqc_jk.h)
template <int N>
__global__ void jk_rys_eval_kernel(const double* rys, const double* x, int count, double* s, double* w, int mode) {
    extern __shared__ __align__(16) double tab[];
    if (mode == 3 || mode == 4) rys_table_copy_f<N>(rys, reinterpret_cast<float*>(tab));
    else if (mode == 7) {
        if constexpr (N <= 4) boys_table_copy<N - 1>(rys, tab);
    } else rys_table_copy<N>(rys, tab);
    __syncthreads();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    if (mode == 3) {
        if constexpr (N <= JK_F32_ROOTS) {
            float rs[N], rw[N];
            rys_table_all_f<N>(reinterpret_cast<const float*>(tab), (float)x[i], rs, rw);
            for (int r = 0; r < N; r++) {
                s[i * N + r] = rs[r];
                w[i * N + r] = rw[r];
            }
        }
    } else if (mode == 4) {
        if constexpr (N <= JK_F32_ROOTS) {
            for (int r = 0; r < N; r++) {
                float rs, rw;
                rys_root_one_f<N>(reinterpret_cast<const float*>(tab), (float)x[i], r, rs, rw);
                s[i * N + r] = rs;
                w[i * N + r] = rw;
            }
        }
    } else if (mode == 7) {
        if constexpr (N <= 4) {
            double F[N];
            boys_all<N - 1>(tab, x[i], F);
            for (int r = 0; r < N; r++) s[i * N + r] = w[i * N + r] = F[r];
        }
    } else if (mode == 0 || mode == 6) {
        double rs[N], rw[N];
        if (mode == 0) rys_roots_all<N>(tab, x[i], rs, rw);
        else rys_table_all<N>(tab, x[i], rs, rw);
        for (int r = 0; r < N; r++) {
            s[i * N + r] = rs[r];
            w[i * N + r] = rw[r];
        }
    } else {
        for (int r = 0; r < N; r++) {
            if (mode == 1) rys_root_one<N>(tab, x[i], r, s[i * N + r], w[i * N + r]);
            else if (mode == 5) rys_root_rt(rys, N, x[i], r, s[i * N + r], w[i * N + r]);
            else rys_root<N>(rys, x[i], r, s[i * N + r], w[i * N + r]);
        }
    }
}

template <int N>
static cudaError_t rys_eval_launch(const double* rys, const double* x, int count, double* s, double* w, int mode,
                                   cudaStream_t st) {
    const size_t smem = std::max<size_t>(RysS<N>::TWORDS, N <= 4 ? (size_t)BoysS::WORDS : 0) * sizeof(double);
    cudaError_t e = cudaFuncSetAttribute(jk_rys_eval_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    jk_rys_eval_kernel<N><<<(count + 127) / 128, 128, smem, st>>>(rys, x, count, s, w, mode);
    return cudaGetLastError();
}

extern "C" int jk_rys_roots_device(int n, const double* x, int count, double* s, double* w, int mode, void* stream) {
    if (n < 1 || n > RYS_NMAX || !x || !s || !w || count < 0 || mode < 0 || mode > 7 ||
        ((mode == 3 || mode == 4) && n > JK_F32_ROOTS) || (mode == 7 && n > 4))
        return set_err(JK_ERR_ARG, "jk_rys_roots_device: bad args");
    if (count == 0) return JK_OK;
    const double* rys;
    int rc = rys_table_device(&rys);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t e;
    switch (n) {
        case 1: e = rys_eval_launch<1>(rys, x, count, s, w, mode, st); break;
        case 2: e = rys_eval_launch<2>(rys, x, count, s, w, mode, st); break;
        case 3: e = rys_eval_launch<3>(rys, x, count, s, w, mode, st); break;
        case 4: e = rys_eval_launch<4>(rys, x, count, s, w, mode, st); break;
        case 5: e = rys_eval_launch<5>(rys, x, count, s, w, mode, st); break;
        case 6: e = rys_eval_launch<6>(rys, x, count, s, w, mode, st); break;
        case 7: e = rys_eval_launch<7>(rys, x, count, s, w, mode, st); break;
        case 8: e = rys_eval_launch<8>(rys, x, count, s, w, mode, st); break;
        case 9: e = rys_eval_launch<9>(rys, x, count, s, w, mode, st); break;
        case 10: e = rys_eval_launch<10>(rys, x, count, s, w, mode, st); break;
        case 11: e = rys_eval_launch<11>(rys, x, count, s, w, mode, st); break;
        case 12: e = rys_eval_launch<12>(rys, x, count, s, w, mode, st); break;
        default: e = rys_eval_launch<13>(rys, x, count, s, w, mode, st); break;
    }
    CUDA_TRY(e);
    return JK_OK;
}

// ---------------------------------------------------------------------------
// internal helpers for the other translation units
// ---------------------------------------------------------------------------
int jk_internal_set_err(int code, const char* msg) { return set_err(code, "%s", msg); }

cudaError_t jk_internal_uploaded() { return cudaStreamSynchronize(cudaStreamLegacy); }

int jk_internal_class_info(const jk_basis_t* b, int cp_ij, int cp_kl, int* n_ij, int* n_kl, int* nao) {
    if (!b || cp_ij < 0 || cp_ij >= b->ncp || cp_kl < 0 || cp_kl > cp_ij)
        return set_err(JK_ERR_ARG, "bad class pair (%d, %d)", cp_ij, cp_kl);
    *n_ij = b->h_pair_locs[cp_ij + 1] - b->h_pair_locs[cp_ij];
    *n_kl = b->h_pair_locs[cp_kl + 1] - b->h_pair_locs[cp_kl];
    *nao = b->nao;
    return JK_OK;
}

void jk_internal_fill_seg(const jk_basis_t* b, int cp_ij, int cp_kl, const long long* qoff, int n_ij,
                          const double* dm, int n_dm, double* vj, double* vk, JKSeg* out) {
    fill_seg(b, cp_ij, cp_kl, qoff, n_ij, dm, n_dm, vj, vk, out);
}

int jk_internal_launch(const jk_basis_t* b, int cp_ij, int cp_kl, const JKSeg* d_seg, const long long* task0,
                       long long max_tasks, int n_dm, void* stream) {
    jk_launch_fn fn = g_tabs.pair[class_index(b, cp_ij, cp_kl)];
    if (!fn) return set_err(JK_ERR_UNSUPPORTED, "no kernel for class pair (%d, %d)", cp_ij, cp_kl);
    CUDA_TRY(fn(d_seg, task0, 1, max_tasks, n_dm, b->nsm, JKBatchCfg{nullptr, 0, 1}, (cudaStream_t)stream));
    return JK_OK;
}

bool jk_internal_pair_runs(const jk_basis_t* b, int cp_ij, int cp_kl, JKSeg* seg, int* ehi, long long* ioff,
                           const int** erank, int* chunk) {
    *chunk = g_tabs.run[class_index(b, cp_ij, cp_kl)];
    if (!*chunk) return false;
    const int v = run_level(b, cp_ij, seg->pst_kl, *chunk, JK_RUN_LEVELS_PAIR, JK_RUN_ITEMS_PAIR);
    seg->nrun = b->h_nrun[v][cp_ij];
    seg->ent = b->d_ent + b->h_pair_locs[cp_ij];
    seg->run0 = b->d_run0 + b->h_run_off[v][cp_ij];
    seg->ehi = ehi;
    seg->ioff = ioff;
    *erank = b->d_erank + b->h_pair_locs[cp_ij];
    return true;
}

int jk_internal_run_items(const JKSeg& seg, int chunk, long long* itm, JKSeg* d_seg, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    long long* ioff = const_cast<long long*>(seg.ioff);
    jk_run_items_kernel<<<(seg.nrun + 255) / 256, 256, 0, st>>>(seg, chunk, ioff);
    jk_run_scan1_kernel<<<1, 1024, 0, st>>>(seg, ioff, itm, d_seg);
    CUDA_TRY(cudaGetLastError());
    return JK_OK;
}

int jk_internal_class_index(const jk_basis_t* b, int cp_ij, int cp_kl) { return class_index(b, cp_ij, cp_kl); }

jk_launch_fn jk_internal_launcher(int class_idx, int fp32) {
    init_tables();
    return fp32 ? g_tab32[class_idx] : g_tab64[class_idx];
}

jk_launch_fn jk_internal_pair_launcher(int class_idx) {
    init_tables();
    return g_tabs.pair[class_idx];
}

int jk_internal_class_runs(int class_idx) {
    init_tables();
    return g_tabs.run[class_idx];
}

int jk_internal_class_team(int class_idx) {
    init_tables();
    return g_tabs.team[class_idx];
}

jk_fill_fn jk_internal_fill_launcher(int class_idx) {
    init_tables();
    return g_tabs.fill[class_idx];
}

void jk_internal_fill_seg_cq(const jk_basis_t* b, const JKScreenCQ& cq, int fp32, JKSeg* out) {
    fill_seg(b, cq.cp_ij, cq.cp_kl, cq.runs ? nullptr : (fp32 ? cq.qoff32 : cq.qoff), cq.n_ij, nullptr, 0, nullptr,
             nullptr, out);
    if (cq.runs) {
        out->nrun = cq.nrun;
        out->ent = cq.ent;
        out->run0 = cq.run0;
        out->elo = fp32 ? cq.klb : nullptr;
        out->ehi = fp32 ? cq.kle : cq.klb;
        out->ioff = fp32 ? cq.ioff32 : cq.ioff;
    } else if (fp32) {
        out->kl_base = cq.klb;
    }
}

int jk_internal_screen_set(const jk_basis_t* b, JKScreenSet* out) {
    // doubles and 64-bit words first, then the ints
    const size_t w = b->zero_bytes / 8 + 2 * (size_t)b->qoff_total + (size_t)b->ioff_total;
    CUDA_TRY(cudaMalloc(&out->mem, 8 * w + 2 * sizeof(int) * (size_t)b->ent_total + 8));
    out->zero = out->mem;
    out->dm_cond = (double*)out->mem;
    long long* counts = (long long*)(out->dm_cond + (size_t)b->ngroups * b->ngroups);
    long long *qoff = (long long*)((char*)out->mem + b->zero_bytes), *qoff32 = qoff + b->qoff_total,
              *ioff = qoff32 + b->qoff_total;
    int *klb = (int*)(ioff + b->ioff_total), *kle = klb + b->ent_total;
    out->cq = b->h_cq;
    for (JKScreenCQ& q : out->cq) {
        q.dm_cond = out->dm_cond;
        q.qoff = qoff + (q.qoff - b->d_qoff);
        q.qoff32 = qoff32 + (q.qoff32 - b->d_qoff32);
        q.ioff = ioff + (q.ioff - b->d_ioff);
        q.ioff32 = ioff + (q.ioff32 - b->d_ioff);
        q.klb = klb + (q.klb - b->d_klb);
        q.kle = kle + (q.kle - b->d_kle);
        q.task0 = counts + (q.task0 - b->d_task0);
        q.task032 = counts + (q.task032 - b->d_task0);
        q.itm = counts + (q.itm - b->d_task0);
        q.itm32 = counts + (q.itm32 - b->d_task0);
    }
    return JK_OK;
}

// pack record of one molecule: dens holds 2 n_dm packed densities (dp, dpb),
// acc as many accumulators (jp, jpb)
JKPackMol jk_internal_pack_mol(const jk_basis_t* b, const double* dm, int n_dm, double* dens, double* acc, double* vj) {
    const size_t n = (size_t)n_dm * b->pack_total;
    return JKPackMol{b->d_pack, b->ncp, b->pack_total, b->d_pair2bra, b->d_pair2ket, b->d_ao_loc, b->d_inv,
                     dm,        b->nao, n_dm,          dens,          dens + n,      acc,         acc + n,  vj,
                     nullptr,   nullptr};
}

int jk_internal_pack_batch(const JKPackMol* d_mols, int nmol, long long max_total, int mode, void* stream) {
    if (nmol <= 0) return JK_OK;
    const unsigned bx = (unsigned)std::max(1LL, std::min<long long>((max_total + 255) / 256, 64));
    jk_pack_batch_kernel<<<dim3(bx, nmol), 256, 0, (cudaStream_t)stream>>>(d_mols, mode);
    CUDA_TRY(cudaGetLastError());
    return JK_OK;
}

int jk_internal_screen(const JKScreenCQ* d_cq, int ncq, double tol, int nbins, int prescreen, double fp32_cutoff,
                       void* stream) {
    if (ncq <= 0) return JK_OK;
    cudaStream_t st = (cudaStream_t)stream;
    // enough blocks for a large class, few enough that small ones (their
    // surplus blocks leave at once) stay cheap: with 512 / 64 / 16 blocks, as it
    // was, and with these, two waters / cc-pVDZ (21 class quartets) take 206 and
    // 191 us, one water / TZVP (666) 1.42 and 1.37 ms, (H2O)64 / cc-pVDZ 98.4 ms both
    const unsigned by = ncq <= 64 ? 128 : (ncq <= 1024 ? 16 : 4);
    jk_screen_kernel<<<dim3(ncq, by), 256, 0, st>>>(d_cq, tol, nbins, prescreen, fp32_cutoff);
    jk_run_scan_kernel<<<ncq, 1024, 0, st>>>(d_cq);
    CUDA_TRY(cudaGetLastError());
    return JK_OK;
}

int jk_internal_dm_cond(const JKDmCond* d_mols, int nmol, int max_groups, int max_nao, void* stream) {
    if (nmol <= 0) return JK_OK;
    cudaStream_t st = (cudaStream_t)stream;
    jk_zero_kernel<<<nmol, 256, 0, st>>>(d_mols);
    const unsigned bx = std::min(16u, dm_cond_blocks(max_nao));
    jk_dm_cond_kernel<<<dim3(bx, max_groups, nmol), 256, 0, st>>>(JKDmCond{}, d_mols);
    CUDA_TRY(cudaGetLastError());
    return JK_OK;
}
