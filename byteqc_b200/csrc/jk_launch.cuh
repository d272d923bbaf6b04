// Launchers of the J/K kernels, one per (li, lj, lk, ll) class and arithmetic
// type, collected in a table indexed by JK_CLASS_INDEX(li, lj, lk, ll).
#pragma once
#include <atomic>

#include "jk_kernels.cuh"
#include "jk_teams.cuh"

// cudaFuncSetAttribute acts on the current device only, so the "already set"
// flag of a kernel is kept per device (bit d of `done` for device d < 64;
// devices beyond that set the attribute on every launch).
template <class K>
cudaError_t jk_smem_attr(K kernel, size_t smem, std::atomic<unsigned long long>& done) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
    if (bit && (done.load(std::memory_order_relaxed) & bit)) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess && bit) done.fetch_or(bit, std::memory_order_relaxed);
    return e;
}


// resident blocks per SM of a kernel at a launch shape, looked up once per
// device (bit d of `done`, the count in cnt[d])
template <class K>
int jk_resident_blocks(K kernel, int threads, size_t smem, std::atomic<unsigned long long>& done, int* cnt) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 1;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
    if (bit && (done.load(std::memory_order_acquire) & bit)) return cnt[dev];
    int nb = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, threads, smem) != cudaSuccess || nb < 1) nb = 1;
    if (bit) {
        cnt[dev] = nb;
        done.fetch_or(bit, std::memory_order_release);
    }
    return nb;
}

template <class C, typename R, bool MULTI, bool KROWS>
cudaError_t jk_launch_run(const JKSeg* segs, const long long* segt, int nseg, long long max_items, int n_dm, int nsm,
                          const JKBatchCfg& cfg, cudaStream_t st) {
    const size_t smem = MULTI ? jk_run_multi_smem<C>(n_dm) : JKRunShape<C>::SMEM;
    static std::atomic<unsigned long long> attr_done{0}, occ_done{0};
    static int occ[64];
    if (cudaError_t e = jk_smem_attr(jk_run_kernel<C, R, MULTI, KROWS>, MULTI ? JK_RUN_SMEM : smem, attr_done); e != cudaSuccess)
        return e;
    // resident grid (the most shared memory a MULTI launch may take)
    const long long res = (long long)nsm * jk_resident_blocks(jk_run_kernel<C, R, MULTI, KROWS>, JK_RUN_THREADS,
                                                              MULTI ? (size_t)JK_RUN_SMEM : smem, occ_done, occ);
    const long long want = (max_items + JK_RUN_THREADS / 32 - 1) / (JK_RUN_THREADS / 32);
    const int blocks = (int)(cfg.queue ? res * cfg.grid_mul : (want < res ? want : res));
    jk_run_kernel<C, R, MULTI, KROWS><<<blocks, JK_RUN_THREADS, smem, st>>>(segs, segt, nseg, cfg.queue, cfg.grab);
    return cudaGetLastError();
}

template <class C, typename R, bool MULTI, bool KROWS>
cudaError_t jk_launch_trun(const JKSeg* segs, const long long* segt, int nseg, long long max_items, int nsm,
                           const JKBatchCfg& cfg, cudaStream_t st) {
    constexpr size_t smem = JKTRunShape<C, R>::SMEM;
    static_assert(smem <= 227 * 1024, "team run kernel shared memory");
    static std::atomic<unsigned long long> attr_done{0}, occ_done{0};
    static int occ[64];
    if (cudaError_t e = jk_smem_attr(jk_trun_kernel<C, R, MULTI, KROWS>, smem, attr_done); e != cudaSuccess) return e;
    const long long res = (long long)nsm * jk_resident_blocks(jk_trun_kernel<C, R, MULTI, KROWS>, JK_RUN_THREADS, smem,
                                                              occ_done, occ);
    const long long want = (max_items + JK_RUN_THREADS / 32 - 1) / (JK_RUN_THREADS / 32);
    const int blocks = (int)(cfg.queue ? res * cfg.grid_mul : (want < res ? want : res));
    jk_trun_kernel<C, R, MULTI, KROWS><<<blocks, JK_RUN_THREADS, smem, st>>>(segs, segt, nseg, cfg.queue, cfg.grab);
    return cudaGetLastError();
}

// The segments of one class (for the team kernels: of one class and one pair
// of primitive counts), task or item prefix segt[0..nseg] on the device.
template <int LI, int LJ, int LK, int LL, typename R, bool KROWS>
cudaError_t jk_launch(const JKSeg* segs, const long long* segt, int nseg, long long max_tasks, int n_dm, int nsm,
                      const JKBatchCfg& cfg, cudaStream_t st) {
    using C = JKClass<LI, LJ, LK, LL>;
    if (max_tasks <= 0 || nseg <= 0) return cudaSuccess;
    if constexpr (C::P == 0) {
        if (n_dm > 1) return jk_launch_run<C, R, true, KROWS>(segs, segt, nseg, max_tasks, n_dm, nsm, cfg, st);
        return jk_launch_run<C, R, false, KROWS>(segs, segt, nseg, max_tasks, n_dm, nsm, cfg, st);
    } else if constexpr (C::TRUN) {
        if (n_dm > 1) return jk_launch_trun<C, R, true, KROWS>(segs, segt, nseg, max_tasks, nsm, cfg, st);
        return jk_launch_trun<C, R, false, KROWS>(segs, segt, nseg, max_tasks, nsm, cfg, st);
    } else {
        using S = JKTeamShape<C>;
        constexpr size_t smem = jk_team_smem<C, R>();
        static std::atomic<unsigned long long> attr_done{0};
        if (cudaError_t e = jk_smem_attr(jk_team_kernel<C, R>, smem, attr_done); e != cudaSuccess) return e;
        int blocks;
        if (cfg.queue) {
            static std::atomic<unsigned long long> occ_done{0};
            static int occ[64];
            blocks = nsm * cfg.grid_mul * jk_resident_blocks(jk_team_kernel<C, R>, S::THREADS, smem, occ_done, occ);
        } else {
            long long want = (max_tasks + S::QPB - 1) / S::QPB;
            long long cap = (long long)nsm * 8;
            blocks = (int)(want < cap ? want : cap);
        }
        jk_team_kernel<C, R><<<blocks, S::THREADS, smem, st>>>(segs, segt, nseg, cfg.queue, cfg.grab);
    }
    return cudaGetLastError();
}

// ERI-tensor fill of one class quartet with the class's templated kernel
// (thread or team shape, FP64), same grid as the J/K launch
template <int LI, int LJ, int LK, int LL>
cudaError_t jk_launch_fill_t(const JKSeg& seg, const long long* task0, long long max_tasks, int nsm,
                             const JKFillOut& out, cudaStream_t st) {
    using C = JKClass<LI, LJ, LK, LL>;
    if (max_tasks <= 0) return cudaSuccess;
    if constexpr (C::P == 0) {
        constexpr size_t smem = RysS<C::NROOTS>::WORDS * sizeof(double);
        static std::atomic<unsigned long long> attr_done{0};
        if (cudaError_t e = jk_smem_attr(jk_thread_fill_kernel<C>, smem, attr_done); e != cudaSuccess) return e;
        long long want = (max_tasks + 127) / 128;
        long long cap = (long long)nsm * 16;
        int blocks = (int)(want < cap ? want : cap);
        jk_thread_fill_kernel<C><<<blocks, 128, smem, st>>>(seg, task0, out);
    } else {
        using S = JKTeamShape<C>;
        constexpr size_t smem = jk_team_smem<C, double>();
        static std::atomic<unsigned long long> attr_done{0};
        if (cudaError_t e = jk_smem_attr(jk_team_fill_kernel<C>, smem, attr_done); e != cudaSuccess) return e;
        long long want = (max_tasks + S::QPB - 1) / S::QPB;
        long long cap = (long long)nsm * 8;
        int blocks = (int)(want < cap ? want : cap);
        jk_team_fill_kernel<C><<<blocks, S::THREADS, smem, st>>>(seg, task0, out);
    }
    return cudaGetLastError();
}
typedef cudaError_t (*jk_fill_fn)(const JKSeg& seg, const long long* task0, long long max_tasks, int nsm,
                                  const JKFillOut& out, cudaStream_t st);

// launcher tables indexed by JK_CLASS_INDEX(li, lj, lk, ll)
struct JKTables {
    // builds (the run kernels write K by rows, see JKRunItem), FP64 and FP32
    // parts; the per-class-pair entries (K in the layout of the C-ABI)
    jk_launch_fn t64[JK_NCLASS], t32[JK_NCLASS], pair[JK_NCLASS];
    // team kernels need one primitive count per launch (their blocks loop
    // over the primitives in step); run and generic kernels read it per
    // segment
    unsigned char team[JK_NCLASS];
    unsigned char run[JK_NCLASS];  // run kernels: ket pairs of an item (0: a row class, task prefix)
    jk_fill_fn fill[JK_NCLASS];  // templated ERI fill (classes up to f)
};

// classes with a shell above f: the generic kernel (jk_generic.cu)
void jk_register_generic(JKTables* T);

// per-instantiation-file registration (jk_inst_*.cu, generated list)
#include "jk_inst_list.h"

#ifndef JK_NO_FP32
#define JK_REG32(LI, LJ, LK, LL)                                         \
    T->t32[JK_CLASS_INDEX(LI, LJ, LK, LL)] = jk_launch<LI, LJ, LK, LL, float, true>;
#else
#define JK_REG32(LI, LJ, LK, LL)
#endif
#define JK_REG(LI, LJ, LK, LL)                                                       \
    T->team[JK_CLASS_INDEX(LI, LJ, LK, LL)] = !JKClass<LI, LJ, LK, LL>::RUNS;     \
    T->fill[JK_CLASS_INDEX(LI, LJ, LK, LL)] = jk_launch_fill_t<LI, LJ, LK, LL>;   \
    T->run[JK_CLASS_INDEX(LI, LJ, LK, LL)] = JKClass<LI, LJ, LK, LL>::RUNS ? JKClass<LI, LJ, LK, LL>::TPW : 0; \
    T->t64[JK_CLASS_INDEX(LI, LJ, LK, LL)] = jk_launch<LI, LJ, LK, LL, double, true>;  \
    T->pair[JK_CLASS_INDEX(LI, LJ, LK, LL)] =                                         \
        jk_launch<LI, LJ, LK, LL, double, !JKClass<LI, LJ, LK, LL>::RUNS>;            \
    JK_REG32(LI, LJ, LK, LL)
