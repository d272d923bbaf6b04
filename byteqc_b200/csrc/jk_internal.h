// Internal helpers of jk_host.cu shared with other translation units of
// libjk.so (not part of the C-ABI).
#pragma once
#include <cublas_v2.h>

#include <exception>
#include <map>
#include <string>
#include <tuple>
#include <vector>

#include "jk_common.cuh"
#include "../../include/byteqc_jk.h"

// One class quartet (cp_ij >= cp_kl) of one basis, as the screening kernels
// see it: pair counts, group indices and the device buffers they read/write.
// Classes of the run kernels (runs != 0) get per-entry ket bounds and an item
// prefix over their runs, the others a task prefix over their rows.
struct JKScreenCQ {
    int cp_ij, cp_kl;
    int gi, gj, gk, gl;
    int n_ij, n_kl;
    int ngroups;
    int runs, nrun;               // ket pairs of an item (0: row class), runs
    const double *lq_ij, *lq_kl;  // clipped log q of the two classes
    const double *rq_ij, *rq_kl;  // unclipped log q (mixed-precision split)
    const double* dm_cond;        // ngroups x ngroups
    // rows: prefixes of the FP64 and FP32 parts and the first FP32 column
    long long *qoff, *qoff32;
    int* klb;                     // (run classes: per entry, the end of the FP64 part)
    // runs: the run table, the end of the FP32 part per entry, item prefixes
    const int *ent, *erank, *run0;  // positions and ranks of the entries
    int bucket;                     // Schwarz ranks per bucket of the ket class
    int* kle;
    long long *ioff, *ioff32;
    long long *itm, *itm32;       // {0, items} of each part
    long long *task0, *task032;   // {0, quartets} of each part
    // host bookkeeping
    int pair_ij0, pair_kl0;
    int level;                    // run length of the table (JK_RUN_LEVELS)
};

int jk_internal_set_err(int code, const char* msg);
// status of a failed CUDA call, taken off the runtime's last error too: the
// check after the next call's launches would report it again
inline int jk_internal_cuda_err(cudaError_t e) {
    cudaGetLastError();
    return jk_internal_set_err(JK_ERR_CUDA, cudaGetErrorString(e));
}
// The body of a C entry that allocates on the host: an exception becomes a status.
template <class F>
int jk_guard(F&& body) {
    try {
        return body();
    } catch (const std::exception& e) {
        return jk_internal_set_err(JK_ERR_CUDA, e.what());
    }
}
// Waits until the tables that cudaMemcpy took from pageable memory lie on the
// device.  It may return with the last transfer still under way on the legacy
// stream, which a caller's non-blocking stream does not wait for; every function
// that uploads tables ends with this.
cudaError_t jk_internal_uploaded();
// pair counts of the two classes and the working-basis size
int jk_internal_class_info(const jk_basis_t* b, int cp_ij, int cp_kl, int* n_ij, int* n_kl, int* nao);
// Class kernel of the per-class-pair entries on the segment at d_seg (device).
// task0: {0, count} as the preparation kernels wrote it.
int jk_internal_launch(const jk_basis_t* b, int cp_ij, int cp_kl, const JKSeg* d_seg, const long long* task0,
                       long long max_tasks, int n_dm, void* stream);
// completes the segment of a run class (seg->nrun > 0 on return, its ehi and
// ioff in the caller's buffers) at the per-class-pair entries' run length, and
// gives the ranks of the run entries; false for a row class
bool jk_internal_pair_runs(const jk_basis_t* b, int cp_ij, int cp_kl, JKSeg* seg, int* ehi, long long* ioff,
                           const int** erank, int* chunk);
// for many bra pairs, in place of jk_pair_prep_kernel: item counts per run from
// the entries' ket ends, their exclusive prefix, itm = {0, total}, and the
// segment to *d_seg
int jk_internal_run_items(const JKSeg& seg, int chunk, long long* itm, JKSeg* d_seg, void* stream);
#define JK_PAIR_PREP_ROWS 8192  // bra pairs up to which one block prepares a call

// Side streams of the class launches.  Every class kernel adds into J and K
// with atomics, so launches of different class quartets (and the FP64 and
// FP32 parts of one) may run concurrently; spreading them over a few
// streams overlaps the ramp-up and tail of the many small launches of a
// build.  begin() forks from the caller's stream with an event, end() joins
// back (both record into a CUDA graph when the caller's stream is captured).
#define JK_SIDE_STREAMS 8
struct JKFanout {
    cudaStream_t s[JK_SIDE_STREAMS] = {};
    cudaEvent_t fork = nullptr;
    cudaEvent_t join[JK_SIDE_STREAMS] = {};
    cudaError_t init() {
        cudaError_t e = cudaEventCreateWithFlags(&fork, cudaEventDisableTiming);
        for (int i = 0; e == cudaSuccess && i < JK_SIDE_STREAMS; i++) {
            e = cudaStreamCreateWithFlags(&s[i], cudaStreamNonBlocking);
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&join[i], cudaEventDisableTiming);
        }
        return e;
    }
    // fork the first n streams from st, join them back
    cudaError_t begin(cudaStream_t st, int n = JK_SIDE_STREAMS) {
        cudaError_t e = cudaEventRecord(fork, st);
        for (int i = 0; e == cudaSuccess && i < n; i++) e = cudaStreamWaitEvent(s[i], fork, 0);
        return e;
    }
    cudaStream_t pick(int i) const { return s[i % JK_SIDE_STREAMS]; }
    cudaError_t end(cudaStream_t st, int n = JK_SIDE_STREAMS) {
        cudaError_t e = cudaSuccess;
        for (int i = 0; e == cudaSuccess && i < n; i++) {
            e = cudaEventRecord(join[i], s[i]);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(st, join[i], 0);
        }
        return e;
    }
    void destroy() {
        for (int i = 0; i < JK_SIDE_STREAMS; i++) {
            if (s[i]) cudaStreamDestroy(s[i]);
            if (join[i]) cudaEventDestroy(join[i]);
            s[i] = nullptr;
            join[i] = nullptr;
        }
        if (fork) cudaEventDestroy(fork);
        fork = nullptr;
    }
};

// one class pair in the pair-packed density / J buffers of jk_build
struct JKPackCls {
    long long off;      // first packed element of the class
    int np, nfi, nfj;   // pairs, Cartesian components of the two shells
    int pair0;          // first pair of the class
};

// one molecule of a batched pack / unpack of the pair-packed J side
struct JKPackMol {
    const JKPackCls* cls;
    int ncls;
    long long total;
    const int *pair2bra, *pair2ket, *ao_loc, *inv;
    const double* dm;
    int nao, n_dm;
    double *dp, *dpb;  // mode 0 output
    double *jp, *jpb;  // mode 1 input
    double* vj;        // mode 1 output
    // K of the run kernels by rows (n_dm x nao x nao, or null), added
    // transposed into vk after the launches
    const double* kt;
    double* vk;
};

// run lengths a run table exists for: long runs save more traffic, short ones
// give a small molecule enough items to fill the device.  The per-class-pair
// entries, whose launch has the device to itself, and contracted class quartets
// go down to single pairs.
#define JK_RUN_LEVELS 3
#define JK_RUN_LEVELS_PAIR 4
static const int JK_RUN_LEN[JK_RUN_LEVELS_PAIR] = {32, 8, 2, 1};

// Class launches of a set of class quartets: one key per class (for the team
// kernels per class and pair of primitive counts), its class quartets as
// segments of one launch.
struct JKPlanKey {
    int cls, np_ij, np_kl;                  // np_* = -1: any primitive count
    std::vector<std::pair<int, int>> segs;  // (molecule, class quartet)
    std::vector<long long> seg_tasks;       // unscreened quartets of each segment
    long long max_tasks = 0;                // their sum
    long long max_items = 0;                // bound of the launch's task or item count
    bool solo = false;                      // a class quartet launched on its own
    JKBatchCfg cfg[2] = {{nullptr, 0, 1}, {nullptr, 0, 1}};  // FP64 part, FP32 part (queue set at launch)
    float tuned_ms[2] = {-1.f, -1.f};
};
struct JKPlan {
    std::vector<JKPlanKey> keys;
    std::map<std::tuple<int, int, int>, int> index;  // key of a class while the plan is put together
    std::vector<int> key_off;  // nkeys + 1 segment offsets
    int nseg = 0;
    JKSeg* d_seg[2] = {nullptr, nullptr};        // FP64, FP32 parts
    long long* d_segt[2] = {nullptr, nullptr};   // task prefix per key: nseg + nkeys entries (keys of one
                                                 // segment use the screening's {0, count} itself)
    std::vector<const long long*> one[2];        // that pair per key, or null
    bool multi = false;                          // some key has several segments
    const long long** d_cnt[2] = {nullptr, nullptr};
    int* d_key_off = nullptr;
    void* mem = nullptr;                         // the tables' allocation
    unsigned long long* d_queue = nullptr;       // 2 work counters per key (persistent launches)
};
void jk_plan_free(JKPlan* p);
// adds class quartet c of basis b (molecule m) to its key
int jk_plan_add(JKPlan* p, const jk_basis* b, int m, int c, bool solo);
// orders the keys (merged ones first) and segments, uploads the tables;
// cqs[m]: the screening records of molecule m
int jk_plan_finish(JKPlan* p, const std::vector<jk_basis*>& mols, const std::vector<const JKScreenCQ*>& cqs);
// exclusive prefixes of the segments' task counts (after the screening)
int jk_plan_prefix(const JKPlan* p, bool mixed, cudaStream_t st);
// direct: the run kernels write K in the layout of the C-ABI (FP64 in both
// parts), otherwise by rows
int jk_plan_launch(const JKPlan* p, int k, int part, const JKBatchCfg& cfg, int n_dm, int nsm, cudaStream_t st,
                   bool direct = false);
// segment s of key k on its own, straight from the screening's counts
int jk_plan_launch_one(const JKPlan* p, int k, int s, int part, const JKScreenCQ& cq, int n_dm, int nsm,
                       cudaStream_t st, bool direct);

// Per-geometry state (opaque to callers of the C-ABI)
struct jk_basis {
    // class quartets and their screening records
    int device = 0, nsm = 148;
    const double* rys = nullptr;  // shared per-device Rys table
    int natm = 0, nbas = 0, nao = 0, ngroups = 0, ncp = 0, ncq = 0;
    double diag_fac = 0.5, cutoff = 1e-13;
    std::vector<int> h_ao_loc, h_group_off, h_group_l, h_group_nprim;
    std::vector<int> h_cls_gi, h_cls_gj, h_pair_locs, h_prim_locs, h_pair2bra, h_pair2ket;
    std::vector<double> h_log_q, h_log_q_raw, h_qcond;
    std::vector<JKScreenCQ> h_cq;
    std::vector<double> h_cq_cost;     // unscreened work of each class quartet (shard plans)
    std::vector<int> h_cq_owner;       // owner of each class quartet in the plan of
    int cq_owner_n = 0;                // cq_owner_n shards
    long long qoff_total = 0, ioff_total = 0, ent_total = 0;
    // Runs of the bra pairs of each class (jk_runs.cuh): entry e of class c is
    // pair d_ent[pair_locs[c] + e] (a position) of the class; run table v (run length
    // JK_RUN_LEN[v]) of class c has h_nrun[v][c] runs at d_run0 + h_run_off[v][c]
    std::vector<int> h_nrun[JK_RUN_LEVELS_PAIR], h_run_off[JK_RUN_LEVELS_PAIR];
    int *d_ent = nullptr, *d_run0 = nullptr;
    int* d_inv = nullptr;  // entry of a pair (the inverse of d_ent)
    int* d_erank = nullptr;  // Schwarz rank of an entry
    int *d_rank = nullptr, *d_pos = nullptr;  // rank of a position of the class, and the inverse
    double *d_bprim = nullptr, *d_bpair = nullptr;  // bra records (JKSeg::bprim, bpair)
    float* d_bprimf = nullptr;
    // device: the arrays of the basis and of its pairs lie in one allocation each
    void *mem_bas = nullptr, *mem_pair = nullptr;
    int *d_atm = nullptr, *d_bas = nullptr, *d_ao_loc = nullptr, *d_group_ao = nullptr;
    double *d_env = nullptr, *d_bas_x = nullptr;
    int *d_pair2bra = nullptr, *d_pair2ket = nullptr;  // by position
    double *d_log_q = nullptr, *d_log_q_raw = nullptr, *d_prim = nullptr;  // prim: a12|e12|x12|y12|z12|1/a12
    float* d_primf = nullptr;  // FP32 path: a12|1/a12|e12/a12|P-R_bra (x, y, z)
    long long nprim_total = 0;
    JKScreenCQ* d_cq = nullptr;
    long long *d_qoff = nullptr, *d_qoff32 = nullptr;  // FP64, FP32 part of the mixed mode
    long long* d_ioff = nullptr;                       // item prefixes, both parts
    int* d_klb = nullptr;
    int* d_kle = nullptr;
    // zeroed at the start of a build, in one piece: the condensed density,
    // then task0, task032, itm, itm32 of every class quartet
    void* d_zero = nullptr;
    size_t zero_bytes = 0;
    double* d_dm_cond = nullptr;
    long long *d_task0 = nullptr, *d_task032 = nullptr;
    // class launches of jk_build: of the whole build (made with the basis), and
    // of every (nshards, shard) asked for.  All are kept, since CUDA graphs
    // hold their tables.
    JKPlan* plan = nullptr;
    std::map<std::pair<int, int>, JKPlan*> shard_plans;
    // a build of this basis was captured: buffers that grow are kept in
    // `retired`, not freed, for the graph's sake
    bool captured = false;
    std::vector<void*> retired;
    // reference-compatible single class-pair path
    long long* d_qoff1 = nullptr;
    long long* d_task01 = nullptr;
    int* d_ehi1 = nullptr;
    JKSeg* d_seg1 = nullptr;
    long long qoff1_cap = 0;
    JKFanout fan;  // side streams of the class launches
    double* d_pgeo = nullptr;  // pair geometry (JKSeg::pgeo)
    std::vector<int> h_pnp;    // primitive pairs above the exponent cutoff, per pair
    int* d_pnp = nullptr;
    int* d_pao = nullptr;      // first AOs of the pair's shells (JKSeg::pao)
    // pair-packed J side of jk_build
    std::vector<JKPackCls> h_pack;
    JKPackCls* d_pack = nullptr;
    long long pack_total = 0;  // packed elements per density
    double* d_pk = nullptr;    // 2 n_dm x pack_total densities, then as many J accumulators
    size_t pk_cap = 0;
    double* d_kt = nullptr;    // K by rows of a jk_build (JKPackMol::kt)
    size_t kt_cap = 0;
    // transform workspace
    cublasHandle_t blas = nullptr;
    double* d_work = nullptr;
    size_t work_cap = 0;
};

int jk_internal_class_index(const jk_basis_t* b, int cp_ij, int cp_kl);
jk_launch_fn jk_internal_launcher(int class_idx, int fp32);
// launcher of the per-class-pair entries: K in the layout of the C-ABI
jk_launch_fn jk_internal_pair_launcher(int class_idx);
// 1 if the class runs a team kernel (one primitive count per launch)
int jk_internal_class_team(int class_idx);
// 1 if the class runs a run kernel
int jk_internal_class_runs(int class_idx);
void jk_internal_fill_seg(const jk_basis_t* b, int cp_ij, int cp_kl, const long long* qoff, int n_ij,
                          const double* dm, int n_dm, double* vj, double* vk, JKSeg* out);
// segment of a class quartet, FP64 or FP32 part (no density, no outputs)
void jk_internal_fill_seg_cq(const jk_basis_t* b, const JKScreenCQ& cq, int fp32, JKSeg* out);
// buffers that a build's screening writes, apart from the basis's own ones: a
// basis that occurs more than once in a batch is screened once per occurrence,
// with other densities
struct JKScreenSet {
    std::vector<JKScreenCQ> cq;
    double* dm_cond;
    void* zero;  // jk_basis::d_zero
    void* mem;   // one allocation, freed by the owner
};
int jk_internal_screen_set(const jk_basis_t* b, JKScreenSet* out);
JKPackMol jk_internal_pack_mol(const jk_basis_t* b, const double* dm, int n_dm, double* dens, double* acc, double* vj);
// pack (mode 0) or unpack (mode 1) the J side of nmol molecules (device
// table); mode 1 adds their kt too
int jk_internal_pack_batch(const JKPackMol* d_mols, int nmol, long long max_total, int mode, void* stream);
// condensed densities (outputs zeroed first) of nmol molecules (device table)
struct JKDmCond {
    const double* dm;
    const int* gao;  // group AO offsets (device)
    double* out;     // ngroups x ngroups
    int nao, n_dm, ngroups;
    unsigned long long* zero;  // words cleared before the condensation (jk_basis::d_zero)
    int nzero;
};
int jk_internal_dm_cond(const JKDmCond* d_mols, int nmol, int max_groups, int max_nao, void* stream);
int jk_internal_screen(const JKScreenCQ* d_cq, int ncq, double tol, int nbins, int prescreen, double fp32_cutoff,
                       void* stream);
