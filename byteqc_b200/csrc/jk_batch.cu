// Batched J/K builds: many molecules (one jk_basis each) in one pass.
//
// The class quartets of all molecules that share a class key become segments
// of ONE launch (jk_plan.cu, as jk_build does for one molecule), so a batch of
// hundreds of molecules costs one launch per class key plus the bookkeeping
// (density condensation, screening, prefixes), with no host synchronisation;
// the whole sequence can be captured into a CUDA graph and replayed every SCF
// iteration.  A key is the class (four angular momenta), plus the two
// primitive counts for the team kernels, whose blocks loop over the primitives
// in step.  Within a key the segments are ordered by descending task count, so
// the largest molecules' work is handed out first.
//
// Class quartets with at least `solo_tasks` unscreened tasks are not merged:
// each is a launch of its own, in molecule order, fanned out over the side
// streams ahead of the merged keys.  Merging costs the run kernels nothing (24
// molecules of 3-30 atoms, 6-31G*: 80.4 ms with a threshold of 2^14, 76.7 at
// 2^16, 75 merged; 12 of 3-60 atoms 260.6, 258.0 and 255.0), so the default
// threshold, 2^24, leaves only launches that run for milliseconds on their own.
//
// Launch shape per key (JKBatchCfg): static, or the persistent mode in which a grid of the device's resident capacity takes
// chunks from a device counter.  jk_batch_tune times the candidate shapes of
// every key on the batch itself and keeps the fastest; its choices can be
// written to and read from a cache file.
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <set>
#include <vector>

#include "jk_internal.h"

#define BCUDA(x)                                                  \
    do {                                                          \
        cudaError_t e_ = (x);                                     \
        if (e_ != cudaSuccess) return jk_internal_cuda_err(e_);   \
    } while (0)

struct JKSym {
    const double* in;
    double* out;
    int nao, n_dm;
};

struct jk_batch {
    int device = 0, nsm = 148, nmol = 0, max_groups = 0, max_nao = 0;
    std::vector<jk_basis*> mols;
    // screening records of every molecule: the basis's own, or those of a set
    // of buffers of the batch where the basis occurred before
    std::vector<const JKScreenCQ*> cqs;
    std::vector<JKScreenSet> own;  // by molecule, empty (mem null) for a first occurrence
    JKPlan* plan = nullptr;  // merged keys, then the class quartets launched on their own
    int nmerged = 0;         // merged keys
    JKScreenCQ* d_cq = nullptr;
    int ncq = 0;
    JKDmCond* d_dmc = nullptr;
    std::vector<JKDmCond> h_dmc;
    // pointer set the segment tables were built for
    std::vector<const double*> seg_dm;
    std::vector<double*> seg_vj, seg_vk;
    int seg_ndm = -1;
    bool seg_krows = false;
    // transform workspace
    cublasHandle_t blas = nullptr;
    double* d_work = nullptr;
    size_t work_cap = 0;
    JKSym* d_sym = nullptr;
    std::vector<size_t> w_dms, w_vj, w_vk, w_sym, w_tmp;  // offsets per molecule
    int w_ndm = -1;
    std::vector<int> w_nao0;  // caller basis sizes they were laid out for
    // captured graph
    cudaGraphExec_t graph = nullptr;
    JKFanout fan;  // side streams of the class launches
    // pair-packed J side: every molecule's packed densities, then every
    // molecule's packed J accumulators (one memset clears them all)
    double* d_pk = nullptr;
    size_t pk_cap = 0, pk_jp = 0;  // capacity; first accumulator element
    JKPackMol* d_pmol = nullptr;
    long long pk_max = 0;          // largest per-molecule packed size
    bool packed = false;
    double* d_kt = nullptr;  // K by rows of jk_batch_build (JKPackMol::kt), every molecule's after the other
    size_t kt_cap = 0, kt_len = 0;
};

// J = 2 (V + V^T), K = V + V^T per molecule (blockIdx.y = molecule)
__global__ void jk_symmetrize_batch_kernel(const JKSym* __restrict__ t, double fac) {
    const JKSym m = t[blockIdx.y];
    long long n = (long long)m.nao * m.nao * m.n_dm;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
         e += (long long)gridDim.x * blockDim.x) {
        long long d = e / ((long long)m.nao * m.nao);
        long long r = e - d * m.nao * m.nao;
        int p = (int)(r / m.nao), q = (int)(r % m.nao);
        const double* b = m.in + d * m.nao * m.nao;
        m.out[e] = fac * (b[(size_t)p * m.nao + q] + b[(size_t)q * m.nao + p]);
    }
}

static void free_batch(jk_batch* t) {
    if (!t) return;
    if (t->graph) cudaGraphExecDestroy(t->graph);
    t->fan.destroy();
    cudaFree(t->d_pk);
    cudaFree(t->d_pmol);
    cudaFree(t->d_kt);
    for (auto& o : t->own) cudaFree(o.mem);
    cudaFree(t->d_cq);
    cudaFree(t->d_dmc);
    jk_plan_free(t->plan);
    cudaFree(t->d_work);
    cudaFree(t->d_sym);
    if (t->blas) cublasDestroy(t->blas);
    delete t;
}

static int batch_create(jk_basis_t* const* bases, int nmol, long long solo_tasks, jk_batch* t) {
    BCUDA(cudaGetDevice(&t->device));
    BCUDA(cudaDeviceGetAttribute(&t->nsm, cudaDevAttrMultiProcessorCount, t->device));
    BCUDA(t->fan.init());
    t->nmol = nmol;
    t->plan = new JKPlan();
    std::vector<JKScreenCQ> cqs;
    std::set<const jk_basis*> seen;
    t->own.resize(nmol, JKScreenSet{});
    for (int m = 0; m < nmol; m++) {
        jk_basis* b = bases[m];
        if (!b) return jk_internal_set_err(JK_ERR_ARG, "jk_batch_create: null basis");
        if (b->device != t->device) return jk_internal_set_err(JK_ERR_ARG, "jk_batch_create: bases on other devices");
        if (!seen.insert(b).second)
            if (int rc = jk_internal_screen_set(b, &t->own[m])) return rc;
        t->mols.push_back(b);
        t->cqs.push_back(t->own[m].mem ? t->own[m].cq.data() : b->h_cq.data());
        t->max_groups = std::max(t->max_groups, b->ngroups);
        t->max_nao = std::max(t->max_nao, b->nao);
        for (int c = 0; c < b->ncq; c++) {
            const JKScreenCQ& cq = t->cqs[m][c];
            cqs.push_back(cq);
            const long long n = cq.cp_ij == cq.cp_kl ? (long long)cq.n_ij * (cq.n_ij + 1) / 2
                                                     : (long long)cq.n_ij * cq.n_kl;
            int rc = jk_plan_add(t->plan, b, m, c, solo_tasks > 0 && n >= solo_tasks);
            if (rc) return rc;
        }
    }
    int rc = jk_plan_finish(t->plan, t->mols, t->cqs);
    if (rc) return rc;
    for (const auto& k : t->plan->keys) t->nmerged += !k.solo;
    t->ncq = (int)cqs.size();
    BCUDA(cudaMalloc(&t->d_cq, sizeof(JKScreenCQ) * std::max(1, t->ncq)));
    if (t->ncq) BCUDA(cudaMemcpy(t->d_cq, cqs.data(), sizeof(JKScreenCQ) * t->ncq, cudaMemcpyHostToDevice));
    BCUDA(cudaMalloc(&t->d_dmc, sizeof(JKDmCond) * nmol));
    BCUDA(jk_internal_uploaded());
    return JK_OK;
}

extern "C" int jk_batch_create_ex(jk_basis_t* const* bases, int nmol, long long solo_tasks, jk_batch_t** out) {
    if (!bases || nmol <= 0 || !out) return jk_internal_set_err(JK_ERR_ARG, "jk_batch_create: invalid arguments");
    jk_batch* t = new jk_batch();
    int rc = jk_guard([&] { return batch_create(bases, nmol, solo_tasks, t); });
    if (rc) {
        free_batch(t);
        *out = nullptr;
        return rc;
    }
    *out = t;
    return JK_OK;
}

extern "C" int jk_batch_create(jk_basis_t* const* bases, int nmol, jk_batch_t** out) {
    return jk_batch_create_ex(bases, nmol, JK_BATCH_SOLO_TASKS, out);
}

extern "C" int jk_batch_destroy(jk_batch_t* t) {
    free_batch(t);
    return JK_OK;
}

// (re)build the segment tables when the density / output buffers change
// (krows as in jk_host.cu's build)
static int batch_segments(jk_batch* t, const double* const* dms, double* const* vjs, double* const* vks, int n_dm,
                          bool krows, cudaStream_t st) {
    bool same = t->seg_ndm == n_dm && t->seg_krows == krows && (int)t->seg_dm.size() == t->nmol;
    for (int m = 0; same && m < t->nmol; m++)
        same = t->seg_dm[m] == dms[m] && t->seg_vj[m] == (vjs ? vjs[m] : nullptr) &&
               t->seg_vk[m] == (vks ? vks[m] : nullptr);
    if (same) return JK_OK;
    // earlier launches may still read the old tables and buffers
    BCUDA(cudaStreamSynchronize(st));
    t->seg_ndm = -1;  // no tables until these are complete (an allocation may fail on the way)
    // pair-packed J side (with J only)
    t->packed = vjs != nullptr;
    std::vector<size_t> dp_off(t->nmol, 0);
    t->pk_max = 0;
    if (t->packed) {
        size_t tot = 0;
        for (int m = 0; m < t->nmol; m++) {
            dp_off[m] = tot;
            tot += 2 * (size_t)n_dm * t->mols[m]->pack_total;
            t->pk_max = std::max(t->pk_max, t->mols[m]->pack_total);
        }
        t->pk_jp = tot;
        if (2 * tot > t->pk_cap) {
            cudaFree(t->d_pk);
            t->d_pk = nullptr;
            t->pk_cap = 0;
            BCUDA(cudaMalloc(&t->d_pk, sizeof(double) * std::max<size_t>(2 * tot, 1)));
            t->pk_cap = 2 * tot;
        }
    }
    // K by rows (jk_batch_build)
    std::vector<size_t> kt_off(t->nmol, 0);
    t->kt_len = 0;
    if (vks && !krows) {
        for (int m = 0; m < t->nmol; m++) {
            kt_off[m] = t->kt_len;
            t->kt_len += (size_t)n_dm * t->mols[m]->nao * t->mols[m]->nao;
        }
        if (t->kt_len > t->kt_cap) {
            cudaFree(t->d_kt);
            t->d_kt = nullptr;
            t->kt_cap = 0;
            BCUDA(cudaMalloc(&t->d_kt, sizeof(double) * t->kt_len));
            t->kt_cap = t->kt_len;
        }
    }
    if (t->packed || t->kt_len) {
        std::vector<JKPackMol> pm(t->nmol);
        for (int m = 0; m < t->nmol; m++) {
            const size_t o = dp_off[m];
            pm[m] = jk_internal_pack_mol(t->mols[m], dms[m], n_dm, t->d_pk + o, t->d_pk + t->pk_jp + o,
                                         vjs ? vjs[m] : nullptr);
            if (!t->packed || !vjs[m]) pm[m].total = 0;  // no J wanted
            if (t->kt_len && vks[m]) {
                pm[m].kt = t->d_kt + kt_off[m];
                pm[m].vk = vks[m];
            }
        }
        if (!t->d_pmol) BCUDA(cudaMalloc(&t->d_pmol, sizeof(JKPackMol) * t->nmol));
        BCUDA(cudaMemcpy(t->d_pmol, pm.data(), sizeof(JKPackMol) * t->nmol, cudaMemcpyHostToDevice));
    }
    JKPlan* p = t->plan;
    std::vector<JKSeg> seg(std::max(1, p->nseg));
    for (int part = 0; part < 2; part++) {
        int i = 0;
        for (auto& k : p->keys)
            for (auto& sgi : k.segs) {
                const int m = sgi.first;
                JKSeg& s = seg[i++];
                jk_internal_fill_seg_cq(t->mols[m], t->cqs[m][sgi.second], part, &s);
                s.dm = dms[m];
                s.vj = vjs ? vjs[m] : nullptr;
                s.vk = vks ? vks[m] : nullptr;
                s.n_dm = n_dm;
                if (t->kt_len && s.vk && s.nrun > 0) s.vk = t->d_kt + kt_off[m];
                if (t->packed) {
                    const size_t n = (size_t)n_dm * t->mols[m]->pack_total;
                    s.dp = t->d_pk + dp_off[m];
                    s.dpb = s.dp + n;
                    s.jp = t->d_pk + t->pk_jp + dp_off[m];
                    s.jpb = s.jp + n;
                }
            }
        BCUDA(cudaMemcpy(p->d_seg[part], seg.data(), sizeof(JKSeg) * p->nseg, cudaMemcpyHostToDevice));
    }
    t->h_dmc.resize(t->nmol);
    for (int m = 0; m < t->nmol; m++) {
        jk_basis* b = t->mols[m];
        const JKScreenSet& o = t->own[m];
        t->h_dmc[m] = JKDmCond{dms[m],     b->d_group_ao, o.mem ? o.dm_cond : b->d_dm_cond, b->nao, n_dm,
                               b->ngroups, (unsigned long long*)(o.mem ? o.zero : b->d_zero),
                               (int)(b->zero_bytes / 8)};
    }
    BCUDA(cudaMemcpy(t->d_dmc, t->h_dmc.data(), sizeof(JKDmCond) * t->nmol, cudaMemcpyHostToDevice));
    BCUDA(jk_internal_uploaded());
    t->seg_dm.assign(dms, dms + t->nmol);
    t->seg_vj.assign(t->nmol, nullptr);
    t->seg_vk.assign(t->nmol, nullptr);
    for (int m = 0; m < t->nmol; m++) {
        if (vjs) t->seg_vj[m] = vjs[m];
        if (vks) t->seg_vk[m] = vks[m];
    }
    t->seg_ndm = n_dm;
    t->seg_krows = krows;
    return JK_OK;
}

// everything before the class launches: segment tables, density
// condensation, screening, task prefixes, pair-packed densities
static int batch_prepare(jk_batch* t, const double* const* dms, double* const* vjs, double* const* vks, int n_dm,
                         bool krows, const jk_opts_t* opts, cudaStream_t st) {
    int rc = batch_segments(t, dms, vjs, vks, n_dm, krows, st);
    if (rc) return rc;
    double tol = opts ? opts->direct_scf_tol : t->mols[0]->cutoff;
    int nbins = opts && opts->nbins > 0 ? opts->nbins : 10;
    int prescreen = opts ? opts->prescreen : 1;
    double fp32_cutoff = opts ? opts->fp32_cutoff : 0.;
    rc = jk_internal_dm_cond(t->d_dmc, t->nmol, t->max_groups, t->max_nao, st);
    if (rc || t->ncq == 0) return rc;
    rc = jk_internal_screen(t->d_cq, t->ncq, tol, nbins, prescreen, fp32_cutoff, st);
    if (!rc) rc = jk_plan_prefix(t->plan, fp32_cutoff > 0, st);
    if (rc) return rc;
    if (t->packed) {
        rc = jk_internal_pack_batch(t->d_pmol, t->nmol, t->pk_max, 0, st);
        if (rc) return rc;
        BCUDA(cudaMemsetAsync(t->d_pk + t->pk_jp, 0, sizeof(double) * t->pk_jp, st));
    }
    if (t->kt_len) BCUDA(cudaMemsetAsync(t->d_kt, 0, sizeof(double) * t->kt_len, st));
    return JK_OK;
}

static int batch_build(jk_batch* t, const double* const* dms, double* const* vjs, double* const* vks, int n_dm,
                       bool krows, const jk_opts_t* opts, void* stream) {
    if (!t || !dms || n_dm <= 0) return jk_internal_set_err(JK_ERR_ARG, "jk_batch_build: invalid arguments");
    if (!vjs && !vks) return JK_OK;
    cudaStream_t st = (cudaStream_t)stream;
    int rc = batch_prepare(t, dms, vjs, vks, n_dm, krows, opts, st);
    if (rc || t->ncq == 0) return rc;
    const bool mixed = opts && opts->fp32_cutoff > 0;
    const int nkeys = (int)t->plan->keys.size();
    // work counters of the persistent launches start at zero every build
    BCUDA(cudaMemsetAsync(t->plan->d_queue, 0, sizeof(unsigned long long) * 2 * nkeys, st));
    BCUDA(t->fan.begin(st));
    // class quartets on their own first; FP64 parts on the even side streams,
    // FP32 parts on the odd ones
    for (int lane = 0; lane < nkeys; lane++) {
        const int k = (t->nmerged + lane) % nkeys;
        for (int part = 0; part < (mixed ? 2 : 1); part++) {
            rc = jk_plan_launch(t->plan, k, part, t->plan->keys[k].cfg[part], n_dm, t->nsm,
                                t->fan.pick(2 * lane + part));
            if (rc) return rc;
        }
    }
    BCUDA(t->fan.end(st));
    if (t->packed || t->kt_len) {
        rc = jk_internal_pack_batch(t->d_pmol, t->nmol, std::max<long long>(t->pk_max, (long long)t->kt_len), 1, stream);
        if (rc) return rc;
    }
    return JK_OK;
}

extern "C" int jk_batch_build(jk_batch_t* t, const double* const* dms, double* const* vjs, double* const* vks,
                              int n_dm, const jk_opts_t* opts, void* stream) {
    return jk_guard([&] { return batch_build(t, dms, vjs, vks, n_dm, false, opts, stream); });
}

// ---------------------------------------------------------------------------
// Autotuner.  For every key (and both parts in the mixed mode) the candidate
// launch shapes are timed on this batch with CUDA events, each launch alone
// on the caller's stream after the bookkeeping of a real build, and the
// fastest is kept.  Candidates: static chunks; the persistent mode at one
// resident grid with three grab sizes (items per warp for the run kernels,
// tasks per team for the team kernels, per block for the generic kernel)
// and at two resident grids with the middle one.  A cache file keeps the
// choices per (class, primitive counts, part, log2 of the task count); keys
// found there are not timed again.
// ---------------------------------------------------------------------------
static int cand_grabs(int cls, int* g) {
    if (jk_internal_class_team(cls)) { g[0] = 2; g[1] = 8; g[2] = 32; }
    else { g[0] = 1; g[1] = 4; g[2] = 16; }
    return 3;
}

static std::string tune_key_str(const JKPlanKey& k, int part) {
    int b = 0;
    for (long long x = k.max_tasks; x > 1; x >>= 1) b++;
    char buf[96];
    snprintf(buf, sizeof(buf), "%d %d %d %d %d", k.cls, k.np_ij, k.np_kl, part, b);
    return buf;
}

// First line of a cache file as the tuner writes it.  The number stands for
// what a grab means: 2, items for the run kernels.  Files written before it
// have the line without a number, and counted quartets there (grabs up to
// 1024, which as items leave most of the device idle): they are not read.
// Files without such a line (written by hand) are.
static const char kTuneHead[] = "# byteqc_b200 batch launch shapes";
static const char kTuneVersion[] = " 2: ";

static int batch_tune(jk_batch* t, const double* const* dms, double* const* vjs, double* const* vks, int n_dm,
                      const jk_opts_t* opts, const char* cache_path, void* stream) {
    if (!t || !dms || n_dm <= 0 || (!vjs && !vks))
        return jk_internal_set_err(JK_ERR_ARG, "jk_batch_tune: invalid arguments");
    cudaStream_t st = (cudaStream_t)stream;
    const int nkeys = t->nmerged;
    const bool mixed = opts && opts->fp32_cutoff > 0;
    // cached choices: "cls np_ij np_kl part log2tasks mode grab grid_mul ms"
    std::map<std::string, std::pair<JKBatchCfg, float>> cache;
    if (cache_path) {
        FILE* f = fopen(cache_path, "r");
        if (f) {
            char line[256];
            while (fgets(line, sizeof(line), f)) {
                if (!strncmp(line, kTuneHead, sizeof(kTuneHead) - 1) &&
                    strncmp(line + sizeof(kTuneHead) - 1, kTuneVersion, sizeof(kTuneVersion) - 1))
                    break;  // of another version
                int cls, a, b, part, lg, grab, gm;
                float ms;
                if (sscanf(line, "%d %d %d %d %d %d %d %f", &cls, &a, &b, &part, &lg, &grab, &gm, &ms) != 8) continue;
                if (grab < 0 || gm < 1 || gm > 64) continue;  // no launch shape
                char key[96];
                snprintf(key, sizeof(key), "%d %d %d %d %d", cls, a, b, part, lg);
                cache[key] = {JKBatchCfg{nullptr, grab, gm}, ms};
            }
            fclose(f);
        }
    }
    // as jk_batch_get_jk launches them
    int rc = batch_prepare(t, dms, vjs, vks, n_dm, true, opts, st);
    if (rc) return rc;
    cudaEvent_t e0, e1;
    BCUDA(cudaEventCreate(&e0));
    BCUDA(cudaEventCreate(&e1));
    for (int k = 0; k < nkeys && t->ncq; k++) {
        JKPlanKey& key = t->plan->keys[k];
        for (int part = 0; part < (mixed ? 2 : 1); part++) {
            const std::string ks = tune_key_str(key, part);
            auto hit = cache.find(ks);
            if (hit != cache.end()) {
                key.cfg[part] = hit->second.first;
                key.tuned_ms[part] = hit->second.second;
                continue;
            }
            int g[3];
            cand_grabs(key.cls, g);
            std::vector<JKBatchCfg> cands = {{nullptr, 0, 1}};
            for (int i = 0; i < 3; i++) cands.push_back({nullptr, g[i], 1});
            cands.push_back({nullptr, g[1], 2});
            // untimed first launch (attributes, instruction cache)
            BCUDA(cudaMemsetAsync(t->plan->d_queue, 0, sizeof(unsigned long long) * 2 * nkeys, st));
            rc = jk_plan_launch(t->plan, k, part, cands[0], n_dm, t->nsm, st);
            if (rc) return rc;
            float best = -1.f;
            for (const JKBatchCfg& c : cands) {
                float tmin = -1.f;
                for (int rep = 0; rep < 1; rep++) {
                    BCUDA(cudaMemsetAsync(t->plan->d_queue, 0, sizeof(unsigned long long) * 2 * nkeys, st));
                    BCUDA(cudaEventRecord(e0, st));
                    rc = jk_plan_launch(t->plan, k, part, c, n_dm, t->nsm, st);
                    if (rc) return rc;
                    BCUDA(cudaEventRecord(e1, st));
                    BCUDA(cudaEventSynchronize(e1));
                    float ms = 0.f;
                    BCUDA(cudaEventElapsedTime(&ms, e0, e1));
                    if (tmin < 0 || ms < tmin) tmin = ms;
                }
                if (best < 0 || tmin < best) {
                    best = tmin;
                    key.cfg[part] = c;
                }
            }
            key.tuned_ms[part] = best;
            cache[ks] = {key.cfg[part], best};
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    BCUDA(cudaStreamSynchronize(st));
    // the timing runs accumulated into the outputs: clear them
    for (int m = 0; m < t->nmol; m++) {
        size_t nn = (size_t)t->mols[m]->nao * t->mols[m]->nao * n_dm;
        if (vjs && vjs[m]) BCUDA(cudaMemset(vjs[m], 0, sizeof(double) * nn));
        if (vks && vks[m]) BCUDA(cudaMemset(vks[m], 0, sizeof(double) * nn));
    }
    if (cache_path) {
        FILE* f = fopen(cache_path, "w");
        if (!f) return jk_internal_set_err(JK_ERR_ARG, "jk_batch_tune: cannot write the cache file");
        fprintf(f, "%s%scls np_ij np_kl part log2tasks grab grid_mul ms\n", kTuneHead, kTuneVersion);
        for (auto& kv : cache)
            fprintf(f, "%s %d %d %.4f\n", kv.first.c_str(), kv.second.first.grab, kv.second.first.grid_mul,
                    kv.second.second);
        fclose(f);
    }
    return JK_OK;
}

extern "C" int jk_batch_tune(jk_batch_t* t, const double* const* dms, double* const* vjs, double* const* vks,
                             int n_dm, const jk_opts_t* opts, const char* cache_path, void* stream) {
    return jk_guard([&] { return batch_tune(t, dms, vjs, vks, n_dm, opts, cache_path, stream); });
}

extern "C" int jk_batch_nsolo(const jk_batch_t* t, int* nsolo) {
    if (!t || !nsolo) return jk_internal_set_err(JK_ERR_ARG, "jk_batch_nsolo: invalid arguments");
    *nsolo = (int)t->plan->keys.size() - t->nmerged;
    return JK_OK;
}

// launch shapes chosen for the batch: per key cls, np_ij, np_kl, then for
// parts 0 and 1 grab, grid_mul and the tuned time in microseconds (-1 if
// not tuned); out holds 12 ints per key
extern "C" int jk_batch_info(const jk_batch_t* t, int* nkeys, int* out) {
    if (!t || !nkeys) return jk_internal_set_err(JK_ERR_ARG, "jk_batch_info: invalid arguments");
    *nkeys = t->nmerged;
    if (!out) return JK_OK;
    for (int k = 0; k < t->nmerged; k++) {
        const JKPlanKey& key = t->plan->keys[k];
        int* o = out + 12 * k;
        o[0] = key.cls;
        o[1] = key.np_ij;
        o[2] = key.np_kl;
        o[3] = (int)std::min<long long>(key.max_tasks, 2147483647LL);
        for (int p = 0; p < 2; p++) {
            o[4 + 4 * p] = key.cfg[p].grab;
            o[5 + 4 * p] = key.cfg[p].grid_mul;
            o[6 + 4 * p] = (int)(key.tuned_ms[p] * 1000.f);
            o[7 + 4 * p] = (int)key.segs.size();
        }
    }
    return JK_OK;
}

static cublasStatus_t gemm_rm_b(cublasHandle_t h, bool ta, bool tb, int M, int N, int K, const double* A, int lda,
                                const double* B, int ldb, double* C, int ldc) {
    const double one = 1.0, zero = 0.0;
    return cublasDgemm(h, tb ? CUBLAS_OP_T : CUBLAS_OP_N, ta ? CUBLAS_OP_T : CUBLAS_OP_N, N, M, K, &one, B, ldb, A,
                       lda, &zero, C, ldc);
}

#define BBLAS(x)                                                                           \
    do {                                                                                   \
        if ((x) != CUBLAS_STATUS_SUCCESS) return jk_internal_set_err(JK_ERR_CUDA, #x);     \
    } while (0)

// Full J/K of every molecule in its own basis: dms_m = C_m D_m C_m^T, one
// batched build, then J_m = 2 C_m^T (V + V^T) C_m, K_m = C_m^T (V + V^T) C_m.
// coeffs[m] (nao_m, nao0s[m]) row-major device; dm0s/vj0s/vk0s device
// (n_dm, nao0, nao0); vj0s/vk0s overwritten (either may be NULL).
static int batch_get_jk(jk_batch* t, const double* const* coeffs, const int* nao0s, const double* const* dm0s,
                        double* const* vj0s, double* const* vk0s, int n_dm, const jk_opts_t* opts, void* stream) {
    if (!t || !coeffs || !nao0s || !dm0s || n_dm <= 0)
        return jk_internal_set_err(JK_ERR_ARG, "jk_batch_get_jk: invalid arguments");
    cudaStream_t st = (cudaStream_t)stream;
    int nmol = t->nmol;
    bool fits = t->w_ndm == n_dm;
    for (int m = 0; fits && m < nmol; m++) fits = nao0s[m] <= t->w_nao0[m];
    if (!fits) {
        size_t off = 0;
        t->w_dms.resize(nmol);
        t->w_vj.resize(nmol);
        t->w_vk.resize(nmol);
        t->w_sym.resize(nmol);
        t->w_tmp.resize(nmol);
        for (int m = 0; m < nmol; m++) {
            size_t nn = (size_t)t->mols[m]->nao * t->mols[m]->nao * n_dm;
            t->w_dms[m] = off;
            off += nn;
            t->w_vj[m] = off;
            off += nn;
            t->w_vk[m] = off;
            off += nn;
            t->w_sym[m] = off;
            off += nn;
            t->w_tmp[m] = off;
            off += (size_t)t->mols[m]->nao * nao0s[m];
        }
        BCUDA(cudaStreamSynchronize(st));
        t->w_ndm = -1;  // until it is laid out
        cudaFree(t->d_work);
        t->d_work = nullptr;
        BCUDA(cudaMalloc(&t->d_work, sizeof(double) * std::max<size_t>(off, 1)));
        t->work_cap = off;
        cudaFree(t->d_sym);
        t->d_sym = nullptr;
        // symmetrisation tables: J inputs in [0, nmol), K inputs in [nmol, 2 nmol)
        BCUDA(cudaMalloc(&t->d_sym, sizeof(JKSym) * 2 * nmol));
        std::vector<JKSym> sy(2 * nmol);
        for (int m = 0; m < nmol; m++) {
            sy[m] = JKSym{t->d_work + t->w_vj[m], t->d_work + t->w_sym[m], t->mols[m]->nao, n_dm};
            sy[nmol + m] = JKSym{t->d_work + t->w_vk[m], t->d_work + t->w_sym[m], t->mols[m]->nao, n_dm};
        }
        BCUDA(cudaMemcpy(t->d_sym, sy.data(), sizeof(JKSym) * 2 * nmol, cudaMemcpyHostToDevice));
        BCUDA(jk_internal_uploaded());
        t->w_ndm = n_dm;
        t->w_nao0.assign(nao0s, nao0s + nmol);
    }
    if (!t->blas) BBLAS(cublasCreate(&t->blas));
    BBLAS(cublasSetStream(t->blas, st));
    std::vector<const double*> dms(nmol);
    std::vector<double*> vjs(nmol), vks(nmol);
    for (int m = 0; m < nmol; m++) {
        jk_basis* b = t->mols[m];
        int nao = b->nao, nao0 = nao0s[m];
        double* w = t->d_work;
        for (int d = 0; d < n_dm; d++) {
            BBLAS(gemm_rm_b(t->blas, false, false, nao, nao0, nao0, coeffs[m], nao0,
                            dm0s[m] + (size_t)d * nao0 * nao0, nao0, w + t->w_tmp[m], nao0));
            BBLAS(gemm_rm_b(t->blas, false, true, nao, nao, nao0, w + t->w_tmp[m], nao0, coeffs[m], nao0,
                            w + t->w_dms[m] + (size_t)d * nao * nao, nao));
        }
        size_t nn = (size_t)nao * nao * n_dm;
        if (vj0s) BCUDA(cudaMemsetAsync(w + t->w_vj[m], 0, sizeof(double) * nn, st));
        if (vk0s) BCUDA(cudaMemsetAsync(w + t->w_vk[m], 0, sizeof(double) * nn, st));
        dms[m] = w + t->w_dms[m];
        vjs[m] = w + t->w_vj[m];
        vks[m] = w + t->w_vk[m];
    }
    int rc = batch_build(t, dms.data(), vj0s ? vjs.data() : nullptr, vk0s ? vks.data() : nullptr, n_dm, true, opts,
                         stream);
    if (rc) return rc;
    for (int pass = 0; pass < 2; pass++) {
        double* const* outs = pass == 0 ? vj0s : vk0s;
        if (!outs) continue;
        dim3 g(32, nmol);
        jk_symmetrize_batch_kernel<<<g, 256, 0, st>>>(t->d_sym + (pass == 0 ? 0 : nmol), pass == 0 ? 2.0 : 1.0);
        BCUDA(cudaGetLastError());
        for (int m = 0; m < nmol; m++) {
            jk_basis* b = t->mols[m];
            int nao = b->nao, nao0 = nao0s[m];
            double* w = t->d_work;
            for (int d = 0; d < n_dm; d++) {
                BBLAS(gemm_rm_b(t->blas, false, false, nao, nao0, nao, w + t->w_sym[m] + (size_t)d * nao * nao, nao,
                                coeffs[m], nao0, w + t->w_tmp[m], nao0));
                BBLAS(gemm_rm_b(t->blas, true, false, nao0, nao0, nao, coeffs[m], nao0, w + t->w_tmp[m], nao0,
                                outs[m] + (size_t)d * nao0 * nao0, nao0));
            }
        }
    }
    return JK_OK;
}

extern "C" int jk_batch_get_jk(jk_batch_t* t, const double* const* coeffs, const int* nao0s,
                               const double* const* dm0s, double* const* vj0s, double* const* vk0s, int n_dm,
                               const jk_opts_t* opts, void* stream) {
    return jk_guard([&] { return batch_get_jk(t, coeffs, nao0s, dm0s, vj0s, vk0s, n_dm, opts, stream); });
}
