// Class launches of a set of class quartets (one molecule for jk_build, many
// for jk_batch_*): the class quartets that share a class become segments of
// one launch.  A launch per class quartet, as jk_build made before, was 666
// launches for a def2-TZVP molecule, most of them too small to fill the
// device; merged they are 59, and the run kernels look a segment up once per
// item (up to 32 x 32 quartets), so that merging costs the large ones nothing.
#include <string.h>

#include <algorithm>

#include "jk_internal.h"

#define PCUDA(x)                                                  \
    do {                                                          \
        cudaError_t e_ = (x);                                     \
        if (e_ != cudaSuccess) return jk_internal_cuda_err(e_);   \
    } while (0)

// exclusive prefix of the segments' counts of every key (blockIdx.x = key, one
// warp); key k's prefix lives at segt[key_off[k] + k], n_k + 1 entries
__global__ void jk_seg_prefix_kernel(const long long* const* __restrict__ cnt, const int* __restrict__ key_off,
                                     long long* __restrict__ segt) {
    const int k = blockIdx.x, lane = threadIdx.x;
    const int s0 = key_off[k], n = key_off[k + 1] - s0;
    long long* out = segt + s0 + k;
    long long carry = 0;
    if (lane == 0) out[0] = 0;
    for (int base = 0; base < n; base += 32) {
        const int i = base + lane;
        long long v = i < n ? *cnt[s0 + i] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const long long y = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += y;
        }
        if (i < n) out[i + 1] = carry + v;
        carry += __shfl_sync(0xffffffffu, v, 31);
    }
}

void jk_plan_free(JKPlan* p) {
    if (!p) return;
    cudaFree(p->mem);
    delete p;
}

// bound of a class quartet's task or item count
static long long cq_items(const JKScreenCQ& cq) {
    if (cq.runs) return (long long)cq.nrun * ((cq.n_kl + cq.runs - 1) / cq.runs + 1);
    return cq.cp_ij == cq.cp_kl ? (long long)cq.n_ij * (cq.n_ij + 1) / 2 : (long long)cq.n_ij * cq.n_kl;
}
// {0, count} of a class quartet's tasks or items
static const long long* cq_count(const JKScreenCQ& cq, int part) {
    if (cq.runs) return part ? cq.itm32 : cq.itm;
    return part ? cq.task032 : cq.task0;
}

int jk_plan_add(JKPlan* p, const jk_basis* b, int m, int c, bool solo) {
    const JKScreenCQ& cq = b->h_cq[c];
    const int cls = jk_internal_class_index(b, cq.cp_ij, cq.cp_kl);
    if (!jk_internal_launcher(cls, 0)) return jk_internal_set_err(JK_ERR_UNSUPPORTED, "no kernel for a class quartet");
    const long long n =
        cq.cp_ij == cq.cp_kl ? (long long)cq.n_ij * (cq.n_ij + 1) / 2 : (long long)cq.n_ij * cq.n_kl;
    int np_ij = b->h_group_nprim[cq.gi] * b->h_group_nprim[cq.gj];
    int np_kl = b->h_group_nprim[cq.gk] * b->h_group_nprim[cq.gl];
    if (!jk_internal_class_team(cls)) np_ij = np_kl = -1;
    JKPlanKey* k = nullptr;
    const auto id = std::make_tuple(cls, np_ij, np_kl);
    if (!solo) {
        auto it = p->index.find(id);
        if (it != p->index.end()) k = &p->keys[it->second];
        else p->index[id] = (int)p->keys.size();
    }
    if (!k) {
        p->keys.emplace_back();
        k = &p->keys.back();
        k->cls = cls;
        k->np_ij = np_ij;
        k->np_kl = np_kl;
        k->solo = solo;
    }
    k->segs.push_back({m, c});
    k->seg_tasks.push_back(n);
    k->max_tasks += n;
    k->max_items += cq_items(cq);
    return JK_OK;
}

int jk_plan_finish(JKPlan* p, const std::vector<jk_basis*>& mols, const std::vector<const JKScreenCQ*>& cqs) {
    p->index.clear();
    std::stable_partition(p->keys.begin(), p->keys.end(), [](const JKPlanKey& k) { return !k.solo; });
    // longest first within every key (stable: ties keep molecule order)
    for (auto& k : p->keys) {
        std::vector<int> ord(k.segs.size());
        for (size_t i = 0; i < ord.size(); i++) ord[i] = (int)i;
        std::stable_sort(ord.begin(), ord.end(), [&](int a, int b) { return k.seg_tasks[a] > k.seg_tasks[b]; });
        std::vector<std::pair<int, int>> segs(ord.size());
        std::vector<long long> tasks(ord.size());
        for (size_t i = 0; i < ord.size(); i++) {
            segs[i] = k.segs[ord[i]];
            tasks[i] = k.seg_tasks[ord[i]];
        }
        k.segs.swap(segs);
        k.seg_tasks.swap(tasks);
    }
    const int nkeys = (int)p->keys.size();
    p->key_off.assign(1, 0);
    for (auto& k : p->keys) p->key_off.push_back(p->key_off.back() + (int)k.segs.size());
    p->nseg = p->key_off.back();
    const size_t ns = std::max(1, p->nseg);
    // one allocation: what the host fills (segments and counts of both parts,
    // key offsets) in front, uploaded as one piece
    auto up = [](size_t bytes) { return (bytes + 255) & ~(size_t)255; };
    const size_t seg_b = up(sizeof(JKSeg) * ns), cnt_b = up(sizeof(long long*) * ns),
                 off_b = up(sizeof(int) * (nkeys + 1)), segt_b = up(sizeof(long long) * (ns + nkeys + 1));
    const size_t host_b = 2 * (seg_b + cnt_b) + off_b;
    PCUDA(cudaMalloc(&p->mem, host_b + 2 * segt_b + sizeof(unsigned long long) * 2 * std::max(1, nkeys)));
    std::vector<char> host(host_b);
    for (int part = 0; part < 2; part++) {
        const size_t seg_at = part * seg_b, cnt_at = 2 * seg_b + part * cnt_b;
        JKSeg* seg = (JKSeg*)(host.data() + seg_at);
        const long long** cnt = (const long long**)(host.data() + cnt_at);
        size_t i = 0;
        for (auto& k : p->keys) {
            if (k.segs.size() != 1) {
                p->one[part].push_back(nullptr);
                p->multi = true;
            }
            for (auto& s : k.segs) {
                const JKScreenCQ& cq = cqs[s.first][s.second];
                jk_internal_fill_seg_cq(mols[s.first], cq, part, &seg[i]);
                if (k.segs.size() == 1) p->one[part].push_back(cq_count(cq, part));
                cnt[i++] = cq_count(cq, part) + 1;
            }
        }
        p->d_seg[part] = (JKSeg*)((char*)p->mem + seg_at);
        p->d_cnt[part] = (const long long**)((char*)p->mem + cnt_at);
        p->d_segt[part] = (long long*)((char*)p->mem + host_b + part * segt_b);
    }
    memcpy(host.data() + 2 * (seg_b + cnt_b), p->key_off.data(), sizeof(int) * (nkeys + 1));
    p->d_key_off = (int*)((char*)p->mem + 2 * (seg_b + cnt_b));
    p->d_queue = (unsigned long long*)((char*)p->mem + host_b + 2 * segt_b);
    PCUDA(cudaMemcpyAsync(p->mem, host.data(), host_b, cudaMemcpyHostToDevice, cudaStreamLegacy));
    PCUDA(jk_internal_uploaded());
    return JK_OK;
}

int jk_plan_prefix(const JKPlan* p, bool mixed, cudaStream_t st) {
    const int nkeys = (int)p->keys.size();
    if (nkeys == 0 || !p->multi) return JK_OK;
    for (int part = 0; part < (mixed ? 2 : 1); part++)
        jk_seg_prefix_kernel<<<nkeys, 32, 0, st>>>(p->d_cnt[part], p->d_key_off, p->d_segt[part]);
    PCUDA(cudaGetLastError());
    return JK_OK;
}

static jk_launch_fn plan_launcher(int cls, int part, bool direct) {
    return direct && jk_internal_class_runs(cls) ? jk_internal_pair_launcher(cls) : jk_internal_launcher(cls, part);
}

int jk_plan_launch(const JKPlan* p, int k, int part, const JKBatchCfg& cfg, int n_dm, int nsm, cudaStream_t st,
                   bool direct) {
    const JKPlanKey& key = p->keys[k];
    const int off = p->key_off[k], n = p->key_off[k + 1] - off;
    jk_launch_fn f = plan_launcher(key.cls, part, direct);
    if (!f) return jk_internal_set_err(JK_ERR_UNSUPPORTED, "no kernel for a class of the build");
    JKBatchCfg c = cfg;
    c.queue = c.grab > 0 ? p->d_queue + 2 * k + part : nullptr;
    const long long* segt = p->one[part][k] ? p->one[part][k] : p->d_segt[part] + off + k;
    PCUDA(f(p->d_seg[part] + off, segt, n, key.max_items, n_dm, nsm, c, st));
    return JK_OK;
}

int jk_plan_launch_one(const JKPlan* p, int k, int s, int part, const JKScreenCQ& cq, int n_dm, int nsm,
                       cudaStream_t st, bool direct) {
    jk_launch_fn f = plan_launcher(p->keys[k].cls, part, direct);
    if (!f) return jk_internal_set_err(JK_ERR_UNSUPPORTED, "no kernel for a class of the build");
    PCUDA(f(p->d_seg[part] + p->key_off[k] + s, cq_count(cq, part), 1, cq_items(cq), n_dm, nsm,
            JKBatchCfg{nullptr, 0, 1}, st));
    return JK_OK;
}
