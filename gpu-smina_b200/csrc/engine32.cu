// Batched mixed-precision docking behind the C ABI (sg_dock_batch32):
// every ligand job's chains run in one persistent search launch (k_mc32, or
// k_mc32_mix where some chains get a block each), the chains of a ligand are
// merged like merge_output_containers with min_rmsd 2 (k_merge32), and every
// merged pose is refined in FP64 on the direct receptor sum (k_refine64).
// Reference: gpu_docking.cpp:560-625 (GpuDocking::dock_batch),
// parallel_mc.cpp:64-98, main.cpp:165-200.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <numeric>
#include "engine.h"

namespace sg {

DTables32 tables32(const sg_engine* e) {
    DTables32 T{};
    T.nc = e->tables.nc;
    T.n = e->tables.n;
    T.factor = (float)e->tables.factor;
    T.cutoff_sqr = (float)e->tables.cutoff_sqr;
    T.tab = e->tab32.as<float4>();
    return T;
}

DMaps32 maps32(const sg_engine* e, const RecState& r) {
    DMaps32 G{};
    for (int i = 0; i < 3; i++) {
        require(r.geom.dim[i] >= 2, "mixed-precision path: the box needs at least one grid cell per axis");
        G.cdim[i] = r.geom.dim[i] - 1;
        G.init[i] = (float)r.geom.init[i];
        G.factor[i] = (float)r.geom.factor[i];
        G.factor_inv[i] = (float)r.geom.factor_inv[i];
        G.dim_fl_minus_1[i] = (float)r.geom.dim_fl_minus_1[i];
    }
    for (int t = 0; t < kNumTypes; t++) {
        G.m32[t] = r.map32[t].as<float4>();
        G.c32[t] = r.cmap32[t].as<float4>();
        G.m16[t] = r.map16[t].as<uint4>();
    }
    G.half = e->precision == SG_PREC_FP32_H16;
    return G;
}

// every grid type the models look up has its packed maps
static void check_packed(const sg_engine* e, const RecState& r, const sg_model_desc* models, int nmodels) {
    for (int k = 0; k < nmodels; k++)
        for (int i = 0; i < models[k].num_movable; i++) {
            const int t = models[k].atom_type[i];
            if (t >= kNumTypes || is_h(t)) continue;
            require(r.map32[t].p && (e->precision != SG_PREC_FP32_H16 || r.map16[t].p) &&
                        (e->tables.nc == 1 || r.cmap32[t].p),
                    "mixed-precision maps missing for a ligand type");
        }
}

// Launch shape for chains on teams of `team` warps: chains per block (wpb)
// with the most resident chains per SM (ties: more chains per block, so
// fewer model copies).  A batch that is resident at once takes the shape that
// loads the fullest SM least (one chain per block up to one chain per SM): with
// 8 chains per block throughout, 1,600 chains of 45-atom ligands at 40 steps took
// 255 ms on one B200, with 4 (11 chains on the fullest SM, not 16) 236 ms; 800 took
// 196 and 191 ms.
// False when no shape fits the shared memory.
bool try_launch(sg_engine* e, size_t stage_stride, size_t ws_stride, int max_chains, int team, long long nchains,
                int& wpb, int& occ) {
    const int cands[4] = {8, 4, 2, 1};
    int best_w = 0, best_occ = 0, best_res = 0;
    long long best_load = 1ll << 60;  // chains on the fullest SM; too high while the batch is not resident
    for (int c : cands) {
        if (c * team > 8) continue;
        if (e->force_wpb && c != e->force_wpb) continue;
        if (!e->force_wpb && c > 1 && c / 2 >= max_chains) continue;  // half the chains' warps would idle
        const size_t smem = stage_stride + (size_t)c * team * ws_stride;
        if (smem > (size_t)e->max_smem) continue;
        const int o = mc32_occupancy(team, c * team, smem);
        if (o == 0) continue;
        const long long blocks = (nchains + c - 1) / c, load = (blocks + e->num_sms - 1) / e->num_sms * c;
        const long long fits = load <= (long long)o * c ? load : 1ll << 59;
        if (fits < best_load || (fits == best_load && fits >= 1ll << 59 && o * c > best_res)) {
            best_load = fits;
            best_res = o * c;
            best_w = c;
            best_occ = o;
        }
    }
    wpb = best_w;
    occ = best_occ;
    return best_res > 0;
}

// ---- which chains get a block each ----------------------------------------------------------
// One B200, 40 steps, milliseconds of search, a block of 8 or 4 warps per chain
// against one warp per chain: ligands of 45 heavy atoms and 10 rotors 73 / 111 (8
// chains, 8 warps), 120 / 183 (296, 8 warps), 140 / 190 (592, 4 warps); of 25 and 5
// 31 / 39, 41 / 50 and 51 / 59 (2 warps lost, 71 / 63 at 1,184 chains).  Past that a
// batch of mixed ligands took the 185 ms of its largest ligand's chains from 592 to
// 2,368 chains: there the largest ones get blocks and the others a warp each: 107,
// 126, 139 and 183 ms at 592, 1,184, 1,600 and 2,368 chains, before 177, 185, 187 and
// 204.
//
// A chain's cost on one warp of a full SM, and a block's time on it as a share of
// that, in pairs: an evaluation costs about 300 pairs' time besides its pairs, and
// a block saves about half of the pairs' time and, having fewer neighbours, a
// third of the rest.
static double chain_cost(const DModel& h, unsigned steps, int maxiters) {
    return (double)steps * std::max(1, maxiters) * (300 + h.npairs);
}
static double block_share(const DModel& h, int warps) {
    return (warps == 8 ? 190 + 0.38 * h.npairs : 210 + 0.5 * h.npairs) / (300 + h.npairs);
}
struct PlanJob {  // chains of one ligand, `cost` each
    int job, chains;
    double cost;
    const DModel* h;
};
struct MixPlan {
    int warps = 0, occ = 0, wide_jobs = 0;  // 0 warps: one warp per chain throughout
    size_t smem = 0;
};
// Time of a batch (jobs by falling cost, the first `wide` of them with blocks) on m
// blocks of `warps` warps taking the longest item first: no less than the work over
// the blocks, nor than the q + 1 shortest of the q m + 1 longest items, which share
// a block.
static double mix_time(const std::vector<PlanJob>& jobs, size_t wide, int warps, long long m) {
    double load = 0, span = 0;
    long long items = 0, next = 0;
    size_t a = 0, b = wide;
    while (a < wide || b < jobs.size()) {  // the two kinds merged, longest first
        const double da = a < wide ? jobs[a].cost * block_share(*jobs[a].h, warps) : -1,
                     db = b < jobs.size() ? jobs[b].cost : -1;
        const double d = std::max(da, db);
        const long long n = da >= db ? jobs[a++].chains : (jobs[b++].chains + warps - 1) / warps;
        load += d * n;
        items += n;
        for (; next < items; next += m) span = std::max(span, d * (double)(next / m + 1));
    }
    return std::max(span, load / (double)m);
}
static MixPlan plan_mix(sg_engine* e, const std::vector<PlanJob>& jobs, size_t stage_stride, size_t ws_stride,
                        size_t wide_bytes) {
    MixPlan best;
    double best_time = 0;
    for (int warps : {8, 4}) {
        const size_t smem = stage_stride + ws_stride + std::max((warps - 1) * ws_stride, wide_bytes);
        if (smem > (size_t)e->max_smem) continue;
        const int occ = mc32_mix_occupancy(warps, smem);
        if (occ == 0) continue;
        const long long m = (long long)occ * e->num_sms;
        if (best_time == 0) {
            // one warp per chain, faster the fewer of them share an SM (a full
            // SM's time at 14 or more, 3/4 of it at 2 to 5); a block per chain has
            // to gain more than the estimate's uncertainty
            long long chains = 0;
            for (const PlanJob& q : jobs) chains += q.chains;
            const double full = std::min(1.0, 0.65 + 0.025 * (double)chains / e->num_sms);
            best_time = 0.95 * full * mix_time(jobs, 0, warps, m);
        }
        for (size_t k = 1;; k = std::min(jobs.size(), k + (k + 1) / 2)) {
            const double t = mix_time(jobs, k, warps, m);
            if (t < best_time) {
                best_time = t;
                best.warps = warps;
                best.occ = occ;
                best.wide_jobs = (int)k;
                best.smem = smem;
            }
            if (k == jobs.size()) break;
        }
    }
    return best;
}

void choose_launch(sg_engine* e, size_t stage_stride, size_t ws_stride, int max_chains, int& wpb, int& occ) {
    require(try_launch(e, stage_stride, ws_stride, max_chains, 1, 1ll << 40, wpb, occ),
            "model too large for the mixed-precision path's shared memory");
}

#ifdef SG_PROFILE
cudaError_t profile_read32(unsigned long long* out16, bool clear);
#endif

}  // namespace sg

using namespace sg;

extern "C" {

int sg_dock_batch32(sg_engine* e, int rid, const sg_model_desc* models, int nmodels, const sg_ligand_job* jobs, int njobs,
                    const sg_mc_params* p, int refine, sg_ligand_result* out) {
    return guarded(e, [&] {
        require(jobs && p && out && njobs > 0 && njobs <= (1 << 22), "dock_batch32: bad arguments");
        require(e->precision != SG_PREC_FP64, "dock_batch32 needs an engine created with SG_PREC_FP32 or SG_PREC_FP32_H16");
        require(p->num_saved_mins >= 1 && p->num_saved_mins <= 1024 && p->maxiters >= 0 && p->temperature > 0,
                "dock_batch32: bad search parameters");
        require(!p->visited, "the QuickVina 2 history (visited) runs on the plain path only");
        require(e->has_tables, "no tables set");
        RecState& r = receptor_for(e, rid);
        CallIo io(e);
        PackedModels pm(e);
        pack_models(io, models, nmodels, kPackWide, pm);
        ensure_model_maps(e, r, models, nmodels);
        check_packed(e, r, models, nmodels);
        uint64_t h2d = pm.mem.bytes, d2h = 0;
        size_t ws_stride = 0, stage_stride = 0, wide_bytes = 0;
        bool wide_packed = true;
        for (const DModel& h : pm.host) {
            require(h.npchunks >= 0, "mixed-precision path: at most 255 atoms per model");
            wide_bytes = std::max(wide_bytes, (size_t)wide32_layout(h.npchunks, h.npairs, h.nmov).total);
            wide_packed = wide_packed && h.wstart;
            ws_stride = std::max(ws_stride, ws32_bytes(h));
            stage_stride = std::max(stage_stride, (size_t)stage32_bytes(h.natoms, h.nframes, h.nheavy, h.npchunks,
                                                                        h.nlig, h.nblocks, h.ntors));
        }
        ws_stride = (ws_stride + 15) & ~(size_t)15;
        const int S = p->num_saved_mins;
        // chains of every job, with their result slots
        std::vector<Chain32> hc;
        std::vector<int> chain_job;
        std::vector<size_t> cres_off, xres_off;
        size_t nconf_res = 0, nxyz_res = 0;
        for (int j = 0; j < njobs; j++) {
            const sg_ligand_job& J = jobs[j];
            require(J.model >= 0 && J.model < nmodels && J.num_chains >= 1 && J.num_chains <= (1 << 16) && J.maxiters >= 0,
                    "dock_batch32: bad ligand job");
            require(out[j].e && out[j].conf && out[j].coords, "dock_batch32: null result arrays");
            const DModel& h = pm.host[J.model];
            for (int c = 0; c < J.num_chains; c++) {
                Chain32 ch{};
                ch.model = J.model;
                ch.steps = J.num_steps;
                ch.maxiters = J.maxiters > 0 ? J.maxiters : p->maxiters;
                ch.key0 = (uint32_t)J.seed;
                ch.key1 = (uint32_t)(J.seed >> 32) ^ (uint32_t)(J.ligand_key >> 32);
                ch.lig = (uint32_t)J.ligand_key;
                ch.chain = (uint32_t)c;
                hc.push_back(ch);
                chain_job.push_back(j);
                cres_off.push_back(nconf_res);
                xres_off.push_back(nxyz_res);
                nconf_res += (size_t)S * h.conf_size;
                nxyz_res += (size_t)S * h.nheavy * 3;
            }
        }
        const int nchains = (int)hc.size();
        require(nchains <= (1 << 24), "dock_batch32: too many chains");
        DevBuf d_e(e), d_conf(e), d_xyz(e), d_order(e), d_count(e), d_evals(e), d_hits(e), d_queue(e);
        d_e.alloc((size_t)nchains * S * sizeof(double));
        d_conf.alloc(std::max<size_t>(1, nconf_res) * sizeof(double));
        d_xyz.alloc(std::max<size_t>(1, nxyz_res) * sizeof(float));
        d_order.alloc((size_t)nchains * S * sizeof(int));
        d_count.alloc((size_t)nchains * sizeof(int));
        d_evals.alloc((size_t)nchains * sizeof(unsigned long long));
        d_hits.alloc((size_t)nchains * 2 * sizeof(unsigned long long));
        d_queue.alloc(sizeof(unsigned));
        // chains of no steps never run: nothing found, nothing counted
        cuda_check(cudaMemsetAsync(d_count.p, 0, d_count.bytes, e->stream), "counts");
        cuda_check(cudaMemsetAsync(d_evals.p, 0, d_evals.bytes, e->stream), "counts");
        cuda_check(cudaMemsetAsync(d_hits.p, 0, d_hits.bytes, e->stream), "counts");
        for (int k = 0; k < nchains; k++) {
            Chain32& ch = hc[k];
            ch.out_e = d_e.as<double>() + (size_t)k * S;
            ch.out_conf = d_conf.as<double>() + cres_off[k];
            ch.out_coords = d_xyz.as<float>() + xres_off[k];
            ch.out_order = d_order.as<int>() + (size_t)k * S;
            ch.out_count = d_count.as<int>() + k;
            ch.evals = d_evals.as<unsigned long long>() + k;
            ch.hits = d_hits.as<unsigned long long>() + 2 * k;
        }
        // work items: up to wpb chains of one job; longest first, so the
        // persistent kernel's queue ends evenly
        int max_chains = 1;
        for (int j = 0; j < njobs; j++) max_chains = std::max(max_chains, jobs[j].num_chains);
        // Threads per chain: as set, or (0) the most warps per chain whose
        // resident chains still hold the whole batch (the reference's
        // threads_per_chain, gpu_kernels_impl.cuh:572-605).
        int wpb = 1, occ = 1, team = std::max(1, e->tpc / 32);
        if (e->tpc == 0) {
            team = 1;
            for (int g : {4, 2}) {
                int w = 0, o = 0;
                if (try_launch(e, stage_stride, ws_stride, max_chains, g, nchains, w, o) &&
                    (long long)nchains <= (long long)o * w * e->num_sms) {
                    team = g;
                    break;
                }
            }
        }
        require(!e->force_wpb || e->force_wpb * team <= 8,
                "chains per block (sg_set_chains_per_block) times warps per chain is above 8 warps per block");
        require(try_launch(e, stage_stride, ws_stride, max_chains, team, nchains, wpb, occ),
                "model too large for the mixed-precision path's shared memory at this many threads per chain");
        MCParams32 P{};
        for (int i = 0; i < 3; i++) {
            P.hunt[i] = (float)p->hunt_cap[i];
            P.auth[i] = (float)p->authentic_v[i];
            P.box[i] = r.gd.begin[i];
            P.box[3 + i] = r.gd.end[i];
        }
        P.slope = (float)p->cache_slope;
        P.temperature = p->temperature;
        P.amplitude = p->mutation_amplitude;
        P.min_rmsd = p->min_rmsd;
        P.num_saved = S;
        P.maxiters = p->maxiters;
        P.accurate_line = p->accurate_line;
        P.early_term = p->early_term;
        // Early stop (--fast): phases ending at (first + k) / checkpoints of
        // every chain's steps, each resuming from the state the previous one
        // saved; the stopping rule between phases.  Without it, one phase.
        const bool phased = e->es_on;
        int es_n = 1, es_first = 1;
        if (phased) {
            es_n = std::max(1, e->es.checkpoints);
            es_first = std::min(es_n, std::max(1, e->es.first));
        }
        const int nphases = es_n - es_first + 1;
        std::vector<size_t> res_off(nchains, 0);
        DevBuf d_resume(e);
        if (phased) {
            size_t nres = 0;
            for (int k = 0; k < nchains; k++) {
                const DModel& h = pm.host[hc[k].model];
                res_off[k] = nres;
                nres += (resume32_doubles(h.conf_size, h.natoms, h.nframes) + 1) & ~(size_t)1;  // 16-byte pieces
            }
            d_resume.alloc(std::max<size_t>(1, nres) * sizeof(double));
            for (int k = 0; k < nchains; k++) hc[k].resume = d_resume.as<double>() + res_off[k];
        }
        std::vector<unsigned> done(nchains, 0);
        std::vector<char> stopped(njobs, 0);
        std::vector<double> hres;
        DevBuf d_chains(e), d_items(e);
        float mc_ms = 0;
        int first_blocks = 0, first_wpb = wpb, first_warps = 0, first_wide = 0;
        cudaEvent_t ev[4];
        for (auto& x : ev) cuda_check(cudaEventCreate(&x), "event");
        struct EvGuard {
            cudaEvent_t* v;
            ~EvGuard() { for (int i = 0; i < 4; i++) cudaEventDestroy(v[i]); }
        } evg{ev};
        for (int ph = 0; ph < nphases; ph++) {
            std::vector<int> active;
            for (int k = 0; k < nchains; k++) {
                if (stopped[chain_job[k]]) continue;
                const unsigned steps = hc[k].steps;
                const unsigned end = ph + 1 < nphases
                                         ? (unsigned)(((unsigned long long)steps * (es_first + ph) + es_n - 1) / es_n)
                                         : steps;
                if (end <= done[k]) continue;
                hc[k].begin = done[k];
                hc[k].end = end;
                done[k] = end;
                active.push_back(k);
            }
            if (active.empty()) continue;
            // the ligands by falling cost, and which of them get a block per chain
            std::vector<PlanJob> jobs_by_cost;
            for (size_t a = 0; a < active.size();) {
                const int k = active[a], j = chain_job[k];
                int n = 0;
                while (a + n < active.size() && chain_job[active[a + n]] == j) n++;
                const DModel& h = pm.host[hc[k].model];
                jobs_by_cost.push_back({j, n, chain_cost(h, hc[k].end - hc[k].begin, hc[k].maxiters), &h});
                a += n;
            }
            std::stable_sort(jobs_by_cost.begin(), jobs_by_cost.end(),
                             [](const PlanJob& a, const PlanJob& b) { return a.cost > b.cost; });
            MixPlan mix;
            if (team == 1 && wide_packed && !e->force_wpb) mix = plan_mix(e, jobs_by_cost, stage_stride, ws_stride, wide_bytes);
            std::vector<char> has_block(njobs, 0);
            std::vector<double> cost(njobs, 0);
            for (size_t k = 0; k < jobs_by_cost.size(); k++) {
                const PlanJob& q = jobs_by_cost[k];
                has_block[q.job] = (int)k < mix.wide_jobs;
                cost[q.job] = q.cost * (has_block[q.job] ? block_share(*q.h, mix.warps) : 1.0);
            }
            const int per_item = mix.warps ? mix.warps : wpb;
            std::vector<Item32> items;
            std::vector<double> item_cost;
            for (size_t a = 0; a < active.size();) {
                const int k = active[a], j = chain_job[k];
                const int most = has_block[j] ? 1 : per_item;
                int n = 0;
                while (a + n < active.size() && chain_job[active[a + n]] == j && n < most && active[a + n] == k + n) n++;
                items.push_back(Item32{hc[k].model, k, n, has_block[j]});
                item_cost.push_back(cost[j]);
                a += n;
            }
            std::vector<int> order(items.size());
            std::iota(order.begin(), order.end(), 0);
            std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return item_cost[x] > item_cost[y]; });
            std::vector<Item32> queue(items.size());
            for (size_t k = 0; k < items.size(); k++) queue[k] = items[order[k]];
            const int nitems = (int)queue.size();
            const int blocks = (int)std::min<long long>((long long)(mix.warps ? mix.occ : occ) * e->num_sms, nitems);
            if (first_blocks == 0) {
                first_blocks = blocks;
                first_warps = mix.warps;
                first_wide = mix.wide_jobs;
                first_wpb = !mix.warps ? wpb : mix.wide_jobs == (int)jobs_by_cost.size() ? 1 : mix.warps;
            }
            io.in(d_chains, hc.data(), hc.size() * sizeof(Chain32));
            io.in(d_items, queue.data(), queue.size() * sizeof(Item32));
            h2d += d_chains.bytes + d_items.bytes;
            cuda_check(cudaMemsetAsync(d_queue.p, 0, sizeof(unsigned), e->stream), "queue reset");
            cuda_check(cudaEventRecord(ev[0], e->stream), "event");
            cuda_check(mix.warps
                           ? launch_mc32_mix(pm.dmodels, tables32(e), maps32(e, r), d_chains.as<Chain32>(),
                                             d_items.as<Item32>(), nitems, P, d_queue.as<unsigned>(), blocks, mix.warps,
                                             stage_stride, ws_stride, mix.smem, e->stream)
                           : launch_mc32(pm.dmodels, tables32(e), maps32(e, r), nullptr, d_chains.as<Chain32>(),
                                         d_items.as<Item32>(), nitems, P, d_queue.as<unsigned>(), blocks, wpb * team,
                                         stage_stride, ws_stride, team, e->stream),
                       "search launch");
            cuda_check(cudaEventRecord(ev[1], e->stream), "event");
            if (phased && ph + 1 < nphases) {  // the stopping rule on the best energies the chains saved
                hres.resize(d_resume.bytes / sizeof(double));
                cuda_check(cudaMemcpyAsync(hres.data(), d_resume.p, d_resume.bytes, cudaMemcpyDeviceToHost, e->stream),
                           "best energies");
                d2h += d_resume.bytes;
            }
            cuda_check(cudaStreamSynchronize(e->stream), "search");
            float ms = 0;
            cuda_check(cudaEventElapsedTime(&ms, ev[0], ev[1]), "event time");
            mc_ms += ms;
            if (phased && ph + 1 < nphases) {
                const int cpu = e->es.chains_per_unit;
                for (int k0 = 0; k0 < nchains;) {  // per job: its units' best energies
                    const int j = chain_job[k0];
                    int k1 = k0;
                    while (k1 < nchains && chain_job[k1] == j) k1++;
                    if (!stopped[j]) {
                        std::vector<double> ub;
                        for (int k = k0; k < k1; k++) {
                            const size_t u = (size_t)((k - k0) / cpu);
                            if (ub.size() <= u) ub.resize(u + 1, DBL_MAX);
                            const int cs = pm.host[hc[k].model].conf_size;
                            ub[u] = std::min(ub[u], hres[res_off[k] + cs + 1]);
                        }
                        if (ub.size() >= 2) {
                            const double best = *std::min_element(ub.begin(), ub.end());
                            int agree = 0;
                            for (double v : ub) agree += (v - best <= e->es.eps);
                            const int need = std::max(2, (int)std::ceil(e->es.fraction * ub.size() - 1e-9));
                            if (agree >= need) stopped[j] = 1;
                        }
                    }
                    k0 = k1;
                }
            }
        }
        const int blocks = first_blocks;
        if (!d_chains.p) io.in(d_chains, hc.data(), hc.size() * sizeof(Chain32));  // no chain had steps
        // merge_output_containers per ligand (chains in job order), then
        // refine_structure of every merged pose, FP64 on the direct sum: both on
        // the device, S places per ligand
        const int cs = pm.max_conf, hs = std::max(1, pm.max_heavy);
        const size_t nplaces = (size_t)njobs * S;
        require(nplaces <= (size_t)1 << 30, "dock_batch32: too many results");
        std::vector<MergeJob32> mj(njobs);
        for (int j = 0, c = 0; j < njobs; j++) {
            mj[j] = {jobs[j].model, c, jobs[j].num_chains};
            c += jobs[j].num_chains;
        }
        DevBuf d_mj(e), d_n(e), dpm(e), de(e), dc(e), dx(e), dmi(e);
        io.in(d_mj, mj.data(), mj.size() * sizeof(MergeJob32));
        h2d += d_mj.bytes;
        d_n.alloc(njobs * sizeof(int));
        dpm.alloc(nplaces * sizeof(int));
        de.alloc(nplaces * sizeof(double));
        dc.alloc(nplaces * cs * sizeof(double));
        dx.alloc(nplaces * hs * 3 * sizeof(double));
        cuda_check(launch_merge32(pm.dmodels, d_mj.as<MergeJob32>(), njobs, d_chains.as<Chain32>(), S, 2.0, d_n.as<int>(),
                                  dpm.as<int>(), de.as<double>(), dc.as<double>(), cs, dx.as<double>(), 3 * hs,
                                  e->stream),
                   "merge launch");
        float ref_ms = 0;
        if (refine) {
            std::vector<int> pmaxit(nplaces);
            for (int j = 0; j < njobs; j++)
                std::fill_n(pmaxit.begin() + (size_t)j * S, S, jobs[j].maxiters > 0 ? jobs[j].maxiters : p->maxiters);
            io.in(dmi, pmaxit.data(), pmaxit.size() * sizeof(int));
            h2d += dmi.bytes;
            const Shape64 sh = plain_shape(e, pm, nplaces, Work64::refine);
            cuda_check(cudaEventRecord(ev[2], e->stream), "event");
            cuda_check(launch_refine64(pm.dmodels, sh, e->tables, r.dhdr.as<DReceptor>(), dpm.as<int>(), (int)nplaces,
                                       dc.as<double>(), cs, p->authentic_v, p->maxiters, dmi.as<int>(), nullptr,
                                       p->accurate_line, p->early_term, de.as<double>(), dx.as<double>(), hs,
                                       e->d_err.as<int>(), e->stream),
                       "refine launch");
            cuda_check(cudaEventRecord(ev[3], e->stream), "event");
        }
        std::vector<double> he(nplaces), hconf(nplaces * cs), hxyz(nplaces * hs * 3);
        std::vector<int> hn(njobs);
        std::vector<unsigned long long> hev(nchains), hhits(2 * (size_t)nchains);
        auto fetch = [&](void* dst, const DevBuf& src, size_t bytes) {
            io.out(dst, src.p, bytes);
            d2h += bytes;
        };
        fetch(hn.data(), d_n, hn.size() * sizeof(int));
        fetch(he.data(), de, he.size() * sizeof(double));
        fetch(hconf.data(), dc, hconf.size() * sizeof(double));
        fetch(hxyz.data(), dx, hxyz.size() * sizeof(double));
        fetch(hev.data(), d_evals, hev.size() * sizeof(unsigned long long));
        fetch(hhits.data(), d_hits, hhits.size() * sizeof(unsigned long long));
        io.finish();
        if (refine) cuda_check(cudaEventElapsedTime(&ref_ms, ev[2], ev[3]), "event time");
        uint64_t tot_evals = 0, tot_grid = 0, tot_pair = 0;
        std::vector<uint64_t> job_evals(njobs, 0);
        for (int k = 0; k < nchains; k++) {
            job_evals[chain_job[k]] += hev[k];
            tot_evals += hev[k];
            tot_grid += hhits[2 * k];
            tot_pair += hhits[2 * k + 1];
        }
        std::vector<int> order(S);
        for (int j = 0; j < njobs; j++) {
            const DModel& h = pm.host[jobs[j].model];
            const int n = std::min(std::max(hn[j], 0), S);
            const double* ej = &he[(size_t)j * S];
            std::iota(order.begin(), order.begin() + n, 0);  // best first (refinement may have changed the order)
            std::stable_sort(order.begin(), order.begin() + n, [&](int a, int b) { return ej[a] < ej[b]; });
            out[j].count = n;
            out[j].evals = job_evals[j];
            for (int i = 0; i < n; i++) {
                const size_t q = (size_t)j * S + order[i];
                out[j].e[i] = he[q];
                std::memcpy(out[j].conf + (size_t)i * h.conf_size, &hconf[q * cs], h.conf_size * sizeof(double));
                std::memcpy(out[j].coords + (size_t)i * h.nheavy * 3, &hxyz[q * hs * 3], (size_t)h.nheavy * 3 * sizeof(double));
            }
        }
        e->last_wpb = first_wpb;
        e->last_team = team;
        e->last_blocks = blocks;
        e->last_block_warps = first_warps;
        e->last_block_ligands = first_wide;
        e->last_mc_ms = mc_ms;
        e->last_refine_ms = ref_ms;
        e->last_evals = tot_evals;
        e->last_grid_hits = tot_grid;
        e->last_pair_hits = tot_pair;
        e->last_h2d = h2d;
        e->last_d2h = d2h;
    });
}

int sg_batch_stats(const sg_engine* e, double* mc_ms, double* refine_ms, int* chains_per_block, int* blocks) {
    if (!e) return SG_ERR_ARG;
    if (mc_ms) *mc_ms = e->last_mc_ms;
    if (refine_ms) *refine_ms = e->last_refine_ms;
    if (chains_per_block) *chains_per_block = e->last_wpb;
    if (blocks) *blocks = e->last_blocks;
    return SG_OK;
}

int sg_batch_blocks(const sg_engine* e, int* warps, int* ligands) {
    if (!e) return SG_ERR_ARG;
    if (warps) *warps = e->last_block_warps;
    if (ligands) *ligands = e->last_block_ligands;
    return SG_OK;
}

int sg_batch_counters(const sg_engine* e, uint64_t* evals, uint64_t* grid_lookups, uint64_t* pair_lookups,
                      uint64_t* h2d_bytes, uint64_t* d2h_bytes) {
    if (!e) return SG_ERR_ARG;
    if (evals) *evals = e->last_evals;
    if (grid_lookups) *grid_lookups = e->last_grid_hits;
    if (pair_lookups) *pair_lookups = e->last_pair_hits;
    if (h2d_bytes) *h2d_bytes = e->last_h2d;
    if (d2h_bytes) *d2h_bytes = e->last_d2h;
    return SG_OK;
}

#ifdef SG_PROFILE
// profiling builds only: clock64() cycles per section summed over warps
int sg_profile_read(unsigned long long* out16, int clear) {
    return profile_read32(out16, clear != 0) == cudaSuccess ? SG_OK : SG_ERR_CUDA;
}
#endif

int sg_set_early_stop(sg_engine* e, const sg_early_stop* es) {
    if (!e) return SG_ERR_ARG;
    if (!es) {
        e->es_on = false;
        return SG_OK;
    }
    if (e->precision == SG_PREC_FP64 || es->checkpoints < 1 || es->checkpoints > 1000 || es->first < 1 ||
        !(es->fraction >= 0 && es->fraction <= 1) || !(es->eps == es->eps) || es->chains_per_unit < 1)
        return SG_ERR_ARG;
    e->es = *es;
    e->es_on = true;
    return SG_OK;
}

int sg_set_threads_per_chain(sg_engine* e, int threads) {
    if (!e || !(threads == 0 || threads == 32 || threads == 64 || threads == 128)) return SG_ERR_ARG;
    e->tpc = threads;
    return SG_OK;
}

int sg_threads_per_chain(const sg_engine* e, int* configured, int* last_batch) {
    if (!e) return SG_ERR_ARG;
    if (configured) *configured = e->tpc;
    if (last_batch) *last_batch = 32 * e->last_team;
    return SG_OK;
}

int sg_set_chains_per_block(sg_engine* e, int n) {
    if (!e || !(n == 0 || n == 1 || n == 2 || n == 4 || n == 8)) return SG_ERR_ARG;
    e->force_wpb = n;
    return SG_OK;
}

int sg_autotune32(sg_engine* e, int rid, const sg_model_desc* models, int nmodels, const sg_ligand_job* jobs, int njobs,
                  const sg_mc_params* p, double step_fraction, double* evals_per_s, int* chosen) {
    if (!e || !jobs || !p || njobs <= 0 || !(step_fraction > 0 && step_fraction <= 1)) return SG_ERR_ARG;
    return guarded(e, [&] {
        const int cands[4] = {8, 4, 2, 1};
        const int keep = e->force_wpb;
        // the sample: every job with its step count scaled (at least one step)
        std::vector<sg_ligand_job> sample(jobs, jobs + njobs);
        for (auto& j : sample) j.num_steps = std::max(1, (int)(j.num_steps * step_fraction));
        const int S = p->num_saved_mins;
        int max_conf = 1, max_heavy = 1;
        for (int k = 0; k < nmodels && models; k++) {
            max_conf = std::max(max_conf, models[k].conf_size);
            max_heavy = std::max(max_heavy, models[k].num_movable);  // bounds the heavy atoms
        }
        std::vector<double> se((size_t)njobs * std::max(S, 1)), sc((size_t)njobs * std::max(S, 1) * max_conf),
            sx((size_t)njobs * std::max(S, 1) * max_heavy * 3);
        std::vector<sg_ligand_result> res(njobs);
        for (int j = 0; j < njobs; j++)
            res[j] = {0, &se[(size_t)j * S], &sc[(size_t)j * S * max_conf], &sx[(size_t)j * S * max_heavy * 3], 0};
        double best = -1;
        int best_c = 0, kept = keep;
        for (int i = 0; i < 5; i++) {  // the shapes, then what sg_dock_batch32 picks by itself
            const bool automatic = i == 4;
            if (!automatic && evals_per_s) evals_per_s[i] = 0;
            e->force_wpb = automatic ? 0 : cands[i];
            const int rc = sg_dock_batch32(e, rid, models, nmodels, sample.data(), njobs, p, 0, res.data());
            if (rc != SG_OK && rc != SG_ERR_ARG) {  // a device error ends the search; the shape stays as it was
                e->force_wpb = keep;
                throw EngineError(rc, std::string(e->err));
            }
            const int c = e->last_wpb;
            if (rc != SG_OK || (!automatic && c != cands[i]) || e->last_mc_ms <= 0) continue;  // shape not possible here
            const double v = (double)e->last_evals / (e->last_mc_ms * 1e-3);
            if (v > best) {
                best = v;
                best_c = c;
                kept = automatic ? 0 : c;
                if (evals_per_s) evals_per_s[std::find(cands, cands + 4, c) - cands] = v;
            } else if (automatic && c == best_c && e->last_block_ligands == 0) {
                kept = 0;  // the same launch as the fastest shape's
            }
            if (!automatic && evals_per_s) evals_per_s[i] = v;
        }
        e->force_wpb = kept;
        if (chosen) *chosen = best_c;
        require(best_c, "autotune: no launch shape ran (" + e->err + ")");
    });
}

}  // extern "C"
