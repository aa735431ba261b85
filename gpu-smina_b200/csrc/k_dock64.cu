// Plain (FP64) path kernels: one block of G warps per item (a conf, a pose or a
// chain); the first warp runs the item and the others take parts of every
// evaluation (dock64_eval.cuh).  Built with -fmad=false so that the arithmetic
// rounds exactly like the CPU restatement compiled with -ffp-contract=off.
#include <algorithm>
#include "dock64_search.cuh"

namespace sg {

// copies n elements behind the workspace
template <int G, typename T>
__device__ __forceinline__ void stage64(int at, const T* src, int n) {
    T* d = reinterpret_cast<T*>(smem64 + at);
    for (int i = threadIdx.x; i < n; i += 32 * G) d[i] = src[i];
}

// The block's header, staged arrays and model state as read (coords and frame
// origins, which mutation reads before the first evaluation).  Every thread
// takes part.
template <int G, bool ST>
__device__ __forceinline__ void init64(const DModel* gm, const DTables& T, const DReceptor* R, const double* box,
                                       int* err) {
    Hdr64& H = hd64();
    static_assert(sizeof(DModel) % 16 == 0, "DModel is read in 16-byte pieces");
    for (int k = threadIdx.x; k < (int)(sizeof(DModel) / 16); k += 32 * G)
        reinterpret_cast<int4*>(&H.m)[k] = reinterpret_cast<const int4*>(gm)[k];
    __syncthreads();
    if (threadIdx.x == 0) {
        H.T = T;
        H.box = box;
        H.err = err;
        H.evals = 0;
        H.L = ws64_layout(H.m.natoms, H.m.nframes, H.m.npairs, H.m.conf_size, H.m.dof, ST, H.m.nheavy, H.m.nlevels,
                          H.m.nlig, H.m.nblocks, H.m.ntors);
        H.R = ST ? reinterpret_cast<const DReceptor*>(smem64 + H.L.s_receptor) : R;
    }
    __syncthreads();
    const DModel& m = H.m;
    const Ws64& L = H.L;
    double* S = smem64;
    if constexpr (ST) {
        const int N = m.natoms, F = m.nframes;
        static_assert(sizeof(DReceptor) % 8 == 0, "the receptor header is copied in 8-byte pieces");
        stage64<G>(L.s_receptor, reinterpret_cast<const double*>(R), (int)(sizeof(DReceptor) / 8));
        uint16_t* csr = reinterpret_cast<uint16_t*>(smem64 + L.s_csr);
        if (L.s_csr)
            for (int i = threadIdx.x; i < m.csr_start[m.nmov]; i += 32 * G) csr[i] = (uint16_t)m.csr[i];
        stage64<G>(L.s_type, m.type, N);
        stage64<G>(L.s_atom_frame, m.atom_frame, N);
        stage64<G>(L.s_csr_start, m.csr_start, m.nmov + 1);
        stage64<G>(L.s_heavy, m.heavy, m.nheavy);
        stage64<G>(L.s_fkind, m.fkind, F);
        stage64<G>(L.s_fparent, m.fparent, F);
        stage64<G>(L.s_fbegin, m.fbegin, F);
        stage64<G>(L.s_fend, m.fend, F);
        stage64<G>(L.s_fconf, m.fconf, F);
        stage64<G>(L.s_fdof, m.fdof, F);
        stage64<G>(L.s_level_start, m.level_start, m.nlevels + 1);
        stage64<G>(L.s_level_frames, m.level_frames, F);
        stage64<G>(L.s_child_start, m.child_start, F + 1);
        stage64<G>(L.s_child_list, m.child_list, m.child_start[F]);
        stage64<G>(L.s_lig_begin, m.lig_begin, m.nlig);
        stage64<G>(L.s_lig_end, m.lig_end, m.nlig);
        stage64<G>(L.s_lig_root, m.lig_root, m.nlig);
        stage64<G>(L.s_lig_pair_end, m.lig_pair_end, m.nlig);
        stage64<G>(L.s_blk_rigid, m.blk_rigid, m.nblocks);
        stage64<G>(L.s_blk_conf, m.blk_conf, m.nblocks);
        stage64<G>(L.s_blk_ntors, m.blk_ntors, m.nblocks);
        stage64<G>(L.s_tor_conf, m.tor_conf, m.ntors);
        stage64<G>(L.s_tor_dof, m.tor_dof, m.ntors);
        stage64<G>(L.s_charge, m.charge, N);
        stage64<G>(L.s_local, m.local, 3 * N);
        stage64<G>(L.s_forigin, m.forigin, 3 * F);
        stage64<G>(L.s_faxis, m.faxis, 3 * F);
    }
    for (int i = threadIdx.x; i < 3 * m.natoms; i += 32 * G) S[L.coords + i] = m.lab[i];
    for (int i = threadIdx.x; i < 3 * m.nframes; i += 32 * G) {
        S[L.origin + i] = m.finit[i];
        S[L.axis + i] = m.faxis[i];
    }
    for (int f = threadIdx.x; f < m.nframes; f += 32 * G) {
        double* q = S + L.q + 4 * f;
        q[0] = 1; q[1] = 0; q[2] = 0; q[3] = 0;
        quat_to_mat(Quat<double>{1, 0, 0, 0}, S + L.rot + 9 * f);
    }
    __syncthreads();
}

// 128 registers a thread: four resident 4-warp blocks or two 8-warp blocks per SM
#define SG_BOUNDS64 __launch_bounds__(32 * G, G == 1 ? 16 : 16 / G)

// model::eval_deriv for a batch of confs of one model
template <int G, bool ST>
__global__ void SG_BOUNDS64 k_eval64(const DModel* model, const __grid_constant__ DTables T, const DReceptor* R,
                                     int nconfs, const double* confs, double v0, double v1, double v2, double slope,
                                     int direct, double* out_e, double* out_g, double* out_coords, int* err) {
    init64<G, ST>(model, T, R, nullptr, err);
    if (threadIdx.x >= 32) return help64<G, ST>(threadIdx.x >> 5);
    const Hdr64& H = hd64();
    const Ws64& L = H.L;
    const int cs = H.m.conf_size, dof = H.m.dof, nmov = H.m.nmov, lane = lane64();
    double *x = smem64 + L.x_tmp, *g = smem64 + L.g;
    const EvalMode em{{v0, v1, v2}, slope, direct != 0};
    for (int k = blockIdx.x; k < nconfs; k += gridDim.x) {
        vcopy(x, confs + (size_t)k * cs, cs);
        const double e = feval<G, ST>(x, g, em);
        if (lane == 0) out_e[k] = e;
        for (int i = lane; i < dof; i += 32) out_g[(size_t)k * dof + i] = g[i];
        if (out_coords)
            for (int i = lane; i < 3 * nmov; i += 32) out_coords[(size_t)k * 3 * nmov + i] = smem64[L.coords + i];
        __syncwarp();
    }
    release64<G>();
}

// quasi_newton on the grid maps, a conf per block (confs updated in place).  Confs
// take very different numbers of evaluations: blocks that each looped over a fixed
// share of them took 20 to 50 % longer past one resident batch.
template <int G, bool ST>
__global__ void SG_BOUNDS64 k_bfgs64(const DModel* model, const __grid_constant__ DTables T, const DReceptor* R,
                                     int nconfs, double* confs, double v0, double v1, double v2, double slope,
                                     int maxiters, int accurate, int early, double* out_e, int* err) {
    const int k = blockIdx.x;
    if (k >= nconfs) return;
    init64<G, ST>(model, T, R, nullptr, err);
    if (threadIdx.x >= 32) return help64<G, ST>(threadIdx.x >> 5);
    const int cs = hd64().m.conf_size, lane = lane64();
    double* x = smem64 + hd64().L.x_tmp;
    const EvalMode em{{v0, v1, v2}, slope, false};
    vcopy(x, confs + (size_t)k * cs, cs);
    const double e = bfgs64<G, ST>(x, maxiters, accurate, early, em);
    if (lane == 0) out_e[k] = e;
    for (int i = lane; i < cs; i += 32) confs[(size_t)k * cs + i] = x[i];
    release64<G>();
}

// monte_carlo::operator() for one chain per block
// VIS: chains may carry a QuickVina 2 history (a separate instantiation, so
// smina's own search compiles exactly as without it)
template <int G, bool ST, bool VIS>
__global__ void SG_BOUNDS64 k_mc64(const DModel* models, const __grid_constant__ DTables T, const DReceptor* R,
                                   const Chain64* chains, int nchains, const __grid_constant__ MCParams64 P,
                                   int* err) {
    const int c = blockIdx.x;
    if (c >= nchains) return;
    const Chain64 ch = chains[c];
    init64<G, ST>(models + ch.model, T, R, nullptr, err);
    if (threadIdx.x >= 32) return help64<G, ST>(threadIdx.x >> 5);
    const Hdr64& H = hd64();
    const int cs = H.m.conf_size, lane = lane64();
    uint32_t* mt = mt64();
    for (int i = lane; i < 625; i += 32) mt[i] = ch.mt[i];
    double *tmp = smem64 + H.L.x_tmp, *cand = smem64 + H.L.x_cand;
    vcopy(tmp, ch.conf0, cs);
    if (lane == 0) *ch.out_count = 0;
    __syncwarp();
    const EvalMode hunt{{P.hunt[0], P.hunt[1], P.hunt[2]}, P.slope, false};
    const EvalMode auth{{P.auth[0], P.auth[1], P.auth[2]}, P.slope, false};
    Hist64 hist_store{};
    const Hist64* vis = nullptr;
    if (VIS && ch.hist && H.m.dof <= kHistMaxN) {
        hist_store = hist64_view(ch.hist, ch.hist_words, H.m.dof);
        vis = &hist_store;
    }
    double tmp_e = 0, best_e = kMaxFl;
    for (unsigned step = 0; step < ch.steps; step++) {
        vcopy(cand, tmp, cs);
        mutate64<ST>(cand, P.amplitude);
        const double cand_e = bfgs64<G, ST>(cand, ch.maxiters, P.accurate_line, P.early_term, hunt, vis);
        if (step == 0 || metropolis64(tmp_e, cand_e, P.temperature)) {
            vcopy(tmp, cand, cs);
            tmp_e = cand_e;
            set_conf64<ST>(tmp);
            const int count = *ch.out_count;
            if (tmp_e < best_e || count < P.num_saved) {
                tmp_e = bfgs64<G, ST>(tmp, ch.maxiters, P.accurate_line, P.early_term, auth, vis);
                set_conf64<ST>(tmp);
                add_to_output64<ST>(ch, tmp, tmp_e, P.min_rmsd, P.num_saved);
                if (tmp_e < best_e) best_e = tmp_e;
            }
        }
    }
    for (int i = lane; i < 625; i += 32) ch.mt[i] = mt[i];
    if (lane == 0) *ch.evals = H.evals;
    release64<G>();
}

// non_cache::within
template <bool ST>
__device__ __forceinline__ bool within64(double margin) {
    using M = MV64<ST>;
    const Hdr64& H = hd64();
    const DGeom& Gm = H.R->g;
    const int* type = M::type();
    bool ok = true;
    for (int i = lane64(); i < H.m.nmov; i += 32) {
        if (is_h(type[i])) continue;
        for (int j = 0; j < 3; j++)
            if (H.box || Gm.gd_n[j] > 0) {
                const double c = smem64[H.L.coords + 3 * i + j];
                const double lo = H.box ? H.box[j] : Gm.gd_begin[j], hi = H.box ? H.box[3 + j] : Gm.gd_end[j];
                if (c < lo - margin || c > hi + margin) ok = false;
            }
    }
    return __all_sync(kFull, ok);
}

// merge_output_containers of one ligand's chains per block: add_to_output_container
// (coords.cpp:25-58) over the chains in order, each one's poses best first.  The
// list holds the energies (ascending), the poses' places and their columns of D.
// Poses are taken in groups of `group`: all distances of a group's poses to the
// list and to one another at once, one thread each (a pose's squares added in
// order, as the host merge does in double precision), then the first warp takes
// the poses one by one with what D holds.  Once the list is full, poses no better
// than its last one are left out of the groups: they would change nothing.  Bound
// by latency.  For 1,000 chains of one 24-atom ligand (9 poses kept, search 36 ms) a
// call took 37 ms on one B200, for 512 chains of a 10-atom one with up to 1,000 poses
// kept (search 8 ms) 95 ms; without leaving poses out 48 and 161, and with one warp that
// measured each pose when its turn came, and one lane that moved the list, 63 and
// 500 ms.
__host__ __device__ constexpr size_t merge32_bytes(int S, int group) {
    return (size_t)S * (sizeof(double) + sizeof(int2) + sizeof(int)) +
           (size_t)group * (sizeof(double) + sizeof(int2) + (S + group) * sizeof(double)) + 16;
}
constexpr int kMergeThreads = 256;
__global__ void __launch_bounds__(kMergeThreads) k_merge32(const DModel* models, const MergeJob32* jobs,
                                                           const Chain32* chains, int S, int group, double min_rmsd,
                                                           int* out_count, int* pose_model, double* out_e,
                                                           double* out_conf, int conf_stride, double* out_xyz,
                                                           int xyz_stride) {
    extern __shared__ __align__(16) double smem_merge[];
    double* le = smem_merge;               // [S] the list: energies,
    double* D = le + S;                    // [group][S + group] distances
    double* ge = D + (size_t)group * (S + group);  // [group] the group: energies,
    int2* at_list = reinterpret_cast<int2*>(ge + group);  // [S] chain and slot,
    int2* at_group = at_list + S;                         // [group] chain and slot
    int* col = reinterpret_cast<int*>(at_group + group);  // [S] column of D
    __shared__ int s_taken;
    const int j = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const MergeJob32 job = jobs[j];
    const int H = models[job.model].nheavy, H3 = 3 * H, cs = models[job.model].conf_size;
    auto coords = [&](int2 q) { return chains[q.x].out_coords + (size_t)q.y * H3; };
    int n = 0;  // the list's length
    // the first warp's place among the chains: of chains [base, base + 32) those in
    // `todo` are left, the first of them from its pose i on
    const int end = job.first + job.count;
    int base = job.first - 32, i = 0;
    unsigned todo = 0;
    bool nan = false;  // the list holds a NaN, or has
    for (;;) {
        if (tid < 32) {  // the next group
            // a pose that is no better than the last one of a full list changes nothing
            const bool full = n == S && !nan;
            const double worst = full ? le[S - 1] : 0;
            int taken = 0;
            while (taken < group) {
                if (!todo) {  // a chain per lane: has it any pose to offer?
                    base += 32;
                    if (base >= end) break;
                    bool some = false;
                    if (base + lane < end) {
                        const Chain32& ch = chains[base + lane];
                        const int cnt = min(max(*ch.out_count, 0), S);
                        some = cnt > 0 && !full;
                        if (full)
                            for (int k = 0; k < cnt && !some; k++)
                                some = !(ch.out_e[min(max(ch.out_order[k], 0), S - 1)] >= worst);
                    }
                    todo = __ballot_sync(kFull, some);
                    continue;
                }
                const int c = base + __ffs(todo) - 1;
                const Chain32& ch = chains[c];
                const int cnt = min(max(*ch.out_count, 0), S), k = min(min(cnt - i, group - taken), 32);
                int slot = 0;
                double e = 0;
                if (lane < k) {
                    slot = min(max(ch.out_order[i + lane], 0), S - 1);
                    e = ch.out_e[slot];
                }
                const unsigned mask = __ballot_sync(kFull, lane < k && !(full && e >= worst));
                if (mask >> lane & 1) {
                    const int at = taken + __popc(mask & ((1u << lane) - 1));
                    at_group[at] = make_int2(c, slot);
                    ge[at] = e;
                }
                taken += __popc(mask);
                i += k;
                if (i >= cnt) { todo &= todo - 1; i = 0; }
            }
            if (lane == 0) s_taken = taken;
        }
        __syncthreads();
        const int g = s_taken;
        if (g == 0) break;
        for (int t = tid; t < g * (n + g); t += kMergeThreads) {
            const int p = t / (n + g), q = t - p * (n + g);
            if (q >= n + p) continue;
            const float *x = coords(at_group[p]), *y = coords(q < n ? at_list[q] : at_group[q - n]);
            double acc = 0;
#pragma unroll 6
            for (int a = 0; a < H3; a++) {
                const double d = (double)x[a] - (double)y[a];
                acc += d * d;
            }
            D[p * (S + group) + q] = H3 ? sqrt(acc / (double)H) : 0.0;
        }
        for (int k = tid; k < n; k += kMergeThreads) col[k] = k;
        __syncthreads();
        if (tid < 32) {
            const int n0 = n;
            for (int p = 0; p < g; p++) {
                const double* d = D + p * (S + group);
                const double e = ge[p];
                double best = kMaxFl;
                int bi = n;
                for (int k = lane; k < n; k += 32) {
                    const double r = d[col[k]];
                    if (k == 0 || r < best) { bi = k; best = r; }
                }
                // pose 0's distance stands unless another's is smaller (a NaN there stays)
                if (__shfl_sync(kFull, best != best, 0)) {
                    bi = 0;
                    best = __shfl_sync(kFull, best, 0);
                } else {
                    for (int o = 16; o > 0; o >>= 1) {
                        const double ob = __shfl_xor_sync(kFull, best, o);
                        const int oi = __shfl_xor_sync(kFull, bi, o);
                        if (ob < best || (ob == best && oi < bi)) { best = ob; bi = oi; }
                    }
                }
                int at = -1;  // the place it takes
                if (bi < n && best < min_rmsd) {
                    if (e < le[bi]) at = bi;
                } else if (n < S) {
                    at = n++;
                } else if (n > 0 && e < le[n - 1]) {
                    at = n - 1;
                }
                __syncwarp();
                if (at < 0) continue;
                nan |= e != e;
                // sorted in behind the last energy before `at` that is not above its own
                int k = 0;
                for (int b = at - 1; b >= 0; b -= 32) {
                    const unsigned keep = __ballot_sync(kFull, b - lane >= 0 && !(le[b - lane] > e));
                    if (keep) {
                        k = b - __ffs(keep) + 2;
                        break;
                    }
                }
                for (int b = at - 1; b >= k; b -= 32) {  // those in between move up by one, the last ones first
                    const int f = b - lane;
                    double ef = 0;
                    int2 af{};
                    int cf = 0;
                    if (f >= k) { ef = le[f]; af = at_list[f]; cf = col[f]; }
                    __syncwarp();
                    if (f >= k) { le[f + 1] = ef; at_list[f + 1] = af; col[f + 1] = cf; }
                    __syncwarp();
                }
                if (lane == 0) {
                    le[k] = e;
                    at_list[k] = at_group[p];
                    col[k] = n0 + p;
                }
                __syncwarp();
            }
            if (lane == 0) s_taken = n;
        }
        __syncthreads();
        n = s_taken;
        __syncthreads();
    }
    if (tid == 0) out_count[j] = n;
    for (int k = tid >> 5; k < S; k += kMergeThreads / 32) {
        const size_t q = (size_t)j * S + k;
        if (lane == 0) pose_model[q] = k < n ? job.model : -1;
        if (k >= n) continue;
        if (lane == 0) out_e[q] = le[k];
        const double* conf = chains[at_list[k].x].out_conf + (size_t)at_list[k].y * cs;
        const float* x = coords(at_list[k]);
        for (int a = lane; a < cs; a += 32) out_conf[q * conf_stride + a] = conf[a];
        for (int a = lane; a < H3; a += 32) out_xyz[q * xyz_stride + a] = x[a];
    }
}

// refine_structure for one pose per block
template <int G, bool ST>
__global__ void SG_BOUNDS64 k_refine64(const DModel* models, const __grid_constant__ DTables T, const DReceptor* R,
                                       const int* pose_model, int nposes, double* confs, int conf_stride, double c0,
                                       double c1, double c2, int maxiters, const int* pose_maxiters,
                                       const double* pose_box, int accurate, int early, double* out_e,
                                       double* out_coords, int coord_stride, int* err) {
    const int k = blockIdx.x;
    if (k >= nposes || pose_model[k] < 0) return;  // (a place of a ligand's list that holds no pose)
    // the pose's own box, if it has one
    init64<G, ST>(models + pose_model[k], T, R, pose_box ? pose_box + 6 * (size_t)k : nullptr, err);
    if (threadIdx.x >= 32) return help64<G, ST>(threadIdx.x >> 5);
    const Hdr64& H = hd64();
    const int cs = H.m.conf_size, lane = lane64(), nheavy = H.m.nheavy;
    double* x = smem64 + H.L.x_tmp;
    vcopy(x, confs + (size_t)k * conf_stride, cs);
    if (pose_maxiters) maxiters = pose_maxiters[k];  // per-ligand iteration limit
    double slope = 10;
    double e = 0;
    for (int p = 0; p < 5; p++) {
        const EvalMode em{{c0, c1, c2}, slope, true};
        e = bfgs64<G, ST>(x, maxiters, accurate, early, em);
        set_conf64<ST>(x);
        if (within64<ST>(0.0001)) break;
        slope *= 10;
    }
    if (!within64<ST>(0.0001)) e = kMaxFl;
    if (lane == 0) out_e[k] = e;
    for (int i = lane; i < cs; i += 32) confs[(size_t)k * conf_stride + i] = x[i];
    if (out_coords) {
        const int* heavy = MV64<ST>::heavy();
        for (int a = lane; a < nheavy; a += 32)
            st3(out_coords + ((size_t)k * coord_stride + a) * 3, ld3(smem64 + H.L.coords + 3 * heavy[a]));
    }
    release64<G>();
}

// Final rescoring (finish_docking, main.cpp:257-282): per pose, model::eval on
// the direct receptor sum (model.cpp:938-967 with non_cache::eval) and
// model::eval_intramolecular (model.cpp:1027-1079), both on the fast table,
// plus the heavy-atom coordinates of the pose.
template <int G, bool ST>
__global__ void SG_BOUNDS64 k_score64(const DModel* models, const __grid_constant__ DTables T, const DReceptor* R,
                                      const int* pose_model, int n, const double* confs, int conf_stride, double v0,
                                      double v1, double v2, double slope, double* out_e, double* out_intra,
                                      double* out_coords, int coord_stride, int* err) {
    const int k = blockIdx.x;
    if (k >= n) return;
    init64<G, ST>(models + pose_model[k], T, R, nullptr, err);
    if (threadIdx.x >= 32) return help64<G, ST>(threadIdx.x >> 5);
    const Hdr64& H = hd64();
    const int lane = lane64(), nheavy = H.m.nheavy;
    double* x = smem64 + H.L.x_tmp;
    vcopy(x, confs + (size_t)k * conf_stride, H.m.conf_size);
    const double v[3] = {v0, v1, v2};
    set_frames64<ST>(x);
    command64<G>(kOpScore, v, slope, 1, 0);
    score_warp64<G, ST>(0);
    release64<G>();
    const double e = energy64<ST>();
    const double intra = intramolecular64<ST>(v);
    if (lane == 0) {
        out_e[k] = e;
        out_intra[k] = intra;
    }
    if (out_coords) {
        const int* heavy = MV64<ST>::heavy();
        for (int a = lane; a < nheavy; a += 32)
            st3(out_coords + ((size_t)k * coord_stride + a) * 3, ld3(smem64 + H.L.coords + 3 * heavy[a]));
    }
}

// ---- host launchers -------------------------------------------------------------------------
void Smem64::add(const DModel& h) {
    auto bytes = [&](bool st) {
        return (size_t)ws64_layout(h.natoms, h.nframes, h.npairs, h.conf_size, h.dof, st, h.nheavy, h.nlevels, h.nlig,
                                   h.nblocks, h.ntors).total * sizeof(double);
    };
    pairs = std::max(pairs, h.npairs);
    plain = std::max(plain, bytes(false));
    staged = std::max(staged, bytes(true));
}

// Warps per item: 8 for refinements, whose direct sums keep them busy (one B200, 8
// warps against 4: 9 poses of a 24-atom ligand 1.04 / 1.39 ms, 296 2.2 / 3.0; 1,890 of a
// 50-atom one 52 / 67), but for many of models with hardly any pairs (without pairs
// 1.97 / 1.50 at 592 poses, 20.3 / 13.9 at 10,000; 61 pairs 3.3 / 2.7 at 1,200; 105 pairs 5.7 / 7.0),
// and for few items; 4 for more chains or evaluations on the maps than two per SM (10 steps of
// 700 chains 60.5 / 53.6 ms, of 296 31.2 / 31.8); 1 with nothing staged for models that
// only fit so, and for many local optimisations of models with few pairs, where
// the leaders' serial work fills the device: milliseconds of 4 warps against 1
// without pairs 0.66 / 0.66 at 592 confs, 1.03 / 0.73 at 1,184, 11.7 / 4.4 at 20,000; 174
// pairs 3.1 / 3.7 at 1,184, 5.2 / 4.1 at 2,400, 9.5 / 7.2 at 5,000; 316 pairs 8.1 / 8.5 at
// 2,400, 15.1 / 14.0 at 5,000; 482 pairs 17.6 / 19.5 at 5,000.
Shape64 shape64(const Smem64& s, long long items, Work64 work, int num_sms, size_t max_smem) {
    const size_t xb = kXbuf64 * sizeof(double);
    const bool one = work == Work64::bfgs && s.pairs <= 350 && items > (long long)num_sms * (4 + s.pairs / 30);
    const bool eight = items <= 2LL * num_sms || (work == Work64::refine && s.pairs > 80);
    if (!one && eight && s.staged + 8 * xb <= max_smem)
        return {8, s.staged + 8 * xb};
    if (!one && s.staged + 4 * xb <= max_smem) return {4, s.staged + 4 * xb};
    return {1, s.plain};
}

static cudaError_t prep64(const void* fn, size_t smem) {
    return smem <= 48 * 1024 ? cudaSuccess : raise_dynamic_smem(fn, smem);
}

// launches kernel<G, ST> with the shape's G
#define SG_LAUNCH64(kernel, blocks, ...)                                                        \
    do {                                                                                        \
        cudaError_t rc = cudaSuccess;                                                           \
        if (sh.warps == 8) {                                                                    \
            if ((rc = prep64((const void*)kernel(8, true), sh.smem)) != cudaSuccess) return rc; \
            kernel(8, true)<<<blocks, 256, sh.smem, s>>>(__VA_ARGS__);                          \
        } else if (sh.warps == 4) {                                                             \
            if ((rc = prep64((const void*)kernel(4, true), sh.smem)) != cudaSuccess) return rc; \
            kernel(4, true)<<<blocks, 128, sh.smem, s>>>(__VA_ARGS__);                          \
        } else {                                                                                \
            if ((rc = prep64((const void*)kernel(1, false), sh.smem)) != cudaSuccess) return rc;\
            kernel(1, false)<<<blocks, 32, sh.smem, s>>>(__VA_ARGS__);                          \
        }                                                                                       \
        return cudaGetLastError();                                                              \
    } while (0)

// blocks that loop over the confs of one model: the model is staged once per block
static int loop_blocks(const Shape64& sh, int n, int num_sms) { return std::min(n, num_sms * (16 / sh.warps)); }

#define SG_K_EVAL(G, ST) k_eval64<G, ST>
#define SG_K_BFGS(G, ST) k_bfgs64<G, ST>
#define SG_K_MC(G, ST) k_mc64<G, ST, false>
#define SG_K_MC_VIS(G, ST) k_mc64<G, ST, true>
#define SG_K_REFINE(G, ST) k_refine64<G, ST>
#define SG_K_SCORE(G, ST) k_score64<G, ST>

cudaError_t launch_eval64(const DModel* dm, const Shape64& sh, int num_sms, const DTables& T, const DReceptor* R, int n,
                          const double* confs, const double v[3], double slope, int direct, double* e, double* g,
                          double* coords, int* err, cudaStream_t s) {
    SG_LAUNCH64(SG_K_EVAL, loop_blocks(sh, n, num_sms), dm, T, R, n, confs, v[0], v[1], v[2], slope, direct, e, g, coords,
                err);
}

cudaError_t launch_bfgs64(const DModel* dm, const Shape64& sh, const DTables& T, const DReceptor* R, int n,
                          double* confs, const double v[3], double slope, int maxiters, int accurate, int early,
                          double* e, int* err, cudaStream_t s) {
    SG_LAUNCH64(SG_K_BFGS, n, dm, T, R, n, confs, v[0], v[1], v[2], slope, maxiters, accurate,
                early, e, err);
}

cudaError_t launch_mc64(const DModel* dms, const Shape64& sh, const DTables& T, const DReceptor* R,
                        const Chain64* chains, int n, const MCParams64& P, bool visited, int* err, cudaStream_t s) {
    if (visited) SG_LAUNCH64(SG_K_MC_VIS, n, dms, T, R, chains, n, P, err);
    SG_LAUNCH64(SG_K_MC, n, dms, T, R, chains, n, P, err);
}

cudaError_t launch_refine64(const DModel* dms, const Shape64& sh, const DTables& T, const DReceptor* R,
                            const int* pose_model, int n, double* confs, int conf_stride, const double cap[3],
                            int maxiters, const int* pose_maxiters, const double* pose_box, int accurate, int early,
                            double* e, double* coords, int coord_stride, int* err, cudaStream_t s) {
    SG_LAUNCH64(SG_K_REFINE, n, dms, T, R, pose_model, n, confs, conf_stride, cap[0], cap[1], cap[2], maxiters,
                pose_maxiters, pose_box, accurate, early, e, coords, coord_stride, err);
}

// merges njobs ligands' chains into S places each (conf_stride and xyz_stride
// doubles apart); places past a ligand's count get pose_model -1
cudaError_t launch_merge32(const DModel* dms, const MergeJob32* jobs, int njobs, const Chain32* chains, int S,
                           double min_rmsd, int* count, int* pose_model, double* e, double* conf, int conf_stride,
                           double* xyz, int xyz_stride, cudaStream_t s) {
    // groups as large as 48 KB allow (32 up to 120 places or so), else of 8 poses
    const int group = merge32_bytes(S, 32) <= 48 * 1024 ? 32 : 8;
    const size_t smem = merge32_bytes(S, group);
    if (smem > 48 * 1024 - 64) {
        const cudaError_t rc = raise_dynamic_smem((const void*)k_merge32, smem);
        if (rc != cudaSuccess) return rc;
    }
    k_merge32<<<njobs, kMergeThreads, smem, s>>>(dms, jobs, chains, S, group, min_rmsd, count, pose_model, e, conf,
                                                 conf_stride, xyz, xyz_stride);
    return cudaGetLastError();
}

cudaError_t launch_score64(const DModel* dms, const Shape64& sh, const DTables& T, const DReceptor* R,
                           const int* pose_model, int n, const double* confs, int conf_stride, const double v[3],
                           double slope, double* e, double* intra, double* coords, int coord_stride, int* err,
                           cudaStream_t s) {
    SG_LAUNCH64(SG_K_SCORE, n, dms, T, R, pose_model, n, confs, conf_stride, v[0], v[1], v[2], slope, e, intra, coords,
                coord_stride, err);
}

}  // namespace sg
