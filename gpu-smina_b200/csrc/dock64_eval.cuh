// Plain (FP64) path, part 1: a block of G warps evaluates model::eval_deriv.
//
// Bit-exact with a CPU FP64 run when compiled with -fmad=false: every
// reduction whose order matters is done in the reference's order (per-atom
// force accumulation over an ordered pair list, sequential energy sums,
// per-frame force/torque sums in atom order, children added in order).
// Reference: model.cpp:837-841,904-928,969-985; grid.cpp:27-46,111-236;
// cache.cpp:69-90; non_cache.cpp:109-191; tree.h:108-243;
// precalculate.h:111-151,245-293.
//
// What bounds it: latency.  An item (a pose or a chain) is one serial chain of
// evaluations, and inside an evaluation the sums have to stay in order.  So the
// terms of those sums are computed by all warps at once and only the additions
// stay serial, as few dependent FP64 adds as the order allows:
//  - frames: the half angles' sines and cosines need no parent, so all torsions
//    compute them at once before the level-by-level composition;
//  - direct receptor sum: 8 lanes per atom compute 8 terms at a time from a
//    packed list (CellAtom, 32 B), pass them through shared memory and 4 of the
//    lanes add energy, x, y and z in list order; terms beyond the cutoff are
//    squeezed out, not added;
//  - pairs: one thread each; a pair beyond the cutoff leaves +0 (adding +0
//    changes no bit of a sum that starts at +0), so no flags are read back;
//  - forces: one thread per (atom, axis) adds its pairs in pair order;
//  - energy: the last warp adds the ordered energy sums while the others add
//    forces and the first warp walks the tree back.
// Measured on one B200 against one warp per item with everything read from
// global memory and lane 0 adding the sums, with calls: refinement of 1,890 poses
// of 210 ligands 197 -> 21 ms, of 9 poses of one ligand 6.3 -> 1.1 ms; 8 chains of 40
// steps 78 -> 62 ms; kernels alone: rescoring of 2,000 poses 0.54 -> 0.18 ms, 1,500
// charge-dependent evaluations 126 -> 77 us.  Bits unchanged.  What is left of an
// evaluation is the leader's instructions, about 3,400 of them at 7 to 8 cycles each
// (frames, tree derivative, BFGS); four lanes per frame (6,500 -> 9,100 cycles an
// evaluation) and one per frame and component (5,900 -> 7,400) took more
// instructions.
// The first warp, the leader, runs the chain (BFGS, line searches, mutation)
// and calls the others in for each evaluation: two numbers of warps (4 and 8)
// by the number of items, plus one warp with nothing staged for models whose
// staged form does not fit an SM's shared memory and for batches of small local
// optimisations (shape64).  There 16 warps of an SM are at 16 places of the code, so
// it is instruction fetch that bounds them: loops that the paths of several warps
// unroll stay rolled with one, and lane-strided loops with any (20,000 local
// optimisations of a 10-atom ligand 5.8 -> 3.9 ms on one B200).
#pragma once
#include "grid64.cuh"

namespace sg {

constexpr unsigned kFull = 0xffffffffu;

// Shared memory of a block: the header Hdr64, then the workspace (Ws64).  With ST
// the model's small arrays and the receptor header are copied behind it;
// without, they stay in global memory.
extern __shared__ __align__(16) double smem64[];
__device__ __forceinline__ Hdr64& hd64() { return *reinterpret_cast<Hdr64*>(smem64); }
__device__ __forceinline__ int lane64() { return threadIdx.x & 31; }

// the model's arrays: the staged copy or the global original
template <bool ST>
struct MV64 {
#define SG_MV(T, name)                                                                             \
    static __device__ __forceinline__ const T* name() {                                            \
        if constexpr (ST) return reinterpret_cast<const T*>(smem64 + hd64().L.s_##name);           \
        else return hd64().m.name;                                                                 \
    }
    SG_MV(int, type) SG_MV(int, atom_frame) SG_MV(int, fkind) SG_MV(int, fparent) SG_MV(int, fbegin) SG_MV(int, fend)
    SG_MV(int, fconf) SG_MV(int, fdof) SG_MV(int, level_start) SG_MV(int, level_frames) SG_MV(int, child_start)
    SG_MV(int, child_list) SG_MV(int, csr_start) SG_MV(int, heavy) SG_MV(int, lig_begin) SG_MV(int, lig_end)
    SG_MV(int, lig_root) SG_MV(int, lig_pair_end) SG_MV(int, blk_rigid) SG_MV(int, blk_conf) SG_MV(int, blk_ntors)
    SG_MV(int, tor_conf) SG_MV(int, tor_dof)
    SG_MV(double, charge) SG_MV(double, local) SG_MV(double, forigin) SG_MV(double, faxis)
#undef SG_MV
};

// every warp of the block (the leader's and the helpers' code meet here)
template <int G>
__device__ __forceinline__ void bar64() {
    if constexpr (G == 1) __syncwarp();
    else asm volatile("bar.sync 0;" ::: "memory");
}
// the warps that add forces: all but the last
template <int G>
__device__ __forceinline__ void bar_forces64() {
    static_assert(G == 1 || G == 4 || G == 8, "1, 4 or 8 warps");
    if constexpr (G == 1) __syncwarp();
    else if constexpr (G == 4) asm volatile("bar.sync 1, 96;" ::: "memory");
    else asm volatile("bar.sync 1, 224;" ::: "memory");
}

__device__ __forceinline__ V3<double> ld3(const double* p) { return {p[0], p[1], p[2]}; }
__device__ __forceinline__ void st3(double* p, V3<double> v) { p[0] = v.x; p[1] = v.y; p[2] = v.z; }

// ---- model::set ---------------------------------------------------------------------------
// frames, by the leader warp: (cos, sin) of every torsion's half angle at once
// (kept where the frame's quaternion goes), then level by level
template <bool ST>
__device__ __noinline__ void set_frames64(const double* conf) {
    using M = MV64<ST>;
    const Hdr64& H = hd64();
    const Ws64& L = H.L;
    double* S = smem64;
    const int lane = lane64(), F = H.m.nframes, nlevels = H.m.nlevels;
    const int *fkind = M::fkind(), *fconf = M::fconf(), *fparent = M::fparent(), *ls = M::level_start(),
              *lf = M::level_frames();
    const double *forigin = M::forigin(), *faxis = M::faxis();
#pragma unroll 1
    for (int t = lane; t < 2 * F; t += 32) {  // a lane each for the cosine and the sine
        const int f = t >> 1;
        if (fkind[f] != SG_FRAME_RIGID) {
            double angle = conf[fconf[f]];
            normalize_angle(angle);
            S[L.q + 4 * f + (t & 1)] = (t & 1) ? fd_sin(angle / 2) : fd_cos(angle / 2);
        }
    }
    __syncwarp();
#pragma unroll 1
    for (int lv = 0; lv < nlevels; lv++) {
#pragma unroll 1
        for (int idx = ls[lv] + lane; idx < ls[lv + 1]; idx += 32) {
            const int f = lf[idx];
            const int kind = fkind[f];
            double* qd = S + L.q + 4 * f;
            Quat<double> q;
            if (kind == SG_FRAME_RIGID) {
                const double* c = conf + fconf[f];
                st3(S + L.origin + 3 * f, V3<double>{c[0], c[1], c[2]});
                q = Quat<double>{c[3], c[4], c[5], c[6]};
            } else if (kind == SG_FRAME_SEGMENT) {
                const int p = fparent[f];
                const double* prot = S + L.rot + 9 * p;
                const V3<double> o = ld3(S + L.origin + 3 * p) + mat_mul(prot, ld3(forigin + 3 * f));
                const V3<double> ax = mat_mul(prot, ld3(faxis + 3 * f));
                st3(S + L.origin + 3 * f, o);
                st3(S + L.axis + 3 * f, ax);
                const double* pq = S + L.q + 4 * p;
                const double c = qd[0], s = qd[1];
                q = qmul(Quat<double>{c, s * ax.x, s * ax.y, s * ax.z}, Quat<double>{pq[0], pq[1], pq[2], pq[3]});
                q_normalize_approx(q);
            } else {
                const V3<double> ax = ld3(faxis + 3 * f);
                st3(S + L.origin + 3 * f, ld3(forigin + 3 * f));
                st3(S + L.axis + 3 * f, ax);
                const double c = qd[0], s = qd[1];
                q = Quat<double>{c, s * ax.x, s * ax.y, s * ax.z};
            }
            qd[0] = q.a; qd[1] = q.b; qd[2] = q.c; qd[3] = q.d;
            quat_to_mat(q, S + L.rot + 9 * f);
        }
        __syncwarp();
    }
}
// atoms t0, t0 + nt, ... from the frames
template <bool ST>
__device__ __forceinline__ void set_atoms64(int t0, int nt) {
    using M = MV64<ST>;
    const Hdr64& H = hd64();
    const Ws64& L = H.L;
    double* S = smem64;
    const int nmov = H.m.nmov;
    const int* atom_frame = M::atom_frame();
    const double* local = M::local();
#pragma unroll(ST ? 4 : 1)
    for (int i = t0; i < nmov; i += nt) {
        const int f = atom_frame[i];
        st3(S + L.coords + 3 * i, ld3(S + L.origin + 3 * f) + mat_mul(S + L.rot + 9 * f, ld3(local + 3 * i)));
    }
}
// model::set by the leader alone
template <bool ST>
__device__ __forceinline__ void set_conf64(const double* conf) {
    set_frames64<ST>(conf);
    set_atoms64<ST>(lane64(), 32);
    __syncwarp();
}

// ---- table lookups --------------------------------------------------------------------------
// precalculate_linear::eval_deriv (type-ordered lookup, charge-weighted
// components); pr: type pair index, sw: the first type is the larger one.
// Samples i and i + 1 lie side by side, 16-byte aligned.
__device__ __forceinline__ double comp_sum64(double c0, double c1, double c2, double c3, double qa, double qb) {
    return c0 + fabs(qa) * c1 + fabs(qb) * c2 + qa * qb * c3;
}
__device__ __forceinline__ void table_deriv64(const DTables& T, int pr, bool sw, double qa, double qb, double r2,
                                              double& e, double& dor) {
    const double rf = T.factor * r2;
    const size_t i1 = (size_t)rf;
    const double rem = rf - (double)i1;
    const double2* s = reinterpret_cast<const double2*>(T.smooth) + ((size_t)pr * T.n + i1) * T.nc;
    double e1, e2, d1, d2;
    if (T.nc == 1) {
        const double2 a = __ldg(s), b = __ldg(s + 1);
        e1 = a.x; d1 = a.y; e2 = b.x; d2 = b.y;
    } else {
        if (sw) { const double q = qa; qa = qb; qb = q; }
        const double2 a0 = __ldg(s), a1 = __ldg(s + 1), a2 = __ldg(s + 2), a3 = __ldg(s + 3);
        const double2 b0 = __ldg(s + 4), b1 = __ldg(s + 5), b2 = __ldg(s + 6), b3 = __ldg(s + 7);
        e1 = comp_sum64(a0.x, a1.x, a2.x, a3.x, qa, qb);
        e2 = comp_sum64(b0.x, b1.x, b2.x, b3.x, qa, qb);
        d1 = comp_sum64(a0.y, a1.y, a2.y, a3.y, qa, qb);
        d2 = comp_sum64(b0.y, b1.y, b2.y, b3.y, qa, qb);
    }
    e = e1 + rem * (e2 - e1);
    dor = d1 + rem * (d2 - d1);
}
// precalculate_linear::eval (precalculate.h:75-83,103-108,191-203): the fast
// table's components at sz(factor r2), weighted by a's and b's charges
// (result_components::eval, result_components.h:75-81); for t_a > t_b the
// (t_b, t_a) entry with its A and B components swapped (swapOrder).
__device__ __forceinline__ double table_fast64(const DTables& T, int pr, bool sw, double qa, double qb, double r2) {
    const double* c = T.fast + ((size_t)pr * T.n + (size_t)(T.factor * r2)) * T.nc;
    double ca = 0, cb = 0, cab = 0;
    if (T.nc > 1) { ca = sw ? c[2] : c[1]; cb = sw ? c[1] : c[2]; cab = c[3]; }
    return c[0] + fabs(qa) * ca + fabs(qb) * cb + qa * qb * cab;
}
__device__ __forceinline__ int type_pair64(int ta, int tb, bool& sw) {
    sw = ta > tb;
    return sw ? tri_index(tb, ta) : tri_index(ta, tb);
}

// ---- receptor terms -------------------------------------------------------------------------
// cache::eval_deriv: per movable atom grid energy and derivative
template <bool ST>
__device__ __forceinline__ void grid_atoms64(int t0, int nt, double v, double slope) {
    using M = MV64<ST>;
    const Hdr64& H = hd64();
    const Ws64& L = H.L;
    const DReceptor& R = *H.R;
    double* S = smem64;
    const int* type = M::type();
    const double* charge = M::charge();
    const int nmov = H.m.nmov;
#pragma unroll 1
    for (int i = t0; i < nmov; i += nt) {
        const int t = type[i];
        double* mf = S + L.mf + 3 * i;
        if (t >= kNumTypes || is_h(t)) {
            mf[0] = mf[1] = mf[2] = 0;
            S[L.eatom + i] = 0;
            continue;
        }
        const V3<double> loc = ld3(S + L.coords + 3 * i);
        V3<double> d;
        double ret = grid_aux64(R.g, R.map[t], loc, slope, v, d);
        const double q = charge[i];
        if (q != 0 && R.cmap[t]) {
            V3<double> cd{0, 0, 0};
            ret += q * grid_aux64(R.g, R.cmap[t], loc, slope, v, cd);
            add_to(d, q * cd);
        }
        S[L.eatom + i] = ret;
        st3(mf, d);
    }
}

// where an atom's direct sum is taken: the atom clamped to the box, the
// out-of-box distance and direction, and the 3 A cell's list [kb, ke)
struct Clamped64 {
    double a[3], adj[3], oobd[3], oob;
    int kb, ke;
    bool inside;
};
__device__ __forceinline__ Clamped64 clamp64(const DReceptor& R, const double* box, const double* x, bool act) {
    const DGeom& G = R.g;
    Clamped64 c;
    c.oob = 0;
    int ci[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
        c.a[j] = c.adj[j] = x[j];
        c.oobd[j] = 0;
        const double lo = box ? box[j] : G.gd_begin[j], hi = box ? box[3 + j] : G.gd_end[j];
        if (box || G.gd_n[j] > 0) {
            if (c.a[j] < lo) { c.adj[j] = lo; c.oobd[j] = -1; c.oob += fabs(c.a[j] - lo); }
            else if (c.a[j] > hi) { c.adj[j] = hi; c.oobd[j] = 1; c.oob += fabs(c.a[j] - hi); }
        }
        ci[j] = (int)floor(c.adj[j] / 3.0) - G.cell_off[j];
    }
    c.inside = ci[0] >= 0 && ci[1] >= 0 && ci[2] >= 0 && ci[0] < G.cell_dim[0] && ci[1] < G.cell_dim[1] &&
               ci[2] < G.cell_dim[2];
    c.kb = c.ke = 0;
    if (act && c.inside) {
        const int cell = ci[0] + G.cell_dim[0] * (ci[1] + G.cell_dim[1] * ci[2]);
        c.kb = R.full_start[cell];
        c.ke = R.full_start[cell + 1];
    }
    return c;
}

// a list entry's lookup under way: its separation and, where one table value is
// one load, the values
template <int NC>
struct Term64 {
    bool in;
    V3<double> r;
    double rem, r2;
    double2 a, b;
    int type;
};
// atom `at` of type t against list entry x (there: the lane has one)
template <int NC, bool ENERGY_ONLY>
__device__ __forceinline__ Term64<NC> look_up64(const DTables& T, bool there, CellAtom x, V3<double> at, int t) {
    Term64<NC> q{false, {0, 0, 0}, 0, 0, {0, 0}, {0, 0}, 0};
    if (there) {
        q.r = V3<double>{at.x - x.x, at.y - x.y, at.z - x.z};
        q.r2 = norm2(q.r);
        q.type = x.type;
        q.in = q.r2 < T.cutoff_sqr;
        if (NC == 1 && q.in) {
            bool sw;
            const size_t row = (size_t)type_pair64(t, q.type, sw) * T.n;
            const double rf = T.factor * q.r2;
            const size_t i1 = (size_t)rf;
            q.rem = rf - (double)i1;
            if (ENERGY_ONLY) {
                q.a.x = __ldg(T.fast + row + i1);
            } else {
                const double2* s = reinterpret_cast<const double2*>(T.smooth) + row + i1;
                q.a = __ldg(s);
                q.b = __ldg(s + 1);
            }
        }
    }
    return q;
}
// The group's terms within the cutoff, squeezed into its exchange buffer X and
// added to its lanes' sums in list order.  charge: of this lane's entry.
template <int NC, bool ENERGY_ONLY>
__device__ __forceinline__ double add_up64(const DTables& T, Term64<NC> q, int t, double qi, const double* charge,
                                           double* X, int* err, double acc) {
    const int lane = lane64(), gl = lane & 7;
    const unsigned gm = (__ballot_sync(kFull, q.in) >> (lane & 24)) & 0xffu;
    const int cnt = __popc(gm);
    if (q.in) {
        double* x = X + 4 * __popc(gm & ((1u << gl) - 1));
        double pe, dor = 0;
        if (!ENERGY_ONLY && q.r2 < kEps) atomicExch(err, kDevOverlap);
        if (NC == 1) {
            pe = q.a.x;
            if (!ENERGY_ONLY) {
                pe = q.a.x + q.rem * (q.b.x - q.a.x);
                dor = q.a.y + q.rem * (q.b.y - q.a.y);
            }
        } else {
            bool sw;
            const int pr = type_pair64(t, q.type, sw);
            if (ENERGY_ONLY) pe = table_fast64(T, pr, sw, qi, *charge, q.r2);
            else table_deriv64(T, pr, sw, qi, *charge, q.r2, pe, dor);
        }
        if (ENERGY_ONLY) {
            x[0] = pe;
        } else {
            const V3<double> f = dor * q.r;
            reinterpret_cast<double2*>(x)[0] = make_double2(pe, f.x);
            reinterpret_cast<double2*>(x)[1] = make_double2(f.y, f.z);
        }
    }
    __syncwarp();
    if (gl < (ENERGY_ONLY ? 1 : 4))
        for (int j = 0; j < cnt; j++) acc += X[4 * j + gl];
    __syncwarp();
    return acc;
}

// non_cache::eval_deriv (ENERGY_ONLY: non_cache::eval on the fast table, into
// eatom only): direct sum over the 3 A cell list of the clamped atom, 8 lanes
// per atom and 16 list entries a round; a round's table values are on their way
// while the round before is added up
template <int G, bool ST, bool ENERGY_ONLY, int NC>
__device__ __forceinline__ void direct_atoms64(int k, double v, double slope) {
    using M = MV64<ST>;
    const Hdr64& H = hd64();
    const Ws64& L = H.L;
    const DReceptor& R = *H.R;
    const DTables& T = H.T;
    double* S = smem64;
    const int lane = lane64(), gl = lane & 7, grp = lane >> 3;
    double* X = S + L.xbuf + k * kXbuf64 + grp * (kXbuf64 / 4);
    const int* type = M::type();
    const int* heavy = M::heavy();
    const double* charge = M::charge();
    const int nmov = H.m.nmov, nheavy = H.m.nheavy;
    const CellAtom* list = R.full_list;
    for (int i = 32 * k + lane; i < nmov; i += 32 * G)
        if (type[i] >= kNumTypes || is_h(type[i])) {
            if (!ENERGY_ONLY) st3(S + L.mf + 3 * i, V3<double>{0, 0, 0});
            S[L.eatom + i] = 0;
        }
    for (int a0 = 4 * k; a0 < nheavy; a0 += 4 * G) {
        const bool there = a0 + grp < nheavy;
        const int i = there ? heavy[a0 + grp] : 0;
        const int t = type[i];
        const bool act = there && t < kNumTypes;
        const Clamped64 c = clamp64(R, ENERGY_ONLY ? nullptr : H.box, S + L.coords + 3 * i, act);
        const double qi = charge[i];
        double acc = 0;  // lane gl < 4 of a group: energy, x, y, z
        CellAtom n0{0, 0, 0, 0, 0}, n1 = n0;
        Term64<NC> q0, q1;
        int kk = c.kb + gl;
        const V3<double> at{c.adj[0], c.adj[1], c.adj[2]};
        const int ke = c.ke;
        const double* list_charge = R.full_charge;
        if (kk < ke) n0 = load_cell_atom(list + kk);
        if (kk + 8 < ke) n1 = load_cell_atom(list + kk + 8);
        q0 = look_up64<NC, ENERGY_ONLY>(T, kk < ke, n0, at, t);
        q1 = look_up64<NC, ENERGY_ONLY>(T, kk + 8 < ke, n1, at, t);
        if (kk + 16 < ke) n0 = load_cell_atom(list + kk + 16);
        if (kk + 24 < ke) n1 = load_cell_atom(list + kk + 24);
        for (; __any_sync(kFull, kk - gl < ke); kk += 16) {
            acc = add_up64<NC, ENERGY_ONLY>(T, q0, t, qi, list_charge + kk, X, H.err, acc);
            q0 = look_up64<NC, ENERGY_ONLY>(T, kk + 16 < ke, n0, at, t);
            if (kk + 32 < ke) n0 = load_cell_atom(list + kk + 32);
            acc = add_up64<NC, ENERGY_ONLY>(T, q1, t, qi, list_charge + kk + 8, X, H.err, acc);
            q1 = look_up64<NC, ENERGY_ONLY>(T, kk + 24 < ke, n1, at, t);
            if (kk + 40 < ke) n1 = load_cell_atom(list + kk + 40);
        }
        double this_e = __shfl_sync(kFull, acc, 8 * grp);
        V3<double> deriv{__shfl_sync(kFull, acc, 8 * grp + 1), __shfl_sync(kFull, acc, 8 * grp + 2),
                         __shfl_sync(kFull, acc, 8 * grp + 3)};
        if (act && gl == 0) {
            if (!c.inside) atomicExch(H.err, kDevBadModel);
            if (ENERGY_ONLY) {
                curl_e(this_e, v);
                S[L.eatom + i] = this_e + c.oob * slope;
            } else {
                if (R.ugrid) {  // the user grid at the atom's own coordinates (non_cache.cpp:180-184)
                    V3<double> ugd;
                    this_e += grid_aux64(R.ug, R.ugrid, V3<double>{c.a[0], c.a[1], c.a[2]}, slope, 1000.0, ugd);
                    add_to(deriv, ugd);
                }
                curl_ed(this_e, deriv, v);
                double* mf = S + L.mf + 3 * i;
                mf[0] = deriv.x + c.oobd[0] * slope;
                mf[1] = deriv.y + c.oobd[1] * slope;
                mf[2] = deriv.z + c.oobd[2] * slope;
                S[L.eatom + i] = this_e + c.oob * slope;
            }
        }
    }
}

// ---- pairs ------------------------------------------------------------------------------------
// intramolecular / other pairs t0, t0 + nt, ...: energy and force per pair
// (ENERGY_ONLY: model::eval_interacting_pairs, model.cpp:885-902, on the fast
// table); +0 beyond the cutoff
template <bool ST, bool ENERGY_ONLY>
__device__ __forceinline__ void pairs64(int t0, int nt, double v_other, double v_lig) {
    using M = MV64<ST>;
    const Hdr64& H = hd64();
    const Ws64& L = H.L;
    const DTables& T = H.T;
    double* S = smem64;
    const int np = H.m.npairs;
    const int2* pairs = reinterpret_cast<const int2*>(H.m.pairs);
    const int *tp = H.m.pair_tp, *group = H.m.pair_group;
    const double* charge = M::charge();
    for (int p = t0; p < np; p += nt) {
        const int2 ab = __ldg(pairs + p);
        const V3<double> r = ld3(S + L.coords + 3 * ab.y) - ld3(S + L.coords + 3 * ab.x);
        const double r2 = norm2(r);
        double pe = 0;
        V3<double> force{0, 0, 0};
        if (r2 < T.cutoff_sqr) {
            const int w = __ldg(tp + p);
            const double v = __ldg(group + p) == 0 ? v_other : v_lig;
            const double qa = T.nc > 1 ? charge[ab.x] : 0.0, qb = T.nc > 1 ? charge[ab.y] : 0.0;
            const bool sw = (w >> 30) & 1;
            if (ENERGY_ONLY) {
                pe = table_fast64(T, w & 0x3fffffff, sw, qa, qb, r2);
                curl_e(pe, v);
            } else {
                double dor;
                table_deriv64(T, w & 0x3fffffff, sw, qa, qb, r2, pe, dor);
                force = dor * r;
                curl_ed(pe, force, v);
            }
        }
        S[L.pe + p] = pe;
        if (!ENERGY_ONLY) st3(S + L.pf + 3 * p, force);
    }
}

// minus_forces: grid derivative, then every pair contribution in pair order;
// one (atom, axis) per thread
template <bool ST>
__device__ __forceinline__ void gather_forces64(int t0, int nt) {
    using M = MV64<ST>;
    const Hdr64& H = hd64();
    const Ws64& L = H.L;
    double* S = smem64;
    const int* csr_start = M::csr_start();
    const int* csr = H.m.csr;
    const uint16_t* csr16 = reinterpret_cast<const uint16_t*>(smem64 + L.s_csr);
    const bool staged = ST && L.s_csr != 0;
    auto entry = [&](int q) { return staged ? (int)csr16[q] : __ldg(csr + q); };
    const int n3 = 3 * H.m.nmov;
    for (int t = t0; t < n3; t += nt) {
        const int i = t / 3, c = t - 3 * i;
        const double* pf = S + L.pf + c;
        double f = S[L.mf + t];
        int q = csr_start[i];
        const int e = csr_start[i + 1];
        for (; q + 4 <= e; q += 4) {
            int w[4];
            double x[4];
#pragma unroll
            for (int u = 0; u < 4; u++) w[u] = entry(q + u);
#pragma unroll
            for (int u = 0; u < 4; u++) x[u] = pf[3 * (w[u] >> 1)];
#pragma unroll
            for (int u = 0; u < 4; u++) f += (w[u] & 1) ? x[u] : -x[u];
        }
#pragma unroll(ST ? 3 : 1)
        for (; q < e; q++) {
            const int w = entry(q);
            const double x = pf[3 * (w >> 1)];
            f += (w & 1) ? x : -x;
        }
        S[L.mf + t] = f;
    }
}

// total energy in the reference's order: grid atoms, other pairs, each ligand.
// One lane per sum; one warp.
template <bool ST>
__device__ __forceinline__ double energy64() {
    using M = MV64<ST>;
    const Hdr64& H = hd64();
    const Ws64& L = H.L;
    const double* S = smem64;
    const int lane = lane64(), nlig = H.m.nlig;
    const int* lig_pair_end = M::lig_pair_end();
    int b = 0, e = 0;
    const double* src = S + L.pe;
    if (lane == 0) {
        src = S + L.eatom;
        e = H.m.nmov;
    } else if (lane == 1) {
        e = H.m.nother;
    } else if (lane - 2 < nlig) {
        b = lane == 2 ? H.m.nother : lig_pair_end[lane - 3];
        e = lig_pair_end[lane - 2];
    }
    double part = 0;
    for (; b + 8 <= e; b += 8) {
        double x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) x[u] = src[b + u];
#pragma unroll
        for (int u = 0; u < 8; u++) part += x[u];
    }
#pragma unroll(ST ? 7 : 1)
    for (; b < e; b++) part += src[b];
    __syncwarp();
    double tot = __shfl_sync(kFull, part, 0);
    tot += __shfl_sync(kFull, part, 1);
#pragma unroll 1
    for (int l = 0; l < nlig && l < 30; l++) tot += __shfl_sync(kFull, part, 2 + l);
    return tot;
}

// model::eval_intramolecular (model.cpp:1027-1079) after the pairs' energies on
// the same coords: each ligand's pairs, then every flexible movable atom
// against every receptor atom (curled per pair), then flex-flex other pairs.
// One running sum in the reference's order; the flex-rigid energies of 32
// receptor atoms are computed at once and those within the cutoff added in
// atom order.
template <bool ST>
__device__ double intramolecular64(const double v[3]) {
    using M = MV64<ST>;
    const Hdr64& H = hd64();
    const Ws64& L = H.L;
    const DReceptor& R = *H.R;
    const DTables& T = H.T;
    const double* S = smem64;
    const int lane = lane64(), nlig = H.m.nlig, nmov = H.m.nmov, nother = H.m.nother;
    const int *lig_begin = M::lig_begin(), *lig_end = M::lig_end(), *lig_pair_end = M::lig_pair_end(), *type = M::type();
    const double* charge = M::charge();
    auto in_ligand = [&](int i) {
        for (int l = 0; l < nlig; l++)
            if (i >= lig_begin[l] && i < lig_end[l]) return true;
        return false;
    };
    double e = 0;
    for (int l = 0, b = nother; l < nlig; l++) {  // every lane adds the same sums
        double el = 0;
        for (int k = b; k < lig_pair_end[l]; k++) el += S[L.pe + k];
        e += el;
        b = lig_pair_end[l];
    }
    for (int i = 0; i < nmov; i++) {  // warp-uniform
        if (in_ligand(i) || type[i] >= kNumTypes) continue;
        const V3<double> a = ld3(S + L.coords + 3 * i);
        for (int j0 = 0; j0 < R.natoms; j0 += 32) {
            const int j = j0 + lane;
            double this_e = 0;
            bool add = false;
            if (j < R.natoms && R.type[j] < kNumTypes) {
                const double r2 = norm2(a - V3<double>{R.xyz[3 * j], R.xyz[3 * j + 1], R.xyz[3 * j + 2]});
                if (r2 < T.cutoff_sqr) {
                    bool sw;
                    const int pr = type_pair64(type[i], R.type[j], sw);
                    this_e = table_fast64(T, pr, sw, charge[i], R.charge[j], r2);
                    curl_e(this_e, v[1]);
                    add = true;
                }
            }
            for (unsigned mask = __ballot_sync(kFull, add); mask; mask &= mask - 1)
                e += __shfl_sync(kFull, this_e, __ffs(mask) - 1);
        }
    }
    for (int k = 0; k < nother; k++) {
        const int a = H.m.pairs[2 * k], b = H.m.pairs[2 * k + 1];
        if (!in_ligand(a) && !in_ligand(b)) e += S[L.pe + k];
    }
    return e;
}

// ---- tree derivative, by the leader warp ------------------------------------------------------
// per-frame sums in atom order, children bottom-up, then the change vector
template <bool ST>
__device__ __forceinline__ void derivative64(double* g) {
    using M = MV64<ST>;
    const Hdr64& H = hd64();
    const Ws64& L = H.L;
    double* S = smem64;
    const int lane = lane64(), F = H.m.nframes, nlevels = H.m.nlevels;
    const int *fbegin = M::fbegin(), *fend = M::fend(), *child_start = M::child_start(), *child_list = M::child_list(),
              *ls = M::level_start(), *lf = M::level_frames(), *fkind = M::fkind(), *fdof = M::fdof();
    if constexpr (ST) {
        // torque terms of all atoms at once, then one sum per (frame, component)
        const int* atom_frame = M::atom_frame();
        const int nmov = H.m.nmov;
        for (int i = lane; i < nmov; i += 32) {
            const int f = atom_frame[i];
            st3(S + L.cr + 3 * i, cross(ld3(S + L.coords + 3 * i) - ld3(S + L.origin + 3 * f), ld3(S + L.mf + 3 * i)));
        }
        __syncwarp();
        for (int t = lane; t < 6 * F; t += 32) {
            const int f = t / 6, c = t - 6 * f;
            const double* src = S + (c < 3 ? L.mf + c : L.cr + c - 3);
            const int e = fend[f];
            int i = fbegin[f];
            double s = 0;
            for (; i + 4 <= e; i += 4) {
                double x[4];
#pragma unroll
                for (int u = 0; u < 4; u++) x[u] = src[3 * (i + u)];
#pragma unroll
                for (int u = 0; u < 4; u++) s += x[u];
            }
            for (; i < e; i++) s += src[3 * i];
            S[(c < 3 ? L.fF + c : L.fT + c - 3) + 3 * f] = s;
        }
    } else {
#pragma unroll 1
        for (int f = lane; f < F; f += 32) {
            V3<double> Fs{0, 0, 0}, Ts{0, 0, 0};
            const V3<double> o = ld3(S + L.origin + 3 * f);
#pragma unroll 1
            for (int i = fbegin[f]; i < fend[f]; i++) {
                const V3<double> fi = ld3(S + L.mf + 3 * i);
                add_to(Fs, fi);
                add_to(Ts, cross(ld3(S + L.coords + 3 * i) - o, fi));
            }
            st3(S + L.fF + 3 * f, Fs);
            st3(S + L.fT + 3 * f, Ts);
        }
    }
    __syncwarp();
#pragma unroll 1
    for (int lv = nlevels - 2; lv >= 0; lv--) {
#pragma unroll 1
        for (int idx = ls[lv] + lane; idx < ls[lv + 1]; idx += 32) {
            const int f = lf[idx];
            const int cb = child_start[f], ce = child_start[f + 1];
            if (cb == ce) continue;
            V3<double> Fs = ld3(S + L.fF + 3 * f), Ts = ld3(S + L.fT + 3 * f);
            const V3<double> o = ld3(S + L.origin + 3 * f);
#pragma unroll(ST ? 4 : 1)
            for (int c = cb; c < ce; c++) {
                const int ch = child_list[c];
                const V3<double> cF = ld3(S + L.fF + 3 * ch);
                add_to(Fs, cF);
                const V3<double> r = ld3(S + L.origin + 3 * ch) - o;
                add_to(Ts, cross(r, cF) + ld3(S + L.fT + 3 * ch));
            }
            st3(S + L.fF + 3 * f, Fs);
            st3(S + L.fT + 3 * f, Ts);
        }
        __syncwarp();
    }
#pragma unroll 1
    for (int f = lane; f < F; f += 32) {
        const V3<double> Fs = ld3(S + L.fF + 3 * f), Ts = ld3(S + L.fT + 3 * f);
        double* d = g + fdof[f];
        if (fkind[f] == SG_FRAME_RIGID) {
            d[0] = Fs.x; d[1] = Fs.y; d[2] = Fs.z; d[3] = Ts.x; d[4] = Ts.y; d[5] = Ts.z;
        } else {
            d[0] = dot(Ts, ld3(S + L.axis + 3 * f));
        }
    }
    __syncwarp();
}

// ---- the block's evaluation ---------------------------------------------------------------------
enum : int { kOpEval = 1, kOpScore = 2, kOpExit = 3 };

// warp k's part of model::eval_deriv after the leader has set the frames;
// `direct` (in the header) selects non_cache instead of the grid maps.  Ends
// with a block barrier, after which the energy and the gradient are in place.
template <int G, bool ST>
__device__ __noinline__ void eval_warp64(int k) {
    Hdr64& H = hd64();
    set_atoms64<ST>(threadIdx.x, 32 * G);
    bar64<G>();
    if (H.direct) {
        if (H.T.nc == 1) direct_atoms64<G, ST, false, 1>(k, H.v[1], H.slope);
        else direct_atoms64<G, ST, false, 4>(k, H.v[1], H.slope);
        pairs64<ST, false>(threadIdx.x, 32 * G, H.v[2], H.v[0]);
    } else {
        // the first warps take the atoms; the pairs start on the others
        const int na = min(G, (H.m.nmov + 31) / 32);
        if (k < na) grid_atoms64<ST>(32 * k + lane64(), 32 * na, H.v[1], H.slope);
        const int kp = (k - na + G) % G;
        pairs64<ST, false>(32 * kp + lane64(), 32 * G, H.v[2], H.v[0]);
    }
    bar64<G>();
    if (G == 1 || k == G - 1) {
        const double e = energy64<ST>();
        if (lane64() == 0) H.e = e;
    }
    if (G == 1 || k < G - 1) {
        gather_forces64<ST>(threadIdx.x, G == 1 ? 32 : 32 * (G - 1));
        bar_forces64<G>();
    }
    if (k == 0) derivative64<ST>(smem64 + H.g_at);
    bar64<G>();
}

// warp k's part of the rescoring energies (eatom and pe)
template <int G, bool ST>
__device__ __noinline__ void score_warp64(int k) {
    Hdr64& H = hd64();
    set_atoms64<ST>(threadIdx.x, 32 * G);
    bar64<G>();
    if (H.T.nc == 1) direct_atoms64<G, ST, true, 1>(k, H.v[1], H.slope);
    else direct_atoms64<G, ST, true, 4>(k, H.v[1], H.slope);
    pairs64<ST, true>(threadIdx.x, 32 * G, H.v[2], H.v[0]);
    bar64<G>();
}

// a helper warp: its part of every evaluation until the leader's exit
template <int G, bool ST>
__device__ __forceinline__ void help64(int k) {
    for (;;) {
        bar64<G>();  // the leader's command and frames are in
        const int op = hd64().op;
        if (op == kOpEval) eval_warp64<G, ST>(k);
        else if (op == kOpScore) score_warp64<G, ST>(k);
        else break;
    }
}

// the leader's side: hands out op and, for an evaluation, does its own part
template <int G>
__device__ __forceinline__ void command64(int op, const double v[3], double slope, int direct, int g_at) {
    Hdr64& H = hd64();
    if (lane64() == 0) {
        H.op = op;
        H.v[0] = v[0]; H.v[1] = v[1]; H.v[2] = v[2];
        H.slope = slope;
        H.direct = direct;
        H.g_at = g_at;
        H.evals += op == kOpEval;
    }
    bar64<G>();
}
template <int G>
__device__ __forceinline__ void release64() {
    if constexpr (G > 1) {
        if (lane64() == 0) hd64().op = kOpExit;
        bar64<G>();
    }
}

// model::eval_deriv of the conf in the workspace, called by the leader
template <int G, bool ST>
__device__ __forceinline__ double eval_deriv64(const double* conf, const double v[3], double slope, bool direct,
                                               double* g) {
    set_frames64<ST>(conf);
    command64<G>(kOpEval, v, slope, direct, (int)(g - smem64));
    eval_warp64<G, ST>(0);
    return hd64().e;
}

}  // namespace sg
