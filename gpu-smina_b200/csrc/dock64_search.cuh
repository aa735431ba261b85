// Plain (FP64) path, part 2: BFGS with its line searches, mutation,
// Metropolis acceptance and the output container, run by an item's leader warp.
// Control flow is warp-uniform.  Scalars that need an order-sensitive reduction
// are added in the reference's order on every lane at once, from terms that the
// lanes computed side by side (a shuffle per term; no lane waits for another's
// loop and nothing is broadcast back).
// Reference: bfgs.h:30-282; conf.h:98-404; mutate.cpp:35-63;
// monte_carlo.cpp:44-48,95-130; coords.cpp:25-58; random.cpp:28-80;
// quaternion.cpp:42-139.
#pragma once
#include "dock64_eval.cuh"

namespace sg {

// ---- mt19937 on lane 0, Boost's uniform_real / uniform_int ------------------------
__device__ __forceinline__ uint32_t* mt64() { return reinterpret_cast<uint32_t*>(smem64 + hd64().L.mt); }
__device__ __noinline__ uint32_t mt_next(uint32_t* st) {
    int i = (int)st[624];
    if (i >= 624) {
        for (int k = 0; k < 624; k++) {
            const uint32_t y = (st[k] & 0x80000000u) | (st[k + 1 < 624 ? k + 1 : 0] & 0x7fffffffu);
            st[k] = st[k + 397 < 624 ? k + 397 : k + 397 - 624] ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
        }
        i = 0;
    }
    uint32_t z = st[i];
    st[624] = (uint32_t)(i + 1);
    z ^= z >> 11;
    z ^= (z << 7) & 0x9d2c5680u;
    z ^= (z << 15) & 0xefc60000u;
    z ^= z >> 18;
    return z;
}
__device__ double rand_fl(double a, double b) {
    double r = 0;
    if (lane64() == 0) {
        for (;;) {
            r = (double)mt_next(mt64()) / (4294967295.0 + 1) * (b - a) + a;
            if (r < b) break;
        }
    }
    return __shfl_sync(kFull, r, 0);
}
__device__ int rand_int(int a, int b) {
    int out = a;
    if (lane64() == 0) {
        const uint32_t range = (uint32_t)b - (uint32_t)a;
        if (range != 0) {
            uint32_t bucket = 0xffffffffu / (range + 1);
            if (0xffffffffu % (range + 1) == range) ++bucket;
            for (;;) {
                const uint32_t r = mt_next(mt64()) / bucket;
                if (r <= range) { out = (int)(r + (uint32_t)a); break; }
            }
        }
    }
    return __shfl_sync(kFull, out, 0);
}
__device__ V3<double> rand_in_sphere() {
    for (;;) {
        const double r1 = rand_fl(-1, 1), r2 = rand_fl(-1, 1), r3 = rand_fl(-1, 1);
        const V3<double> t{r1, r2, r3};
        if (norm2(t) < 1) return t;
    }
}

// ---- ordered scalar products ----------------------------------------------------------
// sum over lanes 0 .. cnt - 1 of t, in lane order, onto s (same on every lane)
template <bool ST>
__device__ __forceinline__ double add_in_order64(double s, double t, int cnt) {
    int j = 0;
    for (; ST && j + 4 <= cnt; j += 4) {
        double x[4];
#pragma unroll
        for (int u = 0; u < 4; u++) x[u] = __shfl_sync(kFull, t, j + u);
#pragma unroll
        for (int u = 0; u < 4; u++) s += x[u];
    }
#pragma unroll 1
    for (; j < cnt; j++) s += __shfl_sync(kFull, t, j);
    return s;
}
template <bool ST>
__device__ __forceinline__ double sprod64(const double* a, const double* b, int n) {
    double s = 0;
#pragma unroll 1
    for (int i0 = 0; i0 < n; i0 += 32) {
        const int i = i0 + lane64();
        s = add_in_order64<ST>(s, i < n ? a[i] * b[i] : 0.0, min(32, n - i0));
    }
    return s;
}
__device__ __forceinline__ void vcopy(double* d, const double* s, int n) {
#pragma unroll 1
    for (int i = lane64(); i < n; i += 32) d[i] = s[i];
    __syncwarp();
}

// conf::increment (torsions normalized, orientation not re-normalized beyond approx)
template <bool ST>
__device__ __noinline__ void conf_increment64(double* x, const double* p, double alpha) {
    using M = MV64<ST>;
    const Hdr64& H = hd64();
    const int *lig_root = M::lig_root(), *fconf = M::fconf(), *fdof = M::fdof(), *tor_conf = M::tor_conf(),
              *tor_dof = M::tor_dof();
    const int nlig = H.m.nlig, ntors = H.m.ntors;
    // the last lanes take the ligands' rigid parts, so that a torsion lane never does both
#pragma unroll 1
    for (int l = 31 - lane64(); l < nlig; l += 32) {
        const int f = lig_root[l];
        double* c = x + fconf[f];
        const double* d = p + fdof[f];
        const V3<double> dp = alpha * V3<double>{d[0], d[1], d[2]};
        c[0] += dp.x; c[1] += dp.y; c[2] += dp.z;
        Quat<double> q{c[3], c[4], c[5], c[6]};
        q_increment(q, alpha * V3<double>{d[3], d[4], d[5]});
        c[3] = q.a; c[4] = q.b; c[5] = q.c; c[6] = q.d;
    }
#pragma unroll 1
    for (int k = lane64(); k < ntors; k += 32) {
        double& t = x[tor_conf[k]];
        t += normalized_angle(alpha * p[tor_dof[k]]);
        normalize_angle(t);
    }
    __syncwarp();
}

// conf::operator()(index): the value of change coordinate i
template <bool ST>
__device__ double conf_value64(const double* x, int i) {
    using M = MV64<ST>;
    const Hdr64& H = hd64();
    const int *lig_root = M::lig_root(), *fconf = M::fconf(), *fdof = M::fdof(), *tor_conf = M::tor_conf(),
              *tor_dof = M::tor_dof();
    for (int l = 0; l < H.m.nlig; l++) {
        const int f = lig_root[l];
        const int d0 = fdof[f];
        if (i >= d0 && i < d0 + 3) return x[fconf[f] + (i - d0)];
        if (i >= d0 + 3 && i < d0 + 6) {
            const double* c = x + fconf[f];
            const V3<double> a = q_to_angle(Quat<double>{c[3], c[4], c[5], c[6]});
            const int j = i - d0 - 3;
            return j == 0 ? a.x : j == 1 ? a.y : a.z;
        }
    }
    for (int k = 0; k < H.m.ntors; k++)
        if (tor_dof[k] == i) return x[tor_conf[k]];
    return 0;
}

struct EvalMode {
    double v[3];
    double slope;
    bool direct;
};

template <int G, bool ST>
__device__ __noinline__ double feval(const double* x, double* g, const EvalMode em) {
    return eval_deriv64<G, ST>(x, em.v, em.slope, em.direct, g);
}

// ---- line searches ----------------------------------------------------------------------
template <int G, bool ST>
__device__ __forceinline__ double fast_line_search64(const double* x, const double* g, double f0, const double* p,
                                                     double* x_new, double* g_new, double& f1, const EvalMode& em) {
    const int n = hd64().m.dof, cs = hd64().m.conf_size;
    double alpha = 1;
    const double pg = sprod64<ST>(p, g, n);
    for (unsigned trial = 0; trial < 10; trial++) {
        vcopy(x_new, x, cs);
        conf_increment64<ST>(x_new, p, alpha);
        f1 = feval<G, ST>(x_new, g_new, em);
        if (f1 - f0 < 0.0001 * alpha * pg) break;
        alpha *= 0.5;
    }
    return alpha;
}

template <int G, bool ST>
__device__ __noinline__ double accurate_line_search64(const double* x, const double* g, double f0, const double* p,
                                                      double* x_new, double* g_new, double& f1, const EvalMode& em) {
    const int n = hd64().m.dof, cs = hd64().m.conf_size;
    double a, alpha, alpha2 = 0, alamin, b, disc, f2 = 0, rhs1, rhs2, tmplam = 0;
    const double ALF = 1.0e-4, FIRST = 1.0;
    const double slope = sprod64<ST>(g, p, n);
    if (slope >= 0) {
        vcopy(x_new, x, cs);
        for (int i = lane64(); i < n; i += 32) g_new[i] = 0;
        __syncwarp();
        return 0;
    }
    double test = 0;
    for (int i = lane64(); i < n; i += 32) {
        const double temp = fabs(p[i]) / fmax(fabs(conf_value64<ST>(x, i)), 1.0);
        if (temp > test) test = temp;
    }
    for (int o = 16; o > 0; o >>= 1) test = fmax(test, __shfl_xor_sync(kFull, test, o));
    alamin = kEps / test;
    alpha = FIRST;
    for (;;) {
        vcopy(x_new, x, cs);
        conf_increment64<ST>(x_new, p, alpha);
        f1 = feval<G, ST>(x_new, g_new, em);
        if (alpha < alamin) {
            vcopy(x_new, x, cs);
            for (int i = lane64(); i < n; i += 32) g_new[i] = 0;
            __syncwarp();
            return 0;
        } else if (f1 <= f0 + ALF * alpha * slope) {
            return alpha;
        } else {
            if (alpha == FIRST) {
                tmplam = -slope / (2.0 * (f1 - f0 - slope));
            } else {
                rhs1 = f1 - f0 - alpha * slope;
                rhs2 = f2 - f0 - alpha2 * slope;
                a = (rhs1 / (alpha * alpha) - rhs2 / (alpha2 * alpha2)) / (alpha - alpha2);
                b = (-alpha2 * rhs1 / (alpha * alpha) + alpha * rhs2 / (alpha2 * alpha2)) / (alpha - alpha2);
                if (a == 0.0) tmplam = -slope / (2.0 * b);
                else {
                    disc = b * b - 3.0 * a * slope;
                    if (disc < 0) tmplam = 0.5 * alpha;
                    else if (b <= 0) tmplam = (-b + sqrt(disc)) / (3.0 * a);
                    else tmplam = -slope / (b + sqrt(disc));
                }
                if (tmplam > .5 * alpha) tmplam = .5 * alpha;
            }
        }
        alpha2 = alpha;
        f2 = f1;
        alpha = fmax(tmplam, 0.1 * alpha);
    }
}

// ---- BFGS on the triangular inverse Hessian -------------------------------------------
// Lane i sums row i: entries (j, i) of column i up to the diagonal, then along
// the row (one more than the column's length further each time).
template <bool ST>
__device__ __forceinline__ void minus_mat_vec64(const double* h, const double* in, double* out, int n) {
#pragma unroll 1
    for (int i = lane64(); i < n; i += 32) {
        double sum = 0;
        int at = i * (i + 1) / 2;
#pragma unroll(ST ? 4 : 1)
        for (int j = 0; j < n; j++) {
            sum += h[at] * in[j];
            at += j < i ? 1 : j + 1;
        }
        out[i] = -sum;
    }
    __syncwarp();
}

template <bool ST>
__device__ __forceinline__ void bfgs_update64(double* h, const double* p, const double* y, double yp, double alpha,
                                              int n) {
    if (alpha * yp < kEps) return;
    double* mhy = smem64 + hd64().L.mhy;
    minus_mat_vec64<ST>(h, y, mhy, n);
    const double yhy = -sprod64<ST>(y, mhy, n);
    const double r = 1 / (alpha * yp);
    const double c1 = alpha * r, c2 = +alpha * alpha * (r * r * yhy + r);
    if (n <= 32) {  // lane i owns p[i] and mhy[i]
        const int i = lane64();
        const double pi = i < n ? p[i] : 0.0, mi = i < n ? mhy[i] : 0.0, c2p = c2 * pi;
#pragma unroll(ST ? 2 : 1)
        for (int j = 0; j < n; j++)
            if (i <= j) h[i + j * (j + 1) / 2] += c1 * (mi * p[j] + mhy[j] * pi) + c2p * p[j];
    } else {
#pragma unroll 1
        for (int j = 0; j < n; j++)
#pragma unroll 1
            for (int i = lane64(); i <= j; i += 32)
                h[i + j * (j + 1) / 2] += c1 * (mhy[i] * p[j] + mhy[j] * p[i]) + c2 * p[i] * p[j];
    }
    __syncwarp();
}

// ---- QuickVina 2 history (not smina's search) ----------------------------------------------
// QuickVina 2 (Alhossary, Handoko, Mu and Kwoh, Bioinformatics 31:2214, 2015)
// skips a local optimisation whose start the chain's recent history already
// accounts for.  The history holds the last 5n points (n = dof) that local
// optimisations visited, with their energies and gradient signs.  A stored
// point e is consistent with a start (x, f, g) when, in every coordinate in
// which both gradients have the same nonzero sign, "gradient positive" equals
// "x_i > e_i" xor "f > f_e".  A start is worth optimising when a consistent
// point is among its 4n nearest (squared distance in change coordinates,
// ties to the lower slot); until 5n points are stored, every start is.  The
// decisions are those of the reference's gpu_mc.cuh:144-264, which the
// checker restates and this path matches bit for bit.
//
// The device layout and the check are this file's own:
//  - coordinates are stored coordinate-major, so for one coordinate the
//    lanes read consecutive slots;
//  - lane l owns slots l, l + 32, ...; their squared distances and "start
//    above the point" bits build up in registers while the coordinates
//    stream past (the start's coordinate comes by shuffle), so nothing is
//    written back but the new point;
//  - the sign test is mask algebra on 64-bit words: it applies where
//    nz_e & nz_x & ~(pos_e ^ pos_x), and a point fails when any of those
//    coordinates has pos_x ^ above ^ uphill set.
constexpr int kHistSlotsPerLane = (5 * kHistMaxN + 31) / 32;

__device__ __forceinline__ Hist64 hist64_view(double* d, unsigned long long* u, int n) {
    const size_t cap = (size_t)5 * n;
    return Hist64{d, d + (size_t)n * cap, u, u + 2 * cap};
}

// (nonzero, positive) masks of the gradient's n coordinates, on every lane
__device__ __forceinline__ ulonglong2 grad_signs64(const double* g, int n) {
    unsigned nz[2], pos[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int i = 32 * h + lane64();
        const double v = i < n ? g[i] : 0.0;
        nz[h] = __ballot_sync(kFull, !(v == 0));
        pos[h] = __ballot_sync(kFull, v > 0);
    }
    return make_ulonglong2(nz[0] | (unsigned long long)nz[1] << 32, pos[0] | (unsigned long long)pos[1] << 32);
}

// stores (x, f, sign(g)) in the next slot (the oldest point once the ring is full)
template <bool ST>
__device__ __noinline__ void hist64_add(const Hist64& H, const double* x, double f, const double* g) {
    const int n = hd64().m.dof, cap = 5 * n;
    const unsigned long long adds = __shfl_sync(kFull, lane64() == 0 ? *H.adds : 0ull, 0);
    const int slot = (int)(adds % (unsigned long long)cap);
    const ulonglong2 sg = grad_signs64(g, n);
    for (int i = lane64(); i < n; i += 32) H.x[(size_t)i * cap + slot] = conf_value64<ST>(x, i);
    if (lane64() == 0) {
        H.f[slot] = f;
        H.mask[2 * slot] = sg.x;
        H.mask[2 * slot + 1] = sg.y;
        *H.adds = adds + 1;
    }
    __syncwarp();
}

// true when a local optimisation from (x, f, g) should run
template <bool ST>
__device__ __noinline__ bool hist64_interesting(const Hist64& H, const double* x, double f, const double* g) {
    const int n = hd64().m.dof, cap = 5 * n;
    const unsigned long long adds = __shfl_sync(kFull, lane64() == 0 ? *H.adds : 0ull, 0);
    if (adds < (unsigned long long)cap) return true;
    const double x_lo = lane64() < n ? conf_value64<ST>(x, lane64()) : 0.0;
    const double x_hi = lane64() + 32 < n ? conf_value64<ST>(x, lane64() + 32) : 0.0;
    const ulonglong2 sx = grad_signs64(g, n);
    double d2[kHistSlotsPerLane];
    unsigned long long above[kHistSlotsPerLane];
#pragma unroll
    for (int k = 0; k < kHistSlotsPerLane; k++) { d2[k] = 0; above[k] = 0; }
    for (int i = 0; i < n; i++) {
        const double xi = __shfl_sync(kFull, i < 32 ? x_lo : x_hi, i & 31);
        const double* row = H.x + (size_t)i * cap;
#pragma unroll
        for (int k = 0; k < kHistSlotsPerLane; k++) {
            const int e = lane64() + 32 * k;
            if (e < cap) {
                const double dx = row[e] - xi;  // summed in coordinate order
                d2[k] += dx * dx;
                if (dx < 0) above[k] |= 1ull << i;
            }
        }
    }
    // nearest consistent point, in (distance, slot) order
    double best = kMaxFl;
    int besti = cap;
#pragma unroll
    for (int k = 0; k < kHistSlotsPerLane; k++) {
        const int e = lane64() + 32 * k;
        if (e < cap) {
            const unsigned long long nz = H.mask[2 * e], pos = H.mask[2 * e + 1];
            const unsigned long long uphill = f - H.f[e] > 0 ? ~0ull : 0ull;
            const unsigned long long applies = nz & sx.x & ~(pos ^ sx.y);
            if ((applies & (sx.y ^ above[k] ^ uphill)) == 0 && d2[k] < best) { best = d2[k]; besti = e; }
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(kFull, best, o);
        const int oi = __shfl_xor_sync(kFull, besti, o);
        if (ob < best || (ob == best && oi < besti)) { best = ob; besti = oi; }
    }
    if (besti >= cap) return false;
    // its rank: the points strictly before it in (distance, slot) order
    int ahead = 0;
#pragma unroll
    for (int k = 0; k < kHistSlotsPerLane; k++) {
        const int e = lane64() + 32 * k;
        if (e < cap) ahead += d2[k] < best || (d2[k] == best && e < besti);
    }
    for (int o = 16; o > 0; o >>= 1) ahead += __shfl_xor_sync(kFull, ahead, o);
    return ahead < 4 * n;
}

template <int G, bool ST>
__device__ __noinline__ double bfgs64(double* x, int maxiters, int accurate, int early, const EvalMode em,
                                      const Hist64* vis = nullptr) {
    const int n = hd64().m.dof, cs = hd64().m.conf_size;
    const Ws64& L = hd64().L;
    double* S = smem64;
    double* h = S + L.h;
    double *g = S + L.g, *g_new = S + L.g_new, *g_orig = S + L.g_orig, *p = S + L.p, *y = S + L.y;
    double *x_new = S + L.x_new, *x_orig = S + L.x_orig;
    const int lane = lane64();
#pragma unroll 1
    for (int t = lane; t < n * (n + 1) / 2; t += 32) h[t] = 0;
    __syncwarp();
#pragma unroll 1
    for (int i = lane; i < n; i += 32) h[i + i * (i + 1) / 2] = 1;
    __syncwarp();
    double f0 = feval<G, ST>(x, g, em);
    if (vis) {
        if (!hist64_interesting<ST>(*vis, x, f0, g)) return f0;
        hist64_add<ST>(*vis, x, f0, g);
    }
    const double f_orig = f0;
    vcopy(g_orig, g, n);
    vcopy(x_orig, x, cs);
    for (int step = 0; step < maxiters; step++) {
        minus_mat_vec64<ST>(h, g, p, n);
        double f1 = 0;
        const double alpha = accurate ? accurate_line_search64<G, ST>(x, g, f0, p, x_new, g_new, f1, em)
                                      : fast_line_search64<G, ST>(x, g, f0, p, x_new, g_new, f1, em);
        if (alpha == 0) break;
#pragma unroll 1
        for (int i = lane; i < n; i += 32) { double t = g_new[i]; t -= g[i]; y[i] = t; }
        __syncwarp();
        const double prevf0 = f0;
        f0 = f1;
        vcopy(x, x_new, cs);
        if (early && fabs(prevf0 - f0) < 1e-5) break;
        vcopy(g, g_new, n);
        const double gn = sprod64<ST>(g, g, n);
        if (!(gn >= 1e-4)) break;
        const double yp = sprod64<ST>(y, p, n);
        if (step == 0) {
            const double yy = sprod64<ST>(y, y, n);
            if (fabs(yy) > kEps) {
                const double d = alpha * yp / yy;
#pragma unroll 1
                for (int i = lane; i < n; i += 32) h[i + i * (i + 1) / 2] = d;
                __syncwarp();
            }
        }
        bfgs_update64<ST>(h, p, y, yp, alpha, n);
        if (vis) hist64_add<ST>(*vis, x, f0, g);
    }
    if (!(f0 <= f_orig)) {
        f0 = f_orig;
        vcopy(x, x_orig, cs);
        vcopy(g, g_orig, n);
    }
    return f0;
}

// ---- Monte Carlo pieces ----------------------------------------------------------------
template <bool ST>
__device__ __forceinline__ double gyration64(int l) {
    using M = MV64<ST>;
    const Ws64& L = hd64().L;
    const double* S = smem64;
    const int *type = M::type();
    const int b = M::lig_begin()[l], e = M::lig_end()[l];
    const V3<double> o = ld3(S + L.origin + 3 * M::lig_root()[l]);
    double acc = 0;
    unsigned counter = 0;
    for (int i0 = b; i0 < e; i0 += 32) {  // squared distances side by side, added in atom order (hydrogens: +0)
        const int i = i0 + lane64();
        const bool heavy = i < e && !is_h(type[i]);
        counter += __popc(__ballot_sync(kFull, heavy));
        acc = add_in_order64<ST>(acc, heavy ? dist2(ld3(S + L.coords + 3 * i), o) : 0.0, min(32, e - i0));
    }
    return counter > 0 ? sqrt(acc / counter) : 0;
}

template <bool ST>
__device__ __forceinline__ void mutate64(double* x, double amplitude) {
    using M = MV64<ST>;
    const int *blk_rigid = M::blk_rigid(), *blk_ntors = M::blk_ntors(), *blk_conf = M::blk_conf();
    const int nblocks = hd64().m.nblocks;
    int num = 0;
    for (int b = 0; b < nblocks; b++) num += (blk_rigid[b] ? 2 : 0) + blk_ntors[b];
    if (num == 0) return;
    int which = rand_int(0, num - 1);
    int lig = 0;
    for (int b = 0; b < nblocks; b++) {
        double* c = x + blk_conf[b];
        if (blk_rigid[b]) {
            if (which == 0) {
                const V3<double> d = amplitude * rand_in_sphere();
                if (lane64() == 0) { c[0] += d.x; c[1] += d.y; c[2] += d.z; }
                __syncwarp();
                return;
            }
            --which;
            if (which == 0) {
                const double gr = gyration64<ST>(lig);
                if (gr > kEps) {
                    const V3<double> rot = amplitude / gr * rand_in_sphere();
                    if (lane64() == 0) {
                        Quat<double> q{c[3], c[4], c[5], c[6]};
                        q_increment(q, rot);
                        c[3] = q.a; c[4] = q.b; c[5] = q.c; c[6] = q.d;
                    }
                    __syncwarp();
                }
                return;
            }
            --which;
            c += 7;
            lig++;
        }
        if (which < blk_ntors[b]) {
            const double t = rand_fl(-kPi, kPi);
            if (lane64() == 0) c[which] = t;
            __syncwarp();
            return;
        }
        which -= blk_ntors[b];
    }
}

__device__ __forceinline__ bool metropolis64(double old_f, double new_f, double temperature) {
    if (new_f < old_f) return true;
    const double p = fd_exp((old_f - new_f) / temperature);
    return rand_fl(0, 1) < p;
}

// add_to_output_container with the container in global memory (slots + sorted
// order).  Lane j measures the pose to saved poses j, j + 32, ... (its atoms in
// order); the first of the nearest ones is picked over the lanes.
template <bool ST>
__device__ __noinline__ void add_to_output64(const Chain64& ch, const double* x, double e, double min_rmsd,
                                             int max_size) {
    using M = MV64<ST>;
    const Hdr64& Hd = hd64();
    const Ws64& L = Hd.L;
    const double* S = smem64;
    const int H = Hd.m.nheavy, cs = Hd.m.conf_size, lane = lane64();
    const int* heavy = M::heavy();
    int count = *ch.out_count;
    int bj = count;
    double best = kMaxFl;
    for (int j = lane; j < count; j += 32) {
        const double* oc = ch.out_coords + (size_t)ch.out_order[j] * H * 3;
        double acc = 0;
#pragma unroll 4
        for (int a = 0; a < H; a++) acc += dist2(ld3(S + L.coords + 3 * heavy[a]), ld3(oc + 3 * a));
        const double r = H > 0 ? sqrt(acc / H) : 0;
        if (j == 0 || r < best) { bj = j; best = r; }
    }
    // pose 0's distance stands unless another's is smaller (a NaN there stays)
    const bool first_nan = __shfl_sync(kFull, best != best, 0);
    if (first_nan) {
        bj = 0;
        best = __shfl_sync(kFull, best, 0);
    } else {
        for (int o = 16; o > 0; o >>= 1) {
            const double ob = __shfl_xor_sync(kFull, best, o);
            const int oj = __shfl_xor_sync(kFull, bj, o);
            if (ob < best || (ob == best && oj < bj)) { best = ob; bj = oj; }
        }
    }
    int target = -1;  // slot to overwrite / fill
    if (lane == 0) {
        if (bj < count && best < min_rmsd) {
            if (e < ch.out_e[ch.out_order[bj]]) target = ch.out_order[bj];
        } else if (count < max_size) {
            target = count;
            ch.out_order[count] = count;
            count++;
        } else if (count > 0 && e < ch.out_e[ch.out_order[count - 1]]) {
            target = ch.out_order[count - 1];
        }
    }
    target = __shfl_sync(kFull, target, 0);
    count = __shfl_sync(kFull, count, 0);
    if (target >= 0) {
        for (int i = lane; i < cs; i += 32) ch.out_conf[(size_t)target * cs + i] = x[i];
        for (int a = lane; a < H; a += 32)
            st3(ch.out_coords + ((size_t)target * H + a) * 3, ld3(S + L.coords + 3 * heavy[a]));
        if (lane == 0) ch.out_e[target] = e;
    }
    __syncwarp();
    if (lane == 0) {
        *ch.out_count = count;
        for (int i = 1; i < count; i++) {  // stable insertion sort by energy
            const int key = ch.out_order[i];
            const double ek = ch.out_e[key];
            int j = i - 1;
            while (j >= 0 && ch.out_e[ch.out_order[j]] > ek) { ch.out_order[j + 1] = ch.out_order[j]; j--; }
            ch.out_order[j + 1] = key;
        }
    }
    __syncwarp();
}

}  // namespace sg
