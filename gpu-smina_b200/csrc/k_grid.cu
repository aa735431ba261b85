// Grid-map construction (cache::populate, cache.cpp:116-206).
//
// 1. Receptor cell lists (szv_grid.h:55-221): for every 3 A cell, the heavy
//    typed receptor atoms within the cutoff of both the search box and the
//    cell's brick, in receptor order.  cache::populate builds each cell's
//    list for the brick of the first grid point that queries the cell (a
//    point on a cell face gives a flat brick); k_cell_lists takes that brick
//    per axis from the host (first query in x, y, z loop order).  The
//    direct-sum path uses full 3 A bricks: the second family of lists.  A block
//    per cell and family, a stretch of the atoms per warp, ordered compaction
//    with ballots.
// 2. k_grid_map64: one lane per ligand type, W lanes per grid point, FP64 sums
//    over the point's cell list in receptor order; identical rounding to the
//    CPU's loop (each type's sum is independent).
//    A user grid (--user_grid) is added to every map at the point's index
//    coordinates (x, y, z), with the cache's slope, as cache::populate does
//    (cache.cpp:204-205).
// 3. k_grid_pack: packed-corner FP32 / FP16 copies for the mixed-precision path.
// Built without FMA contraction, like the CPU code it reproduces.
#include <algorithm>
#include "grid64.cuh"

namespace sg {

__device__ __forceinline__ double closest_between(double b, double e, double x) {
    if (x <= b) return b;
    if (x >= e) return e;
    return x;
}
__device__ __forceinline__ double brick_d2(double b0, double b1, double b2, double e0, double e1, double e2, double x,
                                           double y, double z) {
    const double c0 = closest_between(b0, e0, x), c1 = closest_between(b1, e1, y), c2 = closest_between(b2, e2, z);
    return sq(c0 - x) + sq(c1 - y) + sq(c2 - z);
}

// One cell's list of one family (blockIdx.y).  Without `list`: its length into
// count.  With it: every warp counts its stretch of the atoms again, places it
// behind the warps before it and writes its atoms whole.  bricks: per family lo
// and hi of every cell along x, then y, then z.  Bound by the latency of a
// warp's trips over its stretch: with one warp over all the atoms, and the
// families and passes in four launches, 4 x 181 us for 5,000 atoms and 1,331
// cells on one B200.
constexpr int kCellWarps = 8;
__global__ void __launch_bounds__(32 * kCellWarps) k_cell_lists(int natoms, const double* xyz, const int* type,
                                                               const double* charge, DGeom g, double cutoff_sqr,
                                                               const double* bricks, int* count, CellFamily fam0,
                                                               CellFamily fam1, const __grid_constant__ GridSlots slots) {
    __shared__ int s_count[kCellWarps];
    const int cell = blockIdx.x, nx = g.cell_dim[0], ny = g.cell_dim[1], nz = g.cell_dim[2];
    const CellFamily fam = blockIdx.y ? fam1 : fam0;
    const int cx = cell % nx, cy = (cell / nx) % ny, cz = cell / (nx * ny);
    const double* lo = bricks + (size_t)blockIdx.y * 2 * (nx + ny + nz);
    const double* hi = lo + nx + ny + nz;
    const double l0 = lo[cx], l1 = lo[nx + cy], l2 = lo[nx + ny + cz];
    const double h0 = hi[cx], h1 = hi[nx + cy], h2 = hi[nx + ny + cz];
    const bool empty = !(l0 == l0 && l1 == l1 && l2 == l2);  // NaN brick: no grid point in this cell
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = ((natoms + kCellWarps - 1) / kCellWarps + 31) & ~31;
    const int first = warp * per, last = min(natoms, first + per);
    auto inside = [&](int i, V3<double>& x, int& t) {
        if (empty || i >= last) return false;
        t = type[i];
        if (t >= kNumTypes || is_h(t)) return false;
        x = V3<double>{xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]};
        return brick_d2(g.gd_begin[0], g.gd_begin[1], g.gd_begin[2], g.gd_end[0], g.gd_end[1], g.gd_end[2], x.x, x.y,
                        x.z) < cutoff_sqr &&
               brick_d2(l0, l1, l2, h0, h1, h2, x.x, x.y, x.z) < cutoff_sqr;
    };
    int n = 0;
    for (int base = first; base < last; base += 32) {
        V3<double> x;
        int t;
        n += __popc(__ballot_sync(0xffffffffu, inside(base + lane, x, t)));
    }
    if (lane == 0) s_count[warp] = n;
    __syncthreads();
    int before = 0, all = 0;
    for (int w = 0; w < kCellWarps; w++) {
        if (w < warp) before += s_count[w];
        all += s_count[w];
    }
    if (!fam.list) {
        if (threadIdx.x == 0) count[(size_t)blockIdx.y * gridDim.x + cell] = all;
        return;
    }
    int at = fam.start[cell] + before;
    for (int base = first; base < last; base += 32) {
        V3<double> x;
        int t;
        const bool in = inside(base + lane, x, t);
        const unsigned mask = __ballot_sync(0xffffffffu, in);
        if (in) {
            const int k = at + __popc(mask & ((1u << lane) - 1));
            fam.list[k] = CellAtom{x.x, x.y, x.z, t, slots.of[t]};
            fam.charge[k] = charge[base + lane];
        }
        at += __popc(mask);
    }
}

// The fast table rearranged for the maps: [receptor type slot][sample][lane]
// (lanes past the last ligand type hold 0), NC components side by side, the
// first two already in the order of the lookup (charge of the receptor atom
// first).  All types' values of one (receptor type, distance) then lie in one
// 128-byte line instead of W lines.
template <int NC>
__global__ void k_grid_table(const double* fast, int n, const int* types, int ntypes, const __grid_constant__ GridSlots slots, int W,
                             double* out) {
    const size_t total = (size_t)slots.count * n * W;
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < total; k += (size_t)gridDim.x * blockDim.x) {
        const int j = (int)(k % W);
        const size_t i = (k / W) % n;
        const int t1 = slots.type[k / ((size_t)W * n)];
        double v[NC];
#pragma unroll
        for (int c = 0; c < NC; c++) v[c] = 0;
        if (j < ntypes) {
            const int t2 = types[j];
            const bool sw = t1 > t2;
            const double* f = fast + ((size_t)(sw ? tri_index(t2, t1) : tri_index(t1, t2)) * n + i) * NC;
            v[0] = f[0];
            if constexpr (NC > 1) {
                v[1] = sw ? f[2] : f[1];
                v[2] = sw ? f[1] : f[2];
                v[3] = f[3];
            }
        }
#pragma unroll
        for (int c = 0; c < NC; c++) out[k * NC + c] = v[c];
    }
}

// One chunk of up to W ligand types.  W lanes serve a point: they test W atoms
// of its cell list at once, then, for every atom within the cutoff in list
// order, each lane adds its own type's table value; four lookups are in flight.
// Bound by the table gathers (one 8 W byte line segment per point and in-cutoff
// atom, through L1 and L2).  A thread per point reading each type's table on its
// own took 8 B of W different lines, walked the list twice for more than 8 types
// and waited for a list index, an atom and a table value in turn: 16 maps of 70^3
// points around 5,000 atoms 1,688 us, now 443 us on one B200; 7 charge-dependent
// ones of 67^3 points around 3,000 atoms 2,098 us, now 906 us.
template <int W, int NC>
__global__ void __launch_bounds__(256) k_grid_map64(DGeom g, const CellAtom* list, const double* list_charge,
                                                    const int* cstart, const double* tab, int n,
                                                    double factor, double cutoff_sqr, int ntypes, double** maps,
                                                    double** cmaps, const double* ugrid, DGeom ug, double ug_slope) {
    constexpr int P = 32 / W;  // points a warp serves at a time
    const int lane = threadIdx.x & 31, j = lane % W, sub = lane / W;
    const unsigned submask = (W == 32 ? 0xffffffffu : (1u << W) - 1) << (sub * W);
    const long long npts = (long long)g.dim[0] * g.dim[1] * g.dim[2];
    const long long nwarps = (long long)gridDim.x * (blockDim.x / 32);
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    for (long long p0 = warp * P; p0 < npts; p0 += nwarps * P) {  // warp-uniform
        const long long idx = p0 + sub;
        const bool act = idx < npts;
        const int x = act ? (int)(idx % g.dim[0]) : 0, y = act ? (int)(idx / g.dim[0] % g.dim[1]) : 0,
                  z = act ? (int)(idx / ((long long)g.dim[0] * g.dim[1])) : 0;
        const double px = g.init[0] + g.factor_inv[0] * x, py = g.init[1] + g.factor_inv[1] * y,
                     pz = g.init[2] + g.factor_inv[2] * z;
        const int cx = (int)floor(px / 3.0) - g.cell_off[0], cy = (int)floor(py / 3.0) - g.cell_off[1],
                  cz = (int)floor(pz / 3.0) - g.cell_off[2];
        const bool cell_ok = act && cx >= 0 && cy >= 0 && cz >= 0 && cx < g.cell_dim[0] && cy < g.cell_dim[1] &&
                             cz < g.cell_dim[2];
        const int cell = cell_ok ? cx + g.cell_dim[0] * (cy + g.cell_dim[1] * cz) : 0;
        const int b = cell_ok ? cstart[cell] : 0, e = cell_ok ? cstart[cell + 1] : 0;
        double aff = 0, chg = 0;
        for (int k0 = b; __any_sync(0xffffffffu, k0 < e); k0 += W) {
            int row = 0;  // this lane's atom: its table row
            double q = 0;
            bool in = false;
            if (k0 + j < e) {
                const CellAtom a = load_cell_atom(list + k0 + j);
                const double r2 = sq(a.x - px) + sq(a.y - py) + sq(a.z - pz);
                if (r2 <= cutoff_sqr) {
                    in = true;
                    row = a.slot * n + (int)(factor * r2);
                    if (NC > 1) q = list_charge[k0 + j];
                }
            }
            unsigned m = __ballot_sync(0xffffffffu, in) & submask;
            while (__any_sync(0xffffffffu, m != 0)) {
                double f[4][NC], qa[4];
                bool ok[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    ok[u] = m != 0;
                    const int src = ok[u] ? __ffs(m) - 1 : lane;
                    m &= m - 1;
                    const int r = __shfl_sync(0xffffffffu, row, src);
                    if (NC > 1) qa[u] = __shfl_sync(0xffffffffu, q, src);
                    if (ok[u]) {
                        const double* t = tab + ((size_t)r * W + j) * NC;
                        if constexpr (NC == 1) {
                            f[u][0] = __ldg(t);
                        } else {
                            const double2 t0 = __ldg(reinterpret_cast<const double2*>(t)),
                                          t1 = __ldg(reinterpret_cast<const double2*>(t) + 1);
                            f[u][0] = t0.x; f[u][1] = t0.y; f[u][2] = t1.x; f[u][3] = t1.y;
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (ok[u]) {
                        if constexpr (NC > 1) {
                            aff += f[u][0] + f[u][1] * fabs(qa[u]);
                            chg += f[u][2] + f[u][3] * qa[u];
                        } else {
                            aff += f[u][0];
                        }
                    }
            }
        }
        if (act && j < ntypes) {
            if (ugrid)
                aff += grid_value64(ug, ugrid, V3<double>{(double)x, (double)y, (double)z}, ug_slope, 1000.0);
            maps[j][idx] = aff;
            if (NC > 1) cmaps[j][idx] = chg;
        }
    }
}

// Packed-corner copies for the mixed-precision path: cell (x, y, z) of the
// (dim-1)^3 cells stores its 8 corners contiguously, so one trilinear lookup
// is one 32 B (FP32) or 16 B (FP16) load instead of four row segments.  One
// launch packs every new map (blockIdx.y); bound by the writes.
__global__ void k_grid_pack(DGeom g, const GridPack* maps) {
    const GridPack mp = maps[blockIdx.y];
    const unsigned cx = g.dim[0] - 1, cy = g.dim[1] - 1, cz = g.dim[2] - 1;
    const size_t ncells = (size_t)cx * cy * cz;
    const size_t d0 = g.dim[0], d01 = (size_t)g.dim[0] * g.dim[1];
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < ncells; c += (size_t)gridDim.x * blockDim.x) {
        const size_t row = c / cx, x = c - row * cx, z = row / cy, y = row - z * cy;
        const double* b = mp.src + x + d0 * y + d01 * z;
        const double v[8] = {b[0], b[1], b[d0], b[d0 + 1], b[d01], b[d01 + 1], b[d01 + d0], b[d01 + d0 + 1]};
        if (mp.dst32) {
            mp.dst32[2 * c] = make_float4((float)v[0], (float)v[1], (float)v[2], (float)v[3]);
            mp.dst32[2 * c + 1] = make_float4((float)v[4], (float)v[5], (float)v[6], (float)v[7]);
        }
        if (mp.dst16) {
            uint32_t w[4];
            for (int k = 0; k < 4; k++)
                w[k] = (uint32_t)__half_as_ushort(__double2half(v[2 * k])) |
                       ((uint32_t)__half_as_ushort(__double2half(v[2 * k + 1])) << 16);
            mp.dst16[c] = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

// both families' lengths (lists null) or lists
cudaError_t launch_cell_lists(int natoms, const double* xyz, const int* type, const double* charge, const DGeom& g,
                              double cutoff_sqr, const double* bricks, int* count, const CellFamily& fam0,
                              const CellFamily& fam1, const GridSlots& slots, cudaStream_t s) {
    const dim3 grid(g.cell_dim[0] * g.cell_dim[1] * g.cell_dim[2], 2);
    k_cell_lists<<<grid, 32 * kCellWarps, 0, s>>>(natoms, xyz, type, charge, g, cutoff_sqr, bricks, count, fam0, fam1,
                                                  slots);
    return cudaGetLastError();
}

// lanes per point for a chunk of ntypes ligand types
int grid_lanes(int ntypes) { return ntypes <= 4 ? 4 : ntypes <= 8 ? 8 : ntypes <= 16 ? 16 : 32; }

template <int W, int NC>
static void run_grid_map(const DGeom& g, const CellAtom* list, const double* list_charge, const int* cstart,
                         const DTables& T, const int* types, int ntypes, const GridSlots& slots, double* tab,
                         double** maps, double** cmaps, const double* ugrid, const DGeom& ug, double ug_slope,
                         int num_sms, cudaStream_t s) {
    k_grid_table<NC><<<num_sms * 8, 256, 0, s>>>(T.fast, T.n, types, ntypes, slots, W, tab);
    const long long npts = (long long)g.dim[0] * g.dim[1] * g.dim[2];
    const int blocks = (int)std::min<long long>((npts * W + 255) / 256, num_sms * 64LL);
    k_grid_map64<W, NC><<<blocks, 256, 0, s>>>(g, list, list_charge, cstart, tab, T.n, T.factor, T.cutoff_sqr,
                                               ntypes, maps, cmaps, ugrid, ug, ug_slope);
}

// maps of one chunk of at most 32 ligand types; tab: slots.count * T.n *
// grid_lanes(ntypes) * T.nc doubles
cudaError_t launch_grid_map64(const DGeom& g, const CellAtom* list, const double* list_charge, const int* cstart,
                              const DTables& T, const int* types, int ntypes, const GridSlots& slots, double* tab,
                              double** maps, double** cmaps, const double* ugrid, const DGeom& ug, double ug_slope,
                              int num_sms, cudaStream_t s) {
    const int W = grid_lanes(ntypes);
#define SG_GRID(w, nc) \
    run_grid_map<w, nc>(g, list, list_charge, cstart, T, types, ntypes, slots, tab, maps, cmaps, ugrid, ug, ug_slope, num_sms, s)
    if (T.nc == 1) {
        if (W == 4) SG_GRID(4, 1);
        else if (W == 8) SG_GRID(8, 1);
        else if (W == 16) SG_GRID(16, 1);
        else SG_GRID(32, 1);
    } else {
        if (W == 4) SG_GRID(4, 4);
        else if (W == 8) SG_GRID(8, 4);
        else if (W == 16) SG_GRID(16, 4);
        else SG_GRID(32, 4);
    }
#undef SG_GRID
    return cudaGetLastError();
}

cudaError_t launch_grid_pack(const DGeom& g, const GridPack* maps, int nmaps, cudaStream_t s) {
    const size_t ncells = (size_t)(g.dim[0] - 1) * (g.dim[1] - 1) * (g.dim[2] - 1);
    const dim3 grid((unsigned)std::min<size_t>((ncells + 255) / 256, 148 * 8), nmaps);
    k_grid_pack<<<grid, 256, 0, s>>>(g, maps);
    return cudaGetLastError();
}

}  // namespace sg
