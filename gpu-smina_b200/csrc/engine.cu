// C ABI of the B200 docking engine (include/smina_b200.h): device state,
// input validation, model packing and kernel launches.  Every entry point
// returns a status code; no exception crosses the ABI.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <exception>
#include <map>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <thread>
#include <vector>
#include "engine.h"

namespace sg {

// ---- the devices' pools of call temporaries ------------------------------------------------
// Streams of different engines never wait for one another through a pool: it
// only hands a block to another stream once the first stream's work is done.
// When an allocation fails, what the pools and the dropped maps (below) keep is
// given back and it is tried again.
struct DevPool {
    cudaMemPool_t pool = nullptr;
    int users = 0;
};
static std::atomic<size_t> g_engines{0};  // in the process
static std::mutex g_pools_mu;
static std::map<int, DevPool>& g_pools = *new std::map<int, DevPool>;  // (never destroyed: no CUDA call after main)

static void drop_pin_rings();
cudaMemPool_t pool_acquire(int device) {
    std::lock_guard<std::mutex> lk(g_pools_mu);
    DevPool& d = g_pools[device];
    if (!d.pool) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cuda_check(cudaMemPoolCreate(&d.pool, &props), "memory pool");
        uint64_t keep = kPoolKept;
        int no = 0;
        cuda_check(cudaMemPoolSetAttribute(d.pool, cudaMemPoolAttrReleaseThreshold, &keep), "memory pool");
        cuda_check(cudaMemPoolSetAttribute(d.pool, cudaMemPoolReuseAllowInternalDependencies, &no), "memory pool");
    }
    d.users++;
    g_engines++;
    return d.pool;
}
void pool_release(int device) {
    std::lock_guard<std::mutex> lk(g_pools_mu);
    DevPool& d = g_pools[device];
    g_engines--;
    if (--d.users == 0) {
        cudaMemPoolDestroy(d.pool);
        d.pool = nullptr;
    }
    for (auto& q : g_pools)
        if (q.second.users) return;
    drop_pin_rings();  // the process's last engine is gone
}

// ---- dropped maps ------------------------------------------------------------------------
// A receptor's maps that new tables, a user grid or another receptor in its place
// make void: their allocations wait here for the next map build in that place,
// which takes one that fits and frees the others (18 maps of a 22 A box with a new
// user grid 22 ms of cudaFree and cudaMalloc otherwise, 0.7 to 1.2 ms so).  At most
// kDroppedKept bytes per device, the oldest freed first; a direct sum in that
// place frees them too, and an allocation that fails frees all on its device.
struct DroppedMaps {
    RecState* of;
    int device;
    std::unique_ptr<DevBuf> mem;
};
constexpr size_t kDroppedKept = size_t(2) << 30;
static std::mutex g_dropped_mu;
static std::vector<DroppedMaps>& g_dropped = *new std::vector<DroppedMaps>;  // oldest first

// frees those that `which` picks
template <typename F>
static void free_dropped(F which) {
    std::lock_guard<std::mutex> lk(g_dropped_mu);
    g_dropped.erase(std::remove_if(g_dropped.begin(), g_dropped.end(), which), g_dropped.end());
}
static void free_dropped_of(RecState& r) {
    free_dropped([&](const DroppedMaps& d) { return d.of == &r; });
}
RecState::~RecState() { free_dropped_of(*this); }
// forgets r's maps, their memory kept for its next ones
static void drop_maps(sg_engine* e, RecState& r) {
    size_t kept = 0;
    {
        std::lock_guard<std::mutex> lk(g_dropped_mu);
        g_dropped.reserve(g_dropped.size() + r.map_mem.size());
        for (auto& m : r.map_mem) g_dropped.push_back({&r, e->device, std::move(m)});
        for (const DroppedMaps& d : g_dropped) kept += d.device == e->device ? d.mem->bytes : 0;
    }
    r.clear_maps();
    free_dropped([&](const DroppedMaps& d) {
        if (d.device != e->device || kept <= kDroppedKept) return false;
        kept -= d.mem->bytes;
        return true;
    });
}
// memory for n bytes of r's maps
static std::unique_ptr<DevBuf> map_memory(RecState& r, size_t n) {
    std::unique_ptr<DevBuf> mem;
    {
        std::lock_guard<std::mutex> lk(g_dropped_mu);
        for (auto d = g_dropped.begin(); d != g_dropped.end() && !mem; ++d)
            if (d->of == &r && d->mem->bytes >= n && d->mem->bytes / 2 <= n) {
                mem = std::move(d->mem);
                g_dropped.erase(d);
                break;
            }
    }
    free_dropped_of(r);
    if (!mem) {
        mem.reset(new DevBuf());
        mem->alloc(n);
    }
    return mem;
}

static cudaError_t alloc_device(void** p, size_t n, sg_engine* pooled) {
    if (pooled && pooled->pool) return cudaMallocFromPoolAsync(p, n, pooled->pool, pooled->stream);
    return cudaMalloc(p, n);
}
void DevBuf::reset() {
    if (p) {
        if (pool_of && pool_of->pool) cudaFreeAsync(p, pool_of->stream);
        else cudaFree(p);
    }
    p = nullptr;
    bytes = cap = 0;
}
void DevBuf::alloc(size_t n) {
    if (n == 0) n = 16;
    if (p && n <= cap && cap / 2 <= n + (64 << 10)) {
        bytes = n;
        return;
    }
    reset();
    if (alloc_device(&p, n, pool_of) != cudaSuccess) {
        cudaGetLastError();
        int device = 0;
        cudaGetDevice(&device);
        free_dropped([&](const DroppedMaps& d) { return d.device == device; });
        {
            std::lock_guard<std::mutex> lk(g_pools_mu);
            for (auto& q : g_pools)
                if (q.second.pool) cudaMemPoolTrimTo(q.second.pool, 0);
        }
        if (alloc_device(&p, n, pool_of) != cudaSuccess) {
            cudaGetLastError();
            p = nullptr;
            throw EngineError(SG_ERR_NOMEM, "device allocation of " + std::to_string(n) + " bytes failed");
        }
    }
    bytes = cap = n;
}
void DevBuf::upload(const void* src, size_t n, cudaStream_t s) {
    alloc(n);
    if (n) cuda_check(cudaMemcpyAsync(p, src, n, cudaMemcpyHostToDevice, s), "upload");
}

// ---- a call's copies ----------------------------------------------------------------------
static std::mutex g_rings_mu;
static std::vector<std::unique_ptr<PinRing>>& g_rings = *new std::vector<std::unique_ptr<PinRing>>;  // free ones
static void drop_pin_rings() {
    std::lock_guard<std::mutex> lk(g_rings_mu);
    g_rings.clear();
}

PinRing::~PinRing() {
    for (cudaEvent_t x : ev)
        if (x) cudaEventDestroy(x);
    if (pinned) cudaFreeHost(p);
    else delete[] p;
}
static std::unique_ptr<PinRing> ring_get() {
    {
        std::lock_guard<std::mutex> lk(g_rings_mu);
        if (!g_rings.empty()) {
            auto r = std::move(g_rings.back());
            g_rings.pop_back();
            return r;
        }
    }
    auto r = std::make_unique<PinRing>();
    constexpr size_t n = PinRing::kSlot * PinRing::kSlots;
    r->pinned = cudaHostAlloc((void**)&r->p, n, cudaHostAllocPortable) == cudaSuccess;
    if (!r->pinned) {
        cudaGetLastError();
        r->p = nullptr;
        r->p = new char[n];
    }
    return r;
}
// As many free rings are kept as the process has engines (a call at a time on
// each): with four at most, eight engines on eight threads pinned memory on every
// other call, and 800 evaluations of 64 confs took 293 ms on one B200 (12 ms for
// 400 on four threads).
static void ring_put(std::unique_ptr<PinRing> r) {
    for (cudaEvent_t& x : r->ev) {  // events belong to the call's device
        if (x) cudaEventDestroy(x);
        x = nullptr;
    }
    std::lock_guard<std::mutex> lk(g_rings_mu);
    try {
        if (r->pinned && g_rings.size() < g_engines) g_rings.push_back(std::move(r));
    } catch (std::bad_alloc&) {  // not kept then (callers are destructors)
    }
}
void warm_pin_ring() {
    {
        std::lock_guard<std::mutex> lk(g_rings_mu);
        if (!g_rings.empty()) return;
    }
    ring_put(ring_get());
}
static void mark(PinRing& r, int slot, cudaStream_t s) {
    if (!r.ev[slot]) cuda_check(cudaEventCreateWithFlags(&r.ev[slot], cudaEventDisableTiming), "event");
    cuda_check(cudaEventRecord(r.ev[slot], s), "event");
}
void CallIo::need_ring() {
    if (!ring_) ring_ = ring_get();
}
CallIo::~CallIo() {
    if (busy_) cudaStreamSynchronize(e_->stream);  // an error left copies in flight
    if (ring_) ring_put(std::move(ring_));
}
void CallIo::in(DevBuf& dst, const void* src, size_t n) {
    dst.alloc(n);
    if (!n) return;
    need_ring();
    busy_ = true;
    for (size_t at = 0; at < n;) {
        if (in_used_ == PinRing::kSlot) {  // on to the other slot, once its copies are done
            mark(*ring_, in_slot_, e_->stream);
            in_sent_[in_slot_] = true;
            in_slot_ ^= 1;
            in_used_ = 0;
            if (in_sent_[in_slot_]) cuda_check(cudaEventSynchronize(ring_->ev[in_slot_]), "copy in");
        }
        const size_t k = std::min(n - at, PinRing::kSlot - in_used_);
        char* q = ring_->p + in_slot_ * PinRing::kSlot + in_used_;
        std::memcpy(q, static_cast<const char*>(src) + at, k);
        cuda_check(cudaMemcpyAsync(dst.as<char>() + at, q, k, cudaMemcpyHostToDevice, e_->stream), "copy in");
        in_used_ = std::min(PinRing::kSlot, (in_used_ + k + 15) & ~(size_t)15);
        at += k;
    }
}
void CallIo::out(void* host, const void* dev, size_t n) {
    if (host && n) outs_.push_back({host, dev, n});
}
// Fetches the outputs (behind the device error word, which is cleared for the
// next call and turned into a status).
void CallIo::finish() {
    need_ring();
    busy_ = true;
    int err = kDevOk;
    std::vector<Out> todo;
    todo.push_back({&err, e_->d_err.p, sizeof(int)});
    todo.insert(todo.end(), outs_.begin(), outs_.end());
    outs_.clear();
    std::vector<Piece> pieces[2];
    bool sent[2] = {};
    auto hand_over = [&](int s) {
        if (!sent[s]) return;
        cuda_check(cudaEventSynchronize(ring_->ev[2 + s]), "kernel");
        for (const Piece& p : pieces[s]) std::memcpy(p.host, p.from, p.n);
        pieces[s].clear();
        sent[s] = false;
    };
    int slot = 0;
    size_t used = 0;
    auto flush = [&] {
        mark(*ring_, 2 + slot, e_->stream);
        sent[slot] = true;
        slot ^= 1;
        used = 0;
    };
    for (const Out& o : todo)
        for (size_t at = 0; at < o.n;) {
            if (used == PinRing::kSlot) {
                flush();
                hand_over(slot);
            }
            const size_t k = std::min(o.n - at, PinRing::kSlot - used);
            char* q = ring_->p + (2 + slot) * PinRing::kSlot + used;
            cuda_check(cudaMemcpyAsync(q, static_cast<const char*>(o.dev) + at, k, cudaMemcpyDeviceToHost, e_->stream),
                       "copy out");
            pieces[slot].push_back({static_cast<char*>(o.host) + at, q, k});
            used = std::min(PinRing::kSlot, (used + k + 15) & ~(size_t)15);
            at += k;
        }
    hand_over(slot ^ 1);
    cuda_check(cudaStreamSynchronize(e_->stream), "kernel");  // the last slot
    for (const Piece& p : pieces[slot]) std::memcpy(p.host, p.from, p.n);
    busy_ = false;
    in_used_ = 0;
    in_sent_[0] = in_sent_[1] = false;
    if (err != kDevOk) {
        const int zero = 0;
        cuda_check(cudaMemcpy(e_->d_err.p, &zero, sizeof(int), cudaMemcpyHostToDevice), "clear error word");
        if (err == kDevOverlap) throw EngineError(SG_ERR_OVERLAP, "Ligand atom exactly overlaps receptor atom.");
        throw EngineError(SG_ERR_ARG, "device reported an out-of-range access (error " + std::to_string(err) + ")");
    }
}

cudaError_t raise_dynamic_smem(const void* kernel, size_t smem) {
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    cudaFuncAttributes fa{};
    cudaError_t rc = cudaFuncGetAttributes(&fa, kernel);
    if (rc != cudaSuccess || (size_t)fa.maxDynamicSharedSizeBytes >= smem) return rc;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

void cuda_check(cudaError_t e, const char* what) {
    if (e != cudaSuccess) {
        // a failed call that does not poison the context still stays the
        // thread's last error, which the next launch's check would report
        // again; clear it
        cudaGetLastError();
        throw EngineError(SG_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
    }
}

DGeom make_geom(const sg_grid_dims& gd) {
    DGeom g;
    for (int i = 0; i < 3; i++) {
        g.dim[i] = gd.n[i] + 1;
        g.init[i] = gd.begin[i];
        const double range = gd.end[i] - gd.begin[i];
        g.dim_fl_minus_1[i] = g.dim[i] - 1.0;
        g.factor[i] = g.dim_fl_minus_1[i] / range;
        g.factor_inv[i] = 1 / g.factor[i];
        g.gd_begin[i] = gd.begin[i];
        g.gd_end[i] = gd.end[i];
        g.gd_n[i] = gd.n[i];
        g.cell_off[i] = (int)std::floor(gd.begin[i] / 3.0);
        g.cell_dim[i] = (int)std::ceil(gd.end[i] / 3.0) - g.cell_off[i] + 1;
    }
    return g;
}

}  // namespace sg

using namespace sg;

// ---- engine -----------------------------------------------------------------------------------
sg_engine::~sg_engine() {
    if (stream) cudaStreamDestroy(stream);
    if (pool) pool_release(device);
}

extern "C" {

int sg_create(int device, int precision, sg_engine** out) {
    if (!out) return SG_ERR_ARG;
    *out = nullptr;
    if (precision < SG_PREC_FP64 || precision > SG_PREC_FP32_H16) return SG_ERR_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) return SG_ERR_CUDA;
    std::unique_ptr<sg_engine> e(new (std::nothrow) sg_engine());
    if (!e) return SG_ERR_NOMEM;
    e->device = device;
    e->precision = precision;
    int rc = guarded(e.get(), [&] {
        cuda_check(cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking), "stream");
        e->pool = pool_acquire(device);
        warm_pin_ring();
        e->d_err.alloc(sizeof(int));
        cuda_check(cudaMemsetAsync(e->d_err.p, 0, sizeof(int), e->stream), "memset");
        cudaDeviceProp prop;
        cuda_check(cudaGetDeviceProperties(&prop, device), "device properties");
        e->num_sms = prop.multiProcessorCount;
        e->max_smem = (int)prop.sharedMemPerBlockOptin;
        if (precision != SG_PREC_FP64) noalloc_claim(e.get());
    });
    if (rc != SG_OK) return rc;
    *out = e.release();
    return SG_OK;
}

void sg_destroy(sg_engine* e) {
    if (!e) return;
    cudaSetDevice(e->device);
    serve_shutdown(e);
    cudaStreamSynchronize(e->stream);
    delete e;
}

const char* sg_last_error(const sg_engine* e) { return e ? e->err.c_str() : "no engine"; }
int sg_precision(const sg_engine* e) { return e ? e->precision : -1; }

int sg_device_info(const sg_engine* e, int* device, int* num_sms, int* smem_optin) {
    if (!e) return SG_ERR_ARG;
    if (device) *device = e->device;
    if (num_sms) *num_sms = e->num_sms;
    if (smem_optin) *smem_optin = e->max_smem;
    return SG_OK;
}

int sg_set_tables(sg_engine* e, const sg_tables_desc* t) {
    return guarded(e, [&] {
        require(t && t->smooth && t->fast, "tables: null pointers");
        require(t->num_types == SG_NUM_TYPES, "tables: num_types must be 27");
        require(t->num_components == 1 || t->num_components == 4, "tables: num_components must be 1 or 4");
        require(t->factor > 0 && t->cutoff_sqr > 0, "tables: factor and cutoff must be positive");
        require(t->n >= (int)(size_t)(t->factor * t->cutoff_sqr) + 3 && t->n < (1 << 24), "tables: n too small");
        // (without tables from here on, should one of the uploads fail)
        e->has_tables = false;
        for (auto& r : e->rec) drop_maps(e, r);  // maps depend on the tables
        const size_t np = kNumTypePairs;
        e->tab_smooth.upload(t->smooth, np * t->n * t->num_components * 2 * sizeof(double), e->stream);
        e->tab_fast.upload(t->fast, np * t->n * t->num_components * sizeof(double), e->stream);
        // (e_i, dor_i, e_i+1, dor_i+1) per component: one 16 B load per lookup
        {
            const int nc = t->num_components, n = t->n;
            std::vector<float> t4(np * n * nc * 4, 0.f);
            for (size_t pr = 0; pr < np; pr++)
                for (int i = 0; i < n; i++)
                    for (int c = 0; c < nc; c++) {
                        const double* a = t->smooth + ((pr * n + i) * nc + c) * 2;
                        float* o = &t4[((pr * n + i) * nc + c) * 4];
                        o[0] = (float)a[0];
                        o[1] = (float)a[1];
                        if (i + 1 < n) { o[2] = (float)a[nc * 2]; o[3] = (float)a[nc * 2 + 1]; }
                    }
            e->tab32.upload(t4.data(), t4.size() * sizeof(float), e->stream);
        }
        e->tables.nc = t->num_components;
        e->tables.n = t->n;
        e->tables.factor = t->factor;
        e->tables.cutoff_sqr = t->cutoff_sqr;
        e->tables.smooth = (const double*)e->tab_smooth.p;
        e->tables.fast = (const double*)e->tab_fast.p;
        cuda_check(cudaStreamSynchronize(e->stream), "tables");
        e->has_tables = true;
    });
}

}  // extern "C"

// ---- receptors and grid maps ----------------------------------------------------------------------
namespace sg {

RecState& receptor_for(sg_engine* e, int rid) {
    require(rid >= 0 && rid < SG_MAX_RECEPTORS, "receptor id out of range");
    require(e->rec[rid].set, "receptor " + std::to_string(rid) + " has not been set");
    require(e->has_tables, "no tables set");
    return e->rec[rid];
}

void refresh_header(sg_engine* e, RecState& r) {
    DReceptor& h = r.hdr;
    h.natoms = r.natoms;
    h.xyz = r.xyz.as<double>();
    h.type = r.type.as<int>();
    h.charge = r.charge.as<double>();
    h.full_start = r.full_start.as<int>();
    h.full_list = r.full_list.as<CellAtom>();
    h.full_charge = r.full_charge.as<double>();
    h.g = r.geom;
    for (int t = 0; t < kNumTypes; t++) {
        h.map[t] = r.map64[t].as<double>();
        h.cmap[t] = r.cmap64[t].as<double>();
        h.map32[t] = r.map32[t].as<float4>();
        h.cmap32[t] = r.cmap32[t].as<float4>();
        h.map16[t] = r.map16[t].as<uint4>();
    }
    h.ugrid = r.ugrid.as<double>();
    h.ug = r.ug;
    if (!r.dhdr.p) r.dhdr.alloc(sizeof(DReceptor));
    cuda_check(cudaMemcpyAsync(r.dhdr.p, &h, sizeof(DReceptor), cudaMemcpyHostToDevice, e->stream), "receptor header");
    cuda_check(cudaStreamSynchronize(e->stream), "receptor header");
}

// Brick of every cell along each axis.  Populate: the first grid point of
// the cell in loop order (floor/ceil of its coordinate, flat when it lies on
// a face); direct sum: the full [3c, 3c + 3) brick.
static void cell_bricks(const DGeom& g, bool first_query, std::vector<double>& lo, std::vector<double>& hi) {
    lo.clear();
    hi.clear();
    const double nan = std::nan("");
    for (int d = 0; d < 3; d++) {
        std::vector<double> l(g.cell_dim[d], nan), h(g.cell_dim[d], nan);
        if (first_query) {
            for (int x = 0; x < g.dim[d]; x++) {
                const double c = g.init[d] + g.factor_inv[d] * x;
                const int cell = (int)std::floor(c / 3.0) - g.cell_off[d];
                if (cell < 0 || cell >= g.cell_dim[d] || l[cell] == l[cell]) continue;
                l[cell] = std::floor(c / 3.0) * 3.0;
                h[cell] = std::ceil(c / 3.0) * 3.0;
            }
        } else {
            for (int c = 0; c < g.cell_dim[d]; c++) {
                l[c] = (double)(c + g.cell_off[d]) * 3.0;
                h[c] = l[c] + 3.0;
            }
        }
        lo.insert(lo.end(), l.begin(), l.end());
        hi.insert(hi.end(), h.begin(), h.end());
    }
}

// the receptor's 3 A cell lists (CSR, whole atoms): first-query bricks for the
// maps, full bricks for the direct sum
static void build_receptor_cells(sg_engine* e, RecState& r) {
    const DGeom& g = r.geom;
    const int ncells = g.cell_dim[0] * g.cell_dim[1] * g.cell_dim[2];
    std::vector<double> bricks, lo, hi;
    for (int f = 0; f < 2; f++) {
        cell_bricks(g, f == 0, lo, hi);
        bricks.insert(bricks.end(), lo.begin(), lo.end());
        bricks.insert(bricks.end(), hi.begin(), hi.end());
    }
    DevBuf dbricks(e), dcount(e);
    dbricks.upload(bricks.data(), bricks.size() * sizeof(double), e->stream);
    dcount.alloc(2 * (size_t)ncells * sizeof(int));
    auto launch = [&](const CellFamily& pop, const CellFamily& full) {
        return launch_cell_lists(r.natoms, r.xyz.as<double>(), r.type.as<int>(), r.charge.as<double>(), g,
                                 e->tables.cutoff_sqr, dbricks.as<double>(), dcount.as<int>(), pop, full, r.slots,
                                 e->stream);
    };
    cuda_check(launch({}, {}), "cell count");
    std::vector<int> cnt(2 * (size_t)ncells), st[2];
    cuda_check(cudaMemcpyAsync(cnt.data(), dcount.p, cnt.size() * sizeof(int), cudaMemcpyDeviceToHost, e->stream), "counts");
    cuda_check(cudaStreamSynchronize(e->stream), "cell count");
    DevBuf* const bufs[2][3] = {{&r.pop_start, &r.pop_list, &r.pop_charge}, {&r.full_start, &r.full_list, &r.full_charge}};
    CellFamily fam[2];
    for (int f = 0; f < 2; f++) {
        st[f].assign(ncells + 1, 0);
        for (int c = 0; c < ncells; c++) st[f][c + 1] = st[f][c] + cnt[(size_t)f * ncells + c];
        const size_t n = std::max(1, st[f][ncells]);
        bufs[f][0]->upload(st[f].data(), st[f].size() * sizeof(int), e->stream);
        bufs[f][1]->alloc(n * sizeof(CellAtom));
        bufs[f][2]->alloc(n * sizeof(double));
        fam[f] = {bufs[f][0]->as<int>(), bufs[f][1]->as<CellAtom>(), bufs[f][2]->as<double>()};
    }
    cuda_check(launch(fam[0], fam[1]), "cell fill");
    refresh_header(e, r);
    r.cells = true;
}
void ensure_cells(sg_engine* e, RecState& r) {
    if (!r.cells) build_receptor_cells(e, r);
}
RecState& direct_receptor(sg_engine* e, int rid) {
    RecState& r = receptor_for(e, rid);
    ensure_cells(e, r);
    free_dropped_of(r);
    return r;
}

void ensure_maps(sg_engine* e, RecState& r, const int* types, int ntypes) {
    require(e->has_tables, "no tables set");
    std::vector<int> need;
    for (int k = 0; k < ntypes; k++) {
        const int t = types[k];
        require(t >= 0 && t < kNumTypes, "grid type out of range");
        if (!r.built[t] && std::find(need.begin(), need.end(), t) == need.end()) need.push_back(t);
    }
    if (need.empty()) return;
    ensure_cells(e, r);
    const size_t npts = (size_t)r.geom.dim[0] * r.geom.dim[1] * r.geom.dim[2];
    const bool charged = e->tables.nc > 1;
    const bool packed = e->precision != SG_PREC_FP64, half = e->precision == SG_PREC_FP32_H16;
    // one allocation for all the new maps, each 256-byte aligned
    const size_t ncells = (size_t)(r.geom.dim[0] - 1) * (r.geom.dim[1] - 1) * (r.geom.dim[2] - 1);
    const size_t b64 = npts * sizeof(double), b32 = packed ? ncells * 2 * sizeof(float4) : 0,
                 b16 = half ? ncells * sizeof(uint4) : 0;
    auto up = [](size_t n) { return (n + 255) & ~(size_t)255; };
    const size_t per_type = (up(b64) + up(b32)) * (charged ? 2 : 1) + up(b16), total = per_type * need.size();
    std::unique_ptr<DevBuf> mem = map_memory(r, total);
    char* at = mem->as<char>();
    auto place = [&](MapView& v, size_t n) {
        if (!n) return;
        v.p = at;
        v.bytes = n;
        at += up(n);
    };
    std::vector<double*> maps, cmaps;
    for (int t : need) {
        place(r.map64[t], b64);
        place(r.map32[t], b32);
        place(r.map16[t], b16);
        maps.push_back(r.map64[t].as<double>());
        if (charged) {
            place(r.cmap64[t], b64);
            place(r.cmap32[t], b32);
        }
        cmaps.push_back(r.cmap64[t].as<double>());
    }
    // their memory goes back with its maps when a later step fails
    struct Undo {
        RecState& r;
        const std::vector<int>& need;
        bool done = false;
        ~Undo() {
            if (done) return;
            for (int t : need) r.map64[t] = r.cmap64[t] = r.map32[t] = r.cmap32[t] = r.map16[t] = MapView{};
        }
    } undo{r, need};
    // one upload: map pointers, charge map pointers, maps to pack, type numbers
    const size_t nt = need.size();
    std::vector<GridPack> packs;
    if (packed)
        for (int t : need) {
            packs.push_back({r.map64[t].as<double>(), r.map32[t].as<float4>(), r.map16[t].as<uint4>()});
            if (charged) packs.push_back({r.cmap64[t].as<double>(), r.cmap32[t].as<float4>(), nullptr});
        }
    const size_t at_packs = 2 * nt * sizeof(double*), at_types = at_packs + packs.size() * sizeof(GridPack);
    std::vector<char> args(at_types + nt * sizeof(int));
    std::memcpy(args.data(), maps.data(), nt * sizeof(double*));
    std::memcpy(args.data() + nt * sizeof(double*), cmaps.data(), nt * sizeof(double*));
    if (!packs.empty()) std::memcpy(args.data() + at_packs, packs.data(), packs.size() * sizeof(GridPack));
    std::memcpy(args.data() + at_types, need.data(), nt * sizeof(int));
    DevBuf dargs(e), dtab(e);
    dargs.upload(args.data(), args.size(), e->stream);
    double** dmaps = dargs.as<double*>();
    const int* dtypes = reinterpret_cast<const int*>(dargs.as<char>() + at_types);
    dtab.alloc(std::max<size_t>(1, (size_t)r.slots.count * e->tables.n * grid_lanes((int)nt) * e->tables.nc) * sizeof(double));
    cuda_check(launch_grid_map64(r.geom, r.pop_list.as<CellAtom>(), r.pop_charge.as<double>(), r.pop_start.as<int>(),
                                 e->tables, dtypes, (int)nt, r.slots, dtab.as<double>(), dmaps, dmaps + nt,
                                 r.ugrid.as<double>(), r.ug, r.ug_slope, e->num_sms, e->stream),
               "grid maps");
    if (packed)
        cuda_check(launch_grid_pack(r.geom, reinterpret_cast<const GridPack*>(dargs.as<char>() + at_packs),
                                    (int)packs.size(), e->stream),
                   "pack maps");
    cuda_check(cudaStreamSynchronize(e->stream), "grid maps");
    r.map_mem.push_back(std::move(mem));
    undo.done = true;
    for (int t : need) r.built[t] = true;
    refresh_header(e, r);
}

}  // namespace sg

extern "C" {

int sg_set_receptor(sg_engine* e, int rid, const sg_receptor_desc* r, const sg_grid_dims* gd) {
    return guarded(e, [&] {
        require(rid >= 0 && rid < SG_MAX_RECEPTORS, "receptor id out of range");
        require(r && gd && r->num_atoms >= 0, "receptor: bad arguments");
        require(r->num_atoms == 0 || (r->coords && r->type && r->charge), "receptor: null arrays");
        require(e->has_tables, "set tables before the receptor");
        for (int i = 0; i < 3; i++) {
            require(gd->n[i] >= 1 && gd->n[i] <= 4096, "box: n must be in [1, 4096]");
            require(gd->end[i] > gd->begin[i], "box: end must exceed begin");
        }
        for (int i = 0; i < r->num_atoms; i++) require(std::isfinite(r->coords[3 * i]) && std::isfinite(r->coords[3 * i + 1]) &&
                                                           std::isfinite(r->coords[3 * i + 2]), "receptor: non-finite coordinate");
        RecState& s = e->rec[rid];
        s.set = s.cells = false;  // (no receptor in this place, should a step fail)
        drop_maps(e, s);
        s.ugrid.reset();  // a new receptor starts without a user grid
        s.ug = DGeom{};
        s.gd = *gd;
        s.geom = make_geom(*gd);
        s.natoms = r->num_atoms;
        std::vector<int> types(r->type, r->type + r->num_atoms);
        for (int& t : types) if (t < 0 || t > kNumTypes) t = kNumTypes;
        s.slots = GridSlots{};
        for (int t = 0; t < kNumTypes; t++)
            if (!is_h(t) && std::find(types.begin(), types.end(), t) != types.end()) {
                s.slots.of[t] = (short)s.slots.count;
                s.slots.type[s.slots.count++] = (short)t;
            }
        s.xyz.upload(r->coords, sizeof(double) * 3 * std::max(1, r->num_atoms), e->stream);
        s.type.upload(types.data(), sizeof(int) * std::max<size_t>(1, types.size()), e->stream);
        s.charge.upload(r->charge, sizeof(double) * std::max(1, r->num_atoms), e->stream);
        build_receptor_cells(e, s);
        s.set = true;
    });
}

int sg_build_grids(sg_engine* e, int rid, const int* types, int ntypes) {
    return guarded(e, [&] {
        require(ntypes >= 0 && (ntypes == 0 || types), "build_grids: bad type list");
        RecState& r = receptor_for(e, rid);
        ensure_maps(e, r, types, ntypes);
    });
}

int sg_get_grid(sg_engine* e, int rid, int type, double* data, double* chargedata) {
    return guarded(e, [&] {
        RecState& r = receptor_for(e, rid);
        require(type >= 0 && type < kNumTypes && r.built[type], "grid map not built");
        require(data != nullptr, "null output");
        cuda_check(cudaMemcpy(data, r.map64[type].p, r.map64[type].bytes, cudaMemcpyDeviceToHost), "get grid");
        if (chargedata && r.cmap64[type].p)
            cuda_check(cudaMemcpy(chargedata, r.cmap64[type].p, r.cmap64[type].bytes, cudaMemcpyDeviceToHost), "get grid");
    });
}

int sg_set_user_grid(sg_engine* e, int rid, const sg_grid_dims* gd, const double* data, double cache_slope) {
    return guarded(e, [&] {
        RecState& r = receptor_for(e, rid);
        auto without = [&] {
            r.ugrid.reset();
            r.ug = DGeom{};
            drop_maps(e, r);
            refresh_header(e, r);
        };
        if (gd && data) {
            for (int i = 0; i < 3; i++) {
                require(gd->n[i] >= 1 && gd->n[i] <= 4096, "user grid: n must be in [1, 4096]");
                require(gd->end[i] > gd->begin[i], "user grid: end must exceed begin");
            }
            require(std::isfinite(cache_slope), "user grid: non-finite slope");
            const size_t n = (size_t)(gd->n[0] + 1) * (gd->n[1] + 1) * (gd->n[2] + 1);
            for (size_t k = 0; k < n; k++) require(std::isfinite(data[k]), "user grid: non-finite value");
            try {
                r.ugrid.upload(data, n * sizeof(double), e->stream);
            } catch (...) {  // the old grid's memory is gone
                without();
                throw;
            }
            r.ug = make_geom(*gd);
            r.ug_slope = cache_slope;
            drop_maps(e, r);
            refresh_header(e, r);
        } else {
            without();
        }
    });
}

int sg_drop_receptor(sg_engine* e, int rid) {
    return guarded(e, [&] {
        require(rid >= 0 && rid < SG_MAX_RECEPTORS, "receptor id out of range");
        RecState& s = e->rec[rid];
        s.clear_maps();
        free_dropped_of(s);
        s.pop_start.reset(); s.pop_list.reset(); s.pop_charge.reset();
        s.full_start.reset(); s.full_list.reset(); s.full_charge.reset();
        s.xyz.reset(); s.type.reset(); s.charge.reset(); s.dhdr.reset(); s.ugrid.reset();
        s.set = s.cells = false;
    });
}

}  // extern "C"

// ---- models -------------------------------------------------------------------------------------------
namespace sg {

// Validates one model descriptor on the host so that no device index can
// leave its array, then appends its packed arrays.
// Mixed-precision pair schedule: chunks of 32 slots in which no atom is
// the first atom of two pairs and none is the second atom of two pairs, so
// one warp adds a chunk's forces without atomics (first atoms, then second
// atoms).  A pair may be stored either way round: swapping the atoms toggles
// the charge-role bit.  Within each quarter of a chunk (the 8 lanes that one
// 16-byte shared-memory access serves at a time) the first atoms are
// distinct modulo 8 and so are the second atoms, so the per-atom float4
// loads and stores of a quarter hit 8 different bank groups.  pair_tp[k]:
// type-pair index | (1 << 30) when the pair's first type is the larger.
// Returns false (no schedule) for models of more than 255 atoms.
static bool pack_pair_chunks(const sg_model_desc& d, const std::vector<int>& pair_tp, std::vector<uint32_t>& out) {
    const int N = d.num_atoms, P = d.num_pairs;
    out.clear();
    if (N > 255) return false;  // 8-bit atom indices (inflex atoms take part in pairs too)
    // Chunk c's atoms as bit c of per-atom words, so that a pair meets only the
    // chunks with room for it; its quarters' bank groups as one bit per (quarter,
    // group), a full quarter as all of them.
    struct Chunk {
        uint32_t abank = 0, bbank = 0, slot[32];
        int fill[4] = {};
    };
    std::vector<Chunk> chunks;
    size_t words = 0;
    std::vector<uint64_t> first_in, second_in;  // [word][atom]
    for (int k = 0; k < P; k++) {
        const int u = d.pairs[2 * k], v = d.pairs[2 * k + 1];
        require(u >= 0 && v >= 0 && u < N && v < N && u != v, "model: pair atoms must be distinct atoms");
        require((pair_tp[k] & 0x1ff) < (int)kSlotPairMask, "model: type pair index out of range");
        const uint32_t base = ((uint32_t)(pair_tp[k] & 0x1ff) << 16) | ((pair_tp[k] >> 30) & 1 ? kSlotSwap : 0) |
                              (k >= d.num_other_pairs ? kSlotIntra : 0);
        auto place = [&](size_t c, int o) {
            const int a = o ? v : u, b = o ? u : v;
            Chunk& ch = chunks[c];
            const uint32_t busy = ((ch.abank >> (a & 7)) | (ch.bbank >> (b & 7))) & 0x01010101u;
            if (busy == 0x01010101u) return false;
            const int q = __builtin_ctz(~busy & 0x01010101u) >> 3;
            ch.abank |= 1u << (8 * q + (a & 7));
            ch.bbank |= 1u << (8 * q + (b & 7));
            ch.slot[8 * q + ch.fill[q]++] = (o ? base ^ kSlotSwap : base) | a | (b << 8);
            if (ch.fill[q] == 8) ch.abank |= 0xffu << (8 * q);
            first_in[c / 64 * N + a] |= 1ull << (c & 63);
            second_in[c / 64 * N + b] |= 1ull << (c & 63);
            return true;
        };
        bool placed = false;
        for (size_t w = 0; w < words && !placed; w++) {
            const uint64_t there = chunks.size() - 64 * w >= 64 ? ~0ull : (1ull << (chunks.size() - 64 * w)) - 1;
            const uint64_t as_is = there & ~(first_in[w * N + u] | second_in[w * N + v]),
                           turned = there & ~(first_in[w * N + v] | second_in[w * N + u]);
            for (uint64_t m = as_is | turned; m && !placed; m &= m - 1) {
                const int bit = __builtin_ctzll(m);
                placed = ((as_is >> bit) & 1 && place(64 * w + bit, 0)) || ((turned >> bit) & 1 && place(64 * w + bit, 1));
            }
        }
        if (!placed) {
            chunks.emplace_back();
            for (uint32_t& x : chunks.back().slot) x = kSlotEmpty;
            if (chunks.size() > 64 * words) {
                words++;
                first_in.resize(words * N, 0);
                second_in.resize(words * N, 0);
            }
            place(chunks.size() - 1, 0);
        }
    }
    out.reserve(32 * chunks.size());
    for (const Chunk& ch : chunks) out.insert(out.end(), ch.slot, ch.slot + 32);
    return true;
}

static void pack_one(const sg_model_desc& d, PackFor what, std::vector<int>& I, std::vector<double>& D, std::vector<float>& Fl,
                     std::vector<size_t>& ioff, std::vector<size_t>& doff, std::vector<size_t>& foff, DModel& hm) {
    const int N = d.num_atoms, M = d.num_movable, F = d.num_frames, P = d.num_pairs;
    const bool mixed = what != kPackPlain;
    require(N > 0 && N <= 4096 && M > 0 && M <= N, "model: atom counts out of range");
    require(F > 0 && F <= 1024 && d.num_ligands >= 0 && d.num_flex >= 0 && d.num_ligands + d.num_flex > 0,
            "model: frame / ligand counts out of range");
    require(d.num_ligands <= 30, "model: at most 30 ligands per model");
    require(P >= 0 && P <= 200000 && d.num_other_pairs >= 0 && d.num_other_pairs <= P, "model: pair counts out of range");
    require(d.conf_size > 0 && d.conf_size <= 4096 && d.dof > 0 && d.dof <= 1024, "model: conf/dof sizes out of range");
    require(d.atom_type && d.atom_charge && d.atom_local && d.atom_lab && d.frame_kind && d.frame_parent &&
                d.frame_begin && d.frame_end && d.frame_conf && d.frame_dof && d.frame_origin && d.frame_axis &&
                d.frame_init_origin && (P == 0 || d.pairs) && (d.num_ligands == 0 || (d.lig_pair_end &&
                d.ligand_atom_begin && d.ligand_atom_end && d.ligand_root)),
            "model: null arrays");
    // frames
    std::vector<int> depth(F, 0), atom_frame(N, -1);
    int nlevels = 1, nlig_roots = 0, nflex_roots = 0;
    for (int f = 0; f < F; f++) {
        const int k = d.frame_kind[f], p = d.frame_parent[f];
        require(k >= 0 && k <= 2, "model: bad frame kind");
        require((k == SG_FRAME_SEGMENT) == (p >= 0), "model: only segments have parents");
        require(p < f, "model: frames must be in depth-first order");
        depth[f] = p < 0 ? 0 : depth[p] + 1;
        nlevels = std::max(nlevels, depth[f] + 1);
        require(d.frame_begin[f] >= 0 && d.frame_begin[f] <= d.frame_end[f] && d.frame_end[f] <= M,
                "model: frame atom range out of range");
        for (int i = d.frame_begin[f]; i < d.frame_end[f]; i++) {
            require(atom_frame[i] < 0, "model: frames overlap");
            atom_frame[i] = f;
        }
        if (k == SG_FRAME_RIGID) {
            require(d.frame_conf[f] >= 0 && d.frame_conf[f] + 7 <= d.conf_size && d.frame_dof[f] >= 0 &&
                        d.frame_dof[f] + 6 <= d.dof, "model: rigid conf/dof offsets out of range");
            nlig_roots++;
        } else {
            require(d.frame_conf[f] >= 0 && d.frame_conf[f] < d.conf_size && d.frame_dof[f] >= 0 && d.frame_dof[f] < d.dof,
                    "model: torsion conf/dof offsets out of range");
            if (k == SG_FRAME_FIRST_SEGMENT) nflex_roots++;
        }
        for (int j = 0; j < 3; j++)
            require(std::isfinite(d.frame_origin[3 * f + j]) && std::isfinite(d.frame_axis[3 * f + j]) &&
                        std::isfinite(d.frame_init_origin[3 * f + j]), "model: non-finite frame data");
    }
    require(nlig_roots == d.num_ligands && nflex_roots == d.num_flex, "model: root counts disagree with ligands/flex");
    for (int i = 0; i < M; i++) require(atom_frame[i] >= 0, "model: a movable atom belongs to no frame");
    for (int i = 0; i < N; i++) {
        require(d.atom_type[i] >= 0 && d.atom_type[i] <= kNumTypes, "model: atom type out of range");
        for (int j = 0; j < 3; j++)
            require(std::isfinite(d.atom_local[3 * i + j]) && std::isfinite(d.atom_lab[3 * i + j]), "model: non-finite atom data");
    }
    for (int l = 0; l < d.num_ligands; l++) {
        require(d.ligand_root[l] >= 0 && d.ligand_root[l] < F && d.frame_kind[d.ligand_root[l]] == SG_FRAME_RIGID,
                "model: ligand root is not a rigid frame");
        require(d.ligand_atom_begin[l] >= 0 && d.ligand_atom_begin[l] <= d.ligand_atom_end[l] && d.ligand_atom_end[l] <= M,
                "model: ligand atom range out of range");
        const int prev = l == 0 ? d.num_other_pairs : d.lig_pair_end[l - 1];
        require(d.lig_pair_end[l] >= prev && d.lig_pair_end[l] <= P, "model: ligand pair ranges out of order");
    }
    require(d.num_ligands == 0 || d.lig_pair_end[d.num_ligands - 1] == P, "model: pairs not covered by ligand ranges");
    if (d.num_ligands == 0) require(d.num_other_pairs == P, "model: pairs not covered");
    // levels, children
    std::vector<int> level_start(nlevels + 1, 0), level_frames;
    for (int lv = 0; lv < nlevels; lv++) {
        level_start[lv] = (int)level_frames.size();
        for (int f = 0; f < F; f++) if (depth[f] == lv) level_frames.push_back(f);
    }
    level_start[nlevels] = (int)level_frames.size();
    std::vector<int> child_start(F + 1, 0), child_list;
    for (int f = 0; f < F; f++) {
        child_start[f] = (int)child_list.size();
        for (int c = f + 1; c < F; c++) if (d.frame_parent[c] == f) child_list.push_back(c);
    }
    child_start[F] = (int)child_list.size();
    // pairs, groups, per-atom ordered pair lists
    std::vector<int> group(P, 0), pair_tp(P, 0);
    for (int k = 0; k < P; k++) {
        const int a = d.pairs[2 * k], b = d.pairs[2 * k + 1];
        require(a >= 0 && a < N && b >= 0 && b < N && a != b, "model: pair atom out of range");
        const int ta = d.atom_type[a], tb = d.atom_type[b];
        require(ta < kNumTypes && tb < kNumTypes, "model: a pair atom has no type");
        pair_tp[k] = (ta <= tb ? tri_index(ta, tb) : tri_index(tb, ta)) | (ta > tb ? (1 << 30) : 0);
        if (k >= d.num_other_pairs)
            for (int l = 0; l < d.num_ligands; l++)
                if (k < d.lig_pair_end[l]) { group[k] = l + 1; break; }
    }
    std::vector<std::vector<int>> lists(M);
    for (int k = 0; k < P; k++) {
        const int a = d.pairs[2 * k], b = d.pairs[2 * k + 1];
        if (a < M) lists[a].push_back(k << 1);
        if (b < M) lists[b].push_back((k << 1) | 1);
    }
    std::vector<int> csr_start(M + 1, 0), csr;
    for (int i = 0; i < M; i++) {
        csr_start[i] = (int)csr.size();
        csr.insert(csr.end(), lists[i].begin(), lists[i].end());
    }
    csr_start[M] = (int)csr.size();
    std::vector<int> heavy;
    for (int i = 0; i < M; i++) if (!is_h(d.atom_type[i])) heavy.push_back(i);
    // conf blocks (ligands, then flexible residues) and their torsions
    std::vector<int> root_of(F);
    for (int f = 0; f < F; f++) root_of[f] = d.frame_parent[f] < 0 ? f : root_of[d.frame_parent[f]];
    std::vector<int> blk_rigid, blk_conf, blk_dof, blk_ntors, tor_conf, tor_dof, tor_frame;
    for (int pass = 0; pass < 2; pass++)
        for (int f = 0; f < F; f++) {
            if (d.frame_parent[f] >= 0) continue;
            const bool rigid = d.frame_kind[f] == SG_FRAME_RIGID;
            if ((pass == 0) != rigid) continue;
            blk_rigid.push_back(rigid);
            blk_conf.push_back(d.frame_conf[f]);
            blk_dof.push_back(d.frame_dof[f]);
            int nt = 0;
            for (int g = 0; g < F; g++)
                if (root_of[g] == f && d.frame_kind[g] != SG_FRAME_RIGID) {
                    const int expect_c = d.frame_conf[f] + (rigid ? 7 : 0) + nt;
                    const int expect_d = d.frame_dof[f] + (rigid ? 6 : 0) + nt;
                    require(d.frame_conf[g] == expect_c && d.frame_dof[g] == expect_d,
                            "model: torsions must follow their block in depth-first order");
                    tor_conf.push_back(d.frame_conf[g]);
                    tor_dof.push_back(d.frame_dof[g]);
                    tor_frame.push_back(g);
                    nt++;
                }
            blk_ntors.push_back(nt);
        }
    // pack
    auto pi = [&](const int* src, size_t n) { ioff.push_back(I.size()); I.insert(I.end(), src, src + n); };
    auto pv = [&](const std::vector<int>& v) { ioff.push_back(I.size()); I.insert(I.end(), v.begin(), v.end()); I.push_back(0); };
    auto pd = [&](const double* src, size_t n) { doff.push_back(D.size()); D.insert(D.end(), src, src + n); };
    ioff.clear();
    doff.clear();
    const size_t i0 = I.size(), d0 = D.size();
    (void)i0; (void)d0;
    pi(d.atom_type, N); pi(d.frame_kind, F); pi(d.frame_parent, F); pi(d.frame_begin, F); pi(d.frame_end, F);
    pi(d.frame_conf, F); pi(d.frame_dof, F);
    pv(atom_frame); pv(level_start); pv(level_frames); pv(child_start); pv(child_list);
    if (I.size() & 1) I.push_back(0);  // pairs are read as int2
    if (P) pi(d.pairs, 2 * (size_t)P); else pv({});
    pv(group); pv(csr_start); pv(csr); pv(heavy);
    std::vector<int> lb(d.ligand_atom_begin, d.ligand_atom_begin + d.num_ligands),
        le(d.ligand_atom_end, d.ligand_atom_end + d.num_ligands), lr(d.ligand_root, d.ligand_root + d.num_ligands),
        lp(d.lig_pair_end, d.lig_pair_end + d.num_ligands);
    pv(lb); pv(le); pv(lr); pv(lp);
    pv(blk_rigid); pv(blk_conf); pv(blk_dof); pv(blk_ntors); pv(tor_conf); pv(tor_dof); pv(tor_frame);
    pv(pair_tp);
    {   // subtree atom ranges: a frame's descendants follow its own atoms
        std::vector<int> sub_end(F);
        for (int f = F - 1; f >= 0; f--) {
            sub_end[f] = d.frame_end[f];
            for (int c = f + 1; c < F; c++)
                if (d.frame_parent[c] == f) sub_end[f] = std::max(sub_end[f], sub_end[c]);
        }
        for (int c = 0; c < F; c++)
            for (int a = d.frame_parent[c]; a >= 0; a = d.frame_parent[a])
                require(d.frame_begin[c] >= d.frame_end[a] && d.frame_end[c] <= sub_end[a],
                        "model: a subtree's atoms must follow its root frame's atoms contiguously");
        pv(sub_end);
    }
    {   // mixed-precision pair schedule (pack_pair_chunks)
        std::vector<uint32_t> slots;
        const bool packable = mixed && pack_pair_chunks(d, pair_tp, slots);
        std::vector<int> ps(slots.begin(), slots.end());
        hm.npchunks = packable ? (int)(slots.size() / 32) : -1;
        pv(ps);
        // the same pairs per movable atom: chunk by chunk, in a chunk the atom's
        // pair as first atom before the one as second
        hm.wstart = nullptr;
        if (what == kPackWide && packable && hm.npchunks <= kWideChunks) {
            std::vector<std::vector<uint16_t>> of(M);
            for (size_t c = 0; c < slots.size(); c += 32)
                for (int role = 0; role < 2; role++)
                    for (size_t k = c; k < c + 32; k++) {
                        if (((slots[k] >> 16) & kSlotPairMask) == kSlotPairMask) continue;
                        const int a = (slots[k] >> (8 * role)) & 0xff;
                        if (a < M) of[a].push_back((uint16_t)(k << 1 | role));
                    }
            std::vector<uint16_t> wlist;
            std::vector<int> wide;
            for (int i = 0; i < M; i++) {
                wide.push_back((int)wlist.size());
                wlist.insert(wlist.end(), of[i].begin(), of[i].end());
            }
            wide.push_back((int)wlist.size());
            wide.resize(M + 1 + (wlist.size() + 1) / 2);
            if (!wlist.empty()) std::memcpy(&wide[M + 1], wlist.data(), wlist.size() * sizeof(uint16_t));
            hm.wstart = reinterpret_cast<const int*>(1);  // placed with the pools
            pv(wide);
        }
    }
    auto pf4 = [&](const double* xyz, const double* w4, size_t n) {
        foff.push_back(Fl.size());
        for (size_t i = 0; i < n; i++) {
            Fl.push_back((float)xyz[3 * i]); Fl.push_back((float)xyz[3 * i + 1]); Fl.push_back((float)xyz[3 * i + 2]);
            Fl.push_back(w4 ? (float)w4[i] : 0.f);
        }
    };
    foff.clear();
    if (mixed) {
        pf4(d.atom_local, d.atom_charge, N); pf4(d.atom_lab, nullptr, N);
        pf4(d.frame_origin, nullptr, F); pf4(d.frame_axis, nullptr, F); pf4(d.frame_init_origin, nullptr, F);
    }
    hm.cost = M + P + 8 * F;
    pd(d.atom_charge, N); pd(d.atom_local, 3 * (size_t)N); pd(d.atom_lab, 3 * (size_t)N);
    pd(d.frame_origin, 3 * (size_t)F); pd(d.frame_axis, 3 * (size_t)F); pd(d.frame_init_origin, 3 * (size_t)F);
    hm.natoms = N; hm.nmov = M; hm.nframes = F; hm.nlig = d.num_ligands; hm.nflex = d.num_flex;
    hm.conf_size = d.conf_size; hm.dof = d.dof; hm.npairs = P; hm.nother = d.num_other_pairs;
    hm.nheavy = (int)heavy.size(); hm.nlevels = nlevels; hm.nblocks = (int)blk_rigid.size();
    hm.ntors = (int)tor_conf.size();
    require(hm.ntors + 6 * d.num_ligands == d.dof, "model: dof disagrees with the torsion count");
}

// The pools of a batch of models, as parts that are packed side by side on the
// host's cores, and each descriptor's offsets into its part.
struct PackedPart {
    std::vector<int> I;
    std::vector<double> D;
    std::vector<float> Fl;
    std::vector<std::vector<size_t>> io, dof, fo;
    size_t i0 = 0, d0 = 0, f0 = 0;  // where the part's pools start in the batch's
    std::exception_ptr error;
};
struct PackedPools {
    std::vector<PackedPart> parts;
    int per_part = 0;
    size_t od = 0, of = 0, om = 0, bytes = 0;  // byte offsets of the doubles, floats and descriptors, and the end
};
constexpr int kPackPart = 16;    // models worth a thread (about 1 ms of packing)
constexpr int kPackThreads = 8;
static void pack_pools(const sg_model_desc* models, int nmodels, PackFor what, PackedPools& P, std::vector<DModel>& host) {
    require(models && nmodels > 0 && nmodels <= (1 << 20), "models: bad array");
    host.assign(nmodels, DModel{});
    const int cores = std::max(1, (int)std::thread::hardware_concurrency());
    const int nparts = std::max(1, std::min({nmodels / kPackPart, kPackThreads, cores}));
    P.per_part = (nmodels + nparts - 1) / nparts;
    P.parts.resize((nmodels + P.per_part - 1) / P.per_part);
    auto work = [&](size_t q) {
        PackedPart& part = P.parts[q];
        const int first = (int)q * P.per_part, n = std::min(P.per_part, nmodels - first);
        try {
            part.io.resize(n);
            part.dof.resize(n);
            part.fo.resize(n);
            for (int k = 0; k < n; k++)
                pack_one(models[first + k], what, part.I, part.D, part.Fl, part.io[k], part.dof[k], part.fo[k],
                         host[first + k]);
            if (part.I.size() & 3) part.I.resize((part.I.size() + 3) & ~(size_t)3);  // the next part starts 16 B aligned
        } catch (...) {
            part.error = std::current_exception();
        }
    };
    std::vector<std::thread> threads;
    threads.reserve(P.parts.size());  // (nothing may throw past a thread that has not been joined)
    for (size_t q = 1; q < P.parts.size(); q++) {
        try {
            threads.emplace_back(work, q);
        } catch (...) {  // no thread or no memory for one
            work(q);
        }
    }
    work(0);
    for (std::thread& t : threads) t.join();
    size_t ni = 0, nd = 0, nf = 0;
    for (PackedPart& part : P.parts) {
        if (part.error) std::rethrow_exception(part.error);
        part.i0 = ni;
        part.d0 = nd;
        part.f0 = nf;
        ni += part.I.size();
        nd += part.D.size();
        nf += part.Fl.size();
    }
    auto r16 = [](size_t b) { return (b + 15) & ~(size_t)15; };
    P.od = r16(ni * sizeof(int));
    P.of = P.od + r16(nd * sizeof(double));
    P.om = P.of + r16(nf * sizeof(float));
    P.bytes = P.om + nmodels * sizeof(DModel);
}
// aims every descriptor's pointers at dev_base and writes the image (pools, then
// descriptors, each 16 B aligned)
static void place_pools(const PackedPools& P, std::vector<DModel>& host, char* dev_base, char* image) {
    for (size_t k = 0; k < host.size(); k++) {
        const PackedPart& part = P.parts[k / P.per_part];
        const size_t m = k % P.per_part;
        const int* ib = reinterpret_cast<const int*>(dev_base) + part.i0;
        const double* db = reinterpret_cast<const double*>(dev_base + P.od) + part.d0;
        const float* fb = reinterpret_cast<const float*>(dev_base + P.of) + part.f0;
        DModel& h = host[k];
        const std::vector<size_t>&io = part.io[m], &dd = part.dof[m], &fo = part.fo[m];
        const int** ip[] = {&h.type, &h.fkind, &h.fparent, &h.fbegin, &h.fend, &h.fconf, &h.fdof, &h.atom_frame,
                            &h.level_start, &h.level_frames, &h.child_start, &h.child_list, &h.pairs, &h.pair_group,
                            &h.csr_start, &h.csr, &h.heavy, &h.lig_begin, &h.lig_end, &h.lig_root, &h.lig_pair_end,
                            &h.blk_rigid, &h.blk_conf, &h.blk_dof, &h.blk_ntors, &h.tor_conf, &h.tor_dof,
                            &h.tor_frame, &h.pair_tp, &h.fsub_end};
        size_t j = 0;
        for (const int** q : ip) *q = ib + io[j++];
        h.pslot = h.npchunks >= 0 ? reinterpret_cast<const uint32_t*>(ib + io[j]) : nullptr;
        if (h.wstart) h.wstart = ib + io[j + 1];
        const float4** fp[] = {&h.local32, &h.lab32, &h.forigin32, &h.faxis32, &h.finit32};
        for (j = 0; j < fo.size(); j++) *fp[j] = reinterpret_cast<const float4*>(fb + fo[j]);
        const double** dp[] = {&h.charge, &h.local, &h.lab, &h.forigin, &h.faxis, &h.finit};
        j = 0;
        for (const double** q : dp) *q = db + dd[j++];
    }
    for (const PackedPart& part : P.parts) {
        std::memcpy(image + part.i0 * sizeof(int), part.I.data(), part.I.size() * sizeof(int));
        std::memcpy(image + P.od + part.d0 * sizeof(double), part.D.data(), part.D.size() * sizeof(double));
        if (!part.Fl.empty())
            std::memcpy(image + P.of + part.f0 * sizeof(float), part.Fl.data(), part.Fl.size() * sizeof(float));
    }
    std::memcpy(image + P.om, host.data(), host.size() * sizeof(DModel));
}

void pack_models(CallIo& io, const sg_model_desc* models, int nmodels, PackFor what, PackedModels& out) {
    PackedPools P;
    pack_pools(models, nmodels, what, P, out.host);
    out.mem.alloc(P.bytes);
    std::unique_ptr<char[]> image(new char[P.bytes]);
    place_pools(P, out.host, out.mem.as<char>(), image.get());
    out.dmodels = reinterpret_cast<DModel*>(out.mem.as<char>() + P.om);
    io.in(out.mem, image.get(), P.bytes);
    out.smem64 = Smem64{};
    for (const DModel& h : out.host) {
        out.smem64.add(h);
        out.max_conf = std::max(out.max_conf, h.conf_size);
        out.max_dof = std::max(out.max_dof, h.dof);
        out.max_heavy = std::max(out.max_heavy, h.nheavy);
        out.max_atoms = std::max(out.max_atoms, h.natoms);
        out.max_pairs = std::max(out.max_pairs, h.npairs);
        out.max_frames = std::max(out.max_frames, h.nframes);
    }
}

// Host image of the packed models for a caller that places them in device
// memory it already owns, with every descriptor pointer aimed at dev_base + its
// offset in the image.
void pack_models_image(const sg_model_desc* models, int nmodels, char* dev_base, ModelImage& img) {
    PackedPools P;
    pack_pools(models, nmodels, kPackMixed, P, img.host);
    img.dmodel_off = P.om;
    img.bytes.assign(P.bytes, 0);
    place_pools(P, img.host, dev_base, img.bytes.data());
}

void ensure_model_maps(sg_engine* e, RecState& r, const sg_model_desc* models, int nmodels) {
    bool seen[kNumTypes] = {};
    std::vector<int> types;
    for (int k = 0; k < nmodels; k++)
        for (int i = 0; i < models[k].num_movable; i++) {
            const int t = models[k].atom_type[i];
            if (t < kNumTypes && !is_h(t) && !seen[t]) {
                seen[t] = true;
                types.push_back(t);
            }
        }
    ensure_maps(e, r, types.data(), (int)types.size());
}

}  // namespace sg

Shape64 sg::plain_shape(sg_engine* e, const PackedModels& pm, long long items, Work64 work) {
    const Shape64 sh = shape64(pm.smem64, items, work, e->num_sms, (size_t)e->max_smem);
    require(sh.smem <= (size_t)e->max_smem, "model too large for the plain path's shared memory");
    return sh;
}

// a call's device array: inputs come through the call's copies, results go back
// the same way
template <typename T>
struct Staged {
    CallIo& io;
    sg_engine* e;
    sg::DevBuf d;
    size_t n = 0;
    Staged(CallIo& io_, sg_engine* e_) : io(io_), e(e_), d(e_) {}
    void make(size_t count, const T* init = nullptr) {
        n = count;
        if (init && n) io.in(d, init, n * sizeof(T));
        else d.alloc(std::max<size_t>(1, n) * sizeof(T));
    }
    T* p() { return d.as<T>(); }
    void zero() {  // for outputs with padding the kernel leaves alone
        sg::cuda_check(cudaMemsetAsync(d.p, 0, std::max<size_t>(1, n) * sizeof(T), e->stream), "zero output");
    }
    void fetch(T* host) { io.out(host, d.p, n * sizeof(T)); }
};

extern "C" {

static int eval_common(sg_engine* e, int rid, const sg_model_desc* m, int nconfs, const double* confs, const double v[3],
                       double slope, double* out_e, double* out_g, double* out_coords, int direct) {
    return guarded(e, [&] {
        require(m && confs && v && out_e && out_g && nconfs > 0 && nconfs <= (1 << 24), "eval: bad arguments");
        require(e->has_tables, "no tables set");
        RecState& r = direct ? direct_receptor(e, rid) : receptor_for(e, rid);
        CallIo io(e);
        PackedModels pm(e);
        pack_models(io, m, 1, !direct && e->precision != SG_PREC_FP64 ? kPackMixed : kPackPlain, pm);
        if (!direct) ensure_model_maps(e, r, m, 1);
        const Shape64 sh = plain_shape(e, pm, nconfs, Work64::eval);
        const DModel& h = pm.host[0];
        Staged<double> dc(io, e), de(io, e), dg(io, e), dx(io, e);
        dc.make((size_t)nconfs * h.conf_size, confs);
        de.make(nconfs);
        dg.make((size_t)nconfs * h.dof);
        if (out_coords) dx.make((size_t)nconfs * h.nmov * 3);
        if (!direct && e->precision != SG_PREC_FP64) {  // the mixed-precision evaluation
            require(h.npchunks >= 0, "mixed-precision path: at most 255 atoms per model");
            const size_t ws = (ws32_bytes(h) + 15) & ~(size_t)15;
            const size_t stage =
                (size_t)stage32_bytes(h.natoms, h.nframes, h.nheavy, h.npchunks, h.nlig, h.nblocks, h.ntors);
            require(stage + (size_t)std::max(1, e->tpc / 32) * ws <= (size_t)e->max_smem,
                    "model too large for the mixed-precision path's shared memory");
            cuda_check(launch_eval32(pm.dmodels, stage, ws, tables32(e), maps32(e, r), nconfs, dc.p(), v, slope,
                                     de.p(), dg.p(), out_coords ? dx.p() : nullptr, std::max(1, e->tpc / 32), e->num_sms,
                                     (size_t)e->max_smem, e->stream),
                       "eval launch");
            de.fetch(out_e);
            dg.fetch(out_g);
            if (out_coords) dx.fetch(out_coords);
            io.finish();
            return;
        }
        cuda_check(launch_eval64(pm.dmodels, sh, e->num_sms, e->tables, r.dhdr.as<DReceptor>(), nconfs, dc.p(), v,
                                 slope, direct, de.p(), dg.p(), out_coords ? dx.p() : nullptr, e->d_err.as<int>(), e->stream),
                   "eval launch");
        de.fetch(out_e);
        dg.fetch(out_g);
        if (out_coords) dx.fetch(out_coords);
        io.finish();
    });
}

int sg_eval(sg_engine* e, int rid, const sg_model_desc* m, int nconfs, const double* confs, const double v[3],
            double slope, double* out_e, double* out_g, double* out_coords) {
    return eval_common(e, rid, m, nconfs, confs, v, slope, out_e, out_g, out_coords, 0);
}

int sg_eval_direct(sg_engine* e, int rid, const sg_model_desc* m, int nconfs, const double* confs, const double v[3],
                   double slope, double* out_e, double* out_g) {
    return eval_common(e, rid, m, nconfs, confs, v, slope, out_e, out_g, nullptr, 1);
}

int sg_probe_gather(sg_engine* e, uint64_t working_set_bytes, int bytes_per_lookup, double* out_gbs) {
    return guarded(e, [&] {
        require(out_gbs && (bytes_per_lookup == 16 || bytes_per_lookup == 32) && working_set_bytes >= (1u << 20) &&
                    working_set_bytes <= (64ull << 30),
                "probe_gather: bad arguments");
        cuda_check(gather_probe(working_set_bytes, bytes_per_lookup, e->num_sms, out_gbs, e->stream), "gather probe");
    });
}

int sg_bfgs(sg_engine* e, int rid, const sg_model_desc* m, int nconfs, double* confs, const double v[3], double slope,
            int maxiters, int accurate_line, int early_term, double* out_e) {
    return guarded(e, [&] {
        require(m && confs && v && out_e && nconfs > 0 && nconfs <= (1 << 24) && maxiters >= 0, "bfgs: bad arguments");
        RecState& r = receptor_for(e, rid);
        CallIo io(e);
        PackedModels pm(e);
        pack_models(io, m, 1, e->precision != SG_PREC_FP64 ? kPackWide : kPackPlain, pm);
        ensure_model_maps(e, r, m, 1);
        const DModel& h = pm.host[0];
        Staged<double> dc(io, e), de(io, e);
        dc.make((size_t)nconfs * h.conf_size, confs);
        de.make(nconfs);
        if (e->precision != SG_PREC_FP64) {  // the batched search's mixed-precision BFGS
            require(h.npchunks >= 0, "mixed-precision path: at most 255 atoms per model");
            const size_t ws = (ws32_bytes(h) + 15) & ~(size_t)15;
            const size_t stage =
                (size_t)stage32_bytes(h.natoms, h.nframes, h.nheavy, h.npchunks, h.nlig, h.nblocks, h.ntors);
            require(stage + (size_t)std::max(1, e->tpc / 32) * ws <= (size_t)e->max_smem,
                    "model too large for the mixed-precision path's shared memory");
            const size_t wide = h.wstart ? (size_t)wide32_layout(h.npchunks, h.npairs, h.nmov).total : 0;
            cuda_check(launch_bfgs32(pm.dmodels, stage, ws, wide, h.npairs, tables32(e), maps32(e, r), nconfs, dc.p(), v, slope,
                                     maxiters, accurate_line, early_term, de.p(), std::max(1, e->tpc / 32), e->num_sms,
                                     (size_t)e->max_smem, e->stream),
                       "bfgs launch");
            dc.fetch(confs);
            de.fetch(out_e);
            io.finish();
            return;
        }
        const Shape64 sh = plain_shape(e, pm, nconfs, Work64::bfgs);
        cuda_check(launch_bfgs64(pm.dmodels, sh, e->tables, r.dhdr.as<DReceptor>(), nconfs, dc.p(), v,
                                 slope, maxiters, accurate_line, early_term, de.p(), e->d_err.as<int>(), e->stream),
                   "bfgs launch");
        dc.fetch(confs);
        de.fetch(out_e);
        io.finish();
    });
}

int sg_dock(sg_engine* e, int rid, const sg_model_desc* models, int nmodels, const sg_chain_input* chains, int nchains,
            const sg_mc_params* p, sg_chain_result* out) {
    return guarded(e, [&] {
        require(chains && p && out && nchains > 0 && nchains <= (1 << 22), "dock: bad arguments");
        require(p->num_saved_mins >= 1 && p->num_saved_mins <= 1024 && p->maxiters >= 0 && p->temperature > 0,
                "dock: bad search parameters");
        RecState& r = receptor_for(e, rid);
        CallIo io(e);
        PackedModels pm(e);
        pack_models(io, models, nmodels, kPackPlain, pm);
        ensure_model_maps(e, r, models, nmodels);
        const Shape64 sh = plain_shape(e, pm, nchains, Work64::chain);
        const int S = p->num_saved_mins;
        // per-chain inputs and result storage (one device allocation each)
        std::vector<double> conf0;
        std::vector<uint32_t> mt((size_t)nchains * 625);
        std::vector<size_t> conf_off(nchains), cres_off(nchains), xres_off(nchains);
        size_t nconf_res = 0, nxyz_res = 0;
        for (int k = 0; k < nchains; k++) {
            const sg_chain_input& c = chains[k];
            require(c.model >= 0 && c.model < nmodels && c.conf && c.mt && c.maxiters >= 0, "dock: bad chain input");
            require(c.mt[624] <= 624, "dock: mt19937 index out of range");
            const DModel& h = pm.host[c.model];
            conf_off[k] = conf0.size();
            conf0.insert(conf0.end(), c.conf, c.conf + h.conf_size);
            std::memcpy(&mt[(size_t)k * 625], c.mt, 625 * sizeof(uint32_t));
            cres_off[k] = nconf_res;
            nconf_res += (size_t)S * h.conf_size;
            xres_off[k] = nxyz_res;
            nxyz_res += (size_t)S * h.nheavy * 3;
            require(out[k].e && out[k].conf && out[k].coords, "dock: null result arrays");
        }
        Staged<double> d_conf0(io, e), d_e(io, e), d_conf(io, e), d_xyz(io, e), d_hist(io, e);
        Staged<uint32_t> d_mt(io, e);
        Staged<unsigned long long> d_histw(io, e);
        Staged<int> d_order(io, e), d_count(io, e);
        Staged<unsigned long long> d_evals(io, e);
        // QuickVina 2 histories (MCParams::visited), one block per chain whose dof fits
        std::vector<size_t> hist_off(nchains, SIZE_MAX), histw_off(nchains, SIZE_MAX);
        size_t nhist = 0, nhistw = 0;
        if (p->visited)
            for (int k = 0; k < nchains; k++) {
                const int n = pm.host[chains[k].model].dof;
                if (n > kHistMaxN) continue;
                hist_off[k] = nhist;
                histw_off[k] = nhistw;
                nhist += hist64_doubles(n);
                nhistw += hist64_words(n);
            }
        if (nhist) {
            d_hist.make(nhist);
            d_histw.make(nhistw);
            d_histw.zero();  // empty histories
        }
        d_conf0.make(conf0.size(), conf0.data());
        d_mt.make(mt.size(), mt.data());
        d_e.make((size_t)nchains * S);
        d_conf.make(nconf_res);
        d_xyz.make(nxyz_res);
        d_order.make((size_t)nchains * S);
        d_count.make(nchains);
        d_evals.make(nchains);
        std::vector<Chain64> hc(nchains);
        for (int k = 0; k < nchains; k++) {
            hc[k].model = chains[k].model;
            hc[k].steps = chains[k].num_steps;
            hc[k].maxiters = chains[k].maxiters > 0 ? chains[k].maxiters : p->maxiters;
            hc[k].conf0 = d_conf0.p() + conf_off[k];
            hc[k].mt = d_mt.p() + (size_t)k * 625;
            hc[k].out_e = d_e.p() + (size_t)k * S;
            hc[k].out_conf = d_conf.p() + cres_off[k];
            hc[k].out_coords = d_xyz.p() + xres_off[k];
            hc[k].out_order = d_order.p() + (size_t)k * S;
            hc[k].out_count = d_count.p() + k;
            hc[k].evals = d_evals.p() + k;
            hc[k].hist = hist_off[k] == SIZE_MAX ? nullptr : d_hist.p() + hist_off[k];
            hc[k].hist_words = histw_off[k] == SIZE_MAX ? nullptr : d_histw.p() + histw_off[k];
        }
        DevBuf d_chains(e);
        io.in(d_chains, hc.data(), hc.size() * sizeof(Chain64));
        MCParams64 P;
        P.num_steps = p->num_steps;
        P.temperature = p->temperature;
        P.amplitude = p->mutation_amplitude;
        P.min_rmsd = p->min_rmsd;
        P.num_saved = S;
        for (int i = 0; i < 3; i++) { P.hunt[i] = p->hunt_cap[i]; P.auth[i] = p->authentic_v[i]; }
        P.maxiters = p->maxiters;
        P.accurate_line = p->accurate_line;
        P.early_term = p->early_term;
        P.slope = p->cache_slope;
        cuda_check(launch_mc64(pm.dmodels, sh, e->tables, r.dhdr.as<DReceptor>(),
                               d_chains.as<Chain64>(), nchains, P, nhist > 0, e->d_err.as<int>(), e->stream),
                   "dock launch");
        std::vector<double> he((size_t)nchains * S), hconf(nconf_res), hxyz(nxyz_res);
        std::vector<int> horder((size_t)nchains * S), hcount(nchains);
        std::vector<unsigned long long> hev(nchains);
        d_e.fetch(he.data());
        d_conf.fetch(hconf.data());
        d_xyz.fetch(hxyz.data());
        d_order.fetch(horder.data());
        d_count.fetch(hcount.data());
        d_evals.fetch(hev.data());
        io.finish();
        for (int k = 0; k < nchains; k++) {
            const DModel& h = pm.host[chains[k].model];
            const int cnt = std::min(std::max(hcount[k], 0), S);
            out[k].count = cnt;
            out[k].evals = hev[k];
            for (int j = 0; j < cnt; j++) {
                const int slot = horder[(size_t)k * S + j];
                require(slot >= 0 && slot < S, "dock: corrupt result order");
                out[k].e[j] = he[(size_t)k * S + slot];
                std::memcpy(out[k].conf + (size_t)j * h.conf_size, &hconf[cres_off[k] + (size_t)slot * h.conf_size],
                            h.conf_size * sizeof(double));
                std::memcpy(out[k].coords + (size_t)j * h.nheavy * 3, &hxyz[xres_off[k] + (size_t)slot * h.nheavy * 3],
                            (size_t)h.nheavy * 3 * sizeof(double));
            }
        }
    });
}

int sg_refine(sg_engine* e, int rid, const sg_model_desc* models, int nmodels, const int* pose_model, int nposes,
              double* confs, const double cap[3], int maxiters, int accurate_line, int early_term, double* out_e,
              double* out_coords) {
    return guarded(e, [&] {
        require(pose_model && confs && cap && out_e && nposes > 0 && maxiters >= 0, "refine: bad arguments");
        RecState& r = direct_receptor(e, rid);
        CallIo io(e);
        PackedModels pm(e);
        pack_models(io, models, nmodels, kPackPlain, pm);
        const Shape64 sh = plain_shape(e, pm, nposes, Work64::refine);
        for (int k = 0; k < nposes; k++) require(pose_model[k] >= 0 && pose_model[k] < nmodels, "refine: bad pose model");
        const int cs = pm.max_conf, hs = pm.max_heavy;
        Staged<double> dc(io, e), de(io, e), dx(io, e);
        Staged<int> dpm(io, e);
        dc.make((size_t)nposes * cs, confs);
        de.make(nposes);
        dx.make((size_t)nposes * hs * 3);
        dx.zero();  // atoms past a pose's heavy count stay 0
        dpm.make(nposes, pose_model);
        cuda_check(launch_refine64(pm.dmodels, sh, e->tables, r.dhdr.as<DReceptor>(), dpm.p(), nposes,
                                   dc.p(), cs, cap, maxiters, nullptr, nullptr, accurate_line, early_term, de.p(), dx.p(), hs,
                                   e->d_err.as<int>(), e->stream),
                   "refine launch");
        dc.fetch(confs);
        de.fetch(out_e);
        if (out_coords) dx.fetch(out_coords);
        io.finish();
    });
}

int sg_pair_schedule(const sg_model_desc* m, uint32_t* out, int cap, int* nchunks) {
    if (!m || !nchunks || cap < 0 || (cap > 0 && !out)) return SG_ERR_ARG;
    try {
        const int N = m->num_atoms, P = m->num_pairs;
        if (N <= 0 || P < 0 || (P > 0 && (!m->pairs || !m->atom_type))) return SG_ERR_ARG;
        std::vector<int> pair_tp(P);
        for (int k = 0; k < P; k++) {
            const int a = m->pairs[2 * k], b = m->pairs[2 * k + 1];
            if (a < 0 || a >= N || b < 0 || b >= N || a == b) return SG_ERR_ARG;
            const int ta = m->atom_type[a], tb = m->atom_type[b];
            if (ta < 0 || tb < 0 || ta >= kNumTypes || tb >= kNumTypes) return SG_ERR_ARG;
            pair_tp[k] = (ta <= tb ? tri_index(ta, tb) : tri_index(tb, ta)) | (ta > tb ? (1 << 30) : 0);
        }
        std::vector<uint32_t> slots;
        if (!pack_pair_chunks(*m, pair_tp, slots)) return SG_ERR_ARG;
        *nchunks = (int)(slots.size() / 32);
        if ((size_t)cap >= slots.size()) std::copy(slots.begin(), slots.end(), out);
        return SG_OK;
    } catch (...) {
        return SG_ERR_ARG;
    }
}

int sg_score(sg_engine* e, int rid, const sg_model_desc* models, int nmodels, const int* pose_model, int nposes,
             const double* confs, int conf_stride, const double v[3], double slope, double* out_e, double* out_intra,
             double* out_coords, int coord_stride) {
    return guarded(e, [&] {
        require(pose_model && confs && v && out_e && out_intra && nposes > 0 && nposes <= (1 << 24),
                "score: bad arguments");
        require(e->has_tables, "no tables set");
        RecState& r = direct_receptor(e, rid);
        CallIo io(e);
        PackedModels pm(e);
        pack_models(io, models, nmodels, kPackPlain, pm);
        const Shape64 sh = plain_shape(e, pm, nposes, Work64::eval);
        require(conf_stride >= pm.max_conf && (!out_coords || coord_stride >= pm.max_heavy), "score: strides too small");
        for (int k = 0; k < nposes; k++) require(pose_model[k] >= 0 && pose_model[k] < nmodels, "score: bad pose model");
        Staged<double> dc(io, e), de(io, e), di(io, e), dx(io, e);
        Staged<int> dpm(io, e);
        dc.make((size_t)nposes * conf_stride, confs);
        de.make(nposes);
        di.make(nposes);
        if (out_coords) {
            dx.make((size_t)nposes * coord_stride * 3);
            dx.zero();  // atoms past a pose's heavy count stay 0
        }
        dpm.make(nposes, pose_model);
        cuda_check(launch_score64(pm.dmodels, sh, e->tables, r.dhdr.as<DReceptor>(), dpm.p(),
                                  nposes, dc.p(), conf_stride, v, slope, de.p(), di.p(), out_coords ? dx.p() : nullptr,
                                  coord_stride, e->d_err.as<int>(), e->stream),
                   "score launch");
        de.fetch(out_e);
        di.fetch(out_intra);
        if (out_coords) dx.fetch(out_coords);
        io.finish();
    });
}

int sg_minimize(sg_engine* e, int rid, const sg_model_desc* models, int nmodels, const int* pose_model, int nposes,
                double* confs, int conf_stride, const double* boxes, const double cap[3], const int* maxiters,
                int accurate_line, int early_term, double* out_e, double* out_coords, int coord_stride) {
    return guarded(e, [&] {
        require(pose_model && confs && cap && maxiters && out_e && nposes > 0, "minimize: bad arguments");
        RecState& r = direct_receptor(e, rid);
        CallIo io(e);
        PackedModels pm(e);
        pack_models(io, models, nmodels, kPackPlain, pm);
        const Shape64 sh = plain_shape(e, pm, nposes, Work64::refine);
        require(conf_stride >= pm.max_conf && coord_stride >= pm.max_heavy, "minimize: strides too small");
        for (int k = 0; k < nposes; k++) {
            require(pose_model[k] >= 0 && pose_model[k] < nmodels && maxiters[k] >= 0, "minimize: bad pose");
            if (boxes)  // a pose's box must lie inside the receptor's, where its cell lists are
                for (int d = 0; d < 3; d++)
                    require(boxes[6 * k + d] >= r.gd.begin[d] && boxes[6 * k + 3 + d] <= r.gd.end[d] &&
                                boxes[6 * k + d] <= boxes[6 * k + 3 + d],
                            "minimize: a pose's box must lie inside the receptor's box");
        }
        Staged<double> dc(io, e), de(io, e), dx(io, e), db(io, e);
        Staged<int> dpm(io, e), dmi(io, e);
        dc.make((size_t)nposes * conf_stride, confs);
        de.make(nposes);
        dx.make((size_t)nposes * coord_stride * 3);
        dx.zero();  // atoms past a pose's heavy count stay 0
        dpm.make(nposes, pose_model);
        dmi.make(nposes, maxiters);
        if (boxes) db.make((size_t)nposes * 6, boxes);
        cuda_check(launch_refine64(pm.dmodels, sh, e->tables, r.dhdr.as<DReceptor>(), dpm.p(),
                                   nposes, dc.p(), conf_stride, cap, 0, dmi.p(), boxes ? db.p() : nullptr,
                                   accurate_line, early_term, de.p(), dx.p(), coord_stride, e->d_err.as<int>(),
                                   e->stream),
                   "minimize launch");
        dc.fetch(confs);
        de.fetch(out_e);
        if (out_coords) dx.fetch(out_coords);
        io.finish();
    });
}

}  // extern "C"
