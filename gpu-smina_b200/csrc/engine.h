// Engine state behind the C ABI.
#pragma once
#include <memory>
#include <new>
#include <stdexcept>
#include <string>
#include <utility>
#include <cstdint>
#include <vector>
#include "sg_dev.cuh"

struct sg_engine;

namespace sg {

struct EngineError : std::runtime_error {
    int code;
    EngineError(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

void cuda_check(cudaError_t e, const char* what);

inline void require(bool ok, const std::string& msg) {
    if (!ok) throw EngineError(SG_ERR_ARG, msg);
}

// Owning device memory.  DevBuf(engine) is a call's temporary: it comes from the
// engine's stream-ordered pool and goes back to it on the engine's stream.
// DevBuf() belongs to a receptor or the engine: its own allocation, kept when a
// later one fits it without wasting half.
struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;
    DevBuf() = default;
    explicit DevBuf(sg_engine* e) : pool_of(e) {}
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { reset(); }
    void reset();
    void alloc(size_t n);
    void upload(const void* src, size_t n, cudaStream_t s);
    template <typename T> T* as() const { return reinterpret_cast<T*>(p); }

private:
    sg_engine* pool_of = nullptr;
    size_t cap = 0;
};

// Copies between the caller's memory and the device for one call, in pieces
// through a small ring of pinned memory (PinRing): a piece is copied by the host
// while the one before is in flight.  Inputs go at once; outputs are listed and
// fetched by finish(), after which the caller's arrays are filled.  (Straight
// from and to pageable memory each copy waited for the one before: 20,000
// evaluations of a 13-dof ligand, 4.5 MB both ways, took 2.1 ms a call and take
// 0.68 ms; 2 MB of pinned memory is enough for that, while pinning the whole
// transfer cost a first call 6 ms.)
struct PinRing {
    static constexpr size_t kSlot = size_t(512) << 10;
    static constexpr int kSlots = 4;  // two for inputs, two for outputs
    char* p = nullptr;
    bool pinned = false;  // else, where none could be had, pageable: copies through it then wait
    cudaEvent_t ev[kSlots] = {};
    ~PinRing();
};
class CallIo {
public:
    explicit CallIo(sg_engine* e) : e_(e) {}
    CallIo(const CallIo&) = delete;
    CallIo& operator=(const CallIo&) = delete;
    ~CallIo();
    void in(DevBuf& dst, const void* src, size_t n);   // allocates dst
    void out(void* host, const void* dev, size_t n);   // dev stays as it is until finish()
    void finish();                                     // throws the device's error, if it reported one

private:
    struct Out { void* host; const void* dev; size_t n; };
    struct Piece { void* host; const char* from; size_t n; };
    void need_ring();
    sg_engine* e_;
    std::unique_ptr<PinRing> ring_;
    int in_slot_ = 0;
    size_t in_used_ = 0;
    bool in_sent_[2] = {};
    std::vector<Out> outs_;
    bool busy_ = false;
};
// a ring for the process's next call, so that the first call need not pin one
void warm_pin_ring();
// The device's pool of call temporaries, shared by its engines and destroyed with
// the last of them; it keeps at most kPoolKept bytes between calls.
constexpr size_t kPoolKept = size_t(256) << 20;
cudaMemPool_t pool_acquire(int device);
void pool_release(int device);

// one grid map within its receptor's allocation
struct MapView {
    void* p = nullptr;
    size_t bytes = 0;
    template <typename T> T* as() const { return reinterpret_cast<T*>(p); }
};

DGeom make_geom(const sg_grid_dims& gd);

// one resident receptor with its box, cell lists and maps
struct RecState {
    bool set = false;
    sg_grid_dims gd{};
    DGeom geom{};
    int natoms = 0;
    DevBuf xyz, type, charge, pop_start, pop_list, pop_charge, full_start, full_list, full_charge;
    // the maps of one build share an allocation (void maps' allocations wait for the
    // next build in this place: drop_maps)
    std::vector<std::unique_ptr<DevBuf>> map_mem;
    MapView map64[kNumTypes], cmap64[kNumTypes], map32[kNumTypes], cmap32[kNumTypes], map16[kNumTypes];
    bool built[kNumTypes] = {};
    GridSlots slots{};   // heavy atom types that occur in the receptor
    bool cells = false;  // the cell lists are those of the present receptor
    DevBuf ugrid;  // user grid values, or empty
    DGeom ug{};
    double ug_slope = 1e6;
    DevBuf dhdr;  // device copy of the DReceptor header
    DReceptor hdr{};
    void clear_maps() {
        for (int t = 0; t < kNumTypes; t++) {
            map64[t] = cmap64[t] = map32[t] = cmap32[t] = map16[t] = MapView{};
            built[t] = false;
        }
        map_mem.clear();
    }
    RecState() = default;
    RecState(const RecState&) = delete;
    RecState& operator=(const RecState&) = delete;
    ~RecState();
    size_t map_bytes() const {
        size_t b = 0;
        for (int t = 0; t < kNumTypes; t++)
            b += map64[t].bytes + cmap64[t].bytes + map32[t].bytes + cmap32[t].bytes + map16[t].bytes;
        return b;
    }
};

// a batch of models packed for the device
struct PackedModels {
    std::vector<DModel> host;  // host copies with device pointers
    DevBuf mem;                // pools and descriptors
    DModel* dmodels = nullptr;
    explicit PackedModels(sg_engine* e) : mem(e) {}
    Smem64 smem64;  // plain-path shared memory
    int max_conf = 0, max_dof = 0, max_heavy = 0, max_atoms = 0, max_pairs = 0, max_frames = 0;
};

}  // namespace sg

struct sg_engine {
    int device = 0;
    int precision = 0;
    int num_sms = 148;
    int max_smem = 227 * 1024;
    cudaStream_t stream = nullptr;
    std::string err;
    bool has_tables = false;
    sg::DevBuf tab_smooth, tab_fast, tab32;
    int force_wpb = 0, last_wpb = 0, last_blocks = 0;
    int tpc = 32;        // threads per chain of the batched search: 32, 64, 128, or 0 (by the batch's size)
    int last_team = 1;   // warps per chain of the last batched search
    int last_block_warps = 0, last_block_ligands = 0;  // ... and its chains with a block each
    bool es_on = false;   // early stop of the batched search (--fast; sg_set_early_stop)
    sg_early_stop es{};
    double last_mc_ms = 0, last_refine_ms = 0;
    uint64_t last_evals = 0, last_grid_hits = 0, last_pair_hits = 0, last_h2d = 0, last_d2h = 0;
    sg::DTables tables{};
    sg::RecState rec[SG_MAX_RECEPTORS];
    sg::DevBuf d_err;
    cudaMemPool_t pool = nullptr;  // temporaries of the calls
    ~sg_engine();
};

namespace sg {

// Runs f() on the engine's device and turns exceptions into status codes
// (the message goes to sg_last_error).
template <typename F>
int guarded(sg_engine* e, F f) {
    try {
        if (!e) return SG_ERR_ARG;
        cuda_check(cudaSetDevice(e->device), "cudaSetDevice");
        f();
        return SG_OK;
    } catch (EngineError& x) {
        e->err = x.what();
        return x.code;
    } catch (std::bad_alloc&) {
        e->err = "host allocation failed";
        return SG_ERR_NOMEM;
    } catch (std::exception& x) {
        e->err = x.what();
        return SG_ERR_ARG;
    }
}

// ---- launchers defined in the kernel files ---------------------------------------------------
cudaError_t launch_cell_lists(int natoms, const double* xyz, const int* type, const double* charge, const DGeom& g,
                              double cutoff_sqr, const double* bricks, int* count, const CellFamily& fam0,
                              const CellFamily& fam1, const GridSlots& slots, cudaStream_t s);
int grid_lanes(int ntypes);
cudaError_t launch_grid_map64(const DGeom&, const CellAtom* list, const double* list_charge, const int* cstart,
                              const DTables&, const int* types, int ntypes, const GridSlots&, double* tab,
                              double** maps, double** cmaps, const double* ugrid, const DGeom& ug, double ug_slope,
                              int num_sms, cudaStream_t);
cudaError_t launch_grid_pack(const DGeom&, const GridPack* maps, int nmaps, cudaStream_t);
// warps per item and shared memory of a plain-path launch over `items` items
// within max_smem bytes per block
Shape64 shape64(const Smem64& s, long long items, Work64 work, int num_sms, size_t max_smem);
cudaError_t launch_eval64(const DModel*, const Shape64&, int num_sms, const DTables&, const DReceptor*, int,
                          const double*, const double[3], double, int, double*, double*, double*, int*, cudaStream_t);
cudaError_t launch_bfgs64(const DModel*, const Shape64&, const DTables&, const DReceptor*, int, double*,
                          const double[3], double, int, int, int, double*, int*, cudaStream_t);
cudaError_t launch_mc64(const DModel*, const Shape64&, const DTables&, const DReceptor*, const Chain64*, int,
                        const MCParams64&, bool visited, int*, cudaStream_t);
cudaError_t launch_score64(const DModel* dms, const Shape64&, const DTables& T, const DReceptor* R, const int* pose_model,
                           int n, const double* confs, int conf_stride, const double v[3], double slope, double* e,
                           double* intra, double* coords, int coord_stride, int* err, cudaStream_t s);
cudaError_t launch_refine64(const DModel*, const Shape64&, const DTables&, const DReceptor*, const int*, int, double*, int,
                            const double[3], int, const int* pose_maxiters, const double* pose_box, int, int, double*,
                            double*, int, int*, cudaStream_t);
cudaError_t launch_merge32(const DModel* dms, const MergeJob32* jobs, int njobs, const Chain32* chains, int S,
                           double min_rmsd, int* count, int* pose_model, double* e, double* conf, int conf_stride,
                           double* xyz, int xyz_stride, cudaStream_t s);
size_t ws32_bytes(const DModel& hm);
int mc32_occupancy(int team, int wpb, size_t smem);
cudaError_t launch_mc32_feed(const DTables32& T, const FeedItem32* ring, unsigned cap, FeedCtrl32* ctrl,
                             long long idle_ns, int blocks, int wpb, size_t smem, cudaStream_t s);
cudaError_t mc32_feed_reserve_smem(size_t smem);
cudaError_t mc32_feed_occupancy(int wpb, size_t smem, int* blocks);
cudaError_t mc32_feed_max_dynamic_smem(size_t optin, size_t* out);
cudaError_t mc32_reserve_smem(size_t smem);
cudaError_t mc32_max_dynamic_smem(size_t optin, size_t* out);
cudaError_t launch_mc32_fixed(const DModel*, const DTables32&, const DMaps32&, const DMaps32* maps_tab, const Chain32*,
                              const Item32*, int nitems, const MCParams32&, unsigned* queue, int blocks, int wpb,
                              size_t stage_stride, size_t ws_stride, size_t smem_fixed, cudaStream_t s);
cudaError_t launch_mc32(const DModel*, const DTables32&, const DMaps32&, const DMaps32* maps_tab, const Chain32*,
                        const Item32*, int nitems, const MCParams32&, unsigned*, int blocks, int wpb,
                        size_t stage_stride, size_t ws_stride, int team, cudaStream_t);
int mc32_mix_occupancy(int warps, size_t smem);
cudaError_t launch_mc32_mix(const DModel*, const DTables32&, const DMaps32&, const Chain32*, const Item32*, int nitems,
                             const MCParams32&, unsigned* queue, int blocks, int warps, size_t stage_stride,
                             size_t ws_stride, size_t smem, cudaStream_t);
cudaError_t launch_eval32(const DModel*, size_t stage, size_t ws, const DTables32&, const DMaps32&, int, const double*,
                          const double[3], double, double*, double*, double*, int team, int num_sms, size_t max_smem,
                          cudaStream_t);
cudaError_t gather_probe(size_t working_set, int bytes_per_lookup, int num_sms, double* gbs, cudaStream_t s);
cudaError_t launch_bfgs32(const DModel*, size_t stage, size_t ws, size_t wide, int npairs, const DTables32&,
                          const DMaps32&, int, double*, const double v[3], double slope, int maxiters, int accurate, int early, double* e,
                          int team, int num_sms, size_t max_smem, cudaStream_t);

// FP32 views of the engine's tables and of a receptor's packed maps
DTables32 tables32(const sg_engine* e);
DMaps32 maps32(const sg_engine* e, const RecState& r);
// what is packed beyond the plain path's arrays: the mixed-precision path's
// copies and pair schedules, and the schedules seen from the atoms
enum PackFor { kPackPlain, kPackMixed, kPackWide };
void pack_models(CallIo& io, const sg_model_desc* models, int nmodels, PackFor what, PackedModels& out);
// the plain-path launch of a batch of models; refuses a model that does not fit
Shape64 plain_shape(sg_engine* e, const PackedModels& pm, long long items, Work64 work);
struct ModelImage {
    std::vector<char> bytes;   // pools then descriptors, ready to copy to the device
    size_t dmodel_off = 0;     // byte offset of the descriptor array
    std::vector<DModel> host;  // the descriptors (device addresses)
};
void pack_models_image(const sg_model_desc* models, int nmodels, char* dev_base, ModelImage& img);
RecState& receptor_for(sg_engine* e, int rid);
RecState& direct_receptor(sg_engine* e, int rid);  // for the direct sum: cell lists in place, no dropped maps kept
void ensure_cells(sg_engine* e, RecState& r);
void ensure_maps(sg_engine* e, RecState& r, const int* types, int ntypes);
void ensure_model_maps(sg_engine* e, RecState& r, const sg_model_desc* models, int nmodels);
void refresh_header(sg_engine* e, RecState& r);
void serve_shutdown(sg_engine* e);  // stops the engine's request loop, if one runs
// chains per block and resident blocks per SM of a k_mc32 launch (honours
// e->force_wpb)
void choose_launch(sg_engine* e, size_t stage_stride, size_t ws_stride, int max_chains, int& wpb, int& occ);
void noalloc_claim(sg_engine* e);  // the no-allocation entry point's set-up, at engine creation
}  // namespace sg
