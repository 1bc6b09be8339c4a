// engine.cu -- host side of libmdgb: the C ABI declared in include/mdgb.h.
//
// Drives the kernels of kernels_step.cu / kernels_list.cu / kernels_force.cu
// on one CUDA stream per handle.  A small system's whole chunk of steps is one
// launch (k_steps).  Otherwise one integrator step (integrator.rs:14-59) is:
//   k_pre        (cooperative)  coupling reductions -> kick/drift/wrap -> rebuild
//                               check -> [cell sort, only if needed]
//   k_list_masks, k_build_list  Verlet list of the rebuilt replicas (else return)
//   k_force_mixed               LJ forces + second half kick (+ on NVE chunks the
//                               next step's kick and drift, double-buffered)
//   k_force_band                mixed path: the atoms with a pair in the
//                               FP32-undecidable band around r_cut, with FP64
//                               decisions
//   k_pair_terms, k_pair_sums   FP64 path with pair records (each pair's terms
//                               once, then each atom's sums); k_force_fp64 else
// Steps run in chunks; before each chunk the engine snapshots the mutable
// device state, and if the chunk reports a neighbour-list overflow it grows
// the list, restores the snapshot and re-runs the chunk -- so capacity
// misses never surface as wrong results.  Chunks can be captured once into a
// CUDA graph and replayed.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <thread>
#include <utility>
#include <vector>

#include <sys/mman.h>
#include <unistd.h>

#include "../../include/mdgb.h"
#include "host_math.h"
#include "mdgb_internal.cuh"

namespace mdgb {
__global__ void k_pre(Dev d, StepParams sp);
__global__ void k_macro(Dev d, StepParams sp, int sel);
__global__ void k_apply_pending(Dev d);
__global__ void k_snapshot(Dev d, SnapArrays a);
__global__ void k_set_coupling(Dev d, RepCoupling c);
__global__ void k_gather_out(Dev d, double*, double*, double*, double*, double*);
__global__ void k_type_count(const int4* tiles, const uint16_t* type, int ntypes, int* count, int* bad);
__global__ void k_type_scan(const int2* reps, int ntypes, int* count, int* total);
__global__ void k_scatter_in(Dev d, const double*, const double*, const uint16_t*, const int*, int);
__global__ void k_scatter_forces(Dev d, const double*, const double*, const double*);
__global__ void k_pairs(Dev d, long long capacity, int* out_i, int* out_j, unsigned long long* count);
using force_fn = void (*)(Dev, StepParams);
force_fn force_kernel(int tpa, int precision, bool single, bool kick, bool persistent, bool noe);
using band_fn = void (*)(Dev, StepParams, int);
band_fn band_kernel(int precision);
}  // namespace mdgb

using namespace mdgb;

namespace {

struct LJ {
    double sigma = 0.3418, eps = 1.712, rc = 0.0, ucut = 0.0;  // potential.rs:96 default
    bool set = false;
};

void lj_finish(LJ& p) {
    double out[4];
    mdgb_lj_new(p.sigma, p.eps, out);
    p.rc = out[2];
    p.ucut = out[3];
}

struct ProfEvent { cudaEvent_t a, b; int kind; };

}  // namespace

struct mdgb_engine {
    mdgb_config cfg{};
    std::string err;
    int device = 0;
    cudaStream_t stream = nullptr;
    // the force launches of the size classes after the first run on their own
    // streams, forked from and joined back into `stream` (also inside graphs)
    cudaStream_t aux[3] = {nullptr, nullptr, nullptr};
    cudaEvent_t fork_ev = nullptr;
    cudaEvent_t join_ev[3] = {nullptr, nullptr, nullptr};
    int num_sms = 0;
    // the GPU reads the caller's pageable arrays itself (Grace: address
    // translation through the host's page tables), so uploads skip the copy
    bool host_direct = false;
    int pre_blocks_per_sm = 0, macro_blocks_per_sm = 0, steps_blocks_per_sm = 0;
    int force_blocks_per_sm[4] = {0, 0, 0, 0};
    LJ pot[MAX_TYPES][MAX_TYPES];
    LJ pot_default;

    // state
    bool has_state = false;
    bool forces_valid = false;
    int ntot = 0, nrep = 0, ntypes = 0, ntiles = 0, ncells = 0;
    std::vector<int64_t> offsets;
    std::vector<double> mass;
    std::vector<RepDev> rep_host;
    double rlist = 0, rcmax = 0, skin = 0;
    int cap = 0;
    int tpa = 1;                     // default / single-class threads per atom
    bool tuned = false;
    // size classes of replicas (by atom count): their tiles, threads per atom
    static constexpr int NCLASS = 3;
    std::vector<int> class_of;       // per replica
    int class_tpa[NCLASS] = {1, 1, 1};
    // sizes of the one-launch kernel: whether the lists are in the timed layout,
    // what the timing chose, and steps lately taken that the other layout suits
    bool timed_layout = false, timed = false;
    int timed_tpa[NCLASS] = {1, 1, 1};
    int64_t off_layout = 0;
    int class_ntiles[NCLASS] = {0, 0, 0};
    int class_tile_off[NCLASS] = {0, 0, 0};   // offset into dev.tile_order
    int class_nrep[NCLASS] = {0, 0, 0};
    // Verlet skin of each size class (a replica's list radius is the largest
    // r_cut plus its class's skin): the configured skin, or tuned on the
    // first step call when the configuration leaves it to the engine
    double class_skin[NCLASS] = {0.0, 0.0, 0.0};
    bool skin_tuned = false;

    Dev dev{};
    // allocations
    std::vector<void*> allocs;
    void* nbr_alloc = nullptr;
    void* pair_alloc = nullptr;      // the FP64 path's pair records (Dev::pairs)
    int pair_single = 0;             // Dev::single_type they were sized for
    bool pair_wanted = false;        // the last allocation's answer of pairs_wanted
    double mean_density = 0.0;       // around an atom, at the upload
    // snapshot buffers (chunk retry)
    double4_32a* snap_pos = nullptr;
    double* snap_d = nullptr;   // [8][N]
    int* snap_i = nullptr;      // [4][N]: orig, rank, cell, slot_of_rank
    float4* snap_mir0 = nullptr;
    RepDev* snap_rep = nullptr;
    // device staging in the caller's order; host arrays are copied to and
    // from it directly (no pinned host copy: on this platform the copy engine
    // reads and writes pageable memory at full link speed)
    double* d_out = nullptr;     // [11][N] caller-order staging (pos, vel, force, potential, temp)
    uint16_t* d_in_t = nullptr;  // [N] caller type ids
    // uploads of several types: tiles, counts per tile and type, totals (grown
    // to the largest such upload; not part of the state's allocations, since
    // they are needed before a state may be given up)
    void* type_buf = nullptr;
    size_t type_bytes = 0;
    // pinned: error words, replica 0's record after a step, and room for the
    // outputs of a small download (one copy, then the host's own)
    char* h_pin = nullptr;
    int* h_err = nullptr;        // in h_pin
    RepDev* h_rep = nullptr;     // in h_pin
    bool rep_fresh = false;      // h_rep is the record the last step call left
    bool coupling_set = false;   // some replica's coupling flags may be on
    unsigned long long* trace_buf = nullptr;  // per-phase ns of k_pre (MDGB_FLAG_TRACE)
    int lb_grid = 1, lm_grid = 1, lb_cap = -1, lb_ncells = -1;  // list-build launch shapes for (cap, cells)
    // the other position / mirror buffer of each pair (fused NVE drift)
    double4_32a* pos_alt = nullptr;
    float4* mir_alt = nullptr;
    // coupling (host view of the per-replica settings)
    bool thermo_on = false, baro_on = false, thermo_nh = false;

    // captured step chunks: one graph per distinct chunk length and launch
    // parameters (the key holds everything a capture bakes in), replayed
    // whenever a chunk with the same key comes again; a few are kept
    struct GraphKey {
        int len, lb_grid;
        unsigned flags;
        int precision;
        StepParams sp;
        Dev dev;
        const void* pos_alt;
        const void* mir_alt;
        int class_tpa[3], class_ntiles[3], class_tile_off[3], lm_grid;
    };
    struct GraphEntry {
        GraphKey key;
        cudaGraphExec_t exec;
        int64_t kernels;         // kernel launches one replay makes
        uint64_t used;
    };
    std::vector<GraphEntry> graphs;
    uint64_t graph_clock = 0;
    // the cells and lists were built at the current positions and nothing has
    // moved since (a force evaluation can skip its rebuild)
    bool lists_fresh = false;
    // failure test of the bounded grid barrier (mdgb_test_barrier_timeout):
    // the next step call's first chunk holds this block back (-1: off)
    int test_hold_block = -1, test_hold_step = 0;
    long long test_barrier_cycles = 0;

    // stats
    mdgb_stats st{};
    std::vector<ProfEvent> prof, prof_free;

    ~mdgb_engine();
};

namespace {

// Pinned memory of an engine: head (error words, one replica record), outputs.
constexpr size_t PIN_HEAD = 1024, PIN_OUT = size_t(256) << 10;
static_assert(64 + sizeof(RepDev) <= PIN_HEAD, "the record fits");

int fail(mdgb_engine* e, int code, const std::string& msg) {
    if (e) e->err = msg;
    return code;
}

#define CU(call)                                                                             \
    do {                                                                                     \
        cudaError_t _e = (call);                                                             \
        if (_e != cudaSuccess)                                                               \
            return fail(e, _e == cudaErrorMemoryAllocation ? MDGB_ERR_OUT_OF_MEMORY : MDGB_ERR_CUDA, \
                        std::string(#call) + ": " + cudaGetErrorString(_e));                 \
    } while (0)

template <class T>
int dalloc(mdgb_engine* e, T** p, size_t count) {
    void* q = nullptr;
    CU(cudaMalloc(&q, std::max<size_t>(count, 1) * sizeof(T)));
    e->allocs.push_back(q);
    *p = reinterpret_cast<T*>(q);
    return MDGB_OK;
}

void drop_graphs(mdgb_engine* e) {
    for (auto& g : e->graphs) cudaGraphExecDestroy(g.exec);
    e->graphs.clear();
}

void free_pairs(mdgb_engine* e) {
    if (e->pair_alloc) cudaFree(e->pair_alloc);
    e->pair_alloc = nullptr;
    e->dev.pairs = 0;
}

// Device allocations of a state (kept by an upload of the same shape).
void free_state(mdgb_engine* e) {
    drop_graphs(e);
    for (void* p : e->allocs) cudaFree(p);
    e->allocs.clear();
    if (e->nbr_alloc) { cudaFree(e->nbr_alloc); e->nbr_alloc = nullptr; }
    free_pairs(e);
    e->dev.nn = nullptr;
    e->has_state = false;
    e->forces_valid = false;
    e->lists_fresh = false;
}

const LJ& pot_of(const mdgb_engine* e, int a, int b) {
    if (a > b) std::swap(a, b);
    return e->pot[a][b].set ? e->pot[a][b] : e->pot_default;
}

// Skin of size class c: the tuned one, else the configured (or default) one.
double class_skin_of(const mdgb_engine* e, int c) { return e->skin_tuned ? e->class_skin[c] : e->skin; }

// The configuration asks the engine to choose the skin (skin < 0; 0 means
// the default skin).  The choice comes from timings, and on the mixed path
// the cell grid it implies changes FP32 roundings, so tuning is opt-in: an
// untuned run is reproducible bit for bit.  Reference-order runs keep the
// default (their sums do not depend on the list).
bool skin_auto(const mdgb_engine* e) {
    return e->cfg.skin < 0.0 && !((e->cfg.flags & MDGB_FLAG_REFERENCE_ORDER) && e->cfg.precision == MDGB_PRECISION_FP64);
}

// Skin candidates of the tuning, as fractions of the largest r_cut
// (0.2 .. 0.4 sigma at r_cut = 2.5 sigma).
constexpr double SKIN_FRACTIONS[5] = {0.08, 0.10, 0.12, 0.14, 0.16};

// The largest list radius of any replica (the force kernels' range bounds).
void update_rlist(mdgb_engine* e) {
    double smax = e->skin;
    for (int c = 0; c < mdgb_engine::NCLASS; ++c)
        if (e->class_ntiles[c]) smax = std::max(smax, class_skin_of(e, c));
    e->rlist = e->rcmax + smax;
    e->dev.rlist = e->rlist;
}

// The pair table of the current potentials and the scalars derived from it
// (largest cut-off, list radius, fixed-point scale), on the host.
std::vector<PairDev> pair_table(mdgb_engine* e) {
    std::vector<PairDev> tab(MAX_TYPES * MAX_TYPES);
    double fchar = 0.0;
    e->rcmax = 0.0;
    for (int a = 0; a < MAX_TYPES; ++a)
        for (int b = 0; b < MAX_TYPES; ++b) {
            const LJ& p = pot_of(e, a, b);
            PairDev q{};
            q.sigma = p.sigma; q.eps = p.eps; q.rc = p.rc; q.ucut = p.ucut;
            q.eps4 = 4.0 * p.eps;
            q.eps24 = 24.0 * p.eps;
            q.sig2f = (float)(p.sigma * p.sigma);
            q.eps4f = (float)q.eps4;
            q.eps24f = (float)q.eps24;
            q.ucutf = (float)p.ucut;
            const double rc2 = p.rc * p.rc;
            q.rc2f_lo = (float)(rc2 * (1.0 - 1e-5));
            q.rc2f_hi = (float)(rc2 * (1.0 + 1e-5));
            q.rc2_cut = sqrt_cut(p.rc);
            q.sig2 = p.sigma * p.sigma;
            tab[a * MAX_TYPES + b] = q;
            if (a < e->ntypes && b < e->ntypes) {
                e->rcmax = std::max(e->rcmax, p.rc);
                fchar = std::max(fchar, std::fabs(24.0 * p.eps / p.sigma));
            }
        }
    // fixed-point scale: a power of two putting the characteristic force near 2^31
    if (!(fchar > 0.0)) fchar = 1.0;
    const int ex = 31 - (int)std::ceil(std::log2(fchar));
    e->dev.fscale = std::ldexp(1.0f, ex);
    e->dev.fscale_log2 = ex;
    e->dev.inv_fscale = std::ldexp(1.0, -ex);
    e->dev.inv_fscale_f = std::ldexp(1.0f, -ex);
    e->skin = e->cfg.skin > 0.0 ? e->cfg.skin : 0.12 * e->rcmax;
    update_rlist(e);
    e->dev.rcmax = e->rcmax;
    e->dev.skin = e->skin;
    return tab;
}

int upload_pairs(mdgb_engine* e) {
    const std::vector<PairDev> tab = pair_table(e);
    CU(cudaMemcpyAsync((void*)e->dev.pair, tab.data(), tab.size() * sizeof(PairDev),
                       cudaMemcpyHostToDevice, e->stream));
    CU(cudaStreamSynchronize(e->stream));   // the table is a local copy
    return MDGB_OK;
}

// The FP64 path's pair records for the current list capacity.  From
// PAIR_MIN_ATOMS atoms on the pairs are computed once (kernels_pairs.cu); below,
// steps run as one launch, and with several threads per atom k_force_fp64
// evaluates both sides.  20 NVE steps with records / as one launch, us: tree order
// 1630 / 1245 at 4,000 atoms, 1700 / 1442 at 5,324, 1762 / 2487 at 8,788, reference
// order 1955 / 1762, 2077 / 2192, 2249 / 3966; forces alone 65 / 165 and 78 / 275 at
// 4,000.  The pair kernels walk the lists
// in the layout of one thread per atom, so there are records only while every
// size class has that layout: a state whose records found no room when it was
// uploaded may since have been tuned to another one.  About 4 KB an atom in a
// liquid, which only saves time: half of the device's memory is left to what
// has to be there (other engines' states and lists), and a caller who wants
// all of it sets MDGB_FLAG_NO_PAIR_RECORDS.
// Where an atom lists few others the four launches of the records cost more than
// the pairs: 20 NVE steps with / without them, us, by the entries expected an
// atom, 27,436 and 110,592 atoms in tree order: 2.8 811 / 578 and 1034 / 820, 4.6
// 880 / 797 and 1202 / 1506, 7.4 988 / 1188 and 1526 / 2784; forces alone 28 / 17
// at 1.8, 28 / 25 at 4.6, 52 / 115 at 7.4 (110,592).
constexpr int PAIR_MIN_ATOMS = 4096;
constexpr double PAIR_MIN_LISTED = 4.0;

bool pairs_wanted(const mdgb_engine* e) {
    if (e->cfg.precision != MDGB_PRECISION_FP64 || e->ntot < PAIR_MIN_ATOMS || e->cfg.threads_per_atom > 1 ||
        (e->cfg.flags & MDGB_FLAG_NO_PAIR_RECORDS))
        return false;
    for (int c = 0; c < mdgb_engine::NCLASS; ++c)
        if (e->class_ntiles[c] && e->class_tpa[c] != 1) return false;
    return 4.0 / 3.0 * M_PI * std::pow(e->rlist, 3) * e->mean_density >= PAIR_MIN_LISTED;
}

void alloc_pairs(mdgb_engine* e) {
    Dev& d = e->dev;
    free_pairs(e);
    e->pair_single = d.single_type;
    e->pair_wanted = pairs_wanted(e);
    if (!e->pair_wanted) return;
    const size_t N = e->ntot, room = pair_room(N, d.cap, d.single_type);
    if (room >= (size_t)PAIR_NEG) return;
    // sizes in whole 256 bytes, so that every array starts aligned
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t s_rec = up(room * sizeof(PairRec)), s_ij = up(room * sizeof(uint2)),
                 s_vir = up(room * sizeof(double)), s_of = up((size_t)d.cap * N * sizeof(uint32_t)), s_in = up(room),
                 s_tile = up(e->ntiles * sizeof(int2)), s_cnt = up(e->nrep * sizeof(int));
    const size_t total = s_rec + s_ij + s_vir + s_of + s_in + s_tile + s_cnt;
    size_t free_b = 0, all_b = 0;
    if (cudaMemGetInfo(&free_b, &all_b) != cudaSuccess || total + all_b / 2 > free_b ||
        cudaMalloc(&e->pair_alloc, total) != cudaSuccess) {
        cudaGetLastError();
        e->pair_alloc = nullptr;
        return;
    }
    char* q = static_cast<char*>(e->pair_alloc);
    d.pair_rec = reinterpret_cast<PairRec*>(q); q += s_rec;
    d.pair_ij = reinterpret_cast<uint2*>(q); q += s_ij;
    d.pair_vir = reinterpret_cast<double*>(q); q += s_vir;
    d.pair_of = reinterpret_cast<uint32_t*>(q); q += s_of;
    d.pair_in = reinterpret_cast<unsigned char*>(q); q += s_in;
    d.pair_tile = reinterpret_cast<int2*>(q); q += s_tile;
    d.pair_count = reinterpret_cast<int*>(q);
    // no records until the next rebuild
    cudaMemsetAsync(d.pair_tile, 0, s_tile + s_cnt, e->stream);
    d.pairs = 1;
}

int alloc_nbr(mdgb_engine* e, int cap) {
    // the tpa-interleaved layout (nbr_index) needs cap to be a multiple of every tpa
    cap = std::max(8, (cap + 7) & ~7);
    if (e->nbr_alloc) { cudaFree(e->nbr_alloc); e->nbr_alloc = nullptr; }
    free_pairs(e);   // they index the old list, and the new one may need their memory
    const size_t words = (size_t)cap * (size_t)e->ntot;
    void* q = nullptr;
    CU(cudaMalloc(&q, std::max<size_t>(words, 1) * sizeof(uint32_t)));
    // a fresh list holds valid (zero) entries and zero counts until the next rebuild
    CU(cudaMemsetAsync(q, 0, std::max<size_t>(words, 1) * sizeof(uint32_t), e->stream));
    if (e->dev.nn) CU(cudaMemsetAsync(e->dev.nn, 0, (size_t)e->ntot * sizeof(int), e->stream));
    e->nbr_alloc = q;
    e->dev.nbr = reinterpret_cast<uint32_t*>(q);
    e->dev.cap = cap;
    e->cap = cap;
    e->lists_fresh = false;
    alloc_pairs(e);
    return MDGB_OK;
}

void prof_begin(mdgb_engine* e, int kind, cudaEvent_t* out_b) {
    *out_b = nullptr;
    if (!(e->cfg.flags & MDGB_FLAG_PROFILE)) return;
    ProfEvent p;
    if (!e->prof_free.empty()) { p = e->prof_free.back(); e->prof_free.pop_back(); }
    else { cudaEventCreate(&p.a); cudaEventCreate(&p.b); }
    p.kind = kind;
    cudaEventRecord(p.a, e->stream);
    e->prof.push_back(p);
    *out_b = p.b;
}

void prof_end(mdgb_engine* e, cudaEvent_t b) {
    if (b) cudaEventRecord(b, e->stream);
}

void prof_collect(mdgb_engine* e) {
    for (auto& p : e->prof) {
        float ms = 0.f;
        cudaEventSynchronize(p.b);
        cudaEventElapsedTime(&ms, p.a, p.b);
        if (p.kind == 0) { e->st.force_ms += ms; e->st.force_launches++; }
        else { e->st.integrate_ms += ms; e->st.integrate_launches++; }
        e->prof_free.push_back(p);
    }
    e->prof.clear();
}

// Blocks of k_pre or k_macro: no more than are resident.
int pre_grid(const mdgb_engine* e, int blocks_per_sm) {
    const int maxg = std::min(4096, std::max(1, e->num_sms * blocks_per_sm));  // bsum holds 4096
    // reference order: one block per serial fold (six a replica at most)
    const int folds = e->dev.refmode ? 6 * std::min(e->nrep, maxg) : 1;
    const int want = std::max({e->ntiles, (e->ncells + 1023) / 1024, (e->nrep + TILE - 1) / TILE, folds});
    return std::min(maxg, want);
}

int launch_pre(mdgb_engine* e, const StepParams& sp) {
    cudaEvent_t pe;
    prof_begin(e, 1, &pe);
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3(pre_grid(e, e->pre_blocks_per_sm));
    lc.blockDim = dim3(TILE);
    lc.stream = e->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    lc.attrs = at;
    lc.numAttrs = 1;
    CU(cudaLaunchKernelEx(&lc, k_pre, e->dev, sp));
    if (e->lb_cap != e->dev.cap || e->lb_ncells != e->dev.ncells) {
        e->lb_grid = list_build_grid(e->dev, e->num_sms);
        e->lm_grid = list_masks_grid(e->dev, e->num_sms);
        e->lb_cap = e->dev.cap;
        e->lb_ncells = e->dev.ncells;
    }
    CU(launch_list_build(e->dev, e->lb_grid, e->lm_grid, e->stream));
    prof_end(e, pe);
    e->st.kernel_launches += e->dev.pairs ? 5 : 3;
    return MDGB_OK;
}

// Blocks of size class c's force launch: one per tile, or (persistent) as
// many as are resident.
int force_grid(mdgb_engine* e, int c, bool kick) {
    const int ntl = e->class_ntiles[c];
    if (!(e->cfg.flags & MDGB_FLAG_PERSISTENT)) return ntl;
    const int tpa = e->class_tpa[c];
    force_fn fn = force_kernel(tpa, e->cfg.precision, e->dev.single_type != 0, kick, true, false);
    int bps = 0;
    if (!fn || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, (const void*)fn, TILE * tpa, 0) != cudaSuccess)
        bps = 1;
    return std::min(ntl, std::max(1, bps) * e->num_sms);
}

// One force launch per non-empty size class, each with that class's threads
// per atom (the replicas of a class were listed with the same layout).
int launch_force_class(mdgb_engine* e, const StepParams& sp, bool kick, int c, cudaStream_t st) {
    const bool persistent = (e->cfg.flags & MDGB_FLAG_PERSISTENT) != 0;
    const int tpa = e->class_tpa[c];
    force_fn fn = force_kernel(tpa, e->cfg.precision, e->dev.single_type != 0, kick, persistent,
                               kick && sp.fused);
    if (!fn) return fail(e, MDGB_ERR_INVALID_ARGUMENT, "threads_per_atom must be 1, 2, 4 or 8");
    Dev d = e->dev;
    d.pos_next = e->pos_alt;
    d.mir_next = e->mir_alt;
    d.tile_list = e->dev.tile_order + e->class_tile_off[c];
    d.ntile_list = e->class_ntiles[c];
    d.list_class = c;
    const int grid = force_grid(e, c, kick);
    void* args[] = {(void*)&d, (void*)&sp};
    CU(cudaLaunchKernel((const void*)fn, dim3(grid), dim3(TILE * tpa), args, 0, st));
    e->st.kernel_launches++;
    return MDGB_OK;
}

int launch_force(mdgb_engine* e, const StepParams& sp_in, bool kick) {
    cudaEvent_t pe;
    prof_begin(e, 0, &pe);
    if ((e->cfg.flags & MDGB_FLAG_PERSISTENT) && !e->dev.pairs)
        CU(cudaMemsetAsync(e->dev.queue, 0, mdgb_engine::NCLASS * sizeof(unsigned int), e->stream));
    const StepParams& sp = sp_in;
    if (e->dev.pairs) {
        Dev d = e->dev;
        d.pos_next = e->pos_alt;
        d.mir_next = e->mir_alt;
        CU(launch_pair_forces(d, sp, kick, e->num_sms, e->stream));
        e->st.kernel_launches += 2;
        prof_end(e, pe);
        if (kick && sp.fused) {
            std::swap(e->dev.pos, e->pos_alt);
            std::swap(e->dev.mir, e->mir_alt);
        }
        return MDGB_OK;
    }
    band_fn bk = band_kernel(e->cfg.precision);
    if (bk) CU(cudaMemsetAsync(e->dev.band_count, 0, sizeof(int), e->stream));
    // classes touch disjoint atoms, tiles and queue counters: the second and
    // third run concurrently with the first on their own streams
    int nclasses = 0;
    for (int c = 0; c < mdgb_engine::NCLASS; ++c) nclasses += e->class_ntiles[c] ? 1 : 0;
    bool first = true;
    for (int c = 0; c < mdgb_engine::NCLASS; ++c) {
        if (!e->class_ntiles[c]) continue;
        int rc;
        if (first) {
            if (nclasses > 1) CU(cudaEventRecord(e->fork_ev, e->stream));
            rc = launch_force_class(e, sp, kick, c, e->stream);
            first = false;
        } else {
            CU(cudaStreamWaitEvent(e->aux[c], e->fork_ev, 0));
            rc = launch_force_class(e, sp, kick, c, e->aux[c]);
            if (!rc) CU(cudaEventRecord(e->join_ev[c], e->aux[c]));
            if (!rc) CU(cudaStreamWaitEvent(e->stream, e->join_ev[c], 0));
        }
        if (rc) return rc;
    }
    if (bk) {
        // the atoms the force launches left: same buffers as they used
        Dev d = e->dev;
        d.pos_next = e->pos_alt;
        d.mir_next = e->mir_alt;
        int kk = kick ? 1 : 0;
        void* args[] = {(void*)&d, (void*)&sp, (void*)&kk};
        CU(cudaLaunchKernel((const void*)bk, dim3(4 * e->num_sms), dim3(128), args, 0, e->stream));
        e->st.kernel_launches++;
    }
    prof_end(e, pe);
    if (kick && sp.fused) {   // the next positions/mirrors are in the other buffers now
        std::swap(e->dev.pos, e->pos_alt);
        std::swap(e->dev.mir, e->mir_alt);
    }
    return MDGB_OK;
}

// Write the per-replica threads per atom (the list layout) of every size class.
int apply_class_tpa(mdgb_engine* e) {
    CU(cudaMemcpyAsync(e->rep_host.data(), e->dev.rep, e->nrep * sizeof(RepDev), cudaMemcpyDeviceToHost, e->stream));
    CU(cudaStreamSynchronize(e->stream));
    bool changed = false;
    for (int r = 0; r < e->nrep; ++r) {
        const int t = e->class_tpa[e->class_of[r]];
        changed |= e->rep_host[r].tpa != t;
        e->rep_host[r].tpa = t;
    }
    if (!changed) return MDGB_OK;
    CU(cudaMemcpyAsync(e->dev.rep, e->rep_host.data(), e->nrep * sizeof(RepDev), cudaMemcpyHostToDevice, e->stream));
    e->lists_fresh = false;   // the list layout changed
    return MDGB_OK;
}

// Each replica's list radius: the largest r_cut plus its size class's skin.
int apply_class_skin(mdgb_engine* e) {
    CU(cudaMemcpyAsync(e->rep_host.data(), e->dev.rep, e->nrep * sizeof(RepDev), cudaMemcpyDeviceToHost, e->stream));
    CU(cudaStreamSynchronize(e->stream));
    for (int r = 0; r < e->nrep; ++r) e->rep_host[r].rlist = e->rcmax + class_skin_of(e, e->class_of[r]);
    CU(cudaMemcpyAsync(e->dev.rep, e->rep_host.data(), e->nrep * sizeof(RepDev), cudaMemcpyHostToDevice, e->stream));
    update_rlist(e);
    e->lists_fresh = false;
    return MDGB_OK;
}

StepParams make_sp(const mdgb_engine* e, double dt, bool drift) {
    StepParams sp;
    std::memset(&sp, 0, sizeof(sp));   // byte-wise comparable (graph keys)
    sp.hold_block = -1;
    sp.dt = dt;
    for (int t = 0; t < MAX_TYPES; ++t)
        sp.kick_c[t] = t < (int)e->mass.size() ? dt / (2.0 * e->mass[t]) : 0.0;  // integrator.rs:29-30
    sp.coupled = (e->thermo_on || e->baro_on) ? 1 : 0;
    sp.thermo_nh = e->thermo_nh ? 1 : 0;
    sp.fixed_interval = e->cfg.rebuild_every;
    sp.force_rebuild = 0;
    sp.do_drift = drift ? 1 : 0;
    return sp;
}

int read_err(mdgb_engine* e, int* flags) {
    CU(cudaMemcpyAsync(e->h_err, e->dev.err, 2 * sizeof(int), cudaMemcpyDeviceToHost, e->stream));
    CU(cudaStreamSynchronize(e->stream));
    *flags = e->h_err[0];
    return MDGB_OK;
}

int clear_err(mdgb_engine* e) {
    CU(cudaMemsetAsync(e->dev.err, 0, 2 * sizeof(int), e->stream));
    // bar[5] (direct list builds) is a counter: kept
    CU(cudaMemsetAsync(e->dev.bar, 0, 5 * sizeof(unsigned int), e->stream));
    return MDGB_OK;
}

int snapshot(mdgb_engine* e, bool restore) {
    const size_t N = e->ntot;
    auto cp = [&](void* dst, const void* src, size_t bytes) {
        return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, e->stream);
    };
    Dev& d = e->dev;
    if (!restore) {
        CU(cp(e->snap_pos, d.pos, N * sizeof(double4_32a)));
        CU(cp(e->snap_d, d.vel, 3 * N * sizeof(double)));
        CU(cp(e->snap_d + 3 * N, d.frc, 3 * N * sizeof(double)));
        CU(cp(e->snap_d + 6 * N, d.epot, N * sizeof(double)));
        CU(cp(e->snap_d + 7 * N, d.evir, N * sizeof(double)));
        CU(cp(e->snap_i, d.orig, N * sizeof(int)));
        CU(cp(e->snap_i + N, d.rank, N * sizeof(int)));
        CU(cp(e->snap_i + 2 * N, d.cell, N * sizeof(int)));
        CU(cp(e->snap_i + 3 * N, d.slot_of_rank, N * sizeof(int)));
        CU(cp(e->snap_mir0, d.mir0, N * sizeof(float4)));
        CU(cp(e->snap_rep, d.rep, e->nrep * sizeof(RepDev)));
    } else {
        CU(cp(d.pos, e->snap_pos, N * sizeof(double4_32a)));
        CU(cp(d.vel, e->snap_d, 3 * N * sizeof(double)));
        CU(cp(d.frc, e->snap_d + 3 * N, 3 * N * sizeof(double)));
        CU(cp(d.epot, e->snap_d + 6 * N, N * sizeof(double)));
        CU(cp(d.evir, e->snap_d + 7 * N, N * sizeof(double)));
        CU(cp(d.orig, e->snap_i, N * sizeof(int)));
        CU(cp(d.rank, e->snap_i + N, N * sizeof(int)));
        CU(cp(d.cell, e->snap_i + 2 * N, N * sizeof(int)));
        CU(cp(d.slot_of_rank, e->snap_i + 3 * N, N * sizeof(int)));
        CU(cp(d.mir0, e->snap_mir0, N * sizeof(float4)));
        CU(cp(d.rep, e->snap_rep, e->nrep * sizeof(RepDev)));
    }
    return MDGB_OK;
}

// What a chunk needs to be run again, copied aside, and the error words and the
// barrier cleared, in one launch instead of eleven copies and two clears.  us a
// call of one step, copies / one launch: 70,304 atoms 133 / 79, 256,000 167 / 135,
// 442,368 228 / 188, 1M 432 / 358, 4M 1245 / 1206.
int begin_chunk(mdgb_engine* e) {
    const size_t N = e->ntot;
    Dev& d = e->dev;
    const SnapArrays a{{e->snap_pos, e->snap_d, e->snap_d + 3 * N, e->snap_d + 6 * N, e->snap_d + 7 * N, e->snap_i,
                        e->snap_i + N, e->snap_i + 2 * N, e->snap_i + 3 * N, e->snap_mir0, e->snap_rep},
                       {d.pos, d.vel, d.frc, d.epot, d.evir, d.orig, d.rank, d.cell, d.slot_of_rank, d.mir0, d.rep},
                       {N * sizeof(double4_32a), 3 * N * sizeof(double), 3 * N * sizeof(double), N * sizeof(double),
                        N * sizeof(double), N * sizeof(int), N * sizeof(int), N * sizeof(int), N * sizeof(int),
                        N * sizeof(float4), e->nrep * sizeof(RepDev)}};
    void* args[] = {(void*)&e->dev, (void*)&a};
    const unsigned grid = (unsigned)std::max<size_t>(1, std::min<size_t>((N + 255) / 256, 4 * (size_t)e->num_sms));
    CU(cudaLaunchKernel((const void*)k_snapshot, dim3(grid), dim3(256), args, 0, e->stream));
    return MDGB_OK;
}

int grow_list(mdgb_engine* e) {
    int needed = 0;
    CU(cudaMemcpyAsync(&needed, e->dev.max_needed, sizeof(int), cudaMemcpyDeviceToHost, e->stream));
    CU(cudaStreamSynchronize(e->stream));
    int cap = std::max(e->cap + 8, (int)std::ceil(needed * 1.25));
    cap = (cap + 7) & ~7;
    CU(cudaMemsetAsync(e->dev.max_needed, 0, sizeof(int), e->stream));
    int rc = alloc_nbr(e, cap);
    if (rc) return rc;
    e->st.neighbor_capacity = cap;
    return MDGB_OK;
}

// Forced rebuild + mirror refresh without integration.
int refresh(mdgb_engine* e, bool force_rebuild) {
    StepParams sp = make_sp(e, 0.0, false);
    sp.force_rebuild = force_rebuild ? 1 : 0;
    return launch_pre(e, sp);
}

int check_flags(mdgb_engine* e, int flags) {
    if (flags & E_TIMEOUT) return fail(e, MDGB_ERR_DEVICE_TIMEOUT, "a device-side grid barrier timed out");
    if (flags & E_FIXED)
        return fail(e, MDGB_ERR_FIXED_POINT_OVERFLOW,
                    "a pair force left the 64-bit fixed-point range (atoms overlapping?)");
    if (flags & E_INPUT) return fail(e, MDGB_ERR_INVALID_ARGUMENT, "type id >= ntypes");
    if (flags & (E_BOUNDS | E_CELLS)) return fail(e, MDGB_ERR_CUDA, "internal index check failed");
    return MDGB_OK;
}

// Forced rebuild of cells and lists at the current positions; a list that
// overflows is grown and built again.
int rebuild_lists(mdgb_engine* e) {
    for (int attempt = 0; attempt < 8; ++attempt) {
        int rc = clear_err(e);
        if (rc) return rc;
        rc = refresh(e, true);
        if (rc) return rc;
        int flags = 0;
        rc = read_err(e, &flags);
        if (rc) return rc;
        if (flags & E_NLIST) {
            rc = grow_list(e);
            if (rc) return rc;
            e->st.retries++;
            continue;
        }
        rc = check_flags(e, flags);
        if (rc) return rc;
        e->lists_fresh = true;
        return MDGB_OK;
    }
    return fail(e, MDGB_ERR_NEIGHBOR_OVERFLOW, "neighbour list kept overflowing");
}

// update_force: a rebuild (skipped when the lists were just built at these
// positions -- a second one would give the same cells and lists), then the
// force pass.
int compute_forces_impl(mdgb_engine* e) {
    for (int attempt = 0; attempt < 8; ++attempt) {
        int rc = clear_err(e);
        if (rc) return rc;
        if (!e->lists_fresh) {
            rc = refresh(e, true);
            if (rc) return rc;
        }
        StepParams sp = make_sp(e, 0.0, false);
        rc = launch_force(e, sp, false);
        if (rc) return rc;
        int flags = 0;
        rc = read_err(e, &flags);
        if (rc) return rc;
        if (flags & E_NLIST) {
            rc = grow_list(e);
            if (rc) return rc;
            e->st.retries++;
            continue;
        }
        rc = check_flags(e, flags);
        if (rc) return rc;
        e->lists_fresh = true;
        return MDGB_OK;
    }
    return fail(e, MDGB_ERR_NEIGHBOR_OVERFLOW, "neighbour list kept overflowing");
}

// Whether a chunk of this state's steps runs as one launch (k_steps): few
// enough atoms that the step is launch latency and a mostly idle chip, one
// thread per atom in the list layout, and nothing that looks at single
// launches.  us a step, one launch / launches, mixed path: NVE 19 / 51 at 4,000
// atoms, 23 / 51 at 8,788, 35 / 51 at 23,328, 66 / 59 at 32,000; Berendsen T
// and P 55 / 74, 66 / 75, 68 / 74 at 10,976, 70 / 77 (66 in the timed layout) at
// 13,500, 84 / 76 at 16,384; Nose-Hoover 93 / 97 at 10,976, 98 / 100 (90) at 13,500,
// 107 / 98 at 16,384.
// An ensemble rebuilds some replica at nearly every step, and one block decides
// for all of them: us for 20 NVE steps, one launch / launches, replicas of 64
// atoms 2042 / 2760 at 64, 2748 / 3125 at 150, 3401 / 3365 at 300, 3642 / 3523 at
// 380; of 27 atoms 2510 / 2602 at 300, 3865 / 3254 at 800.  Against launches in the
// timed layout, where threads per atom are the engine's choice: of 64 atoms 1947 /
// 2673 at 60, 2220 / 2292 at 100 (Berendsen T and P 3122 / 2839), 2755 / 2515 at 150.
constexpr int TUNE_MIN_ATOMS = 4096;   // fewer: threads per atom are not worth measuring
constexpr int SMALL_MAX_ATOMS = 24576, SMALL_MAX_COUPLED = 12288, SMALL_MAX_REPLICAS = 300,
              SMALL_MAX_TUNABLE = 96;
bool small_size(const mdgb_engine* e) {
    const bool tunable = e->cfg.threads_per_atom == 0 && e->ntot >= TUNE_MIN_ATOMS && !e->dev.refmode;
    return e->ntot <= SMALL_MAX_ATOMS && e->nrep <= (tunable ? SMALL_MAX_TUNABLE : SMALL_MAX_REPLICAS) && !e->dev.pairs &&
           e->cfg.rebuild_every == 0 && e->steps_blocks_per_sm > 0 && e->cfg.threads_per_atom <= 1 &&
           !(e->cfg.flags & (MDGB_FLAG_PROFILE | MDGB_FLAG_TRACE | MDGB_FLAG_PERSISTENT));
}
// Steps of such a size that run as launches all the same.
bool steps_as_launches(const mdgb_engine* e, bool coupled) { return coupled && e->ntot > SMALL_MAX_COUPLED; }
bool small_system(const mdgb_engine* e, const StepParams& sp) {
    if (!small_size(e) || steps_as_launches(e, sp.coupled || sp.thermo_nh)) return false;
    for (int c = 0; c < mdgb_engine::NCLASS; ++c)
        if (e->class_ntiles[c] && e->class_tpa[c] != 1) return false;
    return true;
}

// n steps.  NVE chunks fuse each step's first kick and drift into the force
// pass of the step before (steps 2..nf+1); nf is even, so the position/mirror
// buffer pair ends the chunk the way round it started (a captured graph stays
// valid), and the chunk's last step is unfused, leaving the state at a whole
// step.
int run_chunk_kernels(mdgb_engine* e, const StepParams& sp, int n) {
    if (small_system(e, sp)) {
        Dev d = e->dev;
        d.pos_next = e->pos_alt;
        d.mir_next = e->mir_alt;
        const bool naive = e->cfg.precision == MDGB_PRECISION_FP32_NAIVE;
        const int blocks = e->num_sms * e->steps_blocks_per_sm;
        // (the failure test in a later step: the steps before it by themselves)
        const int before = sp.hold_block >= 0 ? std::min(sp.hold_step, n - 1) : 0;
        if (before > 0) {
            StepParams clean = sp;
            clean.hold_block = -1;
            CU(launch_steps(d, clean, before, naive, blocks, e->stream));
        }
        CU(launch_steps(d, sp, n - before, naive, blocks, e->stream));
        e->st.kernel_launches++;
        return MDGB_OK;
    }
    const bool fusable = sp.do_drift && !sp.coupled && !sp.thermo_nh;
    const int nf = fusable ? ((n - 1) & ~1) : 0;
    for (int i = 0; i < n; ++i) {
        StepParams pre = sp;
        pre.predrifted = (i >= 1 && i <= nf) ? 1 : 0;
        if (i != sp.hold_step) pre.hold_block = -1;
        int rc = launch_pre(e, pre);
        if (rc) return rc;
        StepParams frc = sp;
        frc.fused = i < nf ? 1 : 0;
        rc = launch_force(e, frc, true);
        if (rc) return rc;
    }
    return MDGB_OK;
}

mdgb_engine::GraphKey graph_key(const mdgb_engine* e, const StepParams& sp, int n) {
    mdgb_engine::GraphKey k;
    std::memset(&k, 0, sizeof(k));   // padding included: keys compare as bytes
    k.len = n;
    k.lb_grid = e->lb_grid;
    k.lm_grid = e->lm_grid;
    k.flags = e->cfg.flags;
    k.precision = e->cfg.precision;
    k.sp = sp;
    k.dev = e->dev;
    k.pos_alt = e->pos_alt;
    k.mir_alt = e->mir_alt;
    for (int c = 0; c < mdgb_engine::NCLASS; ++c) {
        k.class_tpa[c] = e->class_tpa[c];
        k.class_ntiles[c] = e->class_ntiles[c];
        k.class_tile_off[c] = e->class_tile_off[c];
    }
    return k;
}

// The graph of a chunk of n steps with these parameters, captured on first
// use (capture runs nothing).  Returns null when graphs are off or capture is
// not possible here (the engine then stays eager).
mdgb_engine::GraphEntry* chunk_graph(mdgb_engine* e, const StepParams& sp, int n, int* rc_out) {
    *rc_out = MDGB_OK;
    if (!(e->cfg.graph_steps > 1) || (e->cfg.flags & MDGB_FLAG_PROFILE)) return nullptr;
    // the list-build grid is part of the key: settle it before the lookup
    if (e->lb_cap != e->dev.cap || e->lb_ncells != e->dev.ncells) {
        e->lb_grid = list_build_grid(e->dev, e->num_sms);
        e->lm_grid = list_masks_grid(e->dev, e->num_sms);
        e->lb_cap = e->dev.cap;
        e->lb_ncells = e->dev.ncells;
    }
    const mdgb_engine::GraphKey key = graph_key(e, sp, n);
    for (auto& g : e->graphs)
        if (std::memcmp(&g.key, &key, sizeof(key)) == 0) {
            g.used = ++e->graph_clock;
            return &g;
        }
    cudaGraph_t g = nullptr;
    cudaError_t ce = cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeThreadLocal);
    if (ce != cudaSuccess) { *rc_out = fail(e, MDGB_ERR_CUDA, cudaGetErrorString(ce)); return nullptr; }
    const int64_t launches0 = e->st.kernel_launches;
    // capture runs nothing: the buffer pair must read as before afterwards
    double4_32a* const pos0 = e->dev.pos; double4_32a* const pos1 = e->pos_alt;
    float4* const mir0 = e->dev.mir; float4* const mir1 = e->mir_alt;
    int rc = run_chunk_kernels(e, sp, n);
    ce = cudaStreamEndCapture(e->stream, &g);
    e->dev.pos = pos0; e->pos_alt = pos1; e->dev.mir = mir0; e->mir_alt = mir1;
    const int64_t kernels = e->st.kernel_launches - launches0;
    e->st.kernel_launches = launches0;
    cudaGraphExec_t exec = nullptr;
    if (!rc && ce == cudaSuccess) ce = cudaGraphInstantiate(&exec, g, 0);
    if (g) cudaGraphDestroy(g);
    if (rc || ce != cudaSuccess) {
        cudaGetLastError();
        e->cfg.graph_steps = 0;  // capture unsupported here: stay eager
        return nullptr;
    }
    if (e->graphs.size() >= 6) {   // drop the least recently used
        size_t lru = 0;
        for (size_t i = 1; i < e->graphs.size(); ++i)
            if (e->graphs[i].used < e->graphs[lru].used) lru = i;
        cudaGraphExecDestroy(e->graphs[lru].exec);
        e->graphs.erase(e->graphs.begin() + (long)lru);
    }
    e->graphs.push_back(mdgb_engine::GraphEntry{key, exec, kernels, ++e->graph_clock});
    return &e->graphs.back();
}

int run_chunk(mdgb_engine* e, const StepParams& sp, int n) {
    int rc = MDGB_OK;
    mdgb_engine::GraphEntry* g = chunk_graph(e, sp, n, &rc);
    if (rc) return rc;
    if (!g) return run_chunk_kernels(e, sp, n);
    CU(cudaGraphLaunch(g->exec, e->stream));
    e->st.graph_launches++;
    e->st.kernel_launches += g->kernels;
    return MDGB_OK;
}

// Chunk lengths a call of nsteps steps runs: full chunks, then the rest.
int chunk_steps(const mdgb_engine* e) { return e->cfg.graph_steps > 1 ? e->cfg.graph_steps : 64; }

int settle_tpa(mdgb_engine* e, bool launches, int64_t steps);
int autotune_skin(mdgb_engine* e, double dt);

int step_impl(mdgb_engine* e, int64_t nsteps, double dt) {
    if (!e->has_state) return fail(e, MDGB_ERR_NO_STATE, "no state uploaded");
    if (nsteps < 0 || !(dt == dt)) return fail(e, MDGB_ERR_INVALID_ARGUMENT, "bad nsteps or dt");
    {
        const int rc = settle_tpa(e, steps_as_launches(e, e->thermo_on || e->baro_on), nsteps);
        if (rc) return rc;
    }
    if (nsteps > 0 && !e->skin_tuned && skin_auto(e)) {
        int rc = autotune_skin(e, dt);
        if (rc) return rc;
    }
    const StepParams sp = make_sp(e, dt, true);
    const int chunk = chunk_steps(e);
    if (nsteps > 0) e->lists_fresh = false;
    int64_t done = 0;
    int retries = 0;
    while (done < nsteps) {
        const int n = (int)std::min<int64_t>(chunk, nsteps - done);
        e->rep_fresh = false;   // until this chunk's steps stand
        int rc = begin_chunk(e);
        if (rc) return rc;
        if (e->test_hold_block >= 0) {
            // the armed failure test: this chunk eager, one block of its first
            // (or a later) step held back, and a short wait limit
            StepParams t = sp;
            t.hold_block = e->test_hold_block;
            t.hold_step = e->test_hold_step;
            t.barrier_cycles = e->test_barrier_cycles;
            e->test_hold_block = -1;
            rc = run_chunk_kernels(e, t, n);
        } else {
            rc = run_chunk(e, sp, n);
        }
        if (rc) return rc;
        int flags = 0;
        // a single system's coupling state comes back with the error words
        const bool with_rep = e->nrep == 1 && (e->thermo_on || e->baro_on);
        if (with_rep) CU(cudaMemcpyAsync(e->h_rep, e->dev.rep, sizeof(RepDev), cudaMemcpyDeviceToHost, e->stream));
        rc = read_err(e, &flags);
        if (rc) return rc;
        if (flags & E_TIMEOUT) {
            // a grid barrier gave up: the rest of the chunk did nothing; put
            // the state back as the chunk found it, so the engine stays usable
            rc = snapshot(e, true);
            if (!rc) rc = rebuild_lists(e);
            if (rc) return rc;
            return fail(e, MDGB_ERR_DEVICE_TIMEOUT,
                        "a device-side grid barrier timed out; the state is as before the failed chunk");
        }
        if (flags & E_NLIST) {
            if (++retries > 8) return fail(e, MDGB_ERR_NEIGHBOR_OVERFLOW, "neighbour list kept overflowing");
            rc = grow_list(e);
            if (rc) return rc;
            rc = snapshot(e, true);
            if (rc) return rc;
            // the restored state keeps its cells; rebuild lists at the new capacity
            rc = clear_err(e);
            if (rc) return rc;
            rc = refresh(e, true);
            if (rc) return rc;
            e->st.retries++;
            continue;
        }
        rc = check_flags(e, flags);
        if (rc) return rc;
        e->rep_fresh = with_rep;
        done += n;
        e->st.steps += n;
    }
    // finish the last step's barostat update (barostat.rs:45-48)
    if (e->baro_on) {
        void* args[] = {(void*)&e->dev};
        CU(cudaLaunchKernel((const void*)k_apply_pending, dim3(e->ntiles), dim3(TILE), args, 0, e->stream));
        e->st.kernel_launches++;
    }
    e->forces_valid = true;
    return MDGB_OK;
}

// Capture, without running anything, the graphs a call of nsteps steps with
// these coupling kinds will replay (the full chunk and the remainder), so the
// first such call does not pay for the capture.
int prepare_impl(mdgb_engine* e, int64_t nsteps, double dt, bool thermo_on, bool baro_on, bool thermo_nh) {
    if (!e->has_state) return fail(e, MDGB_ERR_NO_STATE, "no state uploaded");
    if (nsteps < 0 || !(dt == dt)) return fail(e, MDGB_ERR_INVALID_ARGUMENT, "bad nsteps or dt");
    if (!(e->cfg.graph_steps > 1)) return MDGB_OK;   // eager engine: nothing to capture
    {
        // the layout that call will choose, without counting its steps here
        const int64_t off = e->off_layout;
        const bool layout = e->timed_layout;
        const int rc = settle_tpa(e, steps_as_launches(e, thermo_on || baro_on), nsteps);
        if (rc) return rc;
        if (layout == e->timed_layout) e->off_layout = off;
    }
    const bool t0 = e->thermo_on, b0 = e->baro_on, n0 = e->thermo_nh;
    if (nsteps > 0 && !e->skin_tuned && skin_auto(e)) {
        // the tuning runs steps: with the coupling kinds of the later call
        e->thermo_on = thermo_on; e->baro_on = baro_on; e->thermo_nh = thermo_nh;
        const int rc = autotune_skin(e, dt);
        e->thermo_on = t0; e->baro_on = b0; e->thermo_nh = n0;
        if (rc) return rc;
    }
    e->thermo_on = thermo_on; e->baro_on = baro_on; e->thermo_nh = thermo_nh;
    const StepParams sp = make_sp(e, dt, true);
    e->thermo_on = t0; e->baro_on = b0; e->thermo_nh = n0;
    const int chunk = chunk_steps(e);
    const int64_t lens[2] = {std::min<int64_t>(chunk, nsteps), nsteps > chunk ? nsteps % chunk : 0};
    for (int64_t len : lens) {
        if (len <= 0) continue;
        int rc = MDGB_OK;
        chunk_graph(e, sp, (int)len, &rc);
        if (rc) return rc;
    }
    return MDGB_OK;
}

// Skin of each size class, for the step's own dynamics: from the state the
// first step call starts from, each candidate (SKIN_FRACTIONS of the largest
// r_cut) runs a short stretch of steps (eager launches, CUDA-event timed, its
// rebuilds included) and the state is put back; classes are tuned one after
// the other, each keeping its fastest.  A larger skin means longer lists but
// fewer rebuilds.  The steps taken here are not counted and leave no trace:
// the state afterwards is the one the call started from.
int autotune_skin(mdgb_engine* e, double dt) {
    constexpr int NC = mdgb_engine::NCLASS;
    constexpr int K = 40;
    for (int c = 0; c < NC; ++c) e->class_skin[c] = e->skin;
    e->skin_tuned = true;   // class_skin now holds the values in use
    const unsigned saved_flags = e->cfg.flags;
    const int64_t launches0 = e->st.kernel_launches;
    e->cfg.flags &= ~MDGB_FLAG_PROFILE;
    const StepParams sp = make_sp(e, dt, true);
    int rc = snapshot(e, false);   // the state the call started from
    unsigned long long trace0[TR_SLOTS];   // the tuning's steps stay out of the phase trace
    if (!rc) {
        CU(cudaMemcpyAsync(trace0, e->trace_buf, sizeof(trace0), cudaMemcpyDeviceToHost, e->stream));
        CU(cudaStreamSynchronize(e->stream));
    }
    cudaEvent_t ev[2] = {nullptr, nullptr};
    if (!rc && (cudaEventCreate(&ev[0]) != cudaSuccess || cudaEventCreate(&ev[1]) != cudaSuccess))
        rc = fail(e, MDGB_ERR_CUDA, "cudaEventCreate failed");
    for (int c = 0; c < NC && !rc; ++c) {
        if (!e->class_ntiles[c]) continue;
        float best = 1e30f;
        double best_skin = e->class_skin[c];
        for (int k = 0; k < 5 && !rc; ++k) {
            e->class_skin[c] = SKIN_FRACTIONS[k] * e->rcmax;
            bool done = false;
            for (int attempt = 0; attempt < 8 && !done && !rc; ++attempt) {
                rc = snapshot(e, true);
                if (!rc) rc = apply_class_skin(e);
                if (!rc) rc = rebuild_lists(e);
                if (!rc) rc = clear_err(e);
                if (rc) break;
                if (cudaEventRecord(ev[0], e->stream) != cudaSuccess) { rc = fail(e, MDGB_ERR_CUDA, "event"); break; }
                rc = run_chunk_kernels(e, sp, K);
                if (rc) break;
                if (cudaEventRecord(ev[1], e->stream) != cudaSuccess) { rc = fail(e, MDGB_ERR_CUDA, "event"); break; }
                int flags = 0;
                rc = read_err(e, &flags);
                if (rc) break;
                if (flags & E_NLIST) {   // longer lists: grow and time this candidate again
                    rc = grow_list(e);
                    continue;
                }
                rc = check_flags(e, flags);
                if (rc) break;
                float ms = 0.f;
                if (cudaEventElapsedTime(&ms, ev[0], ev[1]) != cudaSuccess) { rc = fail(e, MDGB_ERR_CUDA, "event"); break; }
                if (ms < best) { best = ms; best_skin = e->class_skin[c]; }
                done = true;
            }
        }
        e->class_skin[c] = best_skin;
    }
    for (auto& x : ev)
        if (x) cudaEventDestroy(x);
    e->cfg.flags = saved_flags;
    e->st.kernel_launches = launches0;
    if (rc) return rc;
    // back to the starting state; its lists are rebuilt with the chosen skins
    // (a real rebuild, counted and traced like any other)
    CU(cudaMemcpyAsync(e->trace_buf, trace0, sizeof(trace0), cudaMemcpyHostToDevice, e->stream));
    rc = snapshot(e, true);
    if (!rc) rc = apply_class_skin(e);
    if (!rc) rc = rebuild_lists(e);
    return rc;
}

// The lists in the layout of these threads per atom for each size class.
int use_tpa(mdgb_engine* e, const int (&tpa)[mdgb_engine::NCLASS]) {
    const int NC = mdgb_engine::NCLASS;
    for (int c = 0; c < NC; ++c) e->class_tpa[c] = tpa[c];
    e->tpa = tpa[0];
    for (int c = NC - 1; c >= 0; --c)
        if (e->class_ntiles[c]) { e->tpa = tpa[c]; break; }
    e->st.threads_per_atom = e->tpa;
    const int rc = apply_class_tpa(e);
    if (rc) return rc;
    return e->lists_fresh ? MDGB_OK : rebuild_lists(e);
}

int autotune_tpa(mdgb_engine* e);

// Threads per atom for the calls to come.  Sizes of the one-launch kernel take
// one (it shares an atom's list out itself), but what runs as launches there,
// coupled steps of the larger ones and forces alone, is faster with what a timing
// chooses (us, mixed path, one thread / timed: forces of 13,500 atoms 41 / 31, a
// step with both Berendsen couplings 77 / 66).  Changing the layout costs a
// rebuild and the first timing about a millisecond, so it waits for PATIENCE steps
// (a force evaluation is one) that the other layout suits.
constexpr int PATIENCE = 32;
int settle_tpa(mdgb_engine* e, bool launches, int64_t steps) {
    const bool fixed = e->dev.refmode || e->dev.pairs || e->cfg.threads_per_atom > 0;
    if (fixed || small_size(e)) {
        if (!e->tuned) {
            const int t = e->cfg.threads_per_atom > 0 && !e->dev.refmode ? e->cfg.threads_per_atom : 1;
            e->tuned = true;
            e->timed_layout = false;
            e->off_layout = 0;
            const int rc = use_tpa(e, {t, t, t});
            if (rc) return rc;
        }
        if (fixed || e->ntot < TUNE_MIN_ATOMS || launches == e->timed_layout) {
            e->off_layout = 0;
            return MDGB_OK;
        }
        e->off_layout += steps;
        if (e->off_layout < PATIENCE) return MDGB_OK;
        e->off_layout = 0;
        e->timed_layout = launches;
        if (!launches) return use_tpa(e, {1, 1, 1});
        return e->timed ? use_tpa(e, e->timed_tpa) : autotune_tpa(e);
    }
    return e->tuned ? MDGB_OK : autotune_tpa(e);
}

// Threads per atom for each size class: every candidate is timed on every
// class at once (each class's launch bracketed by its own events), and each
// class keeps its fastest.
int autotune_tpa(mdgb_engine* e) {
    e->tuned = true;
    const int NC = mdgb_engine::NCLASS;
    if (!e->lists_fresh) {   // the tuning's rebuilds then keep the atoms' order, and with it the forces'
        const int rc = rebuild_lists(e);
        if (rc) return rc;
    }
    e->lists_fresh = false;
    // Keep the caller's forces: tuning evaluates forces into scratch.
    const size_t N = e->ntot;
    CU(cudaMemcpyAsync(e->snap_d, e->dev.frc, 3 * N * sizeof(double), cudaMemcpyDeviceToDevice, e->stream));
    CU(cudaMemcpyAsync(e->snap_d + 3 * N, e->dev.epot, N * sizeof(double), cudaMemcpyDeviceToDevice, e->stream));
    CU(cudaMemcpyAsync(e->snap_d + 4 * N, e->dev.evir, N * sizeof(double), cudaMemcpyDeviceToDevice, e->stream));
    const int cands[4] = {1, 2, 4, 8};
    float best[NC];
    int best_tpa[NC];
    for (int c = 0; c < NC; ++c) { best[c] = 1e30f; best_tpa[c] = 1; }
    cudaEvent_t ev[NC][2];
    for (int c = 0; c < NC; ++c) { CU(cudaEventCreate(&ev[c][0])); CU(cudaEventCreate(&ev[c][1])); }
    const unsigned saved_flags = e->cfg.flags;
    e->cfg.flags &= ~(MDGB_FLAG_PROFILE | MDGB_FLAG_PERSISTENT);
    StepParams sp = make_sp(e, 0.0, false);
    int rc = MDGB_OK;
    for (int ci = 0; ci < 4 && !rc; ++ci) {
        const int cand = cands[ci];
        if (e->ntot < TUNE_MIN_ATOMS && cand > 1) break;
        for (int c = 0; c < NC; ++c) e->class_tpa[c] = cand;
        rc = apply_class_tpa(e);
        if (!rc) rc = clear_err(e);
        if (!rc) rc = refresh(e, true);
        if (!rc) rc = launch_force(e, sp, false);  // warm-up
        if (rc) break;
        for (int c = 0; c < NC && !rc; ++c) {
            if (!e->class_ntiles[c]) continue;
            CU(cudaEventRecord(ev[c][0], e->stream));
            for (int i = 0; i < 3 && !rc; ++i) rc = launch_force_class(e, sp, false, c, e->stream);
            CU(cudaEventRecord(ev[c][1], e->stream));
        }
        if (rc) break;
        int flags = 0;
        rc = read_err(e, &flags);
        if (rc) break;
        if (flags & E_NLIST) {
            rc = grow_list(e);
            if (!rc) rc = clear_err(e);
            if (e->dev.pairs) {   // the larger list came with pair records: one thread per atom
                for (int c = 0; c < NC; ++c) best_tpa[c] = 1;
                break;
            }
            --ci;  // same candidate again with the larger list
            continue;
        }
        for (int c = 0; c < NC; ++c) {
            if (!e->class_ntiles[c]) continue;
            float ms = 0.f;
            CU(cudaEventElapsedTime(&ms, ev[c][0], ev[c][1]));
            if (ms < best[c]) { best[c] = ms; best_tpa[c] = cand; }
        }
    }
    e->cfg.flags = saved_flags;
    for (int c = 0; c < NC; ++c) { cudaEventDestroy(ev[c][0]); cudaEventDestroy(ev[c][1]); }
    if (rc) return rc;
    for (int c = 0; c < NC; ++c) e->timed_tpa[c] = best_tpa[c];
    e->timed = true;
    CU(cudaMemcpyAsync(e->dev.frc, e->snap_d, 3 * N * sizeof(double), cudaMemcpyDeviceToDevice, e->stream));
    CU(cudaMemcpyAsync(e->dev.epot, e->snap_d + 3 * N, N * sizeof(double), cudaMemcpyDeviceToDevice, e->stream));
    CU(cudaMemcpyAsync(e->dev.evir, e->snap_d + 4 * N, N * sizeof(double), cudaMemcpyDeviceToDevice, e->stream));
    e->lists_fresh = false;
    return use_tpa(e, best_tpa);
}

// Counts of every type per tile (exclusive over the tiles of a replica when
// done, [tile][MAX_TYPES] in *count_out) and each replica's type offsets.
// Refuses a type id >= ntypes and a type without atoms in some replica.
// Few atoms are counted here: the device's two launches and the wait for their
// totals take longer (us an upload, here / device: 195 / 218 at 2,048
// atoms, 176 / 188 at 13,500, 193 / 191 at 23,328, 250 / 216 at 48,668).
constexpr int COUNT_TYPES_HERE = 16384;
int count_types(mdgb_engine* e, int N, const uint16_t* type, int ntypes, const std::vector<int4>& tiles,
                std::vector<RepDev>& reps, int** count_out) {
    const size_t nt = tiles.size(), nr = reps.size();
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t s_cnt = up(nt * MAX_TYPES * sizeof(int)), s_tot = up((nr * MAX_TYPES + 1) * sizeof(int)),
                 s_tiles = up(nt * sizeof(int4)), s_reps = up(nr * sizeof(int2)),
                 s_type = e->host_direct ? 0 : up((size_t)N * sizeof(uint16_t));
    const size_t bytes = s_cnt + s_tot + s_tiles + s_reps + s_type;
    if (bytes > e->type_bytes) {
        if (e->type_buf) cudaFree(e->type_buf);
        e->type_buf = nullptr;
        e->type_bytes = 0;
        CU(cudaMalloc(&e->type_buf, bytes));
        e->type_bytes = bytes;
    }
    char* q = static_cast<char*>(e->type_buf);
    int* count = reinterpret_cast<int*>(q); q += s_cnt;
    int* total = reinterpret_cast<int*>(q); q += s_tot;
    int4* d_tiles = reinterpret_cast<int4*>(q); q += s_tiles;
    int2* d_reps = reinterpret_cast<int2*>(q); q += s_reps;
    std::vector<int> tot(nr * MAX_TYPES + 1, 0);
    if (N <= COUNT_TYPES_HERE) {
        std::vector<int> here(nt * MAX_TYPES);
        for (size_t k = 0; k < nt; ++k) {
            int* t = tot.data() + (size_t)tiles[k].x * MAX_TYPES;
            std::memcpy(&here[k * MAX_TYPES], t, MAX_TYPES * sizeof(int));
            for (int i = tiles[k].y; i < tiles[k].y + tiles[k].z; ++i) {
                if (type[i] >= ntypes) return fail(e, MDGB_ERR_INVALID_ARGUMENT, "type id >= ntypes");
                ++t[type[i]];
            }
        }
        CU(cudaMemcpyAsync(count, here.data(), here.size() * sizeof(int), cudaMemcpyHostToDevice, e->stream));
    } else {
        std::vector<int2> spans(nr);
        for (size_t r = 0; r < nr; ++r) spans[r] = make_int2(reps[r].tile_begin, reps[r].ntiles);
        CU(cudaMemcpyAsync(d_tiles, tiles.data(), nt * sizeof(int4), cudaMemcpyHostToDevice, e->stream));
        CU(cudaMemcpyAsync(d_reps, spans.data(), nr * sizeof(int2), cudaMemcpyHostToDevice, e->stream));
        int* bad = total + nr * MAX_TYPES;
        CU(cudaMemsetAsync(bad, 0, sizeof(int), e->stream));
        const uint16_t* d_type = type;   // read where it lies, as the scatter kernel does
        if (!e->host_direct) {
            CU(cudaMemcpyAsync(q, type, (size_t)N * sizeof(uint16_t), cudaMemcpyHostToDevice, e->stream));
            d_type = reinterpret_cast<const uint16_t*>(q);
        }
        k_type_count<<<(unsigned)nt, TILE, 0, e->stream>>>(d_tiles, d_type, ntypes, count, bad);
        k_type_scan<<<(unsigned)nr, 256, 0, e->stream>>>(d_reps, ntypes, count, total);
        CU(cudaGetLastError());
        CU(cudaMemcpyAsync(tot.data(), total, tot.size() * sizeof(int), cudaMemcpyDeviceToHost, e->stream));
        CU(cudaStreamSynchronize(e->stream));
        if (tot.back()) return fail(e, MDGB_ERR_INVALID_ARGUMENT, "type id >= ntypes");
    }
    for (size_t r = 0; r < nr; ++r) {
        RepDev& R = reps[r];
        for (int t = 0; t < ntypes; ++t) {
            const int c = tot[r * MAX_TYPES + t];
            if (c == 0)
                return fail(e, MDGB_ERR_INVALID_ARGUMENT,
                            "every type 0..ntypes-1 needs at least one atom in every replica "
                            "(the reference indexes particles[type][0])");
            R.type_off[t + 1] = R.type_off[t] + c;
            R.last_type_count = c;
        }
    }
    *count_out = count;
    return MDGB_OK;
}

// Upload of a state (one replica or an ensemble).  An upload whose shape
// (atoms, replicas, tiles, cells, reduction chunks) equals the previous one
// keeps the device allocations, the neighbour list (if large enough), the
// tuned threads per atom and the captured graphs; anything else starts over.
// The caller's arrays are copied straight to the device (pageable memory is
// fine) and scattered into the device layout by a kernel.
int upload_impl(mdgb_engine* e, int nrep, const int64_t* offsets, const uint16_t* type, const double* pos,
                const double* vel, const double* mass_per_type, int ntypes, const double* boxes) {
    if (nrep < 1 || !offsets || !type || !pos || !mass_per_type || !boxes)
        return fail(e, MDGB_ERR_INVALID_ARGUMENT, "null argument");
    if (ntypes < 1 || ntypes > MAX_TYPES)
        return fail(e, MDGB_ERR_INVALID_ARGUMENT, "ntypes must be in 1..16");
    const int64_t n = offsets[nrep];
    if (offsets[0] != 0 || n < 1 || n >= (int64_t)IDX_MASK)
        return fail(e, MDGB_ERR_INVALID_ARGUMENT, "bad offsets / atom count");
    for (int r = 0; r < nrep; ++r) {
        if (offsets[r + 1] <= offsets[r]) return fail(e, MDGB_ERR_INVALID_ARGUMENT, "empty replica");
        for (int a = 0; a < 3; ++a)
            if (!(boxes[3 * r + a] > 0.0) || !std::isfinite(boxes[3 * r + a]))
                return fail(e, MDGB_ERR_INVALID_ARGUMENT, "box must be positive and finite");
    }
    for (int t = 0; t < ntypes; ++t)
        if (!(mass_per_type[t] > 0.0)) return fail(e, MDGB_ERR_INVALID_ARGUMENT, "mass must be positive");
    const int N = (int)n;

    // tiles of each replica, and its type offsets (the reference's order is
    // type-major).  With one type the rank is the index itself and the type ids
    // are checked by the scatter kernel; with several the device counts the
    // types per tile and scans the counts, which gives the scatter kernel every
    // atom's rank (a loop over the atoms here took 1.3 ms of a 500,000-atom
    // frame's 2.8).
    std::vector<RepDev> reps(nrep, RepDev{});
    std::vector<int4> tiles;
    for (int r = 0; r < nrep; ++r) {
        RepDev& R = reps[r];
        const int nr = (int)(offsets[r + 1] - offsets[r]);
        R.begin = offsets[r];
        R.n = nr;
        R.tile_begin = (int)tiles.size();
        for (int b = 0; b < nr; b += TILE) tiles.push_back(make_int4(r, (int)(offsets[r] + b), std::min(TILE, nr - b), 0));
        R.ntiles = (int)tiles.size() - R.tile_begin;
        R.type_off[0] = 0;
        for (int t = 1; t <= MAX_TYPES; ++t) R.type_off[t] = nr;
        R.last_type_count = nr;
    }
    int* d_type_count = nullptr;
    if (ntypes > 1) {
        const int rc = count_types(e, N, type, ntypes, tiles, reps, &d_type_count);
        if (rc) return rc;
    }

    // potentials and list radius (host side: the cell capacity depends on it)
    e->ntypes = ntypes;
    e->dev.ntypes = ntypes;
    const std::vector<PairDev> pair_tab = pair_table(e);

    // tiles and cells (cell capacity for the smallest list radius the skin
    // tuning may choose)
    const bool auto_skin = skin_auto(e);
    const double rl_cells = e->rcmax + (auto_skin ? std::min(e->skin, SKIN_FRACTIONS[0] * e->rcmax) : e->skin);
    std::vector<int> cell_rep;
    int max_rep_n = 0;
    double max_density = 0.0, atom_density = 0.0;
    for (int r = 0; r < nrep; ++r) {
        RepDev& R = reps[r];
        const int nr = (int)(offsets[r + 1] - offsets[r]);
        max_rep_n = std::max(max_rep_n, nr);
        double prod = 1.0;
        for (int a = 0; a < 3; ++a) {
            const double L = boxes[3 * r + a];
            R.box[a] = L; R.box_build[a] = L; R.cs[a] = L; R.inv_cs[a] = 1.0 / L; R.nc[a] = 1;
            prod *= std::max(1.0, std::floor(L / (rl_cells * (1.0 + 1e-6))));
        }
        const double vol = boxes[3 * r] * boxes[3 * r + 1] * boxes[3 * r + 2];
        max_density = std::max(max_density, nr / vol);
        atom_density += nr * (nr / vol);
        // cell capacity: the grid at this box with room to grow (barostat), but
        // no finer than ~8 atoms a cell -- a dilute replica gets larger
        // cells, so its rebuild is not dominated by per-cell work
        const double capd = std::min(std::ceil(prod * 1.3) + 27.0, nr / 8.0 + 27.0);
        R.cell_cap = (int)std::max(27.0, capd);
        R.cell_base = (int)cell_rep.size();
        cell_rep.insert(cell_rep.end(), R.cell_cap, r);
        R.mode = MODE_BRUTE;
        R.pending = 1.0;
        R.lambda = 0.0;
        R.myu = 0.0;
        R.rebuild = 1;
    }
    const int ntiles = (int)tiles.size();
    const int ncells = (int)cell_rep.size();
    // reduction chunks: runs of <= CHUNK_TILES tiles inside one replica
    std::vector<int4> chunks;
    for (int r = 0; r < nrep; ++r) {
        RepDev& R = reps[r];
        R.chunk_begin = (int)chunks.size();
        for (int t = 0; t < R.ntiles; t += CHUNK_TILES)
            chunks.push_back(make_int4(r, R.tile_begin + t, std::min(CHUNK_TILES, R.ntiles - t), 0));
        R.nchunks = (int)chunks.size() - R.chunk_begin;
    }

    // size classes by replica atom count; tile_order = class 0 tiles, class 1, class 2,
    // costliest (densest replica) first inside a class (persistent kernel)
    constexpr int NC = mdgb_engine::NCLASS;
    std::vector<int> class_of(nrep, 0);
    int class_ntiles[NC] = {0, 0, 0}, class_nrep[NC] = {0, 0, 0};
    for (int r = 0; r < nrep; ++r) {
        const int nr = reps[r].n;
        const int c = nr < 2048 ? 0 : (nr < 32768 ? 1 : 2);
        class_of[r] = c;
        reps[r].size_class = c;
        class_nrep[c]++;
        class_ntiles[c] += reps[r].ntiles;
    }
    std::vector<int> order(ntiles);
    for (int i = 0; i < ntiles; ++i) order[i] = i;
    if (nrep > 1) {
        // expected pair work of a tile: its atoms x the replica's neighbours per atom
        const double sphere = 4.0 / 3.0 * M_PI * e->rlist * e->rlist * e->rlist;
        std::vector<double> rep_cost(nrep);
        for (int r = 0; r < nrep; ++r) {
            const RepDev& R = reps[r];
            const double dens = R.n / (R.box[0] * R.box[1] * R.box[2]);
            rep_cost[r] = std::min((double)R.n, 1.0 + dens * sphere);
        }
        struct Key { int cls; double cost; int tile; };
        std::vector<Key> key(ntiles);
        for (int i = 0; i < ntiles; ++i) key[i] = {class_of[tiles[i].x], tiles[i].z * rep_cost[tiles[i].x], i};
        std::stable_sort(key.begin(), key.end(), [](const Key& a, const Key& b) {
            return a.cls != b.cls ? a.cls < b.cls : a.cost > b.cost;
        });
        for (int i = 0; i < ntiles; ++i) order[i] = key[i].tile;
    }

    // keep the allocations when the shape is unchanged
    Dev& d = e->dev;
    const bool reuse = e->has_state && N == e->ntot && nrep == e->nrep && ntiles == e->ntiles &&
                       ncells == e->ncells && (int)chunks.size() == d.nchunks;
    bool same_classes = reuse;
    for (int c = 0; c < NC; ++c)
        same_classes = same_classes && class_ntiles[c] == e->class_ntiles[c] && class_nrep[c] == e->class_nrep[c];
    if (!reuse) free_state(e);
    if (!same_classes) e->skin_tuned = false;
    e->has_state = false;
    e->forces_valid = false;
    e->lists_fresh = false;
    e->ntot = N;
    e->nrep = nrep;
    e->ntiles = ntiles;
    e->ncells = ncells;
    e->offsets.assign(offsets, offsets + nrep + 1);
    e->mass.assign(mass_per_type, mass_per_type + ntypes);
    e->rep_host = reps;
    e->class_of = class_of;
    for (int c = 0; c < NC; ++c) { e->class_ntiles[c] = class_ntiles[c]; e->class_nrep[c] = class_nrep[c]; }
    e->class_tile_off[0] = 0;
    for (int c = 1; c < NC; ++c) e->class_tile_off[c] = e->class_tile_off[c - 1] + e->class_ntiles[c - 1];

    d.ntot = N; d.ntiles = ntiles; d.nrep = nrep; d.ncells = ncells;
    d.refmode = (e->cfg.flags & MDGB_FLAG_REFERENCE_ORDER) && e->cfg.precision == MDGB_PRECISION_FP64 ? 1 : 0;
    d.mixed = e->cfg.precision != MDGB_PRECISION_FP64 ? 1 : 0;
    d.single_type = ntypes == 1 ? 1 : 0;
    d.direct_list = (e->cfg.flags & MDGB_FLAG_DIRECT_LIST) ? 1 : 0;
    d.last_type = ntypes - 1;
    for (int t = 0; t < MAX_TYPES; ++t) d.mass[t] = t < ntypes ? mass_per_type[t] : 1.0;

    int rc = MDGB_OK;
    if (!reuse) {
        if ((rc = dalloc(e, (PairDev**)&d.pair, MAX_TYPES * MAX_TYPES)) ||
            (rc = dalloc(e, &d.pos, N)) || (rc = dalloc(e, &d.vel, 3 * (size_t)N)) ||
            (rc = dalloc(e, &d.frc, 3 * (size_t)N)) || (rc = dalloc(e, &d.epot, N)) ||
            (rc = dalloc(e, &d.evir, N)) || (rc = dalloc(e, &d.mir, N)) || (rc = dalloc(e, &d.mir0, N)) ||
            (rc = dalloc(e, &e->pos_alt, N)) || (rc = dalloc(e, &e->mir_alt, N)) ||
            (rc = dalloc(e, &d.band_list, N)) || (rc = dalloc(e, &d.band_count, 1)) ||
            (rc = dalloc(e, &d.cell, N)) || (rc = dalloc(e, &d.orig, N)) || (rc = dalloc(e, &d.rank, N)) ||
            (rc = dalloc(e, &d.nn, N)) || (rc = dalloc(e, &d.tiles, ntiles)) ||
            (rc = dalloc(e, &d.rep, nrep)) || (rc = dalloc(e, &d.part, 8 * (size_t)ntiles)) ||
            (rc = dalloc(e, &d.cpart, 8 * chunks.size())) || (rc = dalloc(e, &d.chunks, chunks.size())) ||
            (rc = dalloc(e, &d.fx_part, ntiles)) ||
            (rc = dalloc(e, &d.err, 2)) || (rc = dalloc(e, &d.max_needed, 1)) ||
            (rc = dalloc(e, &d.cell_count, ncells)) ||
            (rc = dalloc(e, &d.cell_start, ncells + 1)) || (rc = dalloc(e, &d.cell_rep, ncells)) ||
            (rc = dalloc(e, &d.perm, N)) || (rc = dalloc(e, &d.tmp_pos, N)) ||
            (rc = dalloc(e, &d.tmp_d, 8 * ((size_t)N + (d.refmode ? (size_t)SS_PAD * nrep : 0)))) || (rc = dalloc(e, &d.tmp_i, 4 * (size_t)N)) ||
            (rc = dalloc(e, &d.slot_of_rank, N)) || (rc = dalloc(e, &d.bsum, 4096)) ||
            (rc = dalloc(e, &d.lmask, 27 * (size_t)N)) || (rc = dalloc(e, &d.nbs, 27 * (size_t)ncells)) ||
            (rc = dalloc(e, &d.rb, 4 + 3 * (size_t)nrep)) ||
            (rc = dalloc(e, &d.bar, 8)) || (rc = dalloc(e, &d.queue, NC)) ||
            (rc = dalloc(e, &e->trace_buf, TR_SLOTS)) ||
            (rc = dalloc(e, &d.tile_order, ntiles)) ||
            (rc = dalloc(e, &e->snap_pos, N)) || (rc = dalloc(e, &e->snap_d, 8 * (size_t)N)) ||
            (rc = dalloc(e, &e->snap_i, 4 * (size_t)N)) || (rc = dalloc(e, &e->snap_mir0, N)) ||
            (rc = dalloc(e, &e->snap_rep, nrep)) || (rc = dalloc(e, &e->d_out, 11 * (size_t)N)) ||
            (rc = dalloc(e, &e->d_in_t, N)))
            return rc;
    }
    if (!e->h_pin) {
        CU(cudaMallocHost((void**)&e->h_pin, PIN_HEAD + PIN_OUT));
        e->h_err = reinterpret_cast<int*>(e->h_pin);
        e->h_rep = reinterpret_cast<RepDev*>(e->h_pin + 64);
    }
    e->coupling_set = false;
    e->rep_fresh = false;
    CU(cudaMemcpyAsync((void*)d.pair, pair_tab.data(), pair_tab.size() * sizeof(PairDev), cudaMemcpyHostToDevice,
                       e->stream));

    // threads per atom: kept from the last tuning when the size classes are
    // the same, else the configured (or default) value until the next tuning
    // (before the list is allocated: the pair records go by it)
    if (!same_classes) {
        const int t0 = d.refmode ? 1 : (e->cfg.threads_per_atom > 0 ? e->cfg.threads_per_atom : 1);
        for (int c = 0; c < NC; ++c) e->class_tpa[c] = t0;
        e->tuned = e->timed = false;
    }

    e->mean_density = atom_density / N;
    // neighbour capacity from the densest replica (grows on overflow)
    int cap = e->cfg.neighbor_capacity;
    if (cap <= 0) {
        const double expect = 4.0 / 3.0 * M_PI * std::pow(e->rlist * (1.0 + 1e-5), 3) * max_density;
        cap = (int)std::ceil(expect * 1.35 + 16.0);
        cap = std::min(cap, std::max(max_rep_n - 1, 8));
    }
    cap = std::max(8, (cap + 7) & ~7);
    if (!e->nbr_alloc || cap > e->cap) {
        rc = alloc_nbr(e, cap);
        if (rc) return rc;
    } else if (e->pair_single != d.single_type || e->pair_wanted != pairs_wanted(e)) {
        // as many records as list entries with several types; none for a gas
        alloc_pairs(e);
    }
    e->st = mdgb_stats{};
    e->st.neighbor_capacity = e->cap;

    for (int r = 0; r < nrep; ++r) {
        e->rep_host[r].tpa = e->class_tpa[e->class_of[r]];
        e->rep_host[r].rlist = e->rcmax + class_skin_of(e, e->class_of[r]);
    }
    update_rlist(e);
    e->tpa = e->class_tpa[0];
    for (int c = NC - 1; c >= 0; --c)
        if (e->class_ntiles[c]) { e->tpa = e->class_tpa[c]; break; }
    d.tpa = e->tpa;

    CU(cudaMemcpyAsync(d.tiles, tiles.data(), tiles.size() * sizeof(int4), cudaMemcpyHostToDevice, e->stream));
    d.nchunks = (int)chunks.size();
    CU(cudaMemcpyAsync(d.chunks, chunks.data(), chunks.size() * sizeof(int4), cudaMemcpyHostToDevice, e->stream));
    CU(cudaMemcpyAsync(d.tile_order, order.data(), order.size() * sizeof(int), cudaMemcpyHostToDevice, e->stream));
    CU(cudaMemcpyAsync(d.cell_rep, cell_rep.data(), cell_rep.size() * sizeof(int), cudaMemcpyHostToDevice, e->stream));
    CU(cudaMemsetAsync(d.cell_count, 0, ncells * sizeof(int), e->stream));
    CU(cudaMemsetAsync(d.max_needed, 0, sizeof(int), e->stream));
    CU(cudaMemsetAsync(e->trace_buf, 0, TR_SLOTS * sizeof(unsigned long long), e->stream));
    d.trace = (e->cfg.flags & MDGB_FLAG_TRACE) ? e->trace_buf : nullptr;
    CU(cudaMemsetAsync(d.err, 0, 2 * sizeof(int), e->stream));
    CU(cudaMemsetAsync(d.bar, 0, 8 * sizeof(unsigned int), e->stream));
    CU(cudaMemsetAsync(d.rb, 0, (4 + 3 * (size_t)nrep) * sizeof(int), e->stream));
    CU(cudaMemcpyAsync(d.rep, e->rep_host.data(), nrep * sizeof(RepDev), cudaMemcpyHostToDevice, e->stream));
    // the caller's arrays: read by the scatter kernel where they lie (the
    // GPU reaches pageable host memory), else copied to the device staging
    // first.  Either way they are done with before this call returns (the
    // list rebuild below synchronises).
    const double* dpos = pos;
    const double* vptr = vel;
    const uint16_t* tptr = type;
    if (!e->host_direct) {
        double* spos = e->d_out;
        double* svel = e->d_out + 3 * (size_t)N;
        CU(cudaMemcpyAsync(spos, pos, 3 * (size_t)N * sizeof(double), cudaMemcpyHostToDevice, e->stream));
        if (vel) CU(cudaMemcpyAsync(svel, vel, 3 * (size_t)N * sizeof(double), cudaMemcpyHostToDevice, e->stream));
        CU(cudaMemcpyAsync(e->d_in_t, type, (size_t)N * sizeof(uint16_t), cudaMemcpyHostToDevice, e->stream));
        dpos = spos;
        vptr = vel ? svel : nullptr;
        tptr = e->d_in_t;
    }
    int nt = ntypes;
    void* args[] = {(void*)&e->dev, (void*)&dpos, (void*)&vptr, (void*)&tptr, (void*)&d_type_count, (void*)&nt};
    CU(cudaLaunchKernel((const void*)k_scatter_in, dim3(ntiles), dim3(TILE), args, 0, e->stream));
    // the kernel may read the caller's arrays: done before anything below can
    // return
    if (e->host_direct && ntypes > 1) CU(cudaStreamSynchronize(e->stream));
    e->thermo_on = e->baro_on = e->thermo_nh = false;
    if (ntypes == 1) {   // the type ids were checked on the device
        int flags = 0;
        rc = read_err(e, &flags);
        if (rc) return rc;
        if (flags) return check_flags(e, flags);
    }
    e->has_state = true;
    // bin and build lists now, so a bare mdgb_step starts from a valid list
    return rebuild_lists(e);
}

int set_coupling_impl(mdgb_engine* e, const mdgb_thermostat* th, const mdgb_barostat* ba) {
    if (!e->has_state) return fail(e, MDGB_ERR_NO_STATE, "no state uploaded");
    e->rep_fresh = false;
    if (!th && !ba && !e->coupling_set) return MDGB_OK;   // off already
    if (e->nrep == 1) {
        RepCoupling c{};
        c.thermo_on = th ? 1 : 0;
        if (th) {
            if (th->kind != MDGB_THERMOSTAT_BERENDSEN && th->kind != MDGB_THERMOSTAT_NOSE_HOOVER)
                return fail(e, MDGB_ERR_INVALID_ARGUMENT, "unknown thermostat kind");
            c.thermo_kind = th->kind;
            c.th_tau = th->tau; c.th_T0 = th->target_temperature; c.lambda = th->lambda; c.psi = th->psi;
        }
        c.baro_on = ba ? 1 : 0;
        if (ba) { c.ba_beta = ba->beta; c.ba_tau = ba->tau; c.ba_P0 = ba->target_pressure; c.myu = ba->myu; }
        e->thermo_nh = th && th->kind == MDGB_THERMOSTAT_NOSE_HOOVER;
        e->thermo_on = th != nullptr;
        e->baro_on = ba != nullptr;
        e->coupling_set = th || ba;
        void* args[] = {(void*)&e->dev, (void*)&c};
        CU(cudaLaunchKernel((const void*)k_set_coupling, dim3(1), dim3(32), args, 0, e->stream));
        return MDGB_OK;
    }
    e->coupling_set = th || ba;
    CU(cudaMemcpyAsync(e->rep_host.data(), e->dev.rep, e->nrep * sizeof(RepDev), cudaMemcpyDeviceToHost, e->stream));
    CU(cudaStreamSynchronize(e->stream));
    bool any_nh = false;
    for (int r = 0; r < e->nrep; ++r) {
        RepDev& R = e->rep_host[r];
        R.thermo_on = th ? 1 : 0;
        if (th) {
            if (th[r].kind != MDGB_THERMOSTAT_BERENDSEN && th[r].kind != MDGB_THERMOSTAT_NOSE_HOOVER)
                return fail(e, MDGB_ERR_INVALID_ARGUMENT, "unknown thermostat kind");
            if (th[r].kind == MDGB_THERMOSTAT_NOSE_HOOVER) any_nh = true;
            R.thermo_kind = th[r].kind;
            R.th_tau = th[r].tau; R.th_T0 = th[r].target_temperature;
            R.lambda = th[r].lambda; R.psi = th[r].psi;
        }
        R.baro_on = ba ? 1 : 0;
        if (ba) {
            R.ba_beta = ba[r].beta; R.ba_tau = ba[r].tau; R.ba_P0 = ba[r].target_pressure;
            R.myu = ba[r].myu;
        }
    }
    e->thermo_nh = any_nh;
    e->thermo_on = th != nullptr;
    e->baro_on = ba != nullptr;
    CU(cudaMemcpyAsync(e->dev.rep, e->rep_host.data(), e->nrep * sizeof(RepDev), cudaMemcpyHostToDevice, e->stream));
    return MDGB_OK;
}

int get_coupling_impl(mdgb_engine* e, mdgb_thermostat* th, mdgb_barostat* ba) {
    if (!th && !ba) return MDGB_OK;
    if (e->nrep == 1 && e->rep_fresh) {
        if (th) { th->lambda = e->h_rep->lambda; th->psi = e->h_rep->psi; }
        if (ba) ba->myu = e->h_rep->myu;
        return MDGB_OK;
    }
    CU(cudaMemcpyAsync(e->rep_host.data(), e->dev.rep, e->nrep * sizeof(RepDev), cudaMemcpyDeviceToHost, e->stream));
    CU(cudaStreamSynchronize(e->stream));
    for (int r = 0; r < e->nrep; ++r) {
        const RepDev& R = e->rep_host[r];
        if (th) { th[r].lambda = R.lambda; th[r].psi = R.psi; }
        if (ba) ba[r].myu = R.myu;
    }
    return MDGB_OK;
}

// The caller's output pages that are mapped, marked accessed by host threads
// before the device writes them.  The GPU reaches pageable memory through the
// host's page tables and takes a page whose access flag the host has cleared
// since its last use as a fault of about 10 us, one after the other: an
// 8M-atom state (704 MB) took 4.2 ms to copy where no flag was cleared and 30
// to 100 ms where many were.  A host thread sets a flag in about 0.1 us.  Pages
// not mapped yet (a buffer's first use) are left to the device, which gets
// them in 26 to 58 ms for that state where host threads took 250 ms.  The
// contents stay; the copies are issued after the threads are done.  Below
// MIN_BYTES the time this takes shows (0.1 ms of 8 at 88 MB) and what it saves
// does not.
void settle_pages(const std::vector<std::pair<char*, size_t>>& out) {
    constexpr size_t MIN_BYTES = size_t(128) << 20;
    constexpr size_t PAGES_PER_THREAD = 2048;
    size_t total = 0;
    for (auto& o : out) total += o.second;
    const long ps = sysconf(_SC_PAGESIZE);
    if (total < MIN_BYTES || ps <= 0) return;
    const size_t page = (size_t)ps;
    std::vector<std::thread> pool;
    try {
        struct Run { char* base; std::vector<unsigned char> mapped; };
        std::vector<Run> runs;
        size_t pages = 0;
        for (auto& o : out) {
            // whole pages inside the buffer (its ragged ends stay as they are)
            char* b = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(o.first) + page - 1) / page * page);
            char* e = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(o.first) + o.second) / page * page);
            if (e <= b) continue;
            Run r{b, std::vector<unsigned char>((size_t)(e - b) / page)};
            if (mincore(b, (size_t)(e - b), r.mapped.data()) != 0) continue;
            pages += r.mapped.size();
            runs.push_back(std::move(r));
        }
        const size_t nt = std::max<size_t>(1, std::min({(size_t)8, (size_t)std::thread::hardware_concurrency(),
                                                         pages / PAGES_PER_THREAD}));
        auto work = [&runs, page, nt](size_t t) {
            for (const Run& r : runs) {
                const size_t n = r.mapped.size();
                for (size_t k = n * t / nt; k < n * (t + 1) / nt; ++k)
                    if (r.mapped[k] & 1) {
                        volatile char* p = r.base + k * page;
                        *p = *p;
                    }
            }
        };
        try {
            for (size_t t = 1; t < nt; ++t) pool.emplace_back(work, t);
        } catch (...) {   // no thread to be had: its pages stay as they are
        }
        work(0);
        for (auto& th : pool) th.join();
    } catch (...) {       // out of memory: the copies work all the same
    }
}

// The requested arrays gathered into the caller's order on the device, then
// copied straight into the caller's buffers (pageable memory is fine).
int download_impl(mdgb_engine* e, double* pos, double* vel, double* force, double* pot, double* temp,
                  double* boxes) {
    if (!e->has_state) return fail(e, MDGB_ERR_NO_STATE, "no state uploaded");
    const size_t N = e->ntot;
    double* o = e->d_out;
    double* op = pos ? o : nullptr;
    double* ov = vel ? o + 3 * N : nullptr;
    double* of = force ? o + 6 * N : nullptr;
    double* oe = pot ? o + 9 * N : nullptr;
    double* ot = temp ? o + 10 * N : nullptr;
    if (op || ov || of || oe || ot) {
        void* args[] = {(void*)&e->dev, (void*)&op, (void*)&ov, (void*)&of, (void*)&oe, (void*)&ot};
        CU(cudaLaunchKernel((const void*)k_gather_out, dim3((unsigned)((N + 255) / 256)), dim3(256), args, 0,
                            e->stream));
    }
    const size_t span = 11 * N * sizeof(double);
    if (span <= PIN_OUT && e->nrep == 1) {
        // small: everything gathered in one copy (and the record with it), then
        // the host's own
        double* hp = reinterpret_cast<double*>(e->h_pin + PIN_HEAD);
        if (op || ov || of || oe || ot) CU(cudaMemcpyAsync(hp, o, span, cudaMemcpyDeviceToHost, e->stream));
        if (boxes) CU(cudaMemcpyAsync(e->h_rep, e->dev.rep, sizeof(RepDev), cudaMemcpyDeviceToHost, e->stream));
        CU(cudaStreamSynchronize(e->stream));
        if (pos) std::memcpy(pos, hp, 3 * N * sizeof(double));
        if (vel) std::memcpy(vel, hp + 3 * N, 3 * N * sizeof(double));
        if (force) std::memcpy(force, hp + 6 * N, 3 * N * sizeof(double));
        if (pot) std::memcpy(pot, hp + 9 * N, N * sizeof(double));
        if (temp) std::memcpy(temp, hp + 10 * N, N * sizeof(double));
        if (boxes)
            for (int a = 0; a < 3; ++a) boxes[a] = e->h_rep->box[a];
        return MDGB_OK;
    }
    if (e->host_direct) {
        std::vector<std::pair<char*, size_t>> out;
        auto add = [&](double* p, size_t doubles) {
            if (p) out.emplace_back(reinterpret_cast<char*>(p), doubles * sizeof(double));
        };
        add(pos, 3 * N); add(vel, 3 * N); add(force, 3 * N); add(pot, N); add(temp, N);
        settle_pages(out);
    }
    if (pos) CU(cudaMemcpyAsync(pos, op, 3 * N * sizeof(double), cudaMemcpyDeviceToHost, e->stream));
    if (vel) CU(cudaMemcpyAsync(vel, ov, 3 * N * sizeof(double), cudaMemcpyDeviceToHost, e->stream));
    if (force) CU(cudaMemcpyAsync(force, of, 3 * N * sizeof(double), cudaMemcpyDeviceToHost, e->stream));
    if (pot) CU(cudaMemcpyAsync(pot, oe, N * sizeof(double), cudaMemcpyDeviceToHost, e->stream));
    if (temp) CU(cudaMemcpyAsync(temp, ot, N * sizeof(double), cudaMemcpyDeviceToHost, e->stream));
    if (boxes)
        CU(cudaMemcpyAsync(e->rep_host.data(), e->dev.rep, e->nrep * sizeof(RepDev), cudaMemcpyDeviceToHost,
                           e->stream));
    CU(cudaStreamSynchronize(e->stream));
    if (boxes)
        for (int r = 0; r < e->nrep; ++r)
            for (int a = 0; a < 3; ++a) boxes[3 * r + a] = e->rep_host[r].box[a];
    return MDGB_OK;
}

int macro_impl(mdgb_engine* e, int type, mdgb_macro* out) {
    if (!e->has_state) return fail(e, MDGB_ERR_NO_STATE, "no state uploaded");
    if (type < 0 || type >= e->ntypes) return fail(e, MDGB_ERR_INVALID_ARGUMENT, "type out of range");
    if (!out) return fail(e, MDGB_ERR_INVALID_ARGUMENT, "null output");
    int rc = clear_err(e);
    if (rc) return rc;
    StepParams sp = make_sp(e, 0.0, false);
    cudaLaunchConfig_t lc{};
    // no more blocks than its rounds over the tiles need: 256,000 atoms (2,000
    // tiles, three rounds) took 91 us on 912 blocks, 82 on 760
    const int maxg = pre_grid(e, e->macro_blocks_per_sm), rounds = (e->ntiles + maxg - 1) / maxg;
    lc.gridDim = dim3(e->dev.refmode ? maxg : std::max(1, (e->ntiles + rounds - 1) / rounds));
    lc.blockDim = dim3(TILE);
    lc.stream = e->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    lc.attrs = at;
    lc.numAttrs = 1;
    CU(cudaLaunchKernelEx(&lc, k_macro, e->dev, sp, type));
    e->st.kernel_launches++;
    int flags = 0;
    rc = read_err(e, &flags);
    if (rc) return rc;
    rc = check_flags(e, flags);
    if (rc) return rc;
    CU(cudaMemcpyAsync(e->rep_host.data(), e->dev.rep, e->nrep * sizeof(RepDev), cudaMemcpyDeviceToHost, e->stream));
    CU(cudaStreamSynchronize(e->stream));
    for (int r = 0; r < e->nrep; ++r) {
        const RepDev& R = e->rep_host[r];
        mdgb_macro& m = out[r];
        m.kinetic_energy = R.ke;
        m.potential_energy = R.pe;
        m.thermal_energy = R.thermal;
        m.temperature = R.T;
        m.pressure = R.P;
        for (int a = 0; a < 3; ++a) { m.com_velocity[a] = R.vcm[a]; m.momentum[a] = R.mom[a]; }
        m.count = R.count;
    }
    return MDGB_OK;
}

}  // namespace

mdgb_engine::~mdgb_engine() {
    free_state(this);
    for (auto& p : prof) { cudaEventDestroy(p.a); cudaEventDestroy(p.b); }
    for (auto& p : prof_free) { cudaEventDestroy(p.a); cudaEventDestroy(p.b); }
    if (h_pin) cudaFreeHost(h_pin);
    if (type_buf) cudaFree(type_buf);
    for (int c = 0; c < 3; ++c) {
        if (aux[c]) cudaStreamDestroy(aux[c]);
        if (join_ev[c]) cudaEventDestroy(join_ev[c]);
    }
    if (fork_ev) cudaEventDestroy(fork_ev);
    if (stream) cudaStreamDestroy(stream);
}

// ===========================================================================
extern "C" {

MDGB_API int mdgb_abi_version(void) { return MDGB_ABI_VERSION; }

MDGB_API int mdgb_config_default(mdgb_config* cfg) {
    if (!cfg) return MDGB_ERR_INVALID_ARGUMENT;
    *cfg = mdgb_config{};
    cfg->precision = MDGB_PRECISION_MIXED;
    cfg->skin = 0.0;
    cfg->rebuild_every = 0;
    cfg->threads_per_atom = 0;
    cfg->graph_steps = 0;
    cfg->neighbor_capacity = 0;
    cfg->device = 0;
    cfg->flags = 0;
    return MDGB_OK;
}

MDGB_API int mdgb_create(const mdgb_config* cfg, mdgb_engine** out) {
    if (!out) return MDGB_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    mdgb_config c;
    if (cfg) c = *cfg; else mdgb_config_default(&c);
    if (c.precision != MDGB_PRECISION_FP64 && c.precision != MDGB_PRECISION_MIXED &&
        c.precision != MDGB_PRECISION_FP32_NAIVE)
        return MDGB_ERR_INVALID_ARGUMENT;
    if (c.threads_per_atom != 0 && c.threads_per_atom != 1 && c.threads_per_atom != 2 &&
        c.threads_per_atom != 4 && c.threads_per_atom != 8)
        return MDGB_ERR_INVALID_ARGUMENT;
    if ((c.flags & MDGB_FLAG_REFERENCE_ORDER) && c.precision == MDGB_PRECISION_FP64) c.threads_per_atom = 1;
    mdgb_engine* e = new mdgb_engine();
    e->cfg = c;
    e->device = c.device;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        delete e;
        return MDGB_ERR_CUDA;
    }
    if (cudaSetDevice(c.device) != cudaSuccess) { delete e; return MDGB_ERR_CUDA; }
    cudaDeviceProp prop;
    cudaGetDeviceProperties(&prop, c.device);
    if (!prop.cooperativeLaunch) { delete e; return MDGB_ERR_UNSUPPORTED; }
    e->num_sms = prop.multiProcessorCount;
    {
        int pageable = 0, host_tables = 0;
        cudaDeviceGetAttribute(&pageable, cudaDevAttrPageableMemoryAccess, c.device);
        cudaDeviceGetAttribute(&host_tables, cudaDevAttrPageableMemoryAccessUsesHostPageTables, c.device);
        e->host_direct = pageable == 1 && host_tables == 1;
    }
    if (cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking) != cudaSuccess) { delete e; return MDGB_ERR_CUDA; }
    for (int c = 0; c < mdgb_engine::NCLASS; ++c)
        if (cudaStreamCreateWithFlags(&e->aux[c], cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&e->join_ev[c], cudaEventDisableTiming) != cudaSuccess) {
            delete e;
            return MDGB_ERR_CUDA;
        }
    if (cudaEventCreateWithFlags(&e->fork_ev, cudaEventDisableTiming) != cudaSuccess) { delete e; return MDGB_ERR_CUDA; }
    int bps = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, (const void*)k_pre, TILE, 0);
    int bps2 = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps2, (const void*)k_macro, TILE, 0);
    e->pre_blocks_per_sm = std::max(1, bps);
    e->macro_blocks_per_sm = std::max(1, bps2);
    if (steps_init(&e->steps_blocks_per_sm) != cudaSuccess) { delete e; return MDGB_ERR_CUDA; }
    if (list_build_init() != cudaSuccess) { cudaGetLastError(); delete e; return MDGB_ERR_CUDA; }
    lj_finish(e->pot_default);
    *out = e;
    return MDGB_OK;
}

MDGB_API int mdgb_destroy(mdgb_engine* e) {
    if (!e) return MDGB_ERR_INVALID_ARGUMENT;
    cudaSetDevice(e->device);
    if (e->stream) cudaStreamSynchronize(e->stream);
    delete e;
    return MDGB_OK;
}

MDGB_API const char* mdgb_last_error(const mdgb_engine* e) { return e ? e->err.c_str() : ""; }

MDGB_API const char* mdgb_status_string(int s) {
    switch (s) {
        case MDGB_OK: return "ok";
        case MDGB_ERR_INVALID_ARGUMENT: return "invalid argument";
        case MDGB_ERR_CUDA: return "CUDA error";
        case MDGB_ERR_NO_STATE: return "no state uploaded";
        case MDGB_ERR_NEIGHBOR_OVERFLOW: return "neighbour list overflow";
        case MDGB_ERR_FIXED_POINT_OVERFLOW: return "fixed-point force overflow";
        case MDGB_ERR_UNSUPPORTED: return "unsupported";
        case MDGB_ERR_DEVICE_TIMEOUT: return "device-side wait timed out";
        case MDGB_ERR_OUT_OF_MEMORY: return "out of device memory";
        case MDGB_ERR_SKIN_VIOLATION: return "skin violation";
        default: return "unknown status";
    }
}

MDGB_API void* mdgb_stream(mdgb_engine* e) { return e ? (void*)e->stream : nullptr; }

static int set_pot(mdgb_engine* e, uint16_t t0, uint16_t t1, const LJ& p) {
    if (!e) return MDGB_ERR_INVALID_ARGUMENT;
    if (t0 >= MAX_TYPES || t1 >= MAX_TYPES) return fail(e, MDGB_ERR_INVALID_ARGUMENT, "type id >= 16");
    const int a = std::min(t0, t1), b = std::max(t0, t1);  // potential.rs:142
    e->pot[a][b] = p;
    e->pot[a][b].set = true;
    if (e->has_state) {
        cudaSetDevice(e->device);
        int rc = upload_pairs(e);
        if (rc) return rc;
        e->lists_fresh = false;
        // a changed cutoff needs lists built with the new radius
        CU(cudaMemcpyAsync(e->rep_host.data(), e->dev.rep, e->nrep * sizeof(RepDev), cudaMemcpyDeviceToHost,
                           e->stream));
        CU(cudaStreamSynchronize(e->stream));
        for (int r = 0; r < e->nrep; ++r) {
            e->rep_host[r].rebuild = 1;
            e->rep_host[r].rlist = e->rcmax + class_skin_of(e, e->class_of[r]);
        }
        CU(cudaMemcpyAsync(e->dev.rep, e->rep_host.data(), e->nrep * sizeof(RepDev), cudaMemcpyHostToDevice,
                           e->stream));
    }
    return MDGB_OK;
}

MDGB_API int mdgb_set_potential(mdgb_engine* e, uint16_t t0, uint16_t t1, double sigma, double eps) {
    if (!(sigma > 0.0)) return fail(e, MDGB_ERR_INVALID_ARGUMENT, "sigma must be positive");
    LJ p;
    p.sigma = sigma; p.eps = eps;
    lj_finish(p);
    return set_pot(e, t0, t1, p);
}

MDGB_API int mdgb_set_potential_raw(mdgb_engine* e, uint16_t t0, uint16_t t1, double sigma, double eps,
                                    double r_cut, double u_cut) {
    if (!(sigma > 0.0) || !(r_cut > 0.0)) return fail(e, MDGB_ERR_INVALID_ARGUMENT, "bad potential");
    LJ p;
    p.sigma = sigma; p.eps = eps; p.rc = r_cut; p.ucut = u_cut;
    return set_pot(e, t0, t1, p);
}

MDGB_API int mdgb_upload_state(mdgb_engine* e, int64_t n, const uint16_t* type, const double* pos,
                               const double* vel, const double* mass_per_type, int ntypes, const double box[3]) {
    if (!e) return MDGB_ERR_INVALID_ARGUMENT;
    cudaSetDevice(e->device);
    const int64_t off[2] = {0, n};
    return upload_impl(e, 1, off, type, pos, vel, mass_per_type, ntypes, box);
}

MDGB_API int mdgb_ensemble_upload(mdgb_engine* e, int nrep, const int64_t* offsets, const uint16_t* type,
                                  const double* pos, const double* vel, const double* mass_per_type, int ntypes,
                                  const double* boxes) {
    if (!e) return MDGB_ERR_INVALID_ARGUMENT;
    cudaSetDevice(e->device);
    return upload_impl(e, nrep, offsets, type, pos, vel, mass_per_type, ntypes, boxes);
}

MDGB_API int mdgb_upload_forces(mdgb_engine* e, const double* force, const double* potential,
                                const double* temp) {
    if (!e) return MDGB_ERR_INVALID_ARGUMENT;
    if (!e->has_state) return fail(e, MDGB_ERR_NO_STATE, "no state uploaded");
    cudaSetDevice(e->device);
    const size_t N = e->ntot;
    double* d_f = e->d_out;
    double* d_p = e->d_out + 3 * N;
    double* d_t = e->d_out + 4 * N;
    if (force) CU(cudaMemcpyAsync(d_f, force, 3 * N * sizeof(double), cudaMemcpyHostToDevice, e->stream));
    if (potential) CU(cudaMemcpyAsync(d_p, potential, N * sizeof(double), cudaMemcpyHostToDevice, e->stream));
    if (temp) CU(cudaMemcpyAsync(d_t, temp, N * sizeof(double), cudaMemcpyHostToDevice, e->stream));
    const double* a = force ? d_f : nullptr;
    const double* b = potential ? d_p : nullptr;
    const double* c = temp ? d_t : nullptr;
    void* args[] = {(void*)&e->dev, (void*)&a, (void*)&b, (void*)&c};
    CU(cudaLaunchKernel((const void*)k_scatter_forces, dim3((unsigned)((N + 255) / 256)), dim3(256), args, 0,
                        e->stream));
    CU(cudaStreamSynchronize(e->stream));
    return MDGB_OK;
}

MDGB_API int mdgb_interacting_pairs(mdgb_engine* e, int64_t capacity, int32_t* out_i, int32_t* out_j,
                                    int64_t* count) {
    if (!e || !count || capacity < 0 || (capacity > 0 && (!out_i || !out_j))) return MDGB_ERR_INVALID_ARGUMENT;
    if (!e->has_state) return fail(e, MDGB_ERR_NO_STATE, "no state uploaded");
    cudaSetDevice(e->device);
    int* di = nullptr;
    int* dj = nullptr;
    unsigned long long* dc = nullptr;
    const size_t cap = (size_t)std::max<int64_t>(capacity, 1);
    CU(cudaMalloc(&di, cap * sizeof(int)));
    CU(cudaMalloc(&dj, cap * sizeof(int)));
    CU(cudaMalloc(&dc, sizeof(unsigned long long)));
    CU(cudaMemsetAsync(dc, 0, sizeof(unsigned long long), e->stream));
    long long lcap = capacity;
    void* args[] = {(void*)&e->dev, (void*)&lcap, (void*)&di, (void*)&dj, (void*)&dc};
    cudaError_t ce = cudaLaunchKernel((const void*)k_pairs, dim3((unsigned)((e->ntot + 127) / 128)), dim3(128), args,
                                      0, e->stream);
    unsigned long long total = 0;
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(&total, dc, sizeof(total), cudaMemcpyDeviceToHost, e->stream);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(e->stream);
    const size_t ncopy = (size_t)std::min<unsigned long long>(total, (unsigned long long)capacity);
    if (ce == cudaSuccess && ncopy) ce = cudaMemcpy(out_i, di, ncopy * sizeof(int), cudaMemcpyDeviceToHost);
    if (ce == cudaSuccess && ncopy) ce = cudaMemcpy(out_j, dj, ncopy * sizeof(int), cudaMemcpyDeviceToHost);
    cudaFree(di);
    cudaFree(dj);
    cudaFree(dc);
    if (ce != cudaSuccess) return fail(e, MDGB_ERR_CUDA, cudaGetErrorString(ce));
    *count = (int64_t)total;
    return MDGB_OK;
}

MDGB_API int mdgb_compute_forces(mdgb_engine* e) {
    if (!e) return MDGB_ERR_INVALID_ARGUMENT;
    if (!e->has_state) return fail(e, MDGB_ERR_NO_STATE, "no state uploaded");
    cudaSetDevice(e->device);
    int rc = settle_tpa(e, true, 1);
    if (rc) return rc;
    rc = compute_forces_impl(e);
    if (!rc) e->forces_valid = true;
    return rc;
}

MDGB_API int mdgb_step(mdgb_engine* e, int64_t nsteps, double dt, mdgb_thermostat* thermostat,
                       mdgb_barostat* barostat) {
    if (!e) return MDGB_ERR_INVALID_ARGUMENT;
    if (!e->has_state) return fail(e, MDGB_ERR_NO_STATE, "no state uploaded");
    if (e->nrep != 1) return fail(e, MDGB_ERR_INVALID_ARGUMENT, "ensemble engine: use mdgb_ensemble_step");
    cudaSetDevice(e->device);
    int rc = set_coupling_impl(e, thermostat, barostat);
    if (rc) return rc;
    rc = step_impl(e, nsteps, dt);
    if (rc) return rc;
    return get_coupling_impl(e, thermostat, barostat);
}

MDGB_API int mdgb_prepare_step(mdgb_engine* e, int64_t nsteps, double dt, const mdgb_thermostat* thermostat,
                               const mdgb_barostat* barostat) {
    if (!e) return MDGB_ERR_INVALID_ARGUMENT;
    if (e->nrep != 1 && e->has_state) return fail(e, MDGB_ERR_INVALID_ARGUMENT, "ensemble engine: use mdgb_ensemble_prepare");
    cudaSetDevice(e->device);
    const bool nh = thermostat && thermostat->kind == MDGB_THERMOSTAT_NOSE_HOOVER;
    return prepare_impl(e, nsteps, dt, thermostat != nullptr, barostat != nullptr, nh);
}

MDGB_API int mdgb_ensemble_prepare(mdgb_engine* e, int64_t nsteps, double dt) {
    if (!e) return MDGB_ERR_INVALID_ARGUMENT;
    cudaSetDevice(e->device);
    return prepare_impl(e, nsteps, dt, e->thermo_on, e->baro_on, e->thermo_nh);
}

MDGB_API int mdgb_test_barrier_timeout(mdgb_engine* e, int hold_block, int64_t wait_cycles) {
    return mdgb_test_barrier_timeout_at(e, 0, hold_block, wait_cycles);
}

MDGB_API int mdgb_test_barrier_timeout_at(mdgb_engine* e, int step, int hold_block, int64_t wait_cycles) {
    if (!e || step < 0 || hold_block < 0 || wait_cycles <= 0) return MDGB_ERR_INVALID_ARGUMENT;
    e->test_hold_step = step;
    e->test_hold_block = hold_block;
    e->test_barrier_cycles = wait_cycles;
    return MDGB_OK;
}

MDGB_API int mdgb_download_state(mdgb_engine* e, double* pos, double* vel, double* force, double* potential,
                                 double* temp, double box[3]) {
    if (!e) return MDGB_ERR_INVALID_ARGUMENT;
    cudaSetDevice(e->device);
    return download_impl(e, pos, vel, force, potential, temp, box);
}

MDGB_API int mdgb_macro_parameters(mdgb_engine* e, int type, mdgb_macro* out) {
    if (!e) return MDGB_ERR_INVALID_ARGUMENT;
    if (e->nrep != 1) return fail(e, MDGB_ERR_INVALID_ARGUMENT, "ensemble engine: use mdgb_ensemble_macro");
    cudaSetDevice(e->device);
    return macro_impl(e, type, out);
}

MDGB_API int mdgb_ensemble_set_coupling(mdgb_engine* e, const mdgb_thermostat* thermostats,
                                        const mdgb_barostat* barostats) {
    if (!e) return MDGB_ERR_INVALID_ARGUMENT;
    cudaSetDevice(e->device);
    return set_coupling_impl(e, thermostats, barostats);
}

MDGB_API int mdgb_ensemble_step(mdgb_engine* e, int64_t nsteps, double dt) {
    if (!e) return MDGB_ERR_INVALID_ARGUMENT;
    cudaSetDevice(e->device);
    return step_impl(e, nsteps, dt);
}

MDGB_API int mdgb_ensemble_get_coupling(mdgb_engine* e, mdgb_thermostat* thermostats, mdgb_barostat* barostats) {
    if (!e) return MDGB_ERR_INVALID_ARGUMENT;
    if (!e->has_state) return fail(e, MDGB_ERR_NO_STATE, "no state uploaded");
    cudaSetDevice(e->device);
    return get_coupling_impl(e, thermostats, barostats);
}

MDGB_API int mdgb_ensemble_download(mdgb_engine* e, double* pos, double* vel, double* force, double* potential,
                                    double* temp, double* boxes) {
    if (!e) return MDGB_ERR_INVALID_ARGUMENT;
    cudaSetDevice(e->device);
    return download_impl(e, pos, vel, force, potential, temp, boxes);
}

MDGB_API int mdgb_ensemble_macro(mdgb_engine* e, int type, mdgb_macro* out) {
    if (!e) return MDGB_ERR_INVALID_ARGUMENT;
    cudaSetDevice(e->device);
    return macro_impl(e, type, out);
}

MDGB_API int mdgb_get_stats(mdgb_engine* e, mdgb_stats* out) {
    if (!e || !out) return MDGB_ERR_INVALID_ARGUMENT;
    cudaSetDevice(e->device);
    if (e->stream) cudaStreamSynchronize(e->stream);
    prof_collect(e);
    if (e->has_state) {
        std::vector<RepDev> reps(e->nrep);
        if (cudaMemcpy(reps.data(), e->dev.rep, e->nrep * sizeof(RepDev), cudaMemcpyDeviceToHost) == cudaSuccess) {
            int64_t nb = 0;
            int mx = 0;
            for (auto& R : reps) { nb += R.nrebuilds; mx = std::max(mx, R.max_nn); }
            e->st.rebuilds = nb;
            e->st.max_neighbors = mx;
        }
        unsigned int direct = 0;
        if (cudaMemcpy(&direct, e->dev.bar + 5, sizeof(direct), cudaMemcpyDeviceToHost) == cudaSuccess)
            e->st.direct_list_builds = direct;
    }
    e->st.neighbor_capacity = e->cap;
    e->st.threads_per_atom = e->tpa;
    for (int c = 0; c < mdgb_engine::NCLASS; ++c) {
        e->st.class_threads_per_atom[c] = e->class_tpa[c];
        e->st.class_replicas[c] = e->class_nrep[c];
        e->st.class_skin[c] = class_skin_of(e, c);
    }
    *out = e->st;
    return MDGB_OK;
}

MDGB_API int mdgb_trace_phases(mdgb_engine* e, double* out, int n) {
    if (!e || !out || n < 0) return MDGB_ERR_INVALID_ARGUMENT;
    if (!e->has_state) return fail(e, MDGB_ERR_NO_STATE, "no state uploaded");
    if (!(e->cfg.flags & MDGB_FLAG_TRACE)) return fail(e, MDGB_ERR_INVALID_ARGUMENT, "engine created without MDGB_FLAG_TRACE");
    cudaSetDevice(e->device);
    unsigned long long h[TR_SLOTS];
    CU(cudaMemcpyAsync(h, e->trace_buf, sizeof(h), cudaMemcpyDeviceToHost, e->stream));
    CU(cudaStreamSynchronize(e->stream));
    CU(cudaMemsetAsync(e->trace_buf, 0, sizeof(h), e->stream));
    const int m = std::min(n, 14);
    for (int i = 0; i < m; ++i) out[i] = i < 12 ? h[i] * 1e-3 : (double)h[i];
    return MDGB_OK;
}

MDGB_API int mdgb_reset_stats(mdgb_engine* e) {
    if (!e) return MDGB_ERR_INVALID_ARGUMENT;
    cudaSetDevice(e->device);
    if (e->stream) cudaStreamSynchronize(e->stream);
    prof_collect(e);
    const int cap = e->st.neighbor_capacity;
    e->st = mdgb_stats{};
    e->st.neighbor_capacity = cap;
    if (e->has_state) {
        std::vector<RepDev> reps(e->nrep);
        if (cudaMemcpy(reps.data(), e->dev.rep, e->nrep * sizeof(RepDev), cudaMemcpyDeviceToHost) == cudaSuccess) {
            for (auto& R : reps) R.nrebuilds = 0;
            cudaMemcpy(e->dev.rep, reps.data(), e->nrep * sizeof(RepDev), cudaMemcpyHostToDevice);
        }
        cudaMemset(e->dev.bar + 5, 0, sizeof(unsigned int));
    }
    return MDGB_OK;
}

MDGB_API int mdgb_synchronize(mdgb_engine* e) {
    if (!e) return MDGB_ERR_INVALID_ARGUMENT;
    cudaSetDevice(e->device);
    return cudaStreamSynchronize(e->stream) == cudaSuccess ? MDGB_OK : MDGB_ERR_CUDA;
}

}  // extern "C"
