// kernels_step.cu -- the per-step O(N) work of the engine in one cooperative
// persistent kernel (k_pre), plus the macro-parameter reduction kernel.
//
//   [coupling]  reductions -> Berendsen lambda / mu
//               (solver/src/initializer/thermostat.rs:24-34, barostat.rs:21-31,
//                solver/src/macro_parameters/{mod,energy,pressure,temperature}.rs):
//               exact 128-bit fixed-point sums on the mixed path (integer
//               work, phase_partials_fx), FP64 trees (or the reference's
//               serial order) on the FP64 path
//   [drift]     v += F dt/2m, thermostat scale, pending barostat scale of x,
//               x += v dt, periodic wrap, FP32 mirror, displacement
//               (solver/src/solver/integrator.rs:30-47, core/src/particle.rs:120-141)
//   [rebuild]   per replica, only when the displacement (or a forced rebuild)
//               asks for it: integer counting sort of atoms into cells
//               (count -> exclusive scan -> scatter -> canonical order inside
//               each cell); the Verlet list of brute-mode replicas here, of
//               cell-mode replicas in k_build_list (kernels_list.cu), which
//               follows every k_pre launch.
//   After a force pass that already kicked and drifted (NVE chunks), k_pre
//   only takes the rebuild decision -- without a grid barrier when no replica
//   needs one -- and rebuilds if needed.
//
// On the mixed path the FP64 integration uses fused multiply-adds (explicit
// __fma_rn); the FP64 path keeps the reference's separate multiply and add.
//
// Phases are separated by a bounded grid barrier (the kernel is launched
// cooperatively, so every block is resident).  A barrier that waits longer
// than ~2 s sets E_TIMEOUT and the launch ends: every block stops at its next
// barrier at the latest, so no phase runs on the incomplete results of the
// one before (and the engine puts the chunk's starting state back).  Every
// index derived from scratch data is range-checked as well.  Data produced by
// another block inside the same launch is read with ld.global.cg (L2), never
// from a possibly stale L1 line.
//
// This file is compiled with -fmad=false: its FP64 arithmetic (kick, drift,
// wrap, reductions, coupling factors) keeps the reference's unfused
// multiply-then-add rounding unless a fused operation is written out.
#include <algorithm>
#include <atomic>

#include "force_mixed.cuh"
#include "list_direct.cuh"

namespace mdgb {

constexpr long long BARRIER_LIMIT_CYCLES = 4000000000LL;
constexpr double K_B = 1.380648528;  // core/src/lib.rs:15

static_assert(sizeof(RepDev) % 8 == 0, "RepDev must be a whole number of 8-byte words");


// One replica record per block, in shared memory (phases work tile by tile
// and a tile never straddles replicas).  The copy is kept while consecutive
// tiles of a block belong to the same replica and dropped at every grid
// barrier (the next phase may see fields the previous one changed).
__shared__ RepDev g_tile_rep;
__shared__ int g_tile_rep_id;

__device__ __forceinline__ void tile_rep_reset() {
    if (threadIdx.x == 0) g_tile_rep_id = -1;
    __syncthreads();
}

__device__ __forceinline__ const RepDev& tile_rep(const Dev& d, int r) {
    if (g_tile_rep_id == r) return g_tile_rep;   // block-uniform
    __syncthreads();  // every thread is done with the previous tile's record
    const long long* src = reinterpret_cast<const long long*>(d.rep + r);
    long long* dst = reinterpret_cast<long long*>(&g_tile_rep);
    for (int i = threadIdx.x; i < (int)(sizeof(RepDev) / 8); i += blockDim.x) dst[i] = __ldcg(src + i);
    if (threadIdx.x == 0) g_tile_rep_id = r;
    __syncthreads();
    return g_tile_rep;
}

__device__ __forceinline__ double4_32a ldcg4(const double4_32a* p) {
    const double2 a = __ldcg(reinterpret_cast<const double2*>(p));
    const double2 b = __ldcg(reinterpret_cast<const double2*>(p) + 1);
    return make_double4_32a(a.x, a.y, b.x, b.y);
}

// The grid barrier's wait limit in clock cycles (set at kernel entry) and the
// block's verdict after the last barrier.
__shared__ long long g_bar_limit;
__shared__ int g_bar_abort;
__shared__ int g_bar_spin;    // poll without sleeping in between (k_steps: short phases)

__device__ __forceinline__ void barrier_setup(const StepParams& sp, bool spin = false) {
    if (threadIdx.x == 0) {
        g_bar_spin = spin ? 1 : 0;
        g_bar_limit = sp.barrier_cycles > 0 ? sp.barrier_cycles : BARRIER_LIMIT_CYCLES;
        g_bar_abort = 0;
    }
}

// Returns true when the launch must stop: this block's wait ran out, or
// another block's did (E_TIMEOUT in the error word).  A block that stops
// does no work of the next phase, so no phase ever reads the incomplete
// results of the one before; every block ends at its next barrier at the
// latest, each wait being bounded.  Call sites: if (grid_barrier(d)) return;
__device__ __forceinline__ bool grid_barrier(const Dev& d) {
    __syncthreads();
    if (threadIdx.x == 0) {
        volatile unsigned int* gen = d.bar + 1;
        const unsigned int g = *gen;
        __threadfence();
        const unsigned int arrived = atomicAdd(d.bar, 1u);
        if (arrived == gridDim.x - 1) {
            atomicExch(d.bar, 0u);
            __threadfence();
            atomicAdd(d.bar + 1, 1u);
        } else {
            const long long t0 = clock64();
            while (*gen == g) {
                if (!g_bar_spin) __nanosleep(100);
                if (clock64() - t0 > g_bar_limit) {
                    atomicOr(d.err, E_TIMEOUT);
                    break;
                }
            }
        }
        __threadfence();
        g_tile_rep_id = -1;
        g_bar_abort = (*(volatile int*)d.err & E_TIMEOUT) ? 1 : 0;
    }
    __syncthreads();
    return g_bar_abort != 0;
}

// A grid barrier whose last block to arrive runs f() before it lets the others
// go: f sees everything written before the barrier, and every block everything
// f wrote (k_steps: reductions' last stages and the rebuild decision, which
// would otherwise take a phase and a barrier of their own).
template <class F>
__device__ __forceinline__ bool grid_barrier_then(const Dev& d, F f) {
    __shared__ int s_last_block, s_failed;
    __syncthreads();
    volatile unsigned int* gen = d.bar + 1;
    unsigned int g = 0;
    if (threadIdx.x == 0) {
        g = *gen;
        __threadfence();
        s_last_block = atomicAdd(d.bar, 1u) == gridDim.x - 1 ? 1 : 0;
        s_failed = chunk_failed(d) ? 1 : 0;
        __threadfence();
        g_tile_rep_id = -1;
    }
    __syncthreads();
    if (s_last_block) {
        if (!s_failed) f();
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            atomicExch(d.bar, 0u);
            __threadfence();
            atomicAdd(d.bar + 1, 1u);
        }
    } else if (threadIdx.x == 0) {
        const long long t0 = clock64();
        while (*gen == g) {
            if (!g_bar_spin) __nanosleep(100);
            if (clock64() - t0 > g_bar_limit) {
                atomicOr(d.err, E_TIMEOUT);
                break;
            }
        }
    }
    if (threadIdx.x == 0) {
        __threadfence();
        g_tile_rep_id = -1;
        g_bar_abort = (*(volatile int*)d.err & E_TIMEOUT) ? 1 : 0;
    }
    __syncthreads();
    return g_bar_abort != 0;
}

// Deterministic block sum of NV doubles (fixed shuffle tree, fixed warp order).
// Result valid in thread 0.
// Warp stage: a reduce-scatter butterfly -- at offsets 16, 8, ... each lane
// keeps half of its values and adds the partner's copy of that half, so after
// log2(NV) stages lane L holds one value index (bits of L) and the remaining
// offsets finish plain sums: NV - 1 + log2(32/NV) FP64 adds per lane instead
// of 5 NV (the FP64 pipe is narrow on GB300).  NV is a power of two <= 32.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double* sm) {
    static_assert(NV >= 1 && NV <= 32 && (NV & (NV - 1)) == 0, "power of two");
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int idx = 0;
#pragma unroll
    for (int c = NV, o = 16; c > 1; c >>= 1, o >>= 1) {
        const bool hb = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < c / 2; ++k) {
            const double send = hb ? v[k] : v[c / 2 + k];
            const double keep = hb ? v[c / 2 + k] : v[k];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
        if (hb) idx += c / 2;
    }
#pragma unroll
    for (int o = 16 / NV; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    __syncthreads();
    if ((lane & (32 / NV - 1)) == 0) sm[idx * 32 + w] = v[0];
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            double s = sm[k * 32];
            for (int i = 1; i < nw; ++i) s += sm[k * 32 + i];
            v[k] = s;
        }
    }
    __syncthreads();
}

__device__ __forceinline__ float block_max(float v, float* sm) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_down_sync(0xffffffffu, v, off));
    __syncthreads();
    if (lane == 0) sm[w] = v;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int i = 1; i < nw; ++i) v = fmaxf(v, sm[i]);
    __syncthreads();
    return v;
}

__device__ __forceinline__ int block_max_int(int v, int* sm) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = max(v, __shfl_down_sync(0xffffffffu, v, off));
    __syncthreads();
    if (lane == 0) sm[w] = v;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int i = 1; i < nw; ++i) v = max(v, sm[i]);
    __syncthreads();
    return v;
}

// Two-level deterministic reduction of tile partials: one warp per chunk of
// <= CHUNK_TILES tiles (phase_chunk_sums), then one warp per replica over its
// chunks -- a replica of millions of atoms is summed by many warps in
// parallel, always in the same order.
// Rows of 8 partials (one per tile or chunk, 64 bytes) summed slot by slot by
// one warp: lane l adds rows l, l + 32, ... in order, then a shuffle tree per
// slot.  Each lane loads a row's slots together (four 16-byte loads), so the
// loads of all slots are in flight at once.  Result valid in lane 0.
template <int NS>
__device__ __forceinline__ void warp_sum_rows(const double* rows, int n, double (&s)[NS]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < NS; ++k) s[k] = 0.0;
    for (int t = lane; t < n; t += 32) {
        const double2* row = reinterpret_cast<const double2*>(rows + (size_t)t * 8);
        double v[8];
#pragma unroll
        for (int q = 0; q < (NS + 1) / 2; ++q) {
            const double2 x = __ldcg(row + q);
            v[2 * q] = x.x; v[2 * q + 1] = x.y;
        }
#pragma unroll
        for (int k = 0; k < NS; ++k) s[k] += v[k];
    }
#pragma unroll
    for (int k = 0; k < NS; ++k) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) s[k] += __shfl_down_sync(0xffffffffu, s[k], off);
    }
}

template <int NS>
__device__ void phase_chunk_sums(const Dev& d, int block, int blocks) {
    const int lane = threadIdx.x & 31;
    const int gw = (block * blockDim.x + threadIdx.x) >> 5;
    const int nw = (blocks * blockDim.x) >> 5;
    for (int c = gw; c < d.nchunks; c += nw) {
        const int4 ch = d.chunks[c];
        double s[NS];
        warp_sum_rows<NS>(d.part + (size_t)ch.y * 8, ch.z, s);
        if (lane == 0)
            for (int k = 0; k < NS; ++k) d.cpart[(size_t)c * 8 + k] = s[k];
    }
}

// Sums over the chunk partials of one replica by one warp (fixed order),
// slots 0..NS-1, broadcast to every lane.
template <int NS>
__device__ __forceinline__ void warp_sum_tiles(const Dev& d, const RepDev& R, double (&S)[NS]) {
    warp_sum_rows<NS>(d.cpart + (size_t)R.chunk_begin * 8, R.nchunks, S);
#pragma unroll
    for (int k = 0; k < NS; ++k) S[k] = __shfl_sync(0xffffffffu, S[k], 0);
}


// ---------------------------------------------------------------------------
// Tree-order reductions over atoms of type `sel` (all of one mass m, so m is
// factored out of the sums and applied once per replica; halving is exact
// and applied once too -- fewer FP64-pipe operations per atom).
// Pass 1 slots: 0-2 sum(v), 3 count, 4 sum(temp), 5 sum(v.v), 6 sum(potential).
// One atom's inputs of pass 1, loaded a tile ahead (a block walks its tiles
// one after another; the loads of the next overlap this one's sums).
struct Pass1In {
    int ty;
    double vx, vy, vz, vir, pot;
};

__device__ __forceinline__ void pass1_load(const Dev& d, int s, Pass1In& in) {
    const int N = d.ntot;
    in.ty = (int)__ldcg(reinterpret_cast<const long long*>(d.pos + s) + 3);
    in.vx = __ldcg(d.vel + s); in.vy = __ldcg(d.vel + N + s); in.vz = __ldcg(d.vel + 2 * N + s);
    in.vir = __ldcg(d.evir + s);
    in.pot = __ldcg(d.epot + s);
}

__device__ void phase_partials1(const Dev& d, int sel) {
    __shared__ double sm[8 * 32];
    int t = blockIdx.x;
    int4 tl = t < d.ntiles ? d.tiles[t] : make_int4(0, 0, 0, 0);
    Pass1In cur;
    cur.ty = -1;
    if (t < d.ntiles && (int)threadIdx.x < tl.z) pass1_load(d, tl.y + threadIdx.x, cur);
    for (; t < d.ntiles; t += gridDim.x) {
        const int tn = t + gridDim.x;
        int4 tln = make_int4(0, 0, 0, 0);
        Pass1In nxt;
        nxt.ty = -1;
        if (tn < d.ntiles) {
            tln = d.tiles[tn];
            if ((int)threadIdx.x < tln.z) pass1_load(d, tln.y + threadIdx.x, nxt);
        }
        double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if ((int)threadIdx.x < tl.z && cur.ty == sel) {
            const double vx = cur.vx, vy = cur.vy, vz = cur.vz;
            v[0] = vx; v[1] = vy; v[2] = vz; v[3] = 1.0;
            v[4] = cur.vir;
            v[5] = vx * vx + vy * vy + vz * vz;
            v[6] = cur.pot;
        }
        block_sum<8>(v, sm);
        if (threadIdx.x == 0)
            for (int k = 0; k < 8; ++k) d.part[(size_t)t * 8 + k] = v[k];
        tl = tln;
        cur = nxt;
    }
}

// One warp per replica: COM velocity, momentum, kinetic and potential energy
// (mod.rs:12-34, energy.rs:14-49).
__device__ void phase_finalize1(const Dev& d, int sel, int block, int blocks) {
    const int warps = (blocks * blockDim.x) >> 5;
    const int gw = (block * blockDim.x + threadIdx.x) >> 5;
    const double m = d.mass[sel];
    for (int r = gw; r < d.nrep; r += warps) {
        const RepDev R = load_rep(d.rep + r);
        double S[7];
        warp_sum_tiles<7>(d, R, S);
        RepDev* W = d.rep + r;
        const int lane = threadIdx.x & 31;
        if (lane < 3) W->vcm[lane] = (lane == 0 ? S[0] : lane == 1 ? S[1] : S[2]) / S[3];
        if (lane == 0) {
            W->mom[0] = S[0] * m; W->mom[1] = S[1] * m; W->mom[2] = S[2] * m;
            W->msum = S[3] * m; W->virsum = S[4]; W->ke = 0.5 * (m * S[5]); W->pe = S[6] * 0.5;
            W->count = (long long)S[3];
        }
    }
}

// Pass 2 slot 0: sum(|v - vcm|^2)
__device__ void phase_partials2(const Dev& d, int sel) {
    __shared__ double sm[1 * 32];
    const int N = d.ntot;
    for (int t = blockIdx.x; t < d.ntiles; t += gridDim.x) {
        const int4 tl = d.tiles[t];
        const int s = tl.y + threadIdx.x;
        double v[1] = {0};
        if ((int)threadIdx.x < tl.z) {
            const int ty = (int)__ldcg(reinterpret_cast<const long long*>(d.pos + s) + 3);
            if (ty == sel) {
                const double vc0 = __ldcg(&d.rep[tl.x].vcm[0]), vc1 = __ldcg(&d.rep[tl.x].vcm[1]),
                             vc2 = __ldcg(&d.rep[tl.x].vcm[2]);
                const double dx = __ldcg(d.vel + s) - vc0, dy = __ldcg(d.vel + N + s) - vc1,
                             dz = __ldcg(d.vel + 2 * N + s) - vc2;
                v[0] = dx * dx + dy * dy + dz * dz;
            }
        }
        block_sum<1>(v, sm);
        if (threadIdx.x == 0) d.part[(size_t)t * 8] = v[0];
    }
}

// temperature.rs:4-7
__device__ __forceinline__ double temperature_of(double thermal, long long n) {
    const double t = (2.0 * thermal) / (3.0 * (double)n * K_B);
    return t * 100.0;
}

// Coupling factors from the reduced T and P (thermostat.rs:31-39, barostat.rs:29-30).
__device__ __forceinline__ void thermostat_factor(RepDev* W, const RepDev& R, double T, double dt) {
    if (!R.thermo_on) return;
    if (R.thermo_kind == 0) {
        const double l2 = 1.0 + dt / R.th_tau * (R.th_T0 / T - 1.0);
        W->lambda = sqrt(l2);
    } else {
        const double psi_dot = -((R.th_T0 / T) - 1.0) / R.th_tau;
        const double psi = R.psi + psi_dot * (dt / 2.0);
        W->psi = psi;
        W->lambda = exp(-psi * dt / 2.0);
    }
}
__device__ __forceinline__ void barostat_factor(RepDev* W, const RepDev& R, double P, double dt) {
    if (!R.baro_on) return;
    const double m3 = 1.0 + dt * R.ba_beta / R.ba_tau * (P - R.ba_P0);
    W->myu = cbrt(m3);
}
// A replica's last stage by one warp.  Its dozen FP64 divisions are chains of
// dependent operations at about 64 cycles each: those that do not need one
// another are lanes of the same instructions (argon, 1,000 atoms, a coupled step
// in the reference's order: 85.8 -> 82.8 us).  All lanes call; every lane has
// read its copy of the record before the first store.
//
// The centre-of-mass velocity sum_a / den (lanes 0-2) beside the box part of the
// pending barostat update (lanes 3-5: box *= mu once per type, barostat.rs:45).
__device__ __forceinline__ void finalize_frame(const Dev& d, RepDev* W, const RepDev& R, bool coupling, double s0,
                                               double s1, double s2, double den, double (&vc)[3], double (&box)[3]) {
    const int lane = threadIdx.x & 31, a = lane < 3 ? lane : lane - 3;
    double L = a == 0 ? R.box[0] : a == 1 ? R.box[1] : R.box[2];
    const int nc = a == 0 ? R.nc[0] : a == 1 ? R.nc[1] : R.nc[2];
    const bool scale = coupling && R.pending != 1.0;
    if (scale)
        for (int k = 0; k < d.ntypes; ++k) L *= R.pending;
    const double q = (lane < 3 ? (a == 0 ? s0 : a == 1 ? s1 : s2) : L) / (lane < 3 ? den : (double)nc);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        vc[k] = __shfl_sync(0xffffffffu, q, k);
        box[k] = __shfl_sync(0xffffffffu, L, 3 + k);
    }
    if (lane < 3) W->vcm[a] = q;
    else if (lane < 6 && scale) { W->box[a] = L; W->cs[a] = q; }
}

// Temperature and thermostat factor (lane 0) beside pressure and barostat factor
// (lane 1).  th: thermal energy of n atoms; pv: three times P V.
__device__ __forceinline__ void finalize_coupling(RepDev* W, const RepDev& R, const StepParams& sp, bool coupling,
                                                  bool pressure, double th, long long n, double pv, double volume) {
    const int lane = threadIdx.x & 31;
    const bool t = lane == 0;
    const double dt = sp.dt;
    double q = (t ? 2.0 * th : pv) / (t ? 3.0 * (double)n * K_B : volume);
    if (t) q *= 100.0;                                              // T (temperature_of)
    const double x = (t ? R.th_T0 : q) / (t ? q : 3.0);             // T0 / T; P
    if (t) { W->thermal = th; W->T = q; }
    if (lane == 1 && pressure) W->P = x;
    if (!coupling) return;
    const bool nh = R.thermo_kind != 0;
    const double y = (t ? (nh ? -(x - 1.0) : dt) : dt * R.ba_beta) / (t ? R.th_tau : R.ba_tau);
    if (t && R.thermo_on) {
        if (nh) {
            const double psi = R.psi + y * (dt / 2.0);
            W->psi = psi;
            W->lambda = exp(-psi * dt / 2.0);
        } else {
            W->lambda = sqrt(1.0 + y * (x - 1.0));
        }
    }
    if (lane == 1 && R.baro_on) W->myu = cbrt(1.0 + y * (x - R.ba_P0));
}

// Finalize pass 2.  coupling: first apply the box part of the pending
// barostat update (box *= mu once per type, barostat.rs:45), then T, P and
// the coupling factors.
__device__ void phase_finalize2(const Dev& d, const StepParams& sp, bool coupling, int sel, int block, int blocks) {
    const int warps = (blocks * blockDim.x) >> 5;
    const int gw = (block * blockDim.x + threadIdx.x) >> 5;
    for (int r = gw; r < d.nrep; r += warps) {
        const RepDev R = load_rep(d.rep + r);
        double S1[1];
        warp_sum_tiles<1>(d, R, S1);
        const double sdv = S1[0];
        const double p1 = d.mass[sel] * sdv;              // sum m |v - vcm|^2 (pressure.rs:13-17)
        const double th = 0.5 * p1;                        // energy.rs:25-37
        RepDev* W = d.rep + r;
        double vc[3], box[3];
        // (pass 1 has left the centre-of-mass velocity: divided by one, it stays)
        finalize_frame(d, W, R, coupling, R.vcm[0], R.vcm[1], R.vcm[2], 1.0, vc, box);
        finalize_coupling(W, R, sp, coupling, true, th, R.count, p1 + (-R.virsum) * 0.5, box[0] * box[1] * box[2]);
    }
}

// Mixed path, coupled steps: one pass.  sum_i |v_i - vcm|^2 = sum |v_i|^2 -
// n |vcm|^2 (as sum v_i = n vcm), so pass 2 and its barriers fold into the
// finalize of pass 1; then what phase_finalize2 does (box, T, P, coupling).
// The FP64 path keeps the reference's explicit second pass.
__device__ void phase_finalize_single(const Dev& d, const StepParams& sp, int sel, int block, int blocks) {
    const int warps = (blocks * blockDim.x) >> 5;
    const int gw = (block * blockDim.x + threadIdx.x) >> 5;
    const double m = d.mass[sel];
    for (int r = gw; r < d.nrep; r += warps) {
        const RepDev R = load_rep(d.rep + r);
        double S[7];
        warp_sum_tiles<7>(d, R, S);
        RepDev* W = d.rep + r;
        double vc[3], box[3];
        finalize_frame(d, W, R, true, S[0], S[1], S[2], S[3], vc, box);
        if ((threadIdx.x & 31) == 0) {
            W->mom[0] = S[0] * m; W->mom[1] = S[1] * m; W->mom[2] = S[2] * m;
            W->msum = S[3] * m; W->virsum = S[4]; W->ke = 0.5 * (m * S[5]); W->pe = S[6] * 0.5;
            W->count = (long long)S[3];
        }
        const double p1 = m * (S[5] - S[3] * (vc[0] * vc[0] + vc[1] * vc[1] + vc[2] * vc[2]));
        finalize_coupling(W, R, sp, true, true, 0.5 * p1, (long long)S[3], p1 + (-S[4]) * 0.5,
                          box[0] * box[1] * box[2]);
    }
}

// ---------------------------------------------------------------------------
// Exact sums for the mixed path's coupled steps (replaces the FP64 tree of
// passes partials1 / chunk sums there).  A double x = m 2^(e - 1075)
// (m < 2^53) goes onto a binary grid, unit 2^(T - 1075 - FX_K) with T from the
// largest exponent of that quantity met so far by the warp (fx_grid), as a
// 128-bit integer; lanes, warps, then blocks are added exactly after aligning
// to the larger grid (bits below 2^-96 of the largest value drop, toward zero).
// Integer work only -- GB300's FP64 pipe is narrow -- and the sums do not
// depend on the order of the additions.  Headroom: below 2^100 a value, so a
// replica of up to 2^27 atoms stays below 2^127.
// Below this many atoms the coupled reductions are latency-bound and the
// FP64 tree (fewer dependent steps) is faster; from here on the exact sums
// (no FP64 pipe work) are.
constexpr int FX_MIN_ATOMS = 65536;

__device__ __forceinline__ int fx_exp(double x) {
    const int e = (int)(((unsigned long long)__double_as_longlong(x) >> 52) & 0x7FFull);
    return e ? e : 1;   // subnormals and zero: exponent 1 without the hidden bit
}

// The grid for values up to exponent e: rounded up to the end of a group of
// four, so that warps and blocks nearly always share one and their sums add
// without shifts.  (Exponents near the top stay: 0x7FF marks non-finite values.)
constexpr int FX_T0 = 3;
__device__ __forceinline__ int fx_grid(int e) { return e < 0x7FC ? (e | 3) : e; }

__device__ __forceinline__ __int128 fx_place(double x, int T) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int e = (int)((b >> 52) & 0x7FFull);
    unsigned long long m = b & 0x000FFFFFFFFFFFFFull;
    if (e) m |= 1ull << 52;
    const int s = (e ? e : 1) - T + FX_K;
    if (s >= 0) {   // s <= FX_K: below 2^100 (two 64-bit shifts of the signed mantissa)
        const long long v = (b >> 63) ? -(long long)m : (long long)m;
        const long long hi = (v >> 1) >> (63 - s);
        return (__int128)(((unsigned __int128)(unsigned long long)hi << 64) | ((unsigned long long)v << s));
    }
    const __int128 v = s > -64 ? (__int128)(m >> (-s)) : (__int128)0;
    return (b >> 63) ? -v : v;
}

// v on grid T moved to the coarser grid Tmax >= T, toward zero
__device__ __forceinline__ __int128 fx_align(__int128 v, int T, int Tmax) {
    const int d = Tmax - T;
    if (d == 0) return v;
    if (d >= 127) return 0;
    return v < 0 ? -((-v) >> d) : (v >> d);
}

__device__ __forceinline__ __int128 fx_shfl_xor(__int128 v, int o) {
    const long long lo = __shfl_xor_sync(0xffffffffu, (long long)(unsigned long long)v, o);
    const long long hi = __shfl_xor_sync(0xffffffffu, (long long)(v >> 64), o);
    return (__int128)(((unsigned __int128)(unsigned long long)hi << 64) | (unsigned long long)lo);
}

// x * 2^(T - 1075 - FX_K) rounded to the nearest double (ties to even)
__device__ __forceinline__ double fx_to_double(__int128 v, int T) {
    if (v == 0) return 0.0;
    const bool neg = v < 0;
    const unsigned __int128 u = neg ? (unsigned __int128)(-v) : (unsigned __int128)v;
    const unsigned long long hi = (unsigned long long)(u >> 64), lo = (unsigned long long)u;
    const int p = hi ? 127 - __clzll((long long)hi) : 63 - __clzll((long long)lo);
    unsigned long long mant;
    int sh = 0;
    if (p <= 52) {
        mant = lo;
    } else {
        sh = p - 52;
        mant = (unsigned long long)(u >> sh);
        const unsigned __int128 rem = u & ((((unsigned __int128)1) << sh) - 1);
        const unsigned __int128 half = ((unsigned __int128)1) << (sh - 1);
        if (rem > half || (rem == half && (mant & 1ull))) ++mant;
        if (mant >> 53) { mant >>= 1; ++sh; }
    }
    const double r = ldexp((double)mant, sh + T - 1075 - FX_K);
    return neg ? -r : r;
}

// Pass 1 of a coupled step on the mixed path.  Every warp walks one run of
// consecutive tiles and keeps its lanes' exact sums in registers: nothing is
// exchanged between lanes until the run (or its replica) ends, where a vote
// per pair of atoms is all that a tile needs of the other lanes -- whether a
// quantity's grid has to be widened.  (Before, each tile's sums were reduced
// over the warp and stored as a row -- 120 shuffles and 128 bytes a tile --
// and rows were summed by chunk, then by replica, a grid barrier after each.)
//
// The row of a run stands at the index of its first tile in fx_part; a block
// whose tiles are all of one replica leaves one row for its warps together.
// fx_row_at() below finds a replica's rows again.
//
// Bound by integer issue (about 25 instructions a value): 8M atoms 92 us, 1M 22.
// The whole coupling stage, both Berendsen couplings: 70,304 atoms 36 -> 21 us,
// 1M 94 -> 56, 8M 214 -> 147, 512 replicas of 4.46M atoms 136 -> 97.
struct FxRun {
    __int128 s[FX_NQ];
    int T[FX_NQ];      // grid of every quantity, the same in all lanes
    unsigned cnt;
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int q = 0; q < FX_NQ; ++q) { s[q] = 0; T[q] = FX_T0; }
        cnt = 0;
    }
};

// Tiles per warp; a block's run is its warps' runs one after another.
__device__ __forceinline__ int fx_tiles_per_warp(const Dev& d) {
    const int warps = (int)gridDim.x * (TILE / 32);
    return (d.ntiles + warps - 1) / warps;
}

// One value per lane and quantity onto the lanes' sums (whole warps only).
__device__ __forceinline__ void fx_run_add(FxRun& a, const double (&x)[FX_NQ]) {
    bool wider = false;
#pragma unroll
    for (int q = 0; q < FX_NQ; ++q) wider |= fx_exp(x[q]) > a.T[q];
    if (__any_sync(0xffffffffu, wider)) {
#pragma unroll
        for (int q = 0; q < FX_NQ; ++q) {
            const int T = max(a.T[q], fx_grid(__reduce_max_sync(0xffffffffu, fx_exp(x[q]))));
            a.s[q] = fx_align(a.s[q], a.T[q], T);
            a.T[q] = T;
        }
    }
#pragma unroll
    for (int q = 0; q < FX_NQ; ++q) a.s[q] += fx_place(x[q], a.T[q]);
}

__device__ __forceinline__ void fx_run_tile(const Dev& d, const int4 tl, int sel, FxRun& a) {
    const int lane = threadIdx.x & 31;
    const int N = d.ntot;
#pragma unroll 1
    for (int k = 0; k < TILE; k += 64) {
        if (k >= tl.z) break;
        double x[2][FX_NQ];
        bool in[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = lane + k + 32 * h;
            in[h] = i < tl.z;
            const int s = tl.y + (in[h] ? i : 0);
            x[h][0] = __ldcg(d.vel + s); x[h][1] = __ldcg(d.vel + N + s); x[h][2] = __ldcg(d.vel + 2 * N + s);
            x[h][3] = __ldcg(d.evir + s); x[h][5] = __ldcg(d.epot + s);
            if (!d.single_type && in[h])
                in[h] = (int)__ldcg(reinterpret_cast<const long long*>(d.pos + s) + 3) == sel;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (!in[h]) x[h][0] = x[h][1] = x[h][2] = x[h][3] = x[h][5] = 0.0;
            x[h][4] = __fma_rn(x[h][2], x[h][2], __fma_rn(x[h][1], x[h][1], __dmul_rn(x[h][0], x[h][0])));
            a.cnt += __popc(__ballot_sync(0xffffffffu, in[h]));
            fx_run_add(a, x[h]);
        }
    }
}

// Lane q (below FX_NQ) of a row's readers and writers keeps quantity q, lane
// FX_NQ the count.  An infinity or NaN leaves its exponent, 0x7FF, as the grid.
struct FxTerm {
    __int128 s;
    int T;
};
__device__ __forceinline__ FxTerm fx_add(FxTerm a, FxTerm b) {
    const int T = max(a.T, b.T);
    return FxTerm{fx_align(a.s, a.T, T) + fx_align(b.s, b.T, T), T};
}
__device__ __forceinline__ void fx_set_term(FxRow* row, int q, FxTerm v) {
    if (q < FX_NQ) { row->s[q] = v.s; row->ex[q] = (unsigned short)v.T; }
    else if (q == FX_NQ) row->count = (long long)v.s;
}

// The warp's sums: the term of lane q in that lane.
__device__ __forceinline__ FxTerm fx_run_term(const FxRun& a) {
    const int lane = threadIdx.x & 31;
    FxTerm mine{(__int128)a.cnt, FX_T0};
#pragma unroll
    for (int q = 0; q < FX_NQ; ++q) {
        __int128 v = a.s[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += fx_shfl_xor(v, o);
        if (lane == q) mine = FxTerm{v, a.T[q]};
    }
    return mine;
}

// The block's terms from its warps', in warp order; valid in lanes 0 .. FX_NQ
// of the first warp.
__device__ __forceinline__ FxTerm fx_block_term(FxTerm v) {
    __shared__ __int128 sm_s[TILE / 32][FX_NQ + 1];
    __shared__ int sm_T[TILE / 32][FX_NQ + 1];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();   // a previous call's terms are read
    if (lane <= FX_NQ) { sm_s[w][lane] = v.s; sm_T[w][lane] = v.T; }
    __syncthreads();
    if (threadIdx.x <= FX_NQ)
        for (int i = 1; i < TILE / 32; ++i) v = fx_add(v, FxTerm{sm_s[i][lane], sm_T[i][lane]});
    return v;
}

__device__ void phase_partials_fx(const Dev& d, int sel) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int perw = fx_tiles_per_warp(d), per = perw * (TILE / 32);
    const int b0 = blockIdx.x * per, b1 = min(d.ntiles, b0 + per);
    if (b0 >= b1) return;
    const bool whole = d.tiles[b0].x == d.tiles[b1 - 1].x;
    int first = b0 + w * perw, rep = -1;
    const int end = min(b1, first + perw);
    FxRun run;
    run.init();
    for (int t = first; t < end; ++t) {
        const int4 tl = d.tiles[t];
        if (tl.x != rep && t > first) {
            fx_set_term(d.fx_part + first, lane, fx_run_term(run));
            run.init();
            first = t;
        }
        rep = tl.x;
        fx_run_tile(d, tl, sel, run);
    }
    FxTerm r = fx_run_term(run);
    if (whole) {
        r = fx_block_term(r);
        if (threadIdx.x <= FX_NQ) fx_set_term(d.fx_part + b0, lane, r);
    } else if (first < end) {
        fx_set_term(d.fx_part + first, lane, r);
    }
}

// Where candidate i of a replica with tiles [a, e) has its row, or -1: the
// blocks that hold tiles of it (nb of them) by their first warp, then the other
// warps of the first and the last block, which it may share with neighbours.
__device__ __forceinline__ int fx_row_at(const Dev& d, int a, int e, int perw, int i) {
    const int per = perw * (TILE / 32);
    const int f = a / per, l = (e - 1) / per, nb = l - f + 1;
    int b = f + i, w = 0;
    if (i >= nb) {
        const int k = i - nb;
        w = 1 + (k >> 1);
        b = (k & 1) ? l : f;
        if ((k & 1) && l == f) return -1;
    }
    const int s = b * per;
    if (a <= s && min(s + per, d.ntiles) <= e) return w == 0 ? s : -1;
    const int ws = max(a, s + w * perw);
    return ws < min(e, s + (w + 1) * perw) ? ws : -1;
}

// The rows of the replica with tiles [a, e) added exactly by the block: eight
// lanes a row, one quantity each, sixteen rows at a time, eight loads of each
// lane in flight; then the lanes of a quantity in a fixed order.  (1M atoms, 652
// rows, with the factors: 29 us; a thread a row, all quantities one after
// another, took 45.)  Deterministic: the same rows always go to the same threads
// in the same order.  Valid in lanes 0 .. FX_NQ of the first warp.
__device__ __forceinline__ FxTerm fx_replica_sum(const Dev& d, int a, int e) {
    constexpr int GROUPS = TILE / 8, BATCH = 8;
    const int perw = fx_tiles_per_warp(d), per = perw * (TILE / 32);
    const int n = (e - 1) / per - a / per + 1 + 2 * (TILE / 32 - 1);
    const int q = threadIdx.x & 7;
    FxTerm sum{0, FX_T0};
    for (int i0 = threadIdx.x >> 3; i0 < n; i0 += GROUPS * BATCH) {
        longlong2 h[BATCH];
        unsigned short T[BATCH];
        bool ok[BATCH];
#pragma unroll
        for (int k = 0; k < BATCH; ++k) {   // (nothing here depends on a load)
            const int i = i0 + GROUPS * k;
            const int at = i < n && q <= FX_NQ ? fx_row_at(d, a, e, perw, i) : -1;
            ok[k] = at >= 0;
            const FxRow* row = d.fx_part + (ok[k] ? at : 0);
            h[k] = __ldcg(reinterpret_cast<const longlong2*>(row) + (q < FX_NQ ? q : FX_NQ + 1));
            T[k] = __ldcg(row->ex + (q < FX_NQ ? q : 0));
        }
#pragma unroll
        for (int k = 0; k < BATCH; ++k) {
            const long long hi = ok[k] && q < FX_NQ ? h[k].y : 0, lo = ok[k] ? h[k].x : 0;
            const __int128 v = (__int128)(((unsigned __int128)(unsigned long long)hi << 64) | (unsigned long long)lo);
            sum = fx_add(sum, FxTerm{v, ok[k] && q < FX_NQ ? (int)T[k] : FX_T0});
        }
    }
#pragma unroll
    for (int o = 8; o < 32; o <<= 1)
        sum = fx_add(sum, FxTerm{fx_shfl_xor(sum.s, o), __shfl_xor_sync(0xffffffffu, sum.T, o)});
    return fx_block_term(sum);
}

// Mixed path, coupled steps: the replica's exact sums as doubles, then what
// phase_finalize2 does (box, T, P, coupling).  sum_i |v_i - vcm|^2 = sum
// |v_i|^2 - n |vcm|^2 (as sum v_i = n vcm): one pass over the atoms.
// The FP64 operations are one dependent chain of about 64 cycles each, so what
// can go beside it does: the quantities' conversions and divisions in lanes of
// one warp, the box in another's, the barostat's factor in a third.
__device__ void phase_finalize_fx(const Dev& d, const StepParams& sp, int sel, int block, int blocks) {
    __shared__ double sm_x[FX_NQ + 1], sm_vcm[3], sm_box[3];
    const double m = d.mass[sel];
    const int tid = threadIdx.x;
    for (int r = block; r < d.nrep; r += blocks) {   // one block per replica
        const RepDev R = load_rep(d.rep + r);
        RepDev* W = d.rep + r;
        // (every thread has read the record when this returns: it may be written)
        const FxTerm F = fx_replica_sum(d, R.tile_begin, R.tile_begin + R.ntiles);
        if (tid < 32) {
            const double nan = __longlong_as_double(0x7FF8000000000000ll);
            const bool nonfinite = __any_sync(0xffffffffu, tid < FX_NQ && F.T == 0x7FF);
            const double x = tid >= FX_NQ ? (double)(long long)F.s : nonfinite ? nan : fx_to_double(F.s, F.T);
            const double vc = x / __shfl_sync(0xffffffffu, x, FX_NQ);
            if (tid <= FX_NQ) sm_x[tid] = x;
            if (tid < 3) {
                sm_vcm[tid] = vc;
                W->vcm[tid] = vc;
                W->mom[tid] = x * m;
            }
            if (tid == FX_NQ) W->count = (long long)F.s;
        } else if (tid >= 64 && tid < 67) {
            const int a = tid - 64;
            double L = a == 0 ? R.box[0] : a == 1 ? R.box[1] : R.box[2];
            const int nc = a == 0 ? R.nc[0] : a == 1 ? R.nc[1] : R.nc[2];
            if (R.pending != 1.0) {
                for (int k = 0; k < d.ntypes; ++k) L *= R.pending;
                W->box[a] = L;
                W->cs[a] = L / (double)nc;
            }
            sm_box[a] = L;
        }
        __syncthreads();
        if (tid == 0 || tid == 32) {
            const double n = sm_x[FX_NQ], vv = sm_x[4], vir = sm_x[3];
            const double p1 =
                m * (vv - n * (sm_vcm[0] * sm_vcm[0] + sm_vcm[1] * sm_vcm[1] + sm_vcm[2] * sm_vcm[2]));
            if (tid == 0) {
                const double th = 0.5 * p1;
                const double T = temperature_of(th, (long long)n);
                W->msum = n * m; W->virsum = vir; W->ke = 0.5 * (m * vv); W->pe = sm_x[5] * 0.5;
                W->thermal = th; W->T = T;
                thermostat_factor(W, R, T, sp.dt);
            } else {
                const double volume = sm_box[0] * sm_box[1] * sm_box[2];
                const double P = (p1 + (-vir) * 0.5) / volume / 3.0;
                W->P = P;
                barostat_factor(W, R, P, sp.dt);
            }
        }
    }
}

// thermostat.rs:59-65: psi += psi_dot(T') * dt/2 with T' the temperature
// after the first kick, before the velocity scaling.
__device__ __forceinline__ void nh_update_psi(RepDev* W, const RepDev& R, double T, double dt) {
    if (!R.thermo_on || R.thermo_kind != 1) return;
    const double psi_dot = -((R.th_T0 / T) - 1.0) / R.th_tau;
    W->psi = R.psi + psi_dot * (dt / 2.0);
}

__device__ void phase_finalize_nh(const Dev& d, const StepParams& sp, int sel, int block, int blocks) {
    const int warps = (blocks * blockDim.x) >> 5;
    const int gw = (block * blockDim.x + threadIdx.x) >> 5;
    for (int r = gw; r < d.nrep; r += warps) {
        const RepDev R = load_rep(d.rep + r);
        double S1[1];
        warp_sum_tiles<1>(d, R, S1);
        const double sdv = S1[0];
        if ((threadIdx.x & 31) == 0) nh_update_psi(d.rep + r, R, temperature_of(0.5 * (d.mass[sel] * sdv), R.count), sp.dt);
    }
}

// ---------------------------------------------------------------------------
// Reference-order reductions: the sums of macro_parameters/*.rs are serial
// folds in the reference's atom order, s = RN(s + x_k), and keep its bits.
//
// A fold is cut into segments and every segment is run ahead of its turn, with
// real FP64 additions, from an approximate start (a tree prefix sum).  Let the
// true start be S, the simulated one Z, D = S - Z, and u the unit in the last
// place of the largest binade the segment's running values reach.  When D is
// a multiple of u and every running value of the simulation stays further
// than |D| from a power of two, both runs round every addition alike (the
// exact sums differ by a multiple of the rounding unit): the true end is the
// simulated end + D.  Where a term may make a tie, D must be a multiple of 2u
// (ties then go the same way).  So a segment is run once for each residue of
// S modulo u or 2u (S is a multiple of its own unit: one residue, or two with
// ties, where the segment stays in S's binade; 2, 4 or 8 where it climbs), and
// the segments are then stitched together in integer arithmetic on the bit
// patterns -- a run of segments that change neither binade nor sign as a
// prefix sum, others one by one.  A segment that climbs further, or comes too
// close to a power of two, is added term by term (a start that was exactly
// right is always taken over).
//
// GB300's FP64 add takes 64 cycles of its scheduler's pipe, so one thread that
// folds n terms needs n times that at the least; here 128 threads add at a
// time, and the terms are computed and laid out by the whole grid before.
// Against one thread per replica walking its atoms: a Berendsen T and P step
// of 1,000 atoms 1.85 -> 0.10 ms, a frame of 111,360 atoms with its macro
// parameters (the folds alone) 179 -> 1.2 ms.
constexpr int SS_SEGS = TILE;       // segments a round: one per thread
constexpr int SS_KMAX = 8;          // residues a segment is run for at most
constexpr long long SS_NEAR = 1ll << 30;   // |D| and distance to a power of two, in units

// Terms per segment of a fold of n terms, and where term k lies in scratch:
// rounds of SS_SEGS segments, inside a round [position][segment], so that a
// round's threads read side by side.
__host__ __device__ __forceinline__ int ss_len(long long n) {
    const long long want = (n + SS_SEGS - 1) / SS_SEGS;
    return want < 16 ? 16 : want > SS_PAD ? SS_PAD : (int)want;
}
__device__ __forceinline__ long long ss_place(long long k, long long n) {
    const int len = ss_len(n);
    const long long round = k / (SS_SEGS * len), base = round * (SS_SEGS * len);
    const long long left = n - base;
    const int segs = left >= SS_SEGS * len ? SS_SEGS : (int)((left + len - 1) / len);
    const int i = (int)(k - base);
    return base + (long long)(i % len) * segs + i / len;
}

struct SegRun {
    long long base;       // bits of the simulated start, its low residue bits cleared
    int mask;             // residues - 1
    int lim;              // |D| a start may differ by, in units of the start (0: not at all)
    int shift;            // exponent of the end - of the start
    int flip;             // the sign changed on the way
};

// t + x_0 + x_1 + ... over one segment.  LOOK: lo/hi the smallest and largest
// exponent field of the running values; near: one came within SS_NEAR units of
// a power of two (or is zero, subnormal or not finite); tie: an addition may
// have been a tie -- its term has no bits below half the result's unit (t is
// then a multiple of that half, too, unless the exponent jumped by two).
template <bool LOOK>
__device__ __forceinline__ double ss_run(const double* x, double c, int cnt, int stride, double t, int& lo, int& hi,
                                         bool& near, bool& tie) {
    int ep = LOOK ? (int)(((unsigned long long)__double_as_longlong(t) >> 52) & 0x7FFull) : 0;
    // eight terms at a time, the next eight in flight (+ 0 past the end: no change)
    double nx[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) nx[u] = u < cnt ? (x ? __ldcg(x + (size_t)u * stride) : c) : 0.0;
    for (int q = 0; q < cnt; q += 8) {
        double cur[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) cur[u] = nx[u];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int k = q + 8 + u;
            nx[u] = k < cnt ? (x ? __ldcg(x + (size_t)k * stride) : c) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const double v = cur[u];
            t = __dadd_rn(t, v);
            if (LOOK) {
                const unsigned long long b = (unsigned long long)__double_as_longlong(t);
                const int e = (int)((b >> 52) & 0x7FFull);
                const long long f = (long long)(b & 0x000FFFFFFFFFFFFFull);
                near |= e == 0 || e == 0x7FF || f <= SS_NEAR || f >= (1ll << 52) - SS_NEAR;
                lo = min(lo, e);
                hi = max(hi, e);
                const unsigned long long vb = (unsigned long long)__double_as_longlong(v) << 1;
                const int r = e - (int)(vb >> 53);
                tie |= vb != 0ull && (ep + 1 < e || r <= 1 || (r <= 54 && (vb << (64 - r)) == 0ull));
                ep = e;
            }
        }
    }
    return t;
}

// One segment taken over from the true start sb (bits); the sum's bits after it.
__device__ __forceinline__ bool ss_take(const SegRun& q, long long end, long long sb, int j, long long& out) {
    const long long dl = sb - (q.base | j);
    if (dl == 0) { out = end; return true; }
    if ((dl < 0 ? -dl : dl) >= q.lim || (sb >> 52) != (q.base >> 52)) return false;
    // same sign and exponent: dl is |S| - |Z| in units of S
    const long long du = q.flip ? -dl : dl;
    out = end + (q.shift >= 0 ? du >> q.shift : du << -q.shift);
    return true;
}

// ((0 + x_0) + x_1) + ... + x_(n-1), every addition rounded to nearest, by one
// block of SS_SEGS threads; x in the ss_place order, or null: every term is c.
// The result is valid in every thread.
__device__ double serial_sum(const double* x, long long n, double c) {
    __shared__ SegRun seg[SS_SEGS];
    __shared__ long long ends[SS_KMAX][SS_SEGS];   // bits of the simulated ends, by residue
    __shared__ double wsum[SS_SEGS / 32], s_sum;
    __shared__ int wruns[SS_SEGS / 32];
    __shared__ unsigned short todo[SS_SEGS * (SS_KMAX - 1)];   // runs to do: segment and residue
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int len = ss_len(n);
    if (tid == 0) s_sum = 0.0;
    for (long long base = 0; base < n; base += SS_SEGS * len) {
        const long long left = n - base;
        const int segs = left >= SS_SEGS * len ? SS_SEGS : (int)((left + len - 1) / len);
        const int cnt = (int)max(0ll, min((long long)len, left - (long long)tid * len));
        const double* xs = x ? x + base + tid : nullptr;
        int lo = 0x7FF, hi = 0;
        bool near = false, tie = false;
        // approximate starts: the sum so far plus a tree prefix of the segments' own sums
        double own = ss_run<false>(xs, c, cnt, segs, 0.0, lo, hi, near, tie), incl = own;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const double y = __shfl_up_sync(FULL, incl, off);
            if (lane >= off) incl = __dadd_rn(incl, y);
        }
        if (lane == 31) wsum[w] = incl;
        __syncthreads();
        double z = s_sum;
        for (int k = 0; k < w; ++k) z = __dadd_rn(z, wsum[k]);
        const double before = __shfl_up_sync(FULL, incl, 1);
        if (lane) z = __dadd_rn(z, before);
        // the runs
        const double end = ss_run<true>(xs, c, cnt, segs, z, lo, hi, near, tie);
        const long long zb = __double_as_longlong(z), eb = __double_as_longlong(end);
        const int ez = (int)((zb >> 52) & 0x7FF);
        SegRun r;
        const int climb = hi - ez + (tie ? 1 : 0);       // log2 of the residues (0 or less: one)
        const int deep = max(0, ez - lo);
        const bool ok = !near && ez > 0 && ez < 0x7FF && climb <= 3 && deep < 24;
        r.mask = ok && climb > 0 ? (1 << climb) - 1 : 0;
        r.base = zb & ~(long long)r.mask;
        // (a start lies a multiple of mask + 1 from the run it is taken over from, and
        // so does lim, a power of two: less than lim from z, too, whose running
        // values were looked at)
        r.lim = ok ? (int)(SS_NEAR >> deep) : 0;
        r.shift = (int)((eb >> 52) & 0x7FF) - ez;
        r.flip = (int)((unsigned long long)(zb ^ eb) >> 63);
        ends[zb & r.mask][tid] = eb;
        seg[tid] = r;
        // the other residues' runs, shared out over the block's threads
        int at = r.mask;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(FULL, at, off);
            if (lane >= off) at += y;
        }
        if (lane == 31) wruns[w] = at;
        __syncthreads();
        int runs = 0;
        for (int k = 0; k < SS_SEGS / 32; ++k) {
            if (k < w) at += wruns[k];
            runs += wruns[k];
        }
        for (int k = 1; k <= r.mask; ++k)
            todo[at - k] = (unsigned short)(tid * SS_KMAX + ((int)(zb & r.mask) ^ k));
        __syncthreads();
        for (int k = tid; k < runs; k += SS_SEGS) {
            const int g = todo[k] / SS_KMAX, j = todo[k] % SS_KMAX;
            const int cg = (int)min((long long)len, left - (long long)g * len);
            ends[j][g] = __double_as_longlong(ss_run<false>(x ? x + base + g : nullptr, c, cg, segs,
                                                            __longlong_as_double(seg[g].base | j), lo, hi, near, tie));
        }
        __syncthreads();
        // the stitching, by the first warp (every lane carries the sum)
        if (w == 0) {
            long long sb = __double_as_longlong(s_sum);
            for (int g0 = 0; g0 < segs; g0 += 32) {
                const SegRun q = seg[g0 + lane];
                const bool plain = q.lim > 0 && q.mask == 0 && q.shift == 0 && !q.flip;
                const long long gain = plain ? ends[0][g0 + lane] - q.base : 0;
                const unsigned plains = __ballot_sync(FULL, plain);
                const int m = min(32, segs - g0);
                int f = 0;
                while (f < m) {
                    if (plains >> f & 1u) {
                        // a run of plain segments from f on
                        long long sum = lane >= f ? gain : 0;
#pragma unroll
                        for (int off = 1; off < 32; off <<= 1) {
                            const long long y = __shfl_up_sync(FULL, sum, off);
                            if (lane >= off) sum += y;
                        }
                        const long long start = sb + sum - (lane >= f ? gain : 0);
                        long long out;
                        const bool good = plain && ss_take(q, start + gain, start, 0, out);
                        const unsigned stop = __ballot_sync(FULL, !good) & (0xFFFFFFFFu << f);
                        const int g = stop ? min(__ffs(stop) - 1, m) : m;
                        if (g > f) sb = __shfl_sync(FULL, start + gain, g - 1);
                        f = g;
                        if (f >= m) break;
                    }
                    const SegRun qf = seg[g0 + f];
                    const int j = (int)(sb & qf.mask);
                    if (!ss_take(qf, ends[j][g0 + f], sb, j, sb)) {
                        const int cf = (int)min((long long)len, left - (long long)(g0 + f) * len);
                        sb = __double_as_longlong(ss_run<false>(x ? x + base + g0 + f : nullptr, c, cf, segs,
                                                                __longlong_as_double(sb), lo, hi, near, tie));
                    }
                    ++f;
                }
            }
            if (lane == 0) s_sum = __longlong_as_double(sb);
        }
        __syncthreads();
    }
    return s_sum;
}

// Scratch row f of replica r (in the rebuild's tmp_d, which a reference-order
// engine allocates with SS_PAD more per row and replica).
__device__ __forceinline__ double* ss_row(const Dev& d, int f, int r, long long begin) {
    return d.tmp_d + (size_t)f * ((size_t)d.ntot + (size_t)SS_PAD * d.nrep) + begin + (long long)SS_PAD * r;
}

// The folds' terms, in the reference's order (by rank), into the scratch rows.
// Pass 1, rows 0-4: v m (3), kinetic energy, potential.
__device__ void phase_serial_terms1(const Dev& d, int sel, bool coupling) {
    const int N = d.ntot;
    const double m = d.mass[sel];
    for (int t = blockIdx.x; t < d.ntiles; t += gridDim.x) {
        const int4 tl = d.tiles[t];
        const RepDev& R = tile_rep(d, tl.x);
        const int i = tl.y + threadIdx.x;
        const long long k = i - R.begin - R.type_off[sel], n = R.type_off[sel + 1] - R.type_off[sel];
        if ((int)threadIdx.x >= tl.z || k < 0 || k >= n) continue;
        int s = __ldcg(d.slot_of_rank + i);
        if (s < 0 || s >= N) { atomicOr(d.err, E_BOUNDS); s = i; }
        const double vx = __ldcg(d.vel + s), vy = __ldcg(d.vel + N + s), vz = __ldcg(d.vel + 2 * N + s);
        const long long at = ss_place(k, n);
        ss_row(d, 0, tl.x, R.begin)[at] = vx * m;                                                  // mod.rs:12-25
        ss_row(d, 1, tl.x, R.begin)[at] = vy * m;
        ss_row(d, 2, tl.x, R.begin)[at] = vz * m;
        if (coupling) continue;
        ss_row(d, 3, tl.x, R.begin)[at] = m * (vx * vx + vy * vy + vz * vz) / 2.0;                 // energy.rs:14-22
        ss_row(d, 4, tl.x, R.begin)[at] = __ldcg(d.epot + s);                                      // energy.rs:40-49
    }
}

// Pass 2, with the centre-of-mass velocity from the pass-1 folds: row 0 thermal energy, rows 1-3 (as one) the pressure's three terms
// of every atom, row 4 the negated virial.
__device__ void phase_serial_terms2(const Dev& d, int sel) {
    const int N = d.ntot;
    const double m = d.mass[sel];
    __shared__ double vc[3];
    int vc_rep = -1;                  // replica vc[] belongs to (block-uniform)
    for (int t = blockIdx.x; t < d.ntiles; t += gridDim.x) {
        const int4 tl = d.tiles[t];
        const RepDev& R = tile_rep(d, tl.x);
        if (tl.x != vc_rep) {
            __syncthreads();
            const double* S = d.part + (size_t)R.tile_begin * 8;
            if (threadIdx.x < 3) vc[threadIdx.x] = __ldcg(S + threadIdx.x) / __ldcg(S + 3);
            __syncthreads();
            vc_rep = tl.x;
        }
        const int i = tl.y + threadIdx.x;
        const long long k = i - R.begin - R.type_off[sel], n = R.type_off[sel + 1] - R.type_off[sel];
        if ((int)threadIdx.x >= tl.z || k < 0 || k >= n) continue;
        int s = __ldcg(d.slot_of_rank + i);
        if (s < 0 || s >= N) { atomicOr(d.err, E_BOUNDS); s = i; }
        const double dx = __ldcg(d.vel + s) - vc[0], dy = __ldcg(d.vel + N + s) - vc[1],
                     dz = __ldcg(d.vel + 2 * N + s) - vc[2];
        const long long at = ss_place(k, n);
        ss_row(d, 0, tl.x, R.begin)[at] = m * (dx * dx + dy * dy + dz * dz) / 2.0;                 // energy.rs:25-37
        double* r1 = ss_row(d, 1, 3 * tl.x, 3 * R.begin);                                          // pressure.rs:13-18
        r1[ss_place(3 * k, 3 * n)] = m * dx * dx;
        r1[ss_place(3 * k + 1, 3 * n)] = m * dy * dy;
        r1[ss_place(3 * k + 2, 3 * n)] = m * dz * dz;
        ss_row(d, 4, tl.x, R.begin)[at] = -__ldcg(d.evir + s);
    }
}

// One block per fold.  Pass 1 folds land in the replica's
// first row of d.part (three momentum components, mass, kinetic energy,
// potential), pass 2 folds in its first row of d.cpart (thermal energy, the
// pressure's kinetic and virial sums).  Only the folds somebody reads run:
// a coupled step needs neither energy, and the pressure only with a barostat.
__device__ void phase_serial_folds(const Dev& d, int sel, int pass, bool coupling, bool nh_after_kick) {
    const int nf = pass == 1 ? (coupling || nh_after_kick ? 4 : 6) : (nh_after_kick ? 1 : 3);
    for (int w = blockIdx.x; w < d.nrep * nf; w += gridDim.x) {
        const int r = w / nf, f = w % nf;
        const RepDev* R = d.rep + r;
        if (pass == 2 && f > 0 && coupling && !__ldcg(&R->baro_on)) continue;
        const long long b = __ldcg(&R->begin);
        const long long n = __ldcg(&R->type_off[sel + 1]) - __ldcg(&R->type_off[sel]);
        const double* x;
        if (pass == 1) x = f == 3 ? nullptr : ss_row(d, f < 3 ? f : f - 1, r, b);
        else x = f == 0 ? ss_row(d, 0, r, b) : f == 1 ? ss_row(d, 1, 3 * r, 3 * b) : ss_row(d, 4, r, b);
        const double s = serial_sum(x, pass == 2 && f == 1 ? 3 * n : n, 1.0 * d.mass[sel]);
        if (threadIdx.x == 0)
            (pass == 1 ? d.part + (size_t)__ldcg(&R->tile_begin) * 8
                       : d.cpart + (size_t)__ldcg(&R->chunk_begin) * 8)[f] = s;
        __syncthreads();
    }
}

// What the folds give, per replica: the macro parameters (k_macro), or T, P
// and the coupling factors, or (nh_after_kick) the second psi update.
__device__ void phase_serial_finalize(const Dev& d, const StepParams& sp, int sel, bool coupling, bool nh_after_kick) {
    const int lane = threadIdx.x & 31;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (int r = gw; r < d.nrep; r += nw) {   // one warp per replica
        const RepDev R = load_rep(d.rep + r);
        RepDev* W = d.rep + r;
        const double* A = d.part + (size_t)R.tile_begin * 8;
        const double* B = d.cpart + (size_t)R.chunk_begin * 8;
        const long long n = __ldcg(&W->type_off[sel + 1]) - __ldcg(&W->type_off[sel]);
        const double th = __ldcg(B);
        if (nh_after_kick) {
            if (lane == 0) nh_update_psi(W, R, temperature_of(th, n), sp.dt);
            continue;
        }
        const bool pressure = !coupling || R.baro_on;
        const double kin = pressure ? __ldcg(B + 1) : 0.0, vir = pressure ? __ldcg(B + 2) : 0.0;
        const double m0 = __ldcg(A), m1 = __ldcg(A + 1), m2 = __ldcg(A + 2), msum = __ldcg(A + 3);
        double vc[3], box[3];
        finalize_frame(d, W, R, coupling, m0, m1, m2, msum, vc, box);
        if (lane == 0) {
            W->mom[0] = m0; W->mom[1] = m1; W->mom[2] = m2;
            W->msum = msum; W->count = n;
            if (pressure) W->virsum = -vir;
            if (!coupling) { W->ke = __ldcg(A + 4); W->pe = __ldcg(A + 5) / 2.0; }
        }
        finalize_coupling(W, R, sp, coupling, pressure, th, n, kin + vir * 0.5, box[0] * box[1] * box[2]);
    }
}

// Returns true when the launch must stop.
__device__ bool phase_serial(const Dev& d, const StepParams& sp, int sel, bool coupling, bool nh_after_kick = false) {
    phase_serial_terms1(d, sel, coupling || nh_after_kick);
    if (grid_barrier(d)) return true;
    phase_serial_folds(d, sel, 1, coupling, nh_after_kick);
    if (grid_barrier(d)) return true;
    phase_serial_terms2(d, sel);
    if (grid_barrier(d)) return true;
    phase_serial_folds(d, sel, 2, coupling, nh_after_kick);
    if (grid_barrier(d)) return true;
    phase_serial_finalize(d, sp, sel, coupling, nh_after_kick);
    return false;
}

// The stages that follow a pass over the tiles: chunk sums, then a finalize
// step.  With up to four chunks (a replica has one for every 32,768 atoms)
// the last block to arrive at the barrier does both; otherwise they are phases
// of their own.  Returns true when the launch must stop.
// The block has a warp for each of four chunks, or replicas, at a time: us in the
// last block / as phases, FP64 with both Berendsen couplings, 20 steps: replicas of
// 4,096 atoms 3465 / 3588 at 4, 4376 / 4283 at 6, 8889 / 8339 at 16, one system of
// 110,592 atoms (4 chunks) 10851 / 10999, of 442,368 (14) 31240 / 31007; mixed, 16
// replicas of 512 atoms in one launch 2292 / 1775, Nose-Hoover 3311 / 2365.
constexpr int THEN_MAX_CHUNKS = TILE / 32;
template <int NS, class F>
__device__ __forceinline__ bool sums_then(const Dev& d, F finalize) {
    if (d.nchunks <= THEN_MAX_CHUNKS)
        return grid_barrier_then(d, [&] {
            phase_chunk_sums<NS>(d, 0, 1);
            __syncthreads();
            finalize(0, 1);
        });
    if (grid_barrier(d)) return true;
    phase_chunk_sums<NS>(d, blockIdx.x, gridDim.x);
    if (grid_barrier(d)) return true;
    finalize(blockIdx.x, gridDim.x);
    return grid_barrier(d);
}

// psi += psi_dot(T_t) * dt/2 with T_t the temperature of the atoms of type t
// (thermostat.rs:35-39 before the kick, :59-65 after it), per replica with a
// Nose-Hoover thermostat.  Returns true when the launch must stop.
__device__ __forceinline__ bool nh_psi_of_type(const Dev& d, const StepParams& sp, int t) {
    if (d.refmode) return phase_serial(d, sp, t, false, true) || grid_barrier(d);
    phase_partials1(d, t);
    if (sums_then<7>(d, [&](int b, int n) { phase_finalize1(d, t, b, n); })) return true;
    phase_partials2(d, t);
    return sums_then<1>(d, [&](int b, int n) { phase_finalize_nh(d, sp, t, b, n); });
}

// ---------------------------------------------------------------------------
// Drift: integrator.rs:30-47 for every atom; mirror + displacement.
// Nose-Hoover steps: the first kick alone (integrator.rs:30-36), so the
// thermostat can read the temperature between kick and scaling
// (thermostat.rs:47-52,59-65).
// FM (here and in the phases below): the mixed path's fused multiply-adds,
// a compile-time constant -- the callers dispatch on d.mixed once per phase.
template <bool FM>
__device__ void phase_kick(const Dev& d, const StepParams& sp) {
    const int N = d.ntot;
    for (int t = blockIdx.x; t < d.ntiles; t += gridDim.x) {
        const int4 tl = d.tiles[t];
        const int s = tl.y + threadIdx.x;
        if ((int)threadIdx.x >= tl.z) continue;
        const int ty = (int)reinterpret_cast<const long long*>(d.pos + s)[3];
        const double c = sp.kick_c[ty];
        for (int a = 0; a < 3; ++a)
            d.vel[(size_t)a * N + s] = madd(d.vel[(size_t)a * N + s], d.frc[(size_t)a * N + s], c, FM);
    }
}

// Inputs of one atom's drift, loaded one tile ahead (the loop is latency-
// bound: a block walks its tiles one after another).
struct DriftIn {
    double4_32a p;
    double v[3], f[3];
    int cell;
    float4 m0;
};

__device__ __forceinline__ void drift_load(const Dev& d, int s, bool kicked, DriftIn& in) {
    const int N = d.ntot;
    in.p = d.pos[s];
    for (int a = 0; a < 3; ++a) in.v[a] = __ldcg(d.vel + (size_t)a * N + s);
    if (!kicked)
        for (int a = 0; a < 3; ++a) in.f[a] = __ldcg(d.frc + (size_t)a * N + s);
    in.cell = d.cell[s];
    in.m0 = d.mir0[s];
}

template <bool FM>
__device__ void phase_drift(const Dev& d, const StepParams& sp, bool kicked) {
    __shared__ float smx[32];
    __shared__ float tc[7];   // box (FP32), half box, scale since the last rebuild
    const int N = d.ntot;
    constexpr bool fm = FM;
    int tc_rep = -1;          // replica tc[] and disp belong to (block-uniform)
    float disp = 0.f;         // largest displacement seen by this thread in replica tc_rep
    // a contiguous run of tiles per block: the replica (and with it the
    // constants and the displacement maximum) changes only at its boundaries
    const int per = (d.ntiles + gridDim.x - 1) / gridDim.x;
    const int t_end = min(d.ntiles, ((int)blockIdx.x + 1) * per);
    int t = blockIdx.x * per;
    int4 tl = t < t_end ? d.tiles[t] : make_int4(0, 0, 0, 0);
    DriftIn cur;
    if (t < t_end && (int)threadIdx.x < tl.z) drift_load(d, tl.y + threadIdx.x, kicked, cur);
    for (; t < t_end; ++t) {
        // the next tile's inputs in flight while this one computes
        const int tn = t + 1;
        int4 tln = make_int4(0, 0, 0, 0);
        DriftIn nxt;
        if (tn < t_end) {
            tln = d.tiles[tn];
            if ((int)threadIdx.x < tln.z) drift_load(d, tln.y + threadIdx.x, kicked, nxt);
        }
        if (tl.x != tc_rep) {
            if (tc_rep >= 0) {
                const float m = block_max(disp, smx);
                if (threadIdx.x == 0) atomicMax(&d.rep[tc_rep].max_disp_bits, __float_as_uint(m));
                disp = 0.f;
            }
        }
        const RepDev& R = tile_rep(d, tl.x);
        if (tl.x != tc_rep) {
            __syncthreads();
            if (threadIdx.x == 0) drift_consts(R, tc);
            __syncthreads();
            tc_rep = tl.x;
        }
        const int s = tl.y + threadIdx.x;
        if ((int)threadIdx.x < tl.z) {
            double4_32a p = cur.p;
            if (sp.do_drift) {
                const int ty = type_of(p);
                const double c = sp.kick_c[ty];
                double vx = cur.v[0], vy = cur.v[1], vz = cur.v[2];
                if (!kicked) {
                    vx = madd(vx, cur.f[0], c, fm);                      // :30-36 kick
                    vy = madd(vy, cur.f[1], c, fm);
                    vz = madd(vz, cur.f[2], c, fm);
                }
                if (R.thermo_on) {                                       // thermostat.rs:54-58
                    vx = dmul_nospec(vx, R.lambda); vy = dmul_nospec(vy, R.lambda);
                    vz = dmul_nospec(vz, R.lambda);
                }
                d.vel[s] = vx; d.vel[N + s] = vy; d.vel[2 * N + s] = vz;
                double x = p.x, y = p.y, z = p.z;
                if (__double_as_longlong(R.pending) != 0x3FF0000000000000ll) {   // != 1.0; barostat.rs:46-48
                    x = dmul_nospec(x, R.pending); y = dmul_nospec(y, R.pending);
                    z = dmul_nospec(z, R.pending);
                }
                p.x = x; p.y = y; p.z = z;
                p = drift_wrap(p, vx, vy, vz, sp.dt, R.box, fm);         // :42-46 drift
                d.pos[s] = p;
            }
            const int cl = cur.cell - R.cell_base;
            // cl is out of range only before the first binning (fresh upload);
            // the forced rebuild that follows computes the mirror then.
            if (cl >= 0 && cl < R.nc[0] * R.nc[1] * R.nc[2]) {
                const float4 m = mirror_of(p, cl, R, tc + 3, fm);
                d.mir[s] = m;
                disp = fmaxf(disp, mirror_disp(m, cur.m0, tc));
            }
        }
        tl = tln;
        cur = nxt;
    }
    if (tc_rep >= 0) {
        const float m = block_max(disp, smx);
        if (threadIdx.x == 0) atomicMax(&d.rep[tc_rep].max_disp_bits, __float_as_uint(m));
    }
}

// Per replica: consume the pending barostat factor, decide on a rebuild.
__device__ void phase_decide(const Dev& d, const StepParams& sp, int block, int blocks) {
    const int gt = block * blockDim.x + threadIdx.x;
    const int nt = blocks * blockDim.x;
    for (int r = gt; r < d.nrep; r += nt) decide_replica(d, sp, r);
}

// ---------------------------------------------------------------------------
// Rebuild phases (only tiles/cells of replicas with rebuild set do work).

// The rebuild work list (block 0; the grid barrier after the zero phase
// publishes it): the rebuilding replicas with prefix offsets of their cells
// (the grid the decide phase set; one cell in brute mode) and tiles, so the
// rebuild phases and the list build visit only their work.  Replicas the
// paired list build does not take come first (pass 0), the others after.
__device__ void phase_work_list(const Dev& d) {
    __shared__ int wsum[3][TILE / 32];
    __shared__ int carry[3];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int* rb = d.rb;
    int* ids = rb + 2;
    int* coff = rb + 2 + d.nrep;
    int* toff = rb + 3 + 2 * d.nrep;
    if (threadIdx.x < 3) carry[threadIdx.x] = 0;
    __syncthreads();
    for (int pass = 0; pass < 2; ++pass) {
        for (int base = 0; base < d.nrep; base += blockDim.x) {
            const int r = base + threadIdx.x;
            int v[3] = {0, 0, 0};
            if (r < d.nrep) {
                const RepDev* W = d.rep + r;
                const int cells = __ldcg(&W->nc[0]) * __ldcg(&W->nc[1]) * __ldcg(&W->nc[2]);
                const bool paired = list_paired(W->n, cells) && __ldcg(&W->mode) == MODE_CELLS;
                if (__ldcg(&W->rebuild) && paired == (pass == 1)) {
                    v[0] = 1;
                    v[1] = cells;
                    v[2] = W->ntiles;
                }
            }
            int inc[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                inc[q] = v[q];
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, inc[q], off);
                    if (lane >= off) inc[q] += y;
                }
                if (lane == 31) wsum[q][w] = inc[q];
            }
            __syncthreads();
            if (v[0]) {
                int ex[3];
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    ex[q] = carry[q] + inc[q] - v[q];
                    for (int k = 0; k < w; ++k) ex[q] += wsum[q][k];
                }
                ids[ex[0]] = r;
                coff[ex[0]] = ex[1];
                toff[ex[0]] = ex[2];
            }
            __syncthreads();
            if (threadIdx.x < 3)
                for (int k = 0; k < (int)(blockDim.x >> 5); ++k) carry[threadIdx.x] += wsum[threadIdx.x][k];
            __syncthreads();
        }
        if (pass == 0 && threadIdx.x == 0) rb[1] = carry[0];
    }
    if (threadIdx.x == 0) {
        rb[0] = carry[0];
        coff[carry[0]] = carry[1];
        toff[carry[0]] = carry[2];
    }
}

__device__ void phase_zero_cells(const Dev& d, int block, int blocks) {
    const int gt = block * blockDim.x + threadIdx.x;
    const int nt = blocks * blockDim.x;
    for (int c = gt; c < d.ncells; c += nt) {
        const int r = d.cell_rep[c];
        if (__ldcg(&d.rep[r].rebuild)) d.cell_count[c] = 0;
    }
    if (d.pairs)
        for (int r = gt; r < d.nrep; r += nt)
            if (__ldcg(&d.rep[r].rebuild)) d.pair_count[r] = 0;
}

// Cell of every atom, and its slot among the cell's atoms in arrival order
// (tmp_i row 3): one counter atomic per distinct cell in a warp -- the atoms
// are mostly still sorted by cell, so a warp covers only a few.
__device__ void phase_bin(const Dev& d) {
    const int N = d.ntot;
    const int lane = threadIdx.x & 31;
    // a contiguous run of the rebuilding replicas' tiles per block (the
    // replica record is fetched only when the run crosses into the next)
    const int m = __ldcg(d.rb), nw = __ldcg(rb_tile_off(d) + m);
    const int per = (nw + gridDim.x - 1) / gridDim.x;
    const int w_end = min(nw, ((int)blockIdx.x + 1) * per);
    int wi = blockIdx.x * per;
    int i = wi < w_end ? rb_locate(rb_tile_off(d), m, wi) - 1 : 0;
    int next = wi, shift = 0;   // where replica i's run ends; tile index - work index inside it
    for (; wi < w_end; ++wi) {
        while (wi >= next) {
            ++i;
            next = __ldcg(rb_tile_off(d) + i + 1);
            shift = d.rep[__ldcg(rb_rep(d) + i)].tile_begin - __ldcg(rb_tile_off(d) + i);
        }
        const int4 tl = d.tiles[wi + shift];
        const RepDev& R = tile_rep(d, tl.x);
        const int s = tl.y + threadIdx.x;
        const bool act = (int)threadIdx.x < tl.z;
        const unsigned am = __ballot_sync(0xffffffffu, act);
        if (!act) continue;
        const double4_32a p = d.pos[s];
        int local = 0;
        if (R.mode == MODE_CELLS) {
            const double x[3] = {p.x, p.y, p.z};
            int c[3];
            for (int a = 0; a < 3; ++a) {
                // wrapped positions are >= 0: truncation is the floor
                const int ci = __double2int_rz(__dmul_rn(x[a], R.inv_cs[a]));
                c[a] = min(max(ci, 0), R.nc[a] - 1);
            }
            local = (c[0] * R.nc[1] + c[1]) * R.nc[2] + c[2];
        }
        const int cell = R.cell_base + local;
        d.tmp_i[2 * (size_t)N + s] = cell;
        const unsigned peers = __match_any_sync(am, cell);
        const int leader = __ffs(peers) - 1;
        int base = 0;
        if (lane == leader) base = atomicAdd(d.cell_count + cell, __popc(peers));
        base = __shfl_sync(am, base, leader);
        d.tmp_i[3 * (size_t)N + s] = base + __popc(peers & ((1u << lane) - 1u));
    }
}

// Exclusive scan of cell counts over all cells (block chunks + block sums).
__device__ void phase_scan_a(const Dev& d, int chunk) {
    __shared__ double sm[32];
    const int b0 = blockIdx.x * chunk, b1 = min(b0 + chunk, d.ncells);
    double v[1] = {0.0};
    for (int c = b0 + threadIdx.x; c < b1; c += blockDim.x) v[0] += (double)__ldcg(d.cell_count + c);
    block_sum<1>(v, sm);
    if (threadIdx.x == 0) d.bsum[blockIdx.x] = (int)v[0];
}

// Exclusive scan of the per-block sums by one block (each thread a contiguous run).
__device__ void phase_scan_b(const Dev& d) {
    __shared__ int part[TILE];
    const int G = gridDim.x;
    const int per = (G + blockDim.x - 1) / blockDim.x;
    const int b0 = threadIdx.x * per, b1 = min(b0 + per, G);
    int sum = 0;
    for (int b = b0; b < b1; ++b) sum += __ldcg(d.bsum + b);
    part[threadIdx.x] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int i = 0; i < (int)blockDim.x; ++i) { const int t = part[i]; part[i] = run; run += t; }
        d.cell_start[d.ncells] = run;
    }
    __syncthreads();
    int run = part[threadIdx.x];
    for (int b = b0; b < b1; ++b) {
        const int v = __ldcg(d.bsum + b);
        d.bsum[b] = run;
        run += v;
    }
}

__device__ void phase_scan_c(const Dev& d, int b0, int b1, int before) {
    __shared__ int wsum[32];
    __shared__ int carry;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (threadIdx.x == 0) carry = before;
    __syncthreads();
    for (int base = b0; base < b1; base += blockDim.x) {
        const int c = base + threadIdx.x;
        const int x = (c < b1) ? __ldcg(d.cell_count + c) : 0;
        int inc = x;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, off);
            if (lane >= off) inc += y;
        }
        if (lane == 31) wsum[w] = inc;
        __syncthreads();
        if (threadIdx.x == 0) {
            int run = 0;
            for (int i = 0; i < nw; ++i) { const int t = wsum[i]; wsum[i] = run; run += t; }
        }
        __syncthreads();
        if (c < b1) d.cell_start[c] = carry + wsum[w] + inc - x;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry += wsum[w] + inc;
        __syncthreads();
    }
}

// carry_forces: also move frc/epot/evir (a refresh that no force evaluation
// follows); a step's force pass rewrites them after the rebuild anyway.
// One atom's move to the scratch copy: its inputs (ScatterIn, loaded for two
// tiles before either is stored, so a thread has both in flight) and its
// slot, perm[slot] = s.
struct ScatterIn {
    double4_32a p;
    double v[3];
    int cell, slot, orig, rank;
};

__device__ __forceinline__ void scatter_load(const Dev& d, const RepDev& R, int s, ScatterIn& in) {
    const int N = d.ntot;
    in.cell = d.tmp_i[2 * (size_t)N + s];
    const int within = d.tmp_i[3 * (size_t)N + s];
    in.p = d.pos[s];
    for (int k = 0; k < 3; ++k) in.v[k] = d.vel[(size_t)k * N + s];
    in.orig = d.orig[s];
    in.rank = d.rank[s];
    // brute mode: one cell holds the whole replica in its current order
    const bool cell_ok = in.cell >= R.cell_base && in.cell < R.cell_base + R.cell_cap;
    in.slot = R.mode == MODE_BRUTE ? s : (cell_ok ? __ldcg(d.cell_start + in.cell) + within : -1);
    if (!cell_ok) in.cell = -1;
}

__device__ __forceinline__ void scatter_store(const Dev& d, const RepDev& R, int s, const ScatterIn& in,
                                              bool carry_forces) {
    const int N = d.ntot;
    if (in.cell < 0 || in.slot < R.begin || in.slot >= R.begin + R.n) { atomicOr(d.err, E_CELLS); return; }
    d.perm[in.slot] = s;
    d.tmp_pos[s] = in.p;
    for (int k = 0; k < 3; ++k) d.tmp_d[(size_t)k * N + s] = in.v[k];
    if (carry_forces) {
        for (int k = 0; k < 3; ++k) d.tmp_d[(size_t)(3 + k) * N + s] = d.frc[(size_t)k * N + s];
        d.tmp_d[(size_t)6 * N + s] = d.epot[s];
        d.tmp_d[(size_t)7 * N + s] = d.evir[s];
    }
    d.tmp_i[s] = in.orig;
    d.tmp_i[(size_t)N + s] = in.rank;
}

__device__ void phase_scatter(const Dev& d, bool carry_forces) {
    // a contiguous run of the rebuilding replicas' tiles per block (the
    // replica record is fetched only when the run crosses into the next);
    // two tiles of a replica at a time
    const int m = __ldcg(d.rb), nw = __ldcg(rb_tile_off(d) + m);
    const int per = (nw + gridDim.x - 1) / gridDim.x;
    const int w_end = min(nw, ((int)blockIdx.x + 1) * per);
    int wi = blockIdx.x * per;
    int i = wi < w_end ? rb_locate(rb_tile_off(d), m, wi) - 1 : 0;
    int next = wi, shift = 0;   // where replica i's run ends; tile index - work index inside it
    while (wi < w_end) {
        while (wi >= next) {
            ++i;
            next = __ldcg(rb_tile_off(d) + i + 1);
            shift = d.rep[__ldcg(rb_rep(d) + i)].tile_begin - __ldcg(rb_tile_off(d) + i);
        }
        const bool two = wi + 1 < w_end && wi + 1 < next;
        const int4 ta = d.tiles[wi + shift];
        const int4 tb = two ? d.tiles[wi + 1 + shift] : make_int4(0, 0, 0, 0);
        const RepDev& R = tile_rep(d, ta.x);
        const int sa = ta.y + threadIdx.x, sb = tb.y + threadIdx.x;
        const bool aa = (int)threadIdx.x < ta.z, ab = two && (int)threadIdx.x < tb.z;
        ScatterIn xa, xb;
        if (aa) scatter_load(d, R, sa, xa);
        if (ab) scatter_load(d, R, sb, xb);
        if (aa) scatter_store(d, R, sa, xa, carry_forces);
        if (ab) scatter_store(d, R, sb, xb, carry_forces);
        wi += two ? 2 : 1;
    }
}

// Cells of up to 32 * SORT_MAX_PER_LANE atoms are ranked by shuffles; more
// crowded ones by a serial insertion sort.
constexpr int SORT_MAX_PER_LANE = 4;

// The geometry of one replica that the gather needs, read through L2 (the
// decide phase of this launch may have changed the box).
struct CellGeom {
    double box[3], cs[3];
    float hL[3];
    int nc[3];
    int cell_base, mode, n, r;
    long long begin;
};

__device__ __forceinline__ void load_geom(const Dev& d, int r, CellGeom& g) {
    const RepDev* W = d.rep + r;
    for (int a = 0; a < 3; ++a) {
        g.box[a] = __ldcg(&W->box[a]);
        g.cs[a] = __ldcg(&W->cs[a]);
        g.nc[a] = __ldcg(&W->nc[a]);
        g.hL[a] = 0.5f * dbl_to_flt_rn(g.box[a]);
    }
    g.cell_base = __ldcg(&W->cell_base);
    g.mode = __ldcg(&W->mode);
    g.n = __ldcg(&W->n);
    g.begin = __ldcg(&W->begin);
    g.r = r;
}

// Scratch element i (the atom's index before the rebuild) to slot s of cell
// c: its scratch row loaded (gather_load), then written to the slot with a
// fresh mirror (gather_store).
struct GatherIn {
    double4_32a p;
    double v[3];
    int orig, rank;
};

__device__ __forceinline__ void gather_load(const Dev& d, int i, GatherIn& in) {
    const int N = d.ntot;
    in.p = ldcg4(d.tmp_pos + i);
    for (int k = 0; k < 3; ++k) in.v[k] = __ldcg(d.tmp_d + (size_t)k * N + i);
    in.orig = __ldcg(d.tmp_i + i);
    in.rank = __ldcg(d.tmp_i + (size_t)N + i);
}

template <bool FM>
__device__ __forceinline__ void gather_store(const Dev& d, const CellGeom& g, int c, int i, int s,
                                             const GatherIn& in, bool carry_forces) {
    const int N = d.ntot;
    d.pos[s] = in.p;
    for (int k = 0; k < 3; ++k) d.vel[(size_t)k * N + s] = in.v[k];
    if (carry_forces) {
        for (int k = 0; k < 3; ++k) d.frc[(size_t)k * N + s] = __ldcg(d.tmp_d + (size_t)(3 + k) * N + i);
        d.epot[s] = __ldcg(d.tmp_d + (size_t)6 * N + i);
        d.evir[s] = __ldcg(d.tmp_d + (size_t)7 * N + i);
    }
    d.orig[s] = in.orig;
    d.rank[s] = in.rank;
    d.cell[s] = c;
    const float4 m = mirror_of(in.p, c - g.cell_base, g, g.hL, FM);
    d.mir[s] = m;
    d.mir0[s] = m;
    if (in.rank >= 0 && in.rank < N) d.slot_of_rank[in.rank] = s;
    else atomicOr(d.err, E_BOUNDS);
}

__device__ __forceinline__ bool gather_ok(const Dev& d, const CellGeom& g, int i, int s) {
    if (i < g.begin || i >= g.begin + g.n || s < g.begin || s >= g.begin + g.n) {
        atomicOr(d.err, E_BOUNDS);
        return false;
    }
    return true;
}

template <bool FM>
__device__ __forceinline__ void gather_one(const Dev& d, const CellGeom& g, int c, int i, int s,
                                           bool carry_forces) {
    if (!gather_ok(d, g, i, s)) return;
    GatherIn in;
    gather_load(d, i, in);
    gather_store<FM>(d, g, c, i, s, in, carry_forces);
}

// One cell: canonical order (ascending caller index) and the gather.
template <bool FM>
__device__ void sort_gather_cell(const Dev& d, const CellGeom& g, int c, int b, int n, bool carry_forces) {
    const int N = d.ntot;
    const int lane = threadIdx.x & 31;
    if (g.mode == MODE_BRUTE) {
        // the scatter kept the replica's order: slot i holds element i
        for (int k = lane; k < n; k += 32) gather_one<FM>(d, g, c, __ldcg(d.perm + b + k), b + k, carry_forces);
    } else if (n <= 32 * SORT_MAX_PER_LANE) {
        int e[SORT_MAX_PER_LANE], key[SORT_MAX_PER_LANE], rank[SORT_MAX_PER_LANE];
#pragma unroll
        for (int q = 0; q < SORT_MAX_PER_LANE; ++q) {
            const int i = q * 32 + lane;
            e[q] = i < n ? __ldcg(d.perm + b + i) : -1;
            const bool ok = e[q] >= 0 && e[q] < N;
            if (i < n && !ok) atomicOr(d.err, E_BOUNDS);
            key[q] = ok ? __ldcg(d.tmp_i + e[q]) : 0x7FFFFFFF;
            rank[q] = 0;
        }
        if (n <= 32) {
            // one key a lane, n shuffles
            for (int k = 0; k < n; ++k) rank[0] += (__shfl_sync(0xffffffffu, key[0], k) < key[0]) ? 1 : 0;
        } else {
#pragma unroll
            for (int q2 = 0; q2 < SORT_MAX_PER_LANE; ++q2) {
                if (q2 * 32 >= n) break;
                for (int k = 0; k < 32; ++k) {
                    const int kk = __shfl_sync(0xffffffffu, key[q2], k);
#pragma unroll
                    for (int q = 0; q < SORT_MAX_PER_LANE; ++q) rank[q] += (kk < key[q]) ? 1 : 0;
                }
            }
        }
#pragma unroll
        for (int q = 0; q < SORT_MAX_PER_LANE; ++q) {
            const int i = q * 32 + lane;
            if (i < n && e[q] >= 0 && e[q] < N && rank[q] < n) gather_one<FM>(d, g, c, e[q], b + rank[q], carry_forces);
        }
    } else {
        // very crowded cell: serial insertion sort of the slots, then the gather
        if (lane == 0) {
            for (int a = 1; a < n; ++a) {
                const int e0 = __ldcg(d.perm + b + a);
                if (e0 < 0 || e0 >= N) { atomicOr(d.err, E_BOUNDS); break; }
                const int k0 = __ldcg(d.tmp_i + e0);
                int k = a - 1;
                while (k >= 0) {
                    const int f = __ldcg(d.perm + b + k);
                    if (f < 0 || f >= N || __ldcg(d.tmp_i + f) <= k0) break;
                    d.perm[b + k + 1] = f;
                    --k;
                }
                d.perm[b + k + 1] = e0;
            }
        }
        __syncwarp();
        for (int k = lane; k < n; k += 32) gather_one<FM>(d, g, c, __ldcg(d.perm + b + k), b + k, carry_forces);
    }
}

// Canonical order inside each cell (ascending caller index), and every atom
// moved from the scratch copy to its final slot.  One warp per cell: an
// element's rank is the number of smaller keys (keys are distinct caller
// indices), found by shuffling the cell's keys across the warp; the warp then
// gathers the cell's atoms to cell_start + rank.  A warp takes two
// neighbouring cells (work items 2w, 2w + 1) at a time: when both are in the
// same cell-mode replica and hold at most 32 atoms, their loads, ranks and
// gathers interleave, so twice the memory requests are in flight (the phase
// is latency-bound); otherwise the cells go one after the other.  Cells of
// brute-mode replicas are already in canonical (identity) order.
// carry_forces: also move frc/epot/evir (a refresh that no force evaluation
// follows).
template <bool FM>
__device__ void phase_sort_gather(const Dev& d, bool carry_forces) {
    const int N = d.ntot;
    const int lane = threadIdx.x & 31;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    CellGeom g;
    g.r = -1;
    const int m = __ldcg(d.rb), nwork = __ldcg(rb_cell_off(d) + m);
    for (int wp = gw; 2 * wp < nwork; wp += nw) {
        const int w0 = 2 * wp;
        const int i = rb_locate(rb_cell_off(d), m, w0);
        const int r = __ldcg(rb_rep(d) + i);
        const int off0 = __ldcg(rb_cell_off(d) + i), off1 = __ldcg(rb_cell_off(d) + i + 1);
        const int c0 = __ldcg(&d.rep[r].cell_base) + w0 - off0;
        const bool two = w0 + 1 < off1;   // the second cell is in the same replica
        const int b0 = __ldcg(d.cell_start + c0), n0 = __ldcg(d.cell_count + c0);
        const int b1 = two ? __ldcg(d.cell_start + c0 + 1) : 0, n1 = two ? __ldcg(d.cell_count + c0 + 1) : 0;
        if (r != g.r) load_geom(d, r, g);
        const bool in0 = b0 >= 0 && b0 + n0 <= N, in1 = b1 >= 0 && b1 + n1 <= N;
        if (two && g.mode == MODE_CELLS && n0 <= 32 && n1 <= 32 && in0 && in1) {
            const int e0 = lane < n0 ? __ldcg(d.perm + b0 + lane) : -1;
            const int e1 = lane < n1 ? __ldcg(d.perm + b1 + lane) : -1;
            const bool ok0 = e0 >= 0 && e0 < N, ok1 = e1 >= 0 && e1 < N;
            if ((lane < n0 && !ok0) || (lane < n1 && !ok1)) atomicOr(d.err, E_BOUNDS);
            const int key0 = ok0 ? __ldcg(d.tmp_i + e0) : 0x7FFFFFFF;
            const int key1 = ok1 ? __ldcg(d.tmp_i + e1) : 0x7FFFFFFF;
            int rank0 = 0, rank1 = 0;
            const int nm = max(n0, n1);
            for (int k = 0; k < nm; ++k) {
                rank0 += (__shfl_sync(0xffffffffu, key0, k) < key0) ? 1 : 0;
                rank1 += (__shfl_sync(0xffffffffu, key1, k) < key1) ? 1 : 0;
            }
            const bool go0 = ok0 && rank0 < n0 && gather_ok(d, g, e0, b0 + rank0);
            const bool go1 = ok1 && rank1 < n1 && gather_ok(d, g, e1, b1 + rank1);
            GatherIn g0, g1;
            if (go0) gather_load(d, e0, g0);
            if (go1) gather_load(d, e1, g1);
            if (go0) gather_store<FM>(d, g, c0, e0, b0 + rank0, g0, carry_forces);
            if (go1) gather_store<FM>(d, g, c0 + 1, e1, b1 + rank1, g1, carry_forces);
            continue;
        }
        if (n0 > 0) {
            if (in0) sort_gather_cell<FM>(d, g, c0, b0, n0, carry_forces);
            else if (lane == 0) atomicOr(d.err, E_CELLS);
        }
        if (w0 + 1 >= nwork) continue;
        // the second cell on its own (it may begin the next replica)
        int r1 = r, c1 = c0 + 1, bb = b1, nn = n1;
        if (!two) {
            r1 = __ldcg(rb_rep(d) + i + 1);
            c1 = __ldcg(&d.rep[r1].cell_base);
            bb = __ldcg(d.cell_start + c1);
            nn = __ldcg(d.cell_count + c1);
            if (r1 != g.r) load_geom(d, r1, g);
        }
        if (nn > 0) {
            if (bb >= 0 && bb + nn <= N) sort_gather_cell<FM>(d, g, c1, bb, nn, carry_forces);
            else if (lane == 0) atomicOr(d.err, E_CELLS);
        }
    }
}

// Verlet neighbour list with skin: every j (of type >= type i, the
// reference's t1 <= t2 loop, potential.rs:171-172) within rlist of i.
// Per-atom builder, used for brute-mode replicas (the whole box is one cell).
__device__ void phase_build_list(const Dev& d) {
    __shared__ int smi[32];
    const int cap = d.cap;
    for (int t = blockIdx.x; t < d.ntiles; t += gridDim.x) {
        const int4 tl = d.tiles[t];
        const RepDev& R = tile_rep(d, tl.x);
        if (!R.rebuild || R.mode == MODE_CELLS) continue;  // cell-mode replicas: k_build_list
        const float rl = (float)(R.rlist * (1.0 + 1e-5));
        const float rl2 = rl * rl;
        const int s = tl.y + threadIdx.x;
        const int tpa = R.tpa;
        int cnt = 0;
        if ((int)threadIdx.x < tl.z) {
            const float4 xi = __ldcg(d.mir + s);
            const int ti = type_of(xi);
            const float L[3] = {(float)R.box[0], (float)R.box[1], (float)R.box[2]};
            for (int j = (int)R.begin; j < (int)R.begin + R.n; ++j) {
                if (j == s) continue;
                const float4 xj = __ldcg(d.mir + j);
                if (type_of(xj) < ti) continue;
                float e[3] = {xj.x - xi.x, xj.y - xi.y, xj.z - xi.z};
                for (int a = 0; a < 3; ++a) {
                    if (e[a] < -0.5f * L[a]) e[a] += L[a];
                    else if (e[a] > 0.5f * L[a]) e[a] -= L[a];
                }
                if (e[0] * e[0] + e[1] * e[1] + e[2] * e[2] < rl2) {
                    if (cnt < cap) d.nbr[list_index(s, cnt, tpa, R.begin, R.n, cap)] = (uint32_t)j | ((uint32_t)CODE_ZERO << IDX_BITS);
                    ++cnt;
                }
            }
            const int n = min(cnt, cap);
            if (d.refmode) sort_list_by_rank(d, s, n, tpa, R.begin, R.n);
            d.nn[s] = n;
            if (cnt > cap) {
                atomicOr(d.err, E_NLIST);
                atomicMax(d.max_needed, cnt);
            }
        }
        const int bm = block_max_int(cnt, smi);
        if (threadIdx.x == 0) atomicMax(&d.rep[tl.x].max_nn, bm);
    }
}

// ---------------------------------------------------------------------------
// The per-step cooperative kernel.  Block = TILE threads.
// Phase timing for MDGB_FLAG_TRACE: block 0 stamps the time after each grid
// barrier (all blocks have finished the phase by then).
struct PhaseClock {
    unsigned long long* tr;
    unsigned long long last;
    __device__ __forceinline__ explicit PhaseClock(unsigned long long* t)
        : tr((blockIdx.x == 0 && threadIdx.x == 0) ? t : nullptr), last(0) {
        if (tr) { last = global_ns(); atomicAdd(tr + TR_LAUNCHES, 1ull); }
    }
    __device__ __forceinline__ void mark(int slot) {
        if (!tr) return;
        const unsigned long long now = global_ns();
        atomicAdd(tr + slot, now - last);
        last = now;
    }
};

__device__ __forceinline__ void k_pre_rebuild(const Dev& d, const StepParams& sp, PhaseClock& clk);

// Nose-Hoover steps: the first kick alone, then Thermostat::update per type
// (integrator.rs:35-39): each type's temperature before its scaling adds
// psi_dot * dt/2 (thermostat.rs:59-65); the scaling itself uses the lambda
// computed before the kick, in the drift phase.  Returns true when the launch
// must stop.
__device__ __forceinline__ bool nose_hoover_kick(const Dev& d, const StepParams& sp) {
    if (d.mixed) phase_kick<true>(d, sp); else phase_kick<false>(d, sp);
    // (in tree order a thread sums the atoms it kicked: no barrier in between)
    if (d.refmode && grid_barrier(d)) return true;
    for (int t = 0; t <= d.last_type; ++t)
        if (nh_psi_of_type(d, sp, t)) return true;
    return false;
}

// The coupling factors of a step, before its kick (integrator.rs:20-29), each
// phase closed by a grid barrier.  Returns true when the launch must stop.
// LARGE: the system may have FX_MIN_ATOMS atoms.
template <bool LARGE>
__device__ __forceinline__ bool coupling_phases(const Dev& d, const StepParams& sp) {
    const int sel = d.last_type;
    // Nose-Hoover with several types: calculate_lambda runs once per type,
    // each adding its psi_dot * dt/2 (thermostat.rs:35-39, called per type
    // from integrator.rs:23-26); the last type's pass below adds its own
    // and sets lambda from the sum
    if (sp.thermo_nh)
        for (int t = 0; t < sel; ++t)
            if (nh_psi_of_type(d, sp, t)) return true;
    if (d.refmode) {
        if (phase_serial(d, sp, sel, true)) return true;
        if (grid_barrier(d)) return true;
    } else if (LARGE && d.mixed && d.ntot >= FX_MIN_ATOMS) {
        phase_partials_fx(d, sel);
        // (several replicas: a block each, finalized side by side)
        if (d.nrep == 1) {
            if (grid_barrier_then(d, [&] { phase_finalize_fx(d, sp, sel, 0, 1); })) return true;
        } else {
            if (grid_barrier(d)) return true;
            phase_finalize_fx(d, sp, sel, blockIdx.x, gridDim.x);
            if (grid_barrier(d)) return true;
        }
    } else if (d.mixed) {
        phase_partials1(d, sel);
        if (sums_then<7>(d, [&](int b, int n) { phase_finalize_single(d, sp, sel, b, n); })) return true;
    } else {
        phase_partials1(d, sel);
        if (sums_then<7>(d, [&](int b, int n) { phase_finalize1(d, sel, b, n); })) return true;
        phase_partials2(d, sel);
        if (sums_then<1>(d, [&](int b, int n) { phase_finalize2(d, sp, true, sel, b, n); })) return true;
    }
    return false;
}

// 5 blocks of 128 threads per SM (96 registers): at the default 64 registers
// the phases spilled (the rebuild's sort phases ran ~1.8x slower), at 80 less so
// (8M atoms, a coupled step: 2871 us, 2854 at 96, the same at 128; 512 replicas
// 1760, 1744 and, with the sort phases short of warps, 1793 at 128).
__global__ void __launch_bounds__(TILE, 5) k_pre(Dev d, StepParams sp) {
    if (chunk_failed(d)) return;
    barrier_setup(sp);
    tile_rep_reset();
    if (sp.hold_block == (int)blockIdx.x && threadIdx.x == 0) {
        // failure test: this block enters its first barrier after the others
        // have given up waiting (a bounded delay of twice the wait limit)
        const long long t0 = clock64();
        while (clock64() - t0 < 2 * g_bar_limit) __nanosleep(1000);
    }
    __syncthreads();
    PhaseClock clk(d.trace);
    if (sp.predrifted) {
        // the fused force pass of the previous step kicked and drifted (NVE
        // chunks).  Every block evaluates the rebuild test of every replica
        // (same inputs, same answer); when no replica needs one -- most
        // steps -- block 0 does the bookkeeping and all return without a
        // grid barrier.
        bool any = false;
        for (int r = threadIdx.x; r < d.nrep; r += blockDim.x) any |= rebuild_needed_at(d, sp, d.rep + r);
        if (!__syncthreads_or(any)) {
            if (blockIdx.x == 0) {
                for (int r = threadIdx.x; r < d.nrep; r += blockDim.x) {
                    RepDev* W = d.rep + r;
                    W->pending = W->baro_on ? W->myu : 1.0;
                    W->steps_since = W->steps_since + 1;
                    W->rebuild = 0;
                }
            }
            clk.mark(TR_DECIDE);
            return;
        }
        phase_decide(d, sp, blockIdx.x, gridDim.x);
        if (grid_barrier(d)) return;
        clk.mark(TR_DECIDE);
        if (*(volatile unsigned int*)(d.bar + 2) == 0u) return;
        if (clk.tr) atomicAdd(clk.tr + TR_REBUILD_LAUNCHES, 1ull);
        k_pre_rebuild(d, sp, clk);
        return;
    }
    if (sp.do_drift && sp.coupled) {
        if (coupling_phases<true>(d, sp)) return;
        clk.mark(TR_COUPLING);
    }
    const bool moved = sp.do_drift || !sp.force_rebuild;
    if (moved) {
        // (a forced rebuild without a step -- upload, refresh -- recomputes
        // every mirror in its gather: nothing here to do for it)
        const bool nh = sp.do_drift && sp.thermo_nh;
        if (nh && nose_hoover_kick(d, sp)) return;
        if (d.mixed) phase_drift<true>(d, sp, nh); else phase_drift<false>(d, sp, nh);
    }
    if (moved && d.nrep <= TILE) {
        // a thread per replica: the last block to arrive decides for all
        if (grid_barrier_then(d, [&] { phase_decide(d, sp, 0, 1); })) return;
        clk.mark(TR_DRIFT);
    } else {
        if (moved && grid_barrier(d)) return;
        clk.mark(TR_DRIFT);
        phase_decide(d, sp, blockIdx.x, gridDim.x);
        if (grid_barrier(d)) return;
    }
    clk.mark(TR_DECIDE);
    if (*(volatile unsigned int*)(d.bar + 2) == 0u) return;
    if (clk.tr) atomicAdd(clk.tr + TR_REBUILD_LAUNCHES, 1ull);
    k_pre_rebuild(d, sp, clk);
}

// The rebuild phases of k_pre (replicas with their rebuild flag set).
__device__ __forceinline__ void k_pre_rebuild(const Dev& d, const StepParams& sp, PhaseClock& clk) {
    if (blockIdx.x == 0) phase_work_list(d);
    phase_zero_cells(d, blockIdx.x, gridDim.x);
    if (grid_barrier(d)) return;
    clk.mark(TR_ZERO);
    phase_bin(d);
    if (grid_barrier(d)) return;
    clk.mark(TR_BIN);
    const int chunk = (d.ncells + gridDim.x - 1) / gridDim.x;
    phase_scan_a(d, chunk);
    if (grid_barrier(d)) return;
    clk.mark(TR_SCAN_A);
    if (blockIdx.x == 0) phase_scan_b(d);
    if (grid_barrier(d)) return;
    clk.mark(TR_SCAN_B);
    phase_scan_c(d, blockIdx.x * chunk, min((int)(blockIdx.x + 1) * chunk, d.ncells), __ldcg(d.bsum + blockIdx.x));
    if (grid_barrier(d)) return;
    clk.mark(TR_SCAN_C);
    phase_scatter(d, !sp.do_drift);
    if (grid_barrier(d)) return;
    clk.mark(TR_SCATTER);
    if (d.mixed) phase_sort_gather<true>(d, !sp.do_drift); else phase_sort_gather<false>(d, !sp.do_drift);
    if (grid_barrier(d)) return;
    clk.mark(TR_GATHER);
    if (clk.tr) clk.tr[TR_STAMP] = clk.last;
    // brute-mode replicas here; cell-mode replicas in k_build_list, which
    // follows this kernel and closes the rebuild
    phase_build_list(d);
}

// ---------------------------------------------------------------------------
// Whole chunks of small systems in one cooperative launch.
//
// A step of a few thousand atoms is five or six launches of a few microseconds
// each, most of it launch latency and kernels that fill a tenth of the chip
// with one thread per atom.  k_steps runs all n steps of a chunk: the phases
// of k_pre, the direct list build and the force pass with `lanes` threads per
// atom, separated by grid barriers; the reductions' last stages and the
// rebuild decision run in the last block to arrive at a barrier.
//
// The force sums are exact (mixed path), so sharing an atom's list out over
// more lanes changes no bit of them; the FP32 potential and virial and the
// FP64 path's sums are added entry by entry in list order, as one thread per
// atom adds them.
//
// Data written by this launch is read with plain or L2 loads, never with
// non-coherent ones (the barrier's fences order them).

// Dynamic shared memory of a block: during a rebuild the candidates of a cell
// (16-byte mirrors and 4-byte entries), else the lists of its first atoms.
constexpr int STEPS_WIN = 1800;
constexpr int STEPS_SMEM = STEPS_WIN * 20;

// What a block of k_steps keeps in shared memory besides Dev.
struct StepsShared {
    float4 tab[27];       // cell shifts and displacement constants of replica rep
    float tcs[8];
    int rep;
    // the block's first unit of atoms (the only one of most launches): its
    // tile and its lists, kept from one step to the next until a rebuild
    int4 tile;
    int unit, listed;
    int n[TILE];          // list lengths
    // force sums on their way from the lanes to one thread per atom
    long long f[3][TILE];
    float pe[TILE], vr[TILE];
    int skip[TILE];       // no atom, or left to band_atom
};

// The tile of unit u and its replica's constants; lists that fit are copied
// into `lists` ([atom][entry], row words apart) the first time a block sees
// its first unit after a rebuild.
__device__ __forceinline__ int4 steps_unit(const Dev& d, StepsShared& S, uint32_t* lists, int row, int u, int lanes) {
    const bool first = u == (int)blockIdx.x;
    int4 tl;
    if (first && S.unit == u) tl = S.tile;
    else tl = d.tiles[u / lanes];
    const RepDev* R = d.rep + tl.x;
    if (tl.x != S.rep || (first && !S.listed)) {   // block-uniform
        __syncthreads();
        shift_table(S.tab, R);
        if (threadIdx.x == 0) { drift_consts(*R, S.tcs); S.rep = tl.x; }
        if (first) {
            const int per = TILE / lanes, a = threadIdx.x / lanes, lane = threadIdx.x % lanes;
            const int at = (u % lanes) * per + a;
            const int s = tl.y + at;
            const int n = at < tl.z ? d.nn[s] : 0;
            if (lane == 0) S.n[a] = n;
            const uint32_t* list = d.nbr + list_index(at < tl.z ? s : tl.y, 0, 1, R->begin, R->n, d.cap);
            for (int k = lane; k < min(n, row); k += lanes) lists[a * row + k] = list[(size_t)k * R->n];
            if (threadIdx.x == 0) { S.tile = tl; S.unit = u; S.listed = 1; }
        }
        __syncthreads();
    }
    return tl;
}

// The force pass of a block's atoms (mixed path); lanes: a power of two <= 32.
template <bool NAIVE, bool NOE>
__device__ __noinline__ void steps_force_mixed(const Dev& d, const StepParams& sp, int lanes, StepsShared& S,
                                               uint32_t* lists, int row) {
    const unsigned FULL = 0xffffffffu;
    const int N = d.ntot;
    const int per = TILE / lanes, a = threadIdx.x / lanes, lane = threadIdx.x % lanes;
    const float fscale = d.fscale;
    const float fscale_t = NAIVE ? 1.0f : fscale * 1.1920928955078125e-07f;   // fscale / 2^23 (exact)
    const float rl = (float)(d.rlist * 1.01);
    const float split_limit = 2097152.0f / rl;       // as in k_force_mixed
    const float range_limit = 4294967296.0f / rl;
    for (int u = blockIdx.x; u < d.ntiles * lanes; u += gridDim.x) {
        const int4 tl = steps_unit(d, S, lists, row, u, lanes);
        const RepDev* R = d.rep + tl.x;
        const float4* tab = S.tab;
        const int at = (u % lanes) * per + a;
        const bool act = at < tl.z;
        const int s = tl.y + (act ? at : 0);
        // the epilogue's atom (one thread per atom, from the block's first on)
        // and its operands, on their way
        const int es = tl.y + (u % lanes) * per + (int)threadIdx.x;
        const bool eact = (int)threadIdx.x < per && (u % lanes) * per + (int)threadIdx.x < tl.z;
        if (eact) {
            prefetch_l1(d.vel + es);
            prefetch_l1(d.vel + N + es);
            prefetch_l1(d.vel + 2 * N + es);
            if (sp.fused) {
                prefetch_l1(d.pos + es);
                prefetch_l1(d.mir0 + es);
                prefetch_l1(d.cell + es);
            }
        }
        const bool kept = u == (int)blockIdx.x && d.cap <= row;   // the lists are in shared memory
        const int rn = R->n;
        const float4 xi = d.mir[s];
        const int ty = type_of(xi);
        const bool brute = R->mode == MODE_BRUTE;
        const int n = !act ? 0 : kept ? S.n[a] : d.nn[s];
        const uint32_t* list = kept ? lists + a * row : d.nbr + list_index(s, 0, 1, R->begin, rn, d.cap);
        const size_t step = kept ? 1 : (size_t)rn;
        MixedAcc<NAIVE, NOE> acc;
        acc.init();
        bool band = false;
        FixAcc bs[3];       // NOE: the sums as k_force_band rounds their terms
        for (int c = 0; c < 3; ++c) bs[c].init();
        float pe = 0.f, vr = 0.f, nx = 0.f, ny = 0.f, nz = 0.f;
        const int rounds = __reduce_max_sync(FULL, (n + lanes - 1) / lanes);
        uint32_t e = lane < n ? list[(size_t)lane * step] : 0u;
        for (int i = 0; i < rounds; ++i) {
            const int k = i * lanes + lane;
            const bool have = k < n;
            const float4 xj = d.mir[e & IDX_MASK];
            const uint32_t ec = e;
            if (k + lanes < n) e = list[(size_t)(k + lanes) * step];
            bool in = false;
            float fs = 0.f, uu = 0.f, r2 = 0.f, dz = 0.f;
            f2_t dxy = 0ull;
            if (have) {
                const PairDev& PD = d.pair[ty * MAX_TYPES + type_of(xj)];
                const PairF P = pairf(PD);
                if (!brute) {
                    const float4 sh = tab[ec >> IDX_BITS];
                    dxy = add2(sub2(f2(xj.x, xj.y), f2(xi.x, xi.y)), f2(sh.x, sh.y));
                    dz = __fadd_rn(__fsub_rn(xj.z, xi.z), sh.z);
                    const float dx = f2_lo(dxy), dy = f2_hi(dxy);
                    r2 = fmaf(dz, dz, fmaf(dy, dy, __fmul_rn(dx, dx)));
                    in = r2 < P.rc2_lo;
                    if (!in && r2 <= P.rc2_hi) {
                        band = true;
                        float bx, by;
                        if (NOE && !NAIVE && exact_pair(d, R, s, (int)(ec & IDX_MASK), PD, bx, by, dz)) {
                            in = true;
                            dxy = f2(bx, by);
                            r2 = fmaf(dz, dz, fmaf(by, by, __fmul_rn(bx, bx)));
                        }
                    }
                } else {
                    float dx, dy;
                    in = exact_pair(d, R, s, (int)(ec & IDX_MASK), PD, dx, dy, dz);
                    if (in) {
                        dxy = f2(dx, dy);
                        r2 = fmaf(dz, dz, fmaf(dy, dy, __fmul_rn(dx, dx)));
                    }
                }
                if (in) {
                    lj_f32(P, r2, fs, uu);
                    if (!NAIVE) acc.add(dxy, dz, r2, fs, uu, fscale_t);
                    if (NOE && !NAIVE) {
                        // (there dx g is rounded before it is split; here
                        // the paired instructions fuse the two)
                        const float g = __fmul_rn(fs, fscale_t), dd[3] = {f2_lo(dxy), f2_hi(dxy), dz};
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            const float tt = __fmul_rn(dd[c], g);
                            const float h = __fadd_rn(tt, FIX_MAGIC);
                            bs[c].hi += __float_as_uint(h) - FIX_MAGIC_BITS;
                            bs[c].lo += __float_as_uint(fmaf(__fsub_rn(tt, __fsub_rn(h, FIX_MAGIC)), 8388608.0f,
                                                             FIX_MAGIC)) - FIX_MAGIC_BITS;
                        }
                    }
                }
            }
            if (!NOE || NAIVE) {
                // the sums whose order matters: entry by entry over the lanes
                for (int q = 0; q < lanes; ++q) {
                    const bool qi = __shfl_sync(FULL, in, q, lanes);
                    const float qf = __shfl_sync(FULL, fs, q, lanes);
                    if (NAIVE) {
                        const float qx = __shfl_sync(FULL, f2_lo(dxy), q, lanes), qy = __shfl_sync(FULL, f2_hi(dxy), q, lanes),
                                    qz = __shfl_sync(FULL, dz, q, lanes);
                        if (qi) { nx = fmaf(qx, qf, nx); ny = fmaf(qy, qf, ny); nz = fmaf(qz, qf, nz); }
                    }
                    if (!NOE) {
                        const float qu = __shfl_sync(FULL, uu, q, lanes), qr = __shfl_sync(FULL, r2, q, lanes);
                        if (qi) { pe = __fadd_rn(pe, qu); vr = fmaf(qf, qr, vr); }
                    }
                }
            }
        }
        long long sx = acc.ax.total(), sy = acc.ay.total(), sz = acc.az.total();
        float gmax = acc.gmax;
        for (int off = lanes / 2; off > 0; off >>= 1) {
            gmax = fmaxf(gmax, __shfl_xor_sync(FULL, gmax, off));
            band |= __shfl_xor_sync(FULL, (int)band, off) != 0;
        }
        constexpr bool IN_LANE = NOE && !NAIVE;   // band pairs were decided in the loop
        if (IN_LANE && band) { sx = bs[0].total(); sy = bs[1].total(); sz = bs[2].total(); }
        if (!NAIVE && act && (IN_LANE || !band) && (gmax > split_limit || n > FIX_FOLD)) {
            // a term may exceed the exact range of the split, or the list is
            // as long as k_force_mixed converts: exact conversions
            if (gmax > range_limit) atomicOr(d.err, E_FIXED);
            sx = sy = sz = 0;
            for (int k = lane; k < n; k += lanes) {
                const uint32_t ek = list[(size_t)k * step];
                const int j = (int)(ek & IDX_MASK);
                const float4 xj = d.mir[j];
                const float4 sh = tab[ek >> IDX_BITS];
                float dx = __fadd_rn(__fsub_rn(xj.x, xi.x), sh.x), dy = __fadd_rn(__fsub_rn(xj.y, xi.y), sh.y),
                      dz = __fadd_rn(__fsub_rn(xj.z, xi.z), sh.z);
                const PairDev& PD = d.pair[ty * MAX_TYPES + type_of(xj)];
                const PairF P = pairf(PD);
                if (brute) {
                    if (!exact_pair(d, R, s, j, PD, dx, dy, dz)) continue;
                } else {
                    const float q2 = fmaf(dz, dz, fmaf(dy, dy, __fmul_rn(dx, dx)));
                    if (q2 > P.rc2_hi) continue;
                    if (q2 >= P.rc2_lo && !exact_pair(d, R, s, j, PD, dx, dy, dz)) continue;
                }
                float fs, uu;
                lj_f32(P, fmaf(dz, dz, fmaf(dy, dy, __fmul_rn(dx, dx))), fs, uu);
                const float g = __fmul_rn(fs, fscale);
                sx += __float2ll_rn(__fmul_rn(dx, g));
                sy += __float2ll_rn(__fmul_rn(dy, g));
                sz += __float2ll_rn(__fmul_rn(dz, g));
            }
        }
        for (int off = lanes / 2; off > 0; off >>= 1) {
            sx += __shfl_xor_sync(FULL, sx, off);
            sy += __shfl_xor_sync(FULL, sy, off);
            sz += __shfl_xor_sync(FULL, sz, off);
        }
        // one thread per atom finishes: a warp of them costs the FP64 pipe no
        // more than a single lane would
        if (lane == 0) {
            S.skip[a] = !act || (band && !IN_LANE);
            if (NAIVE) {
                S.f[0][a] = __float_as_int(nx); S.f[1][a] = __float_as_int(ny); S.f[2][a] = __float_as_int(nz);
            } else {
                S.f[0][a] = sx; S.f[1][a] = sy; S.f[2][a] = sz;
            }
            if (!NOE) { S.pe[a] = pe; S.vr[a] = vr; }
        }
        __syncthreads();
        if ((int)threadIdx.x < ((per + 31) & ~31)) {   // whole warps
            float disp = 0.f;
            if (eact && !S.skip[threadIdx.x]) {
                double F[3];
                for (int c = 0; c < 3; ++c) {
                    const long long v = S.f[c][threadIdx.x];
                    F[c] = NAIVE ? flt_to_dbl(__int_as_float((int)v)) : fixed_to_double(v, d.fscale_log2);
                }
                if (!NOE) {
                    d.frc[es] = F[0]; d.frc[N + es] = F[1]; d.frc[2 * N + es] = F[2];
                    d.epot[es] = flt_to_dbl(S.pe[threadIdx.x]); d.evir[es] = flt_to_dbl(S.vr[threadIdx.x]);
                }
                disp = kick_and_drift<true>(d, sp, R, S.tcs, es, type_of(d.mir[es]), F[0], F[1], F[2]);
            }
            if (sp.fused) note_displacement(d, tl.x, disp);
        }
        // atoms with a pair in the band, the whole warp for each (as k_force_band:
        // the order of its potential and virial sums)
        unsigned left = IN_LANE ? 0u : __ballot_sync(FULL, act && band && lane == 0);
        while (left) {
            const int src = __ffs(left) - 1;
            left &= left - 1u;
            band_atom<NAIVE, true>(d, sp, __shfl_sync(FULL, s, src), tl.x, true);
            __syncwarp();
        }
        __syncthreads();
    }
}

// The same for the FP64 path (lanes of at least eight): each lane the terms of
// its entry, added in list order.
__device__ __noinline__ void steps_force_fp64(const Dev& d, const StepParams& sp, int lanes, StepsShared& S,
                                              uint32_t* lists, int row) {
    const unsigned FULL = 0xffffffffu;
    const int N = d.ntot;
    const int per = TILE / lanes, a = threadIdx.x / lanes, lane = threadIdx.x % lanes;
    for (int u = blockIdx.x; u < d.ntiles * lanes; u += gridDim.x) {
        const int4 tl = steps_unit(d, S, lists, row, u, lanes);
        const RepDev* R = d.rep + tl.x;
        const float4* tab = S.tab;
        const int at = (u % lanes) * per + a;
        const bool act = at < tl.z;
        const int s = tl.y + (act ? at : 0);
        const bool kept = u == (int)blockIdx.x && d.cap <= row;
        const double box[3] = {R->box[0], R->box[1], R->box[2]};
        const float Lf[3] = {(float)box[0], (float)box[1], (float)box[2]};
        const bool brute = R->mode == MODE_BRUTE;
        const double4_32a pi = d.pos[s];
        const float4 mi = d.mir[s];
        const int ty = type_of(pi);
        const int n = !act ? 0 : kept ? S.n[a] : d.nn[s];
        const uint32_t* list = kept ? lists + a * row : d.nbr + list_index(s, 0, 1, R->begin, R->n, d.cap);
        const size_t step = kept ? 1 : (size_t)R->n;
        double sum = 0.0;
        const int rounds = __reduce_max_sync(FULL, (n + lanes - 1) / lanes);
        for (int i = 0; i < rounds; ++i) {
            const int k = i * lanes + lane;
            PairTerms o{0.0, 0.0, 0.0, 0.0, 0.0};
            bool in = false;
            if (k < n) {
                const uint32_t e = list[(size_t)k * step];
                const int j = (int)(e & IDX_MASK);
                const float4 mj = d.mir[j];
                const PairDev& P = d.pair[ty * MAX_TYPES + type_of(mj)];
                const float4 sh = tab[e >> IDX_BITS];
                float ex = mj.x - mi.x + sh.x, ey = mj.y - mi.y + sh.y, ez = mj.z - mi.z + sh.z;
                if (brute) {
                    if (ex < -0.5f * Lf[0]) ex += Lf[0]; else if (ex > 0.5f * Lf[0]) ex -= Lf[0];
                    if (ey < -0.5f * Lf[1]) ey += Lf[1]; else if (ey > 0.5f * Lf[1]) ey -= Lf[1];
                    if (ez < -0.5f * Lf[2]) ez += Lf[2]; else if (ez > 0.5f * Lf[2]) ez -= Lf[2];
                }
                if (!(ex * ex + ey * ey + ez * ez > P.rc2f_hi * 1.0001f)) {
                    const double4_32a pj = d.pos[j];
                    const double rx = min_image_ref(__dsub_rn(pj.x, pi.x), box[0]);
                    const double ry = min_image_ref(__dsub_rn(pj.y, pi.y), box[1]);
                    const double rz = min_image_ref(__dsub_rn(pj.z, pi.z), box[2]);
                    const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(rx, rx), __dmul_rn(ry, ry)), __dmul_rn(rz, rz));
                    in = d.refmode ? ref_terms<false>(rx, ry, rz, r2, P, o) : r2_terms<false>(rx, ry, rz, r2, P, o);
                }
            }
            // the sums whose order matters, entry by entry over the lanes; lane
            // c of an atom adds component c (an FP64 add costs the warp 64
            // cycles however many lanes take part)
            unsigned any = __ballot_sync(FULL, in);
            for (int off = 16; off >= lanes; off >>= 1) any |= any >> off;   // entries some atom of the warp has
            for (int q = 0; q < lanes; ++q) {
                if (!(any >> q & 1u)) continue;
                const bool qi = __shfl_sync(FULL, in, q, lanes);
                const double gx = __shfl_sync(FULL, o.gx, q, lanes), gy = __shfl_sync(FULL, o.gy, q, lanes),
                             gz = __shfl_sync(FULL, o.gz, q, lanes), uu = __shfl_sync(FULL, o.u, q, lanes),
                             tt = __shfl_sync(FULL, o.t, q, lanes);
                if (qi) sum = __dadd_rn(sum, lane == 0 ? gx : lane == 1 ? gy : lane == 2 ? gz : lane == 3 ? uu : tt);
            }
        }
        const double fx = __shfl_sync(FULL, sum, 0, lanes), fy = __shfl_sync(FULL, sum, 1, lanes),
                     fz = __shfl_sync(FULL, sum, 2, lanes), pe = __shfl_sync(FULL, sum, 3, lanes),
                     vr = __shfl_sync(FULL, sum, 4, lanes);
        float disp = 0.f;
        if (act && lane == 0) {
            d.frc[s] = fx; d.frc[N + s] = fy; d.frc[2 * N + s] = fz;
            d.epot[s] = pe; d.evir[s] = vr;
            disp = kick_and_drift<false>(d, sp, R, S.tcs, s, ty, fx, fy, fz);
        }
        if (sp.fused) note_displacement(d, tl.x, disp);
    }
}

// Cells up to which one block clears and scans them (a few round trips to L2 for
// 128 cells); more, in ensembles of many replicas above all, take the whole grid
// and three barriers more.  us for 20 NVE steps, one block / grid: 30 replicas of
// 27 atoms (about 900 cells) 1576 / 1652, 64 of 64 atoms (2,240) 2055 / 2042, 128
// (4,480) 2696 / 2450, 300 (10,500) 4406 / 3400.
constexpr int STEPS_FEW_CELLS = 2048;

// The rebuild decision of every replica (one block): decide_replica without
// reading whole records where none is needed.  A rebuild's work list is made
// and its cells, where they are few, are cleared here as well.
__device__ __noinline__ void steps_decide(const Dev& d, const StepParams& sp) {
    bool any = false;
    for (int r = threadIdx.x; r < d.nrep; r += blockDim.x) {
        if (rebuild_needed_at(d, sp, d.rep + r)) {
            any = true;
            decide_replica(d, sp, r);
        } else {
            RepDev* W = d.rep + r;
            W->pending = __ldcg(&W->baro_on) ? __ldcg(&W->myu) : 1.0;
            W->steps_since = __ldcg(&W->steps_since) + 1;
            W->rebuild = 0;
        }
    }
    if (__syncthreads_or(any)) {
        phase_work_list(d);
        if (d.ncells <= STEPS_FEW_CELLS) phase_zero_cells(d, 0, 1);
    }
}

// Lists of the rebuilding cell-mode replicas, one block per cell: the shifted
// mirrors of the 27 neighbour cells in shared memory, then a warp per own atom
// tests 32 of them at a time and appends the hits -- the tests, entries and
// order of list_direct.  (There a warp takes a whole cell; with the few cells
// of a small system that left most of the chip idle and took 49 us for 2,016
// atoms.)

__device__ __noinline__ void steps_lists(const Dev& d, uint32_t* smem) {
    __shared__ int nb_start[28], nb_off[28];
    const unsigned FULL = 0xffffffffu;
    float4* cx = reinterpret_cast<float4*>(smem);
    uint32_t* ce = smem + 4 * STEPS_WIN;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int m = d.rb[0], nwork = rb_cell_off(d)[m];
    for (int wi = blockIdx.x; wi < nwork; wi += gridDim.x) {
        const int i = rb_locate(rb_cell_off(d), m, wi);
        const int r = rb_rep(d)[i];
        const RepDev* W = d.rep + r;
        if (W->mode != MODE_CELLS) continue;
        const int c = W->cell_base + wi - rb_cell_off(d)[i];
        const float rl = (float)(W->rlist * (1.0 + 1e-5));
        const int nc[3] = {W->nc[0], W->nc[1], W->nc[2]};
        const long long rbeg = W->begin;
        const int rn = W->n;
        const float cs[3] = {dbl_to_flt_rn(W->cs[0]), dbl_to_flt_rn(W->cs[1]), dbl_to_flt_rn(W->cs[2])};
        const int ib = d.cell_start[c], in = d.cell_count[c];
        if (ib < rbeg || ib + in > rbeg + rn) {
            if (threadIdx.x == 0) atomicOr(d.err, E_CELLS);
            continue;
        }
        __syncthreads();
        if (w == 0) {
            int ox, oy, oz, start = 0, cnt = 0;
            decode_cell(c - W->cell_base, nc, ox, oy, oz);
            if (lane < 27) {
                int x = ox + lane % 3 - 1, y = oy + (lane / 3) % 3 - 1, z = oz + lane / 9 - 1;
                x = x < 0 ? x + nc[0] : (x >= nc[0] ? x - nc[0] : x);
                y = y < 0 ? y + nc[1] : (y >= nc[1] ? y - nc[1] : y);
                z = z < 0 ? z + nc[2] : (z >= nc[2] ? z - nc[2] : z);
                const int cj = W->cell_base + (x * nc[1] + y) * nc[2] + z;
                start = d.cell_start[cj];
                cnt = d.cell_count[cj];
                if (start < rbeg || start + cnt > rbeg + rn) { atomicOr(d.err, E_CELLS); cnt = 0; }
            }
            int incl = cnt;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int y = __shfl_up_sync(FULL, incl, off);
                if (lane >= off) incl += y;
            }
            if (lane < 28) { nb_start[lane] = start; nb_off[lane] = incl - cnt; }
        }
        __syncthreads();
        const int total = nb_off[27];
        // candidate p of the stream: its entry word and shifted mirror
        auto candidate = [&](int p, uint32_t& e, float4& x) {
            int lo = 0, hi = 26;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (nb_off[mid] <= p) lo = mid; else hi = mid - 1;
            }
            const int j = nb_start[lo] + p - nb_off[lo];
            e = (uint32_t)j | ((uint32_t)lo << IDX_BITS);
            x = d.mir[j];
            x.x = __fadd_rn(x.x, __fmul_rn((float)(lo % 3 - 1), cs[0]));
            x.y = __fadd_rn(x.y, __fmul_rn((float)((lo / 3) % 3 - 1), cs[1]));
            x.z = __fadd_rn(x.z, __fmul_rn((float)(lo / 9 - 1), cs[2]));
        };
        // atom s against the n candidates held, self its own place among them; cnt:
        // its entries so far
        auto scan = [&](int s, int self, int n, int cnt) {
            const float4 xi = d.mir[s];
            const int ti = type_of(xi);
            uint32_t* list = d.nbr + list_index(s, 0, 1, rbeg, rn, d.cap);
            for (int q = 0; q < n; q += 32) {
                const int p = q + lane;
                bool hit = false;
                uint32_t e = 0u;
                if (p < n) {
                    e = ce[p];
                    const float4 x = cx[p];
                    const float ex = __fsub_rn(x.x, xi.x), ey = __fsub_rn(x.y, xi.y), ez = __fsub_rn(x.z, xi.z);
                    hit = fmaf(ez, ez, fmaf(ey, ey, fmaf(ex, ex, -__fmul_rn(rl, rl)))) < 0.f && type_of(x) >= ti &&
                          p != self;
                }
                const unsigned got = __ballot_sync(FULL, hit);
                const int k = cnt + __popc(got & ((1u << lane) - 1u));
                if (hit && k < d.cap) list[(size_t)k * rn] = e;
                cnt += __popc(got);
            }
            return cnt;
        };
        int cmax = 0;
        auto finish = [&](int s, int cnt) {
            const int nfill = min(cnt, d.cap);
            if (d.refmode) sort_lists_by_rank(d, s, lane == 0 ? nfill : 0, rbeg, rn);
            if (lane == 0) {
                d.nn[s] = nfill;
                if (cnt > d.cap) {
                    atomicOr(d.err, E_NLIST);
                    atomicMax(d.max_needed, cnt);
                }
            }
            cmax = max(cmax, cnt);
        };
        if (total <= STEPS_WIN) {
            for (int p = threadIdx.x; p < total; p += blockDim.x) candidate(p, ce[p], cx[p]);
            __syncthreads();
            for (int a = w; a < in; a += TILE / 32) finish(ib + a, scan(ib + a, nb_off[CODE_ZERO] + a, total, 0));
        } else {
            // crowded cells: a window of the stream at a time, an atom's count so far
            // in nn
            for (int w0 = 0; w0 < total; w0 += STEPS_WIN) {
                const int wn = min(STEPS_WIN, total - w0);
                __syncthreads();   // the last window's readers are done
                for (int p = threadIdx.x; p < wn; p += blockDim.x) candidate(w0 + p, ce[p], cx[p]);
                __syncthreads();
                for (int a = w; a < in; a += TILE / 32) {
                    const int s = ib + a;
                    const int cnt = scan(s, nb_off[CODE_ZERO] + a - w0, wn, w0 ? d.nn[s] : 0);
                    __syncwarp();   // every lane has read the count
                    if (w0 + wn == total) finish(s, cnt);
                    else if (lane == 0) d.nn[s] = cnt;
                }
            }
        }
        if (lane == 0 && cmax > 0) atomicMax(&d.rep[r].max_nn, cmax);
    }
}

// Clearing, binning and scanning of many cells by the whole grid, as k_pre does.
__device__ __noinline__ bool steps_sort_many(const Dev& d) {
    const int chunk = (d.ncells + gridDim.x - 1) / gridDim.x;
    phase_zero_cells(d, blockIdx.x, gridDim.x);
    if (grid_barrier(d)) return true;
    phase_bin(d);
    if (grid_barrier(d)) return true;
    phase_scan_a(d, chunk);
    if (grid_barrier_then(d, [&] { phase_scan_b(d); })) return true;
    phase_scan_c(d, blockIdx.x * chunk, min((int)(blockIdx.x + 1) * chunk, d.ncells), __ldcg(d.bsum + blockIdx.x));
    return grid_barrier(d);
}

// The rebuild of k_pre with the scan of few cells in the last block to arrive,
// then the lists and the end of the rebuild.
__device__ __noinline__ bool steps_rebuild(const Dev& d, uint32_t* st_smem) {
    if (d.ncells > STEPS_FEW_CELLS) {
        if (steps_sort_many(d)) return true;
    } else {
        phase_bin(d);
        if (grid_barrier_then(d, [&] { phase_scan_c(d, 0, d.ncells, 0); })) return true;
    }
    phase_scatter(d, false);
    if (grid_barrier(d)) return true;
    if (d.mixed) phase_sort_gather<true>(d, false); else phase_sort_gather<false>(d, false);
    if (grid_barrier(d)) return true;
    phase_build_list(d);
    steps_lists(d, st_smem);
    return grid_barrier_then(d, [&] { close_rebuild(d, d.direct_list != 0); });
}

// Coupling and motion of a step that the previous force pass did not drift.
__device__ __noinline__ bool steps_motion(const Dev& d, const StepParams& sp) {
    if (sp.coupled && coupling_phases<false>(d, sp)) return true;
    if (sp.thermo_nh && nose_hoover_kick(d, sp)) return true;
    if (d.mixed) phase_drift<true>(d, sp, sp.thermo_nh != 0); else phase_drift<false>(d, sp, sp.thermo_nh != 0);
    return false;
}

// One step's motion up to its positions, its list and its forces; the last
// barrier of a step is the next one's rebuild decision.
__global__ void __launch_bounds__(TILE, 4) k_steps(Dev d_in, StepParams sp_in, int n, int naive, int lanes) {
    if (chunk_failed(d_in)) return;
    extern __shared__ __align__(16) uint32_t st_smem[];
    __shared__ __align__(16) unsigned char dev_mem[sizeof(Dev)];
    __shared__ StepsShared S;
    Dev& d = *reinterpret_cast<Dev*>(dev_mem);   // the buffer pair is swapped after every fused step
    if (threadIdx.x == 0) { d = d_in; S.rep = -1; S.unit = -1; S.listed = 0; }
    StepParams sp = sp_in;
    barrier_setup(sp, true);
    tile_rep_reset();
    if (sp.hold_block == (int)blockIdx.x && threadIdx.x == 0) {   // failure test, as in k_pre
        const long long t0 = clock64();
        while (clock64() - t0 < 2 * g_bar_limit) __nanosleep(1000);
    }
    __syncthreads();
    const int row = STEPS_SMEM / 4 / (TILE / lanes);   // list words shared memory holds per atom
    const bool fusable = !sp.coupled && !sp.thermo_nh;
    const int nf = fusable ? ((n - 1) & ~1) : 0;
    for (int i = 0; i < n; ++i) {
        const bool predrifted = i >= 1 && i <= nf;
        if (!predrifted && steps_motion(d, sp)) return;
        if (grid_barrier_then(d, [&] { steps_decide(d, sp); })) return;
        const bool rebuild = *(volatile unsigned int*)(d.bar + 2) != 0u;
        if (rebuild && steps_rebuild(d, st_smem)) return;
        // the force pass's per-replica constants stay in shared memory while
        // neither box nor cells change
        if (rebuild || sp.coupled) {
            __syncthreads();
            if (threadIdx.x == 0) {
                S.rep = -1;
                if (rebuild) S.listed = 0;
            }
            __syncthreads();
        }
        sp.fused = i < nf ? 1 : 0;
        if (!d.mixed) steps_force_fp64(d, sp, lanes, S, st_smem, row);
        else if (naive) steps_force_mixed<true, false>(d, sp, lanes, S, st_smem, row);
        else if (sp.fused) steps_force_mixed<false, true>(d, sp, lanes, S, st_smem, row);
        else steps_force_mixed<false, false>(d, sp, lanes, S, st_smem, row);
        __syncthreads();
        if (sp.fused && threadIdx.x == 0) {
            double4_32a* const p = d.pos; d.pos = d.pos_next; d.pos_next = p;
            float4* const m = d.mir; d.mir = d.mir_next; d.mir_next = m;
        }
        sp.fused = 0;
        // an unfused step's forces are read by the next step's kick or sums
        if (i >= nf && i + 1 < n && grid_barrier(d)) return;
    }
}

// Host side of k_steps: resident blocks per SM.

cudaError_t steps_init(int* blocks_per_sm) {
    // a property of the device: asked once for each (not on every new engine)
    static std::atomic<int> known[64];
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    const bool slot = dev >= 0 && dev < 64;
    if (slot && known[dev].load() > 0) {
        *blocks_per_sm = known[dev].load();
        return cudaSuccess;
    }
    err = cudaFuncSetAttribute(k_steps, cudaFuncAttributeMaxDynamicSharedMemorySize, STEPS_SMEM);
    if (err == cudaSuccess) err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k_steps, TILE, STEPS_SMEM);
    if (err == cudaSuccess && slot) known[dev].store(*blocks_per_sm);
    return err;
}

cudaError_t launch_steps(const Dev& d, const StepParams& sp, int n, bool naive, int max_blocks, cudaStream_t st) {
    // as many lanes per atom as the resident threads allow; the FP64 path adds
    // an entry at a time over a warp, so two atoms a warp at least, and its
    // sums need eight lanes
    int lanes = d.mixed ? 32 : 16;
    while (lanes > (d.mixed ? 1 : 8) && d.ntiles * lanes > max_blocks) lanes /= 2;
    const int folds = d.refmode ? 6 * d.nrep : 1;
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3(std::min(max_blocks, std::max(d.ntiles * lanes, folds)));
    lc.blockDim = dim3(TILE);
    lc.dynamicSmemBytes = STEPS_SMEM;
    lc.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    lc.attrs = at;
    lc.numAttrs = 1;
    return cudaLaunchKernelEx(&lc, k_steps, d, sp, n, naive ? 1 : 0, lanes);
}

// Macro parameters of type `sel` (solver/src/macro_parameters): results land
// in the replica records (vcm, mom, ke, pe, thermal, T, P, count).
// 6 blocks per SM (80 registers), on a grid of its own: at k_pre's five 1.6M atoms
// took 204 us instead of 192.
__global__ void __launch_bounds__(TILE, 6) k_macro(Dev d, StepParams sp, int sel) {
    barrier_setup(sp);
    tile_rep_reset();
    if (d.refmode) {
        phase_serial(d, sp, sel, false);
        return;
    }
    phase_partials1(d, sel);
    if (sums_then<7>(d, [&](int b, int n) { phase_finalize1(d, sel, b, n); })) return;
    phase_partials2(d, sel);
    sums_then<1>(d, [&](int b, int n) { phase_finalize2(d, sp, false, sel, b, n); });
}

// End of an mdgb_step call: finish the barostat update of the last step: x *=
// mu, then (the last block, when every block has read the factor) the box,
// once per type.
__global__ void __launch_bounds__(TILE) k_apply_pending(Dev d) {
    __shared__ int last;
    const int4 tl = d.tiles[blockIdx.x];
    const double f = d.rep[tl.x].pending;
    if (f != 1.0) {
        const int s = tl.y + threadIdx.x;
        if ((int)threadIdx.x < tl.z) {
            double4_32a p = d.pos[s];
            p.x = __dmul_rn(p.x, f); p.y = __dmul_rn(p.y, f); p.z = __dmul_rn(p.z, f);
            d.pos[s] = p;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(d.bar + 6, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    for (int r = threadIdx.x; r < d.nrep; r += blockDim.x) {
        RepDev* W = d.rep + r;
        const double g = W->pending;
        if (g == 1.0) continue;
        for (int k = 0; k < d.ntypes; ++k)
            for (int a = 0; a < 3; ++a) W->box[a] *= g;
        for (int a = 0; a < 3; ++a) W->cs[a] = W->box[a] / (double)W->nc[a];
        W->pending = 1.0;
    }
    if (threadIdx.x == 0) d.bar[6] = 0u;
}

// The arrays a chunk may have to be run again from, copied aside (each with the
// widest words its addresses and length allow), and the error words and the
// barrier cleared (bar[5] on are kept).
template <class T>
__device__ __forceinline__ void copy_words(void* dst, const void* src, size_t bytes) {
    const size_t n = bytes / sizeof(T), step = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step)
        static_cast<T*>(dst)[i] = static_cast<const T*>(src)[i];
}
__global__ void __launch_bounds__(256) k_snapshot(Dev d, SnapArrays a) {
#pragma unroll 1
    for (int k = 0; k < 11; ++k) {
        const uintptr_t bits = (uintptr_t)a.dst[k] | (uintptr_t)a.src[k] | (uintptr_t)a.bytes[k];
        if (!(bits & 15)) copy_words<uint4>(a.dst[k], a.src[k], a.bytes[k]);
        else if (!(bits & 7)) copy_words<uint2>(a.dst[k], a.src[k], a.bytes[k]);
        else copy_words<uint32_t>(a.dst[k], a.src[k], a.bytes[k]);
    }
    if (blockIdx.x == 0 && threadIdx.x < 8) {
        if (threadIdx.x < 2) d.err[threadIdx.x] = 0;
        if (threadIdx.x < 5) d.bar[threadIdx.x] = 0u;
    }
}

// A single system's coupling settings.
__global__ void k_set_coupling(Dev d, RepCoupling c) {
    if (threadIdx.x != 0) return;
    RepDev* W = d.rep;
    W->thermo_on = c.thermo_on;
    if (c.thermo_on) {
        W->thermo_kind = c.thermo_kind;
        W->th_tau = c.th_tau; W->th_T0 = c.th_T0;
        W->lambda = c.lambda; W->psi = c.psi;
    }
    W->baro_on = c.baro_on;
    if (c.baro_on) {
        W->ba_beta = c.ba_beta; W->ba_tau = c.ba_tau; W->ba_P0 = c.ba_P0;
        W->myu = c.myu;
    }
}

// Device -> caller order (for download): out[orig[s]] = value[s]; a null
// output is skipped.
__global__ void k_gather_out(Dev d, double* out_pos, double* out_vel, double* out_frc,
                             double* out_pot, double* out_tmp) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const int N = d.ntot;
    if (s >= N) return;
    const int o = d.orig[s];
    if (o < 0 || o >= N) { atomicOr(d.err, E_BOUNDS); return; }
    if (out_pos) {
        const double4_32a p = d.pos[s];
        out_pos[3 * (size_t)o] = p.x; out_pos[3 * (size_t)o + 1] = p.y; out_pos[3 * (size_t)o + 2] = p.z;
    }
    for (int k = 0; k < 3; ++k) {
        if (out_vel) out_vel[3 * (size_t)o + k] = d.vel[(size_t)k * N + s];
        if (out_frc) out_frc[3 * (size_t)o + k] = d.frc[(size_t)k * N + s];
    }
    if (out_pot) out_pot[o] = d.epot[s];
    if (out_tmp) out_tmp[o] = d.evir[s];
}

// Atoms of each type in every tile (one block each); bad: a type id >= ntypes.
__global__ void __launch_bounds__(TILE) k_type_count(const int4* tiles, const uint16_t* type, int ntypes, int* count,
                                                     int* bad) {
    __shared__ int c[MAX_TYPES];
    const int4 tl = tiles[blockIdx.x];
    const bool act = (int)threadIdx.x < tl.z;
    const int ty = act ? (int)type[tl.y + threadIdx.x] : -1;
    if (ty >= ntypes) atomicOr(bad, 1);
    if (threadIdx.x < MAX_TYPES) c[threadIdx.x] = 0;
    __syncthreads();
    for (int t = 0; t < ntypes; ++t) {
        const unsigned m = __ballot_sync(0xffffffffu, ty == t);
        if ((threadIdx.x & 31) == 0 && m) atomicAdd(c + t, __popc(m));
    }
    __syncthreads();
    if (threadIdx.x < MAX_TYPES) count[(size_t)blockIdx.x * MAX_TYPES + threadIdx.x] = c[threadIdx.x];
}

// The counts of a replica's tiles (reps: first tile, tiles), type by type,
// replaced by their exclusive prefix sums; total: the replica's counts.  One
// block per replica.
__global__ void __launch_bounds__(256) k_type_scan(const int2* reps, int ntypes, int* count, int* total) {
    __shared__ int wsum[8];
    const int2 R = reps[blockIdx.x];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int t = 0; t < ntypes; ++t) {
        int carry = 0;
        for (int b = 0; b < R.y; b += 256) {
            const int i = b + (int)threadIdx.x;
            int* p = count + (size_t)(R.x + i) * MAX_TYPES + t;
            const int v = i < R.y ? *p : 0;
            int incl = v;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, off);
                if (lane >= off) incl += y;
            }
            __syncthreads();
            if (lane == 31) wsum[w] = incl;
            __syncthreads();
            int before = carry, all = 0;
            for (int k = 0; k < 8; ++k) {
                if (k < w) before += wsum[k];
                all += wsum[k];
            }
            if (i < R.y) *p = before + incl - v;
            carry += all;
        }
        if (threadIdx.x == 0) total[blockIdx.x * MAX_TYPES + t] = carry;
    }
}

// Caller order -> device (upload), one block per tile: the device order starts
// as the caller's; the first rebuild sorts it by cell.  type_count: with
// several types, the atoms of each type in the replica's earlier tiles
// (k_type_scan), from which the atom's rank follows; null: one type, the rank
// is the index, and a type id >= ntypes is flagged (E_INPUT) and replaced by
// 0, so no later kernel indexes the pair table with it.
__global__ void __launch_bounds__(TILE) k_scatter_in(Dev d, const double* in_pos, const double* in_vel,
                                                     const uint16_t* in_type, const int* type_count, int ntypes) {
    __shared__ int wcount[TILE / 32][MAX_TYPES];
    const int4 tl = d.tiles[blockIdx.x];
    const bool act = (int)threadIdx.x < tl.z;
    const int s = tl.y + threadIdx.x;
    const int N = d.ntot;
    int ty = act ? (int)in_type[s] : -1;
    if (ty >= ntypes) { atomicOr(d.err, E_INPUT); ty = 0; }
    int rk = s;
    if (type_count) {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        int within = 0;
        for (int t = 0; t < ntypes; ++t) {
            const unsigned m = __ballot_sync(0xffffffffu, ty == t);
            if (lane == 0) wcount[w][t] = __popc(m);
            if (ty == t) within = __popc(m & ((1u << lane) - 1u));
        }
        __syncthreads();
        if (act) {
            for (int k = 0; k < w; ++k) within += wcount[k][ty];
            const RepDev* R = d.rep + tl.x;
            rk = (int)R->begin + R->type_off[ty] + type_count[(size_t)blockIdx.x * MAX_TYPES + ty] + within;
        }
    }
    if (!act) return;
    double4_32a p;
    p.x = in_pos[3 * (size_t)s]; p.y = in_pos[3 * (size_t)s + 1]; p.z = in_pos[3 * (size_t)s + 2];
    p.w = __longlong_as_double((long long)ty);
    d.pos[s] = p;
    for (int k = 0; k < 3; ++k) {
        d.vel[(size_t)k * N + s] = in_vel ? in_vel[3 * (size_t)s + k] : 0.0;
        d.frc[(size_t)k * N + s] = 0.0;
    }
    d.epot[s] = 0.0;
    d.evir[s] = 0.0;
    d.orig[s] = s;
    if (rk < 0 || rk >= N) { atomicOr(d.err, E_BOUNDS); rk = s; }
    d.rank[s] = rk;
    d.slot_of_rank[rk] = s;
    d.cell[s] = -1;
    d.nn[s] = 0;
    d.mir0[s] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// Caller order -> device order for force, potential, temp (mdgb_upload_forces).
__global__ void k_scatter_forces(Dev d, const double* in_frc, const double* in_pot, const double* in_tmp) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const int N = d.ntot;
    if (s >= N) return;
    const int o = d.orig[s];
    if (o < 0 || o >= N) { atomicOr(d.err, E_BOUNDS); return; }
    if (in_frc)
        for (int k = 0; k < 3; ++k) d.frc[(size_t)k * N + s] = in_frc[3 * (size_t)o + k];
    if (in_pot) d.epot[s] = in_pot[o];
    if (in_tmp) d.evir[s] = in_tmp[o];
}

// Interacting pairs from the neighbour list, decided with the reference's
// FP64 arithmetic (potential.rs:181-204), in caller indices.
__global__ void k_pairs(Dev d, long long capacity, int* out_i, int* out_j, unsigned long long* count) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const int N = d.ntot;
    if (s >= N) return;
    int r = 0;
    {
        // replica of s: tiles are contiguous per replica
        int lo = 0, hi = d.nrep - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (d.rep[mid].begin <= s) lo = mid; else hi = mid - 1;
        }
        r = lo;
    }
    const RepDev& R = d.rep[r];
    const double4_32a pi = d.pos[s];
    const int ti = type_of(pi);
    const int n = d.nn[s];
    for (int k = 0; k < n; ++k) {
        const uint32_t e = d.nbr[list_index(s, k, R.tpa, R.begin, R.n, d.cap)];
        const int j = (int)(e & IDX_MASK);
        if (j < 0 || j >= N) { atomicOr(d.err, E_BOUNDS); continue; }
        const double4_32a pj = d.pos[j];
        const PairDev& P = d.pair[ti * MAX_TYPES + type_of(pj)];
        double rx = pj.x - pi.x, ry = pj.y - pi.y, rz = pj.z - pi.z;
        if (rx < -(R.box[0] / 2.0)) rx += R.box[0]; else if (rx > R.box[0] / 2.0) rx -= R.box[0];
        if (ry < -(R.box[1] / 2.0)) ry += R.box[1]; else if (ry > R.box[1] / 2.0) ry -= R.box[1];
        if (rz < -(R.box[2] / 2.0)) rz += R.box[2]; else if (rz > R.box[2] / 2.0) rz -= R.box[2];
        const double ra = sqrt(rx * rx + ry * ry + rz * rz);
        if (ra > P.rc) continue;
        const unsigned long long slot = atomicAdd(count, 1ull);
        if ((long long)slot < capacity) {
            out_i[slot] = d.orig[s];
            out_j[slot] = d.orig[j];
        }
    }
}

}  // namespace mdgb
