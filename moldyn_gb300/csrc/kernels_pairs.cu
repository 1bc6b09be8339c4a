// kernels_pairs.cu -- the FP64 path's force pass over pair records: every pair
// computed once (update_force, solver/src/solver/potential.rs:158-216).
//
// GB300's FP64 pipe takes 64 cycles of a scheduler per warp instruction,
// however few lanes are active, so k_force_fp64 (a thread per atom, both sides
// of every pair, lanes idle where a candidate is outside r_cut) is bound by it.  Here a force pass is two kernels:
//
//   k_pair_terms  one thread per pair record: the pair's force, potential and
//                 virial terms once, from the side of its owner.  Candidates
//                 outside r_cut (FP32 prefilter) are dropped before the FP64
//                 work: a warp queues what passes and computes 32 at a time.
//   k_pair_sums   four lanes per atom: walk its list in list order and add
//                 the records (the partner's with the force negated), then the
//                 second half kick and, on NVE chunks, the next step's kick
//                 and drift.
//
// r_ji = -r_ij, |r|, U and F . r are the same bits from either side, so the
// per-atom sums are those of the one-sided loop, term by term and in the same
// order; with MDGB_FLAG_REFERENCE_ORDER they stay bit-identical to the
// reference.
//
// After every list build k_pair_rows gives each list entry its record -- the
// entry of the atom that comes first in device order, or of the only atom that
// lists the pair (several types) -- and k_pair_link finds the partner's entry
// by binary search in its (ascending) list.  A pair listed by the later atom
// only (within rounding of the list radius, far outside r_cut) has none.
//
// 256,000 atoms, one NVE pass in tree order: 3.66 ms with k_force_fp64 as the
// reference writes the terms, 1.47 with the terms used here; 0.39 + 0.21 ms
// here, and 0.41 ms more at a rebuild (every ninth step).  23,256
// atoms in reference order: 0.53 -> 0.14 ms.  k_pair_terms keeps the FP64 pipe
// busy over 80 % of the time; k_pair_sums waits for its record gathers.
// (Summing runs of tiles on a second stream beside the next run's terms was
// slower: 15.5 to 17.7 ms for 20 steps of 256,000 atoms against 14.9.)
#include <algorithm>

#include "force_mixed.cuh"

namespace mdgb {

// Atom i owns its entry for j: j lists the pair too and comes later, or does
// not list it (the reference's t1 <= t2 loop, potential.rs:171-172).
__device__ __forceinline__ bool pair_owned(const Dev& d, int i, int ti, int j) {
    return j > i || (!d.single_type && type_of(__ldg(d.mir + j)) > ti);
}

// One block per tile: records for the tile's owned entries, numbered by a
// warp's 32 atoms together -- list position by list position, so that stores
// here, and the loads of a warp that walks its atoms' lists in k_pair_sums,
// lie side by side.
__global__ void __launch_bounds__(TILE) k_pair_rows(Dev d) {
    if (*(volatile const unsigned int*)(d.bar + 2) == 0u) return;   // no rebuild this step
    if (chunk_failed(d)) return;
    __shared__ int wsum[TILE / 32];
    __shared__ int s_base;
    const unsigned FULL = 0xffffffffu;
    const int4 tl = d.tiles[blockIdx.x];
    const RepDev* R = d.rep + tl.x;
    if (!R->rebuild) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long rbeg = R->begin;
    const int rn = R->n;
    const int s = tl.y + threadIdx.x;
    const int n = (int)threadIdx.x < tl.z ? d.nn[s] : 0;
    const int nmax = __reduce_max_sync(FULL, n);
    const int ty = n ? type_of(d.mir[s]) : 0;
    const size_t li = list_index(s, 0, 1, rbeg, rn, d.cap);
    int own = 0;
    for (int k = 0; k < n; ++k) {
        const uint32_t e = d.nbr[li + (size_t)k * rn];
        own += pair_owned(d, s, ty, (int)(e & IDX_MASK)) ? 1 : 0;
    }
    own = __reduce_add_sync(FULL, own);
    if (lane == 0) wsum[w] = own;
    __syncthreads();
    if (threadIdx.x == 0) {
        int total = 0;
        for (int k = 0; k < TILE / 32; ++k) { const int t = wsum[k]; wsum[k] = total; total += t; }
        const int room = (int)pair_room(rn, d.cap, d.single_type);
        const int first = (int)pair_room((size_t)rbeg, d.cap, d.single_type);
        const int base = atomicAdd(d.pair_count + tl.x, total);
        s_base = first + base;
        if (base + total > room) {   // lists nearly full everywhere: a longer list makes room
            atomicOr(d.err, E_NLIST);
            atomicMax(d.max_needed, d.cap + 1);
            total = 0;
            s_base = -1;
        }
        d.pair_tile[blockIdx.x] = make_int2(max(s_base, 0), total);
    }
    __syncthreads();
    const bool fits = s_base >= 0;
    uint32_t rec = (uint32_t)(s_base + wsum[w]);
    for (int k = 0; k < nmax; ++k) {
        const uint32_t e = k < n ? d.nbr[li + (size_t)k * rn] : 0u;
        const bool mine = fits && k < n && pair_owned(d, s, ty, (int)(e & IDX_MASK));
        const unsigned got = __ballot_sync(FULL, mine);
        const uint32_t at = rec + __popc(got & ((1u << lane) - 1u));
        if (k < n) d.pair_of[li + (size_t)k * rn] = mine ? at : PAIR_NONE;
        if (mine) d.pair_ij[at] = make_uint2((uint32_t)s, e);
        rec += __popc(got);
    }
}

// One thread per record: the partner's list entry of the pair, by binary
// search -- by rank in the reference's order; else the lists ascend as 32-bit
// words (shift code, then index) and the partner sees the pair at the opposite
// code.  The last block closes the rebuild.
__global__ void __launch_bounds__(TILE) k_pair_link(Dev d) {
    if (*(volatile const unsigned int*)(d.bar + 2) == 0u) return;
    if (chunk_failed(d)) return;
    __shared__ int s_last;
    for (int t = blockIdx.x; t < d.ntiles; t += gridDim.x) {
        const int4 tl = d.tiles[t];
        const RepDev* R = d.rep + tl.x;
        if (!R->rebuild) continue;
        const long long rbeg = R->begin;
        const int rn = R->n;
        const int2 pt = d.pair_tile[t];
        for (int q = threadIdx.x; q < pt.y; q += blockDim.x) {
            const uint2 ij = d.pair_ij[pt.x + q];
            const int i = (int)ij.x, j = (int)(ij.y & IDX_MASK);
            if (!d.single_type && type_of(__ldg(d.mir + j)) > type_of(__ldg(d.mir + i))) continue;
            const size_t lj = list_index(j, 0, 1, rbeg, rn, d.cap);
            const uint32_t want = (uint32_t)i | ((uint32_t)(26 - (int)(ij.y >> IDX_BITS)) << IDX_BITS);
            const int ri = d.refmode ? d.rank[i] : 0;
            int lo = 0, hi = d.nn[j];
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                const uint32_t e = __ldg(d.nbr + lj + (size_t)mid * rn);
                if (d.refmode ? d.rank[e & IDX_MASK] < ri : e < want) lo = mid + 1; else hi = mid;
            }
            if (lo < d.nn[j] && (d.nbr[lj + (size_t)lo * rn] & IDX_MASK) == (uint32_t)i)
                d.pair_of[lj + (size_t)lo * rn] = (uint32_t)(pt.x + q) | PAIR_NEG;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(d.bar + 3, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (s_last) {
        __threadfence();
        close_rebuild(d, d.direct_list || *(volatile const unsigned int*)(d.bar + 4) != 0u);
    }
}

// ---------------------------------------------------------------------------
// Pair terms.

// `parts` blocks per tile, each a share of the tile's records; a warp walks
// its part 32 candidates at a time.
template <bool REF, bool FORCE>
__global__ void __launch_bounds__(TILE) k_pair_terms(Dev d, int parts) {
    if (chunk_failed(d)) return;
    __shared__ float4 tab[27];
    __shared__ uint32_t queue[TILE / 32][64];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int t = blockIdx.x / parts, part = blockIdx.x % parts;
    const int4 tl = d.tiles[t];
    const int2 pt = d.pair_tile[t];
    const RepDev* R = d.rep + tl.x;
    shift_table(tab, R);
    __syncthreads();
    const int per = ((pt.y + parts * TILE - 1) / (parts * TILE)) * 32;   // a warp's share, whole 32s
    const int begin = pt.x + (part * (TILE / 32) + w) * per;
    const int end = min(pt.x + pt.y, begin + per);
    const double box[3] = {R->box[0], R->box[1], R->box[2]};
    const float Lf[3] = {(float)box[0], (float)box[1], (float)box[2]};
    const bool brute = R->mode == MODE_BRUTE;
    uint32_t* qu = queue[w];
    int held = 0;
    auto compute = [&](int at) {
        const uint32_t rec = qu[at];
        const uint2 ij = d.pair_ij[rec];
        const int j = (int)(ij.y & IDX_MASK);
        const double4_32a pi = d.pos[ij.x], pj = d.pos[j];
        const PairDev& P = d.pair[type_of(pi) * MAX_TYPES + type_of(pj)];
        double rx = __dsub_rn(pj.x, pi.x), ry = __dsub_rn(pj.y, pi.y), rz = __dsub_rn(pj.z, pi.z);
        // potential.rs:181-200, by a vote: most warps hold no pair across the
        // boundary (as predicated adds the three would be issued for every warp)
        const bool across = beyond_half(rx, box[0]) || beyond_half(ry, box[1]) || beyond_half(rz, box[2]);
        if (__any_sync(__activemask(), across)) {
            rx = min_image_ref(rx, box[0]);
            ry = min_image_ref(ry, box[1]);
            rz = min_image_ref(rz, box[2]);
        }
        const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(rx, rx), __dmul_rn(ry, ry)), __dmul_rn(rz, rz));
        PairTerms o;
        o.u = 0.0;
        const bool in = REF ? ref_terms<FORCE>(rx, ry, rz, r2, P, o) : r2_terms<FORCE>(rx, ry, rz, r2, P, o);
        if (in) {
            double2* dst = reinterpret_cast<double2*>(d.pair_rec + rec);
            dst[0] = make_double2(o.gx, o.gy);
            dst[1] = make_double2(o.gz, o.u);
            if (!FORCE) d.pair_vir[rec] = o.t;
        }
        d.pair_in[rec] = in ? 1 : 0;
    };
    for (int b = begin; b < end; b += 32) {
        const int rec = b + lane;
        bool pass = false;
        if (rec < end) {
            // certainly outside r_cut in FP32: no FP64 work
            const uint2 ij = d.pair_ij[rec];
            const float4 mi = __ldg(d.mir + ij.x), mj = __ldg(d.mir + (ij.y & IDX_MASK));
            const float4 sh = tab[ij.y >> IDX_BITS];
            float ex = mj.x - mi.x + sh.x, ey = mj.y - mi.y + sh.y, ez = mj.z - mi.z + sh.z;
            if (brute) {
                if (ex < -0.5f * Lf[0]) ex += Lf[0]; else if (ex > 0.5f * Lf[0]) ex -= Lf[0];
                if (ey < -0.5f * Lf[1]) ey += Lf[1]; else if (ey > 0.5f * Lf[1]) ey -= Lf[1];
                if (ez < -0.5f * Lf[2]) ez += Lf[2]; else if (ez > 0.5f * Lf[2]) ez -= Lf[2];
            }
            const PairDev& P = d.pair[type_of(mi) * MAX_TYPES + type_of(mj)];
            pass = !(ex * ex + ey * ey + ez * ez > P.rc2f_hi * 1.0001f);
            if (!pass) d.pair_in[rec] = 0;
        }
        const unsigned got = __ballot_sync(0xffffffffu, pass);
        if (pass) qu[held + __popc(got & ((1u << lane) - 1u))] = (uint32_t)rec;
        held += __popc(got);
        __syncwarp();
        if (held >= 32) {
            held -= 32;
            compute(held + lane);
            __syncwarp();
        }
    }
    if (lane < held) compute(lane);
}

// ---------------------------------------------------------------------------
// Per-atom sums in list order, four lanes per atom: lane c adds component c of
// the records (the fourth potential and virial), so an atom's lanes read a
// record's sector together and a warp adds for eight atoms at a time -- the
// same FP64 work as a thread per atom (three or five adds for 32 atoms against
// one or two for eight) with four times the loads in flight, which is what
// bounds it: 71 -> 36 us at 23,256 atoms, 235 -> 209 us at 256,000.  The block's first warp then finishes its 32 atoms, a thread
// each.  FORCE: a fused NVE pass, whose potential and virial nobody reads (the
// chunk's last pass writes them).
constexpr int SUM_LANES = 4;

template <bool KICK, bool FORCE>
__global__ void __launch_bounds__(TILE) k_pair_sums(Dev d, StepParams sp) {
    if (chunk_failed(d)) return;
    constexpr int PER = TILE / SUM_LANES;
    __shared__ float tcs[8];
    __shared__ double S[5][PER];
    const int N = d.ntot;
    const int4 tl = d.tiles[blockIdx.x / SUM_LANES];
    const int first = (blockIdx.x % SUM_LANES) * PER;
    if (first >= tl.z) return;
    const RepDev* R = d.rep + tl.x;
    const long long rbeg = R->begin;
    const int rn = R->n;
    if (KICK && sp.fused && threadIdx.x == 0) drift_consts(*R, tcs);
    const int a = threadIdx.x / SUM_LANES, c = threadIdx.x % SUM_LANES;
    const unsigned group = ((1u << SUM_LANES) - 1u) << (threadIdx.x & 31 & ~(SUM_LANES - 1));
    const int s = tl.y + first + a;
    const int n = first + a < tl.z ? d.nn[s] : 0;
    if (KICK && threadIdx.x < PER && first + (int)threadIdx.x < tl.z) {   // the epilogue's operands, on their way
        const int es = tl.y + first + threadIdx.x;
        for (int k = 0; k < 3; ++k) prefetch_l2(d.vel + (size_t)k * N + es);
        if (sp.fused) {
            prefetch_l2(d.pos + es);
            prefetch_l2(d.mir0 + es);
            prefetch_l2(d.cell + es);
        }
    }
    double sum = 0.0, vir = 0.0;
    const uint32_t* row = d.pair_of + list_index(first + a < tl.z ? s : tl.y, 0, 1, rbeg, rn, d.cap);
    const double* rec = reinterpret_cast<const double*>(d.pair_rec) + c;
    // 32 entries at a time: which of them lie inside r_cut (a lane looks at
    // eight), then their records in order, four loaded before any is added
    constexpr int NB = 4;
    for (int k0 = 0; k0 < n; k0 += 32) {
        uint32_t in = 0u;
#pragma unroll
        for (int q = 0; q < 32 / SUM_LANES; ++q) {
            const int k = k0 + q * SUM_LANES + c;
            const uint32_t r = k < n ? __ldg(row + (size_t)k * rn) : PAIR_NONE;
            if (r != PAIR_NONE && __ldg(d.pair_in + (r & ~PAIR_NEG))) in |= 1u << (q * SUM_LANES + c);
        }
#pragma unroll
        for (int off = SUM_LANES / 2; off > 0; off >>= 1) in |= __shfl_xor_sync(group, in, off);
        while (in) {
            uint32_t r[NB];
            double x[NB], v[NB];
#pragma unroll
            for (int u = 0; u < NB; ++u) {
                r[u] = PAIR_NONE;
                if (in) r[u] = __ldg(row + (size_t)(k0 + __ffs(in) - 1) * rn);
                in &= in - 1u;
            }
#pragma unroll
            for (int u = 0; u < NB; ++u)
                if (r[u] != PAIR_NONE) {
                    x[u] = __ldg(rec + 4 * (size_t)(r[u] & ~PAIR_NEG));
                    if (!FORCE && c == 3) v[u] = __ldg(d.pair_vir + (r[u] & ~PAIR_NEG));
                }
#pragma unroll
            for (int u = 0; u < NB; ++u)
                if (r[u] != PAIR_NONE) {
                    // the partner's record: the force negated
                    const unsigned long long neg = c < 3 ? (unsigned long long)(r[u] & PAIR_NEG) << 32 : 0ull;
                    const double y =
                        __longlong_as_double((long long)((unsigned long long)__double_as_longlong(x[u]) ^ neg));
                    if (!FORCE || c < 3) sum = __dadd_rn(sum, y);
                    if (!FORCE && c == 3) vir = __dadd_rn(vir, v[u]);
                }
        }
    }
    S[c][a] = sum;
    if (!FORCE && c == 3) S[4][a] = vir;
    __syncthreads();
    if (threadIdx.x >= PER) return;
    float disp = 0.f;
    if (first + (int)threadIdx.x < tl.z) {
        const int es = tl.y + first + threadIdx.x;
        const double fx = S[0][threadIdx.x], fy = S[1][threadIdx.x], fz = S[2][threadIdx.x];
        if (!FORCE) {
            d.frc[es] = fx; d.frc[N + es] = fy; d.frc[2 * N + es] = fz;
            d.epot[es] = S[3][threadIdx.x]; d.evir[es] = S[4][threadIdx.x];
        }
        if (KICK) disp = kick_and_drift<false>(d, sp, R, tcs, es, type_of(d.pos[es]), fx, fy, fz);
    }
    if (KICK && sp.fused) note_displacement(d, tl.x, disp);
}
static_assert(TILE / SUM_LANES == 32, "one warp finishes a block's atoms");

// ---------------------------------------------------------------------------
// Host side.
cudaError_t launch_pair_build(const Dev& d, cudaStream_t st) {
    k_pair_rows<<<d.ntiles, TILE, 0, st>>>(d);
    k_pair_link<<<std::min(d.ntiles, 4096), TILE, 0, st>>>(d);
    return cudaGetLastError();
}

cudaError_t launch_pair_forces(const Dev& d, const StepParams& sp, bool kick, int num_sms, cudaStream_t st) {
    // Blocks per tile: four blocks (four warps a scheduler) keep an SM's FP64
    // pipe busy, and more would cut a warp's share to a few batches of 32, the
    // last of them partly empty.
    const int parts = std::max(1, std::min(16, (4 * num_sms + d.ntiles - 1) / d.ntiles));
    const bool force = kick && sp.fused;
    const int grid = d.ntiles * parts;
    if (d.refmode) {
        if (force) k_pair_terms<true, true><<<grid, TILE, 0, st>>>(d, parts);
        else k_pair_terms<true, false><<<grid, TILE, 0, st>>>(d, parts);
    } else {
        if (force) k_pair_terms<false, true><<<grid, TILE, 0, st>>>(d, parts);
        else k_pair_terms<false, false><<<grid, TILE, 0, st>>>(d, parts);
    }
    if (force) k_pair_sums<true, true><<<d.ntiles * SUM_LANES, TILE, 0, st>>>(d, sp);
    else if (kick) k_pair_sums<true, false><<<d.ntiles * SUM_LANES, TILE, 0, st>>>(d, sp);
    else k_pair_sums<false, false><<<d.ntiles * SUM_LANES, TILE, 0, st>>>(d, sp);
    return cudaGetLastError();
}

}  // namespace mdgb
