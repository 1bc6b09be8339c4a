// kernels_force.cu -- Lennard-Jones pair forces over the Verlet list.
//
// Replaces update_force (solver/src/solver/potential.rs:158-216): per atom i
// the force F_i = sum_j r_ij/|r_ij| * dU/dr(|r_ij|), the potential sum
// U_i = sum_j U(|r_ij|) and temp_i = sum_j F_ij . r_ij over every j with
// |r_ij| <= r_cut, r_ij = x_j - x_i taken to the image picked by the
// reference's single-shift rule (potential.rs:186-200).
//
// k_force_fp64  -- the plain path of systems without pair records
//   (kernels_pairs.cu), with the same pair terms (force_common.cuh): with
//   MDGB_FLAG_REFERENCE_ORDER the bits of the reference's FP64 operation
//   sequence, and the list in the reference's j order, so the per-atom sums are
//   bit-identical too; in tree order functions of r^2.  An FP32 prefilter on
//   the mirror skips candidates that are certainly outside r_cut.
// k_force_mixed -- the chosen path.  FP32 pair maths from the float4 mirror
//   (cell-relative coordinates, periodic cell shift from the list entry),
//   force sums in deterministic 64-bit fixed point, potential/virial in FP32
//   per atom (FP64 across atoms).  An atom with a pair whose FP32 r^2 lies
//   within 1e-5 of r_cut^2 is left whole to k_force_band, which decides those
//   pairs with the reference's FP64 arithmetic, so the set of interacting
//   pairs equals the reference's.
//
// Both end with the second half kick v += F dt/2m (integrator.rs:49-55) when
// called from a step, and on NVE chunks with the next step's first kick and
// drift (kick_and_drift).  TPA threads share one atom's list; their partial
// sums are combined by a fixed shuffle tree.  The fused passes of an NVE chunk
// (NOE) neither sum the per-atom potential and virial nor store them or the
// forces (both kicks take the forces from registers): the chunk's last,
// unfused pass writes all three, and nothing reads them in between.  The
// kick/drift FP64 helpers get the FMA-or-not choice as a compile-time
// constant (a run-time flag made the compiler issue both forms).
#include "force_mixed.cuh"

namespace mdgb {

template <int TPA>
__device__ __forceinline__ long long tpa_sum_ll(long long v) {
#pragma unroll
    for (int off = TPA / 2; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off, TPA);
    return v;
}
template <int TPA>
__device__ __forceinline__ double tpa_sum_d(double v) {
#pragma unroll
    for (int off = TPA / 2; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off, TPA);
    return v;
}
template <int TPA>
__device__ __forceinline__ float tpa_sum_f(float v) {
#pragma unroll
    for (int off = TPA / 2; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off, TPA);
    return v;
}

// The next tile of this launch's tile list: one per block, or (persistent)
// from a work counter over the list, costliest tiles first.
__device__ __forceinline__ int next_tile(const Dev& d, bool persistent, int& iter, int* s_tile) {
    if (!persistent) return (iter++ == 0 && (int)blockIdx.x < d.ntile_list) ? d.tile_list[blockIdx.x] : -1;
    __syncthreads();
    if (threadIdx.x == 0) *s_tile = (int)atomicAdd(d.queue + d.list_class, 1u);
    __syncthreads();
    const int q = *s_tile;
    if (q >= d.ntile_list) return -1;
    return d.tile_list[q];
}

// ---------------------------------------------------------------------------
template <int TPA, bool KICK, bool PERSIST>
__global__ void __launch_bounds__(TILE * TPA) k_force_fp64(Dev d, StepParams sp) {
    if (chunk_failed(d)) return;
    __shared__ float4 tab[27];
    __shared__ float tcs[8];
    __shared__ int s_tile;
    const int N = d.ntot;
    const int a = threadIdx.x / TPA, lane = threadIdx.x % TPA;
    int iter = 0;
    for (;;) {
        const int t = next_tile(d, PERSIST, iter, &s_tile);
        if (t < 0) break;
        const int4 tl = d.tiles[t];
        const RepDev* R = d.rep + tl.x;
        const long long rbeg = R->begin;
        const int rn = R->n;
        __syncthreads();
        shift_table(tab, R);
        if (KICK && sp.fused && threadIdx.x == 0) drift_consts(*R, tcs);
        __syncthreads();
        const double box[3] = {R->box[0], R->box[1], R->box[2]};
        const float Lf[3] = {(float)box[0], (float)box[1], (float)box[2]};
        const bool brute = R->mode == MODE_BRUTE;
        const int s = tl.y + a;
        const bool act = a < tl.z;
        double fx = 0.0, fy = 0.0, fz = 0.0, pe = 0.0, vr = 0.0;
        int ty = 0;
        if (act) {
            const double4_32a pi = d.pos[s];
            const float4 mi = d.mir[s];
            ty = type_of(pi);
            const int n = d.nn[s];
            for (int k = lane; k < n; k += TPA) {
                const uint32_t e = __ldcs(d.nbr + list_index(s, k, TPA, rbeg, rn, d.cap));
                const int j = (int)(e & IDX_MASK);
                const PairDev& P = d.pair[ty * MAX_TYPES + type_of(__ldg(d.mir + j))];
                // FP32 prefilter (certainly outside r_cut -> skip)
                {
                    const float4 mj = __ldg(d.mir + j);
                    const float4 sh = tab[e >> IDX_BITS];
                    float ex = mj.x - mi.x + sh.x, ey = mj.y - mi.y + sh.y, ez = mj.z - mi.z + sh.z;
                    if (brute) {
                        if (ex < -0.5f * Lf[0]) ex += Lf[0]; else if (ex > 0.5f * Lf[0]) ex -= Lf[0];
                        if (ey < -0.5f * Lf[1]) ey += Lf[1]; else if (ey > 0.5f * Lf[1]) ey -= Lf[1];
                        if (ez < -0.5f * Lf[2]) ez += Lf[2]; else if (ez > 0.5f * Lf[2]) ez -= Lf[2];
                    }
                    if (ex * ex + ey * ey + ez * ez > P.rc2f_hi * 1.0001f) continue;
                }
                const double4_32a pj = d.pos[j];
                // the terms of k_pair_terms and k_steps: which of the three
                // kernels runs (memory, size) moves no bit
                const double rx = min_image_ref(__dsub_rn(pj.x, pi.x), box[0]);
                const double ry = min_image_ref(__dsub_rn(pj.y, pi.y), box[1]);
                const double rz = min_image_ref(__dsub_rn(pj.z, pi.z), box[2]);
                const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(rx, rx), __dmul_rn(ry, ry)), __dmul_rn(rz, rz));
                PairTerms o;
                if (!(d.refmode ? ref_terms<false>(rx, ry, rz, r2, P, o) : r2_terms<false>(rx, ry, rz, r2, P, o)))
                    continue;
                fx = __dadd_rn(fx, o.gx); fy = __dadd_rn(fy, o.gy); fz = __dadd_rn(fz, o.gz);
                pe = __dadd_rn(pe, o.u);
                vr = __dadd_rn(vr, o.t);
            }
        }
        if (TPA > 1) {
            fx = tpa_sum_d<TPA>(fx); fy = tpa_sum_d<TPA>(fy); fz = tpa_sum_d<TPA>(fz);
            pe = tpa_sum_d<TPA>(pe); vr = tpa_sum_d<TPA>(vr);
        }
        float disp = 0.f;
        if (act && lane == 0) {
            d.frc[s] = fx; d.frc[N + s] = fy; d.frc[2 * N + s] = fz;
            d.epot[s] = pe; d.evir[s] = vr;
            if (KICK) disp = kick_and_drift<false>(d, sp, R, tcs, s, ty, fx, fy, fz);   // integrator.rs:49-55
        }
        if (KICK && sp.fused) note_displacement(d, tl.x, disp);
    }
}

template <int TPA, bool SINGLE, bool KICK, bool PERSIST, bool NAIVE = false, bool NOE = false>
// 9 blocks of 128 threads per SM (56 registers): the kernel is latency-bound
// on its neighbour gathers, so it keeps as many warps resident as it can.  The
// variants that also sum potential and virial need two more registers than
// that allows (at 56 they spill): 8 blocks, 64 registers.
__global__ void __launch_bounds__(TILE * TPA, ((NOE ? 9 : 8) / TPA) > 0 ? ((NOE ? 9 : 8) / TPA) : 1)
    k_force_mixed(Dev d, StepParams sp) {
    if (chunk_failed(d)) return;
    __shared__ float4 tab[27];
    __shared__ float tcs[8];
    __shared__ int s_tile;
    const int N = d.ntot;
    const int a = threadIdx.x / TPA, lane = threadIdx.x % TPA;
    const float fscale = d.fscale;
    const float fscale_t = NAIVE ? 1.0f : fscale * 1.1920928955078125e-07f;   // fscale / 2^23 (exact)
    // each term |dx * g| <= rlist * gmax; the magic-number split is exact up to
    // 2^44 fixed-point units, i.e. |t| <= 2^21 after the division by 2^23
    const float rl = (float)(d.rlist * 1.01);
    const float split_limit = 2097152.0f / rl;       // 2^44 / 2^23 / rlist
    const float range_limit = 4294967296.0f / rl;    // 2^55 / 2^23 / rlist
    int iter = 0;
    for (;;) {
        const int t = next_tile(d, PERSIST, iter, &s_tile);
        if (t < 0) break;
        const int4 tl = d.tiles[t];
        const RepDev* R = d.rep + tl.x;
        const long long rbeg = R->begin;
        const int rn = R->n;
        __syncthreads();
        shift_table(tab, R);
        if (KICK && sp.fused && threadIdx.x == 0) drift_consts(*R, tcs);
        __syncthreads();
        const bool brute = R->mode == MODE_BRUTE;
        const int s = tl.y + a;
        const bool act = a < tl.z;
        if (KICK && act && lane == 0) {
            // the epilogue's operands: in L2 by the time the pair loop is done
            prefetch_l2(d.vel + s);
            prefetch_l2(d.vel + N + s);
            prefetch_l2(d.vel + 2 * N + s);
            if (sp.fused) {
                prefetch_l2(d.pos + s);
                prefetch_l2(d.mir0 + s);
                prefetch_l2(d.cell + s);
            }
        }
        MixedAcc<NAIVE, NOE> acc;
        acc.init();
        int ty = 0, n_own = 0;
        bool deferred = false;   // an atom with a pair in the band goes to k_force_band whole
        if (act) {
            const float4 xi = d.mir[s];
            ty = type_of(xi);
            PairF P0{};
            if (SINGLE) P0 = pairf(d.pair[ty * MAX_TYPES + ty]);
            const int n = d.nn[s];
            n_own = n;
            if (!brute) {
                // hot loop: FP32 and integer work only, two candidates in flight
                bool band = false;
                const f2_t xixy = f2(xi.x, xi.y);
                auto pair = [&](uint32_t e, float4 xj) {
                    const float4 sh = tab[e >> IDX_BITS];
                    const f2_t dxy = add2(sub2(f2(xj.x, xj.y), xixy), f2(sh.x, sh.y));
                    const float dz = __fadd_rn(__fsub_rn(xj.z, xi.z), sh.z);
                    const PairF P = SINGLE ? P0 : pairf(d.pair[ty * MAX_TYPES + type_of(xj)]);
                    const float dx = f2_lo(dxy), dy = f2_hi(dxy);
                    const float r2 = fmaf(dz, dz, fmaf(dy, dy, __fmul_rn(dx, dx)));
                    if (r2 >= P.rc2_lo) {
                        // within 1e-5 of r_cut^2: the atom is finished by k_force_band
                        band |= r2 <= P.rc2_hi;
                        return;
                    }
                    float fs, u;
                    lj_f32(P, r2, fs, u);
                    acc.add(dxy, dz, r2, fs, u, fscale_t);
                };
                // this lane's entries k = lane, lane + TPA, ...: two per iteration,
                // the next iteration's two list words already in flight (the list
                // streams from HBM; the gathers hit L2)
                const uint32_t* lbase = d.nbr + list_index(s, lane, TPA, rbeg, rn, d.cap);
                const size_t lstride = (size_t)rn * TPA;
                const int m = n > lane ? (n - lane + TPA - 1) / TPA : 0;
                uint32_t ea = 0u, eb = 0u;
                if (m > 0) ea = __ldcs(lbase);
                if (m > 1) eb = __ldcs(lbase + lstride);
                int i = 0;
                for (; i + 1 < m; i += 2) {
                    const float4 xa = __ldg(d.mir + (ea & IDX_MASK));
                    const float4 xb = __ldg(d.mir + (eb & IDX_MASK));
                    uint32_t na = 0u, nb = 0u;
                    if (i + 2 < m) na = __ldcs(lbase + (size_t)(i + 2) * lstride);
                    if (i + 3 < m) nb = __ldcs(lbase + (size_t)(i + 3) * lstride);
                    pair(ea, xa);
                    pair(eb, xb);
                    ea = na;
                    eb = nb;
                }
                if (i < m) pair(ea, __ldg(d.mir + (ea & IDX_MASK)));
                deferred = band;
            } else {
                // brute mode (a box smaller than three list radii): the reference's
                // FP64 displacement for every pair -- these replicas are tiny
                for (int k = lane; k < n; k += TPA) {
                    const uint32_t e = __ldcs(d.nbr + list_index(s, k, TPA, rbeg, rn, d.cap));
                    const int j = (int)(e & IDX_MASK);
                    const PairDev& PD = d.pair[ty * MAX_TYPES + type_of(__ldg(d.mir + j))];
                    float dx, dy, dz;
                    if (!exact_pair(d, R, s, j, PD, dx, dy, dz)) continue;
                    const float r2 = fmaf(dz, dz, fmaf(dy, dy, __fmul_rn(dx, dx)));
                    float fs, u;
                    lj_f32(pairf(PD), r2, fs, u);
                    acc.add(dx, dy, dz, r2, fs, u, fscale_t);
                }
            }
        }
        if (TPA > 1) {
#pragma unroll
            for (int off = TPA / 2; off > 0; off >>= 1) deferred |= __shfl_xor_sync(0xffffffffu, deferred, off, TPA);
        }
        if (deferred && lane == 0) {
            const int slot = atomicAdd(d.band_count, 1);
            d.band_list[slot] = make_int2(s, tl.x);
        }
        long long sx = acc.ax.total(), sy = acc.ay.total(), sz = acc.az.total();
        // terms this lane summed: at most its share of the list
        const int nl = act && n_own > lane ? (n_own - lane + TPA - 1) / TPA : 0;
        if (!NAIVE && act && !deferred && (acc.gmax > split_limit || nl > FIX_FOLD)) {
            // a term may exceed the exact range of the split, or the lane summed
            // more terms than the 32-bit words hold: redo this lane's terms with
            // exact float -> int64 conversions (very close pairs, huge lists)
            if (acc.gmax > range_limit) atomicOr(d.err, E_FIXED);
            sx = sy = sz = 0;
            const float4 xi = d.mir[s];
            const int n = d.nn[s];
            for (int k = lane; k < n; k += TPA) {
                const uint32_t e = __ldcs(d.nbr + list_index(s, k, TPA, rbeg, rn, d.cap));
                const int j = (int)(e & IDX_MASK);
                const float4 xj = __ldg(d.mir + j);
                const float4 sh = tab[e >> IDX_BITS];
                float dx = xj.x - xi.x + sh.x, dy = xj.y - xi.y + sh.y, dz = xj.z - xi.z + sh.z;
                const PairDev& PD = d.pair[ty * MAX_TYPES + type_of(xj)];
                const PairF P = pairf(PD);
                if (brute) {
                    if (!exact_pair(d, R, s, j, PD, dx, dy, dz)) continue;
                } else {
                    const float r2 = fmaf(dz, dz, fmaf(dy, dy, __fmul_rn(dx, dx)));
                    if (r2 > P.rc2_hi) continue;
                    if (r2 >= P.rc2_lo && !exact_pair(d, R, s, j, PD, dx, dy, dz)) continue;
                }
                const float r2 = fmaf(dz, dz, fmaf(dy, dy, __fmul_rn(dx, dx)));
                float fs, u;
                lj_f32(P, r2, fs, u);
                const float g = fs * fscale;
                sx += __float2ll_rn(dx * g);
                sy += __float2ll_rn(dy * g);
                sz += __float2ll_rn(dz * g);
            }
        }
        float pe = acc.pe, vr = acc.vr;
        float nfx = acc.fx, nfy = acc.fy, nfz = acc.fz;
        if (TPA > 1) {
            if (NAIVE) {
                nfx = tpa_sum_f<TPA>(nfx); nfy = tpa_sum_f<TPA>(nfy); nfz = tpa_sum_f<TPA>(nfz);
            } else {
                sx = tpa_sum_ll<TPA>(sx); sy = tpa_sum_ll<TPA>(sy); sz = tpa_sum_ll<TPA>(sz);
            }
            if (!NOE) { pe = tpa_sum_f<TPA>(pe); vr = tpa_sum_f<TPA>(vr); }
        }
        float disp = 0.f;
        if (act && lane == 0 && !deferred) {
            const double fx = NAIVE ? flt_to_dbl(nfx) : fixed_to_double(sx, d.fscale_log2);
            const double fy = NAIVE ? flt_to_dbl(nfy) : fixed_to_double(sy, d.fscale_log2);
            const double fz = NAIVE ? flt_to_dbl(nfz) : fixed_to_double(sz, d.fscale_log2);
            if (!NOE) {
                d.frc[s] = fx; d.frc[N + s] = fy; d.frc[2 * N + s] = fz;
                d.epot[s] = flt_to_dbl(pe); d.evir[s] = flt_to_dbl(vr);
            }
            if (KICK) disp = kick_and_drift<true>(d, sp, R, tcs, s, ty, fx, fy, fz);
        }
        if (KICK && sp.fused) note_displacement(d, tl.x, disp);
    }
}

// ---------------------------------------------------------------------------
// Atoms with a pair whose FP32 r^2 lies within 1e-5 of r_cut^2 (about one in
// six hundred per step): k_force_mixed leaves them (and their kick/drift) to
// this kernel, so its hot loop carries no FP64 code and no second pass
// (an inline second pass cost ~9 % of the force kernel's time although it
// almost never ran).  One warp per atom, lanes over the list; the band pairs
// are decided with the reference's FP64 arithmetic (no square root: the
// r^2 threshold of exact_pair); every term is rounded to fixed point exactly as in
// k_force_mixed (rint(dx * g), here by the conversion instruction), so the
// force sums are the ones the main kernel would have produced.  Potential and
// temp are FP32 sums in a fixed shuffle order.
template <bool NAIVE>
__global__ void __launch_bounds__(128) k_force_band(Dev d, StepParams sp, int kick) {
    if (chunk_failed(d)) return;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    const int count = *(volatile const int*)d.band_count;
    for (int w = gw; w < count; w += nw) {
        const int2 sr = d.band_list[w];
        band_atom<NAIVE, false>(d, sp, sr.x, sr.y, kick != 0);
    }
}

// ---------------------------------------------------------------------------
// Host-side launch table.  precision: 0 FP64 plain, 1 mixed, 2 FP32-naive.
using force_fn = void (*)(Dev, StepParams);

template <int TPA, bool KICK, bool PERSIST>
static force_fn pick_mixed(bool single, bool naive, bool noe) {
    if constexpr (KICK) {
        if (noe && !naive)
            return single ? (force_fn)k_force_mixed<TPA, true, true, PERSIST, false, true>
                          : (force_fn)k_force_mixed<TPA, false, true, PERSIST, false, true>;
    }
    if (naive)
        return single ? (force_fn)k_force_mixed<TPA, true, KICK, PERSIST, true>
                      : (force_fn)k_force_mixed<TPA, false, KICK, PERSIST, true>;
    return single ? (force_fn)k_force_mixed<TPA, true, KICK, PERSIST>
                  : (force_fn)k_force_mixed<TPA, false, KICK, PERSIST>;
}

template <int TPA, bool PERSIST>
static force_fn pick_tpa(int precision, bool single, bool kick, bool noe) {
    if (precision != 0) {
        const bool naive = precision == 2;
        return kick ? pick_mixed<TPA, true, PERSIST>(single, naive, noe)
                    : pick_mixed<TPA, false, PERSIST>(single, naive, noe);
    }
    return kick ? (force_fn)k_force_fp64<TPA, true, PERSIST> : (force_fn)k_force_fp64<TPA, false, PERSIST>;
}

template <bool PERSIST>
static force_fn pick_persist(int tpa, int precision, bool single, bool kick, bool noe) {
    switch (tpa) {
        case 1: return pick_tpa<1, PERSIST>(precision, single, kick, noe);
        case 2: return pick_tpa<2, PERSIST>(precision, single, kick, noe);
        case 4: return pick_tpa<4, PERSIST>(precision, single, kick, noe);
        case 8: return pick_tpa<8, PERSIST>(precision, single, kick, noe);
        default: return nullptr;
    }
}

using band_fn = void (*)(Dev, StepParams, int);
band_fn band_kernel(int precision) {
    if (precision == 0) return nullptr;
    return precision == 2 ? (band_fn)k_force_band<true> : (band_fn)k_force_band<false>;
}

// noe: a fused NVE pass (no per-atom potential/virial); mixed path only.
force_fn force_kernel(int tpa, int precision, bool single, bool kick, bool persistent, bool noe) {
    return persistent ? pick_persist<true>(tpa, precision, single, kick, noe)
                      : pick_persist<false>(tpa, precision, single, kick, noe);
}

}  // namespace mdgb
