// force_mixed.cuh -- the mixed path's pair arithmetic, shared by the force
// kernels (kernels_force.cu) and the whole-chunk kernel of small systems
// (kernels_step.cu).  Every rounding is explicit but two: the assembler fuses the
// paired product and sums of fix_add_xyz, in either translation unit (they are
// compiled with different contraction settings; compared with fmaf over 4M random
// operands).  Both give the same bits, which tests/test_gpu_small_systems.py holds
// them to.
#pragma once
#include "force_common.cuh"

namespace mdgb {

__device__ __forceinline__ void prefetch_l1(const void* p) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}
__device__ __forceinline__ void prefetch_l2(const void* p) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// ---------------------------------------------------------------------------
// 64-bit fixed-point accumulation without float->int64 conversions (those run
// on GB300's narrow FP64 pipe).  A term v (float, already scaled to fixed-point
// units) is split exactly as v = h * 2^23 + l with h = rint(v / 2^23) and
// l = v - h * 2^23 (|l| <= 2^22, exact in FP32).  Both are rounded to integers
// by the magic-number method: adding M = 1.5 * 2^23 to a float of magnitude
// <= 2^22 lands in [2^23, 2^24], where the float's bit pattern is
// bits(M) + rint(x).  Each term's bit pattern minus bits(M) is summed modulo
// 2^32 (one three-input add per word), so
//     sum_k rint(v_k) = (sum h_k) * 2^23 + sum l_k
// exactly, in any order, for |v| <= 2^44 (the kernel re-accumulates an atom
// with exact conversions when one of its terms may be larger).
constexpr float FIX_MAGIC = 12582912.0f;           // 1.5 * 2^23
constexpr unsigned FIX_MAGIC_BITS = 0x4B400000u;   // bits of FIX_MAGIC
constexpr int FIX_FOLD = 256;                      // most terms per lane the words can hold

struct FixAcc {
    unsigned hi, lo;
    __device__ __forceinline__ void init() { hi = lo = 0u; }
    // With at most FIX_FOLD terms the two 32-bit words cannot overflow
    // (|h| <= 2^21, |l| <= 2^22 per term).
    __device__ __forceinline__ long long total() const {
        return ((long long)(int)hi << 23) + (long long)(int)lo;
    }
};

// One term per accumulator pair, with the term already divided by 2^23
// (t = v / 2^23; the scaling is exact): a = t + M holds M + rint(t) = M + h,
// l' = t - h is exact (Sterbenz) and fma(l', 2^23, M) = M + rint(v - h 2^23).
// The x and y components go through the paired instructions together; the
// assembler fuses product and sum there, as the z component is written.  (The
// same written with fma2, bits unchanged: the persistent kernel's force pass of
// 512 replicas 0.66 -> 0.82 ms.)
__device__ __forceinline__ void fix_add_xyz(FixAcc& ax, FixAcc& ay, FixAcc& az, f2_t dxy, float dz, float g) {
    const f2_t M2 = f2(FIX_MAGIC, FIX_MAGIC);
    const f2_t K2 = f2(8388608.0f, 8388608.0f);
    const f2_t t2 = mul2(dxy, f2(g, g));
    const f2_t a2 = add2(t2, M2);
    const f2_t l2 = sub2(t2, sub2(a2, M2));
    const f2_t b2 = fma2(l2, K2, M2);
    ax.hi += (unsigned)a2 - FIX_MAGIC_BITS;
    ay.hi += (unsigned)(a2 >> 32) - FIX_MAGIC_BITS;
    ax.lo += (unsigned)b2 - FIX_MAGIC_BITS;
    ay.lo += (unsigned)(b2 >> 32) - FIX_MAGIC_BITS;
    const float az_ = fmaf(dz, g, FIX_MAGIC);   // one rounding: dz g is not rounded before
    const float lz = fmaf(dz, g, -__fsub_rn(az_, FIX_MAGIC));
    const float bz = fmaf(lz, 8388608.0f, FIX_MAGIC);
    az.hi += __float_as_uint(az_) - FIX_MAGIC_BITS;
    az.lo += __float_as_uint(bz) - FIX_MAGIC_BITS;
}

// ---------------------------------------------------------------------------
// Mixed path.  The per-pair FP32 maths is shared by the loops below.
struct PairF {
    float sig2, eps4, eps24, ucut, rc2_lo, rc2_hi;
};

__device__ __forceinline__ PairF pairf(const PairDev& P) {
    return PairF{P.sig2f, P.eps4f, P.eps24f, P.ucutf, P.rc2f_lo, P.rc2f_hi};
}

// LJ for one pair at displacement (dx,dy,dz): fs = (dU/dr)/r, u = U(r).
__device__ __forceinline__ void lj_f32(const PairF& P, float r2, float& fs, float& u) {
    const float r2i = __fdividef(1.0f, r2);
    const float s2 = __fmul_rn(P.sig2, r2i);
    const float s6 = __fmul_rn(__fmul_rn(s2, s2), s2);
    // (24 eps / r^2) s6 (1 - 2 s6) = (dU/dr) / r ;  4 eps s6 (s6 - 1) - u_cut = U
    fs = __fmul_rn(__fmul_rn(__fmul_rn(P.eps24, r2i), s6), fmaf(-2.0f, s6, 1.0f));
    u = fmaf(__fmul_rn(P.eps4, s6), __fsub_rn(s6, 1.0f), -P.ucut);
}

// NAIVE: the FP32-naive variant of the precision study -- force sums in plain
// FP32 registers instead of fixed point (same pair maths).
template <bool NAIVE, bool NOE = false>
struct MixedAcc {
    FixAcc ax, ay, az;
    float fx, fy, fz;
    float pe, vr, gmax;
    __device__ __forceinline__ void init() {
        ax.init(); ay.init(); az.init();
        fx = fy = fz = 0.f;
        pe = vr = gmax = 0.f;
    }
    // fscale_t: the fixed-point scale divided by 2^23; gmax tracks |fs| * fscale_t
    __device__ __forceinline__ void add(f2_t dxy, float dz, float r2, float fs, float u, float fscale_t) {
        if (!NOE) {
            pe = __fadd_rn(pe, u);
            vr = fmaf(fs, r2, vr);
        }
        if (NAIVE) {
            fx = fmaf(f2_lo(dxy), fs, fx); fy = fmaf(f2_hi(dxy), fs, fy); fz = fmaf(dz, fs, fz);
            return;
        }
        const float g = __fmul_rn(fs, fscale_t);
        gmax = fmaxf(gmax, fabsf(g));
        fix_add_xyz(ax, ay, az, dxy, dz, g);
    }
    __device__ __forceinline__ void add(float dx, float dy, float dz, float r2, float fs, float u, float fscale_t) {
        add(f2(dx, dy), dz, r2, fs, u, fscale_t);
    }
};

// The reference's FP64 decision for one pair (potential.rs:181-204: the
// minimum-image displacement, r = sqrt(r^2), interacting when r <= r_cut);
// on success (dx,dy,dz) is the FP64 displacement rounded to FP32.  No square
// root: sqrt_rn(r^2) <= r_cut exactly when r^2 < rc2_cut, the smallest double
// whose correctly rounded square root exceeds r_cut (computed on the host).
__device__ __forceinline__ bool exact_pair(const Dev& d, const RepDev* R, int s, int j, const PairDev& PD,
                                           float& dx, float& dy, float& dz) {
    const double4_32a pi = d.pos[s], pj = d.pos[j];
    const double rx = min_image_ref(__dsub_rn(pj.x, pi.x), R->box[0]);
    const double ry = min_image_ref(__dsub_rn(pj.y, pi.y), R->box[1]);
    const double rz = min_image_ref(__dsub_rn(pj.z, pi.z), R->box[2]);
    const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(rx, rx), __dmul_rn(ry, ry)), __dmul_rn(rz, rz));
    // both non-negative: the bit patterns order like the values
    if (__double_as_longlong(r2) >= __double_as_longlong(PD.rc2_cut)) return false;
    dx = dbl_to_flt_rn(rx); dy = dbl_to_flt_rn(ry); dz = dbl_to_flt_rn(rz);
    return true;
}

// One atom with a pair in the band around r_cut^2, by one warp: lanes over the
// list, band pairs decided with the reference's FP64 arithmetic, every term
// rounded to fixed point as the main kernel does.  COH: data of this launch
// (no non-coherent loads).
template <bool NAIVE, bool COH>
__device__ __forceinline__ void band_atom(const Dev& d, const StepParams& sp, int s, int rep, bool kick) {
    const int N = d.ntot;
    const int lane = threadIdx.x & 31;
    const float fscale = d.fscale;
    const float rl = (float)(d.rlist * 1.01);
    const float range_limit = 36028797018963968.0f / rl;   // 2^55 / rlist
    const RepDev* R = d.rep + rep;
    const long long rbeg = R->begin;
    const int rn = R->n, tpa = R->tpa;
    const float csf[3] = {(float)R->cs[0], (float)R->cs[1], (float)R->cs[2]};
    const float4 xi = d.mir[s];
    const int ty = type_of(xi);
    const int n = d.nn[s];
    if (kick && lane == 0) {   // the epilogue's operands, on their way
        prefetch_l2(d.vel + s);
        prefetch_l2(d.vel + N + s);
        prefetch_l2(d.vel + 2 * N + s);
        if (sp.fused) {
            prefetch_l2(d.pos + s);
            prefetch_l2(d.mir0 + s);
            prefetch_l2(d.cell + s);
        }
    }
    long long sx = 0, sy = 0, sz = 0;
    float fx = 0.f, fy = 0.f, fz = 0.f, pe = 0.f, vr = 0.f;
    bool over = false;
    // this lane's list words and neighbour mirrors, all loads issued before
    // the maths (the warp handles one atom: latency is the whole cost)
    constexpr int KB = 4;
    uint32_t eb[KB];
    float4 xb[KB];
#pragma unroll
    for (int q = 0; q < KB; ++q) {
        const int k = lane + 32 * q;
        eb[q] = k < n ? (COH ? d.nbr[list_index(s, k, tpa, rbeg, rn, d.cap)] : __ldcs(d.nbr + list_index(s, k, tpa, rbeg, rn, d.cap))) : 0u;
    }
#pragma unroll
    for (int q = 0; q < KB; ++q) xb[q] = COH ? d.mir[eb[q] & IDX_MASK] : __ldg(d.mir + (eb[q] & IDX_MASK));
    auto entry = [&](uint32_t e, float4 xj) {
        const int j = (int)(e & IDX_MASK);
        const int c = (int)(e >> IDX_BITS);
        // the shift table of the main kernel (shift_table)
        const float shx = (float)(c % 3 - 1) * csf[0], shy = (float)((c / 3) % 3 - 1) * csf[1],
                    shz = (float)(c / 9 - 1) * csf[2];
        const f2_t dxy = add2(sub2(f2(xj.x, xj.y), f2(xi.x, xi.y)), f2(shx, shy));
        float dx = f2_lo(dxy), dy = f2_hi(dxy), dz = xj.z - xi.z + shz;
        const PairDev& PD = d.pair[ty * MAX_TYPES + type_of(xj)];
        const PairF P = pairf(PD);
        const float r2 = fmaf(dz, dz, fmaf(dy, dy, __fmul_rn(dx, dx)));
        if (r2 > P.rc2_hi) return;
        float rr2 = r2;
        if (r2 >= P.rc2_lo) {
            if (!exact_pair(d, R, s, j, PD, dx, dy, dz)) return;
            rr2 = fmaf(dz, dz, fmaf(dy, dy, __fmul_rn(dx, dx)));
        }
        float fs, u;
        lj_f32(P, rr2, fs, u);
        pe = __fadd_rn(pe, u);
        vr = fmaf(fs, rr2, vr);
        if (NAIVE) {
            fx = fmaf(dx, fs, fx); fy = fmaf(dy, fs, fy); fz = fmaf(dz, fs, fz);
        } else {
            const float g = fs * fscale;
            over |= fabsf(g) > range_limit;
            sx += __float2ll_rn(dx * g);
            sy += __float2ll_rn(dy * g);
            sz += __float2ll_rn(dz * g);
        }
    };
#pragma unroll
    for (int q = 0; q < KB; ++q)
        if (lane + 32 * q < n) entry(eb[q], xb[q]);
    for (int k = lane + 32 * KB; k < n; k += 32) {
        const uint32_t e = (COH ? d.nbr[list_index(s, k, tpa, rbeg, rn, d.cap)] : __ldcs(d.nbr + list_index(s, k, tpa, rbeg, rn, d.cap)));
        entry(e, COH ? d.mir[e & IDX_MASK] : __ldg(d.mir + (e & IDX_MASK)));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        sx += __shfl_down_sync(0xffffffffu, sx, off);
        sy += __shfl_down_sync(0xffffffffu, sy, off);
        sz += __shfl_down_sync(0xffffffffu, sz, off);
        fx += __shfl_down_sync(0xffffffffu, fx, off);
        fy += __shfl_down_sync(0xffffffffu, fy, off);
        fz += __shfl_down_sync(0xffffffffu, fz, off);
        pe += __shfl_down_sync(0xffffffffu, pe, off);
        vr += __shfl_down_sync(0xffffffffu, vr, off);
    }
    if (over) atomicOr(d.err, E_FIXED);
    if (lane == 0) {
        const double Fx = NAIVE ? flt_to_dbl(fx) : fixed_to_double(sx, d.fscale_log2);
        const double Fy = NAIVE ? flt_to_dbl(fy) : fixed_to_double(sy, d.fscale_log2);
        const double Fz = NAIVE ? flt_to_dbl(fz) : fixed_to_double(sz, d.fscale_log2);
        d.frc[s] = Fx; d.frc[N + s] = Fy; d.frc[2 * N + s] = Fz;
        d.epot[s] = flt_to_dbl(pe); d.evir[s] = flt_to_dbl(vr);
        if (kick) {
            float tcs[8];
            drift_consts(*R, tcs);
            const float disp = kick_and_drift<true>(d, sp, R, tcs, s, ty, Fx, Fy, Fz);
            if (sp.fused && disp > 0.f) atomicMax(&d.rep[rep].max_disp_bits, __float_as_uint(disp));
        }
    }
}

}  // namespace mdgb
