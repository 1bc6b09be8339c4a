// force_common.cuh -- device helpers of the force kernels (kernels_force.cu,
// kernels_pairs.cu, the whole-chunk kernel in kernels_step.cu).
#pragma once
#include "mdgb_internal.cuh"

namespace mdgb {

__device__ __forceinline__ void shift_table(float4* tab, const RepDev* R) {
    if (threadIdx.x < 27) {
        const int c = threadIdx.x;
        const float dx = (float)(c % 3 - 1), dy = (float)((c / 3) % 3 - 1), dz = (float)(c / 9 - 1);
        tab[c] = make_float4(dx * (float)R->cs[0], dy * (float)R->cs[1], dz * (float)R->cs[2], 0.f);
    }
}

// The reference's minimum image of one FP64 displacement component
// (potential.rs:186-200: r < -L/2 -> r + L, r > L/2 -> r - L) with the
// comparisons on the bit patterns (L/2 exact: exponent - 1): integer work
// instead of GB300's narrow FP64 pipe.
__device__ __forceinline__ double min_image_ref(double r, double L) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(r);
    const unsigned long long mag = b & 0x7FFFFFFFFFFFFFFFull;
    const unsigned long long half = (unsigned long long)__double_as_longlong(L) - (1ull << 52);
    if (mag > half) {
        // r + L or r - L: the sign of L set in its bits (-L as an expression
        // costs an FP64 instruction on every call)
        const unsigned long long s = ~b & 0x8000000000000000ull;
        return dadd_nospec(r, __longlong_as_double((long long)((unsigned long long)__double_as_longlong(L) ^ s)));
    }
    return r;
}

// |r| > L/2, as min_image_ref decides it.
__device__ __forceinline__ bool beyond_half(double r, double L) {
    return ((unsigned long long)__double_as_longlong(r) & 0x7FFFFFFFFFFFFFFFull) >
           (unsigned long long)__double_as_longlong(L) - (1ull << 52);
}

// The terms of one pair, from the side of the atom the displacement starts at.
struct PairTerms {
    double gx, gy, gz, u, t;
};

// The reference's operation sequence (potential.rs:57-75, :201-211) with the
// library's square root and divisions.  False: |r| > r_cut.
static __device__ __noinline__ bool ref_terms_plain(double rx, double ry, double rz, double r2, const PairDev& P,
                                             PairTerms& o) {
    const double r = __dsqrt_rn(r2);
    if (r > P.rc) return false;                                          // :202-204
    const double sr = __ddiv_rn(P.sigma, r);
    const double s2 = __dmul_rn(sr, sr);
    const double s4 = __dmul_rn(s2, s2);
    const double s6 = __dmul_rn(s2, s4);
    const double s12 = __dmul_rn(s6, s6);
    o.u = __dsub_rn(__dmul_rn(P.eps4, __dsub_rn(s12, s6)), P.ucut);
    const double dudr = __dmul_rn(__ddiv_rn(P.eps24, r), __dsub_rn(s6, __dmul_rn(2.0, s12)));
    o.gx = __dmul_rn(__ddiv_rn(rx, r), dudr);                            // :207-211
    o.gy = __dmul_rn(__ddiv_rn(ry, r), dudr);
    o.gz = __dmul_rn(__ddiv_rn(rz, r), dudr);
    o.t = __dadd_rn(__dadd_rn(__dmul_rn(o.gx, rx), __dmul_rn(o.gy, ry)), __dmul_rn(o.gz, rz));
    return true;
}

__device__ __forceinline__ int exp_field(double x) { return (__double2hiint(x) >> 20) & 0x7FF; }

// An approximation of 1/sqrt(x) or 1/x to about 2^-22, from FP32; x in the
// FP32 range.
__device__ __forceinline__ double seed_rsqrt(double x) { return flt_to_dbl(rsqrtf(dbl_to_flt_rn(x))); }
__device__ __forceinline__ double seed_rcp(double x) { return flt_to_dbl(__fdividef(1.0f, dbl_to_flt_rn(x))); }

// a / r correctly rounded, from y = 1/r within half a unit in the last place
// (and a rounding of 2^-104) and yl = 1/r - y: q0 is within half a unit plus
// 2^-50 of the quotient, its remainder is exact, and one correction rounds
// correctly (Markstein 1990: a quotient lies at least 2^-106 r^-1 from the
// middle of two doubles, further than the correction's own error; the one
// exception is an r within a few units below a power of two).
__device__ __forceinline__ double div_by(double a, double r, double y, double yl) {
    const double q0 = __fma_rn(a, y, __dmul_rn(a, yl));
    return __fma_rn(__fma_rn(-r, q0, a), y, q0);
}

// The same terms, bit for bit, with one square root and one reciprocal for the
// five divisions by r: 1/sqrt(r2) by Newton's iteration (third order, from the
// FP32 seed), r from it by one correction step whose remainder is checked (a
// correctly rounded root has -u r < r2 - r^2 <= u r, u its unit in the last
// place), 1/r in two words, and div_by.  58 FP64 instructions against about 78
// with the library's divisions.  Values outside a range that keeps every
// intermediate normal take the plain form.
// FORCE: only the force is wanted (50).
template <bool FORCE>
__device__ __forceinline__ bool ref_terms(double rx, double ry, double rz, double r2, const PairDev& P, PairTerms& o) {
    const int e2 = exp_field(r2);
    const auto tame = [](double x) { const int e = exp_field(x); return e > 1023 - 400 || x == 0.0; };
    bool ok = e2 > 1023 - 100 && e2 < 1023 + 100;
    ok = ok && tame(rx) && tame(ry) && tame(rz);
    double r = 0.0, y = 0.0;
    if (ok) {
        // r2 is below r_cut^2 exactly when its rounded root is at most r_cut
        if (__double_as_longlong(r2) >= __double_as_longlong(P.rc2_cut)) return false;
        const double y0 = seed_rsqrt(r2);
        const double e = __fma_rn(-__dmul_rn(r2, y0), y0, 1.0);
        y = __fma_rn(__dmul_rn(y0, e), __fma_rn(0.375, e, 0.5), y0);
        const double g = __dmul_rn(r2, y);
        const double h = __longlong_as_double(__double_as_longlong(y) - (1ll << 52));   // y / 2
        r = __fma_rn(__fma_rn(-g, g, r2), h, g);
        const double rem = __fma_rn(-r, r, r2);
        const long long rb = __double_as_longlong(rem), mag = rb & 0x7FFFFFFFFFFFFFFFll;
        // bits of u r, u = 2^(exponent of r - 52)
        const long long lim = __double_as_longlong(r) + ((long long)(exp_field(r) - 1023 - 52) << 52);
        ok = mag < lim || rb == lim;
        // 1/r of an r just below a power of two does not round from y
        ok = ok && (__double_as_longlong(r) & 0xFFFFFFFFFFFFFll) < 0xFFFFFFFFFFF00ll;
    }
    if (!ok) return ref_terms_plain(rx, ry, rz, r2, P, o);
    y = __fma_rn(__fma_rn(-r, y, 1.0), y, y);
    const double yl = __dmul_rn(__fma_rn(-r, y, 1.0), y);
    const double sr = div_by(P.sigma, r, y, yl);
    const double s2 = __dmul_rn(sr, sr);
    const double s4 = __dmul_rn(s2, s2);
    const double s6 = __dmul_rn(s2, s4);
    const double s12 = __dmul_rn(s6, s6);
    if (!FORCE) o.u = __dsub_rn(__dmul_rn(P.eps4, __dsub_rn(s12, s6)), P.ucut);
    const double dudr = __dmul_rn(div_by(P.eps24, r, y, yl), __fma_rn(-2.0, s12, s6));   // 2 s12 is exact
    o.gx = __dmul_rn(div_by(rx, r, y, yl), dudr);
    o.gy = __dmul_rn(div_by(ry, r, y, yl), dudr);
    o.gz = __dmul_rn(div_by(rz, r, y, yl), dudr);
    if (!FORCE)
        o.t = __dadd_rn(__dadd_rn(__dmul_rn(o.gx, rx), __dmul_rn(o.gy, ry)), __dmul_rn(o.gz, rz));
    return true;
}

// Tree order (no MDGB_FLAG_REFERENCE_ORDER): the same functions of r^2 without
// the root and the divisions by r -- sigma^2 / r^2 by one Newton step, F . r =
// r dU/dr -- 24 FP64 instructions, 21 for the force alone.  Fewer roundings than the reference's form
// ((sigma / r)^6 carries six times the rounding of r and of the quotient).
template <bool FORCE>
__device__ __forceinline__ bool r2_terms(double rx, double ry, double rz, double r2, const PairDev& P, PairTerms& o) {
    const int e2 = exp_field(r2);
    if (!(e2 > 1023 - 100 && e2 < 1023 + 100)) return ref_terms_plain(rx, ry, rz, r2, P, o);
    if (__double_as_longlong(r2) >= __double_as_longlong(P.rc2_cut)) return false;
    const double y0 = seed_rcp(r2);
    const double e = __fma_rn(-r2, y0, 1.0);
    const double y = __fma_rn(__fma_rn(e, e, e), y0, y0);
    const double s2 = __dmul_rn(P.sig2, y);
    const double s6 = __dmul_rn(__dmul_rn(s2, s2), s2);
    if (!FORCE) o.u = __fma_rn(__dmul_rn(P.eps4, s6), __dsub_rn(s6, 1.0), -P.ucut);
    o.t = __dmul_rn(__dmul_rn(P.eps24, s6), __fma_rn(-2.0, s6, 1.0));
    const double f = __dmul_rn(o.t, y);
    o.gx = __dmul_rn(rx, f);
    o.gy = __dmul_rn(ry, f);
    o.gz = __dmul_rn(rz, f);
    return true;
}

// Second half kick v += F dt/2m (integrator.rs:49-55).  With sp.fused (NVE
// chunks) also the next step's first half kick and drift (integrator.rs:30-46)
// into the other position/mirror buffers -- the step kernel that follows only
// decides and rebuilds.  Same operations, in the same order, as the unfused
// kick and drift.  Returns the displacement since the last rebuild.
// FM: the mixed path's fused multiply-adds (a compile-time constant).
template <bool FM>
__device__ __forceinline__ float kick_and_drift(const Dev& d, const StepParams& sp, const RepDev* R,
                                                const float* tcs, int s, int ty, double fx, double fy,
                                                double fz) {
    const int N = d.ntot;
    constexpr bool fm = FM;
    const double c = sp.kick_c[ty];
    double vx = madd(d.vel[s], fx, c, fm);
    double vy = madd(d.vel[N + s], fy, c, fm);
    double vz = madd(d.vel[2 * N + s], fz, c, fm);
    float disp = 0.f;
    if (sp.fused) {
        vx = madd(vx, fx, c, fm);
        vy = madd(vy, fy, c, fm);
        vz = madd(vz, fz, c, fm);
        const double4_32a p = drift_wrap(d.pos[s], vx, vy, vz, sp.dt, R->box, fm);
        d.pos_next[s] = p;
        const int cl = d.cell[s] - R->cell_base;
        if (cl >= 0 && cl < R->nc[0] * R->nc[1] * R->nc[2]) {
            const float4 m = mirror_of(p, cl, *R, tcs + 3, fm);
            d.mir_next[s] = m;
            disp = mirror_disp(m, d.mir0[s], tcs);
        } else {
            atomicOr(d.err, E_CELLS);
        }
    }
    d.vel[s] = vx;
    d.vel[N + s] = vy;
    d.vel[2 * N + s] = vz;
    return disp;
}

// Largest displacement of the warp into the replica's running maximum.
__device__ __forceinline__ void note_displacement(const Dev& d, int r, float disp) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) disp = fmaxf(disp, __shfl_xor_sync(0xffffffffu, disp, off));
    if ((threadIdx.x & 31) == 0 && disp > 0.f) atomicMax(&d.rep[r].max_disp_bits, __float_as_uint(disp));
}

}  // namespace mdgb
