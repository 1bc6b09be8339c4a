// force_common.cuh -- device helpers of the force kernels (kernels_force.cu,
// kernels_pairs.cu).
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

// The reference's FP64 displacement and distance (potential.rs:181-201).
__device__ __forceinline__ double ref_distance(const double4_32a pi, const double4_32a pj, const double* box,
                                               double& rx, double& ry, double& rz) {
    rx = __dsub_rn(pj.x, pi.x);
    ry = __dsub_rn(pj.y, pi.y);
    rz = __dsub_rn(pj.z, pi.z);
    const double hx = 0.5 * box[0], hy = 0.5 * box[1], hz = 0.5 * box[2];
    if (rx < -hx) rx = __dadd_rn(rx, box[0]); else if (rx > hx) rx = __dsub_rn(rx, box[0]);
    if (ry < -hy) ry = __dadd_rn(ry, box[1]); else if (ry > hy) ry = __dsub_rn(ry, box[1]);
    if (rz < -hz) rz = __dadd_rn(rz, box[2]); else if (rz > hz) rz = __dsub_rn(rz, box[2]);
    const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(rx, rx), __dmul_rn(ry, ry)), __dmul_rn(rz, rz));
    return __dsqrt_rn(r2);
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
