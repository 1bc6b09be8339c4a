// list_direct.cuh -- the direct Verlet-list build (every cell against its 27
// neighbour cells; k_build_list, kernels_list.cu) and the reference-order sort
// of a list, which the whole-chunk kernel of small systems (kernels_step.cu)
// uses too.
#pragma once
#include <type_traits>

#include "mdgb_internal.cuh"

namespace mdgb {

constexpr int LB_WIN = 1024;          // candidate stream positions held per window
constexpr int LB_MQ = LB_WIN / 32 + 1;  // mask row stride (odd: conflict-free columns)

// Per-warp shared memory in 32-bit words: candidate window, hit masks
// [own atom][chunk], own atoms (paired coordinates and types: 4 words each),
// the 27 cell shifts (float4).
constexpr int LB_WARP_WORDS = LB_WIN + 32 * LB_MQ + 32 * 4 + 27 * 4 + 4;
static_assert((LB_WIN + 32 * LB_MQ) % 4 == 0 && LB_WARP_WORDS % 4 == 0, "float4 alignment");

// Bit-matrix transpose over a warp: lane l holds row l (bit c = entry (l, c));
// afterwards lane c holds column c (bit l = entry (l, c)).  Five butterfly
// stages; stage j swaps the off-diagonal j x j blocks of every 2j x 2j block.
__device__ __forceinline__ uint32_t warp_transpose32(uint32_t x, int lane) {
    const uint32_t masks[5] = {0x0000FFFFu, 0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
    for (int st = 0; st < 5; ++st) {
        const int j = 16 >> st;
        const uint32_t m = masks[st];
        const uint32_t p = __shfl_xor_sync(0xffffffffu, x, j);
        x = (lane & j) ? ((x & ~m) | ((p >> j) & m)) : ((x & m) | ((p & m) << j));
    }
    return x;
}

// Two own atoms (paired coordinates) against one candidate: r^2 - rlist^2
// for each, negative when the pair is listed.  The sign is exact: the chain
// ends in one rounding of a value that is zero only when r^2 = rlist^2.
__device__ __forceinline__ f2_t pair_r2m(f2_t jx2, f2_t jy2, f2_t jz2, float4 A, float2 Z, f2_t nrl2) {
    const f2_t ex = sub2(jx2, f2(A.x, A.y)), ey = sub2(jy2, f2(A.z, A.w)), ez = sub2(jz2, f2(Z.x, Z.y));
    return fma2(ez, ez, fma2(ey, ey, fma2(ex, ex, nrl2)));
}

// Hit bits of one candidate against the own atoms (bit i: own atom i).  One
// type: the own atoms in descending order, each sign bit shifted in from the
// bottom (one funnel shift per test).  Several types: the reference's t1 <=
// t2 loop (potential.rs:171-172) also decides, separately for each side --
// fwd: own atom i lists the candidate (type_j >= type_i); bwd: the candidate
// lists own atom i (type_i >= type_j).
template <bool SINGLE, bool BWD>
__device__ __forceinline__ void own_hits(f2_t jx2, f2_t jy2, f2_t jz2, int tj, int cpc4, const float4* own_xy,
                                         const float2* own_z, const int* own_t, f2_t nrl2, uint32_t& fwd,
                                         uint32_t& bwd) {
    fwd = 0u;
    bwd = 0u;
    if (SINGLE) {
        for (int i = cpc4 - 4; i >= 0; i -= 4) {
#pragma unroll
            for (int u = 2; u >= 0; u -= 2) {
                const f2_t h = pair_r2m(jx2, jy2, jz2, own_xy[(i + u) >> 1], own_z[(i + u) >> 1], nrl2);
                fwd = __funnelshift_l((unsigned)(h >> 32), fwd, 1);   // own atom i + u + 1
                fwd = __funnelshift_l((unsigned)h, fwd, 1);           // own atom i + u
            }
        }
        bwd = fwd;
    } else {
        for (int i = 0; i < cpc4; i += 4) {
            const uint32_t b0 = 1u << i;
#pragma unroll
            for (int u = 0; u < 4; u += 2) {
                const f2_t h = pair_r2m(jx2, jy2, jz2, own_xy[(i + u) >> 1], own_z[(i + u) >> 1], nrl2);
                const bool h0 = f2_lo(h) < 0.f, h1 = f2_hi(h) < 0.f;
                const int t0 = own_t[i + u], t1 = own_t[i + u + 1];
                if (h0 & (tj >= t0)) fwd |= b0 << u;
                if (h1 & (tj >= t1)) fwd |= b0 << (u + 1);
                if (BWD) {
                    if (h0 & (t0 >= tj)) bwd |= b0 << u;
                    if (h1 & (t1 >= tj)) bwd |= b0 << (u + 1);
                }
            }
        }
    }
}

// Lists of a reference-order engine into the reference's order (ascending
// rank; one thread per atom there, so entry k of atom s lies rn words after
// entry k - 1).  The warp takes its 32 atoms (lane = atom s0 + lane with n
// entries) one after the other: lane l holds entries l, l + 32, ... of the
// list, finds each one's place by counting the smaller keys, broadcast one
// after the other, and stores it there.  An insertion sort per lane in global
// memory took 1.5 ms for 6,912 atoms (a dependent load, rank gather and store
// per move); this one is bound by its instructions (7 per key and round of
// 32): a frame of 111,360 atoms 8.2 -> 5.0 ms, ten saved steps of 23,256 atoms
// 9.4 -> 7.6 ms.  Lists of more than 128 entries keep the insertion sort.
constexpr int SORT_PER_LANE = 4;

static __device__ __noinline__ void sort_lists_by_rank(const Dev& d, int s0, int n, long long rbeg, int rn) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    __syncwarp();   // any lane may have written any entry (k_steps: one atom's list by all 32)
    if (n > 32 * SORT_PER_LANE) sort_list_by_rank(d, s0 + lane, n, 1, rbeg, rn);
    __syncwarp();
    unsigned todo = __ballot_sync(FULL, n > 1 && n <= 32 * SORT_PER_LANE);
    while (todo) {
        const int a = __ffs(todo) - 1;
        todo &= todo - 1u;
        const int na = __shfl_sync(FULL, n, a);
        uint32_t* list = d.nbr + list_index(s0 + a, 0, 1, rbeg, rn, d.cap);
        uint32_t e[SORT_PER_LANE];
        int key[SORT_PER_LANE], place[SORT_PER_LANE];
#pragma unroll
        for (int q = 0; q < SORT_PER_LANE; ++q) {
            const int k = lane + 32 * q;
            e[q] = k < na ? list[(size_t)k * rn] : 0u;
        }
#pragma unroll
        for (int q = 0; q < SORT_PER_LANE; ++q) {
            key[q] = lane + 32 * q < na ? __ldcg(d.rank + (e[q] & IDX_MASK)) : 0x7FFFFFFF;
            place[q] = 0;
        }
        __syncwarp();   // every entry is read before any is stored
        auto rounds = [&](auto nq_) {
            constexpr int NQ = decltype(nq_)::value;
#pragma unroll
            for (int p = 0; p < NQ; ++p) {
                const int m = min(32, na - 32 * p);
                for (int k = 0; k < m; ++k) {
                    const int other = __shfl_sync(FULL, key[p], k);
#pragma unroll
                    for (int q = 0; q < NQ; ++q) place[q] += other < key[q] ? 1 : 0;
                }
            }
        };
        if (na <= 32) rounds(std::integral_constant<int, 1>{});
        else if (na <= 64) rounds(std::integral_constant<int, 2>{});
        else if (na <= 96) rounds(std::integral_constant<int, 3>{});
        else rounds(std::integral_constant<int, 4>{});
#pragma unroll
        for (int q = 0; q < SORT_PER_LANE; ++q)
            if (lane + 32 * q < na) list[(size_t)place[q] * rn] = e[q];
        __syncwarp();
    }
}

// The direct build: every cell against the stream of its 27 neighbour cells.
// all: every rebuilding replica (else those the paired build does not take).
// WARPS: warps per block.
template <bool SINGLE, int WARPS>
__device__ __forceinline__ void list_direct(const Dev& d, uint32_t* lb_smem, bool all) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    uint32_t* cand = lb_smem + (size_t)wib * LB_WARP_WORDS;
    uint32_t* masks = cand + LB_WIN;
    // own atoms in pairs for the paired FP32 instructions: (x_2p, x_2p+1, y_2p,
    // y_2p+1), (z_2p, z_2p+1), and their types
    float4* own_xy = reinterpret_cast<float4*>(masks + 32 * LB_MQ);
    float2* own_z = reinterpret_cast<float2*>(own_xy + 16);
    int* own_t = reinterpret_cast<int*>(own_z + 16);
    float4* tab = reinterpret_cast<float4*>(own_t + 32);
    const int cap = d.cap;
    const int gw = blockIdx.x * WARPS + wib, nw = gridDim.x * WARPS;
    // the cells of the rebuilding replicas this build takes (the step
    // kernel's work list: all, or those before position rb[1])
    const int m = d.rb[0], nwork = rb_cell_off(d)[all ? m : d.rb[1]];
    for (int wi = gw; wi < nwork; wi += nw) {
        const int i = rb_locate(rb_cell_off(d), m, wi);
        const int r = rb_rep(d)[i];
        const RepDev* W = d.rep + r;
        if (W->mode != MODE_CELLS) continue;
        const int c = W->cell_base + wi - rb_cell_off(d)[i];
        const float rl = (float)(W->rlist * (1.0 + 1e-5));
        const f2_t nrl2 = f2(-(rl * rl), -(rl * rl));
        const int nc[3] = {W->nc[0], W->nc[1], W->nc[2]};
        const int base = W->cell_base;
        const int local = c - base;
        if (local >= nc[0] * nc[1] * nc[2]) continue;   // a guard: the work list holds the grid only
        const long long rbeg = W->begin;
        const int rn = W->n, tpa = W->tpa;
        const int ib = d.cell_start[c], in = d.cell_count[c];
        if (ib < rbeg || ib + in > rbeg + rn) {
            if (lane == 0) atomicOr(d.err, E_CELLS);
            continue;
        }
        if (in == 0) continue;
        int ox, oy, oz;
        decode_cell(local, nc, ox, oy, oz);
        __syncwarp();
        // lane k < 27: neighbour cell with shift code k
        int nb_start = 0, nb_cnt = 0;
        if (lane < 27) {
            const int dx = lane % 3 - 1, dy = (lane / 3) % 3 - 1, dz = lane / 9 - 1;
            int x = ox + dx; x = x < 0 ? x + nc[0] : (x >= nc[0] ? x - nc[0] : x);
            int y = oy + dy; y = y < 0 ? y + nc[1] : (y >= nc[1] ? y - nc[1] : y);
            int z = oz + dz; z = z < 0 ? z + nc[2] : (z >= nc[2] ? z - nc[2] : z);
            const int cj = base + (x * nc[1] + y) * nc[2] + z;
            nb_start = d.cell_start[cj];
            nb_cnt = d.cell_count[cj];
            if (nb_start < rbeg || nb_start + nb_cnt > rbeg + rn) {
                atomicOr(d.err, E_CELLS);
                nb_cnt = 0;
            }
            tab[lane] = make_float4((float)dx * dbl_to_flt_rn(W->cs[0]), (float)dy * dbl_to_flt_rn(W->cs[1]),
                                    (float)dz * dbl_to_flt_rn(W->cs[2]), 0.f);
        }
        int incl = nb_cnt;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int v = __shfl_up_sync(FULL, incl, off);
            if (lane >= off) incl += v;
        }
        const int nb_off = incl - nb_cnt;
        const int total = __shfl_sync(FULL, incl, 31);
        const int self_off = __shfl_sync(FULL, nb_off, CODE_ZERO);   // the own cell's segment
        int cmax = 0;
        for (int g = 0; g < in; g += 32) {
            const int cpc = min(32, in - g);
            const int s = ib + g + lane;
            const bool own = lane < cpc;
            __syncwarp();
            // rows past the cell's atoms (up to a multiple of 4) sit far away: no hits
            {
                const float4 xo = own ? d.mir[s] : make_float4(1e18f, 1e18f, 1e18f, __int_as_float(0x7fffffff));
                float* oxy = reinterpret_cast<float*>(own_xy) + ((lane >> 1) << 2) + (lane & 1);
                oxy[0] = xo.x;
                oxy[2] = xo.y;
                reinterpret_cast<float*>(own_z)[lane] = xo.z;
                own_t[lane] = type_of(xo);
            }
            const int cpc4 = (cpc + 3) & ~3;
            const int pself = self_off + g + lane;   // stream position of the atom itself
            int cnt = 0;
            // running output position: entry cnt of atom s is rowp[col],
            // rowp = segment + (cnt / tpa) * n * tpa + (s - begin) * tpa, col = cnt % tpa
            uint32_t* rowp = d.nbr + (size_t)cap * (size_t)rbeg + (size_t)(s - rbeg) * (size_t)tpa;
            const size_t rowstride = (size_t)rn * (size_t)tpa;
            int col = 0;
            for (int w0 = 0; w0 < total; w0 += LB_WIN) {
                const int wn = min(LB_WIN, total - w0);
                const int nq = (wn + 31) >> 5;
                __syncwarp();
                // lane k < 27 writes neighbour cell k's run of the window
                if (lane < 27) {
                    const int lo = max(nb_off, w0), hi = min(nb_off + nb_cnt, w0 + wn);
                    const uint32_t tag = (uint32_t)lane << IDX_BITS;
                    for (int p = lo; p < hi; ++p) cand[p - w0] = (uint32_t)(nb_start + p - nb_off) | tag;
                }
                __syncwarp();
                uint32_t e_n = 0u;
                float4 x_n = make_float4(0.f, 0.f, 0.f, 0.f);
                if (lane < wn) {
                    e_n = cand[lane];
                    x_n = __ldg(d.mir + (e_n & IDX_MASK));
                }
                for (int q = 0; q < nq; ++q) {
                    const bool valid = (q << 5) + lane < wn;
                    const float4 sh = tab[e_n >> IDX_BITS];
                    const float jx = x_n.x + sh.x, jy = x_n.y + sh.y, jz = x_n.z + sh.z;
                    const f2_t jx2 = f2(jx, jx), jy2 = f2(jy, jy), jz2 = f2(jz, jz);
                    const int tj = type_of(x_n);
                    if (((q + 1) << 5) + lane < wn) {   // next chunk in flight
                        e_n = cand[((q + 1) << 5) + lane];
                        x_n = __ldg(d.mir + (e_n & IDX_MASK));
                    }
                    // bit i of `mine`: own atom i lists this lane's candidate
                    uint32_t mine, unused;
                    own_hits<SINGLE, false>(jx2, jy2, jz2, tj, cpc4, own_xy, own_z, own_t, nrl2, mine, unused);
                    if (!valid) mine = 0u;
                    // 32x32 bit transpose across the warp: lane i gets bit k set when
                    // candidate k of the chunk hits own atom i
                    mine = warp_transpose32(mine, lane);
                    masks[lane * LB_MQ + q] = mine;
                }
                __syncwarp();
                // expansion: pass t appends entry t of every lane's atom, so the
                // stores of a pass land side by side
                uint32_t* myrow = masks + lane * LB_MQ;
                int tot = 0;
                if (own) {
                    const int ps = pself - w0;
                    if (ps >= 0 && ps < wn) myrow[ps >> 5] &= ~(1u << (ps & 31));
                    for (int q = 0; q < nq; ++q) tot += __popc(myrow[q]);
                }
                // entries this window writes (the rest of an overflowing list is
                // only counted)
                const int lim = max(0, min(tot, cap - cnt));
                int lmax = lim;
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) lmax = max(lmax, __shfl_xor_sync(FULL, lmax, off));
                if (tpa == 1) {
                    // masks bit-reversed: the next entry is the highest set bit
                    // (one find-leading-one), candidate 32 q + 31 - p
                    uint32_t mr = own ? __brev(myrow[0]) : 0u;
                    int qb = 31;
#pragma unroll 2
                    for (int t = 0; t < lmax; ++t) {
                        if (t < lim) {
                            while (mr == 0u) {   // t < lim <= tot: a set bit remains
                                qb += 32;
                                mr = __brev(myrow[qb >> 5]);
                            }
                            const int p = 31 - __clz(mr);
                            mr ^= 1u << p;
                            rowp[(size_t)t * rowstride] = cand[qb - p];
                        }
                    }
                    rowp += (size_t)tot * rowstride;
                } else {
                    uint32_t m = own ? myrow[0] : 0u;
                    int q = 0;
                    for (int t = 0; t < lmax; ++t) {
                        if (t < lim) {
                            while (m == 0u) m = myrow[++q];
                            const int k = __ffs(m) - 1;
                            m &= m - 1u;
                            rowp[col] = cand[(q << 5) + k];
                            if (++col == tpa) { col = 0; rowp += rowstride; }
                        }
                    }
                    // entries counted past the capacity are never written: no
                    // further window writes either (lim is 0 from here on)
                }
                cnt += tot;
            }
            if (own) {
                const int nfill = min(cnt, cap);
                d.nn[s] = nfill;
                if (cnt > cap) {
                    atomicOr(d.err, E_NLIST);
                    atomicMax(d.max_needed, cnt);
                }
            }
            if (d.refmode) sort_lists_by_rank(d, ib + g, own ? min(cnt, cap) : 0, rbeg, rn);
            cmax = max(cmax, cnt);
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) cmax = max(cmax, __shfl_xor_sync(FULL, cmax, off));
        if (lane == 0 && cmax > 0) atomicMax(&d.rep[r].max_nn, cmax);
    }
}

}  // namespace mdgb
