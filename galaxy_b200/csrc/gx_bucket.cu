// gx_bucket.cu -- the fused particle pass of the mixed-precision step on a
// bucketed particle store.
//
// One step of the reference (step.f:135-290) is, per particle, grdacc
// (grdacc.f:189-266: weights of the current cell, gather of the fields at
// its corners), stpgrp (stpgrp.f:26-32: v += a, x += v) and massgn
// (massgn.f:68-89, 140-172: the weights of the new cell scatter-added into
// the mesh), then scaled (scaled.f:89-92).  Here that is one kernel per
// step, k_push_bkt, over a store that keeps the particles grouped by the
// ring-plane row of their cell:
//
//   * bq[b] holds one segment of slots per row (row nrow: off the grid);
//     segment r starts at bk_base[b][r] and has bk_cap[b][r] slots, planned
//     from the previous step's row counts with 1/8 + 16 slots of slack, so
//     that a particle that changes row usually finds room in its new row's
//     segment.  A particle that does not is appended to an overflow area
//     after the segments (capacity: every particle), so no particle is ever
//     dropped, and the next plan gives its row the room.
//   * k_push_bkt walks work items (up to BK_ITEM particles of one row's
//     segment, or of the overflow area) in the input buffer, and for each
//     particle interpolates the field, moves it, computes its new cell
//     exactly as the reference does (bit-exact keys), writes it into the
//     segment of its new row in the output buffer (warp-aggregated slot
//     atomics), and adds its 4 / 8 CIC weights as 2^-20 fixed-point
//     integers: into unsigned 32-bit shared-memory bins over the window of
//     rows around the item's row (4 rings, and 4 planes in 3D: every cell a
//     particle of the row can reach moving less than a cell), or, for
//     corners outside it (and the rare negative weight), straight into the
//     int64 mesh accumulator.  The bins are flushed into the accumulator
//     (nonzero bins only) after each item.  A bin cannot wrap: the linear
//     weights that reach it are >= 0 and <= 1 + 1e-4, each particle adds at
//     most one to a bin, and an item holds at most 4095 particles, so a bin
//     stays below 4095 (2^20 + 105) < 2^32.
//   * k_bk_plan (one CTA) turns the output buffer's row counts into its
//     work items, the next output buffer's segments and the active ring
//     range (jrad, krad); k_mass_convert turns the accumulator into the mass
//     array (x pmass) and clears it.
//
// Integer sums do not depend on their order, so the mass array is the same
// integers, converted the same way, as the sort-based deposit of
// gx_deposit.cu: the fused path is bitwise identical to it, whatever order
// the atomics resolve in.  A particle's record carries its load index;
// gx_dense() writes the store back to the n contiguous SoA particles of
// pbuf[cur] for the entry points that walk them that way (getacc, tmcent,
// icheck, the adjoint); unload writes the records straight from the store
// in load order, and masset deposits from the store with the same kernel
// run without the field and the move.
#include <limits.h>

#include <algorithm>

#include "gx_common.cuh"

#define BK_FIXQ 1048576.0f  // 2^20: the fixed-point quantum of gx_deposit.cu
// items with fewer particles add straight into the mesh (the flush of a window
// costs about as much; 32 to 256 are within 2 % at 170 to 310 particles a row)
#define BK_SPARSE 128
// items with at least this many particles copy the field rows of their cells
// (4 rows in 3D, 2 in 2D) into shared memory and gather there: a warp's gather
// touches 29 sectors of the first-level cache, in shared memory it takes 11
// wavefronts (10M particles, 3D: the pass 282 -> 262 us; 3M in 2D and short
// items: no change)
#define BK_STAGE 512
// The staged rows grow with the spokes, and past some width they cost CTAs: their
// shared memory is reserved where the SM keeps its CTAs with it, or where the
// particles suffice for items that use it, BK_STAGE_ROW a row on average (they
// crowd a part of the rows).  3D steps on 64 rings x 45 planes, us, rows reserved
// and not: 100k particles (35 a row) 86 and 79 at 256 spokes quadratic, 81 and 76
// at 512 linear; 500k (173 a row) 115 and 123, 110 and 114.
#define BK_STAGE_ROW 64
// Quadratic grids with more spokes than let two CTAs of staged rows onto an SM
// (256 B a spoke each) take the sorted path: fused and sorted steps of 500k and 3M
// particles 115 and 278 against 131 and 302 us at 256 spokes, 148 and 341 against
// 151 and 338 at 384, 160 and 355 against 159 and 347 at 444; with one CTA per SM
// at 512 213 and 526 against 167 and 367 (179 and 372 without the rows).
#define BK_QUAD_NA 444
#define BK_CTASLOT 768      // 2D items with at least this many take their slots by CTA
#define BK_THREADS 256
#define PLAN_THREADS 512
#define PLAN_ROWS 8         // rows per plan thread per pass
#ifndef BK_MINB
#define BK_MINB 5           // resident CTAs per SM the register budget is set for
#endif

__device__ __forceinline__ void red_add_s64(unsigned long long* a, int v) {
    atomicAdd(a, (unsigned long long)(long long)v);  // two's complement sum
}

// round(w 2^20) to the nearest integer, ties to even, for |w 2^20| < 2^22:
// adding 1.5 2^23 leaves the rounded integer in the low mantissa bits (the
// product by a power of two is exact, so one FMA rounds once, exactly as
// __float2int_rn(w * 2^20) does), on the FMA pipe instead of a conversion
__device__ __forceinline__ int bk_fix(float w) {
    return __float_as_int(fmaf(w, BK_FIXQ, 12582912.0f)) - 0x4B400000;
}

// ---------------------------------------------------------------------------
// block-wide exclusive scan of two ints (PLAN_THREADS threads)
__device__ __forceinline__ void plan_scan2(int a, int b, int& ea, int& eb, int& ta, int& tb) {
    __shared__ int wa[PLAN_THREADS / 32], wb[PLAN_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int xa = a, xb = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int ya = __shfl_up_sync(0xffffffffu, xa, o), yb = __shfl_up_sync(0xffffffffu, xb, o);
        if (lane >= o) {
            xa += ya;
            xb += yb;
        }
    }
    if (lane == 31) {
        wa[warp] = xa;
        wb[warp] = xb;
    }
    __syncthreads();
    constexpr int NWP = PLAN_THREADS / 32;  // warps (<= 32): lanes past them hold zeros
    static_assert(NWP <= 32, "one warp scans the warp totals");
    if (warp == 0) {
        int va = (lane < NWP) ? wa[lane] : 0, vb = (lane < NWP) ? wb[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int ya = __shfl_up_sync(0xffffffffu, va, o), yb = __shfl_up_sync(0xffffffffu, vb, o);
            if (lane >= o) {
                va += ya;
                vb += yb;
            }
        }
        if (lane < NWP) {
            wa[lane] = va;
            wb[lane] = vb;
        }
    }
    __syncthreads();
    const int pa = warp ? wa[warp - 1] : 0, pb = warp ? wb[warp - 1] : 0;
    ea = pa + xa - a;
    eb = pb + xb - b;
    ta = wa[NWP - 1];
    tb = wb[NWP - 1];
    __syncthreads();
}

// The plan of one step, one CTA:
//  * with fill_o: the work items of the buffer just written (fill_o, cap_o,
//    base_o, overflow count *ovf_o at slot ovf_base; each item: row, first
//    slot, end slot, ring of the row), and ctl[0] = items, ctl[1] = 0 (the
//    work counter);
//  * the segments of the buffer to be written next from the row counts
//    want: cap_n = want + want/8 + 16 (0 for empty rows), base_n their
//    exclusive sum; its fill counters and overflow count cleared.
// The row tables are padded with zeros to a multiple of PLAN_THREADS x
// PLAN_ROWS entries, so that every thread moves its eight consecutive rows
// with two 16-byte loads per table, all issued before they are used.
__device__ __forceinline__ void ld8(const int32_t* __restrict__ p, int r0, int* v) {
    const int4 a = __ldg(reinterpret_cast<const int4*>(p + r0));
    const int4 b = __ldg(reinterpret_cast<const int4*>(p + r0 + 4));
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void st8(int32_t* __restrict__ p, int r0, const int* v) {
    reinterpret_cast<int4*>(p + r0)[0] = make_int4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<int4*>(p + r0)[1] = make_int4(v[4], v[5], v[6], v[7]);
}
static_assert(PLAN_ROWS == 8, "ld8 / st8 move eight rows");

__global__ void __launch_bounds__(PLAN_THREADS) k_bk_plan(
    int nrow1, int ngz, const int32_t* __restrict__ fill_o, const int32_t* __restrict__ cap_o,
    const int32_t* __restrict__ base_o, const int32_t* __restrict__ ovf_o, int64_t ovf_base,
    int4* __restrict__ items, int32_t* __restrict__ ctl,
    const int32_t* __restrict__ want, int32_t* __restrict__ cap_n, int32_t* __restrict__ base_n,
    int32_t* __restrict__ fill_n, int32_t* __restrict__ ovf_n, int item) {
    int carry_cap = 0, carry_it = 0;
    for (int c0 = 0; c0 < nrow1; c0 += PLAN_THREADS * PLAN_ROWS) {
        const int r0 = c0 + threadIdx.x * PLAN_ROWS;
        int wv[PLAN_ROWS], fv[PLAN_ROWS], cv[PLAN_ROWS], bv[PLAN_ROWS];
        ld8(want, r0, wv);
        if (fill_o) {
            ld8(fill_o, r0, fv);
            ld8(cap_o, r0, cv);
            ld8(base_o, r0, bv);
        }
        int capv[PLAN_ROWS], nit[PLAN_ROWS], val[PLAN_ROWS], zero[PLAN_ROWS];
        int scap = 0, snit = 0;
#pragma unroll
        for (int k = 0; k < PLAN_ROWS; k++) {
            const int w = wv[k];
            zero[k] = 0;
            capv[k] = w + (w >> 3) + (w > 0 ? 16 : 0);
            val[k] = nit[k] = 0;
            if (fill_o) {
                val[k] = min(fv[k], cv[k]);
                nit[k] = (val[k] + item - 1) / item;
            }
            scap += capv[k];
            snit += nit[k];
        }
        int ecap, eit, tcap, tit;
        plan_scan2(scap, snit, ecap, eit, tcap, tit);
        ecap += carry_cap;
        eit += carry_it;
        int basev[PLAN_ROWS];
#pragma unroll
        for (int k = 0; k < PLAN_ROWS; k++) {
            basev[k] = ecap;
            ecap += capv[k];
        }
        st8(cap_n, r0, capv);
        st8(base_n, r0, basev);
        st8(fill_n, r0, zero);
        if (fill_o) {
#pragma unroll
            for (int k = 0; k < PLAN_ROWS; k++) {
                const int ring = (r0 + k) / ngz;
                for (int q = 0; q < nit[k]; q++)
                    items[eit + q] = make_int4(r0 + k, bv[k] + q * item, bv[k] + min((q + 1) * item, val[k]), ring);
                eit += nit[k];
            }
        }
        carry_cap += tcap;
        carry_it += tit;
    }
    if (fill_o && threadIdx.x == 0) {
        const int ov = *ovf_o;
        int it = carry_it;
        for (int q = 0; q * item < ov; q++, it++)
            items[it] = make_int4(-1, (int)ovf_base + q * item, (int)ovf_base + min((q + 1) * item, ov), 0);
        ctl[0] = it;
        ctl[1] = 0;
    }
    if (threadIdx.x == 0) *ovf_n = 0;
}

// ---------------------------------------------------------------------------
// slot of a particle bound for row rk in the output buffer: warp-aggregated
// atomics on the row's fill counter; past the segment's capacity, the
// overflow area (all 32 lanes call; act false lanes take no slot)
__device__ __forceinline__ int64_t bk_slot(bool act, uint32_t rk, const int32_t* __restrict__ cap_o,
                                           const int32_t* __restrict__ base_o, int32_t* __restrict__ fill_o,
                                           int32_t* __restrict__ ovf_o, int64_t ovf_base) {
    const unsigned lane = threadIdx.x & 31;
    const uint32_t am = __ballot_sync(0xffffffffu, act);
    const uint32_t peers = __match_any_sync(0xffffffffu, act ? rk : 0xffffffffu) & am;
    const int leader = __ffs(peers) - 1;
    int b = 0;
    if (act && (int)lane == leader) b = atomicAdd(fill_o + rk, __popc(peers));
    b = __shfl_sync(0xffffffffu, b, leader < 0 ? 0 : leader);
    const int slot = b + __popc(peers & lanemask_lt());
    int64_t dst = -1;
    bool ovf = false;
    if (act) {
        if (slot < __ldg(cap_o + rk)) dst = (int64_t)__ldg(base_o + rk) + slot;
        else ovf = true;
    }
    const uint32_t om = __ballot_sync(0xffffffffu, ovf);
    if (om) {
        const int ol = __ffs(om) - 1;
        int ob = 0;
        if ((int)lane == ol) ob = atomicAdd(ovf_o, __popc(om));
        ob = __shfl_sync(0xffffffffu, ob, ol);
        if (ovf) dst = ovf_base + ob + __popc(om & lanemask_lt());
    }
    return dst;
}

// A particle of the bucketed store is one record: its NP floats (x, y[, z],
// vx, vy[, vz][, the compensated low parts]) then its load index as float
// bits, zero-padded to R float4 words.  The first two words of record s
// are bytes 32 s .. 32 s + 31 (moved with one 32-byte ld/st.v8 access, so a
// warp's loads of consecutive records are contiguous and each store writes
// a whole sector); a third word (the compensated 3D records, R = 3) sits in
// a plane of its own after them, at word 2 bcap + s.
template <int NP>
struct Rec {
    static constexpr int R = (NP + 1 + 3) / 4;
    static_assert(R >= 2 && R <= 3, "records of 5 to 12 floats");
};

__device__ __forceinline__ void ld8f(const float4* p, float* w) {
    asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(w[0]), "=f"(w[1]), "=f"(w[2]), "=f"(w[3]), "=f"(w[4]), "=f"(w[5]), "=f"(w[6]), "=f"(w[7])
                 : "l"(p));
}
__device__ __forceinline__ void st8f(float4* p, const float* w) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(w[0]), "f"(w[1]), "f"(w[2]),
                 "f"(w[3]), "f"(w[4]), "f"(w[5]), "f"(w[6]), "f"(w[7])
                 : "memory");
}

template <int NP>
__device__ __forceinline__ void rec_load(const float4* __restrict__ Q, int64_t bcap, int64_t s, float* P,
                                         int32_t& o) {
    constexpr int R = Rec<NP>::R;
    float w[4 * R];
    ld8f(Q + 2 * s, w);
    if (R == 3) {
        const float4 v = __ldg(Q + 2 * bcap + s);
        w[8] = v.x;
        w[9] = v.y;
        w[10] = v.z;
        w[11] = v.w;
    }
#pragma unroll
    for (int k = 0; k < NP; k++) P[k] = w[k];
    o = __float_as_int(w[NP]);
}

template <int NP>
__device__ __forceinline__ void rec_store(float4* __restrict__ Q, int64_t bcap, int64_t s, const float* P,
                                          int32_t o) {
    constexpr int R = Rec<NP>::R;
    float w[4 * R];
#pragma unroll
    for (int k = 0; k < 4 * R; k++) w[k] = (k < NP) ? P[k] : 0.f;
    w[NP] = __int_as_float(o);
    st8f(Q + 2 * s, w);
    if (R == 3) Q[2 * bcap + s] = make_float4(w[8], w[9], w[10], w[11]);
}

// The fused particle pass of one step.  Persistent CTAs take work items from
// a counter.  bins: int64 [WROWS][na] over the item's window, zero between
// items.  Window of an item of row (ir, iz): rings ir - 1 .. ir + 2 and, in
// 3D, planes iz - 1 .. iz + 2 (bin row 4 a + b for ring ir - 1 + a, plane
// iz - 1 + b); 2D: rows ir - 1 .. ir + 2.
// DEP: the deposit alone (masset on the bucketed store): the cell of each
// particle's current position, its weights into the bins and the mesh, the
// ring and plane range; no field, no move, the store is not rewritten
// Q: the quadratic scheme (3D): 27 nodes around the central one, the window 5
// rings x 5 planes around the item's row, so that the nodes of every cell a
// move of less than a cell reaches lie in it; four CTAs per SM (64 registers) up
// to 220 spokes, where the staged rows leave room for them.
// 500k particles on 64 x 128 x 45: 58.7 us, where the sorted path's push, sort,
// 27-weight deposit and combine took 75
template <int ND, bool COMP, bool DEP = false, bool Q = false>
__global__ void __launch_bounds__(BK_THREADS, Q ? 4 : BK_MINB) k_push_bkt(
    DevGeo g, const float4* __restrict__ Qin, float4* __restrict__ Qout, int64_t bcap,
    const float4* __restrict__ F,
    const int4* __restrict__ items, int32_t* __restrict__ ctl, const int32_t* __restrict__ cap_o,
    const int32_t* __restrict__ base_o, int32_t* __restrict__ fill_o, int32_t* __restrict__ ovf_o,
    int64_t ovf_base, unsigned long long* __restrict__ acc, int32_t* __restrict__ rg, int stage_min) {
    extern __shared__ __align__(16) uint32_t bins[];
    __shared__ int s_it[2];
    __shared__ int4 s_I[2];
    constexpr bool d3 = ND == 3;
    constexpr int WROWS = Q ? 25 : d3 ? 16 : 4;
    constexpr int W = Q ? 5 : 4, WLO = Q ? 2 : 1;  // window rings and planes, those below the item's row
    // 2D: an iteration's particles of each window row and their first slot
    // (double-buffered: the next iteration counts while this one stores)
    constexpr int OWN = 1;  // the item's row in its window
    __shared__ int s_cnt[2][4], s_slot[2][4];
    constexpr int NW = 2 * ND;
    const int na = g.na, ngz = d3 ? g.ngz : 1, nrow = g.nrow;
    const int nit = ctl[0];
    int rmin_l = 0x7fffffff, rmax_l = -1;  // ring range of this lane's new cells
    int zmin_l = 0x7fffffff, zmax_l = -1;  // and their plane range (3D)
    // the field rows of a cell of the item's row: (row, row + 1) and in 3D
    // (row + ngz, row + ngz + 1), na float4 each
    float4* fw = reinterpret_cast<float4*>(bins + (Q ? 28 : WROWS) * na);
    auto fetch = [&](int b) {
        const int it = atomicAdd(ctl + 1, 1);
        s_it[b] = it;
        if (it < nit) s_I[b] = items[it];
    };
    for (int i = threadIdx.x; i < WROWS * na; i += BK_THREADS) bins[i] = 0u;
    if (threadIdx.x == 0) fetch(0);
    if (!d3 && threadIdx.x < 8) (&s_cnt[0][0])[threadIdx.x] = 0;
    __syncthreads();
    int ph = 0;  // buffer of s_cnt, s_slot
    for (int b = 0;; b ^= 1) {
        if (s_it[b] >= nit) break;
        const int4 I = s_I[b];
        if (threadIdx.x == 0) fetch(b ^ 1);  // the next item, while this one runs
        const int row = I.x, s0 = I.y, s1 = I.z;
        const bool win = row >= 0 && row < nrow && (s1 - s0) >= BK_SPARSE;
        // ring and plane of the item's row (the plan stores the ring): the
        // window's origin is one below
        const int wir = I.w;
        const int wiz = d3 ? row - wir * ngz : 0;
        const bool cta = !d3 && (s1 - s0) >= BK_CTASLOT;
        bool stage = !DEP && row >= 0 && row + (d3 ? ngz : 0) + 1 < nrow && (s1 - s0) >= stage_min;
        if (Q) stage = stage && wir >= 1 && wir + 1 < g.nr && wiz >= 1 && wiz + 1 < ngz;
        if (Q && stage) {
            // the 3 x 3 rows around the central one
            for (int i = threadIdx.x; i < 9 * na; i += BK_THREADS) {
                const int q = i / na, j = i - q * na;
                fw[i] = __ldg(F + (size_t)(row + (q / 3 - 1) * ngz + (q % 3 - 1)) * na + j);
            }
            __syncthreads();
        } else if (stage) {
            const float4* f0 = F + (size_t)row * na;
#pragma unroll 4
            for (int i = threadIdx.x; i < (d3 ? 4 : 2) * na; i += BK_THREADS)
                fw[i] = __ldg(f0 + (d3 && i >= 2 * na ? i + (ngz - 2) * na : i));
            __syncthreads();
        }
        constexpr int NP = NW + (COMP ? ND : 0);
        constexpr int NQC = d3 ? 4 : 2;  // corner rows of a cell
        for (int b0 = s0; b0 < s1; b0 += BK_THREADS) {
            const int s = b0 + threadIdx.x;
            const bool act = s < s1;
            float P[NP];
            int32_t o = 0;
            CellW cn;
            cn.key = -1;
            uint32_t rk = 0;
            if (act) {
                rec_load<NP>(Qin, bcap, s, P, o);
                float &x = P[0], &y = P[1];
                float z = d3 ? P[2] : 0.f;
                if (!DEP) {
                    const CellW cw = gx_cell_t<false, ND>(g, x, y, z, true);
                    float ax, ay, az, ph;
                    if (Q && cw.key >= 0) {
                        // grdacc.f:267-299, in the order of gx_accel_cell_t
                        float f[3][3];
                        gx_factors27(cw, f);
                        const bool st = stage && cw.row == row;
                        const int jm = (cw.jt == 0) ? na - 1 : cw.jt - 1, jp = (cw.jt == na - 1) ? 0 : cw.jt + 1;
                        ax = ay = az = ph = 0.f;
#pragma unroll
                        for (int k = 0; k < 3; k++)
#pragma unroll
                            for (int j = 0; j < 3; j++) {
                                const int r = cw.row + (j - 1) + (k - 1) * ngz;
                                if (r < 0 || r >= nrow) continue;
                                float4 v[3];
                                if (st) {
                                    const float4* p = fw + (3 * k + j) * na;
                                    v[0] = p[jm];
                                    v[1] = p[cw.jt];
                                    v[2] = p[jp];
                                } else {
                                    const float4* p = F + (size_t)r * na;
                                    v[0] = __ldg(p + jm);
                                    v[1] = __ldg(p + cw.jt);
                                    v[2] = __ldg(p + jp);
                                }
#pragma unroll
                                for (int i = 0; i < 3; i++) {
                                    const float w = 0.125f * f[0][i] * f[1][j] * f[2][k];
                                    ax += v[i].x * w;
                                    ay += v[i].y * w;
                                    az += v[i].z * w;
                                }
                            }
                        gx_rigid_force(g, x, y, z, ax, ay, az, ph);
                    } else if (!Q && stage && cw.key >= 0 && cw.row == row) {
                        // the common case: the corners from the staged rows
                        // (in the order of gx_accel_cell_t)
                        float w[8];
                        gx_weights<ND>(g, cw, w);
                        const int j0 = cw.jt, j1 = (cw.jt == na - 1) ? 0 : cw.jt + 1;
                        ax = ay = az = ph = 0.f;
#pragma unroll
                        for (int q = 0; q < NQC; q++) {
                            const float4 a = fw[q * na + j0], c = fw[q * na + j1];
                            ax += a.x * w[2 * q];
                            ay += a.y * w[2 * q];
                            if (d3) az += a.z * w[2 * q];
                            ax += c.x * w[2 * q + 1];
                            ay += c.y * w[2 * q + 1];
                            if (d3) az += c.z * w[2 * q + 1];
                        }
                        gx_rigid_force(g, x, y, z, ax, ay, az, ph);
                    } else {
                        gx_accel_cell_t<Q, ND>(g, F, cw, x, y, z, ax, ay, az, ph);
                    }
                    float& vx = P[ND];
                    float& vy = P[ND + 1];
                    vx += ax;
                    vy += ay;
                    if (d3) P[ND + 2] += az;
                    if (COMP) {
                        gx_comp_add(x, P[NW], vx);
                        gx_comp_add(y, P[NW + 1], vy);
                        if (d3) gx_comp_add(P[2], P[NW + 2], P[ND + 2]);
                    } else {
                        x += vx;
                        y += vy;
                        if (d3) P[2] += P[ND + 2];
                    }
                    z = d3 ? P[2] : 0.f;
                }
                cn = gx_cell_t<true, ND>(g, x, y, z, false);
                rk = (cn.key >= 0) ? (uint32_t)cn.row : (uint32_t)nrow;
                if (cn.key >= 0) {
                    rmin_l = min(rmin_l, cn.ju);
                    rmax_l = max(rmax_l, cn.ju);
                    if (Q) {
                        // nodes in the planes below and above; below plane 0 lies
                        // the last plane of the ring below (flat offsets), where
                        // the next pass also reads for a cell just above plane
                        // 0's, whose interpolation cell may come out as plane 0
                        zmin_l = min(zmin_l, max(cn.iz - 1, 0));
                        const bool low = cn.iz == 0 || (cn.iz == 1 && cn.dz < g.eps_z);
                        zmax_l = max(zmax_l, low ? ngz - 1 : cn.iz);
                    } else if (d3) {
                        // a cell in the top plane (a spoke coordinate that
                        // rounded up to na moved it there) has its upper
                        // corners in plane 0 of the next ring
                        zmin_l = min(zmin_l, (cn.iz + 1 == ngz) ? 0 : cn.iz);
                        zmax_l = max(zmax_l, cn.iz);
                    }
                }
            }
            // the slot in the new row's segment, taken before the deposit so that
            // the latency of the fill counter's atomic overlaps it.  3D (rows by
            // the thousand): one atomic per warp and row.  2D: those serialise on
            // the few rows' counters, so a particle takes a rank among the
            // CTA's particles of its row in shared memory (those that stay in
            // the item's row by warp, the others one by one) and one thread per
            // window row takes the slots of all of them (3M particles on 128 x
            // 256, items of 1013: the pass 85 -> 73 us).  In 3D the barriers this
            // needs cost more than the atomics (10M: 262 -> 321 us), as they do
            // for short items.
            const unsigned lane = threadIdx.x & 31;
            uint32_t peers = 0;
            int leader = -1, bslot = 0, capr = 0, baser = 0, wi = -1, rank = 0;
            if (!DEP) {
                if (cta) {
                    if (act && cn.key >= 0 && row >= 0 && row < nrow && (unsigned)(cn.row - row + 1) < 4u)
                        wi = cn.row - row + 1;
                    const uint32_t st = __ballot_sync(0xffffffffu, wi == OWN);
                    if (st) {
                        const int l0 = __ffs(st) - 1;
                        if ((int)lane == l0) rank = atomicAdd(&s_cnt[ph][OWN], __popc(st));
                        rank = __shfl_sync(0xffffffffu, rank, l0) + __popc(st & lanemask_lt());
                    }
                    if (wi >= 0 && wi != OWN) rank = atomicAdd(&s_cnt[ph][wi], 1);
                }
                const bool far = act && wi < 0;
                if (!cta || __any_sync(0xffffffffu, far)) {
                    const uint32_t am = __ballot_sync(0xffffffffu, far);
                    peers = __match_any_sync(0xffffffffu, far ? rk : 0xffffffffu) & am;
                    leader = __ffs(peers) - 1;
                    if (far && (int)lane == leader) bslot = atomicAdd(fill_o + rk, __popc(peers));
                }
                if (act) {
                    capr = __ldg(cap_o + rk);
                    baser = __ldg(base_o + rk);
                }
                if (cta) {
                    __syncthreads();
                    if (threadIdx.x < 4) {
                        const int c = s_cnt[ph][threadIdx.x];
                        if (c) {
                            s_slot[ph][threadIdx.x] = atomicAdd(fill_o + row - 1 + (int)threadIdx.x, c);
                            s_cnt[ph][threadIdx.x] = 0;
                        }
                    }
                }
            }
            // the common case: every corner inside the window (the new cell
            // in its inner 3 x 3 rows, or 3 rows in 2D, no plane wrap, inside
            // the mesh) and no negative weight: eight shared-memory adds
            int va[8];
            bool fast = false;
            if (Q && act && cn.key >= 0) {
                // massgn.f:173-202
                float f[3][3];
                gx_factors27(cn, f);
                const int jm = (cn.jt == 0) ? na - 1 : cn.jt - 1, jp = (cn.jt == na - 1) ? 0 : cn.jt + 1;
                const int a0 = cn.ju - wir + WLO - 1, b0 = cn.iz - wiz + WLO - 1;  // window place of the lowest node
                // only the middle factors can be negative (at clamped indices)
                const bool in = win && (unsigned)a0 <= 2u && (unsigned)b0 <= 2u && cn.iz >= 1 && f[1][1] >= 0.f &&
                                f[2][1] >= 0.f;
                uint32_t* bw = bins + (in ? W * a0 + b0 : 0) * na;
#pragma unroll
                for (int k = 0; k < 3; k++)
#pragma unroll
                    for (int j = 0; j < 3; j++) {
                        int v[3];
#pragma unroll
                        for (int i = 0; i < 3; i++) v[i] = bk_fix(0.125f * f[0][i] * f[1][j] * f[2][k]);
                        if (in) {
                            uint32_t* br = bw + (W * k + j) * na;
                            atomicAdd(br + jm, (uint32_t)v[0]);
                            atomicAdd(br + cn.jt, (uint32_t)v[1]);
                            atomicAdd(br + jp, (uint32_t)v[2]);
                        } else {
                            const int r = cn.row + (j - 1) + (k - 1) * ngz;
                            if (r < 0 || r >= nrow) continue;  // outside the mesh: dropped, as massgn does
                            unsigned long long* ar = acc + (size_t)r * na;
                            if (v[0]) red_add_s64(ar + jm, v[0]);
                            if (v[1]) red_add_s64(ar + cn.jt, v[1]);
                            if (v[2]) red_add_s64(ar + jp, v[2]);
                        }
                    }
            }
            if (!Q && act && cn.key >= 0) {
                float w[8];
                gx_weights<ND>(g, cn, w);
                int neg = 0;
#pragma unroll
                for (int k = 0; k < 2 * NQC; k++) {
                    va[k] = bk_fix(w[k]);
                    neg |= va[k];
                }
                const int a0 = d3 ? cn.ju - wir + 1 : cn.row - row + 1;
                const int b0 = d3 ? cn.iz - wiz + 1 : 0;
                fast = win && neg >= 0 && (unsigned)a0 <= 2u && (unsigned)b0 <= 2u &&
                       (d3 ? (cn.iz + 1 < ngz && cn.ju + 1 < g.nr) : cn.row + 1 < nrow);
                if (fast) {
                    const int jt0 = cn.jt, jt1 = (cn.jt == na - 1) ? 0 : cn.jt + 1;
                    uint32_t* b = bins + (d3 ? 4 * a0 + b0 : a0) * na;
#pragma unroll
                    for (int q = 0; q < NQC; q++) {
                        // corner row q: + 1 (next plane / ring), + ngz (next ring): bin rows + 1, + 4
                        uint32_t* br = b + (d3 ? (q & 1) + 4 * (q >> 1) : q) * na;
                        atomicAdd(br + jt0, (uint32_t)va[2 * q]);
                        atomicAdd(br + jt1, (uint32_t)va[2 * q + 1]);
                    }
                }
            }
            if (!Q && act && cn.key >= 0 && !fast) {
                const int jt0 = cn.jt, jt1 = (cn.jt == na - 1) ? 0 : cn.jt + 1;
                // the corner rows: row, row + 1 (the next plane, or ring in
                // 2D), and in 3D row + ngz, row + ngz + 1, with their window
                // coordinates (a, b)
                int fr[4], wa[4], wb[4];
                fr[0] = cn.row;
                fr[1] = cn.row + 1;
                if (d3) {
                    int ju1 = cn.ju, iz1 = cn.iz + 1;
                    if (iz1 == ngz) {
                        iz1 = 0;
                        ju1 += 1;
                    }
                    wa[0] = cn.ju - wir + 1;
                    wb[0] = cn.iz - wiz + 1;
                    wa[1] = ju1 - wir + 1;
                    wb[1] = iz1 - wiz + 1;
                    fr[2] = cn.row + ngz;
                    fr[3] = cn.row + ngz + 1;
                    wa[2] = wa[0] + 1;
                    wb[2] = wb[0];
                    wa[3] = wa[1] + 1;
                    wb[3] = wb[1];
                } else {
                    wa[0] = cn.row - row + 1;
                    wa[1] = wa[0] + 1;
                    wb[0] = wb[1] = 0;
                }
                constexpr int NQ = d3 ? 4 : 2;
#pragma unroll
                for (int q = 0; q < NQ; q++) {
                    if (fr[q] >= nrow) continue;  // past the mesh end: dropped, as massgn does
                    const int v0 = va[2 * q];
                    const int v1 = va[2 * q + 1];
                    const bool inw = win && wa[q] >= 0 && wa[q] < 4 && wb[q] >= 0 && wb[q] < 4;
                    unsigned long long* ar = acc + (size_t)fr[q] * na;
                    uint32_t* br = bins + (inw ? (d3 ? 4 * wa[q] + wb[q] : wa[q]) * na : 0);
                    if (inw && v0 > 0) atomicAdd(br + jt0, (uint32_t)v0);
                    else if (v0) red_add_s64(ar + jt0, v0);
                    if (inw && v1 > 0) atomicAdd(br + jt1, (uint32_t)v1);
                    else if (v1) red_add_s64(ar + jt1, v1);
                }
            }
            if (!DEP) {
                bslot = __shfl_sync(0xffffffffu, bslot, leader < 0 ? 0 : leader);
                int slot = bslot + __popc(peers & lanemask_lt());
                if (cta) {
                    __syncthreads();
                    if (wi >= 0) slot = s_slot[ph][wi] + rank;
                    ph ^= 1;
                }
                int64_t dst = (int64_t)baser + slot;
                const bool ovf = act && slot >= capr;
                const uint32_t om = __ballot_sync(0xffffffffu, ovf);
                if (om) {
                    const int ol = __ffs(om) - 1;
                    int ob = 0;
                    if ((int)lane == ol) ob = atomicAdd(ovf_o, __popc(om));
                    ob = __shfl_sync(0xffffffffu, ob, ol);
                    if (ovf) dst = ovf_base + ob + __popc(om & lanemask_lt());
                }
                if (act) rec_store<NP>(Qout, bcap, dst, P, o);
            }
        }
        if (win) {
            __syncthreads();
#pragma unroll 4
            for (int wr = 0; wr < WROWS; wr++) {
                const int R = d3 ? (wir - WLO + wr / W) * ngz + (wiz - WLO + wr % W) : wir - 1 + wr;
                uint32_t* br = bins + wr * na;
                for (int j = threadIdx.x; j < na; j += BK_THREADS) {
                    const uint32_t v = br[j];
                    if (v) {
                        atomicAdd(acc + (size_t)R * na + j, (unsigned long long)v);
                        br[j] = 0u;
                    }
                }
            }
        }
        // orders the flush before the next deposits, and the next item's
        // descriptor and field rows after this item's use of theirs
        __syncthreads();
    }
    // the ring range of the new cells (massgn's jrad / krad): one atomic
    // pair per warp
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        rmin_l = min(rmin_l, __shfl_xor_sync(0xffffffffu, rmin_l, o));
        rmax_l = max(rmax_l, __shfl_xor_sync(0xffffffffu, rmax_l, o));
        zmin_l = min(zmin_l, __shfl_xor_sync(0xffffffffu, zmin_l, o));
        zmax_l = max(zmax_l, __shfl_xor_sync(0xffffffffu, zmax_l, o));
    }
    if ((threadIdx.x & 31) == 0 && rmax_l >= 0) {
        atomicMin(rg, rmin_l);
        atomicMax(rg + 1, rmax_l);
        if (d3) {
            atomicMin(rg + 2, zmin_l);
            atomicMax(rg + 3, zmax_l);
        }
    }
}

// mass = pmass 2^-20 acc (as k_mass_combine forms it); acc cleared for the
// next step.  zonly: the array holds a fused pass's mass already, so only the
// planes that held it (zro) or hold it now need converting, a third of a thin
// disc's mesh (128 x 256 x 125: 12.0 us over the mesh, 7.2 over 46 planes).
__global__ void __launch_bounds__(256) k_mass_convert(unsigned long long* __restrict__ acc,
                               float* __restrict__ mass, float pm, const int32_t* __restrict__ rg, int32_t* __restrict__ rgo,
                               int32_t* __restrict__ jrk, int nr, int na,
                               int32_t* __restrict__ zr, const int32_t* __restrict__ zro, int ngz, bool quad,
                               bool zonly) {
    // the active ring range of the new mass, as massgn tracks it (jrad =
    // first ring + 1, krad = min(last ring + 2, nr), 1-based), and the planes
    // holding mass (the cells' planes and the next, clamped), from the
    // ranges the pass gathered (rg); the next pass's (rgo) cleared
    const bool first = blockIdx.x == 0 && threadIdx.x == 0;
    int z0 = 0, z1 = ngz - 1;
    if (zonly || first) {
        const int zn = rg[2], zx = rg[3];
        z0 = (zx >= 0) ? zn : ngz;
        z1 = (zx >= 0) ? min(zx + 1, ngz - 1) : -1;
    }
    if (first) {
        const int mn = rg[0], mx = rg[1];
        jrk[0] = (mx >= 0) ? mn + (quad ? 0 : 1) : nr;  // quadratic: the ring below (massgn.f:180)
        jrk[1] = (mx >= 0) ? min(mx + 2, nr) : 0;
        zr[0] = z0;
        zr[1] = z1;
        rgo[0] = rgo[2] = 0x7fffffff;
        rgo[1] = rgo[3] = -1;
    }
    // one ring-plane row per warp and iteration, two cells per lane
    const int lo = zonly ? min(z0, zro[0]) : 0, hi = zonly ? max(z1, zro[1]) : ngz - 1;
    const int np = hi - lo + 1, lane = threadIdx.x & 31;
    const int nw = gridDim.x * (blockDim.x >> 5);
    for (int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < nr * np; w += nw) {
        const int ir = w / np, row = ir * ngz + lo + (w - ir * np);
        unsigned long long* a = acc + (size_t)row * na;
        float* mr = mass + (size_t)row * na;
#pragma unroll 4
        for (int j = 2 * lane; j < na; j += 64) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(a + j);
            float2 m;
            m.x = (float)((double)(long long)v.x * (1.0 / (double)BK_FIXQ)) * pm;
            m.y = (float)((double)(long long)v.y * (1.0 / (double)BK_FIXQ)) * pm;
            *reinterpret_cast<float2*>(mr + j) = m;
            if (v.x | v.y) *reinterpret_cast<ulonglong2*>(a + j) = make_ulonglong2(0ull, 0ull);
        }
    }
}

// ---------------------------------------------------------------------------
// dense store -> bucketed store: the row of every particle's cell (the
// deposit's exact cell), counted
template <int ND>
__global__ void k_bk_rows(DevGeo g, const float* __restrict__ P, int64_t cap, int64_t n,
                          int32_t* __restrict__ rows, int32_t* __restrict__ cnt) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const bool act = i < n;
    uint32_t rk = 0;
    if (act) {
        const CellW c = gx_cell_t<true, ND>(g, P[i], P[cap + i], ND == 3 ? P[2 * cap + i] : 0.f, false);
        rk = (c.key >= 0) ? (uint32_t)c.row : (uint32_t)g.nrow;
        rows[i] = (int32_t)rk;
    }
    const uint32_t am = __ballot_sync(0xffffffffu, act);
    const uint32_t peers = __match_any_sync(0xffffffffu, act ? rk : 0xffffffffu) & am;
    if (act && (peers & lanemask_lt()) == 0) atomicAdd(cnt + rk, (int)__popc(peers));
}

// The same two steps with the counts gathered per CTA first (grids whose row
// table fits in shared memory): a CTA takes a run of BK_RUN particles, counts
// their rows in shared memory, and touches each global counter once per
// nonzero row instead of once per warp group -- a disc's central rows get
// tens of thousands of particles, whose single-address atomics otherwise
// serialise.  The scatter reserves each row's slots for the CTA with one
// atomic on the row's fill counter and hands them out from shared memory.
// A run is BK_RUN particles, or fewer when that would leave SMs idle (bk_run).
#define BK_RUN 32768
template <int ND>
__global__ void __launch_bounds__(256) k_bk_rows_cta(DevGeo g, const float* __restrict__ P, int64_t cap,
                                                     int64_t n, int run, int32_t* __restrict__ rows,
                                                     int32_t* __restrict__ cnt) {
    extern __shared__ int32_t hist[];  // [nrow + 1]
    const int nr1 = g.nrow + 1;
    for (int r = threadIdx.x; r < nr1; r += blockDim.x) hist[r] = 0;
    __syncthreads();
    const int64_t i0 = (int64_t)blockIdx.x * run, i1 = min(n, i0 + run);
    for (int64_t i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
        const CellW c = gx_cell_t<true, ND>(g, P[i], P[cap + i], ND == 3 ? P[2 * cap + i] : 0.f, false);
        const int rk = (c.key >= 0) ? c.row : g.nrow;
        rows[i] = rk;
        atomicAdd(hist + rk, 1);
    }
    __syncthreads();
    for (int r = threadIdx.x; r < nr1; r += blockDim.x)
        if (hist[r]) atomicAdd(cnt + r, hist[r]);
}

template <int NP>
__global__ void __launch_bounds__(256) k_bk_scatter_cta(const float* __restrict__ P, int64_t cap, int64_t n, int run,
                                                        const int32_t* __restrict__ oin, float4* __restrict__ Qout,
                                                        int64_t bcap, const int32_t* __restrict__ rows, int nr1,
                                                        const int32_t* __restrict__ cap_o,
                                                        const int32_t* __restrict__ base_o,
                                                        int32_t* __restrict__ fill_o, int32_t* __restrict__ ovf_o,
                                                        int64_t ovf_base) {
    extern __shared__ int32_t slot[];  // [nrow + 1]: this CTA's count, then its next slot
    for (int r = threadIdx.x; r < nr1; r += blockDim.x) slot[r] = 0;
    __syncthreads();
    const int64_t i0 = (int64_t)blockIdx.x * run, i1 = min(n, i0 + run);
    for (int64_t i = i0 + threadIdx.x; i < i1; i += blockDim.x) atomicAdd(slot + rows[i], 1);
    __syncthreads();
    for (int r = threadIdx.x; r < nr1; r += blockDim.x)
        if (slot[r]) slot[r] = atomicAdd(fill_o + r, slot[r]);
    __syncthreads();
    for (int64_t i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
        const int rk = rows[i];
        const int sl = atomicAdd(slot + rk, 1);
        int64_t dst;
        if (sl < __ldg(cap_o + rk)) dst = (int64_t)__ldg(base_o + rk) + sl;
        else dst = ovf_base + atomicAdd(ovf_o, 1);  // past the segment (rare): the overflow area
        float w[NP];
#pragma unroll
        for (int k = 0; k < NP; k++) w[k] = P[(size_t)k * cap + i];
        rec_store<NP>(Qout, bcap, dst, w, oin[i]);
    }
}

template <int NP>
__global__ void k_bk_scatter(const float* __restrict__ P, int64_t cap, int64_t n, const int32_t* __restrict__ oin,
                             float4* __restrict__ Qout, int64_t bcap, const int32_t* __restrict__ rows,
                             const int32_t* __restrict__ cap_o, const int32_t* __restrict__ base_o,
                             int32_t* __restrict__ fill_o, int32_t* __restrict__ ovf_o, int64_t ovf_base) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const bool act = i < n;
    const uint32_t rk = act ? (uint32_t)rows[i] : 0u;
    const int64_t dst = bk_slot(act, rk, cap_o, base_o, fill_o, ovf_o, ovf_base);
    if (!act) return;
    float w[NP];
#pragma unroll
    for (int k = 0; k < NP; k++) w[k] = P[(size_t)k * cap + i];
    rec_store<NP>(Qout, bcap, dst, w, oin[i]);
}

// bucketed store -> n contiguous particles (SoA planes and load index),
// item by item (CTA-reserved ranges)
template <int NP>
__global__ void k_bk_densify(const float4* __restrict__ Qin, int64_t bcap, float* __restrict__ P, int64_t cap,
                             int32_t* __restrict__ oout, const int4* __restrict__ items,
                             const int32_t* __restrict__ ctl, int32_t* __restrict__ dense_ctr) {
    __shared__ int s_d0;
    const int nit = ctl[0];
    for (int it = blockIdx.x; it < nit; it += gridDim.x) {
        const int4 I = items[it];
        if (threadIdx.x == 0) s_d0 = atomicAdd(dense_ctr, I.z - I.y);
        __syncthreads();
        const int d0 = s_d0;
        for (int s = I.y + threadIdx.x; s < I.z; s += blockDim.x) {
            const int64_t d = d0 + (s - I.y);
            float w[NP];
            int32_t o;
            rec_load<NP>(Qin, bcap, s, w, o);
#pragma unroll
            for (int k = 0; k < NP; k++) P[(size_t)k * cap + d] = w[k];
            oout[d] = o;
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
bool gx_fast_ok(const GxCtx* c) {
    return !c->fp64 && c->nzones == 1 && !(c->cfg.flags & GX_FLAG_SORTED_DEPOSIT) &&
           !(c->g.quad && c->g.na > BK_QUAD_NA);
}

static inline int bk_nplanes(const GxCtx* c) { return 2 * c->g.ndim + (c->g.comp ? c->g.ndim : 0); }

// bucketed store -> the host records (x, y[, z], vx, vy[, vz]) in load
// order, in two passes: k_bk_inv writes each record's slot at its load
// index (4-byte scattered writes into an n-entry table that stays in L2),
// k_bk_gather walks the load indices in order, reads each record (one
// 32-byte access) and writes the host layout contiguously.  Writing the
// 16 / 24-byte records straight to their scattered load positions (one
// pass) made partial-sector writes over an output larger than L2.
template <int NP>
__global__ void k_bk_inv(const float4* __restrict__ Qin, int64_t bcap, int32_t* __restrict__ inv,
                         const int4* __restrict__ items, const int32_t* __restrict__ ctl) {
    const int nit = ctl[0];
    for (int it = blockIdx.x; it < nit; it += gridDim.x) {
        const int4 I = items[it];
        for (int s = I.y + threadIdx.x; s < I.z; s += blockDim.x) {
            float w[NP];
            int32_t o;
            rec_load<NP>(Qin, bcap, s, w, o);
            inv[o] = s;
        }
    }
}

template <int NP, int NW>
__global__ void k_bk_gather(const float4* __restrict__ Qin, int64_t bcap, const int32_t* __restrict__ inv,
                            float* __restrict__ aos, int64_t n) {
    static_assert(NW == 4 || NW == 6, "2D or 3D records");
    const int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (o >= n) return;
    float w[NP];
    int32_t oo;
    rec_load<NP>(Qin, bcap, __ldg(inv + o), w, oo);
    if (NW == 4) {
        reinterpret_cast<float4*>(aos)[o] = make_float4(w[0], w[1], w[2], w[3]);
    } else {
        float2* d = reinterpret_cast<float2*>(aos + (size_t)o * 6);
        d[0] = make_float2(w[0], w[1]);
        d[1] = make_float2(w[2], w[3]);
        d[2] = make_float2(w[4], w[5]);
    }
}

template <int NP, int NW>
static void bk_unload_launch(GxCtx* c, float* aos) {
    int32_t* inv = c->pkey[0];  // free while the store is bucketed (the keys are recomputed after it)
    k_bk_inv<NP><<<148 * 8, 256, 0, c->stream>>>(c->bq[c->bcur], c->bcap, inv, c->bk_items, c->bk_ctl + 8);
    k_bk_gather<NP, NW><<<(unsigned)((c->n + 255) / 256), 256, 0, c->stream>>>(c->bq[c->bcur], c->bcap, inv,
                                                                                aos, c->n);
}

// float4 words of one record of the bucketed store
int gx_bucket_words(const GxCtx* c) { return (bk_nplanes(c) + 1 + 3) / 4; }

static inline size_t bk_npad(const GxCtx* c);
static int bk_plan(GxCtx* c, int out, bool with_items, cudaStream_t st);

template <typename T>
static int bk_alloc(GxCtx* c, T** p, size_t count) {
    if (*p) return GX_OK;
    if (cudaMalloc((void**)p, sizeof(T) * std::max<size_t>(count, 1)) != cudaSuccess) {
        cudaGetLastError();
        *p = nullptr;
        c->err = "cudaMalloc of the bucketed store's tables failed";
        return GX_ERR_NOMEM;
    }
    return GX_OK;
}

// row tables and the mass accumulator (grid-sized, once per context)
static inline size_t bk_npad(const GxCtx* c) {
    const size_t per = (size_t)PLAN_THREADS * PLAN_ROWS;
    return ((size_t)c->g.nrow + 1 + per - 1) / per * per;
}

int gx_bucket_alloc(GxCtx* c) {
    const size_t nrow1 = bk_npad(c);
    int rc = 0;
    for (int b = 0; b < 2 && !rc; b++) {
        rc = rc ? rc : bk_alloc(c, &c->bk_cap[b], nrow1);
        rc = rc ? rc : bk_alloc(c, &c->bk_base[b], nrow1);
        rc = rc ? rc : bk_alloc(c, &c->bk_fill[b], nrow1);
    }
    rc = rc ? rc : bk_alloc(c, &c->bk_ctl, 24);
    rc = rc ? rc : bk_alloc(c, &c->bk_cnt, nrow1);
    rc = rc ? rc : bk_alloc(c, &c->macc, (size_t)c->g.mesh);
    rc = rc ? rc : bk_alloc(c, &c->zr_d, 4);
    if (rc) return rc;
    for (int b = 0; b < 2; b++) {
        GX_CUDA(c, cudaMemsetAsync(c->bk_fill[b], 0, sizeof(int32_t) * nrow1, c->stream));
        GX_CUDA(c, cudaMemsetAsync(c->bk_cap[b], 0, sizeof(int32_t) * nrow1, c->stream));
        GX_CUDA(c, cudaMemsetAsync(c->bk_base[b], 0, sizeof(int32_t) * nrow1, c->stream));
    }
    GX_CUDA(c, cudaMemsetAsync(c->macc, 0, sizeof(unsigned long long) * c->g.mesh, c->stream));
    int32_t ctl0[24] = {};
    for (int i = 16; i < 24; i += 2) {
        ctl0[i] = 0x7fffffff;
        ctl0[i + 1] = -1;
    }
    GX_CUDA(c, cudaMemcpyAsync(c->bk_ctl, ctl0, sizeof ctl0, cudaMemcpyHostToDevice, c->stream));
    GX_CUDA(c, cudaStreamSynchronize(c->stream));
    return GX_OK;
}

static int bk_plan(GxCtx* c, int out, bool with_items, cudaStream_t st) {
    const DevGeo& g = c->g;
    const int nxt = out ^ 1;
    k_bk_plan<<<1, PLAN_THREADS, 0, st>>>(
        g.nrow + 1, g.ngz, with_items ? c->bk_fill[out] : nullptr, c->bk_cap[out], c->bk_base[out],
        c->bk_ctl + 4 * out, c->bk_main, c->bk_items, c->bk_ctl + 8,
        with_items ? c->bk_fill[out] : c->bk_cnt, c->bk_cap[nxt], c->bk_base[nxt], c->bk_fill[nxt],
        c->bk_ctl + 4 * nxt, c->bk_item);
    GX_LAUNCHED(c);
    return GX_OK;
}

// particles per CTA of the bucketing: two CTAs per SM when the particles
// suffice for runs of at least 1024, BK_RUN at most.  1M particles in runs of
// 32768 (31 CTAs) took 234 us to count and place, in runs of 3584 60 us.
static int bk_run(int64_t n) {
    const int64_t r = (n / (2 * 148) + 256) / 256 * 256;
    return (int)std::min<int64_t>(BK_RUN, std::max<int64_t>(1024, r));
}

template <int NP>
static void bk_scatter_cta_launch(GxCtx* c, int b) {
    const int nr1 = c->g.nrow + 1;
    const int run = bk_run(c->n);
    const unsigned nruns = (unsigned)((c->n + run - 1) / run);
    cudaFuncSetAttribute(k_bk_scatter_cta<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(sizeof(int32_t) * nr1));
    k_bk_scatter_cta<NP><<<nruns, 256, sizeof(int32_t) * nr1, c->stream>>>(
        c->pbuf[c->cur], c->cap, c->n, run, c->origin, c->bq[b], c->bcap, c->pkey[0], nr1, c->bk_cap[b], c->bk_base[b],
        c->bk_fill[b], c->bk_ctl + 4 * b, c->bk_main);
}

template <int NP>
static void bk_scatter_launch(GxCtx* c, unsigned nb, int b) {
    k_bk_scatter<NP><<<nb, 256, 0, c->stream>>>(c->pbuf[c->cur], c->cap, c->n, c->origin, c->bq[b], c->bcap,
                                                c->pkey[0], c->bk_cap[b], c->bk_base[b], c->bk_fill[b],
                                                c->bk_ctl + 4 * b, c->bk_main);
}

template <int NP>
static void bk_densify_launch(GxCtx* c, int32_t* ctr) {
    k_bk_densify<NP><<<148 * 8, 256, 0, c->stream>>>(c->bq[c->bcur], c->bcap, c->pbuf[c->cur], c->cap,
                                                     c->origin, c->bk_items, c->bk_ctl + 8, ctr);
}

// the dense store pbuf[cur] -> the bucketed store bq[b], b = bcur ^ 1
// (becomes bcur); the dense store is left as it was, and is stale from the
// first fused step on
static int gx_bucketize(GxCtx* c) {
    const DevGeo& g = c->g;
    const int64_t n = c->n;
    const int b = c->bcur ^ 1;
    const unsigned nb = (unsigned)((std::max<int64_t>(n, 1) + 255) / 256);
    GX_CUDA(c, cudaMemsetAsync(c->bk_cnt, 0, sizeof(int32_t) * bk_npad(c), c->stream));
    // the row table in shared memory when it fits in 96 KB (two CTAs per SM)
    const size_t hbytes = sizeof(int32_t) * ((size_t)g.nrow + 1);
    const bool cta = hbytes <= 96 * 1024;
    if (n > 0) {
        if (cta) {
            auto kr = (g.ndim == 3) ? k_bk_rows_cta<3> : k_bk_rows_cta<2>;
            cudaFuncSetAttribute(kr, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hbytes);
            const int run = bk_run(n);
            kr<<<(unsigned)((n + run - 1) / run), 256, hbytes, c->stream>>>(g, c->pbuf[c->cur], c->cap, n, run,
                                                                            c->pkey[0], c->bk_cnt);
        } else {
            auto kr = (g.ndim == 3) ? k_bk_rows<3> : k_bk_rows<2>;
            kr<<<nb, 256, 0, c->stream>>>(g, c->pbuf[c->cur], c->cap, n, c->pkey[0], c->bk_cnt);
        }
        GX_LAUNCHED(c);
    }
    // segments of bq[b] from the exact counts (with_items = false plans the
    // layout of buffer "out ^ 1" = b from want = bk_cnt)
    int rc = bk_plan(c, b ^ 1, false, c->stream);
    if (rc) return rc;
    if (n > 0) {
        switch (bk_nplanes(c)) {
            case 4: cta ? bk_scatter_cta_launch<4>(c, b) : bk_scatter_launch<4>(c, nb, b); break;
            case 6: cta ? bk_scatter_cta_launch<6>(c, b) : bk_scatter_launch<6>(c, nb, b); break;
            default: cta ? bk_scatter_cta_launch<9>(c, b) : bk_scatter_launch<9>(c, nb, b); break;
        }
        GX_LAUNCHED(c);
    }
    // items of bq[b]; segments of bq[b ^ 1] for the first fused pass
    rc = bk_plan(c, b, true, c->stream);
    if (rc) return rc;
    c->bcur = b;
    c->bucketed = true;
    return GX_OK;
}

__global__ void k_bk_iota(int32_t* p, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) p[i] = (int32_t)i;
}

// bucketed store -> the dense store pbuf[cur] (its SoA planes and load
// index), in the store's row order; the processing order becomes the
// identity
int gx_dense(GxCtx* c) {
    if (!c->bucketed) return GX_OK;
    int32_t* ctr = c->bk_ctl + 12;
    GX_CUDA(c, cudaMemsetAsync(ctr, 0, sizeof(int32_t), c->stream));
    switch (bk_nplanes(c)) {
        case 4: bk_densify_launch<4>(c, ctr); break;
        case 6: bk_densify_launch<6>(c, ctr); break;
        default: bk_densify_launch<9>(c, ctr); break;
    }
    GX_LAUNCHED(c);
    if (c->n > 0) {
        k_bk_iota<<<(unsigned)((c->n + 255) / 256), 256, 0, c->stream>>>(c->perm, c->n);
        GX_LAUNCHED(c);
    }
    c->bucketed = false;
    return GX_OK;
}

// gx_unload's records from the bucketed store (the store stays as it is)
int gx_bucket_unload(GxCtx* c, float* aos) {
    if (c->n <= 0) return GX_OK;
    // record planes: the phase space (2D: 4, 3D: 6) and the compensated
    // update's low parts of the positions
    if (c->g.ndim == 3) {
        if (c->g.comp) bk_unload_launch<9, 6>(c, aos);
        else bk_unload_launch<6, 6>(c, aos);
    } else {
        if (c->g.comp) bk_unload_launch<6, 4>(c, aos);
        else bk_unload_launch<4, 4>(c, aos);
    }
    c->launches++;  // two kernels: the inversion and the gather
    GX_LAUNCHED(c);
    return GX_OK;
}

template <int ND, bool COMP, bool DEP = false, bool Q = false>
static int bk_launch_push(GxCtx* c, int cur, int nxt) {
    const DevGeo& g = c->g;
    // the deposit window and, for the push, the staged field rows
    const size_t sb = sizeof(uint32_t) * (Q ? 28 : ND == 3 ? 16 : 4) * g.na;  // 25 rows and a pad: 16-byte aligned
    const size_t sf = sb + sizeof(float4) * (Q ? 9 : ND == 3 ? 4 : 2) * g.na;
    if (!c->bk_ctas[0]) {
        // CTAs of the push without and with the rows, once per context; the deposit
        // alone runs as many
        int pb = 0, pf = 0, sms = 148;
        auto kf = k_push_bkt<ND, COMP, false, Q>;
        GX_CUDA(c, cudaFuncSetAttribute(kf, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sf));
        GX_CUDA(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&pf, kf, BK_THREADS, sf));
        GX_CUDA(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&pb, kf, BK_THREADS, sb));
        GX_CUDA(c, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->dev));
        c->bk_ctas[1] = std::max(1, pf) * sms;
        c->bk_ctas[0] = std::max(1, pb) * sms;
    }
    const bool stage = c->bk_ctas[1] >= c->bk_ctas[0] || c->n >= (int64_t)BK_STAGE_ROW * g.nrow;
    const size_t sm = DEP || !stage ? sb : sf;
    auto kp = k_push_bkt<ND, COMP, DEP, Q>;
    GX_CUDA(c, cudaFuncSetAttribute(kp, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    c->acc_open = true;
    kp<<<c->bk_ctas[stage], BK_THREADS, sm, c->stream>>>(g, c->bq[cur], c->bq[nxt], c->bcap, c->field, c->bk_items,
                                                  c->bk_ctl + 8, c->bk_cap[nxt], c->bk_base[nxt],
                                                  c->bk_fill[nxt], c->bk_ctl + 4 * nxt, c->bk_main, c->macc,
                                                  gx_mass_ranges(c), stage ? BK_STAGE : INT_MAX);
    GX_LAUNCHED(c);
    return GX_OK;
}

// the accumulator -> the mass array, its ring and plane ranges; both cleared
int gx_mass_convert(GxCtx* c) {
    const DevGeo& g = c->g;
    const int p = c->mpar, q = p ^ 1;
    k_mass_convert<<<std::min((g.nrow + 7) / 8, 148 * 8), 256, 0, c->stream>>>(
        c->macc, c->mass, g.pmass, c->bk_ctl + 16 + 4 * p, c->bk_ctl + 16 + 4 * q, c->jrk_d, g.nr, g.na,
        c->zr_d + 2 * p, c->zr_d + 2 * q, g.ngz, g.quad, g.ndim == 3 && c->zr_valid);
    GX_LAUNCHED(c);
    c->mpar = q;
    c->acc_open = c->acc_pending = false;
    return GX_OK;
}

// A call that fails between a deposit pass and the conversion of what it
// deposited leaves both accumulators and their ranges as a new context has
// them, so that the next masset adds to nothing; the mass array no longer
// belongs to the particles.  (A call refused before its deposit keeps its mass.)
void gx_mass_discard(GxCtx* c) {
    if (!c->acc_open) return;
    int32_t none[2 * GX_MAX_ZONES];
    for (int i = 0; i < 2 * GX_MAX_ZONES; i += 2) {
        none[i] = 0x7fffffff;
        none[i + 1] = -1;
    }
    static_assert(2 * GX_MAX_ZONES >= 8, "both sets of ranges");
    // (no status: where these fail, so do the calls that follow)
    cudaMemsetAsync(c->macc, 0, sizeof(unsigned long long) * c->g.mesh, c->stream);
    cudaMemcpyAsync(c->bk_ctl + 16, none, 8 * sizeof(int32_t), cudaMemcpyHostToDevice, c->stream);
    if (c->zacc && c->nzones > 1) {
        cudaMemsetAsync(c->zacc, 0, sizeof(unsigned long long) * (c->nzones - 1) * c->g.mesh, c->stream);
        cudaMemcpyAsync(c->zjrk_d + 2 * GX_MAX_ZONES + 2, none, sizeof none, cudaMemcpyHostToDevice, c->stream);
    }
    cudaStreamSynchronize(c->stream);
    c->acc_open = c->acc_pending = false;
    c->have_mass = c->zones_ready = c->zr_valid = false;
}

// 2D: the forward transform converts its ring itself (gx_mixed_findf, which
// has to come next).  Not across ranks, which reduce the ring range first.
int gx_mass_defer(GxCtx* c) {
    if (c->g.ndim != 2 || c->nranks > 1 || c->prof) return gx_mass_convert(c);
    c->acc_pending = true;
    return GX_OK;
}

// the main stream waits for the plan queued on the side stream
static int bk_join(GxCtx* c) {
    if (!c->bk_pending) return GX_OK;
    GX_CUDA(c, cudaStreamWaitEvent(c->stream, c->bk_ev[1], 0));
    c->bk_pending = false;
    return GX_OK;
}

// masset on the fused path: the deposit-only pass over the bucketed store
// (bucketized first when the particles are dense), then the conversion.
// The mass is the same integers, converted the same way, as the sorted
// deposit's (massgn.f:140-172), and the ring and plane ranges of the mass
// are known to the next solve.
int gx_fast_masset(GxCtx* c) {
    const DevGeo& g = c->g;
    int rc = c->bucketed ? bk_join(c) : gx_bucketize(c);
    if (rc) return rc;
    const int cur = c->bcur, nxt = cur ^ 1;
    if (g.quad)
        rc = g.comp ? bk_launch_push<3, true, true, true>(c, cur, nxt) : bk_launch_push<3, false, true, true>(c, cur, nxt);
    else if (g.ndim == 3)
        rc = g.comp ? bk_launch_push<3, true, true>(c, cur, nxt) : bk_launch_push<3, false, true>(c, cur, nxt);
    else
        rc = g.comp ? bk_launch_push<2, true, true>(c, cur, nxt) : bk_launch_push<2, false, true>(c, cur, nxt);
    if (rc) return rc;
    // the pass took the items through the work counter: the next pass starts it afresh
    GX_CUDA(c, cudaMemsetAsync(c->bk_ctl + 9, 0, sizeof(int32_t), c->stream));
    rc = gx_mass_convert(c);
    if (rc) return rc;
    c->zr_valid = true;
    return GX_OK;
}

// one fused step: the solve of the current mass (only the planes that hold
// it once they are known), the pass, its plan on the side stream, the mass
// (left to the next step's solve in 2D, except after the last step of a call)
static int fast_one_step(GxCtx* c, bool lpot, bool last) {
    const DevGeo& g = c->g;
    // once the mass is a fused pass's, the solve knows the planes that
    // hold it, and the field is needed only where the particles are
    int rc = gx_mixed_findf(c, lpot ? 1 : 0, true, nullptr,
                           (c->zr_valid && g.ndim == 3) ? c->zr_d + 2 * (c->mpar ^ 1) : nullptr);
    if (rc) return rc;
    const int cur = c->bcur, nxt = cur ^ 1;
    rc = bk_join(c);
    if (rc) return rc;
    rc = gx_phase_mark(c, PH_PUSH);
    if (rc) return rc;
    if (g.quad)
        rc = g.comp ? bk_launch_push<3, true, false, true>(c, cur, nxt) : bk_launch_push<3, false, false, true>(c, cur, nxt);
    else if (g.ndim == 3) rc = g.comp ? bk_launch_push<3, true>(c, cur, nxt) : bk_launch_push<3, false>(c, cur, nxt);
    else rc = g.comp ? bk_launch_push<2, true>(c, cur, nxt) : bk_launch_push<2, false>(c, cur, nxt);
    if (rc) return rc;
    if (c->prof) {
        // profile mode: the plan in line, so that it has a phase time
        rc = gx_phase_mark(c, PH_SORT);
        if (rc) return rc;
        rc = bk_plan(c, nxt, true, c->stream);
        if (rc) return rc;
    } else {
        // the plan needs only the push: it runs on the side stream while
        // the next field solve runs, and the next push waits for it
        GX_CUDA(c, cudaEventRecord(c->bk_ev[0], c->stream));
        GX_CUDA(c, cudaStreamWaitEvent(c->bk_side, c->bk_ev[0], 0));
        rc = bk_plan(c, nxt, true, c->bk_side);
        if (rc) return rc;
        GX_CUDA(c, cudaEventRecord(c->bk_ev[1], c->bk_side));
        c->bk_pending = true;
    }
    rc = gx_phase_mark(c, PH_COMBINE);
    if (rc) return rc;
    rc = last ? gx_mass_convert(c) : gx_mass_defer(c);
    if (rc) return rc;
    c->zr_valid = true;
    c->bcur = nxt;
    return GX_OK;
}

// two fused steps from the current store captured into a CUDA graph (the
// plans forked to the side stream and joined inside it): the graph, and the
// kernels of one replay in *per; null when the capture is refused, and the
// steps then run as plain launches.  Capturing runs nothing: the host state
// the two steps would change is put back.
static cudaGraphExec_t fast_capture(GxCtx* c, int64_t* per) {
    const int b = c->bcur, mp = c->mpar;
    if (bk_join(c) != GX_OK) return nullptr;
    const int64_t l0 = c->launches;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    // a stream the caller is capturing already is left alone
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(c->stream, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return nullptr;
    }
    if (cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    bool ok = fast_one_step(c, false, false) == GX_OK && fast_one_step(c, false, false) == GX_OK && bk_join(c) == GX_OK;
    const cudaError_t ec = cudaStreamEndCapture(c->stream, &graph);
    ok = ok && ec == cudaSuccess && graph;
    if (ok) ok = cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess;
    if (graph) cudaGraphDestroy(graph);
    cudaGetLastError();
    *per = c->launches - l0;
    c->bcur = b;
    c->mpar = mp;
    c->acc_pending = c->acc_open = true;  // as it was: the caller captures after a deferred step
    c->bk_pending = false;
    c->launches = l0;
    c->err.clear();
    return ok ? exec : nullptr;
}

int gx_fast_step(GxCtx* c, int nsteps, int phys) {
    int rc;
    if (!c->bk_side) {
        int lo = 0, hi = 0;
        GX_CUDA(c, cudaDeviceGetStreamPriorityRange(&lo, &hi));
        GX_CUDA(c, cudaStreamCreateWithPriority(&c->bk_side, cudaStreamNonBlocking, hi));
        GX_CUDA(c, cudaEventCreateWithFlags(&c->bk_ev[0], cudaEventDisableTiming));
        GX_CUDA(c, cudaEventCreateWithFlags(&c->bk_ev[1], cudaEventDisableTiming));
    }
    if (!c->bucketed) {
        rc = gx_bucketize(c);
        if (rc) return rc;
    }
    // 2D contexts (small grids: their steps take tens of microseconds, so the
    // gaps between launches count) replay pairs of steps from a CUDA graph,
    // captured in this call once the state is steady (the mass a fused
    // pass's, every buffer allocated) and released at its end
    const bool graphs = c->g.ndim == 2 && !c->prof && c->nranks <= 1;
    cudaGraphExec_t exec = nullptr;
    int64_t per = 0;
    bool tried = false;
    int s = 0;
    while (s < nsteps) {
        const bool last = (s == nsteps - 1);
        const int pairs = (nsteps - s - 1) / 2;  // the last step runs as plain launches (phys)
        if (graphs && c->zr_valid && c->acc_pending && pairs >= 4 && !tried) {
            tried = true;
            exec = fast_capture(c, &per);
        }
        if (exec && pairs > 0) {
            rc = bk_join(c);
            if (rc) break;
            for (int p = 0; p < pairs && !rc; p++) {
                if (cudaGraphLaunch(exec, c->stream) != cudaSuccess) rc = (c->err = "cudaGraphLaunch failed", GX_ERR_CUDA);
                c->launches += per;
            }
            if (rc) break;
            s += 2 * pairs;
            continue;
        }
        rc = fast_one_step(c, phys && last, last);
        if (rc) break;
        s++;
    }
    if (exec) cudaGraphExecDestroy(exec);
    if (rc) return rc;
    rc = bk_join(c);
    if (rc) return rc;
    rc = gx_phase_end(c);
    if (rc) return rc;
    c->have_field = false;
    return GX_OK;
}
