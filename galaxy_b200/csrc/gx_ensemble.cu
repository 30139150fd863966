// gx_ensemble.cu -- an ensemble of independent 2D discs on one polar grid
// geometry, advanced together by persistent cooperative launches of up to
// ENS_MAXSTEPS steps each.
//
// Each disc is the run the single-disc path makes of it (SRC/progs/galaxy.f
// time loop: findf, getacc + stpgrp, massgn): same cell keys and weights
// (gx_cell, weight.f:61-101), the same integer fixed-point deposit
// (massgn.f:68-89; 2^-20 of a particle mass, summed as integers, so the
// mass array is the same integers), the same forward / contraction /
// synthesis arithmetic (p2manl.f:32-45, p2conv.f:99-187, p2fsyn.f:34-56,
// polcat.f:22-41) with FP32 sums, the m = 0 forward sum in FP64.
//
// One launch:
//   solve   turns a disc's integer mass into its (fx, fy) field grid: forward
//           DFT of the active harmonics per ring, radial contraction with the
//           shared Green table (read from L2), synthesis + polcat; it then
//           zeroes the integer mass and publishes the field with the disc's
//           ready flag (the step's epoch).  The first solves of a launch are
//           dealt over the CTAs; the later ones are made by the CTA that
//           flushed the last chunk of the disc's previous step, so that no
//           disc waits for another and one disc's solve runs beside the
//           others' particles.
//   push    every CTA takes its chunks of particles (one disc each), step by
//           step; it waits (bounded) for the disc's ready flag, stages the
//           disc's field in shared memory, and for each particle interpolates
//           (grdacc), kicks and drifts (stpgrp), and deposits the new position
//           into shared-memory bins over the disc's mesh, flushed with integer
//           atomics (order-free, deterministic).  The particle sums of the m =
//           2 amplitude go to a per-chunk slot; the CTA that completes the
//           disc's step sums them in chunk order (deterministic FP64) into the
//           A2 series.
// The waits end: all CTAs are resident, each takes its (step, chunk) pairs in
// order, and the solve of a disc's step is made by the CTA that completes the
// step before it, inside that step's work.
// The deposit-only launch (mode 0) makes the initial mass (masset) and A2 at
// step 0.
//
// What bounds the pass: shared-memory atomics and instruction issue.  The
// bins are unsigned 32-bit words (native shared-memory atomics; 64-bit ones
// are compare-and-swap loops): a word that wraps adds 2^32 to the cell in the
// mesh, and a negative weight goes straight to the mesh, so the flushed
// integers are the exact 64-bit sums.  Half the bins' size also lets two CTAs
// share an SM when the grid is small enough.  16 discs, 2M particles on 64 x
// 128: 87.0 us a step with one launch per step, 64-bit bins and the solves
// before the pushes, 60.1 so.
#include <algorithm>
#include <vector>

#include "gx_common.cuh"

#define ENS_FIXQ 1048576.0f  // 2^20
#define ENS_MAXACT 64
#define ENS_SPIN (1u << 24)
#define ENS_TUNE_REPS 3
#define ENS_MAXSTEPS 64  // steps per launch
// series entries past max_steps that the tuner's trial steps may write
#define ENS_SPARE (2 + ENS_TUNE_REPS + 1)

struct GxEnsemble {
    GxCtx* ctx = nullptr;  // geometry, Green table, active harmonics, stream
    std::string err;
    int ndisc = 0;
    int64_t ntot = 0;
    std::vector<int64_t> off;  // disc offsets [ndisc + 1]
    int max_steps = 0;
    int64_t steps_done = 0;
    float* P = nullptr;                  // SoA [4][ntot]: x, y, vx, vy
    float* pm = nullptr;                 // particle mass of each disc
    unsigned long long* mass64 = nullptr;  // [ndisc][mesh] fixed point
    float2* field = nullptr;             // [ndisc][mesh] (fx, fy)
    int32_t* chunks = nullptr;           // [nchunks][3]: disc, start, end
    int32_t* dchunk = nullptr;           // [ndisc + 1] first chunk of each disc
    double* a2part = nullptr;            // [nchunks][3]: sum cos 2phi, sum sin 2phi, count
    double* series = nullptr;            // [max_steps + ENS_SPARE][ndisc][2]
    uint32_t* ctl = nullptr;             // [0] entries recorded, [1] CTAs done, [2 + d] ready epoch,
                                         // [2 + ndisc + d] chunks done of the disc's current step
    float* tw = nullptr;                 // twiddle tables (ens_tables)
    // tuning and launch
    int threads = 512, chunk = 16384, nchunks = 0, grid = 0, nchunks_cap = 0;
    size_t smem = 0;
    float last_ms = 0.f;
    int64_t launches = 0;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
};

struct EnsArgs {
    DevGeo g;
    int ndisc, nact, nchunks, mode, tmask;
    float* P;
    int64_t ntot;
    const float* pm;
    unsigned long long* mass64;
    float2* field;
    const int32_t* chunks;
    const int32_t* dchunk;
    double* a2part;
    double* series;
    uint32_t* ctl;
    int32_t* errword;
    const float* green;
    const float* tw;
    int act_m[ENS_MAXACT];
};

// twiddle tables [4][nact][na]: forward cos, forward -sin (p2manl's FFTPACK
// signs), synthesis cosine and sine weights scaled by 1/na (p2fsyn.f)
__global__ void k_ens_tables(DevGeo g, int nact, const int* __restrict__ mlist, float* __restrict__ tw) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int na = g.na;
    if (i >= nact * na) return;
    const int a = i / na, j = i - a * na, m = mlist[a];
    const int idx = (int)(((int64_t)m * j) % na);
    float sn, cs;
    sincospif(2.0f * (float)idx / (float)na, &sn, &cs);
    const float scale = 1.0f / (float)na;
    float tc, ts;
    if (m == 0) {
        tc = 1.f;
        ts = 0.f;
    } else if (m == g.mmax - 1) {
        tc = (j & 1) ? -1.f : 1.f;
        ts = 0.f;
    } else {
        tc = 2.f * cs;
        ts = -2.f * sn;
    }
    const size_t pl = (size_t)nact * na;
    tw[i] = cs;
    tw[pl + i] = -sn;
    tw[2 * pl + i] = tc * scale;
    tw[3 * pl + i] = ts * scale;
}

// ---------------------------------------------------------------------------
// field solve of disc d by the whole CTA (p2fndf.f:25-66 with polcat).  The
// sums of each output run in the same order on any number of threads; the
// threads share operands instead: a forward thread takes ENS_FH harmonics of
// one ring, a contraction thread both components, a synthesis thread two
// rings, which cuts the shared-memory reads that bounded each phase.
#define ENS_FH 3
struct __align__(16) EnsTw {
    float2 f[4];  // (cos, -sin) of harmonics ENS_FH g .. + 2 (one unused)
};

// floats of the solve's workspace: M, forward twiddles [groups][na][8], S, O
__host__ __device__ __forceinline__ size_t ens_solve_floats(int nr, int na, int nact) {
    const size_t ng = (nact + ENS_FH - 1) / ENS_FH;
    return (((size_t)nr * (na + 1) + 3) & ~(size_t)3) + ng * na * 8 + 2 * (size_t)nact * nr + 4 * (size_t)nact * nr;
}

__device__ void ens_solve(const EnsArgs& A, int d, float* sm) {
    const DevGeo& g = A.g;
    const int nr = g.nr, na = g.na, nact = A.nact, mesh = g.mesh;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int ldm = na + 1;
    const size_t pl = (size_t)nact * na;
    const int ngr = (nact + ENS_FH - 1) / ENS_FH;
    float* M = sm;                                                               // [nr][na + 1]
    EnsTw* Tw = reinterpret_cast<EnsTw*>(M + (((size_t)nr * ldm + 3) & ~(size_t)3));  // [ngr][na]
    float2* S = reinterpret_cast<float2*>(Tw + (size_t)ngr * na);                // [nact][nr]: (a_m, b_m)
    float4* O = reinterpret_cast<float4*>(S + (size_t)nact * nr + ((nact * nr) & 1));  // [nact][nr]: (W_c, W_s) of fr, ftheta
    unsigned long long* m64 = A.mass64 + (size_t)d * mesh;
    const float pmass = A.pm[d];
    // integer mass -> FP32 x pmass (scaled.f:89-92); the integers are cleared
    // for the deposit of this step.  Read past the first-level cache: other
    // SMs' atomics made them.
    for (int ir = warp; ir < nr; ir += nw) {
#pragma unroll 4
        for (int j = 2 * lane; j < na; j += 64) {
            ulonglong2* q = reinterpret_cast<ulonglong2*>(m64 + (size_t)ir * na + j);
            const ulonglong2 v = __ldcg(q);
            *q = make_ulonglong2(0ull, 0ull);
            M[ir * ldm + j] = (float)((double)(long long)v.x * (1.0 / (double)ENS_FIXQ)) * pmass;
            M[ir * ldm + j + 1] = (float)((double)(long long)v.y * (1.0 / (double)ENS_FIXQ)) * pmass;
        }
    }
    for (int i = threadIdx.x; i < ngr * na; i += blockDim.x) {
        const int gq = i / na, j = i - gq * na;
        EnsTw t;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int a = gq * ENS_FH + k;
            t.f[k] = (k < ENS_FH && a < nact) ? make_float2(__ldg(A.tw + (size_t)a * na + j), __ldg(A.tw + pl + (size_t)a * na + j))
                                              : make_float2(0.f, 0.f);
        }
        Tw[i] = t;
    }
    __syncthreads();
    // forward transform per ring (p2manl.f:32-45): a_m = sum x cos, b_m = -sum x sin
    {
        // groups of harmonics, then the FP64 sums of m = 0 (in spoke order)
        const int n0 = A.act_m[0] == 0 ? nr : 0;
        const int ng32 = (ngr * nr + 31) & ~31;
        for (int o = threadIdx.x; o < ng32 + n0; o += blockDim.x) {
            if (o >= ng32) {
                const int ir = o - ng32;
                const float* row = M + (size_t)ir * ldm;
                double s = 0.0;
#pragma unroll 8
                for (int j = 0; j < na; j++) s += (double)row[j];
                S[ir] = make_float2((float)s, 0.f);
            } else if (o < ngr * nr) {
                const int gq = o / nr, ir = o - gq * nr;
                const float* row = M + (size_t)ir * ldm;
                const EnsTw* t = Tw + (size_t)gq * na;
                float ca[ENS_FH], sa[ENS_FH];
#pragma unroll
                for (int k = 0; k < ENS_FH; k++) ca[k] = sa[k] = 0.f;
#pragma unroll 4
                for (int j = 0; j < na; j++) {
                    const float x = row[j];
#pragma unroll
                    for (int k = 0; k < ENS_FH; k++) {
                        ca[k] = fmaf(x, t[j].f[k].x, ca[k]);
                        sa[k] = fmaf(x, t[j].f[k].y, sa[k]);
                    }
                }
#pragma unroll
                for (int k = 0; k < ENS_FH; k++) {
                    const int a = gq * ENS_FH + k;
                    if (a < nact && A.act_m[a] != 0) S[(size_t)a * nr + ir] = make_float2(ca[k], sa[k]);
                }
            }
        }
    }
    __syncthreads();
    // radial contraction (p2conv.f:114-181): fr uses (G.M_c, G.M_s), ftheta
    // (+G.M_s, -G.M_c); Green rows of source ring is, columns of field ring ir
    for (int o = threadIdx.x; o < nact * nr; o += blockDim.x) {
        const int a = o / nr, ir = o - a * nr;
        const int m = A.act_m[a];
        const bool v0 = (A.tmask & 1) != 0;
        const bool v1 = ((A.tmask >> 1) & 1) && (m >= 1) && (m <= min(g.ng, g.mmax - 1) - 1);
        const float* G0 = A.green + ((size_t)m * g.nkz) * nr * (size_t)nr + ir;
        const float* G1 = A.green + (((size_t)g.ng + m) * g.nkz) * nr * (size_t)nr + ir;
        const float2* Sa = S + (size_t)a * nr;
        float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
        float wc = 0.f, ws = 0.f;
        if (v0 && v1) {
            // both tables' loads in flight together
#pragma unroll 8
            for (int is = 0; is < nr; is++) {
                const float g0 = __ldg(G0 + (size_t)is * nr), g1 = __ldg(G1 + (size_t)is * nr);
                const float2 sv = Sa[is];
                w.x = fmaf(g0, sv.x, w.x);
                w.y = fmaf(g0, sv.y, w.y);
                wc = fmaf(g1, sv.x, wc);
                ws = fmaf(g1, sv.y, ws);
            }
        } else if (v0 || v1) {
            const float* G = v0 ? G0 : G1;
            float c0 = 0.f, s0 = 0.f;
#pragma unroll 8
            for (int is = 0; is < nr; is++) {
                const float gv = __ldg(G + (size_t)is * nr);
                const float2 sv = Sa[is];
                c0 = fmaf(gv, sv.x, c0);
                s0 = fmaf(gv, sv.y, s0);
            }
            if (v0) {
                w.x = c0;
                w.y = s0;
            } else {
                wc = c0;
                ws = s0;
            }
        }
        if (v1) {
            w.z = ws;
            w.w = -wc;
        }
        O[o] = w;
    }
    __syncthreads();
    // synthesis (p2fsyn.f:34-56, 1/na) and polcat (polcat.f:22-41):
    // f(j) = C + S, f(na - j) = C - S; a warp takes two rings, its lanes spokes
    const float* TC = A.tw + 2 * pl;
    const float* TS = A.tw + 3 * pl;
    const int half = na / 2, nj = half + 1, njb = (nj + 31) >> 5, nrp = (nr + 1) >> 1;
    float2* F = A.field + (size_t)d * mesh;
    for (int o = warp; o < njb * nrp; o += nw) {
        const int jb = o / nrp, ip = o - jb * nrp, j = jb * 32 + lane;
        const int i0 = 2 * ip, i1 = min(2 * ip + 1, nr - 1);
        if (j >= nj) continue;
        float c[2][2] = {{0.f, 0.f}, {0.f, 0.f}}, sn2[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll 3
        for (int a = 0; a < nact; a++) {
            const float tc = __ldg(TC + (size_t)a * na + j), ts = __ldg(TS + (size_t)a * na + j);
            const float4 w0 = O[(size_t)a * nr + i0], w1 = O[(size_t)a * nr + i1];
            c[0][0] = fmaf(w0.x, tc, c[0][0]);
            sn2[0][0] = fmaf(w0.y, ts, sn2[0][0]);
            c[0][1] = fmaf(w0.z, tc, c[0][1]);
            sn2[0][1] = fmaf(w0.w, ts, sn2[0][1]);
            c[1][0] = fmaf(w1.x, tc, c[1][0]);
            sn2[1][0] = fmaf(w1.y, ts, sn2[1][0]);
            c[1][1] = fmaf(w1.z, tc, c[1][1]);
            sn2[1][1] = fmaf(w1.w, ts, sn2[1][1]);
        }
        float sn, cs;
        sincospif(2.0f * (float)j / (float)na, &sn, &cs);
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int ir = 2 * ip + u;
            if (ir >= nr) continue;
            {
                const float fr = c[u][0] + sn2[u][0], ft = c[u][1] + sn2[u][1];
                F[(size_t)ir * na + j] = make_float2(fr * cs - ft * sn, fr * sn + ft * cs);
            }
            if (j > 0 && j < half) {
                const float fr = c[u][0] - sn2[u][0], ft = c[u][1] - sn2[u][1];
                F[(size_t)ir * na + (na - j)] = make_float2(fr * cs + ft * sn, -fr * sn + ft * cs);
            }
        }
    }
}

// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t ens_ld_acquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void ens_st_release(uint32_t* p, uint32_t v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// the field of disc d for the step of epoch e, by the whole CTA
__device__ __forceinline__ void ens_publish(const EnsArgs& A, int d, uint32_t e, unsigned char* sm) {
    ens_solve(A, d, reinterpret_cast<float*>(sm));
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        ens_st_release(&A.ctl[2 + d], e);
    }
    __syncthreads();
}

// mode 0: deposit at the current positions (masset) and A2; mode 1: nsteps steps
template <int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) k_ens_step(EnsArgs A, int nsteps) {
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ uint32_t s_epoch;
    __shared__ int s_last;
    __shared__ double red[2][32];
    __shared__ int redn[32];
    const DevGeo& g = A.g;
    const int mesh = g.mesh;
    if (threadIdx.x == 0) s_epoch = ens_ld_acquire(&A.ctl[0]) + 1u;
    __syncthreads();
    const uint32_t epoch0 = s_epoch;

    // ---- the first step's field solves
    if (A.mode == 1)
        for (int d = blockIdx.x; d < A.ndisc; d += gridDim.x) ens_publish(A, d, epoch0, smraw);

    // ---- particle chunks, step by step
    float2* F = reinterpret_cast<float2*>(smraw);          // [mesh]
    uint32_t* bins = reinterpret_cast<uint32_t*>(F + mesh);  // [mesh]
    bool clean = false;  // the bins are zero
    float* X = A.P;
    float* Y = A.P + A.ntot;
    float* VX = A.P + 2 * A.ntot;
    float* VY = A.P + 3 * A.ntot;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int k = 0; k < nsteps; k++) {
        const uint32_t epoch = epoch0 + (uint32_t)k;
        for (int c = blockIdx.x; c < A.nchunks; c += gridDim.x) {
            const int d = A.chunks[3 * c], s0 = A.chunks[3 * c + 1], s1 = A.chunks[3 * c + 2];
            unsigned long long* m64 = A.mass64 + (size_t)d * mesh;
            if (!clean)
                for (int i = threadIdx.x; i < mesh; i += blockDim.x) bins[i] = 0u;
            if (A.mode == 1) {
                if (threadIdx.x == 0) {
                    uint32_t it = 0;
                    while ((int32_t)(ens_ld_acquire(&A.ctl[2 + d]) - epoch) < 0) {
                        if (++it > ENS_SPIN) {
                            atomicExch(A.errword, 4);
                            break;
                        }
                        __nanosleep(100);
                    }
                }
                __syncthreads();
                const float4* src = reinterpret_cast<const float4*>(A.field + (size_t)d * mesh);
#pragma unroll 4
                for (int i = threadIdx.x; i < mesh / 2; i += blockDim.x)
                    reinterpret_cast<float4*>(F)[i] = __ldcg(src + i);
            }
            __syncthreads();
            double sc = 0.0, ss = 0.0;
            int sn = 0;
            for (int p = s0 + threadIdx.x; p < s1; p += blockDim.x) {
                float x = X[p], y = Y[p];
                if (A.mode == 1) {
                    float vx = VX[p], vy = VY[p];
                    // grdacc.f:40-84 at the old position, halo (frhalo.f:55-56);
                    // the interpolation cell from the fast FP32 arithmetic, as the
                    // single-disc pass forms it (the field is continuous across a
                    // cell boundary, so a cell off by rounding changes nothing)
                    const CellW cw = gx_cell_t<false, 2>(g, x, y, 0.f, true);
                    float ax = 0.f, ay = 0.f;
                    if (cw.key >= 0) {
                        float w[8];
                        int ic[8];
                        gx_weights<2>(g, cw, w);
                        gx_corners_rt<2>(g, cw.key, cw.jt, ic);
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            if (ic[q] < 0) continue;
                            const float2 f = F[ic[q]];
                            ax += f.x * w[q];
                            ay += f.y * w[q];
                        }
                    }
                    if (cw.key >= 0) {
                        float az = 0.f, ph = 0.f;
                        gx_rigid_force(g, x, y, 0.f, ax, ay, az, ph);
                    }
                    // stpgrp.f:26-32
                    vx += ax;
                    vy += ay;
                    x += vx;
                    y += vy;
                    X[p] = x;
                    Y[p] = y;
                    VX[p] = vx;
                    VY[p] = vy;
                }
                // massgn.f:68-89 at the new position
                const CellW cn = gx_cell_t<true, 2>(g, x, y, 0.f, false);
                if (cn.key >= 0) {
                    float w[8];
                    int ic[8];
                    gx_weights<2>(g, cn, w);
                    gx_corners_rt<2>(g, cn.key, cn.jt, ic);
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if (ic[q] >= 0) {
                            // round(w 2^20), ties to even, by one FMA with 1.5 2^23
                            const int v = __float_as_int(fmaf(w[q], ENS_FIXQ, 12582912.0f)) - 0x4B400000;
                            if (v >= 0) {
                                const uint32_t o = atomicAdd(&bins[ic[q]], (uint32_t)v);
                                if (o + (uint32_t)v < o) atomicAdd(&m64[ic[q]], 1ull << 32);  // the word wrapped
                            } else {
                                atomicAdd(&m64[ic[q]], (unsigned long long)(long long)v);
                            }
                        }
                    const double xd = x, yd = y, r2 = xd * xd + yd * yd;
                    if (r2 > 0.0) {
                        const double inv = 1.0 / r2;
                        sc += (xd * xd - yd * yd) * inv;
                        ss += 2.0 * xd * yd * inv;
                    }
                    sn++;
                }
            }
            // chunk sums of the m = 2 amplitude (fixed order: deterministic)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                sc += __shfl_down_sync(0xffffffffu, sc, o);
                ss += __shfl_down_sync(0xffffffffu, ss, o);
                sn += __shfl_down_sync(0xffffffffu, sn, o);
            }
            if (lane == 0) {
                red[0][warp] = sc;
                red[1][warp] = ss;
                redn[warp] = sn;
            }
            __syncthreads();
            // flush the chunk's integer mass (integer atomics: order-free)
            for (int i = threadIdx.x; i < mesh; i += blockDim.x) {
                const uint32_t v = bins[i];
                if (v) {
                    atomicAdd(&m64[i], (unsigned long long)v);
                    bins[i] = 0u;
                }
            }
            clean = true;
            if (threadIdx.x == 0) {
                double a = 0.0, b = 0.0, n = 0.0;
                for (int w = 0; w < nw; w++) {
                    a += red[0][w];
                    b += red[1][w];
                    n += (double)redn[w];
                }
                A.a2part[3 * c] = a;
                A.a2part[3 * c + 1] = b;
                A.a2part[3 * c + 2] = n;
            }
            __syncthreads();
            // the CTA that completes the disc's step records its A2 and makes
            // its next field
            if (threadIdx.x == 0) {
                __threadfence();
                const int nc = A.dchunk[d + 1] - A.dchunk[d];
                const uint32_t prev = atomicAdd(&A.ctl[2 + A.ndisc + d], 1u);
                s_last = (prev == (uint32_t)nc - 1u) ? 1 : 0;
                if (s_last) {
                    __threadfence();
                    A.ctl[2 + A.ndisc + d] = 0u;
                }
            }
            __syncthreads();
            if (s_last) {
                if (threadIdx.x < 32) {
                    // the chunk slots loaded by a warp, added in chunk order
                    double a = 0.0, b = 0.0, n = 0.0;
                    const int q1 = A.dchunk[d + 1];
                    for (int q0 = A.dchunk[d]; q0 < q1; q0 += 32) {
                        const int q = q0 + lane;
                        const double pa = q < q1 ? __ldcg(&A.a2part[3 * q]) : 0.0;
                        const double pb = q < q1 ? __ldcg(&A.a2part[3 * q + 1]) : 0.0;
                        const double pn = q < q1 ? __ldcg(&A.a2part[3 * q + 2]) : 0.0;
                        for (int u = 0; u < min(32, q1 - q0); u++) {
                            a += __shfl_sync(0xffffffffu, pa, u);
                            b += __shfl_sync(0xffffffffu, pb, u);
                            n += __shfl_sync(0xffffffffu, pn, u);
                        }
                    }
                    if (lane == 0) {
                        double* out = A.series + ((size_t)(epoch - 1) * A.ndisc + d) * 2;
                        out[0] = (n > 0.0) ? a / n : 0.0;
                        out[1] = (n > 0.0) ? b / n : 0.0;
                    }
                }
                if (k + 1 < nsteps) {
                    ens_publish(A, d, epoch + 1u, smraw);
                    clean = false;
                }
            }
        }
    }

    // ---- the last CTA to finish records the steps
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const uint32_t prev = atomicAdd(&A.ctl[1], 1u);
        if (prev == gridDim.x - 1) {
            A.ctl[1] = 0u;
            __threadfence();
            ens_st_release(&A.ctl[0], epoch0 + (uint32_t)nsteps - 1u);
        }
    }
}

// ---------------------------------------------------------------------------
// host side
#define ENS_CUDA(e, call)                                                    \
    do {                                                                     \
        cudaError_t e_ = (call);                                             \
        if (e_ != cudaSuccess) {                                             \
            (e)->err = std::string(#call) + ": " + cudaGetErrorString(e_);   \
            cudaGetLastError(); /* reported here, not by the next launch */  \
            return GX_ERR_CUDA;                                              \
        }                                                                    \
    } while (0)

static std::string g_ens_err;

__global__ void k_ens_aos_to_soa(const float* __restrict__ aos, float* __restrict__ P, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int k = 0; k < 4; k++) P[k * n + i] = aos[4 * i + k];
}
__global__ void k_ens_soa_to_aos(const float* __restrict__ P, float* __restrict__ aos, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int k = 0; k < 4; k++) aos[4 * i + k] = P[k * n + i];
}

// the kernel of a block size: 1024 threads take the SM alone, smaller blocks
// share it with the same 64 registers a thread
static const void* ens_kernel(int threads) {
    return threads > 512 ? (const void*)k_ens_step<1024, 1> : (const void*)k_ens_step<512, 2>;
}

// chunk table for the current chunk size, launch geometry for the current
// block size
static int ens_configure(GxEnsemble* e, int threads, int chunk) {
    GxCtx* c = e->ctx;
    std::vector<int32_t> ch;
    std::vector<int32_t> dc(e->ndisc + 1);
    for (int d = 0; d < e->ndisc; d++) {
        dc[d] = (int32_t)(ch.size() / 3);
        for (int64_t s = e->off[d]; s < e->off[d + 1]; s += chunk) {
            ch.push_back(d);
            ch.push_back((int32_t)s);
            ch.push_back((int32_t)std::min<int64_t>(s + chunk, e->off[d + 1]));
        }
    }
    dc[e->ndisc] = (int32_t)(ch.size() / 3);
    const int nch = (int)(ch.size() / 3);
    if (nch > e->nchunks_cap) {
        if (e->chunks) cudaFree(e->chunks);
        if (e->a2part) cudaFree(e->a2part);
        e->chunks = nullptr;
        e->a2part = nullptr;
        ENS_CUDA(e, cudaMalloc((void**)&e->chunks, sizeof(int32_t) * 3 * std::max(nch, 1)));
        ENS_CUDA(e, cudaMalloc((void**)&e->a2part, sizeof(double) * 3 * std::max(nch, 1)));
        e->nchunks_cap = nch;
    }
    if (nch > 0)
        ENS_CUDA(e, cudaMemcpyAsync(e->chunks, ch.data(), sizeof(int32_t) * ch.size(), cudaMemcpyHostToDevice,
                                    c->stream));
    ENS_CUDA(e, cudaMemcpyAsync(e->dchunk, dc.data(), sizeof(int32_t) * dc.size(), cudaMemcpyHostToDevice,
                                c->stream));
    ENS_CUDA(e, cudaStreamSynchronize(c->stream));
    e->nchunks = nch;
    e->threads = threads;
    e->chunk = chunk;
    const DevGeo& g = c->g;
    const size_t solve = sizeof(float) * (ens_solve_floats(g.nr, g.na, c->spec.nact) + 4);
    const size_t push = (sizeof(float2) + sizeof(uint32_t)) * (size_t)g.mesh;
    e->smem = std::max(solve, push);
    int per_sm = 0, sms = 0;
    const void* kern = ens_kernel(threads);
    ENS_CUDA(e, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)e->smem));
    ENS_CUDA(e, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, e->smem));
    ENS_CUDA(e, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->dev));
    if (per_sm < 1) return e->err = "ensemble step kernel does not fit on an SM", GX_ERR_RANGE;
    e->grid = per_sm * sms;
    return GX_OK;
}

static EnsArgs ens_args(GxEnsemble* e, int mode) {
    GxCtx* c = e->ctx;
    EnsArgs A;
    A.g = c->g;
    A.ndisc = e->ndisc;
    A.nact = c->spec.nact;
    A.nchunks = e->nchunks;
    A.mode = mode;
    A.tmask = 1 | (c->g.ng > 1 ? 2 : 0);
    A.P = e->P;
    A.ntot = e->ntot;
    A.pm = e->pm;
    A.mass64 = e->mass64;
    A.field = e->field;
    A.chunks = e->chunks;
    A.dchunk = e->dchunk;
    A.a2part = e->a2part;
    A.series = e->series;
    A.ctl = e->ctl;
    A.errword = c->errword;
    A.green = c->green32;
    A.tw = e->tw;
    for (int a = 0; a < ENS_MAXACT; a++) A.act_m[a] = (a < c->spec.nact) ? c->spec.m[a] : 0;
    return A;
}

// one cooperative launch of nsteps steps (all CTAs resident: the flag waits
// always end)
static int ens_launch(GxEnsemble* e, int mode, int nsteps = 1) {
    EnsArgs A = ens_args(e, mode);
    void* args[] = {&A, &nsteps};
    ENS_CUDA(e, cudaLaunchCooperativeKernel(ens_kernel(e->threads), dim3((unsigned)e->grid), dim3((unsigned)e->threads),
                                            args, e->smem, e->ctx->stream));
    e->launches++;
    return GX_OK;
}

static int ens_check(GxEnsemble* e) {
    int32_t ew = 0;
    ENS_CUDA(e, cudaMemcpy(&ew, e->ctx->errword, sizeof ew, cudaMemcpyDeviceToHost));
    if (ew) {
        char b[96];
        snprintf(b, sizeof b, "device check raised error word %d", ew);
        e->err = b;
        return GX_ERR_DEVICE;
    }
    return GX_OK;
}

extern "C" {

void gx_ensemble_destroy(GxEnsemble* e) {
    if (!e) return;
    if (e->ctx) {
        cudaSetDevice(e->ctx->dev);
        cudaStreamSynchronize(e->ctx->stream);
    }
    void* ptrs[] = {e->P, e->pm, e->mass64, e->field, e->chunks, e->dchunk, e->a2part, e->series, e->ctl, e->tw};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    if (e->ev0) cudaEventDestroy(e->ev0);
    if (e->ev1) cudaEventDestroy(e->ev1);
    if (e->ctx) gx_destroy(e->ctx);
    delete e;
}

const char* gx_ensemble_last_error(const GxEnsemble* e) { return e ? e->err.c_str() : g_ens_err.c_str(); }

int gx_ensemble_create(const GxConfig* cfg, int ndisc, const int64_t* counts, const float* pmass,
                       const float* coords, int max_steps, GxEnsemble** out) {
    if (!cfg || !counts || !pmass || !out || ndisc < 1 || max_steps < 0) {
        g_ens_err = "null argument or ndisc < 1";
        return GX_ERR_ARG;
    }
    *out = nullptr;
    if (cfg->ndim != 2 || cfg->precision != GX_PREC_MIXED) {
        g_ens_err = "the ensemble runs 2D grids on the mixed path";
        return GX_ERR_ARG;
    }
    int64_t ntot = 0;
    for (int d = 0; d < ndisc; d++) {
        if (counts[d] < 0) {
            g_ens_err = "negative particle count";
            return GX_ERR_ARG;
        }
        ntot += counts[d];
    }
    if (ntot > (int64_t)INT32_MAX - 1) {
        g_ens_err = "more than 2^31 - 2 particles";
        return GX_ERR_RANGE;
    }
    if (ntot > 0 && !coords) {
        g_ens_err = "null coords";
        return GX_ERR_ARG;
    }
    GxEnsemble* e = new GxEnsemble();
    GxConfig c1 = *cfg;
    c1.pmass = 1.0f;
    int rc = gx_grdset(&c1, &e->ctx);
    if (rc) {
        g_ens_err = gx_last_error(nullptr);
        delete e;
        return rc;
    }
    GxCtx* c = e->ctx;
    const DevGeo& g = c->g;
    auto fail = [&](int code) {
        g_ens_err = e->err.empty() ? c->err : e->err;
        gx_ensemble_destroy(e);
        return code;
    };
    if (c->spec.nact > ENS_MAXACT) {
        e->err = "more than 64 active harmonics";
        return fail(GX_ERR_RANGE);
    }
    if ((size_t)g.mesh * (sizeof(float2) + sizeof(unsigned long long)) > 200 * 1024 || (g.mesh & 1)) {
        e->err = "grid too large for the ensemble (16 B per cell of shared memory, 200 KB at most)";
        return fail(GX_ERR_RANGE);
    }
    rc = gx_greenm(c);
    if (rc) return fail(rc);
    e->ndisc = ndisc;
    e->ntot = ntot;
    e->max_steps = max_steps;
    e->off.assign(ndisc + 1, 0);
    for (int d = 0; d < ndisc; d++) e->off[d + 1] = e->off[d] + counts[d];
    cudaStream_t st = c->stream;
    rc = [&]() -> int {
        ENS_CUDA(e, cudaMalloc((void**)&e->P, sizeof(float) * 4 * std::max<int64_t>(ntot, 1)));
        ENS_CUDA(e, cudaMalloc((void**)&e->pm, sizeof(float) * ndisc));
        ENS_CUDA(e, cudaMalloc((void**)&e->mass64, sizeof(unsigned long long) * ndisc * (size_t)g.mesh));
        ENS_CUDA(e, cudaMalloc((void**)&e->field, sizeof(float2) * ndisc * (size_t)g.mesh));
        ENS_CUDA(e, cudaMalloc((void**)&e->dchunk, sizeof(int32_t) * (ndisc + 1)));
        ENS_CUDA(e, cudaMalloc((void**)&e->series, sizeof(double) * 2 * ndisc * ((size_t)max_steps + ENS_SPARE)));
        ENS_CUDA(e, cudaMalloc((void**)&e->ctl, sizeof(uint32_t) * (2 + 2 * (size_t)ndisc)));
        ENS_CUDA(e, cudaMalloc((void**)&e->tw, sizeof(float) * 4 * (size_t)c->spec.nact * g.na));
        ENS_CUDA(e, cudaEventCreate(&e->ev0));
        ENS_CUDA(e, cudaEventCreate(&e->ev1));
        ENS_CUDA(e, cudaMemcpyAsync(e->pm, pmass, sizeof(float) * ndisc, cudaMemcpyHostToDevice, st));
        ENS_CUDA(e, cudaMemsetAsync(e->mass64, 0, sizeof(unsigned long long) * ndisc * (size_t)g.mesh, st));
        ENS_CUDA(e, cudaMemsetAsync(e->ctl, 0, sizeof(uint32_t) * (2 + 2 * (size_t)ndisc), st));
        ENS_CUDA(e, cudaMemsetAsync(e->series, 0, sizeof(double) * 2 * ndisc * ((size_t)max_steps + ENS_SPARE), st));
        int* mlist = nullptr;
        ENS_CUDA(e, cudaMallocAsync((void**)&mlist, sizeof(int) * c->spec.nact, st));
        ENS_CUDA(e, cudaMemcpyAsync(mlist, c->spec.m, sizeof(int) * c->spec.nact, cudaMemcpyHostToDevice, st));
        const int nt = c->spec.nact * g.na;
        k_ens_tables<<<(nt + 255) / 256, 256, 0, st>>>(g, c->spec.nact, mlist, e->tw);
        ENS_CUDA(e, cudaGetLastError());
        ENS_CUDA(e, cudaFreeAsync(mlist, st));
        if (ntot > 0) {
            float* stage = nullptr;
            ENS_CUDA(e, cudaMallocAsync((void**)&stage, sizeof(float) * 4 * ntot, st));
            ENS_CUDA(e, cudaMemcpyAsync(stage, coords, sizeof(float) * 4 * ntot, cudaMemcpyHostToDevice, st));
            k_ens_aos_to_soa<<<(unsigned)((ntot + 255) / 256), 256, 0, st>>>(stage, e->P, ntot);
            ENS_CUDA(e, cudaGetLastError());
            ENS_CUDA(e, cudaFreeAsync(stage, st));
        }
        return GX_OK;
    }();
    if (rc) return fail(rc);
    rc = ens_configure(e, 512, 16384);
    if (rc) return fail(rc);
    // masset: the initial integer mass and A2 at step 0
    rc = ens_launch(e, 0);
    if (rc) return fail(rc);
    if (cudaStreamSynchronize(st) != cudaSuccess) {
        e->err = "initial deposit failed";
        return fail(GX_ERR_CUDA);
    }
    rc = ens_check(e);
    if (rc) return fail(rc);
    *out = e;
    return GX_OK;
}

// nsteps steps in launches of at most ENS_MAXSTEPS
int gx_ensemble_step(GxEnsemble* e, int nsteps) {
    if (!e || nsteps < 0) return GX_ERR_ARG;
    if (e->steps_done + nsteps > e->max_steps) return e->err = "more steps than max_steps", GX_ERR_RANGE;
    GxCtx* c = e->ctx;
    cudaSetDevice(c->dev);
    cudaStream_t st = c->stream;
    e->launches = 0;
    ENS_CUDA(e, cudaEventRecord(e->ev0, st));
    for (int left = nsteps; left > 0; left -= ENS_MAXSTEPS) {
        int rc = ens_launch(e, 1, std::min(left, ENS_MAXSTEPS));
        if (rc) return rc;
    }
    ENS_CUDA(e, cudaEventRecord(e->ev1, st));
    ENS_CUDA(e, cudaEventSynchronize(e->ev1));
    ENS_CUDA(e, cudaEventElapsedTime(&e->last_ms, e->ev0, e->ev1));
    e->steps_done += nsteps;
    return ens_check(e);
}

// autotuner: times each (threads, chunk) candidate over a few steps from a
// snapshot of the state, restores the state, keeps the fastest
int gx_ensemble_tune(GxEnsemble* e, int* threads_out, int* chunk_out) {
    if (!e) return GX_ERR_ARG;
    GxCtx* c = e->ctx;
    cudaSetDevice(c->dev);
    cudaStream_t st = c->stream;
    const DevGeo& g = c->g;
    const size_t pbytes = sizeof(float) * 4 * std::max<int64_t>(e->ntot, 1);
    const size_t mbytes = sizeof(unsigned long long) * e->ndisc * (size_t)g.mesh;
    const size_t cbytes = sizeof(uint32_t) * (2 + 2 * (size_t)e->ndisc);
    char *sp = nullptr, *sm = nullptr, *sc = nullptr;
    ENS_CUDA(e, cudaMalloc((void**)&sp, pbytes));
    ENS_CUDA(e, cudaMalloc((void**)&sm, mbytes));
    ENS_CUDA(e, cudaMalloc((void**)&sc, cbytes));
    ENS_CUDA(e, cudaMemcpyAsync(sp, e->P, pbytes, cudaMemcpyDeviceToDevice, st));
    ENS_CUDA(e, cudaMemcpyAsync(sm, e->mass64, mbytes, cudaMemcpyDeviceToDevice, st));
    ENS_CUDA(e, cudaMemcpyAsync(sc, e->ctl, cbytes, cudaMemcpyDeviceToDevice, st));
    const int cand_t[3] = {256, 512, 1024};
    const int cand_c[4] = {4096, 8192, 16384, 32768};
    float best = 1e30f;
    int bt = e->threads, bc = e->chunk;
    int rc = GX_OK;
    const int reps = ENS_TUNE_REPS;
    for (int it = 0; it < 3 && rc == GX_OK; it++) {
        for (int ic = 0; ic < 4 && rc == GX_OK; ic++) {
            rc = ens_configure(e, cand_t[it], cand_c[ic]);
            if (rc) break;
            // warm-up step, then the timed steps; the series entries they
            // write (at most ENS_TUNE_REPS + 1 past the recorded ones, inside
            // the ENS_SPARE spare entries) are rewritten by later steps
            rc = ens_launch(e, 1);
            if (rc) break;
            ENS_CUDA(e, cudaEventRecord(e->ev0, st));
            rc = ens_launch(e, 1, reps);
            ENS_CUDA(e, cudaEventRecord(e->ev1, st));
            if (rc) break;
            ENS_CUDA(e, cudaEventSynchronize(e->ev1));
            float ms = 0.f;
            ENS_CUDA(e, cudaEventElapsedTime(&ms, e->ev0, e->ev1));
            if (ms < best) {
                best = ms;
                bt = cand_t[it];
                bc = cand_c[ic];
            }
            ENS_CUDA(e, cudaMemcpyAsync(e->P, sp, pbytes, cudaMemcpyDeviceToDevice, st));
            ENS_CUDA(e, cudaMemcpyAsync(e->mass64, sm, mbytes, cudaMemcpyDeviceToDevice, st));
            ENS_CUDA(e, cudaMemcpyAsync(e->ctl, sc, cbytes, cudaMemcpyDeviceToDevice, st));
        }
    }
    ENS_CUDA(e, cudaStreamSynchronize(st));
    cudaFree(sp);
    cudaFree(sm);
    cudaFree(sc);
    if (rc) return rc;
    rc = ens_configure(e, bt, bc);
    if (rc) return rc;
    if (threads_out) *threads_out = bt;
    if (chunk_out) *chunk_out = bc;
    return ens_check(e);
}

int gx_ensemble_config(const GxEnsemble* e, int* threads, int* chunk, int* grid, int* graph) {
    if (!e) return GX_ERR_ARG;
    if (threads) *threads = e->threads;
    if (chunk) *chunk = e->chunk;
    if (grid) *grid = e->grid;
    if (graph) *graph = 0;
    return GX_OK;
}

int gx_ensemble_steps_done(const GxEnsemble* e, int64_t* n) {
    if (!e || !n) return GX_ERR_ARG;
    *n = e->steps_done;
    return GX_OK;
}

int gx_ensemble_a2(GxEnsemble* e, double* out, int64_t cap) {
    if (!e || !out) return GX_ERR_ARG;
    const int64_t need = (e->steps_done + 1) * 2 * (int64_t)e->ndisc;
    if (cap < need) return e->err = "output smaller than (steps_done + 1) * ndisc * 2", GX_ERR_RANGE;
    cudaSetDevice(e->ctx->dev);
    ENS_CUDA(e, cudaMemcpy(out, e->series, sizeof(double) * need, cudaMemcpyDeviceToHost));
    return GX_OK;
}

int gx_ensemble_unload(GxEnsemble* e, float* coords) {
    if (!e || (e->ntot > 0 && !coords)) return GX_ERR_ARG;
    if (e->ntot == 0) return GX_OK;
    GxCtx* c = e->ctx;
    cudaSetDevice(c->dev);
    float* stage = nullptr;
    ENS_CUDA(e, cudaMallocAsync((void**)&stage, sizeof(float) * 4 * e->ntot, c->stream));
    k_ens_soa_to_aos<<<(unsigned)((e->ntot + 255) / 256), 256, 0, c->stream>>>(e->P, stage, e->ntot);
    ENS_CUDA(e, cudaGetLastError());
    ENS_CUDA(e, cudaMemcpyAsync(coords, stage, sizeof(float) * 4 * e->ntot, cudaMemcpyDeviceToHost, c->stream));
    ENS_CUDA(e, cudaFreeAsync(stage, c->stream));
    ENS_CUDA(e, cudaStreamSynchronize(c->stream));
    return GX_OK;
}

int gx_ensemble_last_ms(const GxEnsemble* e, float* ms, int64_t* launches) {
    if (!e) return GX_ERR_ARG;
    if (ms) *ms = e->last_ms;
    if (launches) *launches = e->launches;
    return GX_OK;
}

}  // extern "C"
