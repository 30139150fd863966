// gx_adjoint.cu -- adjoint of the 2D mixed-path step for the objective
// J = |A2(x_T)|, A2 = (1/n) sum_p e^{2 i phi_p} over all particles.
//
// Forward: nsteps of massgn, findf (+ polcat), getacc with the ISOT halo,
// stpgrp (the arithmetic of gx_step, but for the rounding of the halo's force,
// on particles kept in load order), with a checkpoint of (x, v) every
// ckpt_every steps.  Reverse sweep, from the
// final state: the trajectory is recomputed backwards by time reversal,
// x_s = x_{s+1} - v_{s+1}, v_s = v_{s+1} - a(x_s), and reset to the
// checkpoint at every checkpoint step; at each step, with
// mu = lambda_v + lambda_x:
//   lambda_v <- mu
//   lambda_x <- lambda_x + sum_c grad W_c(x) (F_c . mu)        (k_adj_a)
//               + halo Jacobian . mu
//               + pmass sum_c grad W_c(x) psi_c                   (k_adj_b)
// with psi = K^T Q, Q_c = sum_p W_c(x_p) mu_p (FP64 atomics into the mesh)
// and K the linear map mass -> (fx, fy): forward DFT of the active
// harmonics (p2manl.f:32-45), radial contraction (p2conv.f:114-181),
// synthesis (p2fsyn.f:34-56), polcat (polcat.f:22-41); K^T runs those
// steps transposed in reverse order (k_adjt_syn, k_adjt_conv).
// dJ/d(halo_rc, halo_v2) accumulate the halo's parameter derivatives . mu
// per block in FP64.
#include <algorithm>
#include <vector>

#include "gx_common.cuh"

#define ADJ_BS 256
#define ADJ_KEEP ((size_t)2 << 30)

// cell, weights and weight gradients at (x, y) (weight.f:61-101); 2D, one sector
__device__ __forceinline__ bool adj_wgrad(const DevGeo& g, float x, float y, CellW& cw, float* w,
                                          float (*dw)[2]) {
    cw = gx_cell_t<true, 2>(g, x, y, 0.f, true);
    if (cw.key < 0) return false;
    gx_weights<2>(g, cw, w);
    const float r2 = x * x + y * y;
    if (!(r2 > 0.f)) {
        for (int k = 0; k < 4; k++) dw[k][0] = dw[k][1] = 0.f;
        return true;
    }
    const float rr = sqrtf(r2);
    const float dudr = (g.rmap == GX_RMAP_STDPOL) ? g.inv_ua / (1.f + rr) : g.inv_ua / rr;
    const float gu[2] = {dudr * x / rr, dudr * y / rr};
    const float ts = g.t_scale / r2;
    const float gt[2] = {-y * ts, x * ts};
    const float du = cw.du, dt = cw.dt;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        dw[0][i] = -(1.f - dt) * gu[i] - (1.f - du) * gt[i];
        dw[1][i] = -dt * gu[i] + (1.f - du) * gt[i];
        dw[2][i] = (1.f - dt) * gu[i] - du * gt[i];
        dw[3][i] = dt * gu[i] + du * gt[i];
    }
    return true;
}

// acceleration at (x, y) from the Cartesian field and the halo (grdacc + halfrc)
__device__ __forceinline__ void adj_accel(const DevGeo& g, const float4* F, const CellW& cw,
                                          const float* w, float x, float y, float& ax, float& ay) {
    ax = ay = 0.f;
    if (cw.key < 0) return;
    int ic[8];
    gx_corners_rt<2>(g, cw.key, cw.jt, ic);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (ic[k] < 0) continue;
        const float4 f = F[ic[k]];
        ax += f.x * w[k];
        ay += f.y * w[k];
    }
    if (g.halo == 1) {
        // from r, with a square root and two divisions where the step
        // (gx_rigid_force) takes one: the step's form moved the gradients of 400k
        // particles over 100 steps by 1e-5 to 4e-4, to errors of the same size
        const float r2 = x * x + y * y, rr = sqrtf(r2);
        float fr = -g.halo_v2 * rr / (r2 + g.halo_rc2);
        if (fr != 0.f) {
            fr = fr / rr;
            ax += fr * x;
            ay += fr * y;
        }
    }
}

// particles in load order from the context's storage order, one record
// (x, y, vx, vy) of 16 bytes each
__global__ void k_adj_gather(const float* __restrict__ Pc, int64_t cap, int64_t n,
                             const int32_t* __restrict__ origin, float4* __restrict__ S) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    S[origin[i]] = make_float4(Pc[i], Pc[cap + i], Pc[2 * cap + i], Pc[3 * cap + i]);
}

// massgn of one particle at (x, y): its four weights as the 2^-20 integers of
// gx_deposit.cu, added straight into the int64 mesh accumulator (integer
// sums: the same mass whatever the order), and its ring into [rlo, rhi]
__device__ __forceinline__ void adj_deposit(const DevGeo& g, float x, float y, unsigned long long* __restrict__ acc,
                                            int& rlo, int& rhi) {
    const CellW cw = gx_cell_t<true, 2>(g, x, y, 0.f, false);
    if (cw.key < 0) return;
    rlo = min(rlo, cw.row);
    rhi = max(rhi, cw.row);
    float w[8];
    int ic[8];
    gx_weights<2>(g, cw, w);
    gx_corners_rt<2>(g, cw.key, cw.jt, ic);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int v = __float2int_rn(w[k] * 1048576.0f);
        if (ic[k] >= 0 && v) atomicAdd(acc + ic[k], (unsigned long long)(long long)v);
    }
}

// the ring range of a pass (rng[0] first, rng[1] last)
__device__ __forceinline__ void adj_range(int rlo, int rhi, int32_t* __restrict__ rng) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        rlo = min(rlo, __shfl_xor_sync(0xffffffffu, rlo, o));
        rhi = max(rhi, __shfl_xor_sync(0xffffffffu, rhi, o));
    }
    if ((threadIdx.x & 31) == 0 && rhi >= 0) gx_atomic_range(rng, rlo, rhi);
}

// The sweeps' particle passes.  The particles stay in load order (16-byte
// records): a pass waits on its gathers from the L2-resident field and on
// its mesh reductions, not on the order.  Depositing the new position with
// four 64-bit reductions into the accumulator inside the pass replaces a
// pass that keyed the particles, their counting sort, the row deposit, the
// combine and two copies of the positions (50 us a solve at 400k particles,
// 128 x 256; the fused forward pass takes 20.4, 23.7 while every warp queued its
// ring range on two words).

// the mass of the records S (the first solve, and the context's mass afterwards)
__global__ void __launch_bounds__(ADJ_BS) k_adj_mass(DevGeo g, const float4* __restrict__ S, int64_t n,
                                                     unsigned long long* __restrict__ acc,
                                                     int32_t* __restrict__ rng) {
    int rlo = 0x7fffffff, rhi = -1;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float4 s = S[i];
        adj_deposit(g, s.x, s.y, acc, rlo, rhi);
    }
    adj_range(rlo, rhi, rng);
}

// forward step: v += a(x); x += v (stpgrp.f:26-32); the new position deposited
__global__ void __launch_bounds__(ADJ_BS) k_adj_fwd(DevGeo g, float4* __restrict__ S, int64_t n,
                                                    const float4* F,
                                                    unsigned long long* __restrict__ acc,
                                                    int32_t* __restrict__ rng) {
    gx_chain();
    int rlo = 0x7fffffff, rhi = -1;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float4 s = __ldcg(S + i);
        const CellW cw = gx_cell_t<true, 2>(g, s.x, s.y, 0.f, true);
        float w[8];
        if (cw.key >= 0) gx_weights<2>(g, cw, w);
        float ax, ay;
        adj_accel(g, F, cw, w, s.x, s.y, ax, ay);
        s.z += ax;
        s.w += ay;
        s.x += s.z;
        s.y += s.w;
        S[i] = s;
        adj_deposit(g, s.x, s.y, acc, rlo, rhi);
    }
    adj_range(rlo, rhi, rng);
}

// per-block FP64 sums of e^{2 i phi} over all particles
__global__ void k_adj_a2(const float4* __restrict__ S, int64_t n, double* __restrict__ part) {
    __shared__ double sh[2][ADJ_BS / 32];
    double c = 0.0, s = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float4 q = S[i];
        const double x = q.x, y = q.y, r2 = x * x + y * y;
        if (r2 > 0.0) {
            c += (x * x - y * y) / r2;
            s += 2.0 * x * y / r2;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        c += __shfl_down_sync(0xffffffffu, c, o);
        s += __shfl_down_sync(0xffffffffu, s, o);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        sh[0][warp] = c;
        sh[1][warp] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int w = 0; w < ADJ_BS / 32; w++) {
            a += sh[0][w];
            b += sh[1][w];
        }
        part[2 * blockIdx.x] = a;
        part[2 * blockIdx.x + 1] = b;
    }
}

// lambda_x at the final time: dJ/dx_T; lambda_v = 0
__global__ void k_adj_init(const float4* __restrict__ S, int64_t n, double a2r, double a2i, double J,
                           float4* __restrict__ L) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float gx = 0.f, gy = 0.f;
    const float4 q = S[i];
    const double x = q.x, y = q.y, r2 = x * x + y * y;
    if (r2 > 0.0 && J > 0.0) {
        const double fr = (x * x - y * y) / r2, fi = 2.0 * x * y / r2, inv = 1.0 / (double)n;
        // dA2/dx = -2 i f y / (n r2), dA2/dy = 2 i f x / (n r2); dJ = Re(conj(A2) dA2) / J
        const double dxr = 2.0 * fi * y / r2 * inv, dxi = -2.0 * fr * y / r2 * inv;
        const double dyr = -2.0 * fi * x / r2 * inv, dyi = 2.0 * fr * x / r2 * inv;
        gx = (float)((a2r * dxr + a2i * dxi) / J);
        gy = (float)((a2r * dyr + a2i * dyi) / J);
    }
    L[i] = make_float4(gx, gy, 0.f, 0.f);
}

// reverse step, first particle pass at x_s: reverse kick (unless the state
// came from a checkpoint), mu, lambda_v <- mu, lambda_x += interpolation
// slope . (F . mu) + halo Jacobian . mu, Q += W mu (x and y of a cell side
// by side), halo parameter terms
__global__ void __launch_bounds__(ADJ_BS) k_adj_a(DevGeo g, float4* __restrict__ S, float4* __restrict__ L,
                                                  int64_t n, const float4* F, int kick,
                                                  double* __restrict__ Q, double* __restrict__ tpart) {
    gx_chain();
    __shared__ double sh[2][ADJ_BS / 32];
    double drc = 0.0, dv2 = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float4 s = __ldcg(S + i), l = __ldcg(L + i);
        const float x = s.x, y = s.y;
        CellW cw;
        float w[8], dw[4][2];
        const bool on = adj_wgrad(g, x, y, cw, w, dw);
        if (kick) {
            float ax, ay;
            adj_accel(g, F, cw, w, x, y, ax, ay);
            s.z -= ax;
            s.w -= ay;
            S[i] = s;
        }
        float lx = l.x, ly = l.y;
        const float m0 = l.z + lx, m1 = l.w + ly;
        if (on) {
            int ic[8];
            gx_corners_rt<2>(g, cw.key, cw.jt, ic);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (ic[k] < 0) continue;
                const float4 f = F[ic[k]];
                const float fdot = f.x * m0 + f.y * m1;
                lx += dw[k][0] * fdot;
                ly += dw[k][1] * fdot;
                atomicAdd(&Q[2 * ic[k]], (double)(w[k] * m0));
                atomicAdd(&Q[2 * ic[k] + 1], (double)(w[k] * m1));
            }
            if (g.halo == 1) {
                // h = -v2 x / d, d = r^2 + rc^2: Jacobian -v2 (I / d - 2 x x^T / d^2)
                const float d = x * x + y * y + g.halo_rc2, v2 = g.halo_v2;
                const float hxx = -v2 * (1.f / d - 2.f * x * x / (d * d));
                const float hyy = -v2 * (1.f / d - 2.f * y * y / (d * d));
                const float hxy = v2 * 2.f * x * y / (d * d);
                lx += hxx * m0 + hxy * m1;
                ly += hxy * m0 + hyy * m1;
                const double xm = (double)x * m0 + (double)y * m1;
                dv2 += -xm / (double)d;
                drc += (double)v2 * 2.0 * sqrt((double)g.halo_rc2) * xm / ((double)d * d);
            }
        }
        L[i] = make_float4(lx, ly, m0, m1);
    }
    for (int o = 16; o > 0; o >>= 1) {
        drc += __shfl_down_sync(0xffffffffu, drc, o);
        dv2 += __shfl_down_sync(0xffffffffu, dv2, o);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        sh[0][warp] = drc;
        sh[1][warp] = dv2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int w = 0; w < ADJ_BS / 32; w++) {
            a += sh[0][w];
            b += sh[1][w];
        }
        // each block owns its slot and the steps run in order: deterministic
        tpart[2 * blockIdx.x] = __ldcg(tpart + 2 * blockIdx.x) + a;
        tpart[2 * blockIdx.x + 1] = __ldcg(tpart + 2 * blockIdx.x + 1) + b;
    }
}

// second particle pass of a reverse step fused with the start of the next:
//   psi (else none yet): lambda_x += pmass sum_c grad W_c(x) psi_c at x_s;
//   move: the reverse drift x_{s-1} = x_s - v_s; with a checkpoint ck its
//   largest |difference| from the reversed position (max of non-negative
//   floats as ordered integers: order-free), then the checkpoint itself; the
//   position deposited for the next solve.
__global__ void __launch_bounds__(ADJ_BS) k_adj_b(DevGeo g, float4* __restrict__ S, float4* __restrict__ L, int64_t n,
                                                  const float* psi, float pmass, int move,
                                                  const float4* __restrict__ ck, unsigned int* __restrict__ drift,
                                                  unsigned long long* __restrict__ acc, int32_t* __restrict__ rng) {
    gx_chain();
    int rlo = 0x7fffffff, rhi = -1;
    float dm = 0.f;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float4 s = __ldcg(S + i);
        if (psi) {
            CellW cw;
            float w[8], dw[4][2];
            if (adj_wgrad(g, s.x, s.y, cw, w, dw)) {
                int ic[8];
                gx_corners_rt<2>(g, cw.key, cw.jt, ic);
                float gx = 0.f, gy = 0.f;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    if (ic[k] < 0) continue;
                    const float p = psi[ic[k]];
                    gx += dw[k][0] * p;
                    gy += dw[k][1] * p;
                }
                float2* l = reinterpret_cast<float2*>(L + i);
                const float2 v = __ldcg(l);
                *l = make_float2(v.x + pmass * gx, v.y + pmass * gy);
            }
        }
        if (!move) continue;
        s.x -= s.z;
        s.y -= s.w;
        if (ck) {
            const float4 c = __ldcg(ck + i);
            dm = fmaxf(dm, fmaxf(fabsf(s.x - c.x), fabsf(s.y - c.y)));
            s = c;
        }
        S[i] = s;
        adj_deposit(g, s.x, s.y, acc, rlo, rhi);
    }
    if (!move) return;
    adj_range(rlo, rhi, rng);
    if (ck) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dm = fmaxf(dm, __shfl_xor_sync(0xffffffffu, dm, o));
        if ((threadIdx.x & 31) == 0 && dm > 0.f) atomicMax(drift, __float_as_uint(dm));
    }
}

// ---------------------------------------------------------------------------
// K^T.  Synthesis weights of harmonic m at spoke j: c_m(j) = 1 (m = 0),
// (-1)^j (m = na/2), 2 cos(2 pi m j / na) otherwise; s_m(j) = -2 sin(...)
// (0 for m = 0, na/2); scale 1/na (p2fsyn.f:42-53).
struct AdjAct {
    int m[64];
};

// polcat^T and synthesis^T: V[t][a][ir] = scale sum_j g_t(ir, j) (c_m(j), s_m(j)).
// One ring per CTA; thread (a, q) sums both components of harmonic a (of a
// block of AT_H) over the spokes j = q (mod AT_Q), with the forward table
// T[j][2a] = cos, T[j][2a + 1] = -sin (k_fwdtab) read through L1, the AT_Q
// partials added in q order.  Q is cleared for the next step.  The sums are
// latency-bound chains: one thread per output (2304 of them at 128 x 256, m =
// 0..8, sines evaluated in place) took 97 us, this split takes 5.5.
#define AT_H 16
#define AT_Q 16
__global__ void __launch_bounds__(AT_H * AT_Q) k_adjt_syn(DevGeo g, AdjAct act, int nact, int ncp,
                                                          double2* __restrict__ Q, const float* __restrict__ T,
                                                          float2* __restrict__ V) {
    gx_chain();
    extern __shared__ __align__(16) float2 gv[];  // [na]: radial, azimuthal
    __shared__ float4 part[AT_Q][AT_H];
    const int nr = g.nr, na = g.na, ir = blockIdx.x;
    for (int j = threadIdx.x; j < na; j += blockDim.x) {
        double2* q = Q + (size_t)ir * na + j;
        const double2 qv = __ldcg(q);
        const float qx = (float)qv.x, qy = (float)qv.y;
        *q = make_double2(0.0, 0.0);
        float sn, cs;
        sincospif(2.0f * (float)j / (float)na, &sn, &cs);
        gv[j] = make_float2(qx * cs + qy * sn, -qx * sn + qy * cs);
    }
    __syncthreads();
    const int h = threadIdx.x % AT_H, q = threadIdx.x / AT_H;
    const float scale = 1.0f / (float)na;
    for (int a0 = 0; a0 < nact; a0 += AT_H) {
        const int a = a0 + h;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        if (a < nact) {
#pragma unroll 4
            for (int j = q; j < na; j += AT_Q) {
                const float2 t = __ldg(reinterpret_cast<const float2*>(T + (size_t)j * ncp + 2 * a));
                const float2 v = gv[j];
                s.x += v.x * t.x;
                s.y += v.x * t.y;
                s.z += v.y * t.x;
                s.w += v.y * t.y;
            }
        }
        part[q][h] = s;
        __syncthreads();
        if (threadIdx.x < AT_H && a < nact) {
            float4 v = part[0][threadIdx.x];
            for (int k = 1; k < AT_Q; k++) {
                const float4 p = part[k][threadIdx.x];
                v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w;
            }
            const int m = act.m[a];
            const bool two = m > 0 && m < g.mmax - 1;
            const float f = two ? 2.f * scale : scale, fs = two ? f : 0.f;
            V[(size_t)a * nr + ir] = make_float2(f * v.x, fs * v.y);
            V[((size_t)nact + a) * nr + ir] = make_float2(f * v.z, fs * v.w);
        }
        __syncthreads();
    }
}

// radial contraction^T and forward DFT^T of one source ring per CTA: AB =
// (A, B) of each harmonic, one warp per harmonic over the field rings; then
// psi(is, j) = sum_a A cos(2 pi m j / na) - B sin(...)
__global__ void __launch_bounds__(ADJ_BS) k_adjt_conv(DevGeo g, AdjAct act, int nact, int ncp,
                                                      const float* __restrict__ G, const float2* __restrict__ V,
                                                      const float* __restrict__ T, float* __restrict__ psi) {
    gx_chain();
    __shared__ float2 AB[64];
    const int lane = threadIdx.x & 31, nr = g.nr, na = g.na, is = blockIdx.x;
    for (int a = threadIdx.x >> 5; a < nact; a += ADJ_BS / 32) {
        const int m = act.m[a];
        const bool hasb = (m > 0 && m < g.mmax - 1);
        const bool ft = (g.ng > 1) && (m >= 1) && (m <= min(g.ng, g.mmax - 1) - 1);
        const float* G0 = G + ((size_t)(0 * g.ng + m) * g.nkz) * nr * (size_t)nr + (size_t)is * nr;
        const float* G1 = G + ((size_t)(1 * g.ng + m) * g.nkz) * nr * (size_t)nr + (size_t)is * nr;
        const float2* V0 = V + (size_t)a * nr;
        const float2* V1 = V + ((size_t)nact + a) * nr;
        float sa = 0.f, sb = 0.f;
#pragma unroll 4
        for (int ir = lane; ir < nr; ir += 32) {
            const float g0 = __ldg(G0 + ir);
            const float2 v0 = __ldcg(V0 + ir);
            sa += g0 * v0.x;
            if (hasb) sb += g0 * v0.y;
            if (ft) {
                const float g1 = __ldg(G1 + ir);
                const float2 v1 = __ldcg(V1 + ir);
                sb += g1 * v1.x;
                sa -= g1 * v1.y;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            sa += __shfl_down_sync(0xffffffffu, sa, o);
            sb += __shfl_down_sync(0xffffffffu, sb, o);
        }
        if (lane == 0) AB[a] = make_float2(sa, hasb ? sb : 0.f);
    }
    __syncthreads();
    for (int j = threadIdx.x; j < na; j += ADJ_BS) {
        float s = 0.f;
        for (int a = 0; a < nact; a++) {
            const float2 t = __ldg(reinterpret_cast<const float2*>(T + (size_t)j * ncp + 2 * a));
            s += AB[a].x * t.x + AB[a].y * t.y;
        }
        psi[(size_t)is * na + j] = s;
    }
}

// ---------------------------------------------------------------------------
__global__ void k_adj_scatter(const float4* __restrict__ S, int64_t n, float* __restrict__ Pc, int64_t cap,
                              int32_t* __restrict__ origin, int32_t* __restrict__ perm) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 s = S[i];
    Pc[i] = s.x;
    Pc[cap + i] = s.y;
    Pc[2 * cap + i] = s.z;
    Pc[3 * cap + i] = s.w;
    origin[i] = (int32_t)i;
    perm[i] = (int32_t)i;
}

// the deposited accumulator -> the mass, then its field
static int adj_solve(GxCtx* c) {
    c->zr_valid = false;  // the mass array is no longer a fused pass's
    int rc = gx_mass_defer(c);
    if (rc) return rc;
    return gx_mixed_findf(c, 0, true);
}

static int adj_run(GxCtx* c, int nsteps, int ckpt_every, double* J_out, float* grad, double* dtheta,
                   float* drift_out) {
    if (!c || nsteps < 0 || ckpt_every < 1 || !J_out || !grad || !dtheta) return GX_ERR_ARG;
    if (c->fp64 || c->g.ndim != 2 || c->g.nsect != 1)
        return c->err = "the adjoint runs 2D one-sector grids on the mixed path", GX_ERR_ARG;
    if (c->nzones > 1) return c->err = "the adjoint runs a single time-step zone", GX_ERR_ARG;
    if (c->g.halo > 1) return c->err = "the adjoint differentiates the ISOT halo only", GX_ERR_ARG;
    if (!c->have_green) return c->err = "no Green table (call gx_greenm)", GX_ERR_STATE;
    if (c->spec.nact > 64) return c->err = "more than 64 active harmonics", GX_ERR_RANGE;
    const int64_t n = c->n;
    if (n < 1) return c->err = "no particles loaded", GX_ERR_STATE;
    if (nsteps > 0 && c->spec.nact == 0) return c->err = "no active harmonics", GX_ERR_ARG;  // (as the solve)
    cudaSetDevice(c->dev);
    {
        const int rc = gx_dense(c);
        if (rc) return rc;
    }
    const DevGeo& g = c->g;
    const int nact = c->spec.nact, ncp = (2 * nact + 3) & ~3;  // row of the forward table (gx_solve.cu)
    AdjAct act;
    for (int a = 0; a < 64; a++) act.m[a] = (a < nact) ? c->spec.m[a] : 0;
    const unsigned nb = (unsigned)((n + ADJ_BS - 1) / ADJ_BS);
    const unsigned np = std::min(nb, 148u * 8u);  // CTAs of the strided passes
    const int nck = nsteps / ckpt_every + 1;
    // the sweeps' buffers: one block, kept with the context up to ADJ_KEEP
    // bytes until the particle arrays grow (allocating and freeing it in every call:
    // 100 steps of 400k particles 12.6 -> 13.6 ms with 323 MB, and now and then
    // hundreds of ms), and given back by the call above that
    struct {
        float4 *S, *L, *ck;
        double2* Q;
        double *part, *tpart;
        float2* V;
        float* psi;
        unsigned int* drift;
    } b;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += (bytes + 255) & ~(size_t)255;
        return o;
    };
    const size_t oS = take(sizeof(float4) * n), oL = take(sizeof(float4) * n),
                 ock = take(sizeof(float4) * n * (size_t)nck), oQ = take(sizeof(double2) * g.mesh),
                 opart = take(sizeof(double) * 2 * np), otpart = take(sizeof(double) * 2 * np),
                 oV = take(sizeof(float2) * 2 * nact * g.nr), opsi = take(sizeof(float) * g.mesh),
                 odrift = take(sizeof(unsigned int));
    if (off > c->adj_bytes) {
        if (c->adj_ws) cudaFree(c->adj_ws);
        c->adj_ws = nullptr;
        c->adj_bytes = 0;
        GX_CUDA(c, cudaMalloc((void**)&c->adj_ws, off));
        c->adj_bytes = off;
    }
    b.S = (float4*)(c->adj_ws + oS);
    b.L = (float4*)(c->adj_ws + oL);
    b.ck = (float4*)(c->adj_ws + ock);
    b.Q = (double2*)(c->adj_ws + oQ);
    b.part = (double*)(c->adj_ws + opart);
    b.tpart = (double*)(c->adj_ws + otpart);
    b.V = (float2*)(c->adj_ws + oV);
    b.psi = (float*)(c->adj_ws + opsi);
    b.drift = (unsigned int*)(c->adj_ws + odrift);
    cudaStream_t st = c->stream;
    c->launches = 0;
    GX_CUDA(c, cudaEventRecord(c->ev0, st));
    // initial state in load order
    k_adj_gather<<<nb, ADJ_BS, 0, st>>>(c->pbuf[c->cur], c->cap, n, c->origin, b.S);
    GX_LAUNCHED(c);
    const size_t sbytes = sizeof(float4) * n;
    GX_CUDA(c, cudaMemcpyAsync(b.ck, b.S, sbytes, cudaMemcpyDeviceToDevice, st));
    // forward sweep with checkpoints
    if (nsteps > 0) {
        c->have_mass = c->have_field = false;  // the sweeps' from here to the end of the call
        c->acc_open = true;
        k_adj_mass<<<np, ADJ_BS, 0, st>>>(g, b.S, n, c->macc, gx_mass_ranges(c));
        GX_LAUNCHED(c);
    }
    for (int s = 0; s < nsteps; s++) {
        int rc = adj_solve(c);
        if (rc) return rc;
        c->acc_open = true;
        GX_CUDA(c, gx_launch_chain(k_adj_fwd, np, ADJ_BS, 0, st, g, b.S, n, c->field, c->macc, gx_mass_ranges(c)));
        GX_LAUNCHED(c);
        if ((s + 1) % ckpt_every == 0)
            GX_CUDA(c, cudaMemcpyAsync(b.ck + (size_t)((s + 1) / ckpt_every) * n, b.S, sbytes,
                                       cudaMemcpyDeviceToDevice, st));
    }
    if (nsteps > 0) {
        // the last pass deposited the final positions, which no solve takes
        int rc = gx_mass_convert(c);
        if (rc) return rc;
    }
    // objective
    k_adj_a2<<<np, ADJ_BS, 0, st>>>(b.S, n, b.part);
    GX_LAUNCHED(c);
    std::vector<double> hp(2 * (size_t)np);
    GX_CUDA(c, cudaMemcpyAsync(hp.data(), b.part, sizeof(double) * 2 * np, cudaMemcpyDeviceToHost, st));
    GX_CUDA(c, cudaStreamSynchronize(st));
    double sre = 0.0, sim = 0.0;
    for (unsigned i = 0; i < np; i++) {
        sre += hp[2 * i];
        sim += hp[2 * i + 1];
    }
    const double a2r = sre / (double)n, a2i = sim / (double)n;
    const double J = sqrt(a2r * a2r + a2i * a2i);
    k_adj_init<<<nb, ADJ_BS, 0, st>>>(b.S, n, a2r, a2i, J, b.L);
    GX_LAUNCHED(c);
    GX_CUDA(c, cudaMemsetAsync(b.tpart, 0, sizeof(double) * 2 * np, st));
    GX_CUDA(c, cudaMemsetAsync(b.drift, 0, sizeof(unsigned int), st));
    GX_CUDA(c, cudaMemsetAsync(b.Q, 0, sizeof(double2) * g.mesh, st));
    // reverse sweep
    for (int s = nsteps - 1; s >= 0; s--) {
        const bool ck = (s % ckpt_every) == 0;
        // the psi term of step s + 1, the drift back to x_s and its deposit
        c->acc_open = true;
        GX_CUDA(c, gx_launch_chain(k_adj_b, np, ADJ_BS, 0, st, g, b.S, b.L, n, s == nsteps - 1 ? nullptr : b.psi, g.pmass,
                                   1, ck ? b.ck + (size_t)(s / ckpt_every) * n : nullptr, b.drift, c->macc,
                                   gx_mass_ranges(c)));
        GX_LAUNCHED(c);
        int rc = adj_solve(c);
        if (rc) return rc;
        GX_CUDA(c, gx_launch_chain(k_adj_a, np, ADJ_BS, 0, st, g, b.S, b.L, n, c->field, ck ? 0 : 1,
                                   reinterpret_cast<double*>(b.Q), b.tpart));
        GX_LAUNCHED(c);
        GX_CUDA(c, gx_launch_chain(k_adjt_syn, g.nr, AT_H * AT_Q, sizeof(float2) * g.na, st, g, act, nact, ncp, b.Q,
                                   c->fwdtab, b.V));
        GX_LAUNCHED(c);
        GX_CUDA(c, gx_launch_chain(k_adjt_conv, g.nr, ADJ_BS, 0, st, g, act, nact, ncp, c->green32, b.V, c->fwdtab,
                                   b.psi));
        GX_LAUNCHED(c);
    }
    if (nsteps > 0) {
        k_adj_b<<<np, ADJ_BS, 0, st>>>(g, b.S, b.L, n, b.psi, g.pmass, 0, nullptr, b.drift, c->macc, gx_mass_ranges(c));
        GX_LAUNCHED(c);
    }
    GX_CUDA(c, cudaEventRecord(c->ev1, st));
    // gradient in load order (x, y, vx, vy): the records as they are
    GX_CUDA(c, cudaMemcpyAsync(grad, b.L, sbytes, cudaMemcpyDeviceToHost, st));
    GX_CUDA(c, cudaMemcpyAsync(hp.data(), b.tpart, sizeof(double) * 2 * np, cudaMemcpyDeviceToHost, st));
    unsigned int hd = 0;
    GX_CUDA(c, cudaMemcpyAsync(&hd, b.drift, sizeof hd, cudaMemcpyDeviceToHost, st));
    GX_CUDA(c, cudaStreamSynchronize(st));
    GX_CUDA(c, cudaEventElapsedTime(&c->last_ms, c->ev0, c->ev1));
    double drc = 0.0, dv2 = 0.0;
    for (unsigned i = 0; i < np; i++) {
        drc += hp[2 * i];
        dv2 += hp[2 * i + 1];
    }
    dtheta[0] = drc;
    dtheta[1] = dv2;
    *J_out = J;
    if (drift_out) {
        float d;
        memcpy(&d, &hd, sizeof d);
        *drift_out = d;
    }
    // the context again holds the initial particles (load order) and their mass
    k_adj_scatter<<<nb, ADJ_BS, 0, st>>>(b.ck, n, c->pbuf[c->cur], c->cap, c->origin, c->perm);
    GX_LAUNCHED(c);
    if (g.comp)  // the low parts of compensated positions start at zero, as after gx_loadup
        GX_CUDA(c, cudaMemsetAsync(c->pbuf[c->cur] + (size_t)4 * c->cap, 0, sizeof(float) * 2 * c->cap, st));
    c->zr_valid = false;
    int rc = gx_mixed_masset(c);
    if (rc) return rc;
    GX_CUDA(c, cudaStreamSynchronize(st));
    c->have_mass = true;
    c->have_field = false;
    int32_t ew = 0;
    GX_CUDA(c, cudaMemcpy(&ew, c->errword, sizeof ew, cudaMemcpyDeviceToHost));
    if (ew) return c->err = "device check raised the error word", GX_ERR_DEVICE;
    return GX_OK;
}

extern "C" int gx_adjoint(GxCtx* c, int nsteps, int ckpt_every, double* J_out, float* grad,
                          double* dtheta, float* drift_out) {
    const int rc = adj_run(c, nsteps, ckpt_every, J_out, grad, dtheta, drift_out);
    if (c && rc) gx_mass_discard(c);
    if (c && c->adj_bytes > ADJ_KEEP) {
        cudaStreamSynchronize(c->stream);  // (a failed call may have launches in flight)
        cudaFree(c->adj_ws);
        c->adj_ws = nullptr;
        c->adj_bytes = 0;
    }
    return rc;
}
