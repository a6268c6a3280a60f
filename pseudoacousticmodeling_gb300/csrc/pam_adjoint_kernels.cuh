// Device code of the receiver-side (adjoint) propagation: receiver injection,
// imaging conditions, anisotropic adjoint operators, the exact discrete
// adjoint, checkpoint compression and the misfit reduction.  Per-cell
// kernels use 2-D blocks of 32 x 8 threads; their neighbour reads are served
// by L1/L2 (these passes are a small share of a migration or gradient run).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "pam_aniso.cuh"
#include "pam_band.cuh"
#include "pam_check.cuh"
#include "pam_kernels.cuh"
#include "pam_types.h"

namespace pam {

// Cerjan factor of a cell in the order x then z (cpp/Modeling.cu:535-550);
// 1 outside the border, for CPML runs and outside the update region.
__device__ __forceinline__ float damp_factor(const GridDims& g, int z, int x) {
    if (!g.cerjan || z < 4 || z >= g.nz - 4 || x < 4 || x >= g.nx - 4) return 1.0f;
    float f = 1.0f;
    if (x < g.N) f = f * g.cerjan[x];
    if (x >= g.nx - g.N) f = f * g.cerjan[g.nx - 1 - x];
    float h = 1.0f;
    if (z < g.N) h = g.cerjan[z];
    if (z >= g.nz - g.N) h = h * g.cerjan[g.nz - 1 - z];
    return f * h;
}

// Multi-step damping applied value by value exactly like cpp/Modeling.cu:535-550.
__device__ __forceinline__ float damp_apply(const GridDims& g, int z, int x, float v) {
    if (!g.cerjan || z < 4 || z >= g.nz - 4 || x < 4 || x >= g.nx - 4) return v;
    if (x < g.N) v = v * g.cerjan[x];
    if (x >= g.nx - g.N) v = v * g.cerjan[g.nx - 1 - x];
    if (z < g.N) v = v * g.cerjan[z];
    if (z >= g.nz - g.N) v = v * g.cerjan[g.nz - 1 - z];
    return v;
}

// ---------------------------------------------------------------- receivers

// field[b][rz][rx] += scale * D * data[b][it][r]  (cpp/Migration.cu:493-502);
// atomics keep coincident receivers correct.  D is the Cerjan factor of the
// receiver cell when g.cerjan is set (the transpose of the damped recording),
// 1 otherwise.
__global__ void inject_receivers_kernel(float* __restrict__ field, const float* __restrict__ data,
                                        const int* __restrict__ rz, const int* __restrict__ rx, int nrec, int B,
                                        int it, int nt_data, int per_shot, float scale, GridDims g)
{
    wait_chained();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)nrec * B) return;
    const int r = (int)(i % nrec);
    const int b = (int)(i / nrec);
    const long long ri = per_shot ? (long long)b * nrec + r : r;
    const int z = rz[ri], x = rx[ri];
    const float v = damp_apply(g, z, x, data[((long long)b * nt_data + it) * nrec + r] * scale);
    atomicAdd(field + (long long)b * g.stride + (long long)z * g.P + x, v);
}

// Residual of the L2 misfit: res = dcal - dobs (or dobs - dcal with sign = -1),
// and per-block partial sums of 0.5 res^2 in double for a deterministic total.
// res may be dobs (the residual overwrites the observed data in place): each
// thread reads and writes only its own sample, so those two are not restrict
__global__ void residual_kernel(const float* __restrict__ dcal, const float* dobs, float* res, long long n,
                                float sign, double* __restrict__ partial)
{
    __shared__ double red[256];
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double acc = 0.0;
    if (i < n) {
        const float r = sign * (dcal[i] - dobs[i]);
        res[i] = r;
        acc = 0.5 * (double)r * (double)r;
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

// ---------------------------------------------------------------- imaging conditions
// Interior cells (z, x) in [N, nz-N) x [N, nx-N), totals [nzi][nxi]:
// - imaging: zero-lag cross-correlation img += Ub(t) P(t) and source
//   illumination ilum += P(t)^2 (cpp/Migration.cu:541-552);
// - reference FWI gradient g += Ub(t) (P(t+1) - 2 P(t) + P(t-1)) / dt^2
//   (cpp/inversion.cu:184-194 per cell);
// - illumination only, the FWI preconditioner (src/Migration.py:1034).
// Each sums the batch in registers (shots in order b = 0 .. B-1) and adds to
// the running totals once per step: one thread per interior cell, 8 B read
// per cell and shot (16 B for the gradient), where per-shot accumulators would
// also read and write 8 B per cell and shot.  The reference sums each shot's
// image over time first (src/Migration.py:553); summing the shots of a step
// first changes only the rounding order.
// One thread per 16-byte quad of field columns [4 q, 4 q + 4), counted from
// column 0 of the pitched row, so each warp reads whole aligned 128-byte lines
// (the interior starts N columns in); cells outside the interior are skipped
// when the sums are added.  Pairs of cells use the packed FP32 instructions.
__global__ void imaging_sum_kernel(const float* __restrict__ ub, const float* __restrict__ P_, float* __restrict__ img,
                                   float* __restrict__ ilum, GridDims g, int nzi, int nxi, long long pstride, int B)
{
    wait_chained();
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const int zi = blockIdx.y * blockDim.y + threadIdx.y;
    const int xf0 = 4 * q;                                   // first field column of the quad
    if (zi >= nzi || xf0 >= g.N + nxi || xf0 + 4 <= g.N) return;
    const long long c = (long long)(zi + g.N) * g.P + xf0;   // 16-byte aligned: P and the strides are multiples of 32
    float2 si0 = make_float2(0.f, 0.f), si1 = si0, sg0 = si0, sg1 = si0;
#pragma unroll 4
    for (int b = 0; b < B; b++) {
        const float4 p = *reinterpret_cast<const float4*>(
            PAM_CHK(P_ + (long long)b * pstride + c, P_, (long long)B * pstride * 4, 16, 60));
        const float4 u = *reinterpret_cast<const float4*>(
            PAM_CHK(ub + (long long)b * g.stride + c, ub, (long long)B * g.stride * 4, 16, 61));
        const float2 p0 = make_float2(p.x, p.y), p1 = make_float2(p.z, p.w);
        si0 = __ffma2_rn(p0, p0, si0);
        si1 = __ffma2_rn(p1, p1, si1);
        sg0 = __ffma2_rn(make_float2(u.x, u.y), p0, sg0);
        sg1 = __ffma2_rn(make_float2(u.z, u.w), p1, sg1);
    }
    const float si[4] = {si0.x, si0.y, si1.x, si1.y}, sg[4] = {sg0.x, sg0.y, sg1.x, sg1.y};
    const long long row = (long long)zi * nxi;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int xi = xf0 + j - g.N;
        if (xi >= 0 && xi < nxi) {
            *PAM_CHK(&ilum[row + xi], ilum, (long long)nzi * nxi * 4, 4, 62) += si[j];
            *PAM_CHK(&img[row + xi], img, (long long)nzi * nxi * 4, 4, 62) += sg[j];
        }
    }
}

// The reference gradient and its illumination in one pass (grad == 0: the
// illumination alone, of the steps outside the gradient's range), by quads like
// the imaging condition: the field at t is read once.
__global__ void fwi_ref_sum_kernel(const float* __restrict__ ub, const float* __restrict__ pp, const float* __restrict__ pc,
                                   const float* __restrict__ pf, float* __restrict__ grad, float* __restrict__ ilum,
                                   GridDims g, int nzi, int nxi, long long pstride, int B, float inv_dt2, int with_grad)
{
    wait_chained();
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const int zi = blockIdx.y * blockDim.y + threadIdx.y;
    const int xf0 = 4 * q;
    if (zi >= nzi || xf0 >= g.N + nxi || xf0 + 4 <= g.N) return;
    const long long c = (long long)(zi + g.N) * g.P + xf0;
    float sg[4] = {0.f, 0.f, 0.f, 0.f}, si[4] = {0.f, 0.f, 0.f, 0.f};
    auto quad = [&](const float* p, long long o, [[maybe_unused]] long long stride, float (&v)[4]) {
        const float4 x = *reinterpret_cast<const float4*>(PAM_CHK(p + o, p, (long long)B * stride * 4, 16, 63));
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    };
#pragma unroll 2
    for (int b = 0; b < B; b++) {
        const long long o = (long long)b * pstride + c;
        float c4[4], f4[4], p4[4], u4[4];
        quad(pc, o, pstride, c4);
        if (with_grad) {
            quad(pf, o, pstride, f4);
            quad(pp, o, pstride, p4);
            quad(ub, (long long)b * g.stride + c, g.stride, u4);
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            si[j] += c4[j] * c4[j];
            if (with_grad) {
                const float d2 = (f4[j] - 2.0f * c4[j] + p4[j]) * inv_dt2;
                sg[j] += u4[j] * d2;
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int xi = xf0 + j - g.N;
        if (xi >= 0 && xi < nxi) {
            const long long i = (long long)zi * nxi + xi;
            ilum[i] += si[j];
            if (with_grad) grad[i] += sg[j];
        }
    }
}

// Sum per-shot accumulators into the running total: out[i] += sum_b part[b][i]
// (fixed order over b, so the total is deterministic).
// Migration::Mute (cpp/Migration.cu:86-115) of observed data [B][nt][nrec] in
// place: zero before t1 = sqrt(dz dz + dx dx) / v0 + shift, scale by
// (t - t1) / (t2 - t1) up to t2 = t1 + window, with t = it * dt.  Each float
// operation rounds separately (no contraction), as the host code does.  One
// thread per (receiver, shot, chunk of `rows` time samples); rows at or after
// t2 are not touched, so a thread stops at the first of them.
__global__ void mute_kernel(float* __restrict__ d, const float* __restrict__ coords, int B, int nt, int nrec,
                            int per_shot, float dt, float v0, float shift, float window, int rows)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const int b = blockIdx.z;
    if (r >= nrec) return;
    const long long R = per_shot ? (long long)B * nrec : nrec;
    const long long ri = (per_shot ? (long long)b * nrec : 0) + r;
    const float ddz = __fsub_rn(coords[2 * B + R + ri], coords[B + b]);
    const float ddx = __fsub_rn(coords[2 * B + ri], coords[b]);
    const float t1 = __fadd_rn(__fdiv_rn(__fsqrt_rn(__fadd_rn(__fmul_rn(ddz, ddz), __fmul_rn(ddx, ddx))), v0), shift);
    const float t2 = __fadd_rn(t1, window);
    const float span = __fsub_rn(t2, t1);
    const int it0 = blockIdx.y * rows, it1 = min(it0 + rows, nt);
    float* col = d + (long long)b * nt * nrec + r;
    for (int it = it0; it < it1; it++) {
        const float t = __fmul_rn((float)it, dt);
        if (t >= t2) break;          // t grows with it: no later sample of this chunk changes
        float* p = col + (long long)it * nrec;
        if (t < t1) *p = 0.0f;
        else if (t < t2) *p = __fmul_rn(*p, __fdiv_rn(__fsub_rn(t, t1), span));
    }
}

__global__ void reduce_shots_kernel(const float* __restrict__ part, float* __restrict__ out, long long n, int B)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float s = out[i];
    for (int b = 0; b < B; b++) s += part[(long long)b * n + i];
    out[i] = s;
}

// ---------------------------------------------------------------- exact discrete adjoint (acoustic)

// 8th-order Laplacian in the stepping kernel's form: literal coefficients,
// sum, then 1/dx^2 and 1/dz^2 (so that its transpose is exact).
__device__ __forceinline__ float laplacian8(const float* W, long long s, float inv_dx2, float inv_dz2) {
    const float pxx = (PAM_C0 * W[0] + PAM_C1 * (W[1] + W[-1]) + PAM_C2 * (W[2] + W[-2]) +
                       PAM_C3 * (W[3] + W[-3]) + PAM_C4 * (W[4] + W[-4])) * inv_dx2;
    const float pzz = (PAM_C0 * W[0] + PAM_C1 * (W[s] + W[-s]) + PAM_C2 * (W[2 * s] + W[-2 * s]) +
                       PAM_C3 * (W[3 * s] + W[-3 * s]) + PAM_C4 * (W[4 * s] + W[-4 * s])) * inv_dz2;
    return pxx + pzz;
}

// The exact adjoint runs on the scaled variable w = kappa D lambda.  With the
// forward recursion U(t+1) = D (2 U(t) - D U(t-1) + kappa L U(t)) + f(t+1),
// the adjoint lambda(t) = 2 D lambda(t+1) + L(kappa D lambda(t+1))
// - D^2 lambda(t+2) + D R^T r(t) becomes
//   w(t) = D (2 w(t+1) - D w(t+2) + kappa L w(t+1)) + kappa D^2 R^T r(t),
// the forward recursion itself (the stepping kernel, no source) plus this
// receiver injection.  data holds the residual r = dcal - dobs.
__global__ void inject_adjoint_kernel(float* __restrict__ w, const float* __restrict__ data,
                                      const int* __restrict__ rz, const int* __restrict__ rx, int nrec, int B, int it,
                                      int nt_data, int per_shot, const float* __restrict__ kap, GridDims g)
{
    wait_chained();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)nrec * B) return;
    const int r = (int)(i % nrec);
    const int b = (int)(i / nrec);
    const long long ri = per_shot ? (long long)b * nrec + r : r;
    const int z = rz[ri], x = rx[ri];
    const long long c = (long long)z * g.P + x;
    const float v = damp_apply(g, z, x, damp_apply(g, z, x, data[((long long)b * nt_data + it) * nrec + r]));
    atomicAdd(w + (long long)b * g.stride + c, kap[c] * v);
}

// ---------------------------------------------------------------- multiparameter gradients

// Per-cell epsilon, delta (and theta) gradient increments of the reference's
// calculateGradientVTI / calculateGradientTTI (src/utils.py:1309-1463):
//   g_eps   += adj ((-2 cos^2 - dSd/deps) pxx - (2 sin^2 + dSd/deps) pzz + 2 sin 2th pxz)
//   g_delta += adj (-dSd/ddelta (pxx + pzz))
//   g_theta += adj ((2 eps sin 2th - dSd/dth) pxx + (-2 eps sin 2th - dSd/dth) pzz + 4 eps cos 2th pxz)
// (theta = 0 for VTI), Sd = num/den of the rotated gradient (h, q).  The
// reference evaluates in float64; here in float32 with (h, q) divided by
// max(|h|, |q|) first - every ratio is homogeneous of degree 0 in (h, q), so
// this is exact in exact arithmetic and keeps den = O(1) instead of |grad U|^4
// (which underflows float32).  Cells within 4 of the physical region's edge
// are skipped, as the reference's interior arrays do.  One thread per
// interior cell sums the batch's shots in registers (shots in order) and adds
// the sums to the running totals [nz][nx] once per step, like the imaging
// condition; the reference sums each shot over time first.  The same pass adds
// the vp gradient and the illumination of the step (fwi_ref_sum_kernel).  The
// cross derivative is the x derivative of the z derivative, which the cells of a
// block pass on through shared memory: 16 loads and 17 operations a cell where
// the 64-point form took 64 and 84.  grid (nx, nz) blocks of 32 x 8.
template <bool TTI>
__global__ void __launch_bounds__(256) mp_grad_kernel(const float* __restrict__ P_, const float* __restrict__ pm,
                                                      const float* __restrict__ pf, const float* __restrict__ ub,
                                                      long long pstride, const float* __restrict__ eps,
                                                      const float* __restrict__ del, const float* __restrict__ cth,
                                                      const float* __restrict__ sth, float* __restrict__ geps,
                                                      float* __restrict__ gdel, float* __restrict__ gth,
                                                      float* __restrict__ grad, float* __restrict__ ilum, GridDims g, int nzi,
                                                      int nxi, int B, float inv_dx, float inv_dz, float inv_dx2,
                                                      float inv_dz2, float inv_dt2)
{
    wait_chained();
    __shared__ float pzs[2][8][40];        // z derivatives of the block's rows, four columns more on each side
    const int x0 = blockIdx.x * 32, z0 = blockIdx.y * 8;
    const int xi = x0 + threadIdx.x, zi = z0 + threadIdx.y;
    const bool cell = xi < nxi && zi < nzi;
    const bool inner = xi >= 4 && xi < nxi - 4 && zi >= 4 && zi < nzi - 4;
    const long long c = (long long)(zi + g.N) * g.P + xi + g.N;
    const long long s = g.P;
    float ct = 1.0f, st = 0.0f, e = 0.0f, d = 0.0f;
    if (inner) {
        if (TTI) {
            ct = cth[c];
            st = sth[c];
        }
        e = eps[c];
        d = del[c];
    }
    const float s2 = 2.0f * st * ct, c2 = ct * ct, sn2 = st * st;
    float sum_e = 0.0f, sum_d = 0.0f, sum_t = 0.0f, sum_g = 0.0f, sum_i = 0.0f;
    auto dz = [&](const float* U) {
        return (PAM_A1 * (U[s] - U[-s]) + PAM_A2 * (U[2 * s] - U[-2 * s]) + PAM_A3 * (U[3 * s] - U[-3 * s]) +
                PAM_A4 * (U[4 * s] - U[-4 * s])) * inv_dz;
    };
    // the block's outer columns: one cell for each of the first 64 threads
    const int tid = threadIdx.y * 32 + threadIdx.x;
    const int hz = z0 + (tid >> 3), hc = tid & 7, hx = x0 + (hc < 4 ? hc - 4 : hc + 28);
    const bool halo = TTI && tid < 64 && hz >= 4 && hz < nzi - 4 && hx >= 0 && hx < nxi;
    const long long hcell = (long long)(hz + g.N) * g.P + hx + g.N;
    for (int b = 0; b < B; b++) {
        const float* U = P_ + (long long)b * pstride + c;
        float pz = 0.0f;
        if (cell && zi >= 4 && zi < nzi - 4) pz = dz(U);
        if (TTI) {
            pzs[b & 1][threadIdx.y][threadIdx.x + 4] = pz;
            if (halo) pzs[b & 1][tid >> 3][hc < 4 ? hc : hc + 32] = dz(P_ + (long long)b * pstride + hcell);
            __syncthreads();
        }
        if (!cell) continue;
        const float u0 = U[0], a = ub[(long long)b * g.stride + c];
        sum_i += u0 * u0;
        sum_g += a * ((pf[(long long)b * pstride + c] - 2.0f * u0 + pm[(long long)b * pstride + c]) * inv_dt2);
        if (!inner) continue;
        const float pxx = (PAM_C0 * u0 + PAM_C1 * (U[1] + U[-1]) + PAM_C2 * (U[2] + U[-2]) +
                           PAM_C3 * (U[3] + U[-3]) + PAM_C4 * (U[4] + U[-4])) * inv_dx2;
        const float pzz = (PAM_C0 * u0 + PAM_C1 * (U[s] + U[-s]) + PAM_C2 * (U[2 * s] + U[-2 * s]) +
                           PAM_C3 * (U[3 * s] + U[-3 * s]) + PAM_C4 * (U[4 * s] + U[-4 * s])) * inv_dz2;
        const float px = (PAM_A1 * (U[1] - U[-1]) + PAM_A2 * (U[2] - U[-2]) + PAM_A3 * (U[3] - U[-3]) +
                          PAM_A4 * (U[4] - U[-4])) * inv_dx;
        float pxz = 0.0f;
        if (TTI) {
            const float* v = &pzs[b & 1][threadIdx.y][threadIdx.x + 4];
            pxz = (PAM_A1 * (v[1] - v[-1]) + PAM_A2 * (v[2] - v[-2]) + PAM_A3 * (v[3] - v[-3]) +
                   PAM_A4 * (v[4] - v[-4])) * inv_dx;
        }
        float h = px * ct - pz * st, q = px * st + pz * ct;
        const float mh = fmaxf(fabsf(h), fabsf(q));
        float dSe = 0.0f, dSdl = 0.0f, dSt = 0.0f;
        if (mh > 0.0f) {
            h /= mh;
            q /= mh;
            const float h2 = h * h, q2 = q * q, t = h2 * q2, h4 = h2 * h2, q4 = q2 * q2;
            const float num = -2.0f * (e - d) * t;
            const float den = (1.0f + 2.0f * e) * h4 + q4 + 2.0f * (1.0f + d) * t;
            const float r = 1.0f / (den * den);
            dSe = (-2.0f * t * den - num * 2.0f * h4) * r;
            dSdl = (2.0f * t * den - num * 2.0f * t) * r;
            if (TTI) {
                const float w = -2.0f * h * q * q2 + 2.0f * h * h2 * q;
                const float dnum = -2.0f * (e - d) * w;
                const float dden =
                    -4.0f * (1.0f + 2.0f * e) * h * h2 * q + 4.0f * h * q * q2 + 2.0f * (1.0f + d) * w;
                dSt = (dnum * den - num * dden) * r;
            }
        }
        sum_e += a * (-(2.0f * c2 + dSe) * pxx - (2.0f * sn2 + dSe) * pzz + 2.0f * s2 * pxz);
        sum_d += a * (-dSdl * (pxx + pzz));
        if (TTI) {
            const float cos2 = c2 - sn2;
            sum_t += a * ((2.0f * e * s2 - dSt) * pxx + (-2.0f * e * s2 - dSt) * pzz + 4.0f * e * cos2 * pxz);
        }
    }
    if (!cell) return;
    const long long o = (long long)zi * nxi + xi;
    grad[o] += sum_g;
    ilum[o] += sum_i;
    if (!inner) return;
    geps[o] += sum_e;
    gdel[o] += sum_d;
    if (TTI) gth[o] += sum_t;
}

// ---------------------------------------------------------------- boundary saving

// Save the band of every shot of `field` into dst[b][nband]; the compressed
// formats keep one scale per chunk of kBandChunk cells (|max| of the chunk
// mapped to `target`), stored as its inverse in inv_scale[b][nchunk].
// grid (nchunk, B, times), block kBandChunk: consecutive times are fstride
// cells apart in field and tshots shots in dst and inv_scale.
template <typename T>
__global__ void __launch_bounds__(kBandChunk)
band_save_kernel(const float* __restrict__ field, T* __restrict__ dst, float* __restrict__ inv_scale, GridDims g,
                 int nzi, int nxi, float target, long long fstride, int tshots)
{
    __shared__ float red[kBandChunk / 32];
    const long long nb = band_cells(nzi, nxi);
    const int nchunk = (int)((nb + kBandChunk - 1) / kBandChunk);
    const int b = blockIdx.y;
    field += blockIdx.z * fstride;
    dst += (long long)blockIdx.z * tshots * nb;
    inv_scale += (long long)blockIdx.z * tshots * nchunk;
    const long long i = (long long)blockIdx.x * kBandChunk + threadIdx.x;
    float v = 0.0f;
    if (i < nb) {
        int z, x;
        band_cell(i, g.N, nzi, nxi, z, x);
        v = field[(long long)b * g.stride + (long long)z * g.P + x];
    }
    float s = 1.0f;
    if (target > 0.0f) {
        float m = fabsf(v);
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
        __syncthreads();
        m = red[0];
        for (int w = 1; w < kBandChunk / 32; w++) m = fmaxf(m, red[w]);
        // a chunk of values below 1e-30 is stored unscaled (and flushes to
        // zero in FP16): scaling it up could overflow target / m
        s = m > 1e-30f ? target / m : 1.0f;
        if (threadIdx.x == 0) inv_scale[(long long)b * nchunk + blockIdx.x] = 1.0f / s;
    }
    if (i < nb) dst[(long long)b * nb + i] = band_pack<T>(v * s);
}

// Write a saved band back into `field` (grid and block as band_save_kernel).
template <typename T>
__global__ void __launch_bounds__(kBandChunk)
band_restore_kernel(const T* __restrict__ src, const float* __restrict__ inv_scale, float* __restrict__ field,
                    GridDims g, int nzi, int nxi, int scaled)
{
    const long long nb = band_cells(nzi, nxi);
    const int nchunk = (int)((nb + kBandChunk - 1) / kBandChunk);
    const int b = blockIdx.y;
    const long long i = (long long)blockIdx.x * kBandChunk + threadIdx.x;
    if (i >= nb) return;
    int z, x;
    band_cell(i, g.N, nzi, nxi, z, x);
    float v = band_unpack(src[(long long)b * nb + i]);
    if (scaled) v *= inv_scale[(long long)b * nchunk + blockIdx.x];
    field[(long long)b * g.stride + (long long)z * g.P + x] = v;
}

// ---------------------------------------------------------------- checkpoints

// Largest |value| of each of `nf` fields of length n: out[f] (as ordered float bits).
__global__ void absmax_kernel(const float* __restrict__ src, long long n, int nf, long long fstride,
                              unsigned* __restrict__ out)
{
    const int f = blockIdx.y;
    float m = 0.f;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        m = fmaxf(m, fabsf(src[(long long)f * fstride + i]));
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out + f, __float_as_uint(m));
}

// dst = src * (1/scale) converted to the storage type (FP32 copies verbatim).
template <typename T>
__global__ void pack_kernel(const float* __restrict__ src, T* __restrict__ dst, long long n, int nf,
                            long long fstride, const unsigned* __restrict__ amax, float target)
{
    const int f = blockIdx.y;
    float inv = 1.0f;
    if (amax) {
        const float m = __uint_as_float(amax[f]);
        inv = m > 1e-30f ? target / m : 1.0f;   // below 1e-30 unscaled: target / m could overflow
    }
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float v = src[(long long)f * fstride + i] * inv;
        if constexpr (sizeof(T) == 4) dst[(long long)f * n + i] = v;
        else if constexpr (std::is_same<T, __nv_bfloat16>::value) dst[(long long)f * n + i] = __float2bfloat16_rn(v);
        else dst[(long long)f * n + i] = __float2half_rn(v);
    }
}

template <typename T>
__global__ void unpack_kernel(const T* __restrict__ src, float* __restrict__ dst, long long n, int nf,
                              long long fstride, const unsigned* __restrict__ amax, float target)
{
    const int f = blockIdx.y;
    float sc = 1.0f;
    if (amax) {
        const float m = __uint_as_float(amax[f]);
        sc = m > 1e-30f ? m / target : 1.0f;
    }
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float v;
        if constexpr (sizeof(T) == 4) v = src[(long long)f * n + i];
        else if constexpr (std::is_same<T, __nv_bfloat16>::value) v = __bfloat162float(src[(long long)f * n + i]);
        else v = __half2float(src[(long long)f * n + i]);
        dst[(long long)f * fstride + i] = v * sc;
    }
}

}  // namespace pam
