// The reference's anisotropic adjoint step (sm_103a), see AnisoArgs.
//
// The reference (cpp/Migration.cu:573-973) runs a step in two kernels: the
// first writes five products of the receiver field U with coefficients taken
// from the source field P (cpp/Migration.cu:573-666 VTI, :757-861 TTI)
//   AU = A U, BU = B U, HU = 2 eps sin(2 theta) U (TTI), QCxU, QCzU,
// the second applies their derivatives (cpp/Migration.cu:668-755, :863-973)
//   new = D (2 U - D U_prev + kappa (dxx AU + dzz BU - dxz HU - dx QCxU - dz QCzU)).
// No product goes to HBM here: per cell and shot a step reads P, U, U_prev and
// writes the new field (16 B).
//
// One warp owns one shot, 64 columns (a pair per lane, 56 of them written) and
// one z segment, and marches down it like the stepping kernel.  At row r it
// has the damped P of rows r-4 .. r+4 in registers and row r with its x
// neighbours in a shared ring, forms row r's products (zero off the update
// region), keeps BU and QCzU of rows r-8 .. r in registers and AU, QCxU (HU) in
// shared rings, and updates row r-4.  The rows arrive through cp.async two
// rows ahead.  The products of the four columns and rows around the written
// cells are formed by the neighbouring warps too: 1.14 x (H + 8) / H times,
// against 1.56 for 32 x 32 tiles with their halo in shared memory, which spent
// as much again on staging and index arithmetic.  Per cell the reference's
// expressions, in its order, with its correctly rounded divisions.
//
// Measured on 8 shots of 901 x 2101, VTI: 142 us a step (187 with the tiles;
// 108 M warp instructions against 182 M); bound by instruction issue (67% of
// the cycles) at 16 warps per SM, 1.8 of 6.8 TB/s.
#pragma once
#include "pam_check.cuh"
#include "pam_kernels.cuh"
#include "pam_types.h"

namespace pam {

struct GridDims {
    int nz, nx, P, N;          // expanded grid, pitch, absorbing width
    long long stride;          // nz * P
    const float* cerjan;       // [N] or nullptr (CPML)
};

struct AnisoArgs {
    const float* ub;      // receiver field U(t) [B][nz][P] (after injection)
    const float* pf;      // source field at t (stored U(t)), [B][...] with pstride
    long long pstride;
    const float *eps, *del, *cth, *sth;   // [nz][P]
    GridDims g;
    int B, tti;
    float inv_dx, inv_dz, inv_dx2, inv_dz2;
    int ntiles, nseg, H;  // tiles of kAnCols columns, segments of H rows
};

#define PAM_C0 (-1435.0f / 504.0f)
#define PAM_C1 (8.0f / 5.0f)
#define PAM_C2 (-1.0f / 5.0f)
#define PAM_C3 (8.0f / 315.0f)
#define PAM_C4 (-1.0f / 560.0f)
#define PAM_A1 (4.0f / 5.0f)
#define PAM_A2 (-1.0f / 5.0f)
#define PAM_A3 (4.0f / 105.0f)
#define PAM_A4 (-1.0f / 280.0f)

// Packed second and first derivatives of a cell pair for the anisotropic
// adjoint: (C0 c + C1 (p1 + m1) + ... + C4 (p4 + m4)) * inv and
// (A1 (p1 - m1) + ... + A4 (p4 - m4)) * inv, the coefficients of the
// reference's adjoint kernels (cpp/Migration.cu:600-640).
__device__ __forceinline__ float2 an_d2(float2 c, float2 p1, float2 m1, float2 p2, float2 m2, float2 p3, float2 m3,
                                       float2 p4, float2 m4, float inv) {
    float2 t = pmul2(bc2(PAM_C0), c);
    t = pfma2(bc2(PAM_C1), padd2(p1, m1), t);
    t = pfma2(bc2(PAM_C2), padd2(p2, m2), t);
    t = pfma2(bc2(PAM_C3), padd2(p3, m3), t);
    t = pfma2(bc2(PAM_C4), padd2(p4, m4), t);
    return pmul2(t, bc2(inv));
}
__device__ __forceinline__ float2 an_d1(float2 p1, float2 m1, float2 p2, float2 m2, float2 p3, float2 m3, float2 p4,
                                       float2 m4, float inv) {
    float2 t = pmul2(bc2(PAM_A1), fsub2(p1, m1));
    t = pfma2(bc2(PAM_A2), fsub2(p2, m2), t);
    t = pfma2(bc2(PAM_A3), fsub2(p3, m3), t);
    t = pfma2(bc2(PAM_A4), fsub2(p4, m4), t);
    return pmul2(t, bc2(inv));
}

// The reference's products of one cell (cpp/Migration.cu:573-666, 757-861).
// (In packed pairs they measured no faster.)
template <bool TTI>
__device__ __forceinline__ void aniso_products(float pxs, float pzs, float pxxs, float pzzs, float e, float d, float u,
                                               float cs, float sn, float& A_u, float& B_u, float& H_u, float& QX_u,
                                               float& QZ_u) {
    float sd = 0.f, Cx = 0.f, Cz = 0.f, A_, B_, hs = 0.f;
    if (!TTI) {
        const float px2 = pxs * pxs, pz2 = pzs * pzs, px4 = px2 * px2, pz4 = pz2 * pz2;
        const float num = -2.0f * (e - d) * px2 * pz2;
        const float den = (1.0f + 2.0f * e) * px4 + pz4 + 2.0f * (1.0f + d) * px2 * pz2;
        if (fabsf(den) > 1.0e-12f) {
            sd = num / den;
            const float inv_den2 = 1.0f / (den * den);
            const float factor = 4.0f * (e - d) * ((1.0f + 2.0f * e) * px4 - pz4) * inv_den2;
            Cx = factor * pxs * pz2;
            Cz = -factor * px2 * pzs;
        }
        A_ = 1.0f + 2.0f * e + sd;
        B_ = 1.0f + sd;
    } else {
        const float xi = pxs * cs - pzs * sn, eta = pxs * sn + pzs * cs;
        const float xi2 = xi * xi, eta2 = eta * eta, xi4 = xi2 * xi2, eta4 = eta2 * eta2;
        const float num = -2.0f * (e - d) * xi2 * eta2;
        const float den = (1.0f + 2.0f * e) * xi4 + eta4 + 2.0f * (1.0f + d) * xi2 * eta2;
        if (fabsf(den) > 1.0e-12f) {
            sd = num / den;
            const float K = (1.0f + 2.0f * e) * xi4 - eta4;
            const float factor = 4.0f * (e - d) * xi * eta * K / (den * den);
            Cx = factor * pzs;
            Cz = -factor * pxs;
        }
        const float cos2 = cs * cs, sin2 = sn * sn;
        A_ = (1.0f + 2.0f * e) * cos2 + sin2 + sd;
        B_ = (1.0f + 2.0f * e) * sin2 + cos2 + sd;
        hs = 2.0f * e * (2.0f * sn * cs);   // 2 eps sin(2 theta)
    }
    const float Q = pxxs + pzzs;
    A_u = A_ * u;
    B_u = B_ * u;
    H_u = hs * u;
    QX_u = Q * Cx * u;
    QZ_u = Q * Cz * u;
}

constexpr int kAnCols = 56;            // columns written per warp (64 held)
constexpr int kAnAhead = 2;            // rows in flight
constexpr int kAnUnroll = 4;           // rows per trip of the march: half a ring of eight
constexpr int kAnPRow = 72;            // P row: the 64 columns and four on each side
constexpr int kAnRing = 8;             // rows of the P, U, AU and QCxU rings
constexpr int kAnHRing = 16;           // rows of the HU ring (nine are read)
constexpr int kAnSlots = 4;            // rows of the model and U_prev ring
static_assert(kAnAhead + 1 <= kAnSlots && 4 + kAnAhead + 1 <= kAnRing, "rings too small for the prefetch distance");
static_assert(kAnUnroll == 4 && kAnRing == 8 && kAnSlots == 4, "a trip takes half a ring of eight");

// resident blocks per SM: the register windows (and the HU ring) set the limit
template <bool TTI>
__host__ __device__ constexpr int aniso_min_blocks() { return TTI ? 3 : 4; }

// floats of shared memory per warp
template <bool TTI>
__host__ __device__ constexpr int aniso_warp_floats() {
    return kAnRing * (kAnPRow + 3 * 64) + kAnSlots * 64 * (TTI ? 6 : 4) + (TTI ? kAnHRing * 64 : 0);
}
template <bool TTI>
__host__ __device__ constexpr int aniso_smem_bytes() { return kWarpsPerBlock * aniso_warp_floats<TTI>() * 4; }

template <bool TTI>
__global__ void __launch_bounds__(128, aniso_min_blocks<TTI>()) aniso_adjoint_kernel(const AnisoArgs a, float* __restrict__ nxt,
                                                                        const float* __restrict__ kap)
{
    wait_chained();
    extern __shared__ float an_sm[];
    const GridDims& g = a.g;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    float* const Pr = an_sm + wib * aniso_warp_floats<TTI>();   // [kAnRing][72] damped P, row z at z & 7
    float* const Ur = Pr + kAnRing * kAnPRow;                    // [kAnRing][64] U
    float* const Ar = Ur + kAnRing * 64;                         // [kAnRing][64] AU
    float* const Xr = Ar + kAnRing * 64;                         // [kAnRing][64] QCxU
    float* const Mr = Xr + kAnRing * 64;                         // [kAnSlots][arrays][64] eps, del, kappa, U_prev (cos, sin)
    constexpr int NM = TTI ? 6 : 4;
    float* const Hr = Mr + kAnSlots * NM * 64;                   // [kAnHRing][64] HU (TTI)

    const int warp = blockIdx.x * kWarpsPerBlock + wib;
    const int shot = warp % a.B;
    const int rest = warp / a.B;
    const int tile = rest % a.ntiles;
    const int seg = rest / a.ntiles;
    if (seg >= a.nseg) return;   // uniform per warp
    const int X0 = tile * kAnCols;
    const int x = X0 + 2 * lane;
    const int z0 = 4 + seg * a.H, z1 = min(z0 + a.H, g.nz - 4);
    const int P = g.P, zmax = g.nz - 1;
    [[maybe_unused]] const long long pbytes = (long long)a.B * a.pstride * 4;
    [[maybe_unused]] const long long fbytes = (long long)a.B * g.stride * 4;
    [[maybe_unused]] const long long mbytes = (long long)g.nz * g.P * 4;
    const float* const Pb = a.pf + (long long)shot * a.pstride;
    const float* const Ub = a.ub + (long long)shot * g.stride;
    float* const Nb = nxt + (long long)shot * g.stride;

    const bool in0 = x >= 4 && x < g.nx - 4, in1 = x + 1 >= 4 && x + 1 < g.nx - 4;
    const bool writer = lane >= 2 && lane < 30 && (in0 || in1);
    // damping factors along x of the lane's columns, and (lanes 0 .. 3) of a pair
    // of the P row's outer columns; 1 off the border and off the update region
    auto fx = [&](int c) {
        if (!g.cerjan || c < 4 || c >= g.nx - 4) return 1.0f;
        return c < g.N ? g.cerjan[c] : c >= g.nx - g.N ? g.cerjan[g.nx - 1 - c] : 1.0f;
    };
    auto fz = [&](int z) {
        return z < g.N ? g.cerjan[z] : z >= g.nz - g.N ? g.cerjan[g.nz - 1 - z] : 1.0f;
    };
    const float cx0 = fx(x), cx1 = fx(x + 1);
    const int hoff = lane < 2 ? 2 * lane : 64 + 2 * lane;             // floats 0 .. 3 and 68 .. 71 of a P row
    const float hx0 = lane < 4 ? fx(X0 - 4 + hoff) : 1.0f, hx1 = lane < 4 ? fx(X0 - 3 + hoff) : 1.0f;
    // warp-uniform: do the columns, or row z, reach into the border?
    const bool xdamp = g.cerjan && (X0 - 4 < g.N || X0 + 68 > g.nx - g.N);
    auto zdamp = [&](int z) { return g.cerjan && (z < g.N || z >= g.nz - g.N); };

    // rows arriving for product row r: P row r + 4, U, eps, delta (cos, sin) of
    // row r, kappa and U_prev of row r - 4, as 16-byte pieces; every piece is
    // aligned (X0 is a multiple of 8), columns off the pitch are left out, rows
    // off the grid are its first or last one (products there are zero).  Row
    // rs + i lies in place i of each ring: a trip of four rows takes one half
    // of the rings of eight, so that every place is a constant from one of two
    // bases (h0: the half of this trip, h1: the other).
    const int rs = z0 - 4;                               // first row of products
    const int half = lane & 15;
    const bool colq = X0 + 4 * half < P, low = lane < 16;
    const int pcol = X0 - 4 + 4 * lane;
    const bool pq = lane < 18 && pcol >= 0 && pcol < P;
    const float* src_p = Pb + (long long)min(rs + 4, zmax) * P + pcol;
    const long long m0 = (long long)rs * P + X0 + 4 * half, u0 = (long long)max(rs - 4, 0) * P + X0 + 4 * half;
    const float* src_a = low ? Ub + m0 : a.eps + m0;     // row r
    const float* src_b = low ? a.del + m0 : (TTI ? a.cth + m0 : nullptr);
    const float* src_c = TTI ? a.sth + m0 : nullptr;
    const float* src_u = low ? Nb + u0 : kap + u0;       // row r - 4
    int rn = rs;                                         // the row that the next issue is for
    auto issue = [&](float* place_p, float* place_u, float* slot) {
        if (pq) cp_async16(place_p + 4 * lane, PAM_CHK(src_p, a.pf, pbytes, 16, 92));
        if (colq) {
            cp_async16(low ? place_u + 4 * half : slot + 4 * half,
                       PAM_CHK(src_a, low ? (const void*)a.ub : (const void*)a.eps, low ? fbytes : mbytes, 16, 94));
            if (TTI || low)
                cp_async16(slot + (low ? 64 : 256) + 4 * half,
                           PAM_CHK(src_b, low ? (const void*)a.del : (const void*)a.cth, mbytes, 16, 93));
            if (TTI && low) cp_async16(slot + 320 + 4 * half, PAM_CHK(src_c, a.sth, mbytes, 16, 93));
            cp_async16(slot + (low ? 192 : 128) + 4 * half,
                       PAM_CHK(src_u, low ? (const void*)nxt : (const void*)kap, low ? fbytes : mbytes, 16, 96));
        }
        cp_async_commit();
        if (rn + 4 < zmax) src_p += P;
        if (rn < zmax) {
            src_a += P;
            if (TTI || low) src_b += P;
            if (TTI) src_c += P;
        }
        if (rn >= 4 && rn - 4 < zmax) src_u += P;
        rn++;
    };
    // the lane's pair of P row z (in the ring), damped; the ring row too
    auto take_p = [&](int z, float* row, bool undamped) {
        float2 v = *reinterpret_cast<const float2*>(row + 4 + 2 * lane);
        if (!undamped && z >= 4 && z < g.nz - 4 && (xdamp || zdamp(z))) {
            const float cz = zdamp(z) ? fz(z) : 1.0f;
            v = make_float2(in0 ? __fmul_rn(__fmul_rn(v.x, cx0), cz) : v.x, in1 ? __fmul_rn(__fmul_rn(v.y, cx1), cz) : v.y);
            *reinterpret_cast<float2*>(row + 4 + 2 * lane) = v;
            if (lane < 4) {
                const int c = X0 - 4 + hoff;
                float2 h = *reinterpret_cast<const float2*>(row + hoff);
                if (c >= 4 && c < g.nx - 4) h.x = __fmul_rn(__fmul_rn(h.x, hx0), cz);
                if (c + 1 >= 4 && c + 1 < g.nx - 4) h.y = __fmul_rn(__fmul_rn(h.y, hx1), cz);
                *reinterpret_cast<float2*>(row + hoff) = h;
            }
        }
        return v;
    };

    // P rows rs - 4 .. rs + 3 before the march
    float2 w[8 + kAnUnroll], bu[8 + kAnUnroll], qz[8 + kAnUnroll];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int z = min(max(rs - 4 + i, 0), zmax);
        if (pq) cp_async16(Pr + ((i + 4) & 7) * kAnPRow + 4 * lane,
                           PAM_CHK(Pb + (long long)z * P + pcol, a.pf, pbytes, 16, 92));
        bu[i] = qz[i] = make_float2(0.f, 0.f);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; i++) w[i] = take_p(rs - 4 + i, Pr + ((i + 4) & 7) * kAnPRow, rs - 4 + i < 0);
    // rows rs - 4 .. rs - 1 are in registers: their places are free
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kAnAhead; i++) issue(Pr + ((i + 4) & 7) * kAnPRow, Ur + i * 64, Mr + i * NM * 64);

    const bool cols_in = X0 >= 4 && X0 + 64 <= g.nx - 4;   // warp-uniform: every column in the update region
    auto row = [&](auto place_tag, int h, int r, float2 p0, float2 p1, float2 p2, float2 p3, float2 p4, float2 p5, float2 p6, float2 p7, float2& p8,
                   float2 b0, float2 b1, float2 b2, float2 b3, float2 b4, float2 b5, float2 b6, float2 b7, float2& b8,
                   float2 q0, float2 q1, float2 q2, float2 q3, float2 q4, float2 q5, float2 q6, float2 q7, float2& q8) {
        // place of row r + k in a ring of eight, and of this row in the others
        constexpr int J = decltype(place_tag)::value;
        auto place8 = [&](float* ring, int stride, int k) {
            const int q = (J + k) & 7;
            return ring + ((q & 4) ^ h) * stride + (q & 3) * stride;
        };
        issue(place8(Pr, kAnPRow, 4 + kAnAhead), place8(Ur, 64, kAnAhead), Mr + ((J + kAnAhead) & 3) * NM * 64);
        cp_async_wait<kAnAhead>();
        __syncwarp();
        p8 = take_p(r + 4, place8(Pr, kAnPRow, 4), false);
        const float* const slot = Mr + J * NM * 64 + 2 * lane;
        auto at = [](const float* p) { return *reinterpret_cast<const float2*>(p); };
        // 1. the products of row r
        float2 av = make_float2(0.f, 0.f), bv = av, hv = av, qxv = av, qzv = av;
        const bool zin = r >= 4 && r < g.nz - 4;
        if (zin && (cols_in || in0 || in1)) {
            const float* const c = place8(Pr, kAnPRow, 0) + 2 * lane;
            const float2 A0 = at(c), A1 = at(c + 2), A2 = p4, A3 = at(c + 6), A4 = at(c + 8);
            const float2 Om3 = make_float2(A0.y, A1.x), Om1 = make_float2(A1.y, A2.x);
            const float2 Op1 = make_float2(A2.y, A3.x), Op3 = make_float2(A3.y, A4.x);
            const float2 pxx = an_d2(A2, Op1, Om1, A3, A1, Op3, Om3, A4, A0, a.inv_dx2);
            const float2 pzz = an_d2(A2, p5, p3, p6, p2, p7, p1, p8, p0, a.inv_dz2);
            const float2 px = an_d1(Op1, Om1, A3, A1, Op3, Om3, A4, A0, a.inv_dx);
            const float2 pz = an_d1(p5, p3, p6, p2, p7, p1, p8, p0, a.inv_dz);
            const float2 e2v = at(slot), d2v = at(slot + 64), u2 = at(place8(Ur, 64, 0) + 2 * lane);
            float2 cs2 = make_float2(0.f, 0.f), sn2 = cs2;
            if (TTI) {
                cs2 = at(slot + 256);
                sn2 = at(slot + 320);
            }
            aniso_products<TTI>(px.x, pz.x, pxx.x, pzz.x, e2v.x, d2v.x, u2.x, cs2.x, sn2.x, av.x, bv.x, hv.x, qxv.x, qzv.x);
            aniso_products<TTI>(px.y, pz.y, pxx.y, pzz.y, e2v.y, d2v.y, u2.y, cs2.y, sn2.y, av.y, bv.y, hv.y, qxv.y, qzv.y);
            if (!cols_in) {
                if (!in0) av.x = bv.x = hv.x = qxv.x = qzv.x = 0.f;
                if (!in1) av.y = bv.y = hv.y = qxv.y = qzv.y = 0.f;
            }
        }
        b8 = bv;
        q8 = qzv;
        *reinterpret_cast<float2*>(place8(Ar, 64, 0) + 2 * lane) = av;
        *reinterpret_cast<float2*>(place8(Xr, 64, 0) + 2 * lane) = qxv;
        if (TTI) *reinterpret_cast<float2*>(Hr + ((r - rs) & (kAnHRing - 1)) * 64 + 2 * lane) = hv;
        // 2. the update of row t = r - 4 (its products' rows r - 8 .. r are complete)
        const int t = r - 4;
        if (t < z0 || t >= z1) return;
        __syncwarp();
        if (writer) {
            const float* const al = place8(Ar, 64, -4) + 2 * lane;
            const float* const xl = place8(Xr, 64, -4) + 2 * lane;
            float2 op;
            {
                const float2 A0 = at(al - 4), A1 = at(al - 2), A2 = at(al), A3 = at(al + 2), A4 = at(al + 4);
                const float2 dxx = an_d2(A2, make_float2(A2.y, A3.x), make_float2(A1.y, A2.x), A3, A1,
                                         make_float2(A3.y, A4.x), make_float2(A0.y, A1.x), A4, A0, a.inv_dx2);
                const float2 dzz = an_d2(b4, b5, b3, b6, b2, b7, b1, b8, b0, a.inv_dz2);
                op = padd2(dxx, dzz);
            }
            if (TTI) {
                // the cross derivative (cpp/Migration.cu:906-928) of HU in the order of
                // sum_ax a_ax sum_az a_az (...): for each az the differences of the rows
                // +az and -az (columns -4 .. +5 around the pair) feed all four ax
                const float aa[5] = {0.f, PAM_A1, PAM_A2, PAM_A3, PAM_A4};
                float2 tax[5] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f),
                                 make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
                for (int az = 1; az <= 4; az++) {
                    const float* const hpr = Hr + ((t - rs + az) & (kAnHRing - 1)) * 64 + 2 * lane;
                    const float* const hmr = Hr + ((t - rs - az) & (kAnHRing - 1)) * 64 + 2 * lane;
                    float2 v[5];
#pragma unroll
                    for (int k = 0; k < 5; k++) v[k] = fsub2(at(hpr - 4 + 2 * k), at(hmr - 4 + 2 * k));
                    const float2 p1 = make_float2(v[2].y, v[3].x), m1 = make_float2(v[1].y, v[2].x);
                    const float2 p3 = make_float2(v[3].y, v[4].x), m3 = make_float2(v[0].y, v[1].x);
                    tax[1] = pfma2(bc2(aa[az]), fsub2(p1, m1), tax[1]);
                    tax[2] = pfma2(bc2(aa[az]), fsub2(v[3], v[1]), tax[2]);
                    tax[3] = pfma2(bc2(aa[az]), fsub2(p3, m3), tax[3]);
                    tax[4] = pfma2(bc2(aa[az]), fsub2(v[4], v[0]), tax[4]);
                }
                float2 dxz = make_float2(0.f, 0.f);
#pragma unroll
                for (int ax = 1; ax <= 4; ax++) dxz = pfma2(bc2(aa[ax]), tax[ax], dxz);
                op = fsub2(op, pmul2(dxz, bc2(a.inv_dx * a.inv_dz)));
            }
            {
                const float2 Y0 = at(xl - 4), Y1 = at(xl - 2), Y2 = at(xl), Y3 = at(xl + 2), Y4 = at(xl + 4);
                op = fsub2(op, an_d1(make_float2(Y2.y, Y3.x), make_float2(Y1.y, Y2.x), Y3, Y1, make_float2(Y3.y, Y4.x),
                                     make_float2(Y0.y, Y1.x), Y4, Y0, a.inv_dx));
                op = fsub2(op, an_d1(q5, q3, q6, q2, q7, q1, q8, q0, a.inv_dz));
            }
            const float2 uc = at(place8(Ur, 64, -4) + 2 * lane), kv = at(slot + 128);
            float2 prev = at(slot + 192);
            const bool damp = xdamp || zdamp(t);
            const float cz = zdamp(t) ? fz(t) : 1.0f;
            if (damp) prev = make_float2(__fmul_rn(__fmul_rn(prev.x, cx0), cz), __fmul_rn(__fmul_rn(prev.y, cx1), cz));
            float2 out = pfma2(kv, op, fsub2(padd2(uc, uc), prev));
            if (damp) out = make_float2(__fmul_rn(__fmul_rn(out.x, cx0), cz), __fmul_rn(__fmul_rn(out.y, cx1), cz));
            float* const dst = Nb + (long long)t * P + x;
            if (in0 && in1) {
                *reinterpret_cast<float2*>(PAM_CHK(dst, nxt, fbytes, 8, 97)) = out;
            } else {
                if (in0) *PAM_CHK(dst, nxt, fbytes, 4, 97) = out.x;
                if (in1) *PAM_CHK(dst + 1, nxt, fbytes, 4, 97) = out.y;
            }
        }
    };
    int h = 0;
    for (int r = rs; r < z1 + 4; r += kAnUnroll, h ^= 4) {
        auto step = [&](auto j_tag) {
            constexpr int j = decltype(j_tag)::value;
            row(j_tag, h, r + j, w[j], w[j + 1], w[j + 2], w[j + 3], w[j + 4], w[j + 5], w[j + 6], w[j + 7], w[j + 8],
                bu[j], bu[j + 1], bu[j + 2], bu[j + 3], bu[j + 4], bu[j + 5], bu[j + 6], bu[j + 7], bu[j + 8],
                qz[j], qz[j + 1], qz[j + 2], qz[j + 3], qz[j + 4], qz[j + 5], qz[j + 6], qz[j + 7], qz[j + 8]);
        };
        step(IntTag<0>{});
        step(IntTag<1>{});
        step(IntTag<2>{});
        step(IntTag<3>{});
#pragma unroll
        for (int i = 0; i < 8; i++) {
            w[i] = w[i + kAnUnroll];
            bu[i] = bu[i + kAnUnroll];
            qz[i] = qz[i + kAnUnroll];
        }
    }
    cp_async_wait<0>();
}

}  // namespace pam
