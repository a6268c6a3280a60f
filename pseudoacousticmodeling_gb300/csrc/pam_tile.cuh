// Time loops of small batches as persistent tiles (sm_103a).
//
// A small grid's step costs far less than the latency of starting it: a graph
// of one-step launches takes 6 us a step for one 301 x 501 shot, and one
// cooperative launch with a grid-wide barrier after every step 2.8 us, most
// of it the barrier and the reload of the field from L2.  Here one block per
// SM owns a tile of one shot for the whole launch and keeps it on chip with a
// halo 4 T cells wide.  It advances T steps between barriers, each on a region
// 4 cells smaller on every side than the one before (the stencil's reach), so
// that the last one ends on the tile itself; then it publishes the tile's two
// fields, waits for the other blocks and reads the halo back from L2.  The
// halo cells are computed by several blocks, from the same values by the same
// operations, so the results are those of the one-step kernels bit for bit
// (acoustic with the matched layer: of those with segments of eight rows).
//
// A thread owns one quad of columns and R rows of the tile with its halo:
// U(t) and U(t-1) of those cells stay in its registers, and two copies of U in
// shared memory (one read, one written, one block barrier per step) give it
// the four rows above and below and the quads left and right.  What a thread
// needs for its cells - addresses, masks, damping factors, kappa - is worked
// out once per launch: the step loop itself is bound by the latency of its
// arithmetic and by instruction issue.
//
// A larger T saves barriers (about 2 us each with the exchange) and costs
// halo cells; tile_plan() on the host weighs the two for the grid at hand.
// Measured per step, tiles against the graph of one-step launches (and the
// one-barrier-per-step persistent kernel): acoustic 301 x 501 1.4 against 5.7
// (2.8) us, 501 x 1101 2.2 against 5.9; VTI 501 x 1101 3.5 against 7.1 (6.3);
// TTI 381 x 681 3.1 against 7.3.  At 1.4 us a step the 301 x 501 tile spends
// about 0.65 us a step in the exchange and issues 28% of the cycles.
#pragma once
#include "pam_band.cuh"
#include "pam_kernels.cuh"

namespace pam {

constexpr int kTileThreads = 512;       // at most
constexpr int kTilePitch = 32;          // quads per row of a shared copy (more than a tile with its halo has)
constexpr int kTileMaxT = 8;

// model arrays of an approximation: kappa, 1 + 2 eps, -2 (eps - delta),
// 2 (1 + delta), cos, sin
template <int APPROX>
__host__ __device__ constexpr int tile_models() { return APPROX == kAcoustic ? 1 : (APPROX == kVTI ? 4 : 6); }

struct TileShape {
    int T;              // steps between barriers
    int TZ, TX;         // cells of a tile (TX a multiple of 4)
    int nty, ntx;       // tiles of one shot
    int halo;           // cells that a step's region loses on each side: 4, with CPML strips 8
    int R;              // rows per thread
    int nrg, EXq;       // row groups and quads of a tile with its halo
};

__host__ __device__ inline int tile_threads(const TileShape& g) { return (g.nrg * g.EXq + 31) / 32 * 32; }
// two copies of U (for TTI a third array, of its z derivative) with four guard
// rows above and below; the models of each thread's cells (the acoustic kappa stays in registers)
__host__ __device__ inline size_t tile_smem_bytes(const TileShape& g, int models) {
    const int copies = models == tile_models<kTTI>() ? 3 : 2;
    return (size_t)copies * (g.nrg * g.R + 8) * kTilePitch * 16 +
           (models > 1 ? (size_t)models * g.R * tile_threads(g) * 16 : 0);
}

struct TileArgs {
    StepArgs s;                          // grid, models, Cerjan factors, sources (no fields)
    TileShape g;
    float* ex[2][2];                     // published state [set][0: U(k), 1: U(k-1)], [B][nz][P]
    int set0;                            // set that holds the state before step k0
    int shot0;                           // first shot of this launch
    const float* __restrict__ wavelet;   // [nt]
    RecordArgs rec;                      // seis == nullptr: no recording
    const int* __restrict__ rec_beg;     // [tiles (per shot) + 1] receivers of each tile ...
    const int2* __restrict__ rec_ent;    // ... as (row << 16 | column, receiver)
    int nt, itlag, k0, k1;
    unsigned* bar;                       // barrier counter, zero at the launch
    int polls;                           // of a barrier before it is given up
    int* status;                         // [0] bit 0 set by a non-finite sample, [1] by a barrier given up
    // every U(k) kept: U(k) at slots + (k - kslot) * slot_stride; the state before
    // step k0 is U(k0), U(k0 - 1) there, and so is what the tiles exchange
    // (nullptr: the two published sets)
    float* slots;
    long long slot_stride;
    int kslot;
    int mem_shots;                       // shots of the memory variables' arrays (CPML)
    // the source field backwards in time (with slots, undamped, kTileReverse): the
    // state before step k1-1 is S(k1-1), S(k1); step t gives
    // S(t-1) = 2 S(t) - S(t+1) + kappa L S(t) + w(t+1), down to S(k0-1), with the
    // saved band of time t-1 written over it (band == nullptr: none)
    const void* band;                    // [nt-1][B][nb] in the storage type
    const float* __restrict__ band_scale;   // [nt-1][B][chunks]
    int band_shots, band_store, nzi, nxi;   // (the bands are kept for max_shots)
};

// Grid-wide barrier of resident blocks: each block's writes before it are
// visible (through L2) to every block after it.  `want` = blocks x barriers so
// far.  False when it was given up (all blocks are resident, so it is not
// unless the limit is far below a step): the block then leaves, and so do the
// others at their next barrier.
__device__ __forceinline__ bool tile_barrier(const TileArgs& t, unsigned want, int* flag) {
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(t.bar) : "memory");
        int left = t.polls;
        unsigned v;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(t.bar) : "memory");
        } while ((int)(v - want) < 0 && --left > 0);
        *flag = left > 0;
        if (left <= 0) t.status[1] = 1;
    }
    __syncthreads();
    return *flag != 0;
}

// The samples that a block which gave up at step k leaves out: NaN, so that the
// holder of a device buffer sees it.
__device__ __forceinline__ void tile_poison(const TileArgs& t, float* seis, int rb, int re, int k) {
    for (int i = rb + threadIdx.x; i < re; i += blockDim.x)
        for (int it = max(k - t.itlag, 0); it < t.k1 - t.itlag; it++)
            seis[(long long)it * t.rec.nrec + t.rec_ent[i].y] = __int_as_float(0x7fc00000);
}

// A quad of row z, column x (a multiple of 4) of a pitched array; zero outside
// [0, nz) x [0, P).  Fields are read past L1, which other SMs' writes do not reach.
__device__ __forceinline__ float4 tile_fetch(const float* src, int z, int x, int nz, int P,
                                             [[maybe_unused]] const void* base, [[maybe_unused]] long long bytes) {
    if (z < 0 || z >= nz || x < 0 || x >= P) return make_float4(0.f, 0.f, 0.f, 0.f);
    return __ldcg(reinterpret_cast<const float4*>(PAM_CHK(src + (long long)z * P + x, base, bytes, 16, 100)));
}

// A quad that another block published, at a cell of the update region.
__device__ __forceinline__ float4 tile_halo(const float* p, [[maybe_unused]] const void* base,
                                            [[maybe_unused]] long long bytes) {
    return __ldcg(reinterpret_cast<const float4*>(PAM_CHK(p, base, bytes, 16, 104)));
}

// What a thread owns, worked out once per launch.
template <int R>
struct TileCells {
    int z, x;                // first row, first column
    int at;                  // quad index in a shared copy
    int need;                // smallest region halo that holds one of its cells
    unsigned valid, mine;    // rows of the update region; rows of the block's own tile
    bool tail, damp;         // columns past the update region; any damped cell
    float4 cx;               // damping factors (1 outside the border)
    float cz[R];
};

template <int R>
__device__ __forceinline__ TileCells<R> tile_cells(const StepArgs& a, const TileShape& g, int tile, int pitch) {
    const int z0 = 4 + (tile / g.ntx) * g.TZ, x0 = 4 + (tile % g.ntx) * g.TX;
    const int z1 = min(z0 + g.TZ, a.nz - 4), x1 = min(x0 + g.TX, a.nx - 4);
    const int rg = threadIdx.x / g.EXq, q = threadIdx.x - rg * g.EXq;
    TileCells<R> c;
    c.z = z0 - g.halo * g.T + rg * R;
    c.x = x0 - g.halo * g.T + 4 * q;
    c.at = (4 + min(rg, g.nrg - 1) * R) * pitch + q;
    c.need = 1 << 20;
    c.valid = c.mine = 0;
    auto factor = [&](int i, int len) {
        float f = 1.0f;
        if (a.cerjan && i >= 0 && i < a.N) f = a.cerjan[i];
        if (a.cerjan && i >= len - a.N && i < len) f = f * a.cerjan[len - 1 - i];
        return f;
    };
    const bool xin = rg < g.nrg && c.x >= 4 && c.x < a.nx - 4;
    const int hx = max(x0 - c.x, c.x >= x1 ? c.x - x1 + 4 : 0);
    c.damp = c.x < a.N || c.x + 4 > a.nx - a.N;
#pragma unroll
    for (int j = 0; j < R; j++) {
        const int z = c.z + j;
        if (xin && z >= 4 && z < a.nz - 4) {
            c.valid |= 1u << j;
            c.need = min(c.need, max(max(max(z0 - z, z - z1 + 1), hx), 0));
            if (z >= z0 && z < z1 && c.x >= x0 && c.x < x1) c.mine |= 1u << j;
        }
        c.cz[j] = factor(z, a.nz);
        c.damp = c.damp || z < a.N || z >= a.nz - a.N;
    }
    c.damp = c.damp && a.cerjan;
    c.cx = make_float4(factor(c.x, a.nx), factor(c.x + 1, a.nx), factor(c.x + 2, a.nx), factor(c.x + 3, a.nx));
    c.tail = c.x + 4 > a.nx - 4;
    return c;
}

// One step of a thread's cells: out[j] = U(k+1) from cur[j] = U(k), old[j] =
// U(k-1) and the neighbours' U(k) in the shared copy A.  model(i, j) gives row
// j of model array i; strips(j, ...) may add CPML strip terms to the derivatives
// of row j.  For TTI every thread that holds cells of the block
// calls it (Z passes the z derivatives on, with a barrier), and out is left
// alone where the thread is not active.
struct TileNoStrips {
    template <class W, class D>
    __device__ __forceinline__ void operator()(int, const W&, D&, D&, D&, D&) const {}
};

template <int APPROX, int R, class Model, class Strips = TileNoStrips>
__device__ __forceinline__ void tile_step(const StepArgs& a, const TileCells<R>& t, int pitch,
                                          const float4* __restrict__ A,
                                          float4* __restrict__ Z, bool active, const float4 (&cur)[R],
                                          const float4 (&old)[R], Model model, float4 (&out)[R],
                                          Strips strips = Strips()) {
    const float4* const col = A + t.at;
    float4 w[R + 8];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        w[j] = col[(j - 4) * pitch];
        w[R + 4 + j] = col[(R + j) * pitch];
    }
#pragma unroll
    for (int j = 0; j < R; j++) w[j + 4] = cur[j];
    // the z derivatives; for the TTI cross derivative (the x derivative of the
    // z derivative) they go to the neighbouring quads through shared memory
    float2 pzv[R][2];
    if (APPROX != kAcoustic) {
#pragma unroll
        for (int j = 0; j < R; j++) {
            pzv[j][0] = d1_pair_ref(lo2(w[j + 5]), lo2(w[j + 3]), lo2(w[j + 6]), lo2(w[j + 2]), lo2(w[j + 7]), lo2(w[j + 1]),
                                    lo2(w[j + 8]), lo2(w[j]), a.inv_dz);
            pzv[j][1] = d1_pair_ref(hi2(w[j + 5]), hi2(w[j + 3]), hi2(w[j + 6]), hi2(w[j + 2]), hi2(w[j + 7]), hi2(w[j + 1]),
                                    hi2(w[j + 8]), hi2(w[j]), a.inv_dz);
            if (APPROX == kTTI && t.valid)
                Z[t.at + j * pitch] = make_float4(pzv[j][0].x, pzv[j][0].y, pzv[j][1].x, pzv[j][1].y);
        }
    }
    if (APPROX == kTTI) __syncthreads();
    if (!active) return;
#pragma unroll
    for (int j = 0; j < R; j++) {
        const float4 c = cur[j], l = col[j * pitch - 1], r = col[j * pitch + 1];
        const float4 kap = model(0, j);
        const float2 P0 = lo2(l), P1 = hi2(l), P2 = lo2(c), P3 = hi2(c), P4 = lo2(r), P5 = hi2(r);
        const float2 O0 = make_float2(l.y, l.z), O1 = make_float2(l.w, c.x), O2 = make_float2(c.y, c.z);
        const float2 O3 = make_float2(c.w, r.x), O4 = make_float2(r.y, r.z);
        float2 pxx[2], pzz[2], px[2], pz[2], pxz[2];
        px[0] = px[1] = pz[0] = pz[1] = pxz[0] = pxz[1] = make_float2(0.f, 0.f);
        pxx[0] = d2_pair(P2, O2, O1, P3, P1, O3, O0, P4, P0, a.inv_dx2);
        pxx[1] = d2_pair(P3, O3, O2, P4, P2, O4, O1, P5, P1, a.inv_dx2);
        pzz[0] = d2_pair(lo2(c), lo2(w[j + 5]), lo2(w[j + 3]), lo2(w[j + 6]), lo2(w[j + 2]), lo2(w[j + 7]), lo2(w[j + 1]),
                         lo2(w[j + 8]), lo2(w[j]), a.inv_dz2);
        pzz[1] = d2_pair(hi2(c), hi2(w[j + 5]), hi2(w[j + 3]), hi2(w[j + 6]), hi2(w[j + 2]), hi2(w[j + 7]), hi2(w[j + 1]),
                         hi2(w[j + 8]), hi2(w[j]), a.inv_dz2);
        if (APPROX != kAcoustic) {
            px[0] = d1_pair_ref(O2, O1, P3, P1, O3, O0, P4, P0, a.inv_dx);
            px[1] = d1_pair_ref(O3, O2, P4, P2, O4, O1, P5, P1, a.inv_dx);
            pz[0] = pzv[j][0];
            pz[1] = pzv[j][1];
        }
        if (APPROX == kTTI) {
            const float4 zl = Z[t.at + j * pitch - 1], zr = Z[t.at + j * pitch + 1];
            const float2 V0 = lo2(zl), V1 = hi2(zl), V4 = lo2(zr), V5 = hi2(zr);
            const float2 W0 = make_float2(zl.y, zl.z), W1 = make_float2(zl.w, pz[0].x);
            const float2 W2 = make_float2(pz[0].y, pz[1].x), W3 = make_float2(pz[1].y, zr.x);
            const float2 W4 = make_float2(zr.y, zr.z);
            pxz[0] = d1_pair(W2, W1, pz[1], V1, W3, W0, V4, V0, a.cx1);
            pxz[1] = d1_pair(W3, W2, V4, pz[0], W4, W1, V5, V1, a.cx1);
        }
        strips(j, w, pxx, pzz, px, pz);
        float4 e4 = kap, n4 = kap, b4 = kap, c4 = kap, s4 = kap;
        if (APPROX != kAcoustic) { e4 = model(1, j); n4 = model(2, j); b4 = model(3, j); }
        if (APPROX == kTTI) { c4 = model(4, j); s4 = model(5, j); }
        float2 o[2];
#pragma unroll
        for (int m = 0; m < 2; m++) {
            const float2 uc = m ? hi2(c) : lo2(c), cxm = m ? hi2(t.cx) : lo2(t.cx);
            float2 u1 = m ? hi2(old[j]) : lo2(old[j]);
            if (t.damp) u1 = pmul2(pmul2(u1, cxm), bc2(t.cz[j]));   // damping of U(t-1) deferred to this read
            const float2 base = fsub2(padd2(uc, uc), u1);
            float2 v = update_pair<APPROX>(m ? hi2(kap) : lo2(kap), base, pxx[m], pzz[m], px[m], pz[m], pxz[m],
                                           m ? hi2(e4) : lo2(e4), m ? hi2(n4) : lo2(n4), m ? hi2(b4) : lo2(b4),
                                           m ? hi2(c4) : lo2(c4), m ? hi2(s4) : lo2(s4));
            if (t.damp) v = pmul2(pmul2(v, cxm), bc2(t.cz[j]));
            o[m] = v;
        }
        out[j] = make_float4(o[0].x, o[0].y, o[1].x, o[1].y);
    }
    // cells off the update region stay zero
    if (t.valid != (1u << R) - 1u)
#pragma unroll
        for (int j = 0; j < R; j++)
            if (!(t.valid >> j & 1u)) out[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t.tail)
#pragma unroll
        for (int j = 0; j < R; j++) {
            if (t.x + 1 >= a.nx - 4) out[j].y = 0.f;
            if (t.x + 2 >= a.nx - 4) out[j].z = 0.f;
            if (t.x + 3 >= a.nx - 4) out[j].w = 0.f;
        }
}

// Index of a cell in the list of saved band cells (band_cell's inverse), -1 off
// the band.
__device__ __forceinline__ int tile_band_index(int zi, int xi, int nzi, int nxi) {
    if (zi < 0 || zi >= nzi || xi < 0 || xi >= nxi) return -1;
    if (zi < 4) return zi * nxi + xi;
    if (zi >= nzi - 4) return (zi - (nzi - 8)) * nxi + xi;
    if (xi < 4) return 8 * nxi + (zi - 4) * 4 + xi;
    if (xi >= nxi - 4) return 8 * nxi + 4 * (nzi - 8) + (zi - 4) * 4 + xi - (nxi - 4);
    return -1;
}

// The saved value of band cell i of a shot at time `tt`.
__device__ __forceinline__ float tile_band_value(const TileArgs& t, int shot, int tt, int i) {
    const long long nb = band_cells(t.nzi, t.nxi);
    const long long nchunk = (nb + kBandChunk - 1) / kBandChunk;
    const long long row = (long long)tt * t.band_shots + shot;
    if (t.band_store == 0) return reinterpret_cast<const float*>(t.band)[row * nb + i];
    const float v = t.band_store == 1 ? band_unpack(reinterpret_cast<const __nv_bfloat16*>(t.band)[row * nb + i])
                                      : band_unpack(reinterpret_cast<const __half*>(t.band)[row * nb + i]);
    return v * t.band_scale[row * nchunk + i / kBandChunk];
}

// Forward time loop, steps k0 .. k1-1, of the shots shot0 .. (one block per
// tile of each): see the head of the file.
template <int APPROX, int R, bool REVERSE = false>
__global__ void __launch_bounds__(kTileThreads, 1) tile_forward_kernel(const TileArgs t)
{
    extern __shared__ float4 tsm[];
    __shared__ int alive;
    const StepArgs& a = t.s;
    const TileShape& g = t.g;
    const int ntiles = g.nty * g.ntx;
    const int shot = t.shot0 + blockIdx.x / ntiles, tile = blockIdx.x % ntiles;
    const int tid = threadIdx.x, nthr = blockDim.x;
    const TileCells<R> own = tile_cells<R>(a, g, tile, kTilePitch);
    const int copy = (g.nrg * R + 8) * kTilePitch;
    float4* A = tsm;                       // U(k)
    float4* B = tsm + copy;                // U(k+1)
    constexpr int ncopy = APPROX == kTTI ? 3 : 2;
    float4* const Z = tsm + 2 * copy;      // TTI: z derivative of U(k)
    float4* const M = tsm + ncopy * copy + tid;
    const long long so = (long long)shot * a.shot_stride;
    [[maybe_unused]] const long long fbytes = (long long)a.B * a.shot_stride * 4;
    [[maybe_unused]] const long long mbytes = (long long)a.nz * a.P * 4;

    constexpr int dir = REVERSE ? -1 : 1;

    // the state and the models of the thread's cells
    float4 cur[R], old[R], kap[R];
    {
        for (int i = tid; i < ncopy * copy; i += nthr) tsm[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        const float* const in0 = t.slots ? t.slots + ((REVERSE ? t.k1 - 1 : t.k0) - t.kslot) * t.slot_stride
                                 : t.set0 ? t.ex[1][0] : t.ex[0][0];
        const float* const in1 = t.slots ? in0 - dir * t.slot_stride : t.set0 ? t.ex[1][1] : t.ex[0][1];
        const float* const mod[6] = {a.kap, a.e2, a.m1, a.m2, a.cth, a.sth};
#pragma unroll
        for (int j = 0; j < R; j++) {
            const bool v = own.valid >> j & 1u;
            const int z = v ? own.z + j : -1;
            cur[j] = tile_fetch(in0 + so, z, own.x, a.nz, a.P, in0, fbytes);
            old[j] = tile_fetch(in1 + so, z, own.x, a.nz, a.P, in1, fbytes);
            kap[j] = tile_fetch(a.kap, z, own.x, a.nz, a.P, a.kap, mbytes);
            if (APPROX != kAcoustic)
#pragma unroll
                for (int i = 0; i < tile_models<APPROX>(); i++)
                    M[(i * R + j) * nthr] = tile_fetch(mod[i], z, own.x, a.nz, a.P, mod[i], mbytes);
        }
        __syncthreads();
        if (own.valid)
#pragma unroll
            for (int j = 0; j < R; j++) A[own.at + j * kTilePitch] = cur[j];
    }
    auto model = [&](int i, int j) { return APPROX == kAcoustic ? kap[j] : M[(i * R + j) * nthr]; };

    // the source, if it is one of the thread's cells
    const int sz = *PAM_CHK(&a.src_z[shot], a.src_z, a.B * 4, 4, 101);
    const int sx = *PAM_CHK(&a.src_x[shot], a.src_x, a.B * 4, 4, 101);
    const int srow = sz - own.z;
    const bool has_src = own.valid && srow >= 0 && srow < R && (own.valid >> srow & 1u) && sx >= own.x && sx < own.x + 4 &&
                         sx < a.nx - 4;
    // the first of the receivers that the thread records: place and damping
    // factors, x then z, as in the one-step kernels' recording
    const int rl = t.rec.per_shot ? shot * ntiles + tile : tile;
    const int rb = t.rec.seis ? t.rec_beg[rl] : 0, re = t.rec.seis ? t.rec_beg[rl + 1] : 0;
    const int ez0 = 4 + (tile / g.ntx) * g.TZ - g.halo * g.T - 4, ex0 = 4 + (tile % g.ntx) * g.TX - g.halo * g.T;
    [[maybe_unused]] const long long sbytes = (long long)a.B * t.rec.nt_data * t.rec.nrec * 4;
    float* const seis = t.rec.seis + (long long)shot * t.rec.nt_data * t.rec.nrec;
    auto place = [&](int2 e, int& off, float& fx, float& fz) {
        const int z = e.x >> 16, x = e.x & 0xffff;
        off = (z - ez0) * (4 * kTilePitch) + x - ex0;
        fx = x < a.N ? a.cerjan[x] : x >= a.nx - a.N ? a.cerjan[a.nx - 1 - x] : 1.0f;
        fz = z < a.N ? a.cerjan[z] : z >= a.nz - a.N ? a.cerjan[a.nz - 1 - z] : 1.0f;
    };
    auto sample = [&](int it, int r, int off, float fx, float fz) {
        const float v = reinterpret_cast<const float*>(A)[off] * fx * fz;
        *PAM_CHK(&seis[(long long)it * t.rec.nrec + r], t.rec.seis, sbytes, 4, 102) = v;
        if (!isfinite(v)) atomicOr(t.status, 1);
    };
    int roff = 0, rr = -1;
    float rfx = 1.0f, rfz = 1.0f;
    if (rb + tid < re) {
        const int2 e = t.rec_ent[rb + tid];
        rr = e.y;
        place(e, roff, rfx, rfz);
    }
    __syncthreads();

    int k = REVERSE ? t.k1 - 1 : t.k0, left = t.k1 - t.k0, set = t.set0;
    unsigned want = 0;
    const long long o = so + (long long)own.z * a.P + own.x;   // the thread's first cell in a field
    float amp = k + 1 < t.nt ? t.wavelet[k + 1] : 0.0f;
    // rows with cells of the saved band, and their values at the next time
    unsigned brow = 0;
    float4 bval[REVERSE ? R : 1];
    auto band_fetch = [&](int tt) {
#pragma unroll
        for (int j = 0; j < R; j++)
            if (REVERSE && (brow >> j & 1u) && tt >= 0) {
                float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int c = tile_band_index(own.z + j - a.N, own.x + i - a.N, t.nzi, t.nxi);
                    if (c >= 0) v[i] = tile_band_value(t, shot, tt, c);
                }
                bval[j] = make_float4(v[0], v[1], v[2], v[3]);
            }
    };
    if (REVERSE && t.band) {
#pragma unroll
        for (int j = 0; j < R; j++)
#pragma unroll
            for (int i = 0; i < 4; i++)
                if ((own.valid >> j & 1u) && tile_band_index(own.z + j - a.N, own.x + i - a.N, t.nzi, t.nxi) >= 0)
                    brow |= 1u << j;
        band_fetch(k - 1);
    }
    while (left > 0) {
        const int nsub = min(g.T, left);
        for (int s = 0; s < nsub; s++, k += dir, left--) {
            const int kn = k + dir + 1;
            const float next_amp = kn < t.nt && kn >= 0 ? t.wavelet[kn] : 0.0f;
            if (!REVERSE && k >= t.itlag) {
                if (rr >= 0) sample(k - t.itlag, rr, roff, rfx, rfz);
                for (int i = rb + tid + nthr; i < re; i += nthr) {
                    const int2 e = t.rec_ent[i];
                    int off;
                    float fx, fz;
                    place(e, off, fx, fz);
                    sample(k - t.itlag, e.y, off, fx, fz);
                }
            }
            // a region of halo 4 (nsub - 1 - s) around the tile, whole threads of it
            const bool active = own.need <= 4 * (nsub - 1 - s);
            float4 out[R];
            if (active || APPROX == kTTI) tile_step<APPROX, R>(a, own, kTilePitch, A, Z, active, cur, old, model, out);
            if (active) {
                if (has_src)
#pragma unroll
                    for (int j = 0; j < R; j++)
                        if (j == srow) {
                            out[j].x += sx == own.x ? amp : 0.f;
                            out[j].y += sx == own.x + 1 ? amp : 0.f;
                            out[j].z += sx == own.x + 2 ? amp : 0.f;
                            out[j].w += sx == own.x + 3 ? amp : 0.f;
                        }
                if (REVERSE && brow)
#pragma unroll
                    for (int j = 0; j < R; j++)
                        if (brow >> j & 1u) {
                            const int zi = own.z + j - a.N, xi = own.x - a.N;
                            if (tile_band_index(zi, xi, t.nzi, t.nxi) >= 0) out[j].x = bval[j].x;
                            if (tile_band_index(zi, xi + 1, t.nzi, t.nxi) >= 0) out[j].y = bval[j].y;
                            if (tile_band_index(zi, xi + 2, t.nzi, t.nxi) >= 0) out[j].z = bval[j].z;
                            if (tile_band_index(zi, xi + 3, t.nzi, t.nxi) >= 0) out[j].w = bval[j].w;
                        }
#pragma unroll
                for (int j = 0; j < R; j++) {
                    old[j] = cur[j];
                    cur[j] = out[j];
                    B[own.at + j * kTilePitch] = out[j];
                }
            }
            if (REVERSE && brow) band_fetch(k - 2);
            float4* const sw = A;
            A = B;
            B = sw;
            amp = next_amp;
            if (t.slots && own.mine) {
                float* const u = t.slots + (k + dir - t.kslot) * t.slot_stride;
#pragma unroll
                for (int j = 0; j < R; j++)
                    if (own.mine >> j & 1u)
                        *reinterpret_cast<float4*>(PAM_CHK(u + o + j * a.P, u, fbytes, 16, 105)) = cur[j];
            }
            if (s + 1 < nsub) __syncthreads();
        }
        // publish the tile into the other set
        float* const pub0 = t.slots ? t.slots + (k - t.kslot) * t.slot_stride : set ? t.ex[0][0] : t.ex[1][0];
        float* const pub1 = t.slots ? pub0 - dir * t.slot_stride : set ? t.ex[0][1] : t.ex[1][1];
        if (!t.slots)
#pragma unroll
            for (int j = 0; j < R; j++)
                if (own.mine >> j & 1u) {
                    *reinterpret_cast<float4*>(PAM_CHK(pub0 + o + j * a.P, pub0, fbytes, 16, 103)) = cur[j];
                    *reinterpret_cast<float4*>(PAM_CHK(pub1 + o + j * a.P, pub1, fbytes, 16, 103)) = old[j];
                }
        set ^= 1;
        if (left <= 0) break;
        want += gridDim.x;
        if (!tile_barrier(t, want, &alive)) {
            if (!REVERSE) tile_poison(t, seis, rb, re, k);
            return;
        }
        // the halo, both fields, from the other tiles
        const unsigned halo = own.valid & ~own.mine;
        if (halo) {
#pragma unroll
            for (int j = 0; j < R; j++)
                if (halo >> j & 1u) {
                    cur[j] = tile_halo(pub0 + o + j * a.P, pub0, fbytes);
                    old[j] = tile_halo(pub1 + o + j * a.P, pub1, fbytes);
                }
#pragma unroll
            for (int j = 0; j < R; j++)
                if (halo >> j & 1u) A[own.at + j * kTilePitch] = cur[j];
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------- backward sweeps

// The backward sweep of a small acoustic batch over the steps t = k1-1 .. k0
// of a segment whose source fields U(t) are stored, with the fields as
// tiles, like the forward loop; the receiver-side field advances by the forward
// recursion (see inject_adjoint_kernel), and the sums of each cell over time
// stay in the block until the launch ends.
//   kTileExact: w(t) from w(t+1), w(t+2), then the residual of time t at the
//               receivers; G += w(t+1) L U(t) (t <= nt-2), I += U(t)^2
//   kTileRtm:   G += Ub(t) U(t), I += U(t)^2, Ub(t-1) from Ub(t), Ub(t+1), then
//               the data of time t-1
// U(t) of the tile and four cells around it comes through a ring of shared
// copies filled by cp.async three steps ahead; the data of a group's steps are
// staged in shared memory one group ahead.
enum TileMode { kTileExact = 0, kTileRtm = 1 };

constexpr int kTileRing = 4;
constexpr int kTileInject = 1024;      // most receiver entries of a tile with its halo

struct TileAdjArgs {
    TileArgs f;                          // k0, k1: the segment; slots: U(t); ex: the receiver-side field
    const int* __restrict__ inj_beg;     // [tiles (per shot)][threads + 1] entries of each thread's cells
    const int2* __restrict__ inj_ent;    // (row << 16 | column of the expanded grid, receiver)
    const float* __restrict__ data;      // [B][nt_data][nrec] residual or observed data
    float scale;                         // of the data (kTileRtm)
    float* gsum;                         // [B][nz][P] sums, continued
    float* isum;
};

__host__ __device__ inline int tile_pitch(const TileShape& g) { return g.EXq; }
__host__ __device__ inline size_t tile_adj_smem_bytes(const TileShape& g) {
    const size_t copy = (size_t)(g.nrg * g.R + 8) * tile_pitch(g) * 16;
    return (2 + kTileRing) * copy + (size_t)2 * g.R * tile_threads(g) * 16 + (size_t)kTileInject * (16 + 2 * 4 * g.T);
}

__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}

// s + a b, the product rounded before it is added, as where the one-step
// kernels pass it through shared memory
__device__ __forceinline__ float4 add_product(float4 s, float4 a, float4 b) {
    return make_float4(__fadd_rn(s.x, __fmul_rn(a.x, b.x)), __fadd_rn(s.y, __fmul_rn(a.y, b.y)),
                       __fadd_rn(s.z, __fmul_rn(a.z, b.z)), __fadd_rn(s.w, __fmul_rn(a.w, b.w)));
}

template <int MODE, int R>
__global__ void __launch_bounds__(kTileThreads, 1) tile_adjoint_kernel(const TileAdjArgs ta)
{
    extern __shared__ float4 tsm[];
    __shared__ int alive;
    const TileArgs& t = ta.f;
    const StepArgs& a = t.s;
    const TileShape& g = t.g;
    const int ntiles = g.nty * g.ntx;
    const int shot = t.shot0 + blockIdx.x / ntiles, tile = blockIdx.x % ntiles;
    const int tid = threadIdx.x, nthr = blockDim.x, pitch = tile_pitch(g);
    const TileCells<R> own = tile_cells<R>(a, g, tile, pitch);
    const int copy = (g.nrg * R + 8) * pitch;
    float4* A = tsm;                               // the field read by the step
    float4* B = tsm + copy;                        // the field it writes
    float4* const ring = tsm + 2 * copy;           // copies of U(t), at t & 3
    float4* const G = ring + kTileRing * copy + tid;   // [R] sums of the thread's cells
    float4* const I = G + R * nthr;
    float4* const ient = ring + kTileRing * copy + 2 * R * nthr;       // entries: offset, factors, kappa
    float* const idat = reinterpret_cast<float*>(ient + kTileInject);  // [2][T][entries] staged data
    const long long so = (long long)shot * a.shot_stride;
    const long long o = so + (long long)own.z * a.P + own.x;
    [[maybe_unused]] const long long fbytes = (long long)a.B * a.shot_stride * 4;
    [[maybe_unused]] const long long mbytes = (long long)a.nz * a.P * 4;

    // U(t) is needed on the tile (kTileRtm) and four cells around it (kTileExact)
    const bool want_u = own.need <= (MODE == kTileExact ? 4 : 0);
    auto fetch_u = [&](int tt) {
        if (tt >= t.k0 && want_u) {
            const float* const u = t.slots + (tt - t.kslot) * t.slot_stride;
            float4* const dst = ring + (tt & (kTileRing - 1)) * copy + own.at;
#pragma unroll
            for (int j = 0; j < R; j++)
                if (own.valid >> j & 1u) cp_async16(dst + j * pitch, PAM_CHK(u + o + j * a.P, u, fbytes, 16, 110));
        }
        cp_async_commit();
    };

    float4 cur[R], old[R], kap[R];
    for (int i = tid; i < (2 + kTileRing) * copy; i += nthr) tsm[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    {
        const float* const in0 = t.set0 ? t.ex[1][0] : t.ex[0][0];
        const float* const in1 = t.set0 ? t.ex[1][1] : t.ex[0][1];
#pragma unroll
        for (int j = 0; j < R; j++) {
            const int z = own.valid >> j & 1u ? own.z + j : -1;
            cur[j] = tile_fetch(in0 + so, z, own.x, a.nz, a.P, in0, fbytes);
            old[j] = tile_fetch(in1 + so, z, own.x, a.nz, a.P, in1, fbytes);
            kap[j] = tile_fetch(a.kap, z, own.x, a.nz, a.P, a.kap, mbytes);
            // the sums go on from the last segment's
            G[j * nthr] = tile_fetch(ta.gsum + so, z, own.x, a.nz, a.P, ta.gsum, fbytes);
            I[j * nthr] = tile_fetch(ta.isum + so, z, own.x, a.nz, a.P, ta.isum, fbytes);
        }
    }
    auto model = [&](int, int j) { return kap[j]; };

    // the receivers of the thread's cells: entries [ib, ie) of the tile's list,
    // which starts at il; the field time of the injection after step t is t - lag
    const long long list = (long long)(t.rec.per_shot ? shot * ntiles + tile : tile) * (nthr + 1);
    const int il = ta.inj_beg[list], nent = ta.inj_beg[list + nthr] - il;
    const int ib = ta.inj_beg[list + tid] - il, ie = ta.inj_beg[list + tid + 1] - il;
    constexpr int lag = MODE == kTileExact ? 0 : 1;
    const float* const data = ta.data + (long long)shot * t.rec.nt_data * t.rec.nrec;
    for (int i = ib; i < ie; i++) {
        const int2 e = ta.inj_ent[il + i];
        const int z = e.x >> 16, x = e.x & 0xffff;
        const float fx = x < a.N ? a.cerjan[x] : x >= a.nx - a.N ? a.cerjan[a.nx - 1 - x] : 1.0f;
        const float fz = z < a.N ? a.cerjan[z] : z >= a.nz - a.N ? a.cerjan[a.nz - 1 - z] : 1.0f;
        const int off = (own.at + (z - own.z) * pitch) * 4 + x - own.x;
        ient[i] = make_float4(__int_as_float(off), fx, fz, a.kap[(long long)z * a.P + x]);
    }
    // the data of the group of n steps whose first is tt, staged at parity p
    auto stage = [&](int tt, int n, int p) {
        for (int i = tid; i < nent; i += nthr) {
            const int r = ta.inj_ent[il + i].y;
            for (int s = 0; s < n; s++) {
                const int it = tt - s - lag - t.itlag;
                float* const dst = idat + (p * g.T + s) * nent + i;
                if (it >= 0) cp_async4(dst, data + (long long)it * t.rec.nrec + r);
                else *dst = 0.0f;
            }
        }
    };

    int k = t.k1 - 1, set = t.set0, parity = 0;
    unsigned want = 0;
    stage(k, min(g.T, k - t.k0 + 1), 0);
    __syncthreads();                               // the copies are zero before they are written
    fetch_u(k);
    fetch_u(k - 1);
    fetch_u(k - 2);
    if (own.valid)
#pragma unroll
        for (int j = 0; j < R; j++) A[own.at + j * pitch] = cur[j];
    cp_async_wait<2>();                            // U(k) and the first group's data
    __syncthreads();

    while (k >= t.k0) {
        const int nsub = min(g.T, k - t.k0 + 1);
        if (k - nsub >= t.k0) stage(k - nsub, min(g.T, k - nsub - t.k0 + 1), parity ^ 1);
        for (int s = 0; s < nsub; s++, k--) {
            fetch_u(k - 3);
            if (own.mine) {
                // the sums of the tile's cells
                const float4* const U = ring + (k & (kTileRing - 1)) * copy + own.at;
                float4 w[R + 8];
                if (MODE == kTileExact)
#pragma unroll
                    for (int j = 0; j < R + 8; j++) w[j] = U[(j - 4) * pitch];
#pragma unroll
                for (int j = 0; j < R; j++) {
                    if (!(own.mine >> j & 1u)) continue;
                    const float4 c = MODE == kTileExact ? w[j + 4] : U[j * pitch];
                    float4 q = I[j * nthr];
                    if (MODE == kTileExact) {
                        const float4 l = U[j * pitch - 1], r = U[j * pitch + 1];
                        const float2 P0 = lo2(l), P1 = hi2(l), P2 = lo2(c), P3 = hi2(c), P4 = lo2(r), P5 = hi2(r);
                        const float2 O0 = make_float2(l.y, l.z), O1 = make_float2(l.w, c.x), O2 = make_float2(c.y, c.z);
                        const float2 O3 = make_float2(c.w, r.x), O4 = make_float2(r.y, r.z);
                        q = add_product(q, c, c);
                        if (k <= t.nt - 2) {
                            const float2 L0 = padd2(d2_pair(P2, O2, O1, P3, P1, O3, O0, P4, P0, a.inv_dx2),
                                                    d2_pair(lo2(c), lo2(w[j + 5]), lo2(w[j + 3]), lo2(w[j + 6]),
                                                            lo2(w[j + 2]), lo2(w[j + 7]), lo2(w[j + 1]), lo2(w[j + 8]),
                                                            lo2(w[j]), a.inv_dz2));
                            const float2 L1 = padd2(d2_pair(P3, O3, O2, P4, P2, O4, O1, P5, P1, a.inv_dx2),
                                                    d2_pair(hi2(c), hi2(w[j + 5]), hi2(w[j + 3]), hi2(w[j + 6]),
                                                            hi2(w[j + 2]), hi2(w[j + 7]), hi2(w[j + 1]), hi2(w[j + 8]),
                                                            hi2(w[j]), a.inv_dz2));
                            G[j * nthr] = add_product(G[j * nthr], cur[j], make_float4(L0.x, L0.y, L1.x, L1.y));
                        }
                    } else {
                        const float2 i0 = pfma2(lo2(c), lo2(c), lo2(q)), i1 = pfma2(hi2(c), hi2(c), hi2(q));
                        q = make_float4(i0.x, i0.y, i1.x, i1.y);
                        const float4 p = G[j * nthr];
                        const float2 g0 = pfma2(lo2(cur[j]), lo2(c), lo2(p)), g1 = pfma2(hi2(cur[j]), hi2(c), hi2(p));
                        G[j * nthr] = make_float4(g0.x, g0.y, g1.x, g1.y);
                    }
                    I[j * nthr] = q;
                }
            }
            if (own.need <= 4 * (nsub - 1 - s)) {
                float4 out[R];
                tile_step<kAcoustic, R>(a, own, pitch, A, nullptr, true, cur, old, model, out);
#pragma unroll
                for (int j = 0; j < R; j++) {
                    old[j] = cur[j];
                    cur[j] = out[j];
                    B[own.at + j * pitch] = out[j];
                }
                if (ie > ib) {
                    const float* const d = idat + (parity * g.T + s) * nent;
                    for (int i = ib; i < ie; i++) {
                        const float4 e = ient[i];
                        float* const p = reinterpret_cast<float*>(B) + __float_as_int(e.x);
                        float v = d[i];
                        if (MODE == kTileExact) {
                            v = __fmul_rn(__fmul_rn(v, e.y), e.z);
                            v = __fmul_rn(e.w, __fmul_rn(__fmul_rn(v, e.y), e.z));
                        } else {
                            v = __fmul_rn(v, ta.scale);
                        }
                        *p = __fadd_rn(*p, v);
                    }
#pragma unroll
                    for (int j = 0; j < R; j++) cur[j] = B[own.at + j * pitch];
                }
            }
            float4* const sw = A;
            A = B;
            B = sw;
            if (s + 1 < nsub) {
                cp_async_wait<2>();                // U of the next step
                __syncthreads();
            }
        }
        parity ^= 1;
        float* const pub0 = set ? t.ex[0][0] : t.ex[1][0];
        float* const pub1 = set ? t.ex[0][1] : t.ex[1][1];
#pragma unroll
        for (int j = 0; j < R; j++)
            if (own.mine >> j & 1u) {
                *reinterpret_cast<float4*>(PAM_CHK(pub0 + o + j * a.P, pub0, fbytes, 16, 111)) = cur[j];
                *reinterpret_cast<float4*>(PAM_CHK(pub1 + o + j * a.P, pub1, fbytes, 16, 111)) = old[j];
            }
        set ^= 1;
        if (k < t.k0) break;
        cp_async_wait<0>();                        // the next group's data (and U)
        want += gridDim.x;
        if (!tile_barrier(t, want, &alive)) return;
        const unsigned halo = own.valid & ~own.mine;
        if (halo) {
#pragma unroll
            for (int j = 0; j < R; j++)
                if (halo >> j & 1u) {
                    cur[j] = tile_halo(pub0 + o + j * a.P, pub0, fbytes);
                    old[j] = tile_halo(pub1 + o + j * a.P, pub1, fbytes);
                }
#pragma unroll
            for (int j = 0; j < R; j++)
                if (halo >> j & 1u) A[own.at + j * pitch] = cur[j];
        }
        __syncthreads();
    }
    cp_async_wait<0>();
#pragma unroll
    for (int j = 0; j < R; j++)
        if (own.mine >> j & 1u) {
            *reinterpret_cast<float4*>(PAM_CHK(ta.gsum + o + (long long)j * a.P, ta.gsum, fbytes, 16, 112)) = G[j * nthr];
            *reinterpret_cast<float4*>(PAM_CHK(ta.isum + o + (long long)j * a.P, ta.isum, fbytes, 16, 112)) = I[j * nthr];
        }
}

// ---------------------------------------------------------------- CPML

// Steps of a field with the perfectly matched layer as tiles: the forward loop
// (kTileForwardRole) and the receiver side of acoustic migration (kTileRtmRole,
// as tile_adjoint_kernel<kTileRtm>).  A step needs the new psi of the strip
// cells four cells away, hence U eight cells away, so the regions lose eight
// cells a step; psi goes to the neighbours through two more shared copies
// (a second barrier per step), zeta stays with its thread in shared memory.
// Per cell the expressions of the strip kernels and of step_kernel.
//
// One shot of 377 x 743 cells takes 10.7 us a step as a graph of four launches
// (two strip kernels, the step, the recording).
enum TileRole { kTileForwardRole = 0, kTileRtmRole = 1 };

struct TileCpmlArgs {
    TileAdjArgs r;                   // r.f: the loop; the rest of r: kTileRtmRole
    float* mem[2];                   // [set][4][B][nz][P] psi x, zeta x, psi z, zeta z as published; [0] zero before step 0
    const float2* __restrict__ cxab; // [nz][2N]
    const float2* __restrict__ czab; // [2N][P]
};

__host__ __device__ inline size_t tile_cpml_smem_bytes(const TileShape& g, int models, int role) {
    const size_t copy = (size_t)(g.nrg * g.R + 8) * tile_pitch(g) * 16, rows = (size_t)g.R * tile_threads(g) * 16;
    return 4 * copy + 6 * rows + (models > 1 ? models * rows : 0) +
           (role == kTileRtmRole ? 2 * rows + (size_t)kTileInject * (16 + 2 * 4 * g.T) : 0);
}

// Sums and differences of pairs, each half on its own: the packed forms of a
// product and a sum that follow each other in straight-line code are contracted
// into one operation whatever their rounding mode says.  step_kernel's branch
// around its strip terms and the strip kernels keep them apart here.
__device__ __forceinline__ float2 add_apart(float2 a, float2 b) {
    return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y));
}
// The recursions of psi and zeta, a old + b v, contracted as in the strip
// kernels; d1_pair_ref and d2_pair are their derivatives, bit for bit.
__device__ __forceinline__ float2 cpml_recursion(float2 a, float2 b, float2 old, float2 v) {
    return pfma2(a, old, pmul2(b, v));
}
// Second derivative without its 1/d^2 (d2_pair is this times inv).
__device__ __forceinline__ float2 d2_pair_sum(float2 c, float2 p1, float2 m1, float2 p2, float2 m2, float2 p3, float2 m3,
                                              float2 p4, float2 m4) {
    float2 t = pmul2(bc2(kC0), c);
    t = pfma2(bc2(kC1), padd2(p1, m1), t);
    t = pfma2(bc2(kC2), padd2(p2, m2), t);
    t = pfma2(bc2(kC3), padd2(p3, m3), t);
    return pfma2(bc2(kC4), padd2(p4, m4), t);
}
__device__ __forceinline__ void d2_quad_sum(const float4& l, const float4& c, const float4& r, float2 (&d)[2]) {
    const float2 P0 = lo2(l), P1 = hi2(l), P2 = lo2(c), P3 = hi2(c), P4 = lo2(r), P5 = hi2(r);
    const float2 O0 = make_float2(l.y, l.z), O1 = make_float2(l.w, c.x), O2 = make_float2(c.y, c.z);
    const float2 O3 = make_float2(c.w, r.x), O4 = make_float2(r.y, r.z);
    d[0] = d2_pair_sum(P2, O2, O1, P3, P1, O3, O0, P4, P0);
    d[1] = d2_pair_sum(P3, O3, O2, P4, P2, O4, O1, P5, P1);
}
// First derivative along x of the two pairs of a quad c with its neighbours l, r.
__device__ __forceinline__ void d1_quad(const float4& l, const float4& c, const float4& r, float inv, float2 (&d)[2]) {
    const float2 P0 = lo2(l), P1 = hi2(l), P2 = lo2(c), P3 = hi2(c), P4 = lo2(r), P5 = hi2(r);
    const float2 O0 = make_float2(l.y, l.z), O1 = make_float2(l.w, c.x), O2 = make_float2(c.y, c.z);
    const float2 O3 = make_float2(c.w, r.x), O4 = make_float2(r.y, r.z);
    d[0] = d1_pair_ref(O2, O1, P3, P1, O3, O0, P4, P0, inv);
    d[1] = d1_pair_ref(O3, O2, P4, P2, O4, O1, P5, P1, inv);
}

// One row per thread, in 64 registers: a cut that fits with two rows in twice the
// registers (384 threads at most) fits with one too, in no more shared memory and
// with a cheaper exchange.
constexpr int kTileCpmlRows = 1, kTileCpmlThreads = 1024;

template <int APPROX, int ROLE>
__global__ void __launch_bounds__(kTileCpmlThreads, 1) tile_cpml_kernel(const TileCpmlArgs tc)
{
    constexpr int R = kTileCpmlRows;
    extern __shared__ float4 tsm[];
    __shared__ int alive;
    const TileAdjArgs& ta = tc.r;
    const TileArgs& t = ta.f;
    const StepArgs& a = t.s;
    const TileShape& g = t.g;
    const int ntiles = g.nty * g.ntx;
    const int shot = t.shot0 + blockIdx.x / ntiles, tile = blockIdx.x % ntiles;
    const int tid = threadIdx.x, nthr = blockDim.x, pitch = tile_pitch(g);
    const TileCells<R> own = tile_cells<R>(a, g, tile, pitch);
    const int copy = (g.nrg * R + 8) * pitch;
    float4* A = tsm;                               // U(k)
    float4* B = tsm + copy;                        // U(k+1)
    float4* __restrict__ const PX = tsm + 2 * copy;             // psi of the x strips, of the z strips
    float4* __restrict__ const PZ = tsm + 3 * copy;
    float4* __restrict__ const ZX = tsm + 4 * copy + tid;       // [R] zeta of the thread's cells
    float4* __restrict__ const ZZ = ZX + R * nthr;
    float4* __restrict__ const AX = ZZ + R * nthr;              // [R] (a, b) of the thread's cells, zero off the strips
    float4* __restrict__ const BX = AX + R * nthr;
    float4* __restrict__ const AZ = BX + R * nthr;
    float4* __restrict__ const BZ = AZ + R * nthr;
    float4* const M = BZ + R * nthr;               // models (not acoustic)
    constexpr int nmod = APPROX == kAcoustic ? 0 : tile_models<APPROX>();
    float4* const G = M + nmod * R * nthr;         // kTileRtmRole: the sums, the entries and the staged data
    float4* const I = G + R * nthr;
    float4* const ient = I + R * nthr - tid;
    float* const idat = reinterpret_cast<float*>(ient + kTileInject);
    const long long so = (long long)shot * a.shot_stride;
    const long long o = so + (long long)own.z * a.P + own.x;
    [[maybe_unused]] const long long fbytes = (long long)a.B * a.shot_stride * 4;
    [[maybe_unused]] const long long mbytes = (long long)a.nz * a.P * 4;
    const long long mstride = (long long)t.mem_shots * a.shot_stride;

    // which of the thread's cells lie in a strip
    unsigned xin = 0;                              // columns
    unsigned zin = 0;                              // rows
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int x = own.x + i;
        if ((x >= 4 && x < a.N) || (x >= a.nx - a.N && x < a.nx - 4)) xin |= 1u << i;
    }
#pragma unroll
    for (int j = 0; j < R; j++) {
        const int z = own.z + j;
        if ((own.valid >> j & 1u) && (z < a.N || z >= a.nz - a.N)) zin |= 1u << j;
    }
    if (!own.valid) xin = 0;
    // acoustic: rows that step_kernel takes in its march without border code (a
    // 128-column tile and an 8-row segment, the height that small batches run
    // with, clear of the border), where its sum of the two second derivatives
    // takes the x one's scaling with it in one operation; elsewhere the branch
    // around the strip terms keeps the two apart
    unsigned inner = 0;
    if (APPROX == kAcoustic) {
        const int tx = own.x / kTileWide * kTileWide - 4;
        if (own.valid && tx >= a.N && tx + kTileWide + 8 <= a.nx - a.N)
#pragma unroll
            for (int j = 0; j < R; j++) {
                const int z = 4 + (own.z + j - 4) / 8 * 8;
                if ((own.valid >> j & 1u) && z >= a.N && min(z + 8, a.nz - 4) <= a.nz - a.N) inner |= 1u << j;
            }
    }

    float4 cur[R], old[R], kap[R];
    for (int i = tid; i < 4 * copy; i += nthr) tsm[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    {
        const float* const in0 = t.slots && ROLE == kTileForwardRole ? t.slots + (t.k0 - t.kslot) * t.slot_stride
                                 : t.set0                            ? t.ex[1][0] : t.ex[0][0];
        const float* const in1 = t.slots && ROLE == kTileForwardRole ? in0 - t.slot_stride
                                 : t.set0                            ? t.ex[1][1] : t.ex[0][1];
        const float* const mod[6] = {a.kap, a.e2, a.m1, a.m2, a.cth, a.sth};
        const float* const mem = t.set0 ? tc.mem[1] : tc.mem[0];
#pragma unroll
        for (int j = 0; j < R; j++) {
            const int z = own.valid >> j & 1u ? own.z + j : -1;
            cur[j] = tile_fetch(in0 + so, z, own.x, a.nz, a.P, in0, fbytes);
            old[j] = tile_fetch(in1 + so, z, own.x, a.nz, a.P, in1, fbytes);
            kap[j] = tile_fetch(a.kap, z, own.x, a.nz, a.P, a.kap, mbytes);
            if (APPROX != kAcoustic)
#pragma unroll
                for (int i = 0; i < tile_models<APPROX>(); i++)
                    M[(i * R + j) * nthr] = tile_fetch(mod[i], z, own.x, a.nz, a.P, mod[i], mbytes);
            const int zx = xin ? z : -1, zz = zin >> j & 1u ? z : -1;
            const float4 px = tile_fetch(mem + so, zx, own.x, a.nz, a.P, mem, fbytes);
            ZX[j * nthr] = tile_fetch(mem + mstride + so, zx, own.x, a.nz, a.P, mem + mstride, fbytes);
            const float4 pz = tile_fetch(mem + 2 * mstride + so, zz, own.x, a.nz, a.P, mem + 2 * mstride, fbytes);
            ZZ[j * nthr] = tile_fetch(mem + 3 * mstride + so, zz, own.x, a.nz, a.P, mem + 3 * mstride, fbytes);
            if (own.valid) {
                A[own.at + j * pitch] = cur[j];
                PX[own.at + j * pitch] = px;
                PZ[own.at + j * pitch] = pz;
            }
            if (ROLE == kTileRtmRole) {
                G[j * nthr] = tile_fetch(ta.gsum + so, z, own.x, a.nz, a.P, ta.gsum, fbytes);
                I[j * nthr] = tile_fetch(ta.isum + so, z, own.x, a.nz, a.P, ta.isum, fbytes);
            }
        }
    }
    auto model = [&](int i, int j) { return APPROX == kAcoustic ? kap[j] : M[(i * R + j) * nthr]; };
    // (a, b) of the thread's cells; zero off the strips, where psi and zeta stay zero
#pragma unroll
    for (int j = 0; j < R; j++) {
        float2 x[4], z[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int xx = own.x + i, zz = own.z + j;
            const int c = xx < a.N ? xx : xx - (a.nx - 2 * a.N), r = zz < a.N ? zz : zz - (a.nz - 2 * a.N);
            x[i] = z[i] = make_float2(0.f, 0.f);
            if ((own.valid >> j & 1u) && (xin >> i & 1u))
                x[i] = __ldg(PAM_CHK(&tc.cxab[(long long)zz * (2 * a.N) + c], tc.cxab, (long long)a.nz * 2 * a.N * 8, 8, 120));
            if ((zin >> j & 1u) && xx < a.nx - 4)
                z[i] = __ldg(PAM_CHK(&tc.czab[(long long)r * a.P + xx], tc.czab, (long long)2 * a.N * a.P * 8, 8, 121));
        }
        AX[j * nthr] = make_float4(x[0].x, x[1].x, x[2].x, x[3].x);
        BX[j * nthr] = make_float4(x[0].y, x[1].y, x[2].y, x[3].y);
        AZ[j * nthr] = make_float4(z[0].x, z[1].x, z[2].x, z[3].x);
        BZ[j * nthr] = make_float4(z[0].y, z[1].y, z[2].y, z[3].y);
    }

    // source and recording (kTileForwardRole), as in tile_forward_kernel
    int sz = 0, sx = 0, srow = 0, rb = 0, re = 0, roff = 0, rr = -1;
    bool has_src = false;
    const int ez0 = 4 + (tile / g.ntx) * g.TZ - g.halo * g.T - 4, ex0 = 4 + (tile % g.ntx) * g.TX - g.halo * g.T;
    [[maybe_unused]] const long long sbytes = (long long)a.B * t.rec.nt_data * t.rec.nrec * 4;
    float* const seis = t.rec.seis + (long long)shot * t.rec.nt_data * t.rec.nrec;
    auto place = [&](int2 e) { return ((e.x >> 16) - ez0) * (4 * pitch) + (e.x & 0xffff) - ex0; };
    auto sample = [&](int it, int r, int off) {
        const float v = reinterpret_cast<const float*>(A)[off];
        *PAM_CHK(&seis[(long long)it * t.rec.nrec + r], t.rec.seis, sbytes, 4, 122) = v;
        if (!isfinite(v)) atomicOr(t.status, 1);
    };
    if (ROLE == kTileForwardRole) {
        sz = *PAM_CHK(&a.src_z[shot], a.src_z, a.B * 4, 4, 101);
        sx = *PAM_CHK(&a.src_x[shot], a.src_x, a.B * 4, 4, 101);
        srow = sz - own.z;
        has_src = own.valid && srow >= 0 && srow < R && (own.valid >> srow & 1u) && sx >= own.x && sx < own.x + 4 &&
                  sx < a.nx - 4;
        const int rl = t.rec.per_shot ? shot * ntiles + tile : tile;
        rb = t.rec.seis ? t.rec_beg[rl] : 0;
        re = t.rec.seis ? t.rec_beg[rl + 1] : 0;
        if (rb + tid < re) {
            const int2 e = t.rec_ent[rb + tid];
            rr = e.y;
            roff = place(e);
        }
    }
    // the data injected (kTileRtmRole), as in tile_adjoint_kernel
    int il = 0, nent = 0, ib = 0, ie = 0;
    const float* const data = ta.data + (long long)shot * t.rec.nt_data * t.rec.nrec;
    auto stage = [&](int tt, int n, int p) {
        for (int i = tid; i < nent; i += nthr) {
            const int r = ta.inj_ent[il + i].y;
            for (int s = 0; s < n; s++) {
                const int it = tt - s - 1 - t.itlag;
                float* const dst = idat + (p * g.T + s) * nent + i;
                if (it >= 0) cp_async4(dst, data + (long long)it * t.rec.nrec + r);
                else *dst = 0.0f;
            }
        }
    };
    float4 pc[R], pn[R];                           // source field U(t) of the tile's cells, and the next one
    auto fetch_p = [&](int tt, float4 (&p)[R]) {
        const float* const u = t.slots + (tt - t.kslot) * t.slot_stride;
#pragma unroll
        for (int j = 0; j < R; j++)
            p[j] = tile_fetch(u + so, tt >= t.k0 && (own.mine >> j & 1u) ? own.z + j : -1, own.x, a.nz, a.P, u, fbytes);
    };
    int k = ROLE == kTileForwardRole ? t.k0 : t.k1 - 1;
    constexpr int dir = ROLE == kTileForwardRole ? 1 : -1;
    int left = t.k1 - t.k0;                        // steps to go
    if (ROLE == kTileRtmRole) {
        const long long list = (long long)(t.rec.per_shot ? shot * ntiles + tile : tile) * (nthr + 1);
        il = ta.inj_beg[list];
        nent = ta.inj_beg[list + nthr] - il;
        ib = ta.inj_beg[list + tid] - il;
        ie = ta.inj_beg[list + tid + 1] - il;
        for (int i = ib; i < ie; i++) {
            const int2 e = ta.inj_ent[il + i];
            ient[i].x = __int_as_float((own.at + ((e.x >> 16) - own.z) * pitch) * 4 + (e.x & 0xffff) - own.x);
        }
        stage(k, min(g.T, left), 0);
        cp_async_commit();
        fetch_p(k, pc);
        cp_async_wait<0>();
    }
    __syncthreads();

    int set = t.set0, parity = 0;
    unsigned want = 0;
    while (left > 0) {
        const int nsub = min(g.T, left);
        if (ROLE == kTileRtmRole && left > nsub) {
            stage(k - nsub, min(g.T, left - nsub), parity ^ 1);
            cp_async_commit();
        }
        for (int s = 0; s < nsub; s++, k += dir, left--) {
            const int h = g.halo * (nsub - 1 - s);
            const float amp = ROLE == kTileForwardRole && k + 1 < t.nt ? t.wavelet[k + 1] : 0.0f;
            if (ROLE == kTileForwardRole && k >= t.itlag) {
                if (rr >= 0) sample(k - t.itlag, rr, roff);
                for (int i = rb + tid + nthr; i < re; i += nthr) sample(k - t.itlag, t.rec_ent[i].y, place(t.rec_ent[i]));
            }
            if (ROLE == kTileRtmRole) {
                fetch_p(k - 1, pn);
                if (own.mine)
#pragma unroll
                    for (int j = 0; j < R; j++) {
                        const float4 p = pc[j], q = I[j * nthr], v = G[j * nthr];
                        const float2 i0 = pfma2(lo2(p), lo2(p), lo2(q)), i1 = pfma2(hi2(p), hi2(p), hi2(q));
                        const float2 g0 = pfma2(lo2(cur[j]), lo2(p), lo2(v)), g1 = pfma2(hi2(cur[j]), hi2(p), hi2(v));
                        I[j * nthr] = make_float4(i0.x, i0.y, i1.x, i1.y);
                        G[j * nthr] = make_float4(g0.x, g0.y, g1.x, g1.y);
                    }
            }
            const float4* const col = A + own.at;
            // psi of the strip cells, four cells past the region
            if (own.need <= h + 4 && (xin | zin)) {
                if (xin)
#pragma unroll
                    for (int j = 0; j < R; j++) {
                        if (!(own.valid >> j & 1u)) continue;
                        float2 px[2];
                        d1_quad(col[j * pitch - 1], cur[j], col[j * pitch + 1], a.inv_dx, px);
                        const float4 ps = PX[own.at + j * pitch], aa = AX[j * nthr], bb = BX[j * nthr];
                        const float2 n0 = cpml_recursion(lo2(aa), lo2(bb), lo2(ps), px[0]);
                        const float2 n1 = cpml_recursion(hi2(aa), hi2(bb), hi2(ps), px[1]);
                        PX[own.at + j * pitch] = make_float4(n0.x, n0.y, n1.x, n1.y);
                    }
                if (zin) {
                    float4 w[R + 8];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        w[j] = col[(j - 4) * pitch];
                        w[R + 4 + j] = col[(R + j) * pitch];
                    }
#pragma unroll
                    for (int j = 0; j < R; j++) w[j + 4] = cur[j];
#pragma unroll
                    for (int j = 0; j < R; j++) {
                        if (!(zin >> j & 1u)) continue;
                        const float4 ps = PZ[own.at + j * pitch], aa = AZ[j * nthr], bb = BZ[j * nthr];
                        const float2 p0 = d1_pair_ref(lo2(w[j + 5]), lo2(w[j + 3]), lo2(w[j + 6]), lo2(w[j + 2]),
                                                      lo2(w[j + 7]), lo2(w[j + 1]), lo2(w[j + 8]), lo2(w[j]), a.inv_dz);
                        const float2 p1 = d1_pair_ref(hi2(w[j + 5]), hi2(w[j + 3]), hi2(w[j + 6]), hi2(w[j + 2]),
                                                      hi2(w[j + 7]), hi2(w[j + 1]), hi2(w[j + 8]), hi2(w[j]), a.inv_dz);
                        const float2 n0 = cpml_recursion(lo2(aa), lo2(bb), lo2(ps), p0);
                        const float2 n1 = cpml_recursion(hi2(aa), hi2(bb), hi2(ps), p1);
                        PZ[own.at + j * pitch] = make_float4(n0.x, n0.y, n1.x, n1.y);
                    }
                }
            }
            __syncthreads();
            if (own.need <= h) {
                float4 out[R];
                // the strip terms of a row: zeta, and (d psi, d psi + zeta) added to the derivatives
                tile_step<APPROX, R>(
                    a, own, pitch, A, nullptr, true, cur, old, model, out,
                    [&](int j, const float4 (&w)[R + 8], float2 (&pxx)[2], float2 (&pzz)[2], float2 (&px)[2], float2 (&pz)[2]) {
                        if (APPROX == kAcoustic && (inner >> j & 1u)) {
                            float2 s[2];
                            d2_quad_sum(col[j * pitch - 1], cur[j], col[j * pitch + 1], s);
#pragma unroll
                            for (int m = 0; m < 2; m++) {
                                pxx[m] = pfma2(s[m], bc2(a.inv_dx2), pzz[m]);
                                pzz[m] = make_float2(0.f, 0.f);
                            }
                            return;
                        }
                        if (!(xin | zin)) return;
                        float2 hx[2], hz[2];
                        hx[0] = hx[1] = hz[0] = hz[1] = make_float2(0.f, 0.f);
                        if (xin && (own.valid >> j & 1u)) {
                            float2 d[2];
                            d1_quad(PX[own.at + j * pitch - 1], PX[own.at + j * pitch], PX[own.at + j * pitch + 1], a.inv_dx, d);
                            const float4 zo = ZX[j * nthr], aa = AX[j * nthr], bb = BX[j * nthr];
                            const float2 z0 = cpml_recursion(lo2(aa), lo2(bb), lo2(zo), add_apart(pxx[0], d[0]));
                            const float2 z1 = cpml_recursion(hi2(aa), hi2(bb), hi2(zo), add_apart(pxx[1], d[1]));
                            ZX[j * nthr] = make_float4(z0.x, z0.y, z1.x, z1.y);
                            // (psi's derivative reaches past the strip, its term does not)
                            if (!(xin & 1u)) d[0].x = 0.f;
                            if (!(xin & 2u)) d[0].y = 0.f;
                            if (!(xin & 4u)) d[1].x = 0.f;
                            if (!(xin & 8u)) d[1].y = 0.f;
                            hx[0] = add_apart(d[0], z0);
                            hx[1] = add_apart(d[1], z1);
                            if (APPROX != kAcoustic) {
                                px[0] = add_apart(px[0], d[0]);
                                px[1] = add_apart(px[1], d[1]);
                            }
                        }
                        if (zin >> j & 1u) {
                            float4 q[8];
#pragma unroll
                            for (int i = 0; i < 4; i++) {
                                q[i] = PZ[own.at + (j - 4 + i) * pitch];
                                q[4 + i] = PZ[own.at + (j + 1 + i) * pitch];
                            }
                            const float2 d0 = d1_pair_ref(lo2(q[4]), lo2(q[3]), lo2(q[5]), lo2(q[2]), lo2(q[6]), lo2(q[1]),
                                                          lo2(q[7]), lo2(q[0]), a.inv_dz);
                            const float2 d1 = d1_pair_ref(hi2(q[4]), hi2(q[3]), hi2(q[5]), hi2(q[2]), hi2(q[6]), hi2(q[1]),
                                                          hi2(q[7]), hi2(q[0]), a.inv_dz);
                            const float2 s0 = d2_pair_sum(lo2(w[j + 4]), lo2(w[j + 5]), lo2(w[j + 3]), lo2(w[j + 6]),
                                                          lo2(w[j + 2]), lo2(w[j + 7]), lo2(w[j + 1]), lo2(w[j + 8]), lo2(w[j]));
                            const float2 s1 = d2_pair_sum(hi2(w[j + 4]), hi2(w[j + 5]), hi2(w[j + 3]), hi2(w[j + 6]),
                                                          hi2(w[j + 2]), hi2(w[j + 7]), hi2(w[j + 1]), hi2(w[j + 8]), hi2(w[j]));
                            const float4 zo = ZZ[j * nthr], aa = AZ[j * nthr], bb = BZ[j * nthr];
                            const float2 z0 = cpml_recursion(lo2(aa), lo2(bb), lo2(zo), pfma2(s0, bc2(a.inv_dz2), d0));
                            const float2 z1 = cpml_recursion(hi2(aa), hi2(bb), hi2(zo), pfma2(s1, bc2(a.inv_dz2), d1));
                            ZZ[j * nthr] = make_float4(z0.x, z0.y, z1.x, z1.y);
                            hz[0] = add_apart(d0, z0);
                            hz[1] = add_apart(d1, z1);
                            if (APPROX != kAcoustic) {
                                pz[0] = add_apart(pz[0], d0);
                                pz[1] = add_apart(pz[1], d1);
                            }
                        }
#pragma unroll
                        for (int m = 0; m < 2; m++) {
                            if (APPROX == kAcoustic) {
                                pxx[m] = add_apart(pxx[m], pzz[m]);
                                pzz[m] = add_apart(hx[m], hz[m]);
                            } else {
                                pxx[m] = add_apart(pxx[m], hx[m]);
                                pzz[m] = add_apart(pzz[m], hz[m]);
                            }
                        }
                    });
                if (has_src)
#pragma unroll
                    for (int j = 0; j < R; j++)
                        if (j == srow) {
                            out[j].x += sx == own.x ? amp : 0.f;
                            out[j].y += sx == own.x + 1 ? amp : 0.f;
                            out[j].z += sx == own.x + 2 ? amp : 0.f;
                            out[j].w += sx == own.x + 3 ? amp : 0.f;
                        }
#pragma unroll
                for (int j = 0; j < R; j++) {
                    old[j] = cur[j];
                    cur[j] = out[j];
                    B[own.at + j * pitch] = out[j];
                }
                if (ROLE == kTileRtmRole && ie > ib) {
                    const float* const d = idat + (parity * g.T + s) * nent;
                    for (int i = ib; i < ie; i++) {
                        float* const p = reinterpret_cast<float*>(B) + __float_as_int(ient[i].x);
                        *p = __fadd_rn(*p, __fmul_rn(d[i], ta.scale));
                    }
#pragma unroll
                    for (int j = 0; j < R; j++) cur[j] = B[own.at + j * pitch];
                }
            }
            float4* const sw = A;
            A = B;
            B = sw;
            if (ROLE == kTileRtmRole)
#pragma unroll
                for (int j = 0; j < R; j++) pc[j] = pn[j];
            if (ROLE == kTileForwardRole && t.slots && own.mine) {
                float* const u = t.slots + (k + 1 - t.kslot) * t.slot_stride;
#pragma unroll
                for (int j = 0; j < R; j++)
                    if (own.mine >> j & 1u)
                        *reinterpret_cast<float4*>(PAM_CHK(u + o + j * a.P, u, fbytes, 16, 123)) = cur[j];
            }
            if (s + 1 < nsub) __syncthreads();
        }
        parity ^= 1;
        // publish the tile: fields (unless the slots hold them) and memory variables
        const bool slots = ROLE == kTileForwardRole && t.slots;
        float* const pub0 = slots ? t.slots + (k - t.kslot) * t.slot_stride : set ? t.ex[0][0] : t.ex[1][0];
        float* const pub1 = slots ? pub0 - t.slot_stride : set ? t.ex[0][1] : t.ex[1][1];
        float* const pubm = set ? tc.mem[0] : tc.mem[1];
#pragma unroll
        for (int j = 0; j < R; j++)
            if (own.mine >> j & 1u) {
                const long long c = o + j * a.P;
                auto put = [&](float* base, float4 v) {
                    *reinterpret_cast<float4*>(PAM_CHK(base + c, base, fbytes, 16, 124)) = v;
                };
                if (!slots) {
                    put(pub0, cur[j]);
                    put(pub1, old[j]);
                }
                if (xin) {
                    put(pubm, PX[own.at + j * pitch]);
                    put(pubm + mstride, ZX[j * nthr]);
                }
                if (zin >> j & 1u) {
                    put(pubm + 2 * mstride, PZ[own.at + j * pitch]);
                    put(pubm + 3 * mstride, ZZ[j * nthr]);
                }
            }
        set ^= 1;
        if (left <= 0) break;
        if (ROLE == kTileRtmRole) cp_async_wait<0>();
        want += gridDim.x;
        if (!tile_barrier(t, want, &alive)) {
            if (ROLE == kTileForwardRole) tile_poison(t, seis, rb, re, k);
            return;
        }
        const unsigned halo = own.valid & ~own.mine;
        if (halo) {
            float4 px[R], pz[R];
#pragma unroll
            for (int j = 0; j < R; j++)
                if (halo >> j & 1u) {
                    const float* const m = pubm + o + j * a.P;
                    cur[j] = tile_halo(pub0 + o + j * a.P, pub0, fbytes);
                    old[j] = tile_halo(pub1 + o + j * a.P, pub1, fbytes);
                    if (xin) {
                        px[j] = tile_halo(m, pubm, fbytes);
                        ZX[j * nthr] = tile_halo(m + mstride, pubm + mstride, fbytes);
                    }
                    if (zin >> j & 1u) {
                        pz[j] = tile_halo(m + 2 * mstride, pubm + 2 * mstride, fbytes);
                        ZZ[j * nthr] = tile_halo(m + 3 * mstride, pubm + 3 * mstride, fbytes);
                    }
                }
#pragma unroll
            for (int j = 0; j < R; j++)
                if (halo >> j & 1u) {
                    A[own.at + j * pitch] = cur[j];
                    if (xin) PX[own.at + j * pitch] = px[j];
                    if (zin >> j & 1u) PZ[own.at + j * pitch] = pz[j];
                }
        }
        __syncthreads();
    }
    if (ROLE == kTileRtmRole)
#pragma unroll
        for (int j = 0; j < R; j++)
            if (own.mine >> j & 1u) {
                *reinterpret_cast<float4*>(PAM_CHK(ta.gsum + o + (long long)j * a.P, ta.gsum, fbytes, 16, 125)) = G[j * nthr];
                *reinterpret_cast<float4*>(PAM_CHK(ta.isum + o + (long long)j * a.P, ta.isum, fbytes, 16, 125)) = I[j * nthr];
            }
}

}  // namespace pam
