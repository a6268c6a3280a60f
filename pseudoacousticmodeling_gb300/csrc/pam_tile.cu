// Host side of the persistent tiles (pam_tile.cuh): which runs take them, how
// a grid is cut, and the launches.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <vector>

#include "../../include/pam.h"
#include "pam_engine.h"
#include "pam_tile.cuh"

using namespace pam;

#define CU(call)                                                                                 \
    do {                                                                                         \
        cudaError_t _e = (call);                                                                 \
        if (_e != cudaSuccess)                                                                   \
            return e->fail(PAM_E_CUDA, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(_e),    \
                           __FILE__, __LINE__);                                                  \
    } while (0)

namespace {

constexpr int kMaxDevices = 64;
// dynamic shared memory of a block: 227 KB less the kernel's own few bytes
constexpr int kTileSmemMax = 226 * 1024;

// cost in microseconds of a barrier with the exchange of the halo (a part of it
// for each row that a thread publishes and reloads), of a step's own overhead,
// and of a cell update on one SM by approximation: fitted to runs of 0.04 to
// 0.5 million cells with T = 1 .. 8 and R = 2 .. 4, which they meet within 10%
constexpr double kTileBarrierUs = 1.62, kTileRowUs = 0.265, kTileStepUs = 0.05;
constexpr double kTileCellUs[3] = {3.2e-4, 5.5e-4, 9.0e-4};
// the same of a graph of one-step launches, by approximation: the latency of a
// step, and a cell of the batch (0.15 to 2.2 million cells: 5.7 to 9.2 us
// acoustic, 6.9 to 10.3 us VTI, 7.6 to 10.2 us TTI)
constexpr double kGraphStepUs[3] = {5.5, 6.6, 7.2}, kGraphCellUs[3] = {1.6e-6, 2.1e-6, 3.5e-6};

int models_of(int approx) {
    return approx == PAM_ACOUSTIC ? tile_models<kAcoustic>() : approx == PAM_VTI ? tile_models<kVTI>() : tile_models<kTTI>();
}

TileShape shape_of(const pam_engine::TilePlan& p) {
    TileShape g;
    g.T = p.T;
    g.TZ = p.TZ;
    g.TX = p.TX;
    g.nty = p.nty;
    g.ntx = p.ntx;
    g.R = p.R;
    g.nrg = (p.TZ + 8 * p.T + p.R - 1) / p.R;
    g.EXq = p.TX / 4 + 2 * p.T;
    return g;
}

template <int A, int R>
cudaError_t launch_forward(const TileArgs& t, int blocks, size_t smem, cudaStream_t s) {
    // the shared-memory opt-in is a per-device attribute of the kernel
    static bool configured[kMaxDevices] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= kMaxDevices || !configured[dev]) {
        cudaError_t err = cudaFuncSetAttribute(tile_forward_kernel<A, R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               kTileSmemMax);
        if (err != cudaSuccess) return err;
        if (dev >= 0 && dev < kMaxDevices) configured[dev] = true;
    }
    TileArgs q = t;
    void* args[] = {&q};
    return cudaLaunchCooperativeKernel((const void*)tile_forward_kernel<A, R>, dim3(blocks), dim3(tile_threads(t.g)), args,
                                       smem, s);
}

template <int A>
cudaError_t launch_forward(const TileArgs& t, int blocks, size_t smem, cudaStream_t s) {
    return t.g.R == 2   ? launch_forward<A, 2>(t, blocks, smem, s)
           : t.g.R == 3 ? launch_forward<A, 3>(t, blocks, smem, s)
                        : launch_forward<A, 4>(t, blocks, smem, s);
}

}  // namespace

// How to run this batch as persistent tiles, or nullptr for the one-step
// launches.  Every cut of the grid into at most one tile per SM and every
// number T of steps between barriers that fits in shared memory is weighed by
// its cost per step: a barrier with the exchange of the halo every T steps,
// and the cells of each step's region at the rate one SM updates them; a batch
// may go in several launches of some shots each.  The tiles are taken where
// the best of these is below the cost of the one-step launches.
const pam_engine::TilePlan* pam_engine::tile_plan(int nshots) {
    if (cfg.boundary != PAM_CERJAN || prof_stride > 0 || std::getenv("PAM_NO_PERSISTENT")) return nullptr;
    auto it = tile_plans.find(nshots);
    if (it == tile_plans.end()) {
        TilePlan best;
        int sms = 0, coop = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) sms = 0;
        if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess) coop = 0;
        cudaGetLastError();
        const int rows = nza - 8, cols = nxa - 8;
        // (a receiver's place is held in 16 bits each way)
        const bool fits = nza < 32768 && nxa < 65536;
        const int approx = cfg.approximation;
        double best_cost = kGraphStepUs[approx] + kGraphCellUs[approx] * nshots * (double)nza * nxa;
        for (int group = nshots; fits && coop && group >= 1; group = group > 1 ? (group + 1) / 2 : 0) {
            const int launches = (nshots + group - 1) / group;
            for (int ntx0 = 1; ntx0 * group <= sms && ntx0 <= (cols + 3) / 4; ntx0++) {
                const int TX = ((cols + ntx0 - 1) / ntx0 + 3) / 4 * 4, ntx = (cols + TX - 1) / TX;
                const int nty0 = std::min(sms / (ntx * group), rows);
                if (nty0 < 1) break;
                const int TZ = (rows + nty0 - 1) / nty0, nty = (rows + TZ - 1) / TZ;
                for (int R = 2; R <= 4; R++)
                    for (int T = 1; T <= kTileMaxT; T++) {
                        TilePlan p;
                        p.usable = true;
                        p.T = T;
                        p.TZ = TZ;
                        p.TX = TX;
                        p.nty = nty;
                        p.ntx = ntx;
                        p.R = R;
                        p.group = group;
                        const TileShape g = shape_of(p);
                        if (tile_threads(g) > kTileThreads || g.EXq >= kTilePitch ||
                            tile_smem_bytes(g, models_of(approx)) > (size_t)kTileSmemMax)
                            break;
                        double cost = kTileBarrierUs + kTileRowUs * R;
                        for (int s = 0; s < T; s++) {
                            const double cells =
                                (double)std::min(TZ + 8 * s, rows) * std::min(TX + 8 * s, (cols + 3) / 4 * 4);
                            cost += kTileStepUs + cells * kTileCellUs[approx];
                        }
                        cost *= (double)launches / T;
                        if (cost < best_cost) {
                            best_cost = cost;
                            best = p;
                        }
                    }
            }
        }
        it = tile_plans.emplace(nshots, best).first;
    }
    return it->second.usable ? &it->second : nullptr;
}

// The buffers of the persistent tiles, and each tile's list of the receivers
// in it (receivers off the update region, whose samples are zero, go to the
// nearest tile, which holds those cells in its halo).
int pam_engine::tile_begin(const TilePlan& p, cudaStream_t s) {
    pam_engine* e = this;
    const size_t field = (size_t)shot_stride * B;
    for (float*& d : d_tile)
        if (!d) {
            if (dalloc_bytes((void**)&d, field * 4)) return PAM_E_CUDA;
            CU(cudaMemsetAsync(d, 0, field * 4, s));
        }
    if (!d_tile_bar && dalloc_bytes((void**)&d_tile_bar, 128)) return PAM_E_CUDA;
    tile_set = 0;
    if (!tile_lists_stale && tile_lists_TZ == p.TZ && tile_lists_TX == p.TX) return PAM_OK;
    const int nt = p.nty * p.ntx, lists = rec_per_shot ? B : 1;
    std::vector<int> beg((size_t)nt * lists + 1, 0);
    std::vector<int> where((size_t)lists * nrec);
    for (int l = 0; l < lists; l++)
        for (int r = 0; r < nrec; r++) {
            const size_t i = (size_t)l * nrec + r;
            const int ty = std::min(std::max(h_rz[i] - 4, 0) / p.TZ, p.nty - 1);
            const int tx = std::min(std::max(h_rx[i] - 4, 0) / p.TX, p.ntx - 1);
            where[i] = l * nt + ty * p.ntx + tx;
            beg[where[i] + 1]++;
        }
    for (size_t i = 0; i + 1 < beg.size(); i++) beg[i + 1] += beg[i];
    std::vector<int> at(beg.begin(), beg.end() - 1);
    std::vector<int2> ent(where.size());
    for (size_t i = 0; i < where.size(); i++) ent[at[where[i]]++] = make_int2(h_rz[i] << 16 | h_rx[i], (int)(i % nrec));
    dfree(d_tile_beg);
    dfree(d_tile_ent);
    d_tile_beg = nullptr;
    d_tile_ent = nullptr;
    if (dalloc_bytes((void**)&d_tile_beg, beg.size() * sizeof(int)) ||
        dalloc_bytes((void**)&d_tile_ent, ent.size() * sizeof(int2)))
        return PAM_E_CUDA;
    CU(cudaMemcpyAsync(d_tile_beg, beg.data(), beg.size() * sizeof(int), cudaMemcpyHostToDevice, s));
    CU(cudaMemcpyAsync(d_tile_ent, ent.data(), ent.size() * sizeof(int2), cudaMemcpyHostToDevice, s));
    CU(cudaStreamSynchronize(s));   // the vectors go out of scope
    tile_lists_stale = false;
    tile_lists_TZ = p.TZ;
    tile_lists_TX = p.TX;
    return PAM_OK;
}

int pam_engine::tile_forward(const TilePlan& p, int nshots, float* d_seis, int k0, int k1, cudaStream_t s) {
    if (k1 <= k0) return PAM_OK;
    TileArgs t;
    t.s = step_args(0, nshots, nullptr, nullptr, 0);
    t.g = shape_of(p);
    t.ex[0][0] = d_u[0];
    t.ex[0][1] = d_u[1];
    t.ex[1][0] = d_tile[0];
    t.ex[1][1] = d_tile[1];
    t.set0 = tile_set;
    t.wavelet = d_wavelet;
    t.rec = RecordArgs{};
    t.rec.seis = d_seis;
    t.rec.nrec = nrec;
    t.rec.nt_data = nt_data;
    t.rec.per_shot = rec_per_shot;
    t.rec_beg = d_tile_beg;
    t.rec_ent = d_tile_ent;
    t.nt = cfg.nt;
    t.itlag = cfg.itlag;
    t.k0 = k0;
    t.k1 = k1;
    t.bar = d_tile_bar;
    t.status = d_status;
    const size_t smem = tile_smem_bytes(t.g, models_of(cfg.approximation));
    for (int b = 0; b < nshots; b += p.group) {
        t.shot0 = b;
        const int blocks = std::min(p.group, nshots - b) * p.nty * p.ntx;
        cudaError_t err = cudaMemsetAsync(d_tile_bar, 0, sizeof(unsigned), s);
        if (err == cudaSuccess)
            err = cfg.approximation == PAM_ACOUSTIC ? launch_forward<kAcoustic>(t, blocks, smem, s)
                : cfg.approximation == PAM_VTI      ? launch_forward<kVTI>(t, blocks, smem, s)
                                                    : launch_forward<kTTI>(t, blocks, smem, s);
        if (err != cudaSuccess) return fail(PAM_E_CUDA, "cooperative launch failed: %s", cudaGetErrorString(err));
    }
    // every group of T steps publishes into the other set
    tile_set ^= ((k1 - k0 + p.T - 1) / p.T) & 1;
    return PAM_OK;
}
