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
// ... more for a step with CPML strips
constexpr double kTileStripUs = 1.2, kTileStripCellUs[2] = {1.1e-3, 1.9e-3};
// ... and of the sums over time of a tile's cell (backward sweeps, by job)
constexpr double kTileSumUs[3] = {0.0, 4.0e-4, 1.5e-4};
// the same of a graph of one-step launches, by approximation: the latency of a
// step, and a cell of the batch (0.15 to 2.2 million cells: 5.7 to 9.2 us
// acoustic, 6.9 to 10.3 us VTI, 7.6 to 10.2 us TTI)
constexpr double kGraphStepUs[3] = {5.5, 6.6, 7.2}, kGraphCellUs[3] = {1.6e-6, 2.1e-6, 3.5e-6};

// ... and of a step of the graph where the callers of three engines keep the GPU
// busy together, which an asynchronous run (device output) allows and a
// cooperative launch, taking every SM, does not.  Every such run is weighed with
// these figures, since the engine cannot know who else uses the GPU: one engine
// that waits after each batch would do better as tiles (eight acoustic shots of
// 301 x 501: 5.3 against 7.4 us a step by the figures above), as before there
// were tiles.  (Three engines in turn, measured:
// CPML of 0.18 / 0.36 / 0.53 million cells 3.7 / 4.1 / 4.6 us acoustic, 4.1 / 4.9 /
// 5.6 us VTI, against 4.6 / 9.3 us and 5.3 us as tiles; Cerjan of 1.06 million
// cells 3.0 us acoustic, 4.2 us VTI against 4.4 and 7.0.)  Cerjan batches up to
// kPersistCells are one cooperative launch either way.
constexpr double kSharedStepUs[3] = {1.8, 2.1, 2.4}, kSharedCellUs[3] = {1.15e-6, 2.0e-6, 2.8e-6};
constexpr double kCpmlSharedStepUs[2] = {3.3, 3.6}, kCpmlSharedCellUs[2] = {2.3e-6, 3.3e-6};

constexpr double kCpmlGraphStepUs = 9.6, kCpmlGraphCellUs[2] = {1.9e-6, 3.5e-6};
// ... and of the one-barrier-per-step persistent loop (0.3 to 0.9 million cells:
// 3.6 to 4.9 us acoustic, 4.6 to 5.9 us VTI, 5.4 to 8.5 us TTI)
constexpr double kPersistStepUs[3] = {3.1, 4.1, 4.2}, kPersistCellUs[3] = {1.9e-6, 2.1e-6, 4.0e-6};
// ... and what a step costs more as separate launches than as a graph (the
// forward sweeps of migration and gradient jobs)
constexpr double kLaunchUs = 1.0, kCpmlLaunchUs = 4.0;
// ... and of a backward step as launches of its own
constexpr double kBackStepUs = 10.0, kBackCellUs = 4.5e-6;

int models_of(int approx) {
    return approx == PAM_ACOUSTIC ? tile_models<kAcoustic>() : approx == PAM_VTI ? tile_models<kVTI>() : tile_models<kTTI>();
}

TileShape shape_of(const pam_engine::TilePlan& p) {
    TileShape g;
    g.halo = p.halo;
    g.T = p.T;
    g.TZ = p.TZ;
    g.TX = p.TX;
    g.nty = p.nty;
    g.ntx = p.ntx;
    g.R = p.R;
    g.nrg = (p.TZ + 2 * p.halo * p.T + p.R - 1) / p.R;
    g.EXq = p.TX / 4 + p.halo / 2 * p.T;
    return g;
}

size_t smem_of(const TileShape& g, int approx, int job) {
    const bool forward = job != pam_engine::kTileExactJob && job != pam_engine::kTileRtmJob;
    if (g.halo == 8) return tile_cpml_smem_bytes(g, models_of(approx), forward ? kTileForwardRole : kTileRtmRole);
    return forward ? tile_smem_bytes(g, models_of(approx)) : tile_adj_smem_bytes(g);
}

int threads_of(const TileShape& g) { return g.halo == 8 ? kTileCpmlThreads : kTileThreads; }

// A cooperative launch; the shared-memory opt-in is a per-device attribute of
// the kernel.
template <class Args>
cudaError_t launch(void (*kernel)(const Args), bool* configured, const Args& args, int blocks, int threads, size_t smem,
                   cudaStream_t s) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= kMaxDevices || !configured[dev]) {
        cudaError_t err = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmemMax);
        if (err != cudaSuccess) return err;
        if (dev >= 0 && dev < kMaxDevices) configured[dev] = true;
    }
    Args q = args;
    void* list[] = {&q};
    return cudaLaunchCooperativeKernel((const void*)kernel, dim3(blocks), dim3(threads), list, smem, s);
}

template <int A, int R, bool REVERSE>
cudaError_t launch_forward(const TileArgs& t, int blocks, size_t smem, cudaStream_t s) {
    static bool configured[kMaxDevices] = {};
    return launch<TileArgs>(tile_forward_kernel<A, R, REVERSE>, configured, t, blocks, tile_threads(t.g), smem, s);
}

template <int A, bool REVERSE>
cudaError_t launch_forward(const TileArgs& t, int blocks, size_t smem, cudaStream_t s) {
    return t.g.R == 2   ? launch_forward<A, 2, REVERSE>(t, blocks, smem, s)
           : t.g.R == 3 ? launch_forward<A, 3, REVERSE>(t, blocks, smem, s)
                        : launch_forward<A, 4, REVERSE>(t, blocks, smem, s);
}

template <bool REVERSE>
cudaError_t launch_forward(int approx, const TileArgs& t, int blocks, size_t smem, cudaStream_t s) {
    return approx == PAM_ACOUSTIC ? launch_forward<kAcoustic, REVERSE>(t, blocks, smem, s)
           : approx == PAM_VTI    ? launch_forward<kVTI, REVERSE>(t, blocks, smem, s)
                                  : launch_forward<kTTI, REVERSE>(t, blocks, smem, s);
}

template <int A, int ROLE>
cudaError_t launch_cpml(const TileCpmlArgs& t, int blocks, size_t smem, cudaStream_t s) {
    static bool configured[kMaxDevices] = {};
    return launch<TileCpmlArgs>(tile_cpml_kernel<A, ROLE>, configured, t, blocks, tile_threads(t.r.f.g), smem, s);
}

template <int MODE, int R>
cudaError_t launch_adjoint(const TileAdjArgs& t, int blocks, size_t smem, cudaStream_t s) {
    static bool configured[kMaxDevices] = {};
    return launch<TileAdjArgs>(tile_adjoint_kernel<MODE, R>, configured, t, blocks, tile_threads(t.f.g), smem, s);
}

template <int MODE>
cudaError_t launch_adjoint(const TileAdjArgs& t, int blocks, size_t smem, cudaStream_t s) {
    return t.f.g.R == 2   ? launch_adjoint<MODE, 2>(t, blocks, smem, s)
           : t.f.g.R == 3 ? launch_adjoint<MODE, 3>(t, blocks, smem, s)
                          : launch_adjoint<MODE, 4>(t, blocks, smem, s);
}

__global__ void tile_fold_image_kernel(const float* __restrict__ gsum, const float* __restrict__ isum, long long stride,
                                       int B, int P, int N, int nzi, int nxi, float* __restrict__ img,
                                       float* __restrict__ ilum)
{
    const int xi = blockIdx.x * blockDim.x + threadIdx.x, zi = blockIdx.y;
    if (xi >= nxi || zi >= nzi) return;
    const long long c = (long long)(zi + N) * P + xi + N;
    float g = 0.0f, i = 0.0f;
    for (int b = 0; b < B; b++) {
        g += gsum[(long long)b * stride + c];
        i += isum[(long long)b * stride + c];
    }
    img[(long long)zi * nxi + xi] += g;
    ilum[(long long)zi * nxi + xi] += i;
}

}  // namespace

// How to run this batch as persistent tiles, or nullptr for the one-step
// launches.  Every cut of the grid into at most one tile per SM and every
// number T of steps between barriers that fits in shared memory is weighed by
// its cost per step: a barrier with the exchange of the halo every T steps,
// and the cells of each step's region at the rate one SM updates them; a batch
// may go in several launches of some shots each.  The tiles are taken where
// the best of these is below the cost of the one-step launches.
pam_engine::TilePlan* pam_engine::tile_plan(int nshots, TileJob job) {
    const int approx = cfg.approximation;
    const bool cpml = cfg.boundary == PAM_CPML && job != kTileReverse;
    if (prof_stride > 0 || std::getenv("PAM_NO_PERSISTENT")) return nullptr;
    // with the matched layer: the forward loop of the acoustic and VTI operators, acoustic migration
    if (cpml && (approx == PAM_TTI || job == kTileExactJob)) return nullptr;
    std::map<int, TilePlan>& plans = tile_plans[job];
    auto it = plans.find(nshots);
    if (it == plans.end()) {
        TilePlan best;
        int sms = 0, coop = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) sms = 0;
        if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess) coop = 0;
        cudaGetLastError();
        const int rows = nza - 8, cols = nxa - 8;
        // (a receiver's place is held in 16 bits each way)
        const bool fits = nza < 32768 && nxa < 65536;
        const bool forward = job != kTileExactJob && job != kTileRtmJob;
        const double cells_all = nshots * (double)nza * nxa;
        double best_cost = forward ? kGraphStepUs[approx] + kGraphCellUs[approx] * cells_all
                                   : kBackStepUs + kBackCellUs * cells_all;
        if ((job == kTileForward || job == kTileForwardAsync) && !cpml && cells_all <= kPersistCells)
            best_cost = std::min(best_cost, kPersistStepUs[approx] + kPersistCellUs[approx] * cells_all);
        if (cpml) best_cost = kCpmlGraphStepUs + kCpmlGraphCellUs[approx] * cells_all + (forward ? 0.0 : kBackStepUs);
        if (job == kTileForwardAsync && (cpml || cells_all > kPersistCells))
            best_cost = cpml ? kCpmlSharedStepUs[approx] + kCpmlSharedCellUs[approx] * cells_all
                             : kSharedStepUs[approx] + kSharedCellUs[approx] * cells_all;
        if (job == kTileForwardLaunched) best_cost += cpml ? kCpmlLaunchUs : kLaunchUs;
        const int halo = cpml ? 8 : 4;
        for (int group = nshots; fits && coop && group >= 1; group = group > 1 ? (group + 1) / 2 : 0) {
            const int launches = (nshots + group - 1) / group;
            for (int ntx0 = 1; ntx0 * group <= sms && ntx0 <= (cols + 3) / 4; ntx0++) {
                const int TX = ((cols + ntx0 - 1) / ntx0 + 3) / 4 * 4, ntx = (cols + TX - 1) / TX;
                const int nty0 = std::min(sms / (ntx * group), rows);
                if (nty0 < 1) break;
                const int TZ = (rows + nty0 - 1) / nty0, nty = (rows + TZ - 1) / TZ;
                for (int R = cpml ? kTileCpmlRows : 2; R <= (cpml ? kTileCpmlRows : 4); R++)
                    for (int T = 1; T <= kTileMaxT; T++) {
                        TilePlan p;
                        p.usable = true;
                        p.T = T;
                        p.TZ = TZ;
                        p.TX = TX;
                        p.nty = nty;
                        p.ntx = ntx;
                        p.R = R;
                        p.halo = halo;
                        p.group = group;
                        const TileShape g = shape_of(p);
                        if (tile_threads(g) > threads_of(g) || g.EXq >= kTilePitch ||
                            smem_of(g, approx, job) > (size_t)kTileSmemMax)
                            break;
                        double cost = kTileBarrierUs + kTileRowUs * R;
                        for (int s = 0; s < T; s++) {
                            const double cells = (double)std::min(TZ + 2 * halo * s, rows) *
                                                 std::min(TX + 2 * halo * s, (cols + 3) / 4 * 4);
                            cost += kTileStepUs + cells * kTileCellUs[approx];
                            if (cpml) cost += kTileStripUs + cells * kTileStripCellUs[approx];
                            if (!forward) cost += (double)TZ * TX * kTileSumUs[job];
                        }
                        cost *= (double)launches / T;
                        if (cost < best_cost) {
                            best_cost = cost;
                            best = p;
                        }
                    }
            }
        }
        it = plans.emplace(nshots, best).first;
    }
    return it->second.usable ? &it->second : nullptr;
}

// One array of the workspace: `fields` fields of every shot of it.
bool pam_engine::tile_alloc(float** d, size_t fields, bool zero, cudaStream_t s) {
    if (*d) return true;
    const size_t bytes = fields * (size_t)tile_field() * 4;
    const bool allowed = bytes <= tile_limit && tile_bytes <= tile_limit - bytes;
    if (!allowed || cudaMalloc((void**)d, bytes) != cudaSuccess) {
        if (allowed) cudaGetLastError();
        *d = nullptr;
        tile_tight = true;   // until tile_reserve makes room
        return false;
    }
    allocs.push_back(*d);
    tile_bytes += bytes;
    if (zero) cudaMemsetAsync(*d, 0, bytes, s);   // (its error is the caller's next one)
    return true;
}

void pam_engine::tile_free(float** d, size_t fields) {
    if (!*d) return;
    dfree(*d);
    *d = nullptr;
    tile_bytes -= fields * (size_t)tile_field() * 4;
}

bool pam_engine::tile_release() {
    if (!tile_bytes) return false;
    for (float** d : {d_tile, d_tile_b, d_tile_sum})
        for (int i = 0; i < 2; i++) tile_free(d + i, 1);
    for (float** d : {d_tile_mem, d_tile_bmem})
        for (int i = 0; i < 2; i++) tile_free(d + i, 4);
    tile_free(&d_tile_slots, tile_slot_count());
    tile_held_shots = 0;
    return true;
}

// The workspace grows with the batch; where the larger one has not fitted, it is
// made anew for the smaller.
void pam_engine::tile_reserve(int nshots) {
    if (nshots <= tile_shots && !(nshots < tile_shots && tile_tight)) return;
    tile_release();
    tile_shots = nshots;
    tile_tight = false;
}

// The second published state.
bool pam_engine::tile_buffers(cudaStream_t s) {
    if (!d_tile_bar) {
        if (cudaMalloc((void**)&d_tile_bar, 128) != cudaSuccess) {
            cudaGetLastError();
            d_tile_bar = nullptr;
            return false;
        }
        allocs.push_back(d_tile_bar);
    }
    return tile_alloc(&d_tile[0], 1, true, s) && tile_alloc(&d_tile[1], 1, true, s);
}

// The source fields of a segment (their outer rows and columns stay zero).
bool pam_engine::tile_slots(cudaStream_t s) {
    return tile_buffers(s) && tile_alloc(&d_tile_slots, tile_slot_count(), true, s);
}

// The lists of a plan to the device, behind the work queued on s.  Buffers that
// are large enough are used again; what is waited for is the plan's last upload
// (still queued only if the receivers changed twice meanwhile), and the device
// where the buffers have to grow.
bool pam_engine::tile_upload(TileLists& l, const std::vector<int>& beg, const std::vector<int2>& ent, cudaStream_t s) {
    l.entries = (beg.size() * sizeof(int) + 15) / 16 * 16;
    const size_t need = l.entries + ent.size() * sizeof(int2);
    if (!l.uploaded && cudaEventCreateWithFlags(&l.uploaded, cudaEventDisableTiming) != cudaSuccess) return false;
    cudaEventSynchronize(l.uploaded);   // the last upload has left the pinned copy
    if (need > l.bytes) {
        l.bytes = 0;
        dfree(l.d);
        l.d = nullptr;
        if (l.h) host_allocs.erase(std::find(host_allocs.begin(), host_allocs.end(), (void*)l.h));
        cudaFreeHost(l.h);
        l.h = nullptr;
        if (cudaMalloc((void**)&l.d, need) != cudaSuccess) {
            l.d = nullptr;
            cudaGetLastError();
            return false;
        }
        allocs.push_back(l.d);
        if (cudaMallocHost((void**)&l.h, need) != cudaSuccess) {
            l.h = nullptr;
            cudaGetLastError();
            return false;
        }
        host_allocs.push_back(l.h);
        l.bytes = need;
    }
    std::copy(beg.begin(), beg.end(), (int*)l.h);
    std::copy(ent.begin(), ent.end(), (int2*)(l.h + l.entries));
    l.ready = cudaMemcpyAsync(l.d, l.h, need, cudaMemcpyHostToDevice, s) == cudaSuccess &&
              cudaEventRecord(l.uploaded, s) == cudaSuccess;
    return l.ready;
}

// The buffers of the persistent tiles, and each tile's list of the receivers
// in it (receivers off the update region, whose samples are zero, go to the
// nearest tile, which holds those cells in its halo).  False: there is no room
// for them.
bool pam_engine::tile_begin(TilePlan& p, int nshots, cudaStream_t s) {
    if (!tile_buffers(s)) return false;
    tile_set = 0;
    if (p.halo == 8) {
        if (!tile_alloc(&d_tile_mem[0], 4, false, s) || !tile_alloc(&d_tile_mem[1], 4, false, s)) return false;
        // (what is published into the other set covers all that is read from it)
        for (int i = 0; i < 4; i++)
            cudaMemsetAsync(d_tile_mem[0] + i * tile_field(), 0, (size_t)shot_stride * nshots * 4, s);
    }
    if (p.record.ready) return true;
    const int nt = p.nty * p.ntx, lists = rec_per_shot ? nshots : 1;
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
    return tile_upload(p.record, beg, ent, s);
}

TileArgs pam_engine::tile_args(const TilePlan& p, int nshots) const {
    TileArgs t{};
    t.s = step_args(0, nshots, nullptr, nullptr, 0);
    t.g = shape_of(p);
    t.wavelet = d_wavelet;
    t.rec.nrec = nrec;
    t.rec.nt_data = nt_data;
    t.rec.per_shot = rec_per_shot;
    t.nt = cfg.nt;
    t.itlag = cfg.itlag;
    t.bar = d_tile_bar;
    t.polls = tile_polls;
    t.status = d_status;
    t.mem_shots = tile_shots;
    return t;
}

int pam_engine::tile_forward(const TilePlan& p, int nshots, float* d_seis, int k0, int k1, cudaStream_t s, float* slots,
                             int kslot, long long slot_stride) {
    if (k1 <= k0) return PAM_OK;
    TileArgs t = tile_args(p, nshots);
    t.ex[0][0] = d_u[0];
    t.ex[0][1] = d_u[1];
    t.ex[1][0] = d_tile[0];
    t.ex[1][1] = d_tile[1];
    t.set0 = tile_set;
    t.rec.seis = d_seis;
    t.rec_beg = p.record.beg();
    t.rec_ent = p.record.ent();
    t.k0 = k0;
    t.k1 = k1;
    t.slots = slots;
    t.kslot = kslot;
    t.slot_stride = slot_stride;
    const size_t smem = smem_of(t.g, cfg.approximation, kTileForward);
    for (int b = 0; b < nshots; b += p.group) {
        t.shot0 = b;
        const int blocks = std::min(p.group, nshots - b) * p.nty * p.ntx;
        cudaError_t err = cudaMemsetAsync(d_tile_bar, 0, sizeof(unsigned), s);
        if (err == cudaSuccess && p.halo == 8) {
            TileCpmlArgs c{};
            c.r.f = t;
            c.mem[0] = d_tile_mem[0];
            c.mem[1] = d_tile_mem[1];
            c.cxab = d_cxab;
            c.czab = d_czab;
            err = cfg.approximation == PAM_ACOUSTIC ? ::launch_cpml<kAcoustic, kTileForwardRole>(c, blocks, smem, s)
                                                    : ::launch_cpml<kVTI, kTileForwardRole>(c, blocks, smem, s);
        } else if (err == cudaSuccess) {
            err = launch_forward<false>(cfg.approximation, t, blocks, smem, s);
        }
        if (err != cudaSuccess) return fail(PAM_E_CUDA, "cooperative launch failed: %s", cudaGetErrorString(err));
    }
    // every group of T steps publishes into the other set
    if (!slots || p.halo == 8) tile_set ^= ((k1 - k0 + p.T - 1) / p.T) & 1;
    return PAM_OK;
}

// Steps t = k1-1 .. k0 of the source field backwards in time, undamped, from
// S(k1-1), S(k1) in the slots to S(k0-1): with the random border (its kappa) or
// the saved bands written over each new field.
int pam_engine::tile_reverse(const TilePlan& p, int nshots, int k0, int k1, cudaStream_t s, float* slots, int kslot,
                             const float* kap, bool bands) {
    if (k1 <= k0) return PAM_OK;
    TileArgs t = tile_args(p, nshots);
    t.s.kap = kap;
    t.s.cerjan = nullptr;
    t.k0 = k0;
    t.k1 = k1;
    t.slots = slots;
    t.kslot = kslot;
    t.slot_stride = tile_field();
    if (bands) {
        t.band = d_band;
        t.band_shots = B;
        t.band_scale = d_band_scale;
        t.band_store = adj_store;
        t.nzi = cfg.nz;
        t.nxi = cfg.nx;
    }
    const size_t smem = smem_of(t.g, cfg.approximation, kTileReverse);
    for (int b = 0; b < nshots; b += p.group) {
        t.shot0 = b;
        const int blocks = std::min(p.group, nshots - b) * p.nty * p.ntx;
        cudaError_t err = cudaMemsetAsync(d_tile_bar, 0, sizeof(unsigned), s);
        if (err == cudaSuccess) err = launch_forward<true>(cfg.approximation, t, blocks, smem, s);
        if (err != cudaSuccess) return fail(PAM_E_CUDA, "cooperative launch failed: %s", cudaGetErrorString(err));
    }
    return PAM_OK;
}

// Steps 0 .. nt-1 of the source field with the random border, undamped, from
// d_u[0], d_u[1]; leaves U(nt - 1), U(nt) in the two field buffers.
int pam_engine::tile_undamped(const TilePlan& p, int nshots, const float* kap, cudaStream_t s) {
    pam_engine* e = this;
    TileArgs t = tile_args(p, nshots);
    t.ex[0][0] = d_u[0];
    t.ex[0][1] = d_u[1];
    t.ex[1][0] = d_tile[0];
    t.ex[1][1] = d_tile[1];
    t.s.kap = kap;
    t.s.cerjan = nullptr;
    t.k1 = cfg.nt;
    const size_t smem = smem_of(t.g, cfg.approximation, kTileReverse);
    for (int b = 0; b < nshots; b += p.group) {
        t.shot0 = b;
        const int blocks = std::min(p.group, nshots - b) * p.nty * p.ntx;
        cudaError_t err = cudaMemsetAsync(d_tile_bar, 0, sizeof(unsigned), s);
        if (err == cudaSuccess) err = launch_forward<false>(cfg.approximation, t, blocks, smem, s);
        if (err != cudaSuccess) return fail(PAM_E_CUDA, "cooperative launch failed: %s", cudaGetErrorString(err));
    }
    // from the set that holds the state: U(nt) into d_u[nt & 1], U(nt - 1) into the other
    const bool second = ((cfg.nt + p.T - 1) / p.T) & 1;
    const size_t bytes = (size_t)shot_stride * nshots * 4;
    const float* cur = second ? d_tile[0] : d_u[0];
    const float* prev = second ? d_tile[1] : d_u[1];
    if (!second && (cfg.nt & 1)) {   // in the field buffers, the wrong way round
        CU(cudaMemcpyAsync(d_tile[0], d_u[0], bytes, cudaMemcpyDeviceToDevice, s));
        cur = d_tile[0];
    }
    if (prev != d_u[(cfg.nt + 1) & 1])
        CU(cudaMemcpyAsync(d_u[(cfg.nt + 1) & 1], prev, bytes, cudaMemcpyDeviceToDevice, s));
    if (cur != d_u[cfg.nt & 1]) CU(cudaMemcpyAsync(d_u[cfg.nt & 1], cur, bytes, cudaMemcpyDeviceToDevice, s));
    return PAM_OK;
}

// ---------------------------------------------------------------- backward sweeps

// The plan of a backward sweep, with its buffers and each thread's receivers
// ready; nullptr for the one-step launches.  Receivers off the update region,
// which the one-step kernels inject into cells that no step writes, and lists
// too long for shared memory stay with those.
const pam_engine::TilePlan* pam_engine::tile_adjoint_begin(int nshots, TileJob job, cudaStream_t s) {
    if (cfg.approximation != PAM_ACOUSTIC) return nullptr;
    TilePlan* p = tile_plan(nshots, job);
    if (!p) return nullptr;
    TileLists& l = p->inject;
    if (!l.ready) {
        const TileShape g = shape_of(*p);
        const int nt = p->nty * p->ntx, lists = rec_per_shot ? nshots : 1, nthr = tile_threads(g);
        std::vector<int> beg((size_t)nt * lists * (nthr + 1));
        std::vector<int2> ent;
        std::vector<std::vector<int2>> of(nthr);
        l.ok = true;
        for (size_t i = 0; i < (size_t)lists * nrec && l.ok; i++)
            l.ok = h_rz[i] >= 4 && h_rz[i] < nza - 4 && h_rx[i] >= 4 && h_rx[i] < nxa - 4;
        for (int t = 0; t < lists * nt && l.ok; t++) {
            const int tile = t % nt;
            const int ez0 = 4 + (tile / p->ntx) * p->TZ - p->halo * p->T, ex0 = 4 + (tile % p->ntx) * p->TX - p->halo * p->T;
            for (auto& v : of) v.clear();
            for (int r = 0; r < nrec; r++) {
                const size_t i = (size_t)(t / nt) * nrec + r;
                const int er = h_rz[i] - ez0, ec = h_rx[i] - ex0;
                if (er < 0 || er >= g.nrg * g.R || ec < 0 || ec >= 4 * g.EXq) continue;
                of[(er / g.R) * g.EXq + ec / 4].push_back(make_int2(h_rz[i] << 16 | h_rx[i], r));
            }
            const size_t first = ent.size();
            int* const b = &beg[(size_t)t * (nthr + 1)];
            for (int j = 0; j < nthr; j++) {
                b[j] = (int)ent.size();
                ent.insert(ent.end(), of[j].begin(), of[j].end());
            }
            b[nthr] = (int)ent.size();
            if (ent.size() - first > (size_t)kTileInject) l.ok = false;
        }
        if (l.ok && !tile_upload(l, beg, ent, s)) return nullptr;
        l.ready = true;
    }
    if (!l.ok) return nullptr;
    if (!tile_buffers(s)) return nullptr;
    for (int i = 0; i < 2; i++)
        if (!tile_alloc(&d_tile_b[i], 1, true, s) || !tile_alloc(&d_tile_sum[i], 1, false, s) ||
            (p->halo == 8 && !tile_alloc(&d_tile_bmem[i], 4, false, s)))
            return nullptr;
    const size_t bytes = (size_t)shot_stride * nshots * 4;
    for (float* d : d_tile_sum) cudaMemsetAsync(d, 0, bytes, s);
    if (p->halo == 8)
        for (int i = 0; i < 4; i++) cudaMemsetAsync(d_tile_bmem[0] + i * tile_field(), 0, bytes, s);
    tile_bset = 0;
    return p;
}

int pam_engine::tile_adjoint(const TilePlan& p, TileJob job, int nshots, int k0, int k1, const float* slots, int kslot,
                             long long slot_stride, const float* data, float scale, cudaStream_t s) {
    if (k1 <= k0) return PAM_OK;
    TileAdjArgs t{};
    t.f = tile_args(p, nshots);
    t.f.ex[0][0] = d_ub[0];
    t.f.ex[0][1] = d_ub[1];
    t.f.ex[1][0] = d_tile_b[0];
    t.f.ex[1][1] = d_tile_b[1];
    t.f.set0 = tile_bset;
    t.f.k0 = k0;
    t.f.k1 = k1;
    t.f.slots = const_cast<float*>(slots);
    t.f.kslot = kslot;
    t.f.slot_stride = slot_stride;
    t.inj_beg = p.inject.beg();
    t.inj_ent = p.inject.ent();
    t.data = data;
    t.scale = scale;
    t.gsum = d_tile_sum[0];
    t.isum = d_tile_sum[1];
    const size_t smem = smem_of(t.f.g, cfg.approximation, job);
    for (int b = 0; b < nshots; b += p.group) {
        t.f.shot0 = b;
        const int blocks = std::min(p.group, nshots - b) * p.nty * p.ntx;
        cudaError_t err = cudaMemsetAsync(d_tile_bar, 0, sizeof(unsigned), s);
        if (err == cudaSuccess && p.halo == 8) {
            TileCpmlArgs c{};
            c.r = t;
            c.mem[0] = d_tile_bmem[0];
            c.mem[1] = d_tile_bmem[1];
            c.cxab = d_cxab;
            c.czab = d_czab;
            err = ::launch_cpml<kAcoustic, kTileRtmRole>(c, blocks, smem, s);
        } else if (err == cudaSuccess) {
            err = job == kTileExactJob ? launch_adjoint<kTileExact>(t, blocks, smem, s)
                                       : launch_adjoint<kTileRtm>(t, blocks, smem, s);
        }
        if (err != cudaSuccess) return fail(PAM_E_CUDA, "cooperative launch failed: %s", cudaGetErrorString(err));
    }
    tile_bset ^= ((k1 - k0 + p.T - 1) / p.T) & 1;
    return PAM_OK;
}

void pam_engine::tile_fold_image(int nshots, float* img, float* ilum, cudaStream_t s) const {
    tile_fold_image_kernel<<<dim3((cfg.nx + 255) / 256, cfg.nz), 256, 0, s>>>(d_tile_sum[0], d_tile_sum[1], shot_stride, nshots,
                                                                             P, N, cfg.nz, cfg.nx, img, ilum);
}
