// spread_standalone.cu -- sfg_spread_forces: ImmersedBoundary::spreadForces
// (reference immersed_boundary.cpp:25-100) on caller-provided device buffers.
//
// Deterministic gather without floating-point atomics: markers are binned by
// the 32 x 8 force tiles their 4 x 4 stencil covers (counts, list space taken by
// atomics, fill); one CTA per tile applies its markers in ascending order,
// so every cell sums its contributions in the reference's serial order.  The sum is
// added to the caller's field as the reference's OpenMP reduction does
// (F += sum, immersed_boundary.cpp:70-79).  Built with --fmad=false.
#include <algorithm>
#include <climits>
#include <cmath>
#include <mutex>
#include <string>

#include <cuda.h>

#include "../../include/softflow_gpu.h"
#include "markers.cuh"
#include "sfg_internal.h"
#include "launch.cuh"
#include "spread_standalone.cuh"
#include "spread_wide.cuh"

namespace sfg_host {
void set_error(const std::string& msg);
}

namespace sfg {

__device__ __forceinline__ int ring_of(const int* __restrict__ off, int ncaps, int m) {
    int lo = 0, hi = ncaps - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= m) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ int sa_tiles(int nx, int ny, int tiles_x, int ix0, int iy0, int out[8]) {
    int tys[2], nty = 0;
    for (int iy = iy0 - 1; iy <= iy0 + 2; ++iy) {
        if (iy < 0 || iy >= ny) continue;
        const int ty = iy / TILE_H;
        if (nty == 0 || tys[nty - 1] != ty) tys[nty++] = ty;
    }
    int txs[4], ntx = 0;
    for (int ix = ix0 - 1; ix <= ix0 + 2; ++ix) {
        int jx = ix;
        if (jx < 0) jx += nx;
        if (jx >= nx) jx -= nx;
        if (jx < 0 || jx >= nx) continue;
        const int tx = jx / TILE_W;
        bool dup = false;
        for (int a = 0; a < ntx; ++a) dup |= (txs[a] == tx);
        if (!dup) txs[ntx++] = tx;
    }
    int n = 0;
    for (int a = 0; a < nty; ++a)
        for (int b = 0; b < ntx; ++b) out[n++] = tys[a] * tiles_x + txs[b];
    return n;
}

// Arc length (min image, Lx = nx), stencil origin and tile counts.
__global__ void k_sa_prep(int nx, int ny, int tiles_x, int ncaps, const int* __restrict__ off,
                          const double2* __restrict__ pos, const double2* __restrict__ frc, int M,
                          SpreadScratch sc) {
    chain_begin();
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    // num_markers must equal off[ncaps]; a marker beyond the rings (a larger
    // count) is skipped instead of reading past the caller's arrays
    if (m >= off[ncaps]) {
        sc.ds[m] = 0.0;
        sc.ix0[m] = INT_MIN;
        sc.iy0[m] = 0;
        return;
    }
    const int c = ring_of(off, ncaps, m);
    const int o = off[c], n = off[c + 1] - o, k = m - o;
    const double Lx = (double)nx;
    const double2 p = pos[m];
    const double dp = norm_d(min_image_d(p, pos[o + (k - 1 + n) % n], Lx));
    const double dn = norm_d(min_image_d(pos[o + (k + 1) % n], p, Lx));
    sc.ds[m] = 0.5 * (dp + dn);
    int ix0 = INT_MIN, iy0 = 0;
    const double2 f = frc[m];
    // NaN / Inf guards of immersed_boundary.cpp:248-252 and the stencil row
    // test of :257-258; markers beyond one period outside are skipped
    if (finite2(p) && !(isnan(f.x) || isnan(f.y)) && p.x >= -Lx + 2.0 && p.x < 2.0 * Lx - 3.0 &&
        fabs(p.y) < 1e9) {
        const int a = (int)floor(p.x), b = (int)floor(p.y);
        if (!(b < -2 || b >= ny + 2)) {
            ix0 = a;
            iy0 = b;
        }
    }
    sc.ix0[m] = ix0;
    sc.iy0[m] = iy0;
    if (ix0 == INT_MIN) return;
    int t[8];
    const int nt = sa_tiles(nx, ny, tiles_x, ix0, iy0, t);
    for (int i = 0; i < nt; ++i) atomicAdd(&sc.tile_cnt[t[i]], 1);
}

// Clears the per-tile counters and writes the Peskin table
// (delta_function.h:29-37: phi on 1025 points of [0, 2]) into the scratch.
// Every operation is exact in double except the square root, which is
// correctly rounded on the device as in the host library, and the unit is
// built without contraction, so the table equals the host-built one of the
// simulation contexts bit for bit.
__global__ void k_sa_init(int T, SpreadScratch sc) {
    chain_begin();
    const int n = T > 1025 ? T : 1025;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (i < T) sc.tile_cnt[i] = 0;
        if (i == 0) *sc.total = 0;
        if (i <= 1024) {
            const double ar = 2.0 * static_cast<double>(i) / 1024;
            double v = 0.0;
            if (ar <= 1.0) v = 0.125 * (3.0 - 2.0 * ar + sqrt(1.0 + 4.0 * ar - 4.0 * ar * ar));
            else v = 0.125 * (5.0 - 2.0 * ar - sqrt(-7.0 + 12.0 * ar - 4.0 * ar * ar));
            sc.phi[i] = v;
        }
    }
}

// List space of every tile, one atomic per warp (where a list lies does not
// matter): tile_pos[t] is the next free entry, tile_off[t] the first.
__global__ void k_sa_alloc(int T, SpreadScratch sc) {
    chain_begin();
    const int t = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    const int cnt = t < T ? sc.tile_cnt[t] : 0;
    int inc = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    int base = 0;
    if (lane == 31 && inc > 0) base = atomicAdd(sc.total, inc);
    base = __shfl_sync(0xffffffffu, base, 31) + inc - cnt;
    if (cnt > 0) {
        sc.tile_off[t] = base;
        sc.tile_pos[t] = base;
    }
}

__global__ void k_sa_fill(int nx, int ny, int tiles_x, int M, SpreadScratch sc) {
    chain_begin();
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M || sc.ix0[m] == INT_MIN) return;
    int t[8];
    const int nt = sa_tiles(nx, ny, tiles_x, sc.ix0[m], sc.iy0[m], t);
    for (int i = 0; i < nt; ++i) sc.list[atomicAdd(&sc.tile_pos[t[i]], 1)] = m;
}

// One CTA per tile (spread_wide.cuh).  The staging lanes evaluate their markers'
// weights.  Marker by marker, with two loads and the table lookups in a row for
// each, one warp a tile, 500 rings of 40 markers on 1000 x 700 took 112 us.
__global__ void __launch_bounds__(BAND_WARPS * 32)
k_sa_gather(int nx, int ny, int tiles_x, int T, const double2* __restrict__ pos,
            const double2* __restrict__ frc, const double* phi_tbl, SpreadScratch sc,
            double* __restrict__ Fx, double* __restrict__ Fy) {
    __shared__ BandTile s_band[BAND_WARPS];
    __shared__ __align__(16) int s_sort[SORT_SMEM];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    BandTile& B = s_band[warp];
    chain_begin();
    for (int t = blockIdx.x; t < T; t += gridDim.x) {   // uniform in the CTA
        const int cnt = sc.tile_cnt[t];
        if (cnt == 0) continue;
        int* list = sc.list + sc.tile_off[t];
        const int x0 = (t % tiles_x) * TILE_W + BAND_W * warp, y0 = (t / tiles_x) * TILE_H;
        const int first = tile_list_sort<32 * BAND_WARPS>(list, cnt, s_sort, threadIdx.x, false);
        __syncwarp();
        for (int c = lane; c < BandTile::CELLS; c += 32) B.ax[c] = B.ay[c] = 0.0;
        auto org_of = [&](int m) { return make_int2(sc.ix0[m], sc.iy0[m]); };
        auto load = [&](int m, int sy, BandMarker& k) {
            const double2 p = pos[m];
            k.f = frc[m];
            k.org = make_int2(sc.ix0[m], sc.iy0[m]);
            k.ds = sc.ds[m];
#pragma unroll
            for (int q = 0; q < 4; ++q) k.wx[q] = phi_lut(phi_tbl, p.x - (double)(k.org.x - 1 + q));
            k.wy = phi_lut(phi_tbl, p.y - (double)(k.org.y - 1 + sy));
        };
        band_spread<true>(B, list, cnt, first, nx, ny, x0, 0, y0, lane, org_of, load);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = (lane >> 3) + 4 * h, a = r * BandTile::ROW + (lane & 7);
            const int jx = x0 + (lane & 7), jy = y0 + r;
            if (jx < nx && jy < ny) {
                const size_t n = (size_t)jy * nx + jx;
                Fx[n] = Fx[n] + B.ax[a];
                Fy[n] = Fy[n] + B.ay[a];
            }
        }
    }
}

size_t spread_scratch_bytes(int M, int T) {
    const size_t a = 256;
    auto up = [a](size_t b) { return (b + a - 1) / a * a; };
    return up(sizeof(double) * M) + 2 * up(sizeof(int) * M) + up(sizeof(int) * 8 * (size_t)M) +
           3 * up(sizeof(int) * T) + up(sizeof(int)) + up(sizeof(double) * 1025);
}

SpreadScratch carve_spread_scratch(void* base, int M, int T) {
    const size_t a = 256;
    auto up = [a](size_t b) { return (b + a - 1) / a * a; };
    char* p = static_cast<char*>(base);
    SpreadScratch sc;
    sc.ds = reinterpret_cast<double*>(p);         p += up(sizeof(double) * M);
    sc.ix0 = reinterpret_cast<int*>(p);           p += up(sizeof(int) * M);
    sc.iy0 = reinterpret_cast<int*>(p);           p += up(sizeof(int) * M);
    sc.list = reinterpret_cast<int*>(p);          p += up(sizeof(int) * 8 * (size_t)M);
    sc.tile_cnt = reinterpret_cast<int*>(p);      p += up(sizeof(int) * T);
    sc.tile_off = reinterpret_cast<int*>(p);      p += up(sizeof(int) * T);
    sc.tile_pos = reinterpret_cast<int*>(p);      p += up(sizeof(int) * T);
    sc.total = reinterpret_cast<int*>(p);         p += up(sizeof(int));
    sc.phi = reinterpret_cast<double*>(p);
    return sc;
}

// Enqueues the whole spread on `st` with the scratch in `sc`.  Everything the
// scratch must start with (zero counters, the Peskin table) is written by
// k_sa_init on the stream, so the scratch may hold anything on entry.
int run_spread(int nx, int ny, int ncaps, const int* off, const double* pos, const double* frc,
               double* Fx, double* Fy, SpreadScratch sc, int M, int T, int tiles_x,
               cudaStream_t st) {
    int nsm = 0, dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) {
        sfg_host::set_error(std::string("spread: ") + cudaGetErrorString(e));
        return SFG_ERR_CUDA;
    }
    const int B = 256, G = (M + B - 1) / B;
    const int Gi = std::min((std::max(T, 1025) + B - 1) / B, nsm * 8);
    const double2* p2 = reinterpret_cast<const double2*>(pos);
    const double2* f2 = reinterpret_cast<const double2*>(frc);
    const int grid = std::max(1, std::min(T, nsm * 6));
    launch_chain(false, k_sa_init, Gi, B, 0, st, T, sc);
    launch_chain(true, k_sa_prep, G, B, 0, st, nx, ny, tiles_x, ncaps, off, p2, f2, M, sc);
    launch_chain(true, k_sa_alloc, (T + B - 1) / B, B, 0, st, T, sc);
    launch_chain(true, k_sa_fill, G, B, 0, st, nx, ny, tiles_x, M, sc);
    launch_chain(true, k_sa_gather, grid, BAND_WARPS * 32, 0, st, nx, ny, tiles_x, T, p2, f2,
                 (const double*)sc.phi, sc, Fx, Fy);
    e = cudaGetLastError();
    if (e != cudaSuccess) {
        sfg_host::set_error(std::string("spread: ") + cudaGetErrorString(e));
        return SFG_ERR_CUDA;
    }
    return SFG_OK;
}

int check_spread_args(int nx, int ny, int ncaps, const int* off, const double* pos,
                      const double* frc, const double* Fx, const double* Fy, const char* who) {
    if (nx < 4 || ny < 1) {
        sfg_host::set_error(std::string(who) + ": need nx >= 4 and ny >= 1");
        return SFG_ERR_ARG;
    }
    if (ncaps < 0 || (ncaps > 0 && (!off || !pos || !frc)) || !Fx || !Fy) {
        sfg_host::set_error(std::string(who) + ": null or negative argument");
        return SFG_ERR_ARG;
    }
    return SFG_OK;
}

}  // namespace sfg

using namespace sfg;

namespace {

// Scratch memory of sfg_spread_forces: a pool of its own per device context that
// keeps at most 32 MiB (one chunk of the driver's) between calls, until
// sfg_release_scratch.  The device's default pool gives its memory back
// whenever the stream is waited for, and the next call maps it anew: a caller
// that waits for each spread paid 600 us for 140 us of work.
struct ScratchPool {
    unsigned long long context = 0;   // cuCtxGetId: no two contexts of a process share one
    cudaMemPool_t pool = nullptr;     // null: it could not be made
};
constexpr int MAX_POOLS = 64;
std::mutex g_pool_mutex;
ScratchPool g_pools[MAX_POOLS];
int g_num_pools = 0;

// The current context's id, 0 without one.  A pool ends with its context
// (cudaDeviceReset); by the id its handle is never used in the next one.
unsigned long long context_id() {
    using GetId = CUresult (*)(CUcontext, unsigned long long*);
    static const GetId get = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &found) !=
                cudaSuccess || found != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return reinterpret_cast<GetId>(f);
    }();
    unsigned long long id = 0;
    return get && get(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}

// The current context's entry, null without one (all callers hold the mutex).
ScratchPool* find_pool(unsigned long long context) {
    for (int i = 0; i < g_num_pools; ++i)
        if (g_pools[i].context == context) return &g_pools[i];
    return nullptr;
}

// Null while the stream is being captured (the call's allocation then becomes a
// node of the graph, from the default pool) or when the pool cannot be made.
cudaMemPool_t scratch_pool(cudaStream_t st) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    int dev = 0;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone ||
        cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    const unsigned long long context = context_id();
    if (context == 0) return nullptr;
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    if (ScratchPool* known = find_pool(context)) return known->pool;
    if (g_num_pools == MAX_POOLS) return nullptr;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    unsigned long long keep = 32ull << 20;
    cudaMemPool_t pool = nullptr;
    // (another thread's stream capture forbids neither call to this one)
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess ||
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
        cudaGetLastError();
        if (pool) cudaMemPoolDestroy(pool);
        pool = nullptr;
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
    g_pools[g_num_pools++] = {context, pool};
    return pool;
}

}  // namespace

extern "C" int sfg_spread_forces(int nx, int ny, int ncaps, const int* d_offsets,
                                 const double* d_pos, const double* d_force, double* d_Fx,
                                 double* d_Fy, int num_markers, void* stream) {
    int rc = check_spread_args(nx, ny, ncaps, d_offsets, d_pos, d_force, d_Fx, d_Fy,
                               "sfg_spread_forces");
    if (rc) return rc;
    if (ncaps == 0 || num_markers <= 0) return SFG_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int tiles_x = (nx + TILE_W - 1) / TILE_W, tiles_y = (ny + TILE_H - 1) / TILE_H;
    const int T = tiles_x * tiles_y, M = num_markers;
    void* base = nullptr;
    const cudaMemPool_t pool = scratch_pool(st);
    const size_t bytes = spread_scratch_bytes(M, T);
    cudaError_t e = pool ? cudaMallocFromPoolAsync(&base, bytes, pool, st) : cudaErrorMemoryAllocation;
    if (e == cudaErrorMemoryAllocation) {   // the default pool may still hold enough
        if (pool) cudaGetLastError();
        e = cudaMallocAsync(&base, bytes, st);
    }
    if (e != cudaSuccess) {
        sfg_host::set_error(std::string("sfg_spread_forces: ") + cudaGetErrorString(e));
        return SFG_ERR_CUDA;
    }
    rc = run_spread(nx, ny, ncaps, d_offsets, d_pos, d_force, d_Fx, d_Fy,
                    carve_spread_scratch(base, M, T), M, T, tiles_x, st);
    e = cudaFreeAsync(base, st);
    if (rc == SFG_OK && e != cudaSuccess) {
        sfg_host::set_error(std::string("sfg_spread_forces: ") + cudaGetErrorString(e));
        return SFG_ERR_CUDA;
    }
    return rc;
}

extern "C" int sfg_release_scratch(void) {
    const unsigned long long context = context_id();
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    const ScratchPool* known = context ? find_pool(context) : nullptr;
    const cudaError_t e = known && known->pool ? cudaMemPoolTrimTo(known->pool, 0) : cudaSuccess;
    if (e != cudaSuccess) {
        sfg_host::set_error(std::string("sfg_release_scratch: ") + cudaGetErrorString(e));
        return SFG_ERR_CUDA;
    }
    return SFG_OK;
}
