// ivp_noalloc.cu -- SPH density and k = 1/(Aii + eps) for one scene without
// any device allocation.
//
// Who needs this: callers that cannot allocate device memory themselves or let
// a library do it -- code that runs inside another runtime's memory arena
// (for example a host whose GPU memory is managed by Warp's or a renderer's
// fixed-budget allocator), and real-time loops that cannot afford the
// implicit device synchronisation of cudaMalloc/cudaFree.  The
// regular engine needs a caller-provided workspace sized by
// ivp_workspace_bytes; this entry point needs none.  Instead it works in one
// file-scope device array of fixed size (kScratchBytes below, about 6.3 MB),
// which every GPU that loads the library holds until the process exits.
//
// Limits: at most IVP_NOALLOC_MAX_PARTICLES particles and at most
// IVP_NOALLOC_MAX_CELLS grid cells (ceil(L/h) per axis multiplied).  Larger
// inputs are rejected with IVP_ERR_BAD_ARG before any device work.
//
// Sharing: every call, on every stream, uses the same array and leaves its
// contents behind.  The cell counters that must start at zero are cleared by
// each call; everything else is overwritten before it is read.  Two calls
// whose work overlaps on the GPU (different streams, or different host
// threads) race on the array and give wrong results: serialise them.
//
// Set-up: the device address of the array is looked up with
// cudaGetSymbolAddress the first time the entry point runs on a device (with
// that device current) and cached.  Make that first call on a device before
// any stream capture.
#include <cuda_runtime.h>

#include <cmath>
#include <mutex>

#include <string>

#include "../../include/ivp.h"
#include "ivp_device.cuh"
#include "ivp_scan.cuh"
#include "ivp_window.cuh"

namespace ivp {
// the engine's thread-local error text (ivp_last_error), set in ivp_engine.cu
void set_last_error(const std::string& msg);
}  // namespace ivp

namespace {

using ivp::cell_coord;
using ivp::dot3;

constexpr int kMaxParticles = IVP_NOALLOC_MAX_PARTICLES;
constexpr int kMaxKeys = 2 * IVP_NOALLOC_MAX_CELLS;
constexpr int kMaxDevices = 64;

struct Scratch {
    int cell_count[kMaxKeys];
    int cell_start[kMaxKeys + 64];
    int block_sums[(kMaxKeys + ivp::SCAN_TILE - 1) / ivp::SCAN_TILE];
    int key[kMaxParticles];
    int rank[kMaxParticles];
    int placed[kMaxParticles];
    int pid[kMaxParticles];
    float4 xm[kMaxParticles];
};
constexpr size_t kScratchBytes = sizeof(Scratch);

static __device__ __align__(256) unsigned char g_scratch[kScratchBytes];

std::mutex g_setup_mutex;
Scratch* g_scratch_addr[kMaxDevices] = {};

struct Grid {
    int dims[3];
    int ncell;
    float cell_inv, h, inv_h, cubic_k, spiky_k, W0, r2_max;
    int cap;
};

__global__ void na_keys(const float* __restrict__ x, const int* __restrict__ dyn, int n, Grid g, Scratch* S) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int cx = cell_coord(x[3 * p], g.cell_inv, g.dims[0]);
    const int cy = cell_coord(x[3 * p + 1], g.cell_inv, g.dims[1]);
    const int cz = cell_coord(x[3 * p + 2], g.cell_inv, g.dims[2]);
    const int key = (dyn[p] ? 0 : g.ncell) + (cz * g.dims[1] + cy) * g.dims[0] + cx;
    S->key[p] = key;
    S->rank[p] = atomicAdd(&S->cell_count[key], 1);
}

__global__ void na_place(int n, Scratch* S) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    S->placed[S->cell_start[S->key[p]] + S->rank[p]] = p;
}

// Stable order by particle id inside each cell, and the slot-ordered copies.
__global__ void na_order(const float* __restrict__ x, const float* __restrict__ m, int n, Scratch* S) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int p = S->placed[s];
    const int key = S->key[p];
    const int b = S->cell_start[key], e = S->cell_start[key + 1];
    int before = 0;
    for (int q = b; q < e; ++q) before += (S->placed[q] < p);
    const int slot = b + before;
    S->pid[slot] = p;
    S->xm[slot] = make_float4(x[3 * p], x[3 * p + 1], x[3 * p + 2], m[p]);
}

// Density (pressure_base.py:12-46) and k (pressure_base.py:49-87) of every
// dynamic particle over its first `cap` neighbours |x_i - x_j| < h, j != i
// (neighbour_search.py:10-51), in the same candidate order as the engine's
// neighbour build, but without storing the lists.  Static particles get k = 0.
//
// One warp per eight slots, as in the engine's build for small scenes: a thread
// per particle walked 270 candidates one after another, on 176 CTAs of 256
// threads for 40,000 particles (99 us), and left most of the chip waiting.  One
// warp per CTA: 60 us a call; two: 63 to 73.
constexpr int kSub = 8;

__global__ void __launch_bounds__(32) na_density_aii(int n, Grid g, Scratch* S, float* __restrict__ density,
                                                     float* __restrict__ kdiag) {
    __shared__ ivp::BuildShared<kSub> B;
    const int lane = threadIdx.x;
    const int i0 = blockIdx.x * kSub;
    const int n_dyn = S->cell_start[g.ncell];
    if (lane < kSub && i0 + lane < n && i0 + lane >= n_dyn) kdiag[S->pid[i0 + lane]] = 0.0f;
    const int m = min(kSub, n_dyn - i0);
    if (m <= 0) return;
    ivp::WindowGrid W;
    W.cell_start = S->cell_start;
    W.xm = S->xm;
    W.ncell = g.ncell;
    for (int a = 0; a < 3; ++a) W.dims[a] = g.dims[a];
    W.r2_max = g.r2_max;
    float4 xl = make_float4(0.f, 0.f, 0.f, 0.f);
    int3 cell = make_int3(0, 0, 0);
    int pid = 0;
    if (lane < m) {
        xl = W.xm[i0 + lane];
        pid = S->pid[i0 + lane];
        cell = make_int3(cell_coord(xl.x, g.cell_inv, g.dims[0]), cell_coord(xl.y, g.cell_inv, g.dims[1]),
                         cell_coord(xl.z, g.cell_inv, g.dims[2]));
    }
    const int run = ivp::filter_hits<kSub>(W, B, i0, m, xl, cell, ivp::kHits).run;
    __syncwarp();
    ivp::HitSums s;  // lane p's own particle
    const int found = lane < m ? B.found[lane] : 0;
    // more hits than a list holds (a cache_size above it only), or a window
    // that does not fit the filter: the whole warp on one particle
    const unsigned alone = __ballot_sync(0xffffffffu, found < 0 || (found > ivp::kHits && g.cap > ivp::kHits));
    for (int p0 = 0; p0 < m; p0 += 4) {
        // eight lanes per particle
        const int p = p0 + (lane >> 3), q = min(p, m - 1);
        const int n_hit = p < m ? min(min(B.found[p], ivp::kHits), g.cap) : 0;
        const int* delta = B.delta[__shfl_sync(0xffffffffu, run, q)];
        const float4 xi = B.pos[q];
        ivp::HitSums a;
        for (int k = lane & 7; k < n_hit; k += 8) {
            const int code = B.hit[k][p];
            const int j = delta[code >> ivp::kOrdShift] + (code & ((1 << ivp::kOrdShift) - 1));
            const float4 xj = __ldg(W.xm + j);
            const float3 r = make_float3(xi.x - xj.x, xi.y - xj.y, xi.z - xj.z);
            float w;
            ivp::hit_terms(r, ivp::norm2_rn(r), xj.w, j < n_dyn, g.h, g.inv_h, g.spiky_k, g.cubic_k, a, &w);
        }
        __syncwarp();
        ivp::sum_lanes<8>(a);
        ivp::own_sums(a, p0, 4, s);
    }
    for (unsigned left = alone; left; left &= left - 1u) {
        const int p = __ffs(left) - 1, i = i0 + p;
        const float4 xi = B.pos[p];
        int b, len, at = 0;
        ivp::window_range(W, cell_coord(xi.x, g.cell_inv, g.dims[0]), cell_coord(xi.x, g.cell_inv, g.dims[0]),
                          cell_coord(xi.y, g.cell_inv, g.dims[1]), cell_coord(xi.z, g.cell_inv, g.dims[2]), lane, b, len);
        ivp::HitSums a;
        for (int q = 0; q < 18; ++q) {
            const int jb = __shfl_sync(0xffffffffu, b, q), c = __shfl_sync(0xffffffffu, len, q);
            for (int base = 0; base < c; base += 32) {
                const int j = jb + base + lane;
                float4 xj = xi;
                if (base + lane < c) xj = __ldg(W.xm + j);
                const float3 r = make_float3(xi.x - xj.x, xi.y - xj.y, xi.z - xj.z);
                const float r2 = ivp::norm2_rn(r);
                const bool in = base + lane < c && j != i && r2 <= W.r2_max;
                const unsigned ball = __ballot_sync(0xffffffffu, in);
                float w;
                if (in && at + __popc(ball & ((1u << lane) - 1u)) < g.cap)
                    ivp::hit_terms(r, r2, xj.w, j < n_dyn, g.h, g.inv_h, g.spiky_k, g.cubic_k, a, &w);
                at += __popc(ball);
            }
        }
        ivp::sum_lanes<32>(a);
        if (lane == p) s = a;
    }
    if (lane < m) {
        const float mi = xl.w;
        float rho = 0.0f;
        rho = rho + mi * g.W0;
        rho += s.rho;
        const float aii = s.aii + dot3(s.jii, s.jii) * __frcp_rn(mi);
        density[pid] = rho;
        kdiag[pid] = __frcp_rn(aii + 1e-3f);
    }
}

// Every failure leaves its reason where ivp_last_error() reads it.
int fail(int code, const char* msg) {
    ivp::set_last_error(msg);
    return code;
}

// One launch; its own status (cudaLaunchKernel reports this launch's error,
// not one left pending by earlier work of the caller).
int launch(const void* fn, int grid, int block, void** args, cudaStream_t s, const char* what) {
    const cudaError_t e = cudaLaunchKernel(fn, dim3(grid), dim3(block), args, 0, s);
    if (e != cudaSuccess) {
        cudaGetLastError();  // this launch's error is now the last error: clear it, it is reported here
        return fail(IVP_ERR_CUDA, (std::string(what) + ": " + cudaGetErrorString(e)).c_str());
    }
    return IVP_OK;
}

}  // namespace

extern "C" int ivp_density_aii_noalloc(const float* x, const float* m, const int32_t* is_dynamic, int32_t n_particles,
                                       float particle_radius, const float* domain_size, int32_t cache_size,
                                       float* density, float* kdiag, void* stream) {
    if (n_particles < 0 || !domain_size || cache_size <= 0 || !(particle_radius > 0.0f))
        return fail(IVP_ERR_BAD_ARG, "ivp_density_aii_noalloc: bad argument");
    if (n_particles > kMaxParticles)
        return fail(IVP_ERR_BAD_ARG, "more particles than IVP_NOALLOC_MAX_PARTICLES");
    if (n_particles == 0) return IVP_OK;
    if (!x || !m || !is_dynamic || !density || !kdiag)
        return fail(IVP_ERR_BAD_ARG, "ivp_density_aii_noalloc: null array");
    Grid g;
    const float h = 4.0f * particle_radius;  // config_builder.py:51-52
    long ncell = 1;
    for (int a = 0; a < 3; ++a) {
        if (!(domain_size[a] > 0.0f)) return fail(IVP_ERR_BAD_ARG, "ivp_density_aii_noalloc: bad domain");
        double dd = std::ceil((double)domain_size[a] / (double)h);
        if (dd > 65536.0) return fail(IVP_ERR_BAD_ARG, "ivp_density_aii_noalloc: grid too large");
        g.dims[a] = dd < 1.0 ? 1 : (int)dd;
        ncell *= g.dims[a];
    }
    if (ncell > IVP_NOALLOC_MAX_CELLS)
        return fail(IVP_ERR_BAD_ARG, "more grid cells than IVP_NOALLOC_MAX_CELLS");
    g.ncell = (int)ncell;
    g.h = h;
    g.cell_inv = 1.0f / h;
    g.inv_h = 1.0f / h;
    g.r2_max = ivp::strict_r2_max(h);
    float k = 8.0f / 3.14159265359f;
    k = k / (h * h * h);
    g.cubic_k = k;
    g.W0 = k * (6.0f * 0.0f - 6.0f * 0.0f + 1.0f);
    g.spiky_k = 45.0f / (3.14159265359f * h * h * h * h * h * h);
    g.cap = cache_size;

    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
        return fail(IVP_ERR_CUDA, "ivp_density_aii_noalloc: no current device");
    Scratch* S = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_setup_mutex);
        if (!g_scratch_addr[dev]) {
            void* addr = nullptr;
            cudaError_t e = cudaGetSymbolAddress(&addr, g_scratch);
            if (e != cudaSuccess || !addr) {
                if (e != cudaSuccess) cudaGetLastError();  // reported here
                return fail(IVP_ERR_CUDA, (std::string("ivp_density_aii_noalloc: cudaGetSymbolAddress: ") +
                                           cudaGetErrorString(e)).c_str());
            }
            g_scratch_addr[dev] = static_cast<Scratch*>(addr);
        }
        S = g_scratch_addr[dev];
    }
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const int n = n_particles, n_keys = 2 * g.ncell;
    const int B = 256, nb = (n + B - 1) / B;
    {
        const cudaError_t e = cudaMemsetAsync(S->cell_count, 0, sizeof(int) * (size_t)n_keys, s);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return fail(IVP_ERR_CUDA, (std::string("ivp_density_aii_noalloc: memset: ") + cudaGetErrorString(e)).c_str());
        }
    }
    int* counts = S->cell_count;
    int* starts = S->cell_start;
    int* bsums = S->block_sums;
    int nk = n_keys, nsb = (n_keys + ivp::SCAN_TILE - 1) / ivp::SCAN_TILE, nn = n;
    const float* px = x;
    const float* pm = m;
    const int* pd = is_dynamic;
    void* a_keys[] = {&px, &pd, &nn, &g, &S};
    void* a_scan1[] = {&counts, &starts, &bsums, &nk};
    void* a_scan2[] = {&starts, &bsums, &nk, &nsb};
    void* a_place[] = {&nn, &S};
    void* a_order[] = {&px, &pm, &nn, &S};
    void* a_dens[] = {&nn, &g, &S, &density, &kdiag};
    int st = launch((const void*)na_keys, nb, B, a_keys, s, "na_keys");
    if (st == IVP_OK) st = launch((const void*)ivp::k_scan_local, nsb, ivp::SCAN_BLOCK, a_scan1, s, "scan_local");
    if (st == IVP_OK) st = launch((const void*)ivp::k_scan_add, nsb, ivp::SCAN_BLOCK, a_scan2, s, "scan_add");
    if (st == IVP_OK) st = launch((const void*)na_place, nb, B, a_place, s, "na_place");
    if (st == IVP_OK) st = launch((const void*)na_order, nb, B, a_order, s, "na_order");
    if (st == IVP_OK) st = launch((const void*)na_density_aii, (n + kSub - 1) / kSub, 32, a_dens, s, "na_density_aii");
    if (st != IVP_OK) return st;
    return IVP_OK;
}
