// ivp_window.cuh -- the neighbour search of a few consecutive slots by one
// warp: hit lists and the SPH sums over them, shared by the engine's neighbour
// build and the allocation-free density.
#pragma once
#include <cmath>

#include "ivp_device.cuh"

namespace ivp {

constexpr int kHits = 64;         // >= every cache_size the rows can hold
constexpr int kMaxChunks = 16;    // window candidates / 32 of the filter pass
constexpr int kOrdShift = 9;      // hit code: (range ordinal << 9) | window position (< 512)
static_assert(kMaxChunks * 32 <= (1 << kOrdShift) && 18 << kOrdShift <= 65536, "hit codes are 16 bits");

template <int SUB>
struct BuildShared {
    static constexpr bool kLists = SUB < 32;           // the hits as lists, or as the ballots' bits
    static constexpr int VMAX = SUB < 16 ? SUB : 16;   // runs with a kept window
    static constexpr int kRunFill = kLists ? 3 : 12;   // a run takes in up to two more cells while it holds no more particles
    float4 pos[SUB + 1];                               // (the tests go over particles in pairs)
    unsigned mask[kMaxChunks][SUB + 1];
    int delta[VMAX][18];                               // slot = delta[run][ordinal] + window position
    int2 starts[kLists ? 1 : VMAX][kLists ? 1 : kMaxChunks];  // {range starts in the chunk, ordinal before it}
    int found[SUB];                                    // hits of each particle (not capped); -1: scan it alone
    alignas(16) unsigned short code[kLists ? kMaxChunks * 32 : 2];
    unsigned short hit[kLists ? kHits : 1][SUB];
};

// A lane's particle after the filter pass: its run and the run's chunk count.
struct RunOf {
    int run = 0, chunks = 0;
};

// Largest float r2 with sqrtf(r2) < h: `r2 <= r2_max` is the strict `|r| < h` test
// (IEEE sqrt is monotone and correctly rounded on host and device alike).
inline float strict_r2_max(float h) {
    float t = h * h;
    while (std::sqrt(t) >= h) t = std::nextafter(t, 0.0f);
    while (std::sqrt(std::nextafter(t, INFINITY)) < h) t = std::nextafter(t, INFINITY);
    return t;
}

// What the scan of a cell's window needs (one scene of an engine, or the grid
// of ivp_density_aii_noalloc).
struct WindowGrid {
    const int* cell_start;  // of the scene's keys: dynamic cells, then static cells
    const float4* xm;
    int ncell, dims[3];
    float r2_max;
};

// Lane q < 18: the q-th slot range of the window of cells (cx .. cx1, cy, cz).
__device__ __forceinline__ void window_range(const WindowGrid& W, int cx, int cx1, int cy, int cz, int q, int& b,
                                             int& len) {
    b = len = 0;
    const int rr = q >> 1;
    const int z = cz + rr / 3 - 1, y = cy + rr % 3 - 1;
    if (q < 18 && z >= 0 && z < W.dims[2] && y >= 0 && y < W.dims[1]) {
        const int x0 = cx > 0 ? cx - 1 : 0, x1 = cx1 < W.dims[0] - 1 ? cx1 + 1 : W.dims[0] - 1;
        const int* cs = W.cell_start + ((q & 1) ? W.ncell : 0) + (z * W.dims[1] + y) * W.dims[0];
        b = __ldg(cs + x0);
        len = __ldg(cs + x1 + 1) - b;
    }
}

// Filter pass of one warp over slots i0 .. i0 + n - 1 (n <= SUB).  Lane l < n
// passes its particle's position and cell.  With lists, every particle's hit
// count and list are left in S; without, the ballots of a test with fused
// products and a slack of 1e-5, which lets a few more through (and the particle
// itself), for the exact test to come.
template <int SUB>
__device__ __forceinline__ RunOf filter_hits(const WindowGrid& W, BuildShared<SUB>& S, int i0, int n, float4 xi,
                                             int3 cell, int cap) {
    constexpr bool LISTS = BuildShared<SUB>::kLists;
    const int lane = threadIdx.x & 31;
    const unsigned le = 0xffffffffu >> (31 - lane);
    const float r2_near = W.r2_max * 1.00001f;
    if (lane < n) {
        S.pos[lane] = xi;
        S.found[lane] = 0;
    }
    const int row = lane < n ? cell.z * W.dims[1] + cell.y : -1;
    RunOf mine;
    __syncwarp();
    for (int first = 0, run = 0; first < n; ++run) {
        const int cx = __shfl_sync(0xffffffffu, cell.x, first);
        const int cy = __shfl_sync(0xffffffffu, cell.y, first);
        const int cz = __shfl_sync(0xffffffffu, cell.z, first);
        const bool after = lane >= first && row == cz * W.dims[1] + cy;
        int ext = 0;
        int np = __popc(__ballot_sync(0xffffffffu, after && cell.x == cx));
        for (int e = 1; e <= 2 && np < BuildShared<SUB>::kRunFill; ++e) {
            const int more = __popc(__ballot_sync(0xffffffffu, after && cell.x <= cx + e));
            if (more > BuildShared<SUB>::kRunFill) break;
            np = more;
            ext = e;
        }
        int b, len;
        window_range(W, cx, cx + ext, cy, cz, lane, b, len);
        int incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        const int L = __shfl_sync(0xffffffffu, incl, 31);
        if (L > kMaxChunks * 32 || run >= BuildShared<SUB>::VMAX) {
            // a crowded window, or particles scattered over many cells: each
            // is scanned on its own by the whole warp
            if (lane < np) S.found[first + lane] = -1;
            first += np;
            continue;
        }
        const int off = incl - len;
        const unsigned some = __ballot_sync(0xffffffffu, len > 0);
        if (len > 0) S.delta[run][__popc(some & le) - 1] = b - off;
        const int self = __shfl_sync(0xffffffffu, b - off, 8);  // range 8: the run's own cell row
        __syncwarp();
        int ord = -1;  // last range begun before the chunk
        auto chunk = [&](int c) {
            const unsigned rel = (unsigned)(off - 32 * c);
            const unsigned starts = __reduce_or_sync(0xffffffffu, (len > 0 && rel < 32u) ? 1u << rel : 0u);
            const int o = ord + __popc(starts & le);
            if constexpr (!LISTS)
                if (lane == 0) S.starts[run][c] = make_int2((int)starts, ord);
            ord += __popc(starts);
            const int v = 32 * c + lane;
            float4 x = make_float4(__int_as_float(0x7fc00000), 0.f, 0.f, 0.f);  // past the end: never within h
            if (v < L) {
                if constexpr (LISTS) S.code[v] = (unsigned short)((o << kOrdShift) | v);
                x = __ldg(W.xm + (S.delta[run][o] + v));
            }
            return x;
        };
        const int nch = (L + 31) >> 5;
        float4 xn = chunk(0);
        for (int c = 0; c < nch; ++c) {
            const float4 xj = xn;
            if (c + 1 < nch) xn = chunk(c + 1);
            // two particles at a time; a last odd one tests its successor's
            // place along, whose ballots its own run writes later
#pragma unroll 2
            for (int p = first; p < first + np; p += 2) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float4 xp = S.pos[p + u];
                    const float3 r = make_float3(xp.x - xj.x, xp.y - xj.y, xp.z - xj.z);
                    const bool in = LISTS ? norm2_rn(r) <= W.r2_max
                                          : __fmaf_rn(r.z, r.z, __fmaf_rn(r.y, r.y, r.x * r.x)) <= r2_near;
                    const unsigned ball = __ballot_sync(0xffffffffu, in);
                    if (lane == 0) S.mask[c][p + u] = ball;
                }
            }
        }
        __syncwarp();
        if (lane >= first && lane < first + np) {
            mine.run = run;
            mine.chunks = nch;
        }
        if constexpr (LISTS) {
            // expand: lane (c0, p) takes chunks c0, c0 + nc, ... of particle p
            const int sh = np <= 8 ? 3 : np <= 16 ? 4 : 5;
            const int p = lane & ((1 << sh) - 1), c0 = lane >> sh, nc = 32 >> sh;
            const int vself = i0 + first + p - self;  // the particle's own window position
            int count = 0;
            for (int cb = 0; cb < nch; cb += nc) {
                const int c = cb + c0;
                unsigned m = (p < np && c < nch) ? S.mask[c][first + p] : 0u;
                if (c == (vself >> 5)) m &= ~(1u << (vself & 31));
                int sum = __popc(m);
                const int own = sum;
#pragma unroll
                for (int o = 8; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, sum, o);
                    if (o >= (1 << sh) && lane >= o) sum += t;
                }
                int at = count + sum - own;
                count += __shfl_sync(0xffffffffu, sum, p | (32 - (1 << sh)));
                while (m) {
                    const int bit = __ffs(m) - 1;
                    m &= m - 1u;
                    if (at < cap) S.hit[at][first + p] = S.code[32 * c + bit];
                    ++at;
                }
            }
            if (c0 == 0 && p < np) S.found[first + p] = count;
            __syncwarp();
        }
        first += np;
    }
    return mine;
}

// Sums of one particle over its hits.  One reciprocal mass is kept: the
// dynamic neighbours of a particle nearly always have the same mass (m_of starts
// as no mass at all, so that a mass of zero takes its reciprocal too).
struct HitSums {
    float rho = 0.0f, aii = 0.0f, m_of = NAN, inv_m = 0.0f;
    float3 jii = make_float3(0.0f, 0.0f, 0.0f);
};

// |a|^2, its roundings written out: left to the compiler, the product that stays
// outside the fused steps differed between two kernels, and with it the last bit
// of k.
__device__ __forceinline__ float length2(float3 a) {
    return __fmaf_rn(a.z, a.z, __fmaf_rn(a.x, a.x, __fmul_rn(a.y, a.y)));
}

// The pair terms of hit j at squared distance r2 (sph_kernel.py:8-61) onto the
// sums; returns J_ij, its weight and, where asked, the spline's value and the
// squared length of a dynamic neighbour's J_ij (its 1 / m is then s.inv_m).
__device__ __forceinline__ float3 hit_terms(float3 r, float r2, float mj, bool dynamic, float h, float inv_h,
                                            float spk, float ck, HitSums& s, float* weight,
                                            float* W = nullptr, float* JJ = nullptr) {
    // spiky gradient (sph_kernel.py:52-61): -k (h - |r|)^2 r / |r|
    const float rn = sqrtf(r2);
    const float rc = rn < 1e-6f ? 1e-6f : rn;
    const float t = h - rc;
    const float sg = -spk * (t * t);
    const float ir = __frcp_rn(rc);
    const float w = mj * (sg * ir);
    const float3 J = make_float3(__fmul_rn(w, r.x), __fmul_rn(w, r.y), __fmul_rn(w, r.z));
    const float Wr = cubic_Wq(rn * inv_h, ck);
    s.rho = __fmaf_rn(mj, Wr, s.rho);
    if (W) *W = Wr;
    if (dynamic) {
        if (mj != s.m_of) {
            s.m_of = mj;
            s.inv_m = __frcp_rn(mj);
        }
        const float jj = length2(J);
        s.aii = __fmaf_rn(jj, s.inv_m, s.aii);
        if (JJ) *JJ = jj;
    }
    s.jii = sub3(s.jii, J);
    *weight = w;
    return J;
}

template <int LANES>
__device__ __forceinline__ void sum_lanes(HitSums& s) {
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) {
        s.rho += __shfl_xor_sync(0xffffffffu, s.rho, o);
        s.aii += __shfl_xor_sync(0xffffffffu, s.aii, o);
        s.jii.x += __shfl_xor_sync(0xffffffffu, s.jii.x, o);
        s.jii.y += __shfl_xor_sync(0xffffffffu, s.jii.y, o);
        s.jii.z += __shfl_xor_sync(0xffffffffu, s.jii.z, o);
    }
}

// The sums that lane `from` holds.
__device__ __forceinline__ HitSums sums_of_lane(const HitSums& a, int from) {
    HitSums g;
    g.rho = __shfl_sync(0xffffffffu, a.rho, from);
    g.aii = __shfl_sync(0xffffffffu, a.aii, from);
    g.jii.x = __shfl_sync(0xffffffffu, a.jii.x, from);
    g.jii.y = __shfl_sync(0xffffffffu, a.jii.y, from);
    g.jii.z = __shfl_sync(0xffffffffu, a.jii.z, from);
    return g;
}

// The sums of particles p0 .. p0 + count - 1 (count <= 4), in the eight lanes of
// each, to the lanes p0 .. p0 + count - 1.
__device__ __forceinline__ void own_sums(const HitSums& a, int p0, int count, HitSums& s) {
    const int lane = threadIdx.x & 31;
    const HitSums g = sums_of_lane(a, ((lane - p0) * 8) & 31);
    if (lane >= p0 && lane < p0 + count) s = g;
}

// Sums in list order by N lanes, one hit each: five sums (rho, Aii, J_ii), each a
// chain of fma(first, second, sum) over the hits.  The lanes leave their hits'
// factors in shared memory and lane q < 5 of the N runs the chain of sum q.
template <int N>
struct ListOrder {
    static constexpr int kWords = 7 * N;  // m_j, W, |J|^2, 1 / m_j, J of N hits
    float sum = 0.0f;

    // Factors of zero add nothing; `group` is the mask of the N lanes, `mem` their
    // kWords words (16-byte aligned).
    __device__ __forceinline__ void add(float* mem, unsigned group, float mj, float W, float jj, float inv_m,
                                        float3 J) {
        const int sub = threadIdx.x & (N - 1);
        mem[sub] = mj;
        mem[N + sub] = W;
        mem[2 * N + sub] = jj;
        mem[3 * N + sub] = inv_m;
        mem[4 * N + sub] = J.x;
        mem[5 * N + sub] = J.y;
        mem[6 * N + sub] = J.z;
        __syncwarp(group);
        const int q = min(sub, 4);
        const float4* first = reinterpret_cast<const float4*>(mem + N * (q < 2 ? 2 * q : 2 + q));
        const float4* second = reinterpret_cast<const float4*>(mem + N * (q < 2 ? 2 * q + 1 : 0));
#pragma unroll 2
        for (int u = 0; u < N / 4; ++u) {
            const float4 a = first[u];
            float4 b = second[u];
            if (q >= 2) b = make_float4(-1.0f, -1.0f, -1.0f, -1.0f);
            sum = __fmaf_rn(a.x, b.x, sum);
            sum = __fmaf_rn(a.y, b.y, sum);
            sum = __fmaf_rn(a.z, b.z, sum);
            sum = __fmaf_rn(a.w, b.w, sum);
        }
        __syncwarp(group);
    }

    // The five sums in every lane of the N (the whole warp calls it).
    __device__ __forceinline__ void get(HitSums& s) const {
        const int g = threadIdx.x & (32 - N);
        s.rho = __shfl_sync(0xffffffffu, sum, g);
        s.aii = __shfl_sync(0xffffffffu, sum, g + 1);
        s.jii.x = __shfl_sync(0xffffffffu, sum, g + 2);
        s.jii.y = __shfl_sync(0xffffffffu, sum, g + 3);
        s.jii.z = __shfl_sync(0xffffffffu, sum, g + 4);
    }
};

}  // namespace ivp
