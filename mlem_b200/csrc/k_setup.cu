// k_setup.cu -- one-time and bookkeeping kernels: prefix sums, the
// deterministic CSR -> CSC transpose, matrix validation, image statistics,
// frame-layout transposes, and the synthetic Siddon generator on the device.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "kernels.h"
#include "siddon_core.h"

namespace mlem {

namespace {

constexpr int kScanThreads = 1024;
constexpr int kScanTile = 2 * kScanThreads;

__device__ __forceinline__ uint64_t warp_incl_scan(uint64_t v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint64_t t = __shfl_up_sync(MLEM_FULL_MASK, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Block-level inclusive scan of a 2048-element tile; out[i+1] = inclusive
// sum within the tile; tile_sums[tile] = tile total.
__global__ void __launch_bounds__(kScanThreads) k_scan_tile(const uint64_t* __restrict__ in,
                                                             uint64_t* __restrict__ out,
                                                             uint64_t n,
                                                             uint64_t* __restrict__ tile_sums) {
    __shared__ uint64_t warp_tot[32];
    const uint64_t base = (uint64_t)blockIdx.x * kScanTile;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const uint64_t i0 = base + 2 * t, i1 = i0 + 1;
    const uint64_t a = i0 < n ? in[i0] : 0, b = i1 < n ? in[i1] : 0;
    uint64_t s = warp_incl_scan(a + b, lane);
    if (lane == 31) warp_tot[w] = s;
    __syncthreads();
    if (w == 0) {
        uint64_t v = warp_tot[lane];
        v = warp_incl_scan(v, lane);
        warp_tot[lane] = v;
    }
    __syncthreads();
    const uint64_t before = (w > 0 ? warp_tot[w - 1] : 0) + s - (a + b);
    if (i0 < n) out[i0 + 1] = before + a;
    if (i1 < n) out[i1 + 1] = before + a + b;
    if (t == kScanThreads - 1) tile_sums[blockIdx.x] = before + a + b;
}

// out[i+1] += offsets[tile of i]  (offsets = exclusive scan of tile sums).
__global__ void k_scan_add(uint64_t* __restrict__ out, uint64_t n,
                           const uint64_t* __restrict__ offsets) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i + 1] += offsets[i / kScanTile];
    if (i == 0) out[0] = 0;
}

inline uint64_t ceil_div(uint64_t a, uint64_t b) { return (a + b - 1) / b; }
inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// ---------------------------------------------------------------------------
// Transpose.
// ---------------------------------------------------------------------------
__global__ void k_count_cols(SparseView csr, unsigned long long* __restrict__ cnt) {
    const uint2* el = reinterpret_cast<const uint2*>(csr.pairs);
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < csr.nnz;
         k += (uint64_t)gridDim.x * blockDim.x)
        atomicAdd(cnt + el[k].x, 1ull);
}

// Warp per row: every element gets a slot in its column through an atomic
// cursor; the slot holds {row (or its key), position in row} until the
// columns are sorted.
__global__ void k_fill_csc(SparseView csr, const uint64_t* __restrict__ col_ptr,
                           unsigned long long* __restrict__ cursor, uint2* __restrict__ ce,
                           const uint32_t* __restrict__ row_key) {
    const uint2* el = reinterpret_cast<const uint2*>(csr.pairs);
    const int lane = threadIdx.x & 31;
    const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t r = warp; r < csr.n; r += nwarps) {
        const uint64_t b = csr.ptr[r], e = csr.ptr[r + 1];
        for (uint64_t k = b + lane; k < e; k += 32) {
            const uint32_t col = el[k].x;
            const uint64_t slot = col_ptr[col] + atomicAdd(cursor + col, 1ull);
            ce[slot] = make_uint2(row_key ? row_key[r] : (uint32_t)r, (uint32_t)(k - b));
        }
    }
}

__global__ void k_col_len_max(const uint64_t* __restrict__ col_ptr, uint32_t C,
                              unsigned long long* __restrict__ out) {
    unsigned long long m = 0;
    for (uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; c < C;
         c += (uint64_t)gridDim.x * blockDim.x)
        m = max(m, (unsigned long long)(col_ptr[c + 1] - col_ptr[c]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(MLEM_FULL_MASK, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

__device__ __forceinline__ uint64_t key_of(uint2 q) { return ((uint64_t)q.x << 32) | q.y; }
__device__ __forceinline__ uint2 entry_of(uint64_t k) {
    return make_uint2((uint32_t)(k >> 32), (uint32_t)k);
}

constexpr int kSortCap = 4096;  // keys per column sorted in shared memory (32 KB)

// Block per column: bitonic sort of the column's (row, position) keys.
__global__ void __launch_bounds__(256) k_sort_cols(const uint64_t* __restrict__ col_ptr,
                                                   uint32_t C, uint2* __restrict__ ce) {
    __shared__ uint64_t key[kSortCap];
    for (uint32_t col = blockIdx.x; col < C; col += gridDim.x) {
        const uint64_t b = col_ptr[col], len = col_ptr[col + 1] - b;
        if (len <= 1 || len > kSortCap) continue;  // block-uniform
        uint32_t N = 2;
        while (N < len) N <<= 1;
        for (uint32_t i = threadIdx.x; i < N; i += blockDim.x)
            key[i] = i < len ? key_of(ce[b + i]) : ~0ull;
        __syncthreads();
        for (uint32_t k = 2; k <= N; k <<= 1)
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                for (uint32_t i = threadIdx.x; i < N; i += blockDim.x) {
                    const uint32_t ixj = i ^ j;
                    if (ixj > i) {
                        const uint64_t a = key[i], c = key[ixj];
                        const bool up = (i & k) == 0;
                        if ((a > c) == up) { key[i] = c; key[ixj] = a; }
                    }
                }
                __syncthreads();
            }
        for (uint32_t i = threadIdx.x; i < len; i += blockDim.x) ce[b + i] = entry_of(key[i]);
        __syncthreads();
    }
}

__global__ void k_long_load(const uint2* __restrict__ ce, uint64_t b, uint64_t len, uint64_t N,
                            uint64_t* __restrict__ tmp) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < N;
         i += (uint64_t)gridDim.x * blockDim.x)
        tmp[i] = i < len ? key_of(ce[b + i]) : ~0ull;
}

__global__ void k_bitonic_step(uint64_t* __restrict__ tmp, uint64_t N, uint64_t j, uint64_t k) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < N;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t ixj = i ^ j;
        if (ixj > i) {
            const uint64_t a = tmp[i], c = tmp[ixj];
            const bool up = (i & k) == 0;
            if ((a > c) == up) { tmp[i] = c; tmp[ixj] = a; }
        }
    }
}

__global__ void k_long_store(const uint64_t* __restrict__ tmp, uint2* __restrict__ ce, uint64_t b,
                             uint64_t len) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < len;
         i += (uint64_t)gridDim.x * blockDim.x)
        ce[b + i] = entry_of(tmp[i]);
}

__global__ void k_list_long(const uint64_t* __restrict__ col_ptr, uint32_t C,
                            uint32_t* __restrict__ list, unsigned int* __restrict__ count) {
    for (uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; c < C;
         c += (uint64_t)gridDim.x * blockDim.x)
        if (col_ptr[c + 1] - col_ptr[c] > (uint64_t)kSortCap) list[atomicAdd(count, 1u)] = (uint32_t)c;
}

// {row (or key), position} -> {row (or key), value}.
__global__ void k_materialize(SparseView csr, uint2* __restrict__ ce,
                              const uint32_t* __restrict__ key_row) {
    const uint2* el = reinterpret_cast<const uint2*>(csr.pairs);
    for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < csr.nnz;
         s += (uint64_t)gridDim.x * blockDim.x) {
        const uint2 q = ce[s];
        const uint32_t r = key_row ? key_row[q.x] : q.x;
        ce[s] = make_uint2(q.x, el[csr.ptr[r] + q.y].y);
    }
}

__global__ void k_invert(const uint32_t* __restrict__ order, uint32_t* __restrict__ pos, uint64_t n) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
         v += (uint64_t)gridDim.x * blockDim.x)
        pos[order[v]] = (uint32_t)v;
}

__global__ void k_validate(SparseView csr, uint32_t C, unsigned int* __restrict__ bad) {
    const uint2* el = reinterpret_cast<const uint2*>(csr.pairs);
    const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t r = tid; r < csr.n; r += stride)
        if (csr.ptr[r] > csr.ptr[r + 1]) atomicOr(bad, 1u);
    if (tid == 0 && csr.ptr[csr.n] != csr.nnz) atomicOr(bad, 2u);
    for (uint64_t k = tid; k < csr.nnz; k += stride)
        if (el[k].x >= C) atomicOr(bad, 4u);
}

// ---------------------------------------------------------------------------
// Image statistics: per frame, double sum, zero count, subnormal count, in
// fixed-order trees (the same order on every call).
//
// A pass over the image that is in L2 or HBM anyway: 16 bytes per lane, and a
// lane always holds the same frames (V frames per blockIdx.y, Q = V / 4 lanes
// per voxel; with one or two frames a lane takes four or two voxels).  One
// float per lane and frame and a launch of its own for the blocks' partials
// took 53 us of an iteration at 16 frames of 1,048,576 voxels and 13 us at one
// frame of 16,384; this form takes 32 and 7 (event times, the last block
// adding the partials).  FINAL: the last block to finish adds the blocks'
// partials; otherwise k_stats_final does.
// ---------------------------------------------------------------------------
constexpr int kStatsThreads = 256;
constexpr int kStatsBlocks = 2 * kB200SMs;

struct StatsOut {
    unsigned int* slot;
    double* sums;
    unsigned long long* zeros;
    unsigned long long* subn;
};

// Adds the blocks' partials of every frame: a warp per frame, lanes in a
// fixed stride, then a fixed butterfly.  Every thread of one block calls it.
__device__ __forceinline__ void stats_finish(const double* ps, const unsigned long long* pz,
                                             const unsigned long long* pn, uint32_t nblocks,
                                             uint32_t B, uint32_t n_out, const StatsOut& o) {
    const uint64_t row = o.slot ? *o.slot : 0;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (uint32_t f = w; f < n_out; f += nw) {
        double a = 0.0;
        unsigned long long b = 0, c = 0;
#pragma unroll 4
        for (uint32_t k = lane; k < nblocks; k += 32) {
            a += __ldcg(ps + (uint64_t)k * B + f);
            b += __ldcg(pz + (uint64_t)k * B + f);
            c += __ldcg(pn + (uint64_t)k * B + f);
        }
#pragma unroll
        for (int o2 = 16; o2 > 0; o2 >>= 1) {
            a += __shfl_xor_sync(MLEM_FULL_MASK, a, o2);
            b += __shfl_xor_sync(MLEM_FULL_MASK, b, o2);
            c += __shfl_xor_sync(MLEM_FULL_MASK, c, o2);
        }
        if (lane == 0) {
            if (o.sums) o.sums[row * n_out + f] = a;
            if (o.zeros) o.zeros[row * n_out + f] = b;
            if (o.subn) o.subn[row * n_out + f] = c;
        }
    }
    __syncthreads();
    if (o.slot && threadIdx.x == 0) *o.slot = (unsigned int)row + 1;
}

template <int V, bool FINAL>
__global__ void __launch_bounds__(kStatsThreads) k_stats(const float* x, uint32_t C,
                                                         uint32_t B, double* __restrict__ ps,
                                                         unsigned long long* __restrict__ pz,
                                                         unsigned long long* __restrict__ pn,
                                                         unsigned int* __restrict__ ticket,
                                                         uint32_t n_out, StatsOut out) {
    constexpr int Q = V >= 4 ? V / 4 : 1;   // lanes per voxel
    constexpr int NS = V >= 4 ? 4 : V;      // frames per lane
    constexpr int VPL = V >= 4 ? 1 : 4 / V; // voxels per lane
    __shared__ double ss[kStatsThreads / 32][V];
    __shared__ uint32_t sz[kStatsThreads / 32][V], sn[kStatsThreads / 32][V];
    __shared__ bool s_last;
    pdl_wait();
    pdl_release();
    const uint32_t g = blockIdx.y;  // frames [g*V, g*V+V)
    double s[NS];
    uint32_t z[NS], n[NS];  // a thread sees fewer than 2^32 values
#pragma unroll
    for (int i = 0; i < NS; ++i) { s[i] = 0.0; z[i] = 0; n[i] = 0; }
    auto take = [&](float v, int i) {
        const uint32_t bits = __float_as_uint(v) & 0x7fffffffu;
        s[i] += (double)v;
        z[i] += bits == 0;
        n[i] += bits != 0 && bits < 0x00800000u;
    };
    const uint64_t items = V >= 4 ? (uint64_t)C * Q : (uint64_t)C / VPL;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < items;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t at = V >= 4 ? (i / Q) * B + (uint64_t)g * V + (i % Q) * 4 : i * 4;
        const float4 v = *reinterpret_cast<const float4*>(x + at);
        take(v.x, 0);
        take(v.y, 1 % NS);
        take(v.z, 2 % NS);
        take(v.w, 3 % NS);
    }
    if (V < 4 && blockIdx.x == 0 && threadIdx.x == 0)  // the last voxels that fill no 16 bytes
        for (uint64_t c = items * VPL; c < C; ++c) {
            take(x[c * V], 0);
            if (V == 2) take(x[c * V + 1], 1 % NS);
        }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < NS; ++i) {
#pragma unroll
        for (int o = 16; o >= Q; o >>= 1) {
            s[i] += __shfl_xor_sync(MLEM_FULL_MASK, s[i], o);
            z[i] += __shfl_xor_sync(MLEM_FULL_MASK, z[i], o);
            n[i] += __shfl_xor_sync(MLEM_FULL_MASK, n[i], o);
        }
        if (lane < Q) { ss[w][lane * NS + i] = s[i]; sz[w][lane * NS + i] = z[i]; sn[w][lane * NS + i] = n[i]; }
    }
    __syncthreads();
    if (threadIdx.x < V) {
        double a = 0.0;
        unsigned long long b = 0, c = 0;
        for (int k = 0; k < kStatsThreads / 32; ++k) {
            a += ss[k][threadIdx.x]; b += sz[k][threadIdx.x]; c += sn[k][threadIdx.x];
        }
        const uint64_t o = (uint64_t)blockIdx.x * B + (uint64_t)g * V + threadIdx.x;
        ps[o] = a; pz[o] = b; pn[o] = c;
        if (FINAL) __threadfence();
    }
    if constexpr (FINAL) {
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            s_last = atomicAdd(ticket, 1u) == gridDim.x * gridDim.y - 1;
            if (s_last) *ticket = 0u;
        }
        __syncthreads();
        if (s_last) {
            __threadfence();
            stats_finish(ps, pz, pn, gridDim.x, B, n_out, out);
        }
    }
}

__global__ void k_stats_final(const double* __restrict__ ps, const unsigned long long* __restrict__ pz,
                              const unsigned long long* __restrict__ pn, uint32_t nblocks,
                              uint32_t B, uint32_t n_out, StatsOut out) {
    pdl_wait();
    pdl_release();
    stats_finish(ps, pz, pn, nblocks, B, n_out, out);
}

__global__ void k_fill_frames(float* __restrict__ x, uint64_t total, uint32_t Bp,
                              const FrameValues vals) {
    __shared__ float v[64];
    if (threadIdx.x < 64) v[threadIdx.x] = vals.v[threadIdx.x];
    __syncthreads();
    for (uint64_t o = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; o < total;
         o += (uint64_t)gridDim.x * blockDim.x)
        x[o] = v[o % Bp];
}

__global__ void k_correl(const float* __restrict__ f, const int32_t* __restrict__ s,
                         float* __restrict__ c, uint64_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        c[i] = correl_of(s[i], f[i]);
}

// Whole-number sums of every frame's counts, and of their magnitudes, over the
// interleaved sinogram: a thread keeps to one frame (the grid's threads are a
// multiple of Bp), blocks add in shared memory, then one atomic per block and
// frame.  Integer sums, so their order does not matter.
__global__ void k_count_sums(const int32_t* __restrict__ s, uint64_t total, uint32_t Bp,
                             unsigned long long* __restrict__ sums,
                             unsigned long long* __restrict__ mags) {
    __shared__ unsigned long long ss[64], sm[64];
    for (uint32_t f = threadIdx.x; f < Bp; f += blockDim.x) ss[f] = sm[f] = 0ull;
    __syncthreads();
    const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    long long a = 0;
    unsigned long long m = 0;
#pragma unroll 4
    for (uint64_t i = t; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
        const long long v = s[i];
        a += v;
        m += (unsigned long long)(v < 0 ? -v : v);
    }
    // lanes of one frame first where a warp holds them
    const uint32_t f = (uint32_t)(t % Bp);
    if (Bp <= 16) {
        for (uint32_t o = 16; o >= Bp; o >>= 1) {
            a += __shfl_xor_sync(MLEM_FULL_MASK, a, o);
            m += __shfl_xor_sync(MLEM_FULL_MASK, m, o);
        }
        if ((threadIdx.x & 31) < Bp) {
            atomicAdd(&ss[f], (unsigned long long)a);
            atomicAdd(&sm[f], m);
        }
    } else {
        atomicAdd(&ss[f], (unsigned long long)a);
        atomicAdd(&sm[f], m);
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < Bp; k += blockDim.x) {
        if (ss[k]) atomicAdd(&sums[k], ss[k]);
        if (sm[k]) atomicAdd(&mags[k], sm[k]);
    }
}

// Frame-major [B][n] <-> interleaved [n][Bp], V frames per access on the
// interleaved side; a thread keeps to one item, so the frame-major side is
// coalesced and no thread divides an index.  Pad frames are written as 0.  Where
// the items do not fill the SMs, blockIdx.y takes a share of the frames (1,001
// voxels of 32 frames: a thread's 32 loads in turn cost 4 us).
template <typename T, int V>
struct alignas(V * sizeof(T)) FrameVec {
    T v[V];
};

template <typename T, int V>
__global__ void k_interleave(const T* __restrict__ in, T* __restrict__ out, uint64_t n, uint32_t B,
                             uint32_t Bp, const uint32_t* __restrict__ perm) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        T* to = out + (perm ? (uint64_t)perm[i] : i) * Bp;
        for (uint32_t b0 = blockIdx.y * V; b0 < Bp; b0 += gridDim.y * V) {
            FrameVec<T, V> f;
#pragma unroll
            for (int k = 0; k < V; ++k) f.v[k] = b0 + k < B ? in[(uint64_t)(b0 + k) * n + i] : T(0);
            *reinterpret_cast<FrameVec<T, V>*>(to + b0) = f;
        }
    }
}

template <typename T, int V>
__global__ void k_deinterleave(const T* __restrict__ in, T* __restrict__ out, uint64_t n,
                               uint32_t B, uint32_t Bp, const uint32_t* __restrict__ perm) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const T* from = in + (perm ? (uint64_t)perm[i] : i) * Bp;
        for (uint32_t b0 = blockIdx.y * V; b0 < B; b0 += gridDim.y * V) {
            const FrameVec<T, V> f = *reinterpret_cast<const FrameVec<T, V>*>(from + b0);
#pragma unroll
            for (int k = 0; k < V; ++k)
                if (b0 + k < B) out[(uint64_t)(b0 + k) * n + i] = f.v[k];
        }
    }
}

template <bool TO_DEVICE, typename I>
__global__ void k_permute(const float* __restrict__ in, float* __restrict__ out,
                          const uint32_t* __restrict__ perm, I n, uint32_t B, uint32_t Bd) {
    const I S = TO_DEVICE ? Bd : B, total = n * S;
    for (I j = blockIdx.x * (I)blockDim.x + threadIdx.x; j < total; j += (I)gridDim.x * blockDim.x) {
        const I i = j / S, b = j - i * S;
        const uint64_t d = (uint64_t)(perm ? perm[i] : i) * Bd + b;
        if (TO_DEVICE) out[d] = b < B ? in[(uint64_t)i * B + b] : 0.0f;
        else out[j] = in[d];
    }
}

__global__ void k_remap_columns(uint2* __restrict__ el, uint64_t nnz,
                                const uint32_t* __restrict__ perm) {
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < nnz;
         k += (uint64_t)gridDim.x * blockDim.x)
        el[k].x = perm[el[k].x];
}

// ---------------------------------------------------------------------------
// Synthetic Siddon generator (thread per row), bit-identical to the host build.
// ---------------------------------------------------------------------------
__device__ __forceinline__ siddon_geom geom_of(const SiddonSpec& s) {
    siddon_geom g;
    g.nx = s.nx; g.ny = s.ny; g.nz = s.nz; g.pad_ = 0;
    g.min_count = s.min_count; g.max_count = s.max_count;
    g.radius_scale = s.radius_scale; g.min_len = s.min_len; g.seed = s.seed;
    return g;
}

__global__ void k_siddon_counts(SiddonSpec s, uint64_t* __restrict__ counts) {
    const siddon_geom g = geom_of(s);
    for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < s.n_rows;
         r += (uint64_t)gridDim.x * blockDim.x)
        counts[r] = sd_row(&g, (uint32_t)r, nullptr);
}

__global__ void k_siddon_fill(SiddonSpec s, const uint64_t* __restrict__ row_ptr,
                              uint2* __restrict__ elems) {
    const siddon_geom g = geom_of(s);
    for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < s.n_rows;
         r += (uint64_t)gridDim.x * blockDim.x)
        sd_row(&g, (uint32_t)r, reinterpret_cast<uint32_t*>(elems + row_ptr[r]));
}

__global__ void k_project_f64(SparseView csr, const float* __restrict__ x, double* __restrict__ out) {
    const uint2* el = reinterpret_cast<const uint2*>(csr.pairs);
    for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < csr.n;
         r += (uint64_t)gridDim.x * blockDim.x) {
        double s = 0.0;
        for (uint64_t k = csr.ptr[r]; k < csr.ptr[r + 1]; ++k) {
            const uint2 q = el[k];
            s = __dadd_rn(s, __dmul_rn((double)__uint_as_float(q.y), (double)x[q.x]));
        }
        out[r] = s;
    }
}

}  // namespace

// ---------------------------------------------------------------------------
// Scan.
// ---------------------------------------------------------------------------
size_t scan_scratch_bytes(uint64_t n) {
    size_t total = 256;
    uint64_t m = n;
    while (true) {
        const uint64_t tiles = std::max<uint64_t>(1, ceil_div(m, kScanTile));
        total += align256(tiles * 8) + align256((tiles + 1) * 8);
        if (tiles <= 1) break;
        m = tiles;
    }
    return total;
}

// Three-phase scan: tile-local scans, a (recursive) scan of the tile sums,
// then every output adds the prefix of the tiles before it.
static cudaError_t scan_impl(const uint64_t* in, uint64_t* out, uint64_t n, char* scratch,
                             cudaStream_t st) {
    if (n == 0) return cudaMemsetAsync(out, 0, 8, st);
    const uint64_t tiles = ceil_div(n, kScanTile);
    uint64_t* sums = reinterpret_cast<uint64_t*>(scratch);
    uint64_t* offs = reinterpret_cast<uint64_t*>(scratch + align256(tiles * 8));
    char* next = scratch + align256(tiles * 8) + align256((tiles + 1) * 8);
    k_scan_tile<<<(unsigned)tiles, kScanThreads, 0, st>>>(in, out, n, sums);
    cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    err = tiles > 1 ? scan_impl(sums, offs, tiles, next, st) : cudaMemsetAsync(offs, 0, 8, st);
    if (err != cudaSuccess) return err;
    k_scan_add<<<(unsigned)ceil_div(n, 256), 256, 0, st>>>(out, n, offs);
    return cudaGetLastError();
}

cudaError_t exclusive_scan_u64(const uint64_t* in, uint64_t* out, uint64_t n, void* scratch,
                               size_t scratch_bytes, cudaStream_t st) {
    if (scratch_bytes < scan_scratch_bytes(n)) return cudaErrorInvalidValue;
    return scan_impl(in, out, n, static_cast<char*>(scratch), st);
}

// ---------------------------------------------------------------------------
// Transpose.
// ---------------------------------------------------------------------------
size_t transpose_scratch_bytes(uint32_t C) {
    return align256(((size_t)C + 1) * 8)            // counts / cursor
           + align256(((size_t)C + 1) * 4)          // long-column list
           + 256                                    // counters
           + scan_scratch_bytes((uint64_t)C);
}

cudaError_t invert_permutation(const uint32_t* order, uint32_t* pos, uint64_t n, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    k_invert<<<kB200SMs * 8, 256, 0, st>>>(order, pos, n);
    return cudaGetLastError();
}

cudaError_t transpose(const SparseView& csr, uint32_t C, uint64_t* col_ptr, uint2* ce,
                      void* scratch, uint32_t* max_col_len, cudaStream_t st,
                      const uint32_t* row_key, const uint32_t* key_row) {
    char* p = static_cast<char*>(scratch);
    unsigned long long* cnt = reinterpret_cast<unsigned long long*>(p);
    p += align256(((size_t)C + 1) * 8);
    uint32_t* long_list = reinterpret_cast<uint32_t*>(p);
    p += align256(((size_t)C + 1) * 4);
    unsigned long long* counters = reinterpret_cast<unsigned long long*>(p);  // [0]=max len, [1]=n long
    p += 256;
    void* scan_scratch = p;

    cudaError_t err;
#define MLEM_TRY(x) do { if ((err = (x)) != cudaSuccess) return err; } while (0)
    MLEM_TRY(cudaMemsetAsync(cnt, 0, ((size_t)C + 1) * 8, st));
    MLEM_TRY(cudaMemsetAsync(counters, 0, 256, st));
    const int grid = kB200SMs * 8;
    if (csr.nnz) {
        k_count_cols<<<grid, 256, 0, st>>>(csr, cnt);
        MLEM_TRY(cudaGetLastError());
    }
    MLEM_TRY(exclusive_scan_u64(reinterpret_cast<const uint64_t*>(cnt), col_ptr, C, scan_scratch,
                                scan_scratch_bytes(C), st));
    if (csr.nnz == 0) {
        if (max_col_len) *max_col_len = 0;
        return cudaStreamSynchronize(st);
    }
    MLEM_TRY(cudaMemsetAsync(cnt, 0, ((size_t)C + 1) * 8, st));
    k_fill_csc<<<grid, 256, 0, st>>>(csr, col_ptr, cnt, ce, row_key);
    MLEM_TRY(cudaGetLastError());
    k_col_len_max<<<kB200SMs * 2, 256, 0, st>>>(col_ptr, C, counters);
    MLEM_TRY(cudaGetLastError());
    k_list_long<<<kB200SMs * 2, 256, 0, st>>>(col_ptr, C, long_list,
                                              reinterpret_cast<unsigned int*>(counters + 1));
    MLEM_TRY(cudaGetLastError());
    k_sort_cols<<<kB200SMs * 6, 256, 0, st>>>(col_ptr, C, ce);
    MLEM_TRY(cudaGetLastError());

    unsigned long long host_counters[2] = {0, 0};
    MLEM_TRY(cudaMemcpyAsync(host_counters, counters, 16, cudaMemcpyDeviceToHost, st));
    MLEM_TRY(cudaStreamSynchronize(st));
    const uint64_t max_len = host_counters[0];
    const uint32_t n_long = (uint32_t)(host_counters[1] & 0xffffffffu);
    if (max_col_len) *max_col_len = (uint32_t)std::min<uint64_t>(max_len, 0xffffffffu);
    if (n_long) {
        // Columns too long for shared memory: global bitonic sort, one column at a time.
        std::vector<uint32_t> cols(n_long);
        std::vector<uint64_t> hptr(2);
        MLEM_TRY(cudaMemcpy(cols.data(), long_list, n_long * 4, cudaMemcpyDeviceToHost));
        uint64_t N = 2;
        while (N < max_len) N <<= 1;
        uint64_t* tmp = nullptr;
        MLEM_TRY(cudaMalloc(&tmp, N * 8));
        for (uint32_t c : cols) {
            MLEM_TRY(cudaMemcpy(hptr.data(), col_ptr + c, 16, cudaMemcpyDeviceToHost));
            const uint64_t b = hptr[0], len = hptr[1] - hptr[0];
            uint64_t n2 = 2;
            while (n2 < len) n2 <<= 1;
            const unsigned g = (unsigned)std::min<uint64_t>(ceil_div(n2, 256), kB200SMs * 8);
            k_long_load<<<g, 256, 0, st>>>(ce, b, len, n2, tmp);
            for (uint64_t k = 2; k <= n2; k <<= 1)
                for (uint64_t j = k >> 1; j > 0; j >>= 1) k_bitonic_step<<<g, 256, 0, st>>>(tmp, n2, j, k);
            k_long_store<<<g, 256, 0, st>>>(tmp, ce, b, len);
            if ((err = cudaGetLastError()) != cudaSuccess) { cudaFree(tmp); return err; }
        }
        MLEM_TRY(cudaStreamSynchronize(st));
        cudaFree(tmp);
    }
    k_materialize<<<grid, 256, 0, st>>>(csr, ce, key_row);
    MLEM_TRY(cudaGetLastError());
    return cudaStreamSynchronize(st);
#undef MLEM_TRY
}

cudaError_t validate_csr(const SparseView& csr, uint32_t C, unsigned int* bad_flag,
                         cudaStream_t st) {
    cudaError_t err = cudaMemsetAsync(bad_flag, 0, sizeof(unsigned int), st);
    if (err != cudaSuccess) return err;
    k_validate<<<kB200SMs * 4, 256, 0, st>>>(csr, C, bad_flag);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Statistics and layouts.
// ---------------------------------------------------------------------------
size_t stats_scratch_bytes(uint32_t B) { return (size_t)kStatsBlocks * B * 24 + 256; }

namespace {
template <int V>
cudaError_t run_stats(const float* x, uint32_t C, uint32_t B, uint32_t n_out, bool one_launch,
                      double* ps, unsigned long long* pz, unsigned long long* pn,
                      unsigned int* ticket, const StatsOut& out, cudaStream_t st) {
    // four loads of 16 bytes per thread, up to two blocks per SM
    const uint64_t items = ceil_div((uint64_t)C * V, 4);
    const uint32_t nb = (uint32_t)std::max<uint64_t>(
        1, std::min<uint64_t>(kStatsBlocks, ceil_div(items, (uint64_t)kStatsThreads * 4)));
    const dim3 grid(nb, B / V);
    const bool early = (uint64_t)C * B <= kDependentMost;
    if (one_launch)
        return launch_dependent(early, k_stats<V, true>, grid, kStatsThreads, 0, st, x, C, B, ps, pz, pn,
                                ticket, n_out, out);
    cudaError_t e = launch_dependent(early, k_stats<V, false>, grid, kStatsThreads, 0, st, x, C, B, ps, pz, pn,
                                     ticket, n_out, out);
    if (e != cudaSuccess) return e;
    return launch_dependent(early, k_stats_final, 1, 512, 0, st, ps, pz, pn, nb, B, n_out, out);
}
}  // namespace

cudaError_t image_stats(const float* x, uint32_t C, uint32_t B, uint32_t n_out, void* partial,
                        unsigned int* slot, double* sums, unsigned long long* zeros,
                        unsigned long long* subnormals, bool one_launch, cudaStream_t st) {
    double* ps = static_cast<double*>(partial);
    unsigned long long* pz = reinterpret_cast<unsigned long long*>(ps + (size_t)kStatsBlocks * B);
    unsigned long long* pn = pz + (size_t)kStatsBlocks * B;
    unsigned int* ticket = reinterpret_cast<unsigned int*>(pn + (size_t)kStatsBlocks * B);
    const StatsOut out{slot, sums, zeros, subnormals};
    if (B % 16 == 0) return run_stats<16>(x, C, B, n_out, one_launch, ps, pz, pn, ticket, out, st);
    if (B % 8 == 0) return run_stats<8>(x, C, B, n_out, one_launch, ps, pz, pn, ticket, out, st);
    if (B % 4 == 0) return run_stats<4>(x, C, B, n_out, one_launch, ps, pz, pn, ticket, out, st);
    if (B == 2) return run_stats<2>(x, C, B, n_out, one_launch, ps, pz, pn, ticket, out, st);
    if (B == 1) return run_stats<1>(x, C, B, n_out, one_launch, ps, pz, pn, ticket, out, st);
    return cudaErrorInvalidValue;  // padded frame counts only
}

static unsigned elementwise_grid(uint64_t n) {
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(ceil_div(n, 256), kB200SMs * 16));
}

cudaError_t count_sums(const int32_t* sino, uint64_t R, uint32_t Bp, unsigned long long* sums,
                       unsigned long long* mags, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(sums, 0, Bp * 8, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(mags, 0, Bp * 8, st);
    if (e != cudaSuccess || R == 0) return e;
    const unsigned threads = Bp == 48 ? 192 : 256;  // a multiple of every padded frame count
    const uint64_t total = R * Bp;
    const unsigned grid = (unsigned)std::min<uint64_t>(ceil_div(total, threads * 4ull), kB200SMs * 8);
    k_count_sums<<<grid, threads, 0, st>>>(sino, total, Bp, sums, mags);
    return cudaGetLastError();
}

namespace {
template <typename T, bool TO_FRAMES>
cudaError_t run_interleave(const T* in, T* out, uint64_t n, uint32_t B, uint32_t Bp,
                           const uint32_t* perm, cudaStream_t st) {
    if (n * B == 0) return cudaSuccess;
    auto go = [&](auto v) {
        constexpr int V = decltype(v)::value;
        const unsigned gx = elementwise_grid(n);
        const dim3 grid(gx, std::min<unsigned>((unsigned)ceil_div(Bp, V), std::max(1u, kB200SMs * 4u / gx)));
        if (TO_FRAMES) k_deinterleave<T, V><<<grid, 256, 0, st>>>(in, out, n, B, Bp, perm);
        else k_interleave<T, V><<<grid, 256, 0, st>>>(in, out, n, B, Bp, perm);
        return cudaGetLastError();
    };
    if (Bp % 4 == 0) return go(std::integral_constant<int, 4>{});
    if (Bp % 2 == 0) return go(std::integral_constant<int, 2>{});
    return go(std::integral_constant<int, 1>{});
}
}  // namespace

cudaError_t interleave_i32(const int32_t* in, int32_t* out, uint64_t n, uint32_t B, uint32_t Bp,
                           cudaStream_t st) {
    return run_interleave<int32_t, false>(in, out, n, B, Bp, nullptr, st);
}

cudaError_t interleave_f32(const float* in, float* out, uint64_t n, uint32_t B, uint32_t Bp,
                           const uint32_t* perm, cudaStream_t st) {
    return run_interleave<float, false>(in, out, n, B, Bp, perm, st);
}

cudaError_t deinterleave_f32(const float* in, float* out, uint64_t n, uint32_t B, uint32_t Bp,
                             const uint32_t* perm, cudaStream_t st) {
    return run_interleave<float, true>(in, out, n, B, Bp, perm, st);
}

namespace {
template <bool TO_DEVICE>
cudaError_t run_permute(const float* in, float* out, const uint32_t* perm, uint64_t n, uint32_t B,
                        uint32_t Bd, cudaStream_t st) {
    if (n * B == 0) return cudaSuccess;
    const uint64_t total = n * Bd;
    // 32-bit indexes (a 64-bit division per value costs several times the copy)
    // while the last index plus a stride fits
    if (total < 0xf0000000ull)
        k_permute<TO_DEVICE, uint32_t><<<elementwise_grid(total), 256, 0, st>>>(in, out, perm,
                                                                               (uint32_t)n, B, Bd);
    else
        k_permute<TO_DEVICE, uint64_t><<<elementwise_grid(total), 256, 0, st>>>(in, out, perm, n, B, Bd);
    return cudaGetLastError();
}
}  // namespace

cudaError_t permute_to_device(const float* in, float* out, const uint32_t* perm, uint64_t n,
                              uint32_t B, uint32_t Bd, cudaStream_t st) {
    return run_permute<true>(in, out, perm, n, B, Bd, st);
}

cudaError_t permute_to_natural(const float* in, float* out, const uint32_t* perm, uint64_t n,
                               uint32_t B, uint32_t Bd, cudaStream_t st) {
    return run_permute<false>(in, out, perm, n, B, Bd, st);
}

cudaError_t remap_columns(uint2* elems, uint64_t nnz, const uint32_t* perm, cudaStream_t st) {
    if (nnz == 0) return cudaSuccess;
    k_remap_columns<<<elementwise_grid(nnz), 256, 0, st>>>(elems, nnz, perm);
    return cudaGetLastError();
}

cudaError_t fill_frames(float* x, uint64_t n, uint32_t Bp, const FrameValues& vals, cudaStream_t st) {
    if (n * Bp == 0) return cudaSuccess;
    if (Bp > 64) return cudaErrorInvalidValue;
    k_fill_frames<<<elementwise_grid(n * Bp), 256, 0, st>>>(x, n * Bp, Bp, vals);
    return cudaGetLastError();
}

cudaError_t correl_elementwise(const float* f, const int32_t* s, float* c, uint64_t n,
                               cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    k_correl<<<elementwise_grid(n), 256, 0, st>>>(f, s, c, n);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Generator.
// ---------------------------------------------------------------------------
cudaError_t siddon_counts(const SiddonSpec& s, uint64_t* counts, cudaStream_t st) {
    if (s.n_rows == 0) return cudaSuccess;
    k_siddon_counts<<<elementwise_grid(s.n_rows), 256, 0, st>>>(s, counts);
    return cudaGetLastError();
}

cudaError_t siddon_fill(const SiddonSpec& s, const uint64_t* row_ptr, uint2* elems,
                        cudaStream_t st) {
    if (s.n_rows == 0) return cudaSuccess;
    k_siddon_fill<<<elementwise_grid(s.n_rows), 256, 0, st>>>(s, row_ptr, elems);
    return cudaGetLastError();
}

cudaError_t project_f64(const SparseView& csr, const float* x, double* out, cudaStream_t st) {
    if (csr.n == 0) return cudaSuccess;
    k_project_f64<<<elementwise_grid(csr.n), 256, 0, st>>>(csr, x, out);
    return cudaGetLastError();
}

}  // namespace mlem
