// k_gather.cu -- the gather passes of the two-pass methods: forward projection
// (+ calcCorrel) over the CSR and back projection (+ calcUpdate) over a CSC
// (calcFwProj/calcCorrel/calcBkProj/calcUpdate, mlem_seq/seqcsr4mlem.cpp:69-134).
//
// Both are the same walk: for every row (column) sum value * vec[index] over
// its elements and hand the sums to an epilogue.  G lanes own one row; a warp
// owns 32/G rows; the element loads are coalesced (one element per lane per
// load), and with BT > 4 frames each element's BT floats are split over FL
// lanes of four, the elements handed around by shuffles.
//
// What bounds the pass is memory latency unless enough loads are in flight, so
// every lane group runs a software pipeline of its own over its rows: while
// the gathers of one batch of D x G elements are out, the elements of the next
// batch (of this row or of the group's next row) are already loading, and the
// next row's range and the epilogue's operands load a row ahead.  The loads
// are volatile predicated instructions: written as conditional expressions,
// the compiler serialised them behind one another to save registers (40
// registers with 16 frames, two to three gathers in flight).
//
// The groups of a warp advance independently (ragged rows do not wait for one
// another).  A lane adds its elements batch by batch and a butterfly combines
// the lanes, so the sums are a fixed function of G, BT and the matrix.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "row_dev.cuh"

namespace mlem {

namespace {

constexpr int kGatherThreads = 256;

// Frame tile split: VW <= 8 floats (a 32-byte sector) per lane.
template <int BT>
struct GLanes {
    static constexpr int VW = BT < 8 ? BT : 8;
    static constexpr int FL = BT / VW;
};

// VW <= 8 values as 16-byte (or narrower) accesses: the outputs and the counts
// need no more alignment than a tile of four frames does.
template <int VW>
__device__ __forceinline__ void g_counts(const int32_t* p, int32_t (&v)[VW]) {
    if constexpr (VW == 8) {
        int32_t a[4], b[4];
        ld_counts<4>(p, a);
        ld_counts<4>(p + 4, b);
#pragma unroll
        for (int i = 0; i < 4; ++i) { v[i] = a[i]; v[4 + i] = b[i]; }
    } else {
        ld_counts<VW>(p, v);
    }
}
template <int VW>
__device__ __forceinline__ void g_load(const float* p, float (&v)[VW]) {
    if constexpr (VW == 8) {
        float a[4], b[4];
        ld_plain<4>(p, a);
        ld_plain<4>(p + 4, b);
#pragma unroll
        for (int i = 0; i < 4; ++i) { v[i] = a[i]; v[4 + i] = b[i]; }
    } else {
        ld_plain<VW>(p, v);
    }
}
template <int VW>
__device__ __forceinline__ void g_store(float* p, const float (&v)[VW]) {
    if constexpr (VW == 8) {
        st_vec<4>(p, {v[0], v[1], v[2], v[3]});
        st_vec<4>(p + 4, {v[4], v[5], v[6], v[7]});
    } else {
        st_vec<VW>(p, v);
    }
}

// Batches of D elements per lane slot, and the resident CTAs per SM the
// registers are bounded for: the gathered floats in flight per lane (D * VW)
// against the warps that hide what is left.  Measured, forward + back
// projection on 1,048,576 rows (1.9e8 elements), sorted visit, 8 lanes:
// 1 frame D 4 / 6 CTAs 546 us, 8 / 4 507, 12 / 3 513; 2 frames 4 / 5 682,
// 6 / 4 663, 8 / 4 706; 8 frames 2 / 5 1477, 3 / 4 1403; 16 frames 1 / 6
// 3268, 2 / 5 2953 (spills), 2 / 4 2076, 3 / 3 2124, 4 / 3 2213.
template <int BT>
constexpr int gather_depth() { return BT == 1 ? 8 : BT == 2 ? 6 : BT == 4 ? 4 : BT == 8 ? 3 : 2; }
constexpr int kGatherCtas = 4;

// ---------------------------------------------------------------------------
// Forward projection: rows of the CSR in visiting order; y = the sums, c =
// calcCorrel.  SKIP: only the correlation is wanted and the visit is not a
// list of rows with counts, so a row whose counts are zero in the tile's
// frames (calcCorrel 0 whatever its projection) is walked as an empty one.
// Tiles of up to four frames only: with eight or sixteen few rows are empty in
// every frame, and the counts of two rows held per lane left the gathers no
// registers (1.50 ms against 1.03 on 1,048,576 rows, 16 frames).
// ---------------------------------------------------------------------------
template <int G, int BT, bool SKIP>
struct FwOp {
    static constexpr int VW = GLanes<BT>::VW;
    SparseView csr;
    const int32_t* sino;
    float* c;
    float* y;
    uint32_t B, off;
    uint32_t gmask;
    bool writer, each;
    struct Row {
        const uint2* b;
        uint64_t n;                // elements
        uint32_t r;
        int32_t s[SKIP ? VW : 1];  // SKIP: the counts, loaded with the range
    };
    struct Pre {
        uint32_t o;                      // output row
        uint32_t r;
        int32_t s[VW < 8 ? VW : 1];      // the counts, a row ahead
    };
    __device__ __forceinline__ uint64_t count() const { return visit_count(csr); }
    __device__ __forceinline__ bool by_line() const { return csr.by_line; }
    // Row of visiting position v: loaded two rows ahead, so that its counts
    // (SKIP) can load beside its range.
    __device__ __forceinline__ uint32_t id(uint32_t v) const { return (uint32_t)row_at(csr, v); }
    __device__ __forceinline__ Row row(uint32_t v, uint32_t r) const {
        const uint2* el = reinterpret_cast<const uint2*>(csr.pairs);
        Row q;
        q.r = r;
        if (csr.vrange) {
            const ulonglong2 t = csr.vrange[v];
            q.b = el + t.x;
            q.n = t.y - t.x;
        } else {
            const uint64_t b = csr.ptr[q.r];
            q.b = el + b;
            q.n = csr.ptr[q.r + 1ull] - b;
        }
        if constexpr (SKIP) g_counts<VW>(sino + (size_t)q.r * B + off, q.s);
        return q;
    }
    // Elements of the row that the walk takes.
    __device__ __forceinline__ uint64_t take(const Row& q) const {
        if constexpr (SKIP) {
            int any = 0;
#pragma unroll
            for (int i = 0; i < VW; ++i) any |= q.s[i];
            return any ? q.n : 0;
        } else {
            return q.n;
        }
    }
    __device__ __forceinline__ Pre pre(const Row& q, uint32_t v) const {
        Pre p;
        p.o = p.r = q.r;
        if constexpr (VW < 8) {
#pragma unroll
            for (int i = 0; i < VW; ++i) p.s[i] = 0;
            if constexpr (SKIP) {
#pragma unroll
                for (int i = 0; i < VW; ++i) p.s[i] = q.s[i];
            } else if (c && writer) {
                g_counts<VW>(sino + (size_t)q.r * B + off, p.s);
            }
        }
        if (csr.out_by_visit && writer) p.o = csr.out_pos ? csr.out_pos[q.r] : v;
        return p;
    }
    __device__ __forceinline__ void finish(const Pre& p, uint32_t, const float (&acc)[VW]) const {
        if (!writer) return;
        const size_t o = (size_t)p.o * B + off;
        if (y) g_store<VW>(y + o, acc);
        if (c) {
            int32_t s[VW];
            if constexpr (VW < 8) {
#pragma unroll
                for (int i = 0; i < VW; ++i) s[i] = p.s[i];
            } else {  // eight counts held over the row cost more than this wait
                g_counts<VW>(sino + (size_t)p.r * B + off, s);
            }
            // A count of 0 has calcCorrel 0 whatever the projection, NaN included, where the
            // row has none in the tile or (each) in its frame.
            int any = 0;
#pragma unroll
            for (int i = 0; i < VW; ++i) any |= s[i];
            if constexpr (BT > VW) {  // two writers hold the tile's counts
                static_assert(BT == 2 * VW, "one exchange between the writing lanes");
                any |= __shfl_xor_sync((gmask & (0u - gmask)) * 3u, any, 1);
            }
            float t[VW];
#pragma unroll
            for (int i = 0; i < VW; ++i) t[i] = (each ? s[i] : any) ? correl_of(s[i], acc[i]) : 0.0f;
            g_store<VW>(c + o, t);
        }
    }
};

// ---------------------------------------------------------------------------
// Back projection: columns of the CSC; x *= calcUpdate's factor (norm given),
// or u = the sums.
// ---------------------------------------------------------------------------
template <int G, int BT>
struct BkOp {
    static constexpr int VW = GLanes<BT>::VW;
    SparseView csc;
    const float* norm;
    float* x;
    float* u;
    uint32_t B, off;
    uint32_t gmask;
    bool writer;
    struct Row {
        const uint2* b;
        uint64_t n;
    };
    struct Pre {
        float n;
        float x[VW < 8 ? VW : 1];
    };
    __device__ __forceinline__ uint64_t count() const { return csc.n; }
    __device__ __forceinline__ bool by_line() const { return csc.by_line; }
    __device__ __forceinline__ uint32_t id(uint32_t v) const { return v; }
    __device__ __forceinline__ Row row(uint32_t v, uint32_t) const {
        const uint2* el = reinterpret_cast<const uint2*>(csc.pairs);
        uint64_t b, e;
        span_of(csc, v, b, e);
        return Row{el + b, e - b};
    }
    __device__ __forceinline__ uint64_t take(const Row& q) const { return q.n; }
    __device__ __forceinline__ Pre pre(const Row&, uint32_t v) const {
        Pre p;
        p.n = 0.0f;
        if (norm && writer) {
            p.n = norm[v];
            if constexpr (VW < 8) g_load<VW>(x + (size_t)v * B + off, p.x);
        }
        return p;
    }
    __device__ __forceinline__ void finish(const Pre& p, uint32_t v, const float (&acc)[VW]) const {
        if (!writer) return;
        const size_t o = (size_t)v * B + off;
        if (norm) {
            float t[VW];
            if constexpr (VW < 8) {
#pragma unroll
                for (int i = 0; i < VW; ++i) t[i] = p.x[i];
            } else {
                g_load<VW>(x + o, t);
            }
#pragma unroll
            for (int i = 0; i < VW; ++i) t[i] *= update_factor(acc[i], p.n);
            g_store<VW>(x + o, t);
        } else {
            g_store<VW>(u + o, acc);
        }
    }
};

// The pipelined walk of one lane group over rows v, v + stride, ... < count.
template <int G, int BT, class Op>
__device__ __forceinline__ void gather_walk(const Op& op, const float* __restrict__ vec, uint32_t B,
                                            uint32_t off, uint32_t v, uint32_t stride,
                                            uint32_t gmask) {
    constexpr int VW = GLanes<BT>::VW, FL = GLanes<BT>::FL, EPS = G / FL;
    constexpr int D = gather_depth<BT>();
    constexpr uint32_t kBatch = D * EPS;
    const uint32_t slot = (threadIdx.x & (G - 1)) / FL;
    const uint64_t ps = l2_evict_first(), ph = l2_evict_last();
    pdl_wait();
    pdl_release();
    const uint32_t n = (uint32_t)op.count();
    if (v >= n) return;
    uint32_t rows = (n - v - 1) / stride;  // rows after the current one
    // A row is walked from the last line (or the last multiple of a load's span)
    // before it, `head` elements masked off.  At one frame the pass is bound by the
    // L1's wavefronts (79 % busy), one for each 128-byte line that an instruction
    // touches, and a third of them were a load's 64-byte pieces crossing lines:
    // plain-full forward + back projection 1.93 -> 1.82 ms, 1,048,576 rows at 2 and 4
    // frames 669 -> 635 and 912 -> 882; at 8 and 16
    // frames the gathers' own lines leave nothing to gain (loading 16 bytes a lane
    // there changed nothing either).  Batches of the row from there (at least one,
    // an empty one for an empty row) and the elements of the last.
    constexpr uint32_t kAlign = EPS < 16 ? EPS : 16;
    auto enter = [&](const typename Op::Row& q, const uint2*& p, uint32_t& nb, uint32_t& tail) {
        const uint64_t len = op.take(q);
        const uint32_t head =
            len && op.by_line() ? (uint32_t)(reinterpret_cast<uintptr_t>(q.b) >> 3) & (kAlign - 1) : 0u;
        p = q.b + (int)(slot - head);
        nb = len == 0 ? 1u : (uint32_t)((len + head + kBatch - 1) / kBatch);
        tail = (uint32_t)(len + head - (uint64_t)(nb - 1) * kBatch);
        return head;
    };
    typename Op::Row nx = op.row(v, op.id(v));
    typename Op::Pre pre = op.pre(nx, v);
    const uint2* p;
    uint32_t nb, tail;  // of the current row, from the loaded batch q on
    uint32_t head = enter(nx, p, nb, tail);
    if (rows) nx = op.row(v + stride, op.id(v + stride));
    uint32_t id2 = rows > 1 ? op.id(v + 2 * stride) : 0u;
    // element t of this lane is in the batch when t * EPS + s0 < m (unsigned)
    uint2 q[D];
    uint32_t s0 = slot - head, m0 = (nb == 1 ? tail : kBatch) - head;
#pragma unroll
    for (int t = 0; t < D; ++t) q[t] = ld_elem_if(p + t * EPS, t * EPS + s0 < m0, ps);
    float acc[VW];
#pragma unroll
    for (int i = 0; i < VW; ++i) acc[i] = 0.0f;
    for (;;) {
        // the next batch: the rest of this row, else the group's next row
        const bool last = nb == 1;
        head = 0;
        if (!last) {
            p += kBatch;
            --nb;
        } else if (rows) {
            head = enter(nx, p, nb, tail);
        } else {
            tail = 0;
        }
        const uint32_t s = slot - head, m = (nb == 1 ? tail : kBatch) - head;
        uint2 qn[D];
#pragma unroll
        for (int t = 0; t < D; ++t) qn[t] = ld_elem_if(p + t * EPS, t * EPS + s < m, ps);
        // this batch's gathers
        float xv[D][VW];
#pragma unroll
        for (int t = 0; t < D; ++t)
            ld_vec_if<VW>(vec + off + (size_t)q[t].x * B, t * EPS + s0 < m0, xv[t], ph);
        // the batch's products by pairs, then as a tree, into the running sum: a
        // chain of len / (D x G) additions instead of len / G
#pragma unroll
        for (int i = 0; i < VW; ++i) {
            float sum[(D + 1) / 2];
#pragma unroll
            for (int t = 0; t < D; t += 2) {
                sum[t / 2] = __uint_as_float(q[t].y) * xv[t][i];
                if (t + 1 < D) sum[t / 2] = fmaf(__uint_as_float(q[t + 1].y), xv[t + 1][i], sum[t / 2]);
            }
#pragma unroll
            for (int h = 1; h < (D + 1) / 2; h <<= 1)
#pragma unroll
                for (int t = 0; t + h < (D + 1) / 2; t += 2 * h) sum[t] += sum[t + h];
            acc[i] += sum[0];
        }
        if (last) {
#pragma unroll
            for (int o = FL; o < G; o <<= 1)
#pragma unroll
                for (int i = 0; i < VW; ++i) acc[i] += __shfl_xor_sync(gmask, acc[i], o);
            op.finish(pre, v, acc);
            if (rows == 0) return;
            --rows;
            v += stride;
            pre = op.pre(nx, v);
            if (rows) nx = op.row(v + stride, id2);
            if (rows > 1) id2 = op.id(v + 2 * stride);
#pragma unroll
            for (int i = 0; i < VW; ++i) acc[i] = 0.0f;
        }
        s0 = s;
        m0 = m;
#pragma unroll
        for (int t = 0; t < D; ++t) q[t] = qn[t];
    }
}

#define MLEM_GATHER_SETUP                                                                       \
    constexpr int FL = GLanes<BT>::FL, VW = GLanes<BT>::VW;                                       \
    const int lw = threadIdx.x & 31, lane = lw & (G - 1);                                       \
    const uint32_t gmask = G == 32 ? MLEM_FULL_MASK : ((1u << (G & 31)) - 1u) << (lw & ~(G - 1)); \
    const uint32_t off = f0 + (uint32_t)(lane % FL) * VW;                                       \
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;                         \
    const uint32_t stride = ((gridDim.x * blockDim.x) >> 5) * (32 / G);                         \
    const uint32_t v = warp * (32 / G) + lw / G;

template <int G, int BT, bool SKIP>
__global__ void __launch_bounds__(kGatherThreads, kGatherCtas)
    k_fwproj(SparseView csr, const float* __restrict__ x, uint32_t B, uint32_t f0,
             const int32_t* __restrict__ sino, float* __restrict__ c, float* __restrict__ y, bool each) {
    MLEM_GATHER_SETUP
    const FwOp<G, BT, SKIP> op{csr, sino, c, y, B, off, gmask, lane < FL, each};
    gather_walk<G, BT>(op, x, B, off, v, stride, gmask);
}

template <int G, int BT>
__global__ void __launch_bounds__(kGatherThreads, kGatherCtas)
    k_bkproj_csc(SparseView csc, const float* __restrict__ c, uint32_t B, uint32_t f0,
                 const float* __restrict__ norm, float* __restrict__ x, float* __restrict__ u) {
    MLEM_GATHER_SETUP
    const BkOp<G, BT> op{csc, norm, x, u, B, off, gmask, lane < FL};
    gather_walk<G, BT>(op, c, B, off, v, stride, gmask);
}
#undef MLEM_GATHER_SETUP

// The resident CTAs (the configuration's blocks per SM at most), fewer when
// the rows do not fill them.
template <int G, int BT>
int gather_grid(const LaunchCfg& cfg, uint64_t rows) {
    const int per_sm = std::min(cfg.blocks_per_sm, kGatherCtas);
    const uint64_t rows_per_cta = (uint64_t)(kGatherThreads / 32) * (32 / G);
    const uint64_t need = (rows + rows_per_cta - 1) / rows_per_cta;
    return (int)std::max<uint64_t>(1, std::min<uint64_t>(need, (uint64_t)per_sm * cfg.sm_count));
}

template <int G, int BT>
struct FwRun {
    static cudaError_t run(const LaunchCfg& cfg, cudaStream_t st, const SparseView& csr,
                           const float* x, uint32_t B, uint32_t f0, const int32_t* sino, float* c,
                           float* y) {
        const int grid = gather_grid<G, BT>(cfg, csr.n);
        if constexpr (BT <= 4)
            if (c && !y && !csr.n_dev)
                return launch_dependent(cfg.dependent && csr.n <= kDependentMost, k_fwproj<G, BT, true>, grid, kGatherThreads, 0, st, csr, x, B,
                                        f0, sino, c, y, cfg.each_frame);
        return launch_dependent(cfg.dependent && csr.n <= kDependentMost, k_fwproj<G, BT, false>, grid, kGatherThreads, 0, st, csr, x, B, f0,
                                sino, c, y, cfg.each_frame);
    }
};

template <int G, int BT>
struct BkRun {
    static cudaError_t run(const LaunchCfg& cfg, cudaStream_t st, const SparseView& csc,
                           const float* c, uint32_t B, uint32_t f0, const float* norm, float* x,
                           float* u) {
        return launch_dependent(cfg.dependent && csc.n <= kDependentMost, k_bkproj_csc<G, BT>, gather_grid<G, BT>(cfg, csc.n), kGatherThreads, 0,
                                st, csc, c, B, f0, norm, x, u);
    }
};

// Lanes per row.  A configuration's group (32 is the default) means at most that many,
// and as few as 8 lanes where rows are many, 4 where they also have few elements: the
// rows (or columns) next to one another in a warp are neighbouring rays
// (voxels), which share lines of the gathered vector, and no lane idles
// behind the end of a row.  Plain-full forward + back projection at one frame
// 2.38 ms with 32 lanes, 1.98 with 16, 1.93 with 8; 1,048,576 rows at 16
// frames 2.42, 2.13, 2.08 ms; 200,003 rows at one frame forward 70.7 us with 16 and 54.6
// with 8, back projection 84.1 and 62.6.  Four lanes: 500,000 rows of 0 to 3 elements,
// forward at one frame 50 us with 8 and 26 with 4, of 4 to 12 elements 54 and 30 (98 and 72
// at 16 frames), the back projections alike; forward passes of up to eight frames also on
// rows of up to kFourLaneRow elements: 400,000 rows of 15, 31, 44 and 60 on average 50 ->
// 29, 50 -> 37, 52 -> 42 and 63 -> 48 us at one frame, 58 -> 42, 70 -> 49, 76 -> 58 and 86
// -> 72 at four, 20,000 to 60,000 rows alike with either; at 16 frames 120,000 rows of 17
// and of 59 lose (34 -> 38, 48 -> 52).  Back projections of columns of 54 elements lose at
// one frame (95 -> 121 us), of 38 at 16 (130 -> 142).  More lanes where 8 would leave half
// of the resident warps without a row, or where the longest row would outlast four times a
// group's share of the elements.
constexpr uint64_t kFourLaneRow = 64, kFourLane = 12;
// (`four`: elements a row up to which four lanes take it.)
int gather_lanes(const SparseView& s, const LaunchCfg& cfg, uint64_t four) {
    for (int g : {4, 8, 16}) {
        if (g >= cfg.group) return cfg.group;
        if (g == 4 && s.nnz > four * s.n) continue;
        const uint64_t groups = (uint64_t)cfg.sm_count * kGatherCtas * kGatherThreads / g;
        const uint64_t used = std::min<uint64_t>(s.n, groups);
        if (used * 2 >= groups && s.max_len <= 4 * (s.nnz / used)) return g;
    }
    return 32;
}

// The widest frame tile of at most `tile` whose vector accesses the pointers
// allow: gathers of 8 floats (tiles of 8 and 16) want 32-byte rows, everything
// else min(tile, 4) floats.
int aligned_tile(int tile, const void* gathered, const void* a, const void* b, const void* c) {
    const uintptr_t rest = (uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)gathered;
    if (tile >= 8 && ((uintptr_t)gathered & 31)) tile = 4;
    while (tile > 1 && (rest & (uintptr_t)(std::min(tile, 4) * 4 - 1))) tile >>= 1;
    return tile;
}

template <template <int, int> class K, int G, typename... Args>
cudaError_t dispatch_tile(const LaunchCfg& cfg, cudaStream_t st, Args... args) {
    switch (cfg.frame_tile) {
        case 1: return K<G, 1>::run(cfg, st, args...);
        case 2: return K<G, 2>::run(cfg, st, args...);
        case 4: return K<G, 4>::run(cfg, st, args...);
        case 8: return K<G, 8>::run(cfg, st, args...);
        case 16: return K<G, 16>::run(cfg, st, args...);
        default: return cudaErrorInvalidValue;
    }
}

template <template <int, int> class K, typename... Args>
cudaError_t dispatch_lanes(uint64_t four, const SparseView& s, const LaunchCfg& cfg, cudaStream_t st,
                           Args... args) {
    switch (gather_lanes(s, cfg, four)) {
        case 4: return dispatch_tile<K, 4>(cfg, st, s, args...);
        case 8: return dispatch_tile<K, 8>(cfg, st, s, args...);
        case 16: return dispatch_tile<K, 16>(cfg, st, s, args...);
        case 32: return dispatch_tile<K, 32>(cfg, st, s, args...);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

cudaError_t fwproj(const SparseView& csr, const float* x, uint32_t B, uint32_t f0,
                   const int32_t* sino, float* c, float* y, const LaunchCfg& cfg,
                   cudaStream_t st) {
    if (!cfg_valid(cfg) || (B % cfg.frame_tile) || (f0 % cfg.frame_tile)) return cudaErrorInvalidValue;
    if (csr.n == 0) return cudaSuccess;
    LaunchCfg t = cfg;
    t.frame_tile = aligned_tile(cfg.frame_tile, x, sino, c, y);
    cudaError_t e = cudaSuccess;
    for (uint32_t f = f0; f < f0 + (uint32_t)cfg.frame_tile && e == cudaSuccess; f += (uint32_t)t.frame_tile)
        e = dispatch_lanes<FwRun>(t.frame_tile < 16 ? kFourLaneRow : kFourLane, csr, t, st, x, B, f, sino, c, y);
    return e;
}

cudaError_t bkproj_csc(const SparseView& csc, const float* c, uint32_t B, uint32_t f0,
                       const float* norm, float* x, float* u, const LaunchCfg& cfg,
                       cudaStream_t st) {
    if (!cfg_valid(cfg) || (B % cfg.frame_tile) || (f0 % cfg.frame_tile)) return cudaErrorInvalidValue;
    if (csc.n == 0) return cudaSuccess;
    LaunchCfg t = cfg;
    t.frame_tile = aligned_tile(cfg.frame_tile, c, norm ? x : u, nullptr, nullptr);
    cudaError_t e = cudaSuccess;
    for (uint32_t f = f0; f < f0 + (uint32_t)cfg.frame_tile && e == cudaSuccess; f += (uint32_t)t.frame_tile)
        e = dispatch_lanes<BkRun>(kFourLane, csc, t, st, c, B, f, norm, x, u);
    return e;
}

}  // namespace mlem
