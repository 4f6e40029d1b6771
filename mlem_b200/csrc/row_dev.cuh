// row_dev.cuh -- per-row device building blocks of the row-wise kernels
// (k_project.cu) and the multi-matrix kernel (k_batch.cu).
//
// Work decomposition.  G lanes (4..32) own one row (or column); a warp owns
// 32/G rows.  A tile of BT frames of the B frames interleaved in the vectors
// is handled per pass: each element's BT floats are split over FL = BT/VW
// lanes of VW <= 4 floats, so the G lanes work on EPS = G/FL consecutive
// elements at a time (lane (slot, sub) takes element b + slot + j*EPS and
// frames [sub*VW, sub*VW + VW) of the tile).
#pragma once

#include "common.cuh"
#include "kernels.h"

namespace mlem {
namespace {

template <int BT>
struct Lanes {
    static constexpr int VW = BT < 4 ? BT : 4;  // floats per lane
    static constexpr int FL = BT / VW;          // lanes per element
};

__device__ __forceinline__ float2 ld_hot2(const float2* ptr, uint64_t pol) {
    float2 r;
    asm("ld.global.L2::cache_hint.v2.f32 {%0,%1}, [%2], %3;" : "=f"(r.x), "=f"(r.y)
        : "l"(ptr), "l"(pol));
    return r;
}

template <int VW>
__device__ __forceinline__ void ld_vec(const float* __restrict__ p, float (&v)[VW], uint64_t pol) {
    if constexpr (VW == 4) {
        const float4 t = ld_hot4(reinterpret_cast<const float4*>(p), pol);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else if constexpr (VW == 2) {
        const float2 t = ld_hot2(reinterpret_cast<const float2*>(p), pol);
        v[0] = t.x; v[1] = t.y;
    } else {
        v[0] = ld_hot(p, pol);
    }
}

template <int VW>
__device__ __forceinline__ void ld_plain(const float* __restrict__ p, float (&v)[VW]) {
    if constexpr (VW == 4) {
        const float4 t = *reinterpret_cast<const float4*>(p);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else if constexpr (VW == 2) {
        const float2 t = *reinterpret_cast<const float2*>(p);
        v[0] = t.x; v[1] = t.y;
    } else {
        v[0] = *p;
    }
}

template <int VW>
__device__ __forceinline__ void st_vec(float* __restrict__ p, const float (&v)[VW]) {
    if constexpr (VW == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else if constexpr (VW == 2) *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
    else *p = v[0];
}

template <int VW>
__device__ __forceinline__ void ld_counts(const int32_t* __restrict__ p, int32_t (&v)[VW]) {
    if constexpr (VW == 4) {
        const int4 t = *reinterpret_cast<const int4*>(p);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else if constexpr (VW == 2) {
        const int2 t = *reinterpret_cast<const int2*>(p);
        v[0] = t.x; v[1] = t.y;
    } else {
        v[0] = *p;
    }
}

// Visiting positions of a one-pass walk: *csr.n_dev for a device-built list
// (rows with counts), else csr.n.
__device__ __forceinline__ uint64_t visit_count(const SparseView& csr) {
    return csr.n_dev ? (uint64_t)__ldg(csr.n_dev) : (uint64_t)csr.n;
}

// L2 prefetch of the bytes [p, p + bytes) rounded out to 16-byte bounds (at
// most 64 KiB): a hint -- nothing completes or waits on it.  The caller keeps
// the rounded range inside the allocation (the element arrays carry a spare
// 16 bytes).
__device__ __forceinline__ void prefetch_l2(const void* p, uint64_t bytes) {
    const uint64_t a0 = reinterpret_cast<uint64_t>(p) & ~15ull;
    const uint64_t a1 = (reinterpret_cast<uint64_t>(p) + bytes + 15) & ~15ull;
    const uint32_t n = (uint32_t)(a1 - a0 < 65536 ? a1 - a0 : 65536);
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a0), "r"(n) : "memory");
}

// u[...] += w * c[...] for VW floats (one vector reduction, 4..16 bytes).
template <int VW>
__device__ __forceinline__ void red_vec(float* __restrict__ p, float w, const float (&c)[VW]) {
    if constexpr (VW == 4)
        atomicAdd(reinterpret_cast<float4*>(p), make_float4(w * c[0], w * c[1], w * c[2], w * c[3]));
    else if constexpr (VW == 2)
        atomicAdd(reinterpret_cast<float2*>(p), make_float2(w * c[0], w * c[1]));
    else
        atomicAdd(p, w * c[0]);
}

// Predicated loads: the value when `in`, else zeros.  Volatile, so that a batch of
// them goes out before anything waits: as conditional expressions the compiler
// put most of them behind one another (16 frames in chunks 2,996 -> 2,639 us per
// iteration of 1,048,576 rows with these and batches of 4, sorted 3,994 -> 3,481,
// staged 2,615 -> 2,529; 8 frames of 120,007 rows 79 -> 63 us).
// One element of the stream, past L1.
__device__ __forceinline__ uint2 ld_elem_if(const uint2* p, bool in, uint64_t pol) {
    uint2 r;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\tmov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\t"
        "@p ld.global.nc.L1::no_allocate.L2::cache_hint.v2.u32 {%0, %1}, [%2], %3;\n\t}"
        : "=r"(r.x), "=r"(r.y)
        : "l"(p), "l"(pol), "r"((uint32_t)in));
    return r;
}
// One element through L1 (a row that is read again).
__device__ __forceinline__ uint2 ld_elem_keep_if(const uint2* p, bool in, uint64_t pol) {
    uint2 r;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\tmov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\t"
        "@p ld.global.nc.L2::cache_hint.v2.u32 {%0, %1}, [%2], %3;\n\t}"
        : "=r"(r.x), "=r"(r.y)
        : "l"(p), "l"(pol), "r"((uint32_t)in));
    return r;
}
// VW floats when `in`, else zeros.  Not the .nc form: the kernel before this one
// (which it may overlap up to pdl_wait) writes the vector.
template <int VW>
__device__ __forceinline__ void ld_vec_if(const float* p, bool in, float (&v)[VW], uint64_t pol) {
    if constexpr (VW == 8) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %10, 0;\n\tmov.f32 %0, 0f00000000;\n\t"
            "mov.f32 %1, 0f00000000;\n\tmov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t"
            "mov.f32 %4, 0f00000000;\n\tmov.f32 %5, 0f00000000;\n\tmov.f32 %6, 0f00000000;\n\t"
            "mov.f32 %7, 0f00000000;\n\t"
            "@p ld.global.L2::cache_hint.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8], %9;\n\t}"
            : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]),
              "=f"(v[7])
            : "l"(p), "l"(pol), "r"((uint32_t)in));
    } else if constexpr (VW == 4) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %6, 0;\n\tmov.f32 %0, 0f00000000;\n\t"
            "mov.f32 %1, 0f00000000;\n\tmov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t"
            "@p ld.global.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;\n\t}"
            : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
            : "l"(p), "l"(pol), "r"((uint32_t)in));
    } else if constexpr (VW == 2) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\tmov.f32 %0, 0f00000000;\n\t"
            "mov.f32 %1, 0f00000000;\n\t"
            "@p ld.global.L2::cache_hint.v2.f32 {%0, %1}, [%2], %3;\n\t}"
            : "=f"(v[0]), "=f"(v[1])
            : "l"(p), "l"(pol), "r"((uint32_t)in));
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\tmov.f32 %0, 0f00000000;\n\t"
            "@p ld.global.L2::cache_hint.f32 %0, [%1], %2;\n\t}"
            : "=f"(v[0])
            : "l"(p), "l"(pol), "r"((uint32_t)in));
    }
}

// How a row's elements and gathers are loaded.  In a sorted visit neighbouring rows
// share image lines and the loads are latency-bound: batches of volatile predicated
// loads (eager).  In file order at four and more frames the rows share nothing and
// the L2 is the limit: all of a batch at once made it 12 % slower than conditional
// loads, which the compiler spaces out (1,048,576 rows: 16 frames 4,499 us eager,
// 3,864 conditional; 4 frames 1,322 and 1,127).  At one frame, and at two with a
// warp per row, eager is at least as fast in either order (two frames, 16 lanes: 992
// and 963).  Four lanes a row want conditional loads at two frames in the sorted visit
// too (1,048,576 rows 1,951 us eager, 1,858 conditional; 200,003 rows 95.2 and 93.0).
template <int G, int BT, bool SORTED>
constexpr bool eager_loads() {
    return BT == 1 || (BT == 2 && G == 32) || (SORTED && !(BT == 2 && G == 4));
}

// Elements a lane loads before it gathers (memory-level parallelism).  A
// full-warp group takes 8 (a 150-250-element row is one batch) at one and two
// frames and of conditional loads; with four floats per lane, and in narrower
// groups, 4 eager ones keep the registers, and so the occupancy.  Kernels whose
// rows want another depth at four frames pass their own.
template <int G, int BT, bool EAGER>
constexpr int batch_depth() { return G == 32 && (BT < 4 || !EAGER) ? 8 : 4; }

// acc[0..VW) = sum over the row's elements of value * vec[col*B + off + ...].
// Each batch issues all of its (predicated) element loads, then all of its
// gathers, so a row costs about two memory latencies per batch instead of
// two per element.  When `keep` is non-null and the whole row fits in one
// batch, the lane's elements are left in keep[] (fused kernel) and true is
// returned.
template <int G, int BT, bool KEEP, bool EAGER, int kBatch>
__device__ __forceinline__ bool row_dot(const uint2* __restrict__ el, uint64_t b, uint64_t e,
                                        int lane, const float* __restrict__ vec, uint32_t B,
                                        uint32_t off, float (&acc)[Lanes<BT>::VW], uint64_t ps,
                                        uint64_t ph, uint2* keep = nullptr) {
    constexpr int VW = Lanes<BT>::VW, FL = Lanes<BT>::FL, EPS = G / FL;
    const float* base = vec + off;
#pragma unroll
    for (int i = 0; i < VW; ++i) acc[i] = 0.0f;
    const bool one_batch = e - b <= (uint64_t)kBatch * EPS;
    // Elements go through L1 when the fused kernel may re-read them for its
    // scatter (rows longer than one batch).  A full warp at one frame holds 256
    // elements per batch, so the rows of a typical matrix stay in registers
    // and their elements skip L1, leaving its lines to the image gathers
    // (plain-full, chunked walk: 2.450 vs 2.471 ms; at 16 frames, where rows
    // span several batches, skipping L1 cost 13 %).
    constexpr bool kL1 = KEEP && !(G == 32 && BT == 1);
    for (uint64_t k0 = b + lane / FL; k0 < e; k0 += (uint64_t)kBatch * EPS) {
        uint2 q[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const uint64_t k = k0 + (uint64_t)u * EPS;
            if constexpr (EAGER) {
                q[u] = kL1 ? ld_elem_keep_if(el + k, k < e, ps) : ld_elem_if(el + k, k < e, ps);
            } else {
                q[u] = make_uint2(0u, 0u);  // value 0: contributes nothing
                if (k < e) q[u] = kL1 ? ld_keep2(el + k, ps) : ld_stream2(el + k, ps);
            }
        }
        float xv[kBatch][VW];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const bool in = k0 + (uint64_t)u * EPS < e;
            if constexpr (EAGER) {
                ld_vec_if<VW>(base + (size_t)q[u].x * B, in, xv[u], ph);
            } else if (in) {
                ld_vec<VW>(base + (size_t)q[u].x * B, xv[u], ph);
            } else {
#pragma unroll
                for (int i = 0; i < VW; ++i) xv[u][i] = 0.0f;
            }
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const float v = __uint_as_float(q[u].y);
#pragma unroll
            for (int i = 0; i < VW; ++i) acc[i] = fmaf(v, xv[u][i], acc[i]);
        }
        if (keep && one_batch) {
#pragma unroll
            for (int u = 0; u < kBatch; ++u) keep[u] = q[u];
        }
    }
    return one_batch;
}

// Sum over the element slots of the group: afterwards every lane holds the
// row totals of its frames.  Every lane of the warp must call it.
template <int G, int BT>
__device__ __forceinline__ void slot_allreduce(float (&acc)[Lanes<BT>::VW]) {
    constexpr int VW = Lanes<BT>::VW, FL = Lanes<BT>::FL;
#pragma unroll
    for (int o = FL; o < G; o <<= 1)
#pragma unroll
        for (int i = 0; i < VW; ++i) acc[i] += __shfl_xor_sync(MLEM_FULL_MASK, acc[i], o);
}


// One pass per row over rows [r_begin, r_end): forward projection, calcCorrel
// and the scatter of the row into the update vector.  `warp` / `nwarps`
// number the warps that share the range (grid-wide or block-wide).
// SORTED: the view carries the sorted visiting order with its row ranges
// (csr.vrange); otherwise rows are visited in file order (csr.order null).
// A compile-time choice: the file-order loop measured 2.49 vs 3.15 ms on the
// plain-full matrix when the sorted path was a runtime branch inside it.
// kBatch: elements a lane holds at once.
template <int G, int BT, bool SORTED, int kBatch = batch_depth<G, BT, eager_loads<G, BT, SORTED>()>()>
__device__ __forceinline__ void fused_row_range(const SparseView& csr, const float* __restrict__ x,
                                                uint32_t B, uint32_t f0,
                                                const int32_t* __restrict__ sino,
                                                float* __restrict__ u, uint64_t r_begin,
                                                uint64_t r_end, uint64_t warp, uint64_t nwarps) {
    // [r_begin, r_end) are visiting positions (rows in csr.order when set)
    constexpr int RPW = 32 / G;
    constexpr int VW = Lanes<BT>::VW, FL = Lanes<BT>::FL, EPS = G / FL;
    const int lw = threadIdx.x & 31;
    const int lane = lw & (G - 1);
    const int sub = lane % FL;
    const uint64_t ps = l2_evict_first(), ph = l2_evict_last();
    const uint2* el = reinterpret_cast<const uint2*>(csr.pairs);
    for (uint64_t base = r_begin + warp * RPW; base < r_end; base += nwarps * RPW) {
        const uint64_t v = base + lw / G;  // visiting position
        const bool active = v < r_end;
        uint64_t r = 0, b = 0, e = 0;
        if constexpr (SORTED) {
            if (active) {
                const ulonglong2 q = csr.vrange[v];
                r = csr.order[v];
                b = q.x;
                e = q.y;
            }
            // the row this lane group takes next: its range load goes out beside
            // this row's, and its elements are prefetched into L2 while this row
            // is worked on (in file order the next row of a grid-stride walk is
            // thousands of rows away and a prefetch only adds L2 requests)
            const uint64_t nv = v + nwarps * RPW;
            if (lane == 0 && nv < r_end) {
                const ulonglong2 nq = csr.vrange[nv];
                if (nq.y > nq.x) prefetch_l2(el + nq.x, (nq.y - nq.x) * 8);
            }
        } else {
            r = v;
            if (active) {
                b = csr.ptr[r];
                e = csr.ptr[r + 1];
            }
        }
        if (e - b > csr.long_len) e = b;  // left to the long-row kernels
        float acc[VW];
        uint2 kept[kBatch];
        const bool in_regs =
            row_dot<G, BT, true, eager_loads<G, BT, SORTED>(), kBatch>(el, b, e, lane, x, B,
                                                                    f0 + sub * VW, acc, ps, ph, kept);
        slot_allreduce<G, BT>(acc);
        if (!active) continue;
        const uint64_t idx = r * B + f0 + sub * VW;
        int32_t s[VW];
        ld_counts<VW>(sino + idx, s);
        float cv[VW];
        bool any = false;
#pragma unroll
        for (int i = 0; i < VW; ++i) {
            cv[i] = correl_of(s[i], acc[i]);
            any |= (cv[i] != 0.0f);
        }
        if (!any) continue;
        float* ub = u + f0 + sub * VW;
        if (in_regs) {
            // the whole row is still in registers: scatter from there
#pragma unroll
            for (int q = 0; q < kBatch; ++q)
                if (b + lane / FL + (uint64_t)q * EPS < e)
                    red_vec<VW>(ub + (size_t)kept[q].x * B, __uint_as_float(kept[q].y), cv);
        } else {
            for (uint64_t k = b + lane / FL; k < e; k += EPS) {
                const uint2 q = ld_keep2(el + k, ps);
                red_vec<VW>(ub + (size_t)q.x * B, __uint_as_float(q.y), cv);
            }
        }
    }
}

// One pass over the sorted visiting positions v, v + S, ... < end at one frame, a
// warp per row: forward sum, calcCorrel, scatter.  What the whole machine waits
// for is the L2's float reductions (plain-full: 299 M sector reductions, 1.63 ms
// at the measured rate); the rest of a row is a chain of memory round trips
// (range and row, elements, gathers, count), which this walk takes off the path:
// while row k's image values are gathered, row k+1's elements load into
// registers, its range and index loaded before that.  Loads are volatile and
// predicated, so a batch of 256 elements goes out at once; the elements stay in
// registers for the scatter.  For matrices of short rows (SparseView::short_rows):
// beyond 256 elements a row's rest is read one load at a time, which on rows of
// 1,500 elements cost a third (6.2e9 elements: 44 ms against 33 for
// fused_row_range) and behind 1 % of rows of 2,000 a fifth, and row lengths have
// 32 bits.  Against
// fused_row_range (B200): plain-full 2.11 -> 2.08 ms, 1,048,576 rows 543 -> 532
// us, eight subsets of 500,003 rows 282 -> 248 us in chunks, 253 -> 247 in grid
// stride, 65,536 rows 22.6 -> 19.4 and 21.0 -> 18.3 us.  The adjoint kernels'
// form of it (counts two rows ahead, to skip rows) was no faster than theirs.
__device__ __forceinline__ void one_pass_rows(const SparseView& csr, const float* __restrict__ x,
                                              const int32_t* __restrict__ sino,
                                              float* __restrict__ u, uint32_t v, uint32_t end,
                                              uint32_t S) {
    constexpr int D = 8;
    constexpr uint32_t kBatch = D * 32;
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t ps = l2_evict_first(), ph = l2_evict_last();
    if (v >= end) return;
    struct Row {
        const uint2* b;
        uint32_t n, r;
    };
    auto row = [&](uint32_t k) {
        const ulonglong2 t = csr.vrange[k];
        const uint64_t n = t.y - t.x;
        return Row{reinterpret_cast<const uint2*>(csr.pairs) + t.x + lane,
                   n > csr.long_len ? 0u : (uint32_t)n, csr.order[k]};
    };
    uint32_t left = (end - v - 1) / S;  // rows after the current one
    Row cur = row(v), nx = cur;
    int32_t s = sino[cur.r];
    if (left) nx = row(v + S);
    uint2 q[D];
    int m = (int)min(cur.n, kBatch) - (int)lane;
#pragma unroll
    for (int t = 0; t < D; ++t) q[t] = ld_elem_if(cur.b + t * 32, t * 32 < m, ps);
    for (;;) {
        const int mn = left ? (int)min(nx.n, kBatch) - (int)lane : 0;
        uint2 qn[D];
#pragma unroll
        for (int t = 0; t < D; ++t) qn[t] = ld_elem_if(nx.b + t * 32, t * 32 < mn, ps);
        const int32_t sn = sino[nx.r];
        float xv[D][1];
#pragma unroll
        for (int t = 0; t < D; ++t) ld_vec_if<1>(x + q[t].x, t * 32 < m, xv[t], ph);
        float acc = 0.0f;
#pragma unroll
        for (int t = 0; t < D; ++t) acc = fmaf(__uint_as_float(q[t].y), xv[t][0], acc);
        for (uint32_t k = kBatch; k + lane < cur.n; k += 32) {
            const uint2 e = ld_keep2(cur.b + k, ps);
            acc = fmaf(__uint_as_float(e.y), ld_hot(x + e.x, ph), acc);
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) acc += __shfl_xor_sync(MLEM_FULL_MASK, acc, o);
        const float c = correl_of(s, acc);
        if (c != 0.0f) {
#pragma unroll
            for (int t = 0; t < D; ++t)
                if (t * 32 < m) atomicAdd(u + q[t].x, __uint_as_float(q[t].y) * c);
            for (uint32_t k = kBatch; k + lane < cur.n; k += 32) {
                const uint2 e = ld_keep2(cur.b + k, ps);
                atomicAdd(u + e.x, __uint_as_float(e.y) * c);
            }
        }
        if (left == 0) return;
        --left;
        v += S;
        cur = nx;
        s = sn;
        m = mn;
        if (left) nx = row(v + S);
#pragma unroll
        for (int t = 0; t < D; ++t) q[t] = qn[t];
    }
}

}  // namespace
}  // namespace mlem
