// Row-segment stream kernels (layout in cb_rowseg.hpp) and the balanced
// schedule:
//   * cb_rowseg_kernel       y = A x, one right-hand side (below);
//   * cb_rowseg_mrhs_kernel  Y = A X, G lanes per entry, several right-hand
//                            sides (rs_mrhs_segment);
//   * cb_rowseg_gv_kernel    the fused adjoint: A^T G and the value gradient;
//   * cb_rowseg_batch_kernel every matrix of a batch in one launch;
//   * cb_balanced_kernel     plans built with row_owned = 0: the reference's
//                            block order, atomics into y;
//   * the balanced stream's value refresh after cbspmv_set_values.
//
// One right-hand side: one CTA of 32 warps per SM.  Per chunk a lane
//   * holds the NEXT chunk's words and values in registers, loaded with
//     coalesced 16-byte loads that do not allocate in L1 (L1 is left to the
//     x gathers) and are marked evict-first in L2 (x stays in L2),
//   * gathers x for its kRsK entries, all loads in flight at once: from the
//     CTA's window of x in shared memory (staged at the start) when the
//     entry's word says so, else from global memory,
//   * counts the row starts of the lanes before it (one ballot per entry),
//     which gives the ordinal of the row it starts in,
//   * adds its entries along its rows in registers; a row that starts and
//     ends inside the lane is stored at once,
//   * joins the rows that run across lanes with one segmented inclusive scan
//     (reset at lanes holding a row start, its steps' lanes read off the
//     ballots, ended once no row reaches further), carrying the chunk's last
//     row into the next chunk.
// Bound by L1 (76% of its rate) and issue (63%) on large power-law matrices,
// by issue (63%) on stencils, and by the latency of a warp's few chunks in a
// row on mid-sized matrices (issue 52%, L1 49%).  Row starts and the scan's
// flags from ballots instead of shuffles, with windows no longer than they
// pay, took 13% off, n = 1048576, mean 16, FP64 and n = 300007, FP32.
// The products of one row are added in entry order within a lane and in lane
// order across lanes, fixed by the layout: results are bitwise reproducible
// (the balanced schedule's atomics excepted).  The reference adds each entry
// into its row with an atomic (cb-spmv-dcu.hpp:423-426); the sums here are
// the same rows' sums.
#include <cuda/atomic>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "cb_device.cuh"
#include "cb_kernels.hpp"
#include "cb_rowseg.hpp"

namespace cb {
namespace {

using dev::kFull;

template <typename T> struct RsVec;
template <> struct RsVec<double> { using V = double2; static constexpr int n = 2; };
template <> struct RsVec<float> { using V = float4; static constexpr int n = 4; };

// Words and values of the stream.  The launch before may have written the
// values (cbspmv_set_values), so the loads are coherent ones (see
// launch_behind), and volatile, which keeps them after behind_wait's wait.
__device__ __forceinline__ uint4 ld_stream(const uint4 *p, uint64_t pol) {
    uint4 r;
    asm volatile("ld.global.L1::no_allocate.L2::cache_hint.v4.u32 {%0,%1,%2,%3}, [%4], %5;"
        : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
        : "l"(p), "l"(pol));
    return r;
}
__device__ __forceinline__ double2 ld_stream(const double2 *p, uint64_t pol) {
    double2 r;
    asm volatile("ld.global.L1::no_allocate.L2::cache_hint.v2.f64 {%0,%1}, [%2], %3;"
        : "=d"(r.x), "=d"(r.y)
        : "l"(p), "l"(pol));
    return r;
}
__device__ __forceinline__ float4 ld_stream(const float4 *p, uint64_t pol) {
    float4 r;
    asm volatile("ld.global.L1::no_allocate.L2::cache_hint.v4.f32 {%0,%1,%2,%3}, [%4], %5;"
        : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w)
        : "l"(p), "l"(pol));
    return r;
}
// Values of x, which the launch before may have written: the same loads, with
// no hint.
__device__ __forceinline__ double ld_x(const double *p) {
    double r;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(r) : "l"(p));
    return r;
}
__device__ __forceinline__ float ld_x(const float *p) {
    float r;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(r) : "l"(p));
    return r;
}
__device__ __forceinline__ double2 ld_x(const double2 *p) {
    double2 r;
    asm volatile("ld.global.v2.f64 {%0,%1}, [%2];" : "=d"(r.x), "=d"(r.y) : "l"(p));
    return r;
}
__device__ __forceinline__ float4 ld_x(const float4 *p) {
    float4 r;
    asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];"
                 : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w)
                 : "l"(p));
    return r;
}
__device__ __forceinline__ void unpack(const double2 &v, double *o) {
    o[0] = v.x;
    o[1] = v.y;
}
__device__ __forceinline__ void unpack(const float4 &v, float *o) {
    o[0] = v.x;
    o[1] = v.y;
    o[2] = v.z;
    o[3] = v.w;
}

// A row that crosses one segment boundary (a span of two segments; kRsPair in
// its id): the two parts meet in the span's exchange word, which holds kEmpty
// between launches.  Whoever exchanges its part in second gets the first part
// back, has the row's sum (two addends: the same in either order) and empties
// the word.  The value travels in the atomic, so no fence is needed: the
// acquire-release counter below made each warp wait for all its stores of y
// (8-10% of the warps' cycles on power-law matrices; device time without it
// -8% at n = 300007, FP32, -30% on a 256 x 256 grid, -14% for a batch of 32).
// A part with kEmpty's bits, a NaN, goes in as the ordinary NaN.  Returns true
// with v the sum.
template <typename T> struct RsBits;
template <> struct RsBits<float> {
    using U = unsigned int;
    static constexpr U kEmpty = 0xffffdeadu, kNan = 0x7fffffffu;
    static __device__ __forceinline__ U to(float v) { return __float_as_uint(v); }
    static __device__ __forceinline__ float from(U u) { return __uint_as_float(u); }
};
template <> struct RsBits<double> {
    using U = unsigned long long;
    static constexpr U kEmpty = 0xffffdeadffffdeadull, kNan = 0x7fffffffffffffffull;
    static __device__ __forceinline__ U to(double v) {
        return (U)__double_as_longlong(v);
    }
    static __device__ __forceinline__ double from(U u) {
        return __longlong_as_double((long long)u);
    }
};
template <typename T>
__device__ __forceinline__ bool rs_meet(void *xch, int64_t i, T &v) {
    using B = RsBits<T>;
    typename B::U *w = static_cast<typename B::U *>(xch) + i;
    typename B::U mine = B::to(v);
    if (mine == B::kEmpty) mine = B::kNan;
    const typename B::U old = atomicExch(w, mine);
    if (old == B::kEmpty) return false;
    *w = B::kEmpty;
    v += B::from(old);
    return true;
}

// A row over more segments: this segment's part into its slot; the last
// part to arrive (acquire-release counter) adds the slots in segment order,
// stores y and resets the counter.  Called by one lane.
template <typename T>
__device__ __forceinline__ void rs_arrive(const RowSegDev &rs, T *__restrict__ y, int span,
                                          T v, int slot, int64_t row) {
    if (span & kRsPair) {
        if (rs_meet(rs.xch, (int64_t)(span & ~kRsPair) * kRsSlotValues, v)) y[row] = v;
        return;
    }
    T *part = static_cast<T *>(rs.part);
    part[slot] = v;
    cuda::atomic_ref<int32_t, cuda::thread_scope_device> ctr(rs.counters[span]);
    const int old = ctr.fetch_add(1, cuda::memory_order_acq_rel);
    const int4 sp = __ldg(&rs.spans[span]);
    if (old + 1 == sp.y - sp.x + 1) {
        T tot = __ldcg(&part[2 * sp.x + 1]);
        for (int s = sp.x + 1; s <= sp.y; ++s) tot += __ldcg(&part[2 * s]);
        y[rs.rowmap ? __ldg(&rs.rowmap[sp.z]) : sp.z] = tot;
        ctr.store(0, cuda::memory_order_relaxed);
    }
}

// src[0 .. len) into shared memory by asynchronous copies of the whole CTA:
// all of a thread's copies are in flight at once and take no registers, so
// the staging costs one memory latency and its bytes (a load-then-store loop
// waited for memory once per few values).  16-byte copies when src is aligned
// to them, else value by value.  stage_wait before the CTA's barrier.
template <typename T>
__device__ __forceinline__ void stage_window(T *dst, const T *src, int len, int tid) {
    constexpr int NV = 16 / sizeof(T);
    int i0 = 0;
    if (reinterpret_cast<uintptr_t>(src) % 16 == 0) {
        for (int i = tid; i < len / NV; i += kRsWarps * 32)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                             dev::smem_u32(dst + i * NV)),
                         "l"(src + i * NV)
                         : "memory");
        i0 = len / NV * NV;
    }
    for (int i = i0 + tid; i < len; i += kRsWarps * 32)
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dev::smem_u32(dst + i)),
                     "l"(src + i), "n"((int)sizeof(T))
                     : "memory");
}
__device__ __forceinline__ void stage_wait() {
    asm volatile("cp.async.wait_all;" ::: "memory");
}

template <typename T, bool UNIT, bool MAP>
__global__ void __launch_bounds__(kRsWarps * 32, 1)
    cb_rowseg_kernel(const RowSegDev rs, const T *x, T *__restrict__ y) {
    dev::behind_wait();
    using V = typename RsVec<T>::V;
    constexpr int K = kRsK, NV = RsVec<T>::n;
    constexpr int64_t CB = 32 * K * (4 + (UNIT ? 0 : (int64_t)sizeof(T)));
    extern __shared__ __align__(16) unsigned char rs_smem[];
    T *xs = reinterpret_cast<T *>(rs_smem);  // x[wb .. wb + wl)
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int G = gridDim.x, b = blockIdx.x;
    const int wb = __ldg(&rs.wbase[b]);
    const int wl = __ldg(&rs.wlen[b]);
    const int sb0 = (int)((int64_t)b * rs.nseg / G);
    const int sb1 = (int)((int64_t)(b + 1) * rs.nseg / G);
    int s = sb0 + wib;
    const int M = rs.M, nch = rs.nch, nord = rs.nord;
    const uint64_t pol = dev::policy_evict_first();
    uint4 nw[K / 4];
    V nv[K / NV];
    auto load = [&](int c) {
        const uint4 *gw = reinterpret_cast<const uint4 *>(rs.chunks + (int64_t)c * CB);
        const V *gv = reinterpret_cast<const V *>(rs.chunks + (int64_t)c * CB + 32 * K * 4);
#pragma unroll
        for (int q = 0; q < K / 4; ++q) nw[q] = ld_stream(gw + q * 32 + lane, pol);
        if (!UNIT) {
#pragma unroll
            for (int q = 0; q < K / NV; ++q) nv[q] = ld_stream(gv + q * 32 + lane, pol);
        }
    };
    auto rid = [&](int32_t o) { return MAP ? __ldg(&rs.rowmap[o]) : o; };
    const uint32_t below = (1u << lane) - 1u;
    int c = s * M;
    if (s < sb1) load(c);  // in flight while the window is staged
    stage_window(xs, x + wb, wl, threadIdx.x);
    for (int i = (blockIdx.x * kRsWarps + wib) * 32 + lane; i < rs.nempty;
         i += gridDim.x * kRsWarps * 32)
        y[__ldg(&rs.empty[i])] = T(0);
    stage_wait();
    __syncthreads();
    if (s >= sb1) return;
    while (true) {
        // segment s: meta = {ordinal running before its first entry, its first
        // entry starts a row, head span, tail span}
        const int4 meta = __ldg(&rs.meta[s]);
        const int32_t first = meta.x;
        int32_t ord0 = meta.x;
        T carry = T(0);
        const int cend = min(nch, c + M);
        for (; c < cend; ++c) {
            uint32_t w[K];
            T v[K], xv[K];
#pragma unroll
            for (int q = 0; q < K / 4; ++q) {
                w[4 * q] = nw[q].x;
                w[4 * q + 1] = nw[q].y;
                w[4 * q + 2] = nw[q].z;
                w[4 * q + 3] = nw[q].w;
            }
            if (UNIT) {
#pragma unroll
                for (int j = 0; j < K; ++j) v[j] = T(1);
            } else {
#pragma unroll
                for (int q = 0; q < K / NV; ++q) unpack(nv[q], v + q * NV);
            }
            {  // the next chunk of this segment, or the first of the warp's next
                int cn = c + 1;
                if (cn >= cend) {
                    const int sn = s + kRsWarps;
                    cn = sn < sb1 ? sn * M : -1;
                }
                if (cn >= 0) load(cn);
            }
#pragma unroll
            for (int j = 0; j < K; ++j) {
                const uint32_t col = w[j] & kRsColMask;
                xv[j] = (w[j] & kRsWin) ? xs[(int)col - wb] : ld_x(x + col);
            }
            // row starts of the lanes before this one, and the lanes that hold
            // one, from one ballot per entry
            uint32_t heads = 0;
            int32_t ordS = ord0;  // the row this lane starts in
#pragma unroll
            for (int j = 0; j < K; ++j) {
                const uint32_t bal = __ballot_sync(kFull, (w[j] >> 31) != 0);
                heads |= bal;
                ordS += __popc(bal & below);
            }
            int32_t ord = ordS;
            T run = T(0), head = T(0);
            bool seen = false;  // a row starts in this lane
#pragma unroll
            for (int j = 0; j < K; ++j) {
                const bool f = (w[j] >> 31) != 0;
                if (f && seen) y[rid(ord)] = run;  // a row whole inside the lane
                head = (f && !seen) ? run : head;
                seen = seen || f;
                ord += f ? 1 : 0;
                run = fma(v[j], xv[j], f ? T(0) : run);
            }
            // rows across lanes: inclusive scan of run, reset at lanes that
            // hold a row start; lane 0 continues the previous chunk's row
            T sc = run;
            if (lane == 0 && !seen) sc += carry;
            // bit l of cont: the d lanes up to l all go on from the lane before
            uint32_t cont = ~heads & ~1u;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                if (cont == 0) break;  // no row reaches d lanes further
                const T su = __shfl_up_sync(kFull, sc, d);
                if ((cont >> lane) & 1u) sc += su;
                cont &= cont << d;
            }
            T cin = __shfl_up_sync(kFull, sc, 1);
            if (lane == 0) cin = carry;
            if (seen) {  // the row this lane started in ends here
                const T val = cin + head;
                if (ordS == first && meta.z >= 0)
                    rs_arrive<T>(rs, y, meta.z, val, 2 * s, rid(ordS));
                else if (!(ordS == first && meta.y) && ordS < nord)
                    y[rid(ordS)] = val;
            }
            carry = __shfl_sync(kFull, sc, 31);
            ord0 = __shfl_sync(kFull, ord, 31);
        }
        // the segment's last row: a span's part, or whole here
        if (lane == 0) {
            if (ord0 == first && meta.z >= 0)
                rs_arrive<T>(rs, y, meta.z, carry, 2 * s, rid(ord0));
            else if (meta.w >= 0)
                rs_arrive<T>(rs, y, meta.w, carry, 2 * s + 1, rid(ord0));
            else if (ord0 < nord && !(ord0 == first && meta.y))
                y[rid(ord0)] = carry;
        }
        s += kRsWarps;
        if (s >= sb1) break;
        c = s * M;
    }
}

// Several right-hand sides over the same stream: G lanes per entry, lane q
// of a group holding the V = 16 / sizeof(T) right-hand sides q*V .. q*V+V-1
// of its rows; P = 32 / G groups per warp, group p taking the 4G consecutive
// entries 4Gp .. 4Gp+4G-1 of each chunk (the entries lanes Gp .. Gp+G-1 take
// in the one-vector kernel).  A group walks its entries in steps of 4: the
// step's words and values are loaded by every lane of the group (one 16-byte
// access, broadcast), its four x rows gathered (one 16-byte load per lane
// and entry), then added along the rows in registers.  Row starts are
// counted per group and scanned over the groups; one segmented scan over the
// groups joins rows across groups.  No x window (the window holds single
// vectors).
constexpr int kRsMaxRhs = kRsSlotValues;  // right-hand sides per launch (slots hold this many)

// One matrix as the several-right-hand-side segment code reads it.
template <typename T>
struct RsMat {
    const uint8_t *chunks;
    const int32_t *rowmap;  // NULL: ordinals are rows
    const T *x;
    T *y;
    int64_t ldx, ldy;
    int32_t nrhs, nord;
    int32_t xvec, yvec;     // 16-byte loads of x rows / stores of y rows allowed
};

// The spans of one segmentation: per span {first segment, last segment,
// ordinal, -}, an arrival counter each (zero between launches), kRsMaxRhs
// values per slot and two slots per segment.
template <typename T>
struct RsSpans {
    const int4 *spans;
    int32_t *counters;
    T *part;
    void *xch;  // exchange words, kRsMaxRhs per span
};

// The value gradient of a transposed stream (the fused adjoint): per stream
// entry e of row j (a column of A) gathering row i of G, gv[e] = sum over the
// right-hand sides of G[i, :] . xo[j, :] (written, or added when accum).
template <typename T>
struct RsGV {
    const T *xo;
    int64_t ldo;
    int32_t xovec;  // 16-byte loads of xo rows allowed
    int32_t accum;
    T *gv;
};

// Chunks [cb, ce) of matrix A as segment s, meta = {ordinal running before
// chunk cb, chunk cb starts a row, head span, tail span}.  Called by a whole
// warp.  GV: also the value gradient of every entry (gvp).
template <typename T, int G, bool UNIT, bool GV = false>
__device__ __forceinline__ void rs_mrhs_segment(const RsMat<T> &A, int cb, int ce, int4 meta,
                                                int s, const RsSpans<T> &S, int lane,
                                                uint64_t pol, const RsGV<T> *gvp = nullptr) {
    using VT = typename RsVec<T>::V;
    constexpr int V = RsVec<T>::n, P = 32 / G, NV = RsVec<T>::n;
    constexpr int64_t CB = 128 * (4 + (UNIT ? 0 : (int64_t)sizeof(T)));
    const int p = lane / G, q = lane % G, c0 = q * V;
    const unsigned gmask = (G == 32 ? kFull : ((1u << G) - 1u)) << (p * G);
    const int nrhs = A.nrhs, nord = A.nord;
    auto rid = [&](int32_t o) -> int64_t { return A.rowmap ? __ldg(&A.rowmap[o]) : o; };
    auto load_x = [&](uint32_t col, T *o) {
        const T *px = A.x + (int64_t)col * A.ldx + c0;
        if (A.xvec) {
            if (c0 < nrhs) unpack(ld_x(reinterpret_cast<const VT *>(px)), o);
            else
#pragma unroll
                for (int k = 0; k < V; ++k) o[k] = T(0);
        } else {
#pragma unroll
            for (int k = 0; k < V; ++k) o[k] = c0 + k < nrhs ? ld_x(px + k) : T(0);
        }
    };
    auto store_y = [&](int64_t row, const T *v) {
        T *py = A.y + row * A.ldy + c0;
        if (A.yvec && c0 + V <= nrhs) {
            VT t;
            T *tv = reinterpret_cast<T *>(&t);
#pragma unroll
            for (int k = 0; k < V; ++k) tv[k] = v[k];
            *reinterpret_cast<VT *>(py) = t;
        } else {
#pragma unroll
            for (int k = 0; k < V; ++k)
                if (c0 + k < nrhs) py[k] = v[k];
        }
    };
    // a row across segments: every lane of the group writes its columns of
    // the slot; lane 0 of the group takes the arrival; the last part's group
    // adds the slots in segment order and stores y
    auto arrive = [&](int span, const T *v, int slot, int32_t o) {
        if (span & kRsPair) {  // every lane's columns meet on their own
#pragma unroll
            for (int k = 0; k < V; ++k) {
                T t = v[k];
                if (c0 + k < nrhs &&
                    rs_meet(S.xch, (int64_t)(span & ~kRsPair) * kRsMaxRhs + c0 + k, t))
                    A.y[rid(o) * A.ldy + c0 + k] = t;
            }
            return;
        }
#pragma unroll
        for (int k = 0; k < V; ++k)
            if (c0 + k < nrhs) S.part[(int64_t)slot * kRsMaxRhs + c0 + k] = v[k];
        __threadfence();
        __syncwarp(gmask);
        int last = 0;
        const int4 sp = __ldg(&S.spans[span]);
        if (q == 0) {
            cuda::atomic_ref<int32_t, cuda::thread_scope_device> ctr(S.counters[span]);
            last = ctr.fetch_add(1, cuda::memory_order_acq_rel) + 1 == sp.y - sp.x + 1;
            if (last) ctr.store(0, cuda::memory_order_relaxed);
        }
        last = __shfl_sync(gmask, last, p * G);
        if (last) {
            __threadfence();
            T tot[V];
#pragma unroll
            for (int k = 0; k < V; ++k)
                tot[k] = c0 + k < nrhs
                             ? __ldcg(&S.part[(int64_t)(2 * sp.x + 1) * kRsMaxRhs + c0 + k])
                             : T(0);
            for (int w = sp.x + 1; w <= sp.y; ++w)
#pragma unroll
                for (int k = 0; k < V; ++k)
                    if (c0 + k < nrhs)
                        tot[k] += __ldcg(&S.part[(int64_t)(2 * w) * kRsMaxRhs + c0 + k]);
            store_y(rid(sp.z), tot);
        }
    };
    const int32_t first = meta.x;
    int32_t ord0 = meta.x;
    T carry[V];
#pragma unroll
    for (int k = 0; k < V; ++k) carry[k] = T(0);
    for (int c = cb; c < ce; ++c) {
        const uint4 *gw = reinterpret_cast<const uint4 *>(A.chunks + (int64_t)c * CB);
        const uint8_t *gv = A.chunks + (int64_t)c * CB + 4 * 128;
        // row starts of the group's entries: each lane counts one 4-entry
        // step, the group adds them
        int cnt;
        {
            const uint4 t = __ldg(gw + G * p + q);
            cnt = (int)((t.x >> 31) + (t.y >> 31) + (t.z >> 31) + (t.w >> 31));
#pragma unroll
            for (int d = 1; d < G; d <<= 1) cnt += __shfl_xor_sync(kFull, cnt, d);
        }
        int inc = cnt;  // inclusive scan over the groups
#pragma unroll
        for (int d = 1; d < P; d <<= 1) {
            const int t = __shfl_up_sync(kFull, inc, d * G);
            if (p >= d) inc += t;
        }
        const int32_t ordS = ord0 + inc - cnt;  // the row this group starts in
        int32_t ord = ordS;
        T run[V], head[V];
#pragma unroll
        for (int k = 0; k < V; ++k) run[k] = head[k] = T(0);
        bool seen = false;
#pragma unroll 1
        for (int i = 0; i < G; ++i) {
            const int ls = G * p + i;  // the one-vector lane whose 4 entries these are
            const uint4 t = __ldg(gw + ls);
            const uint32_t w[4] = {t.x, t.y, t.z, t.w};
            T v[4];
            if (UNIT) {
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = T(1);
            } else if (NV == 4) {
                unpack(ld_stream(reinterpret_cast<const VT *>(gv) + ls, pol), v);
            } else {
                unpack(ld_stream(reinterpret_cast<const VT *>(gv) + ls, pol), v);
                unpack(ld_stream(reinterpret_cast<const VT *>(gv) + 32 + ls, pol), v + 2);
            }
            T xv[4][V];
#pragma unroll
            for (int j = 0; j < 4; ++j) load_x(w[j] & kRsColMask, xv[j]);
            T xo[GV ? 4 : 1][V];
            if (GV) {  // the entries' own rows of xo (the padding row: zeros)
                int32_t o = ord;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    o += (int32_t)(w[j] >> 31);
                    const T *po = gvp->xo + (o < nord ? rid(o) : 0) * gvp->ldo + c0;
                    if (o < nord && c0 < nrhs && gvp->xovec) {
                        unpack(__ldg(reinterpret_cast<const VT *>(po)), xo[GV ? j : 0]);
                    } else {
#pragma unroll
                        for (int k = 0; k < V; ++k)
                            xo[GV ? j : 0][k] = o < nord && c0 + k < nrhs ? __ldg(po + k) : T(0);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool f = (w[j] >> 31) != 0;
                if (GV) {  // value gradient of this entry: the group's dot product
                    T dot = T(0);
#pragma unroll
                    for (int k = 0; k < V; ++k)
                        if (c0 + k < nrhs) dot = fma(xv[j][k], xo[GV ? j : 0][k], dot);
#pragma unroll
                    for (int d = 1; d < G; d <<= 1) dot += __shfl_xor_sync(kFull, dot, d);
                    if (q == 0) {
                        T *pg = gvp->gv + (int64_t)c * 128 + 4 * ls + j;
                        *pg = gvp->accum ? *pg + dot : dot;
                    }
                }
                if (f && seen) store_y(rid(ord), run);  // a row whole inside the group
#pragma unroll
                for (int k = 0; k < V; ++k) {
                    head[k] = (f && !seen) ? run[k] : head[k];
                    run[k] = fma(v[j], xv[j][k], f ? T(0) : run[k]);
                }
                seen = seen || f;
                ord += f ? 1 : 0;
            }
        }
        // rows across groups: inclusive scan over the groups, reset at groups
        // holding a row start; group 0 continues the previous chunk
        T sc[V];
#pragma unroll
        for (int k = 0; k < V; ++k) sc[k] = (p == 0 && !seen) ? run[k] + carry[k] : run[k];
        bool r = seen;
#pragma unroll
        for (int d = 1; d < P; d <<= 1) {
            const bool ru = __shfl_up_sync(kFull, (int)r, d * G) != 0;
#pragma unroll
            for (int k = 0; k < V; ++k) {
                const T su = __shfl_up_sync(kFull, sc[k], d * G);
                if (p >= d && !r) sc[k] += su;
            }
            if (p >= d) r = r || ru;
        }
        T cin[V];
#pragma unroll
        for (int k = 0; k < V; ++k) {
            const T t = __shfl_up_sync(kFull, sc[k], G);
            cin[k] = p == 0 ? carry[k] : t;
        }
        if (seen) {  // the row this group started in ends here
            T val[V];
#pragma unroll
            for (int k = 0; k < V; ++k) val[k] = cin[k] + head[k];
            if (ordS == first && meta.z >= 0)
                arrive(meta.z, val, 2 * s, ordS);
            else if (!(ordS == first && meta.y) && ordS < nord)
                store_y(rid(ordS), val);
        }
#pragma unroll
        for (int k = 0; k < V; ++k) carry[k] = __shfl_sync(kFull, sc[k], (P - 1) * G + q);
        ord0 = __shfl_sync(kFull, ord, (P - 1) * G);
    }
    // the segment's last row: a span's part, or whole here (group 0)
    if (p == 0) {
        if (ord0 == first && meta.z >= 0)
            arrive(meta.z, carry, 2 * s, ord0);
        else if (meta.w >= 0)
            arrive(meta.w, carry, 2 * s + 1, ord0);
        else if (ord0 < nord && !(ord0 == first && meta.y))
            store_y(rid(ord0), carry);
    }
    __syncwarp();
}

template <typename T, int G, bool UNIT>
__global__ void __launch_bounds__(kRsWarps * 32, 1)
    cb_rowseg_mrhs_kernel(const RowSegDev rs, const T *x, T *__restrict__ y,
                          int nrhs, int64_t ldx, int64_t ldy, int xvec, int yvec) {
    dev::behind_wait();
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    {  // rows without entries
        const int64_t total = (int64_t)rs.nempty * nrhs;
        for (int64_t i = ((int64_t)blockIdx.x * kRsWarps + wib) * 32 + lane; i < total;
             i += (int64_t)gridDim.x * kRsWarps * 32)
            y[(int64_t)__ldg(&rs.empty[i / nrhs]) * ldy + i % nrhs] = T(0);
    }
    const int NB = gridDim.x, b = blockIdx.x;
    const int sb0 = (int)((int64_t)b * rs.nseg / NB);
    const int sb1 = (int)((int64_t)(b + 1) * rs.nseg / NB);
    const RsMat<T> A{rs.chunks, rs.rowmap, x, y, ldx, ldy, nrhs, rs.nord, xvec, yvec};
    const RsSpans<T> S{rs.spans, rs.counters, static_cast<T *>(rs.part), rs.xch};
    const uint64_t pol = dev::policy_evict_first();
    for (int s = sb0 + wib; s < sb1; s += kRsWarps)
        rs_mrhs_segment<T, G, UNIT>(A, s * rs.M, min(rs.nch, s * rs.M + rs.M),
                                    __ldg(&rs.meta[s]), s, S, lane, pol);
}

// The fused adjoint on a transposed stream: A^T G into y and the value
// gradient of every entry (kRsGvWarps warps per CTA: the gradient's registers fit without
// spills; each CTA's warps stride over its share of the segments).
template <typename T, int G>
__global__ void __launch_bounds__(kRsGvWarps * 32, 1)
    cb_rowseg_gv_kernel(const RowSegDev rs, const T *__restrict__ x, T *__restrict__ y,
                        int nrhs, int64_t ldx, int64_t ldy, int xvec, int yvec,
                        const RsGV<T> gvp) {
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    {  // rows without entries
        const int64_t total = (int64_t)rs.nempty * nrhs;
        for (int64_t i = ((int64_t)blockIdx.x * kRsGvWarps + wib) * 32 + lane; i < total;
             i += (int64_t)gridDim.x * kRsGvWarps * 32)
            y[(int64_t)__ldg(&rs.empty[i / nrhs]) * ldy + i % nrhs] = T(0);
    }
    const int NB = gridDim.x, b = blockIdx.x;
    const int sb0 = (int)((int64_t)b * rs.nseg / NB);
    const int sb1 = (int)((int64_t)(b + 1) * rs.nseg / NB);
    const RsMat<T> A{rs.chunks, rs.rowmap, x, y, ldx, ldy, nrhs, rs.nord, xvec, yvec};
    const RsSpans<T> S{rs.spans, rs.counters, static_cast<T *>(rs.part), rs.xch};
    const uint64_t pol = dev::policy_evict_first();
    for (int s = sb0 + wib; s < sb1; s += kRsGvWarps)
        rs_mrhs_segment<T, G, false, true>(A, s * rs.M, min(rs.nch, s * rs.M + rs.M),
                                           __ldg(&rs.meta[s]), s, S, lane, pol, &gvp);
}

// A batch over the streams (kRsBatchWarps warps per CTA: the kernel holds
// every lanes-per-entry variant, so it is given more registers per thread):
// warps take segments segs[0 .. nseg) ({matrix, first chunk, end chunk, -},
// with meta[] and the batch's own spans; queued by lanes per entry) from
// sched[0], choosing the segment code from the matrix's entry; the last warp
// out (sched[1]) resets both words for the next launch.
template <typename T>
__global__ void __launch_bounds__(kRsBatchWarps * 32, 1)
    cb_rowseg_batch_kernel(const RsBatchMat *__restrict__ mats, const int4 *__restrict__ segs,
                           const int4 *__restrict__ meta, int32_t nseg, uint32_t *sched,
                           const int2 *__restrict__ empty, int64_t nempty, const int4 *spans,
                           int32_t *counters, T *part, void *xch) {
    dev::behind_wait();
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    for (int64_t i = ((int64_t)blockIdx.x * kRsBatchWarps + wib) * 32 + lane; i < nempty;
         i += (int64_t)gridDim.x * kRsBatchWarps * 32) {  // rows without entries
        const int2 e = __ldg(&empty[i]);
        const RsBatchMat &m = mats[e.x];
        for (int k = 0; k < m.nrhs; ++k) static_cast<T *>(m.y)[(int64_t)e.y * m.ldy + k] = T(0);
    }
    const RsSpans<T> S{spans, counters, part, xch};
    const uint64_t pol = dev::policy_evict_first();
    while (true) {
        int si = 0;
        if (lane == 0) si = (int)atomicAdd(&sched[0], 1u);
        si = __shfl_sync(kFull, si, 0);
        if (si >= nseg) break;
        const int4 sg = __ldg(&segs[si]);
        const RsBatchMat &m = mats[sg.x];
        const RsMat<T> A{m.chunks, m.rowmap, static_cast<const T *>(m.x), static_cast<T *>(m.y),
                         m.ldx, m.ldy, m.nrhs, m.nord, m.xvec, m.yvec};
        const int4 mt = __ldg(&meta[si]);
        constexpr int GMAX = sizeof(T) == 4 ? 4 : 8;
        switch (m.g * 2 + (m.unit ? 1 : 0)) {
            case 2: rs_mrhs_segment<T, 1, false>(A, sg.y, sg.z, mt, si, S, lane, pol); break;
            case 3: rs_mrhs_segment<T, 1, true>(A, sg.y, sg.z, mt, si, S, lane, pol); break;
            case 4: rs_mrhs_segment<T, 2, false>(A, sg.y, sg.z, mt, si, S, lane, pol); break;
            case 5: rs_mrhs_segment<T, 2, true>(A, sg.y, sg.z, mt, si, S, lane, pol); break;
            case 8: rs_mrhs_segment<T, 4, false>(A, sg.y, sg.z, mt, si, S, lane, pol); break;
            case 9: rs_mrhs_segment<T, 4, true>(A, sg.y, sg.z, mt, si, S, lane, pol); break;
            case 16: rs_mrhs_segment<T, GMAX, false>(A, sg.y, sg.z, mt, si, S, lane, pol); break;
            case 17: rs_mrhs_segment<T, GMAX, true>(A, sg.y, sg.z, mt, si, S, lane, pol); break;
            default: break;
        }
    }
    // the last warp out resets the scheduler words for the next launch
    if (lane == 0) {
        __threadfence();
        if (atomicAdd(&sched[1], 1u) == gridDim.x * kRsBatchWarps - 1) {
            atomicExch(&sched[0], 0u);
            atomicExch(&sched[1], 0u);
        }
    }
}

// The balanced schedule (plans built with row_owned = 0): warps take whole
// groups (the reference's CTAs of waves_per_block blocks, balanced by its
// permutation), each lane a quad of 4 entries at a time; a run of one row
// inside the quad is summed in registers and added into y with an atomic
// (the reference's accumulate_output without CB_ROW_OWNED,
// cb-spmv-dcu.hpp:149-157).  y is zeroed before the launch.
constexpr int kBalWarps = 8;
template <typename T>
__global__ void __launch_bounds__(kBalWarps * 32)
    cb_balanced_kernel(const BalancedDev b, const T *__restrict__ x, T *__restrict__ y) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = (int64_t)gridDim.x * kBalWarps;
    for (int64_t g = (int64_t)blockIdx.x * kBalWarps + (threadIdx.x >> 5); g < b.ngroups;
         g += nw) {
        const int64_t q1 = __ldg(&b.gstart[g + 1]);
        for (int64_t q = __ldg(&b.gstart[g]) + lane; q < q1; q += 32) {
            const uint4 r4 = __ldg(&b.rows[q]), c4 = __ldg(&b.cols[q]);
            const uint32_t r[4] = {r4.x, r4.y, r4.z, r4.w}, c[4] = {c4.x, c4.y, c4.z, c4.w};
            T v[4];
            if (sizeof(T) == 4) {
                unpack(__ldg(reinterpret_cast<const float4 *>(b.vals) + q),
                       reinterpret_cast<float *>(v));
            } else {
                unpack(__ldg(reinterpret_cast<const double2 *>(b.vals) + 2 * q),
                       reinterpret_cast<double *>(v));
                unpack(__ldg(reinterpret_cast<const double2 *>(b.vals) + 2 * q + 1),
                       reinterpret_cast<double *>(v) + 2);
            }
            T xv[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) xv[j] = r[j] != kBalSkip ? __ldg(x + c[j]) : T(0);
            uint32_t rr = r[0];
            T run = v[0] * xv[0];
#pragma unroll
            for (int j = 1; j < 4; ++j) {
                if (r[j] == rr) {
                    run = fma(v[j], xv[j], run);
                } else {
                    if (rr != kBalSkip) atomicAdd(&y[rr], run);
                    rr = r[j];
                    run = v[j] * xv[j];
                }
            }
            if (rr != kBalSkip) atomicAdd(&y[rr], run);
        }
    }
}

// Balanced stream values refreshed from the tile payload (skip entries 0).
template <typename T>
__global__ void cb_balanced_values_kernel(const BalancedDev b, const uint8_t *__restrict__ payload) {
    T *vals = static_cast<T *>(const_cast<void *>(b.vals));
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < 4 * b.nquads;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t off = __ldg(&b.eoff[e]);
        vals[e] = off >= 0 ? *reinterpret_cast<const T *>(payload + off) : T(0);
    }
}

}  // namespace

// Launches a kernel that begins with dev::behind_wait: its blocks are set up
// while the launch before it drains, so a call in a solver's loop does not pay
// the launch latency between its kernels.  Time a call, one after another,
// without and with: 256 x 256 grid, FP64 6.1 and 5.1 us; n = 300007, FP32 18.2
// and 16.0; uniform A x and A^T y 30.8 and 27.9.  Such a kernel reads what a
// launch before it may have written (x, the stream's values) by coherent
// volatile loads (ld_x, ld_stream, stage_window): one through the read-only
// path (__ldg) could be moved before behind_wait and need not see those
// writes.  __ldg is for what stays as uploaded (words, meta, spans, row maps).
template <typename... P, typename... A>
cudaError_t launch_behind(void (*kernel)(P...), unsigned grid, unsigned threads, size_t smem,
                          cudaStream_t stream, A... args) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = stream;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

template <typename T, bool UNIT, bool MAP>
const void *rowseg_fn() {
    return reinterpret_cast<const void *>(cb_rowseg_kernel<T, UNIT, MAP>);
}

template <typename T, bool UNIT, bool MAP>
cudaError_t launch_rowseg_m(const DevLayout &d, const void *x, void *y, size_t smem,
                            cudaStream_t stream) {
    const void *fn = rowseg_fn<T, UNIT, MAP>();
    cudaError_t e = dev_enable_smem(fn, smem);
    if (e != cudaSuccess) return e;
    // the carveout: what the window leaves is L1 for the other gathers.  In
    // powers of two, so that plans of about one window size share a setting
    // (a change costs the host a call)
    size_t keep = size_t(16) << 10;
    while (keep < smem) keep *= 2;
    dev_resident_l1(fn, kRsWarps * 32, keep);
    // the grid the segments and windows were assigned for
    return launch_behind(cb_rowseg_kernel<T, UNIT, MAP>, (unsigned)d.rs.G, kRsWarps * 32, smem,
                         stream, d.rs, static_cast<const T *>(x), static_cast<T *>(y));
}

template <typename T, bool UNIT>
cudaError_t launch_rowseg_t(const DevLayout &d, const void *x, void *y, size_t smem,
                            cudaStream_t stream) {
    return d.rs.rowmap ? launch_rowseg_m<T, UNIT, true>(d, x, y, smem, stream)
                       : launch_rowseg_m<T, UNIT, false>(d, x, y, smem, stream);
}

int64_t rowseg_warps(int f32) {
    // the x window in shared memory; the carveout leaves the rest of the
    // unified L1/shared memory to the L1 (the other x gathers)
    const void *fn = f32 ? rowseg_fn<float, false, true>() : rowseg_fn<double, false, true>();
    if (dev_enable_smem(fn, (size_t)kRsWindowBytes) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return (int64_t)dev_sms() * dev_resident_l1(fn, kRsWarps * 32, (size_t)kRsWindowBytes) *
           kRsWarps;
}

cudaError_t launch_rowseg(const DevLayout &d, const void *x, void *y, cudaStream_t stream) {
    if (!d.rs.chunks || d.rs.nseg <= 0 || d.rs.G <= 0 || !d.rs.wbase || !d.rs.wlen)
        return cudaErrorInvalidValue;
    const size_t smem = (size_t)d.rs.W * (d.f32 ? 4 : 8);
    const cudaError_t e =
        d.f32 ? (d.rs.unit ? launch_rowseg_t<float, true>(d, x, y, smem, stream)
                           : launch_rowseg_t<float, false>(d, x, y, smem, stream))
              : (d.rs.unit ? launch_rowseg_t<double, true>(d, x, y, smem, stream)
                           : launch_rowseg_t<double, false>(d, x, y, smem, stream));
    if (e != cudaSuccess) return e;
    note_launch();
    return cudaGetLastError();
}

template <typename T, int G, bool UNIT>
cudaError_t launch_mrhs_g(const DevLayout &d, const T *x, T *y, int r, int64_t ldx, int64_t ldy,
                          int xvec, int yvec, cudaStream_t stream) {
    const void *fn = reinterpret_cast<const void *>(cb_rowseg_mrhs_kernel<T, G, UNIT>);
    dev_resident_l1(fn, kRsWarps * 32, 0);  // sets the carveout: all L1
    const cudaError_t e =
        launch_behind(cb_rowseg_mrhs_kernel<T, G, UNIT>, (unsigned)d.rs.G, kRsWarps * 32, 0,
                      stream, d.rs, x, y, r, ldx, ldy, xvec, yvec);
    if (e != cudaSuccess) return e;
    note_launch();
    return cudaGetLastError();
}

template <typename T, bool UNIT>
cudaError_t launch_mrhs_t(const DevLayout &d, const T *x, T *y, int nrhs, int64_t ldx,
                          int64_t ldy, cudaStream_t stream) {
    constexpr int V = 16 / sizeof(T);
    // slabs of at most kRsMaxRhs right-hand sides, one launch each
    for (int c = 0; c < nrhs; c += kRsMaxRhs) {
        const int r = std::min(kRsMaxRhs, nrhs - c);
        const int xvec = ldx % V == 0 && reinterpret_cast<uintptr_t>(x + c) % 16 == 0;
        const int yvec = ldy % V == 0 && reinterpret_cast<uintptr_t>(y + c) % 16 == 0;
        const int g = rs_lanes_per_entry(sizeof(T) == 4, r);
        cudaError_t e;
        switch (g) {
            case 1: e = launch_mrhs_g<T, 1, UNIT>(d, x + c, y + c, r, ldx, ldy, xvec, yvec, stream); break;
            case 2: e = launch_mrhs_g<T, 2, UNIT>(d, x + c, y + c, r, ldx, ldy, xvec, yvec, stream); break;
            case 4: e = launch_mrhs_g<T, 4, UNIT>(d, x + c, y + c, r, ldx, ldy, xvec, yvec, stream); break;
            default: e = launch_mrhs_g<T, (16 / sizeof(T) == 2 ? 8 : 4), UNIT>(
                         d, x + c, y + c, r, ldx, ldy, xvec, yvec, stream);
        }
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_rowseg_mrhs(const DevLayout &d, const void *x, void *y, int nrhs,
                               int64_t ldx, int64_t ldy, cudaStream_t stream) {
    if (!d.rs.chunks || d.rs.nseg <= 0 || d.rs.G <= 0 || nrhs < 1) return cudaErrorInvalidValue;
    if (d.f32)
        return d.rs.unit ? launch_mrhs_t<float, true>(d, static_cast<const float *>(x),
                                                      static_cast<float *>(y), nrhs, ldx, ldy, stream)
                         : launch_mrhs_t<float, false>(d, static_cast<const float *>(x),
                                                       static_cast<float *>(y), nrhs, ldx, ldy, stream);
    return d.rs.unit ? launch_mrhs_t<double, true>(d, static_cast<const double *>(x),
                                                   static_cast<double *>(y), nrhs, ldx, ldy, stream)
                     : launch_mrhs_t<double, false>(d, static_cast<const double *>(x),
                                                    static_cast<double *>(y), nrhs, ldx, ldy, stream);
}

template <typename T, int G>
cudaError_t launch_gv_g(const DevLayout &d, const T *g, T *gx, int r, int64_t ldg,
                        int64_t ldgx, int xvec, int yvec, const RsGV<T> &gvp,
                        cudaStream_t stream) {
    const void *fn = reinterpret_cast<const void *>(cb_rowseg_gv_kernel<T, G>);
    dev_resident_l1(fn, kRsGvWarps * 32, 0);  // sets the carveout: all L1
    cb_rowseg_gv_kernel<T, G><<<(unsigned)d.rs.G, kRsGvWarps * 32, 0, stream>>>(
        d.rs, g, gx, r, ldg, ldgx, xvec, yvec, gvp);
    note_launch();
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_gv_t(const DevLayout &d, const T *g, T *gx, int nrhs, int64_t ldg,
                        int64_t ldgx, const T *x, int64_t ldx, T *gv, cudaStream_t stream) {
    constexpr int V = 16 / sizeof(T);
    for (int c = 0; c < nrhs; c += kRsMaxRhs) {  // slabs of 16: the gradient adds up
        const int r = std::min(kRsMaxRhs, nrhs - c);
        const int xvec = ldg % V == 0 && reinterpret_cast<uintptr_t>(g + c) % 16 == 0;
        const int yvec = ldgx % V == 0 && reinterpret_cast<uintptr_t>(gx + c) % 16 == 0;
        const RsGV<T> gvp{x + c, ldx,
                          (int32_t)(ldx % V == 0 && reinterpret_cast<uintptr_t>(x + c) % 16 == 0),
                          (int32_t)(c > 0), gv};
        const int gl = rs_lanes_per_entry(sizeof(T) == 4, r);
        cudaError_t e;
        switch (gl) {
            case 1: e = launch_gv_g<T, 1>(d, g + c, gx + c, r, ldg, ldgx, xvec, yvec, gvp, stream); break;
            case 2: e = launch_gv_g<T, 2>(d, g + c, gx + c, r, ldg, ldgx, xvec, yvec, gvp, stream); break;
            case 4: e = launch_gv_g<T, 4>(d, g + c, gx + c, r, ldg, ldgx, xvec, yvec, gvp, stream); break;
            default: e = launch_gv_g<T, (16 / sizeof(T) == 2 ? 8 : 4)>(
                         d, g + c, gx + c, r, ldg, ldgx, xvec, yvec, gvp, stream);
        }
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_rowseg_adjoint(const DevLayout &d, const void *g, void *gx, int nrhs,
                                  int64_t ldg, int64_t ldgx, const void *x, int64_t ldx,
                                  void *gv, cudaStream_t stream) {
    if (!d.rs.chunks || d.rs.unit || d.rs.nseg <= 0 || d.rs.G <= 0 || nrhs < 1)
        return cudaErrorInvalidValue;
    if (d.f32)
        return launch_gv_t<float>(d, static_cast<const float *>(g), static_cast<float *>(gx),
                                  nrhs, ldg, ldgx, static_cast<const float *>(x), ldx,
                                  static_cast<float *>(gv), stream);
    return launch_gv_t<double>(d, static_cast<const double *>(g), static_cast<double *>(gx),
                               nrhs, ldg, ldgx, static_cast<const double *>(x), ldx,
                               static_cast<double *>(gv), stream);
}

cudaError_t launch_balanced(const DevLayout &d, const void *x, void *y, cudaStream_t stream) {
    if (!d.bal.rows) return cudaErrorInvalidValue;
    const size_t vsz = d.f32 ? 4 : 8;
    cudaError_t e = cudaMemsetAsync(y, 0, (size_t)d.m * vsz, stream);
    if (e != cudaSuccess) return e;
    const void *fn = d.f32 ? reinterpret_cast<const void *>(cb_balanced_kernel<float>)
                           : reinterpret_cast<const void *>(cb_balanced_kernel<double>);
    const int64_t grid = std::max<int64_t>(
        1, std::min<int64_t>((d.bal.ngroups + kBalWarps - 1) / kBalWarps,
                             (int64_t)dev_sms() * dev_resident(fn, kBalWarps * 32, 0)));
    if (d.f32)
        cb_balanced_kernel<float><<<(unsigned)grid, kBalWarps * 32, 0, stream>>>(
            d.bal, static_cast<const float *>(x), static_cast<float *>(y));
    else
        cb_balanced_kernel<double><<<(unsigned)grid, kBalWarps * 32, 0, stream>>>(
            d.bal, static_cast<const double *>(x), static_cast<double *>(y));
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_balanced_values(const DevLayout &d, cudaStream_t stream) {
    if (!d.bal.rows || !d.bal.eoff || d.bal.nquads <= 0) return cudaSuccess;
    const unsigned grid =
        (unsigned)std::min<int64_t>((4 * d.bal.nquads + 255) / 256, (int64_t)dev_sms() * 16);
    if (d.f32)
        cb_balanced_values_kernel<float><<<grid, 256, 0, stream>>>(d.bal, d.payload);
    else
        cb_balanced_values_kernel<double><<<grid, 256, 0, stream>>>(d.bal, d.payload);
    note_launch();
    return cudaGetLastError();
}

int rs_lanes_per_entry(int f32, int nrhs) {
    const int V = f32 ? 4 : 2, gmax = f32 ? 4 : 8;
    int g = 1;
    while (g * V < std::min(nrhs, kRsMaxRhs) && g < gmax) g *= 2;
    return g;
}

int64_t rowseg_batch_warps(int f32) {
    const void *fn = f32 ? reinterpret_cast<const void *>(cb_rowseg_batch_kernel<float>)
                         : reinterpret_cast<const void *>(cb_rowseg_batch_kernel<double>);
    return (int64_t)dev_sms() * dev_resident_l1(fn, kRsBatchWarps * 32, 0) * kRsBatchWarps;
}

cudaError_t launch_rowseg_batch(int f32, const RsBatchMat *mats, const int4 *segs,
                                const int4 *meta, int32_t nseg, uint32_t *sched, int64_t nwarps,
                                const int2 *empty, int64_t nempty, const int4 *spans,
                                int32_t *counters, void *part, void *xch,
                                cudaStream_t stream) {
    if (nwarps <= 0 || nwarps % kRsBatchWarps) return cudaErrorInvalidValue;
    const unsigned grid = (unsigned)(nwarps / kRsBatchWarps);
    const cudaError_t e =
        f32 ? launch_behind(cb_rowseg_batch_kernel<float>, grid, kRsBatchWarps * 32, 0, stream,
                            mats, segs, meta, nseg, sched, empty, nempty, spans, counters,
                            static_cast<float *>(part), xch)
            : launch_behind(cb_rowseg_batch_kernel<double>, grid, kRsBatchWarps * 32, 0, stream,
                            mats, segs, meta, nseg, sched, empty, nempty, spans, counters,
                            static_cast<double *>(part), xch);
    if (e != cudaSuccess) return e;
    note_launch();
    return cudaGetLastError();
}

}  // namespace cb
