// Block primitives of the pivot-set closures (open.cu, node_build.cu, kernels.cu): the
// Floyd-Warshall of a 64-pivot block, alone or with the pivot rows of a column tile.
// All run on a 256-thread CTA.
#pragma once
#include "minplus.cuh"

#include <cstdint>

namespace hb {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int B = 64;  // pivots per round

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc) {
    const uint32_t sa = (uint32_t)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

constexpr int kTLD = B + 8;  // padded row of T (144 bytes): column reads hit distinct banks

// Floyd-Warshall over the round's pivot block T (mk <= B rows, identity
// beyond) in shared memory: thread t owns row t / 4 and 16 columns.  Step kk
// reads row kk and column kk, whose values it rewrites unchanged
// (T[kk][kk] = 0), so one barrier per step orders it before step kk + 1; a
// = INF gives no change through the clamped form, so no branch is needed.
__device__ __forceinline__ void close_pivot_block(uint16_t (*Ts)[kTLD], int mk) {
    const int tid = threadIdx.x;
    const int a = tid >> 2, c0 = (tid & 3) * 16;
    uint32_t v[8];
    const uint4 x0 = *reinterpret_cast<const uint4*>(&Ts[a][c0]);
    const uint4 y0 = *reinterpret_cast<const uint4*>(&Ts[a][c0 + 8]);
    v[0] = x0.x; v[1] = x0.y; v[2] = x0.z; v[3] = x0.w; v[4] = y0.x; v[5] = y0.y; v[6] = y0.z; v[7] = y0.w;
    for (int kk = 0; kk < mk; ++kk) {
        const uint32_t t = Ts[a][kk];
        const uint4 x = *reinterpret_cast<const uint4*>(&Ts[kk][c0]);
        const uint4 y = *reinterpret_cast<const uint4*>(&Ts[kk][c0 + 8]);
        const uint32_t rw[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
        const uint32_t aa = splat(t), tt = INF2 - aa;
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = acc_clamp(v[i], rw[i], aa, tt);
        *reinterpret_cast<uint4*>(&Ts[a][c0]) = make_uint4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<uint4*>(&Ts[a][c0 + 8]) = make_uint4(v[4], v[5], v[6], v[7]);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Closure of a round's pivot block together with its pivot rows: the augmented
// matrix M = [T | Bt], 64 rows x 32 CW columns (T the pivot block in the first 64,
// Bt the pivot rows of a column tile), becomes [T* | T* (x) Bt]: a shortest path
// from pivot a to column j through pivots ends with one entry of a pivot row.
// Floyd-Warshall with M in registers: thread (rg, cg) = (t / 16, t % 16) owns rows
// 4 rg .. and columns 2 CW cg ..; a step needs the pivot row only (T is symmetric, so its
// T part is the pivot column too), which its owners put into one of two shared rows
// at the step before: one barrier and two shared loads a step.  Blocks of 16
// pivots with 6 barriers each, which this replaces, cost 4 us however few the
// pivots are and no less than this at 64 (device time of an opening with 1 cell, 256 x 256
// open map, b = 16: 128 -> 115 us; 256 cells, 1024 x 1024 street map, b = 8: 4351 -> 4147 us).
// HALF: every finite value is <= kHalfMax and INF stands as kHalfInf: sums need
// no clamp, one fused add-and-min per pair.  Values then saturate at kHalfInf, which
// is exact while no finite distance reaches it; fw_panel checks that.
// ---------------------------------------------------------------------------
constexpr int kHalfMax = 16383;
constexpr uint32_t kHalfInf = 32767u;
constexpr uint32_t kHalfInf2 = 0x7FFF7FFFu;

template <bool HALF>
__device__ __forceinline__ uint32_t acc_mode(uint32_t c, uint32_t b, uint32_t aa) {
    if constexpr (HALF) return acc_fast(c, b, aa);
    else return acc_clamp(c, b, aa, INF2 - aa);
}

template <int CW>
struct alignas(16) FwSmem {
    static constexpr int LD = 32 * CW + 8;  // padded row: the 8 rows of a 16-byte access phase hit distinct banks
    uint16_t M[64][LD];
    uint16_t P[2][LD];  // pivot rows of this step and the next
    int mx[2];
};

// CW packed words at p (8-byte aligned).
template <int CW>
__device__ __forceinline__ void ld_words(const uint16_t* p, uint32_t (&w)[CW]) {
    static_assert(CW % 2 == 0, "pairs of words");
    if constexpr (CW % 4 == 0) {
#pragma unroll
        for (int x = 0; x < CW / 4; ++x) {
            const uint4 v = reinterpret_cast<const uint4*>(p)[x];
            w[4 * x] = v.x; w[4 * x + 1] = v.y; w[4 * x + 2] = v.z; w[4 * x + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int x = 0; x < CW / 2; ++x) {
            const uint2 v = reinterpret_cast<const uint2*>(p)[x];
            w[2 * x] = v.x; w[2 * x + 1] = v.y;
        }
    }
}
template <int CW>
__device__ __forceinline__ void st_words(uint16_t* p, const uint32_t (&w)[CW]) {
    if constexpr (CW % 4 == 0) {
#pragma unroll
        for (int x = 0; x < CW / 4; ++x)
            reinterpret_cast<uint4*>(p)[x] = make_uint4(w[4 * x], w[4 * x + 1], w[4 * x + 2], w[4 * x + 3]);
    } else {
#pragma unroll
        for (int x = 0; x < CW / 2; ++x) reinterpret_cast<uint2*>(p)[x] = make_uint2(w[2 * x], w[2 * x + 1]);
    }
}

// m[r][.] = min(m[r][.], min_{k < B} A[k][4 rg + r] (+) A[k][columns]) for the
// thread's tile; A has rows of stride LD with the pivot columns first.
template <int CW, bool HALF>
__device__ __forceinline__ void fw_product(const uint16_t* A, uint32_t (&m)[4][CW]) {
    constexpr int LD = FwSmem<CW>::LD;
    const int rg = threadIdx.x >> 4, cg = threadIdx.x & 15;
    const uint16_t *ap = A + 4 * rg, *bp = A + 2 * CW * cg;
#pragma unroll 2
    for (int k = 0; k < B; ++k) {
        const uint2 a2 = *reinterpret_cast<const uint2*>(ap + k * LD);
        uint32_t b[CW];
        ld_words<CW>(bp + k * LD, b);
        const uint32_t a[4] = {splat(a2.x), splat(a2.x >> 16), splat(a2.y), splat(a2.y >> 16)};
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int w = 0; w < CW; ++w) m[r][w] = acc_mode<HALF>(m[r][w], b[w], a[r]);
    }
}

// The thread's tile m of M -> the closed tile.
template <int CW, bool HALF>
__device__ __forceinline__ void fw_close(FwSmem<CW>& F, int mk, uint32_t (&m)[4][CW]) {
    const int rg = threadIdx.x >> 4, cg = threadIdx.x & 15;
    if (rg == 0) st_words<CW>(&F.P[0][2 * CW * cg], m[0]);
    __syncthreads();
#pragma unroll 1
    for (int s0 = 0; s0 < mk; s0 += 4) {
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            if (s0 + x >= mk) break;  // uniform
            const uint2 a2 = *reinterpret_cast<const uint2*>(&F.P[x & 1][4 * rg]);
            uint32_t b[CW];
            ld_words<CW>(&F.P[x & 1][2 * CW * cg], b);
            const uint32_t a[4] = {splat(a2.x), splat(a2.x >> 16), splat(a2.y), splat(a2.y >> 16)};
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int w = 0; w < CW; ++w) m[r][w] = acc_mode<HALF>(m[r][w], b[w], a[r]);
            if (rg == (s0 + x + 1) >> 2) st_words<CW>(&F.P[(x + 1) & 1][2 * CW * cg], m[(x + 1) & 3]);
            __syncthreads();
        }
    }
}

// Largest finite value of packed words, INF (full range) or kHalfInf (half range, no value
// above it) aside: the words are shifted so that INF becomes 0.
template <bool HALF>
__device__ __forceinline__ uint32_t top_of(uint32_t top, uint32_t w) {
    constexpr uint32_t shift = 0x10000u - (HALF ? kHalfInf : (uint32_t)INF);
    return max2(top, add2(w, shift * 0x00010001u));
}
template <bool HALF>
__device__ __forceinline__ int top_value(uint32_t top) {
    constexpr int shift = 0x10000 - (HALF ? (int)kHalfInf : (int)INF);
    return max((int)max(top & 0xffffu, top >> 16) - shift, 0);
}
template <bool HALF, int R, int W>
__device__ __forceinline__ int tile_top(const uint32_t (&m)[R][W]) {
    uint32_t top = 0;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int w = 0; w < W; ++w) top = top_of<HALF>(top, m[r][w]);
    return top_value<HALF>(top);
}
// Half-range sums (65534 at most; kHalfInf or more: INF) as full-range values.
__device__ __forceinline__ uint32_t half_to_full(uint32_t w) {
    const uint32_t inf = (w + 0x00010001u) & 0x80008000u;  // the top bit of a half that is INF ..
    return min2(w | (2 * inf - (inf >> 15)), INF2);         // .. -> all its bits
}

// The whole of it for the tile in F.M (synchronised; raw values, INF = 60000):
// with Q, first M = min(M, Q_T^T (x) Q) (a 64 x 32 CW panel of the round before).
// m receives the closed tile with INF = 60000.  The half range is tried with Q, whose
// product is most of the work; without it the checks cost more than the clamps.
// Returns false when the half range turned out too small (Q is used up; call again on
// fresh copies with half off).  A finite distance of kHalfInf or more would have a
// prefix, itself a distance between pivots, within one entry of M of kHalfInf: none is there when
// the largest finite result and the largest finite entry add up to less.
template <int CW>
__device__ __forceinline__ bool fw_panel(FwSmem<CW>& F, uint16_t* Q, int mk, bool try_half, uint32_t (&m)[4][CW]) {
    constexpr int LD = FwSmem<CW>::LD;
    const int tid = threadIdx.x, rg = tid >> 4, cg = tid & 15;
#pragma unroll
    for (int r = 0; r < 4; ++r) ld_words<CW>(&F.M[4 * rg + r][2 * CW * cg], m[r]);
    bool half = false;
    if (Q) {
        uint32_t q[4][CW];
#pragma unroll
        for (int r = 0; r < 4; ++r) ld_words<CW>(Q + (4 * rg + r) * LD + 2 * CW * cg, q[r]);
        if (tid < 2) F.mx[tid] = 0;
        half = __syncthreads_and(try_half && max(tile_top<false>(m), tile_top<false>(q)) <= kHalfMax);
    }
    if (!half) {
        if (Q) fw_product<CW, false>(Q, m);
        fw_close<CW, false>(F, mk, m);
        return true;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        uint32_t q[CW];
        uint16_t* p = Q + (4 * rg + r) * LD + 2 * CW * cg;
        ld_words<CW>(p, q);
#pragma unroll
        for (int w = 0; w < CW; ++w) {
            m[r][w] = min2(m[r][w], kHalfInf2);
            q[w] = min2(q[w], kHalfInf2);
        }
        st_words<CW>(p, q);
    }
    __syncthreads();
    fw_product<CW, true>(Q, m);
    const int m0 = tile_top<true>(m);
    fw_close<CW, true>(F, mk, m);
    const int a = __reduce_max_sync(0xffffffffu, m0), z = __reduce_max_sync(0xffffffffu, tile_top<true>(m));
    if ((tid & 31) == 0) {
        atomicMax(&F.mx[0], a);
        atomicMax(&F.mx[1], z);
    }
    __syncthreads();
    if (F.mx[0] + F.mx[1] >= (int)kHalfInf) return false;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int w = 0; w < CW; ++w) m[r][w] = half_to_full(m[r][w]);
    return true;
}

// Upper-triangle tile pair t of an nt x nt tile grid: I <= J.
__device__ __forceinline__ void tri_pair(int t, int nt, int& I, int& J) {
    int i = 0;
    while (t >= nt - i) {
        t -= nt - i;
        ++i;
    }
    I = i;
    J = i + t;
}

}  // namespace
}  // namespace hb
