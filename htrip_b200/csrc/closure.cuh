// Block primitives of the pivot-set closures (open.cu, node_build.cu): the
// Floyd-Warshall of a 64-pivot block with the pivot rows of a column tile, and
// the 64 x 64 min-plus product.  All run on a 256-thread CTA.
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
// Blocked Floyd-Warshall in steps of 16 pivots K: the 16 x 16 block is closed by
// four squarings (T is symmetric, so a squared entry is a product of two
// rows), then the rows K follow as block* (x) M[K, :], then M = min(M, P^T (x) P).
// Thread (rg, cg) = (t / 16, t % 16) owns rows 4 rg .. and columns 2 CW cg .. in
// registers; 6 CTA barriers per 16 pivots.  A step per pivot with a barrier each, as
// before, is a chain of 64 shared-memory round trips; the opening kernel's mixed
// stages (panel with the old panel's update, beside the update) went from 35-38 to
// 26-30 us, its first panels from 18-20 to 15-17 us.
// HALF: every finite value is <= kHalfMax and INF stands as kHalfInf: sums need
// no clamp, one fused add-and-min per pair.  Values then saturate at kHalfInf, which
// is exact while no finite distance reaches it; fw_exact checks that.
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
    uint16_t P[16][LD];
    uint16_t S[2][16][24];
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

// m[r][.] = min(m[r][.], min_{k < K} A[k][4 rg + r] (+) A[k][columns]) for the
// thread's tile; A has rows of stride LD with the pivot columns first.
template <int CW, bool HALF, int K>
__device__ __forceinline__ void fw_product(const uint16_t* A, uint32_t (&m)[4][CW]) {
    constexpr int LD = FwSmem<CW>::LD;
    const int rg = threadIdx.x >> 4, cg = threadIdx.x & 15;
    const uint16_t *ap = A + 4 * rg, *bp = A + 2 * CW * cg;
#pragma unroll 2
    for (int k = 0; k < K; ++k) {
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

// M (synchronised) and the thread's tile m of it -> the closed tile in m.
template <int CW, bool HALF>
__device__ __forceinline__ void fw_close(FwSmem<CW>& F, int mk, uint32_t (&m)[4][CW]) {
    constexpr int LD = FwSmem<CW>::LD;
    const int tid = threadIdx.x, rg = tid >> 4, cg = tid & 15;
#pragma unroll 1
    for (int k0 = 0; k0 < mk; k0 += 16) {
        {
            const uint16_t *ri = &F.M[k0 + rg][k0], *rj = &F.M[k0 + cg][k0];
#pragma unroll 1
            for (int q = 0; q < 4; ++q) {
                uint32_t a[8], b[8], v = HALF ? kHalfInf2 : INF2;
                ld_words<8>(ri, a);
                ld_words<8>(rj, b);
#pragma unroll
                for (int x = 0; x < 8; ++x) v = acc_mode<HALF>(v, b[x], a[x]);
                F.S[q & 1][rg][cg] = (uint16_t)min(v & 0xffffu, v >> 16);
                __syncthreads();
                ri = F.S[q & 1][rg];
                rj = F.S[q & 1][cg];
            }
        }
        {
            uint32_t acc[CW];
#pragma unroll
            for (int w = 0; w < CW; ++w) acc[w] = HALF ? kHalfInf2 : INF2;
            const uint16_t* bp = &F.M[k0][2 * CW * cg];
#pragma unroll 4
            for (int e = 0; e < 16; ++e) {
                uint32_t b[CW];
                ld_words<CW>(bp + e * LD, b);
                const uint32_t a = splat(F.S[1][rg][e]);
#pragma unroll
                for (int w = 0; w < CW; ++w) acc[w] = acc_mode<HALF>(acc[w], b[w], a);
            }
            st_words<CW>(&F.P[rg][2 * CW * cg], acc);
        }
        __syncthreads();
        fw_product<CW, HALF, 16>(&F.P[0][0], m);
        if ((rg >> 2) == (k0 >> 4) + 1) {  // the next step's pivot rows
#pragma unroll
            for (int r = 0; r < 4; ++r) st_words<CW>(&F.M[4 * rg + r][2 * CW * cg], m[r]);
        }
        __syncthreads();
    }
}

// Whether every value of w fits the half range (INF aside).
__device__ __forceinline__ bool half_ok(uint32_t w) {
    const uint32_t lo = w & 0xffffu, hi = w >> 16;
    return (lo <= (uint32_t)kHalfMax || lo >= INF) && (hi <= (uint32_t)kHalfMax || hi >= INF);
}
// Half-range sums (kHalfInf or more: INF) as full-range values.
__device__ __forceinline__ uint32_t half_to_full(uint32_t w) {
    const uint32_t lo = w & 0xffffu, hi = w >> 16;
    return (lo >= kHalfInf ? (uint32_t)INF : lo) | ((hi >= kHalfInf ? (uint32_t)INF : hi) << 16);
}
// Largest value below kHalfInf of a tile.
template <int CW>
__device__ __forceinline__ int half_max(const uint32_t (&m)[4][CW]) {
    uint32_t mx = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int w = 0; w < CW; ++w) {
            const uint32_t lo = m[r][w] & 0xffffu, hi = m[r][w] >> 16;
            if (lo < kHalfInf) mx = max(mx, lo);
            if (hi < kHalfInf) mx = max(mx, hi);
        }
    return (int)mx;
}

// The whole of it for the tile in F.M (synchronised; raw values, INF = 60000):
// with Q, first M = min(M, Q_T^T (x) Q) (a 64 x 32 CW panel of the round before).
// m receives the closed tile with INF = 60000.  Returns false when the half range
// turned out too small (F is used up; call again on fresh copies with half
// off).  A finite distance of kHalfInf or more would have a prefix, itself a
// distance between pivots, within one entry of M of kHalfInf: none is there when
// the largest finite result and the largest finite entry add up to less.
template <int CW>
__device__ __forceinline__ bool fw_panel(FwSmem<CW>& F, uint16_t* Q, int mk, bool try_half, uint32_t (&m)[4][CW]) {
    constexpr int LD = FwSmem<CW>::LD;
    const int tid = threadIdx.x, rg = tid >> 4, cg = tid & 15;
    bool ok = try_half;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        ld_words<CW>(&F.M[4 * rg + r][2 * CW * cg], m[r]);
#pragma unroll
        for (int w = 0; w < CW; ++w) ok &= half_ok(m[r][w]);
    }
    if (Q) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            uint32_t q[CW];
            ld_words<CW>(Q + (4 * rg + r) * LD + 2 * CW * cg, q);
#pragma unroll
            for (int w = 0; w < CW; ++w) ok &= half_ok(q[w]);
        }
    }
    if (tid < 2) F.mx[tid] = 0;
    if (!__syncthreads_and(ok)) {
        if (Q) {
            fw_product<CW, false, 64>(Q, m);
#pragma unroll
            for (int r = 0; r < 4; ++r) st_words<CW>(&F.M[4 * rg + r][2 * CW * cg], m[r]);
            __syncthreads();
        }
        fw_close<CW, false>(F, mk, m);
        return true;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int w = 0; w < CW; ++w) m[r][w] = min2(m[r][w], kHalfInf2);
    if (Q) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            uint32_t q[CW];
            uint16_t* p = Q + (4 * rg + r) * LD + 2 * CW * cg;
            ld_words<CW>(p, q);
#pragma unroll
            for (int w = 0; w < CW; ++w) q[w] = min2(q[w], kHalfInf2);
            st_words<CW>(p, q);
        }
        __syncthreads();
        fw_product<CW, true, 64>(Q, m);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) st_words<CW>(&F.M[4 * rg + r][2 * CW * cg], m[r]);
    const int m0 = half_max<CW>(m);
    __syncthreads();
    fw_close<CW, true>(F, mk, m);
    const int a = __reduce_max_sync(0xffffffffu, m0), z = __reduce_max_sync(0xffffffffu, half_max<CW>(m));
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
