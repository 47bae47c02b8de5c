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

// Floyd-Warshall over the round's pivots on the augmented rows [T | Bt]:
// T the pivot block as above, Bt the pivot rows of a 64-column tile.  After
// the last pivot, Bt = T* (x) Bt: a shortest path from pivot a to column j
// through pivots ends with one entry D[c][j] of a pivot row.  Thread t owns
// row t / 4 and 16 columns of each part; its Bt values end in vb.  Row kk of
// both parts is rewritten unchanged at step kk (T[kk][kk] = 0), so one
// barrier per step; rows >= mk of Bt are never read (T[a][kk] = INF there).
__device__ __forceinline__ void close_pivot_panel(uint16_t (*Ts)[kTLD], uint16_t (*Bt)[kTLD], int mk,
                                                  uint32_t (&vb)[8]) {
    const int tid = threadIdx.x;
    const int a = tid >> 2, c0 = (tid & 3) * 16;
    uint32_t v[8];
    {
        const uint4 x0 = *reinterpret_cast<const uint4*>(&Ts[a][c0]);
        const uint4 y0 = *reinterpret_cast<const uint4*>(&Ts[a][c0 + 8]);
        const uint4 x1 = *reinterpret_cast<const uint4*>(&Bt[a][c0]);
        const uint4 y1 = *reinterpret_cast<const uint4*>(&Bt[a][c0 + 8]);
        v[0] = x0.x; v[1] = x0.y; v[2] = x0.z; v[3] = x0.w; v[4] = y0.x; v[5] = y0.y; v[6] = y0.z; v[7] = y0.w;
        vb[0] = x1.x; vb[1] = x1.y; vb[2] = x1.z; vb[3] = x1.w; vb[4] = y1.x; vb[5] = y1.y; vb[6] = y1.z; vb[7] = y1.w;
    }
    for (int kk = 0; kk < mk; ++kk) {
        const uint32_t t = Ts[a][kk];
        const uint4 x = *reinterpret_cast<const uint4*>(&Ts[kk][c0]);
        const uint4 y = *reinterpret_cast<const uint4*>(&Ts[kk][c0 + 8]);
        const uint4 xb = *reinterpret_cast<const uint4*>(&Bt[kk][c0]);
        const uint4 yb = *reinterpret_cast<const uint4*>(&Bt[kk][c0 + 8]);
        const uint32_t rw[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
        const uint32_t rb[8] = {xb.x, xb.y, xb.z, xb.w, yb.x, yb.y, yb.z, yb.w};
        const uint32_t aa = splat(t), tt = INF2 - aa;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            v[i] = acc_clamp(v[i], rw[i], aa, tt);
            vb[i] = acc_clamp(vb[i], rb[i], aa, tt);
        }
        *reinterpret_cast<uint4*>(&Ts[a][c0]) = make_uint4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<uint4*>(&Ts[a][c0 + 8]) = make_uint4(v[4], v[5], v[6], v[7]);
        *reinterpret_cast<uint4*>(&Bt[a][c0]) = make_uint4(vb[0], vb[1], vb[2], vb[3]);
        *reinterpret_cast<uint4*>(&Bt[a][c0 + 8]) = make_uint4(vb[4], vb[5], vb[6], vb[7]);
        __syncthreads();
    }
}

// 64 x 64 block product of the panel unit (kn <= B pivot steps):
//   acc[i][q] = min_k A[k][row i] (+) Bm[k][column pair q]
// Warp w owns rows 8w .. 8w + 7 and skips (class 0) or takes the 2-op form
// (class 1) for pivot k by cls[k * kWarps + w]; lane 8 rp + cg holds rows
// 8w + 2rp, 8w + 2rp + 1 and columns 8cg .. 8cg + 7 (four packed pairs), so
// a pivot step is one 4-byte and one 16-byte shared load for 8 updates.
__device__ __forceinline__ void gemm64(const uint16_t (*A)[kTLD], const uint16_t* Bm, int ldb, int kn,
                                       const uint8_t* cls, uint32_t (&acc)[2][4]) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint16_t* ap = &A[0][warp * 8 + 2 * (lane >> 3)];
    const uint16_t* bp = Bm + (lane & 7) * 8;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[i][q] = INF2;
#pragma unroll 2
    for (int k = 0; k < kn; ++k) {
        const int c = cls[k * kWarps + warp];
        if (c == 0) continue;  // uniform over the warp
        const uint32_t a2 = *reinterpret_cast<const uint32_t*>(ap + k * kTLD);
        const uint4 b4 = *reinterpret_cast<const uint4*>(bp + k * ldb);
        const uint32_t b[4] = {b4.x, b4.y, b4.z, b4.w};
        const uint32_t aa[2] = {splat(a2), splat(a2 >> 16)};
        if (c == 1) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[i][q] = acc_fast(acc[i][q], b[q], aa[i]);
        } else {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint32_t tt = INF2 - aa[i];
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[i][q] = acc_clamp(acc[i][q], b[q], aa[i], tt);
            }
        }
    }
}

// dst[row i][8 cg .. 8 cg + 7] = min(dst, acc[i]) for the rows of gemm64's
// thread layout below `rows`.
__device__ __forceinline__ void min_into(uint16_t* dst, int ld, int rows, const uint32_t (&acc)[2][4]) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int a = warp * 8 + 2 * (lane >> 3) + i;
        if (a >= rows) continue;
        uint4* p = reinterpret_cast<uint4*>(dst + a * ld + (lane & 7) * 8);
        const uint4 o = *p;
        *p = make_uint4(min2(o.x, acc[i][0]), min2(o.y, acc[i][1]), min2(o.z, acc[i][2]), min2(o.w, acc[i][3]));
    }
}

// Class of step k for warp w's rows of a 64 x 64 operand A (entries
// A[k][8w .. 8w+7]): 0 all INF (skip), 1 all <= INF_HEADROOM (2-op form),
// 2 otherwise.
__device__ __forceinline__ void block_classes(const uint16_t (*A)[kTLD], int kn, uint8_t* cls) {
    for (int idx = threadIdx.x; idx < kn * kWarps; idx += kThreads) {
        const int k = idx / kWarps, w = idx % kWarps;
        const uint4 v = *reinterpret_cast<const uint4*>(&A[k][w * 8]);
        const uint32_t x[4] = {v.x, v.y, v.z, v.w};
        uint32_t mn = 0xffffu, mx = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            mn = min(mn, min(x[q] & 0xffffu, x[q] >> 16));
            mx = max(mx, max(x[q] & 0xffffu, x[q] >> 16));
        }
        cls[idx] = mn >= INF ? 0 : (mx <= INF_HEADROOM ? 1 : 2);
    }
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
