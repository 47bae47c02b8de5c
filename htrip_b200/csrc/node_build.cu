// Internal-node matrices from their children and seams (reference
// InternalNode::recomputeFromChildren, src/internal_node.cpp:94-245): the
// shortest-path closure D of a node's boundary vertices V_U, given every
// child's closed summary S_q and the seam edges between the children.
//
// The seam edges are contracted: a path between two boundary vertices is a
// chain of child segments joined by seam edges, so all that has to be closed
// is the matrix T over the node's active seam edges E (both cells passable),
// about half the pivots of a closure over the edges' endpoints and an eighth
// of the node's order.  Edge e = (u, v, w) stands for its vertex u; it is incident
// to u's child with offset 0 and to v's child with offset w.  With R_q[k][j] =
// o_k (+) S_q[x_k][j] for the incidences k = (x_k, e_k, o_k) of child q:
//   T0[e][e'] = min over common children q of R_q[e][x_e'] (+) o_e'
//   T  = closure of T0 (blocked Floyd-Warshall, 64 pivots a round)
//   U_p[e][i]  = min_k T[e][e_k] (+) R_p[k][i]            (k over child p's)
//   D[i][j]    = min([p == q] S_p[i][j], min_k U_p[e_k][i] (+) R_q[k][j])
//                for i in child p, j in child q, p <= q, and transposed.
// Every sum is the exact clamped tropical product and the closure is unique,
// so D equals the reference's sequential relaxation over the seam endpoints
// bit for bit; each matrix is written once instead of once per 64 pivots.
// Measured against the blocked closure over the seam endpoints that it
// replaces (device time, B200): building a 1024 x 1024 street map, b = 8, 22.8 ->
// 5.9 ms; one weight change on a 256 x 256 map, b = 8, 2.45 -> 0.75 ms.
#include "closure.cuh"
#include "kernels.cuh"

#include <algorithm>
#include <type_traits>

namespace hb {

namespace {

constexpr unsigned FULL = 0xffffffffu;

// Distances of at most kHalfMax add up below kHalfInf, so with INF replaced
// by kHalfInf a sum needs no clamp: it never wraps (65534 at most) and a sum
// of kHalfInf or more means INF.
constexpr int kHalfMax = 16383;
constexpr uint32_t kHalfInf = 32767u;
constexpr uint32_t kHalfInf2 = 0x7FFF7FFFu;

__device__ __forceinline__ int node_id(const NodeBuild& P, int i) { return P.list ? P.list[i] : P.first + i; }

__device__ __forceinline__ int child_id(const NodeBuild& P, int node, int q) {
    const int tx = node % P.nodes_x, ty = node / P.nodes_x;
    return (ty * P.g + q / P.g) * P.child_nodes_x + tx * P.g + q % P.g;
}

__device__ __forceinline__ const uint16_t* child_mat(const NodeBuild& P, int node, int q) {
    return P.C.base + (size_t)child_id(P, node, q) * P.C.NP * P.C.NP;
}

__device__ __forceinline__ uint16_t* node_mat(const NodeBuild& P, int node) {
    return P.N.base + (size_t)node * P.N.NP * P.N.NP;
}

// Weight of seam candidate s of a node (INF: a cell is not passable).
__device__ __forceinline__ uint16_t seam_weight(const NodeBuild& P, int node, int s) {
    const int* e = P.seams + 6 * s;
    const int R0 = (node / P.nodes_x) * P.side, C0 = (node % P.nodes_x) * P.side;
    const size_t a = (size_t)(R0 + e[2]) * P.S + C0 + e[3], c = (size_t)(R0 + e[4]) * P.S + C0 + e[5];
    if (!P.pass[a] || !P.pass[c]) return INF;
    return P.wts ? edge_weight(P.wts[a], P.wts[c]) : (uint16_t)1;  // internal_node.cpp:160-161
}

// Largest number of active seams of the launch's nodes into *most.
__global__ void __launch_bounds__(128) seam_count_kernel(const NodeBuild P, int* most) {
    const int node = node_id(P, blockIdx.x);
    int c = 0;
    for (int s = threadIdx.x; s < P.n_seams; s += blockDim.x) c += seam_weight(P, node, s) < INF;
    c = __reduce_add_sync(FULL, c);
    __shared__ int w[4];
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(most, w[0] + w[1] + w[2] + w[3]);
}

// Seam edge record: x = qu | qv << 8, y = iu | iv << 16 (incidence rows in the
// two children), z = xu | xv << 16 (ports in the two children), w = weight.
// Incidence record: x = port | offset << 16, y = edge.

// Active seams of every node: its edges and each child's incidences.
__global__ void __launch_bounds__(256) seam_list_kernel(const NodeBuild P) {
    __shared__ int q_cnt[256];
    __shared__ int wtot[8];
    __shared__ int base;
    const int i = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (P.active && !P.active[i]) return;
    const int node = node_id(P, i), g2 = P.g * P.g;
    if (tid < g2) q_cnt[tid] = 0;
    if (tid == 0) base = 0;
    __syncthreads();
    int4* edge = P.edge + (size_t)i * P.TP;
    uint2* inc = P.inc + (size_t)i * g2 * P.capI;
    for (int s0 = 0; s0 < P.n_seams; s0 += 256) {
        const int s = s0 + tid;
        const uint16_t w = s < P.n_seams ? seam_weight(P, node, s) : INF;
        const bool on = w < INF;
        const unsigned bal = __ballot_sync(FULL, on);
        if (lane == 0) wtot[warp] = __popc(bal);
        __syncthreads();
        int e = base + __popc(bal & ((1u << lane) - 1u));
        for (int k = 0; k < warp; ++k) e += wtot[k];
        if (on) {
            const int u = P.seams[6 * s], v = P.seams[6 * s + 1];
            const int qu = u / P.nP, qv = v / P.nP, xu = u - qu * P.nP, xv = v - qv * P.nP;
            const int iu = atomicAdd(&q_cnt[qu], 1), iv = atomicAdd(&q_cnt[qv], 1);
            edge[e] = make_int4(qu | (qv << 8), iu | (iv << 16), xu | (xv << 16), w);
            inc[(size_t)qu * P.capI + iu] = make_uint2((unsigned)xu, (unsigned)e);
            inc[(size_t)qv * P.capI + iv] = make_uint2((unsigned)xv | ((unsigned)w << 16), (unsigned)e);
        }
        __syncthreads();
        if (tid == 0)
            for (int k = 0; k < 8; ++k) base += wtot[k];
        __syncthreads();
    }
    int* cnt = P.cnt + (size_t)i * (1 + g2);
    if (tid == 0) cnt[0] = base;
    if (tid < g2) cnt[1 + tid] = q_cnt[tid];
    if (tid < 4) P.vmax[4 * i + tid] = 0;
}

// R_q rows of every incidence (one warp per row) and the largest finite one.
__global__ void __launch_bounds__(kThreads) lift_rows_kernel(const NodeBuild P) {
    __shared__ int s_max;
    const int i = blockIdx.z, q = blockIdx.y, g2 = P.g * P.g;
    if (P.active && !P.active[i]) return;
    const int n = P.cnt[(size_t)i * (1 + g2) + 1 + q];
    if ((int)blockIdx.x * kWarps >= n) return;
    const int k = blockIdx.x * kWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) s_max = 0;
    __syncthreads();
    if (k < n) {
        const uint2 rec = P.inc[((size_t)i * g2 + q) * P.capI + k];
        const uint32_t o = rec.x >> 16;
        const uint16_t* crow = child_mat(P, node_id(P, i), q) + (size_t)P.cext[rec.x & 0xffffu] * P.C.NP;
        uint32_t* row = reinterpret_cast<uint32_t*>(P.R + (((size_t)i * g2 + q) * P.capI + k) * P.RP);
        uint32_t mx = 0;
        for (int j2 = lane; j2 < P.RP / 2; j2 += 32) {
            uint32_t v[2] = {INF, INF};
#pragma unroll
            for (int x = 0; x < 2; ++x)
                if (2 * j2 + x < P.nP) {
                    v[x] = sat_add(crow[P.cext[2 * j2 + x]], o);
                    if (v[x] < INF) mx = max(mx, v[x]);
                }
            row[j2] = v[0] | (v[1] << 16);
        }
        mx = __reduce_max_sync(FULL, mx);
        if (lane == 0) atomicMax(&s_max, (int)mx);
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_max) atomicMax(P.vmax + 4 * i, s_max);
}

// T0 in 64 x 64 tiles (INF beyond the node's edges, up to the 128-tile edge).
__global__ void __launch_bounds__(kThreads) seam_block_kernel(const NodeBuild P) {
    __shared__ int4 er[64], ec[64];
    const int i = blockIdx.y, g2 = P.g * P.g, tid = threadIdx.x;
    if (P.active && !P.active[i]) return;
    const int nE = P.cnt[(size_t)i * (1 + g2)];
    const int tiles = P.TP / 64, I = blockIdx.x / tiles, J = blockIdx.x % tiles;
    const int used = (nE + 127) / 128 * 128;
    if (I * 64 >= used || J * 64 >= used) return;
    const int4* edge = P.edge + (size_t)i * P.TP;
    if (tid < 64) {
        if (I * 64 + tid < nE) er[tid] = edge[I * 64 + tid];
    } else if (tid < 128) {
        if (J * 64 + tid - 64 < nE) ec[tid - 64] = edge[J * 64 + tid - 64];
    }
    __syncthreads();
    const uint16_t* R = P.R + (size_t)i * g2 * P.capI * P.RP;
    uint16_t* T = P.T + (size_t)i * P.TP * P.TP;
    for (int idx = tid; idx < 64 * 64; idx += kThreads) {
        const int a = idx >> 6, c = idx & 63;
        uint32_t v = INF;
        if (I * 64 + a < nE && J * 64 + c < nE) {
            const int4 r = er[a], k = ec[c];
            const int qr[2] = {r.x & 255, r.x >> 8}, qc[2] = {k.x & 255, k.x >> 8};
            const int ir[2] = {r.y & 0xffff, (int)((unsigned)r.y >> 16)};
            const int xc[2] = {k.z & 0xffff, (int)((unsigned)k.z >> 16)};
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int y = 0; y < 2; ++y)
                    if (qr[x] == qc[y])
                        v = min(v, sat_add(R[((size_t)qr[x] * P.capI + ir[x]) * P.RP + xc[y]], y ? (uint32_t)k.w : 0u));
        }
        T[(size_t)(I * 64 + a) * P.TP + J * 64 + c] = (uint16_t)v;
    }
}

// ---------------------------------------------------------------------------
// Min-plus product of one TM x TN tile (TM = 8 RW, TN = 64 CP, 8 warps):
//   acc[r][c] = min(acc[r][c], min_k A_k[row r] (+) B_k[column pair c]),  k < K
// A_k = arow(k) (8-column chunks from a_lim on are taken from the row's start:
// their results are not used), B_k = Bp + k ldb (b_lim alike).  Warp w owns
// rows RW w .. RW w + RW - 1, a lane CP column pairs.  Steps come in chunks of
// kKC, double-buffered: the A rows through registers, splatted so that a row
// value is one broadcast word, the B rows by cp.async.
// half: every finite operand is <= kHalfMax, INF is taken as kHalfInf and no
// sum needs a clamp (results >= kHalfInf mean INF).  Otherwise each step of a
// warp is skipped (its rows all INF), unclamped (all <= INF_HEADROOM) or clamped.
// ---------------------------------------------------------------------------
constexpr int kKC = 32;

template <int RW, int CP>
constexpr size_t tile_smem_bytes() {
    return 2 * (size_t)kKC * (8 * RW * sizeof(uint32_t) + 64 * CP * sizeof(uint16_t) + kWarps);
}

template <int RW, int CP, class ARow>
__device__ __forceinline__ void tile_minplus(uint32_t (&acc)[RW][CP], ARow arow, int a_lim, const uint16_t* Bp,
                                             size_t ldb, int b_lim, int K, bool half, unsigned char* smem) {
    constexpr int TM = 8 * RW, TN = 64 * CP;
    constexpr int NA = kKC * (TM / 8) / kThreads, NB = kKC * (TN / 8) / kThreads;
    static_assert(NA * kThreads == kKC * (TM / 8) && NB * kThreads == kKC * (TN / 8), "whole chunks per thread");
    uint32_t* As = reinterpret_cast<uint32_t*>(smem);
    uint16_t* Bs = reinterpret_cast<uint16_t*>(As + 2 * kKC * TM);
    uint8_t* cls = reinterpret_cast<uint8_t*>(Bs + 2 * kKC * TN);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n_c = (K + kKC - 1) / kKC;
    uint4 va[NA];
    auto load = [&](int c) {
#pragma unroll
        for (int x = 0; x < NA; ++x) {
            const int idx = tid + x * kThreads, k = c * kKC + idx / (TM / 8), c8 = (idx % (TM / 8)) * 8;
            va[x] = make_uint4(INF2, INF2, INF2, INF2);
            if (k < K) va[x] = *reinterpret_cast<const uint4*>(arow(k) + (c8 < a_lim ? c8 : 0));
        }
#pragma unroll
        for (int x = 0; x < NB; ++x) {
            const int idx = tid + x * kThreads, kk = idx / (TN / 8), c8 = (idx % (TN / 8)) * 8;
            if (c * kKC + kk < K)
                cp_async16(Bs + (size_t)((c & 1) * kKC + kk) * TN + c8,
                           Bp + (size_t)(c * kKC + kk) * ldb + (c8 < b_lim ? c8 : 0));
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    if (n_c > 0) load(0);
    for (int c = 0; c < n_c; ++c) {
        uint32_t* Ab = As + (c & 1) * kKC * TM;
        uint8_t* cb = cls + (c & 1) * kKC * kWarps;
#pragma unroll
        for (int x = 0; x < NA; ++x) {
            const int idx = tid + x * kThreads, kk = idx / (TM / 8), c8 = idx % (TM / 8);
            uint32_t w[4] = {va[x].x, va[x].y, va[x].z, va[x].w};
            if (half) {
#pragma unroll
                for (int t = 0; t < 4; ++t) w[t] = min2(w[t], kHalfInf2);
            } else {
                uint32_t mn = w[0], mx = w[0];
#pragma unroll
                for (int t = 1; t < 4; ++t) {
                    mn = min2(mn, w[t]);
                    mx = max2(mx, w[t]);
                }
                if constexpr (RW == 16) {  // a warp's rows are two neighbouring chunks
                    mn = min2(mn, __shfl_xor_sync(FULL, mn, 1));
                    mx = max2(mx, __shfl_xor_sync(FULL, mx, 1));
                }
                mn = min(mn & 0xffffu, mn >> 16);
                mx = max(mx & 0xffffu, mx >> 16);
                cb[kk * kWarps + c8 / (RW / 8)] = mn >= INF ? 0 : (mx <= INF_HEADROOM ? 1 : 2);
            }
            uint4* dst = reinterpret_cast<uint4*>(Ab + kk * TM + c8 * 8);
            dst[0] = make_uint4(splat(w[0]), splat(w[0] >> 16), splat(w[1]), splat(w[1] >> 16));
            dst[1] = make_uint4(splat(w[2]), splat(w[2] >> 16), splat(w[3]), splat(w[3] >> 16));
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();  // chunk c is staged; every warp is done with chunk c - 1
        if (c + 1 < n_c) load(c + 1);
        const int kn = min(kKC, K - c * kKC);
        const uint32_t* bp = reinterpret_cast<const uint32_t*>(Bs + (size_t)(c & 1) * kKC * TN) + lane * CP;
        const uint32_t* ap = Ab + warp * RW;
        auto step = [&](int k, auto mode) {
            constexpr int M = decltype(mode)::value;  // 0 half range, 1 unclamped, 2 clamped
            uint32_t bv[CP], av[RW];
#pragma unroll
            for (int cc = 0; cc < CP; ++cc) bv[cc] = bp[k * (TN / 2) + cc];
#pragma unroll
            for (int r4 = 0; r4 < RW / 4; ++r4) {
                const uint4 a4 = *reinterpret_cast<const uint4*>(ap + k * TM + 4 * r4);
                av[4 * r4] = a4.x;
                av[4 * r4 + 1] = a4.y;
                av[4 * r4 + 2] = a4.z;
                av[4 * r4 + 3] = a4.w;
            }
            if constexpr (M == 0) {
#pragma unroll
                for (int cc = 0; cc < CP; ++cc) bv[cc] = min2(bv[cc], kHalfInf2);
            }
#pragma unroll
            for (int r = 0; r < RW; ++r) {
                const uint32_t tt = INF2 - av[r];
#pragma unroll
                for (int cc = 0; cc < CP; ++cc) {
                    if constexpr (M == 2) acc[r][cc] = acc_clamp(acc[r][cc], bv[cc], av[r], tt);
                    else acc[r][cc] = acc_fast(acc[r][cc], bv[cc], av[r]);
                }
            }
        };
        if (half) {
#pragma unroll 4
            for (int k = 0; k < kn; ++k) step(k, std::integral_constant<int, 0>());
        } else {
            for (int k = 0; k < kn; ++k) {
                const int cl = cb[k * kWarps + warp];
                if (cl == 0) continue;  // uniform over the warp
                if (cl == 1) step(k, std::integral_constant<int, 1>());
                else step(k, std::integral_constant<int, 2>());
            }
        }
    }
    __syncthreads();  // the staging buffers are free
    if (half) {
#pragma unroll
        for (int r = 0; r < RW; ++r)
#pragma unroll
            for (int cc = 0; cc < CP; ++cc) {
                const uint32_t lo = acc[r][cc] & 0xffffu, hi = acc[r][cc] >> 16;
                acc[r][cc] = (lo >= kHalfInf ? (uint32_t)INF : lo) | ((hi >= kHalfInf ? (uint32_t)INF : hi) << 16);
            }
    }
}

// The tile transposed through shared memory: Tt[j][i] of TN x TM u16, in
// 16-byte chunks of 8 rows i.  Chunk q of row j sits at q ^ ((j / (2 CP)) & 7), so
// the 8 lanes of a 16-byte store phase (8 different rows) hit 8 different
// bank groups.  transposed_chunk reads chunk q of row j.
template <int RW, int CP>
__device__ __forceinline__ void transpose_store(uint16_t* Tt, const uint32_t (&acc)[RW][CP]) {
    constexpr int TM = 8 * RW;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int cc = 0; cc < CP; ++cc)
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const int j = lane * 2 * CP + 2 * cc + x;
            const int key = (j / (2 * CP)) & 7;
#pragma unroll
            for (int h = 0; h < RW / 8; ++h) {
                uint32_t w4[4];
#pragma unroll
                for (int t = 0; t < 4; ++t)
                    w4[t] = __byte_perm(acc[8 * h + 2 * t][cc], acc[8 * h + 2 * t + 1][cc], x ? 0x7632 : 0x5410);
                const int q = warp * (RW / 8) + h;
                *reinterpret_cast<uint4*>(Tt + j * TM + ((q ^ key) * 8)) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
            }
        }
}
template <int TM, int CP>
__device__ __forceinline__ uint4 transposed_chunk(const uint16_t* Tt, int j, int q) {
    return *reinterpret_cast<const uint4*>(Tt + j * TM + ((q ^ ((j / (2 * CP)) & 7)) * 8));
}

template <int RW, int CP>
__device__ __forceinline__ void fill_inf(uint32_t (&acc)[RW][CP]) {
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
        for (int c = 0; c < CP; ++c) acc[r][c] = INF2;
}

// ---------------------------------------------------------------------------
// Closure of T, stage t of one launch per stage: the panel units of round t
// (64-column tiles) and the update units of round t - 1 (upper-triangle tile
// pairs) side by side; a panel applies round t - 1's update to its own rows
// itself (from round t - 1's panel), so the two only meet at the next launch.
// The rows a panel reads may or may not hold that update yet: the minimum is
// the updated value either way.
// ---------------------------------------------------------------------------
constexpr size_t kStagePanelSmem = ((size_t)3 * B * kTLD + (size_t)B * 64) * sizeof(uint16_t) + (size_t)B * kWarps;

__device__ void stage_panel(const NodeBuild& P, int i, int nE, int j0, int t, unsigned char* smem) {
    uint16_t (*Ts)[kTLD] = reinterpret_cast<uint16_t (*)[kTLD]>(smem);
    uint16_t (*Ag)[kTLD] = Ts + B;  // old panel at the pivot columns
    uint16_t (*Bt)[kTLD] = Ag + B;  // the tile's pivot rows
    uint16_t* Pj = &Bt[B][0];       // old panel at the tile's columns
    uint8_t* cls = reinterpret_cast<uint8_t*>(Pj + B * 64);
    const int tid = threadIdx.x, TP = P.TP, k0 = t * B, mk = min(B, nE - k0);
    const bool ahead = t > 0;
    const uint16_t* T = P.T + (size_t)i * TP * TP;
    const uint16_t* Pp = P.P + ((size_t)((t - 1) & 1) * P.n + i) * B * TP;
    for (int idx = tid; idx < B * 8; idx += kThreads) {
        const int a = idx >> 3, c = (idx & 7) * 8;
        cp_async16(&Ts[a][c], T + (size_t)(k0 + a) * TP + k0 + c);
        cp_async16(&Bt[a][c], T + (size_t)(k0 + a) * TP + j0 + c);
        if (ahead) {
            cp_async16(&Ag[a][c], Pp + (size_t)a * TP + k0 + c);
            cp_async16(Pj + a * 64 + c, Pp + (size_t)a * TP + j0 + c);
        }
    }
    cp_async_wait_all();
    __syncthreads();
    if (ahead) {
        uint32_t acc[2][4];
        block_classes(Ag, B, cls);
        __syncthreads();
        gemm64(Ag, &Ag[0][0], kTLD, B, cls, acc);
        min_into(&Ts[0][0], kTLD, B, acc);
        gemm64(Ag, Pj, 64, B, cls, acc);
        min_into(&Bt[0][0], kTLD, B, acc);
        __syncthreads();
    }
    uint32_t vb[8];
    close_pivot_panel(Ts, Bt, mk, vb);
    uint16_t* out = P.P + ((size_t)(t & 1) * P.n + i) * B * TP;
    const int a = tid >> 2, c0 = (tid & 3) * 16;
    uint4* dst = reinterpret_cast<uint4*>(out + (size_t)a * TP + j0 + c0);
    if (a >= mk) {
#pragma unroll
        for (int x = 0; x < 8; ++x) vb[x] = INF2;
    }
    dst[0] = make_uint4(vb[0], vb[1], vb[2], vb[3]);
    dst[1] = make_uint4(vb[4], vb[5], vb[6], vb[7]);
}

template <int RW, int CP>
__device__ void stage_update(const NodeBuild& P, int i, int nE, int I, int J, int t, unsigned char* smem) {
    constexpr int TT = 8 * RW;
    static_assert(TT == 64 * CP, "square tiles");
    const int TP = P.TP, mk = min(B, nE - t * B);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint16_t* T = P.T + (size_t)i * TP * TP;
    const uint16_t* Pp = P.P + ((size_t)(t & 1) * P.n + i) * B * TP;
    uint32_t acc[RW][CP];
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        const uint32_t* row = reinterpret_cast<const uint32_t*>(T + (size_t)(I * TT + warp * RW + r) * TP + J * TT);
#pragma unroll
        for (int c = 0; c < CP; ++c) acc[r][c] = row[lane * CP + c];
    }
    tile_minplus<RW, CP>(acc, [&](int k) { return Pp + (size_t)k * TP + I * TT; }, TP - I * TT, Pp + J * TT, TP,
                         TP - J * TT, mk, false, smem);
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        uint32_t* row = reinterpret_cast<uint32_t*>(T + (size_t)(I * TT + warp * RW + r) * TP + J * TT);
#pragma unroll
        for (int c = 0; c < CP; ++c) row[lane * CP + c] = acc[r][c];
    }
    if (I == J) return;
    uint16_t* Tt = reinterpret_cast<uint16_t*>(smem);
    transpose_store<RW, CP>(Tt, acc);
    __syncthreads();
    for (int idx = threadIdx.x; idx < TT * (TT / 8); idx += kThreads) {
        const int j = idx / (TT / 8), q = idx % (TT / 8);
        reinterpret_cast<uint4*>(T + (size_t)(J * TT + j) * TP + I * TT)[q] = transposed_chunk<TT, CP>(Tt, j, q);
    }
}

__global__ void __launch_bounds__(kThreads, 2) seam_stage_kernel(const NodeBuild P, int t) {
    extern __shared__ __align__(16) unsigned char nsm[];
    const int i = blockIdx.y;
    if (P.active && !P.active[i]) return;
    const int nE = P.cnt[(size_t)i * (1 + P.g * P.g)];
    const int rounds = (nE + B - 1) / B;
    if (t > rounds) return;
    // the panel covers whole update tiles
    const int n_panel = t < rounds ? (P.TP >= 128 ? (nE + 127) / 128 * 2 : 1) : 0;
    int u = blockIdx.x;
    if (u < n_panel) {
        stage_panel(P, i, nE, u * 64, t, nsm);
        return;
    }
    u -= n_panel;
    const int TT = P.TP >= 128 ? 128 : 64;
    const int nt = (nE + TT - 1) / TT;
    if (t == 0 || u >= nt * (nt + 1) / 2) return;
    int I, J;
    tri_pair(u, nt, I, J);
    if (TT == 128) stage_update<16, 2>(P, i, nE, I, J, t - 1, nsm);
    else stage_update<8, 1>(P, i, nE, I, J, t - 1, nsm);
}

// Largest finite value of every node's T (one 64-row strip per CTA).
__global__ void __launch_bounds__(kThreads) seam_max_kernel(const NodeBuild P) {
    const int i = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (P.active && !P.active[i]) return;
    const int nE = P.cnt[(size_t)i * (1 + P.g * P.g)];
    const uint16_t* T = P.T + (size_t)i * P.TP * P.TP;
    uint32_t mx = 0;
    for (int r = blockIdx.x * 64 + warp; r < min(nE, (int)blockIdx.x * 64 + 64); r += kWarps)
        for (int c = lane * 8; c < nE; c += 256) {
            const uint4 v = *reinterpret_cast<const uint4*>(T + (size_t)r * P.TP + c);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const uint32_t lo = w[t] & 0xffffu, hi = w[t] >> 16;
                if (lo < INF) mx = max(mx, lo);
                if (hi < INF) mx = max(mx, hi);
            }
        }
    mx = __reduce_max_sync(FULL, mx);
    if (lane == 0 && mx) atomicMax(P.vmax + 4 * i + 1, (int)mx);
}

// U_p tiles: rows = edges, columns = ports of child p.
template <int RW, int CP>
__global__ void __launch_bounds__(kThreads, 2) lift_kernel(const NodeBuild P) {
    constexpr int TM = 8 * RW, TN = 64 * CP;
    extern __shared__ __align__(16) unsigned char nsm[];
    __shared__ int s_max;
    const int i = blockIdx.z, p = blockIdx.y, g2 = P.g * P.g;
    if (P.active && !P.active[i]) return;
    const int* cnt = P.cnt + (size_t)i * (1 + g2);
    const int tn = (P.RP + TN - 1) / TN;
    const int m0 = (blockIdx.x / tn) * TM, n0 = (blockIdx.x % tn) * TN;
    if (m0 >= cnt[0]) return;
    const int* vm = P.vmax + 4 * i;
    const bool half = max(vm[0], vm[1]) <= kHalfMax;
    const uint2* inc = P.inc + ((size_t)i * g2 + p) * P.capI;
    const uint16_t* T = P.T + (size_t)i * P.TP * P.TP;
    const uint16_t* R = P.R + ((size_t)i * g2 + p) * P.capI * P.RP;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t acc[RW][CP];
    fill_inf<RW, CP>(acc);
    if (threadIdx.x == 0) s_max = 0;
    tile_minplus<RW, CP>(acc, [&](int k) { return T + (size_t)inc[k].y * P.TP + m0; }, P.TP - m0, R + n0, P.RP,
                         P.RP - n0, cnt[1 + p], half, nsm);
    uint16_t* U = P.U + ((size_t)i * g2 + p) * P.TP * P.RP;
    uint32_t mx = 0;
    const int col = n0 + lane * 2 * CP;
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        const int e = m0 + warp * RW + r;
#pragma unroll
        for (int c = 0; c < CP; ++c) {
            if (col + 2 * c >= P.RP) continue;
            *reinterpret_cast<uint32_t*>(U + (size_t)e * P.RP + col + 2 * c) = acc[r][c];
            const uint32_t lo = acc[r][c] & 0xffffu, hi = acc[r][c] >> 16;
            if (lo < INF) mx = max(mx, lo);
            if (hi < INF) mx = max(mx, hi);
        }
    }
    mx = __reduce_max_sync(FULL, mx);
    __syncthreads();
    if (lane == 0 && mx) atomicMax(&s_max, (int)mx);
    __syncthreads();
    if (threadIdx.x == 0 && s_max) atomicMax(P.vmax + 4 * i + 2, s_max);
}

// D tiles: unit = (children p <= q, tile of p's ports x tile of q's ports).
template <int RW, int CP>
__global__ void __launch_bounds__(kThreads, 2) node_tile_kernel(const NodeBuild P) {
    constexpr int TM = 8 * RW, TN = 64 * CP;
    static_assert(TM == TN, "square tiles");
    extern __shared__ __align__(16) unsigned char nsm[];
    __shared__ int s_chg;
    const int i = blockIdx.y, g2 = P.g * P.g, nP = P.nP, NP = P.N.NP;
    if (P.active && !P.active[i]) return;
    const int nt = (nP + TM - 1) / TM, tri = nt * (nt + 1) / 2;
    int u = blockIdx.x, p, q, I, J;
    if (u < g2 * tri) {  // p == q: the upper triangle
        p = q = u / tri;
        tri_pair(u % tri, nt, I, J);
    } else {
        u -= g2 * tri;
        tri_pair(u / (nt * nt), g2 - 1, p, q);  // pairs p < q as (p, q - 1) with p <= q - 1
        ++q;
        I = u % (nt * nt) / nt;
        J = u % nt;
    }
    const int node = node_id(P, i), m0 = I * TM, n0 = J * TN;
    const int* vm = P.vmax + 4 * i;
    const bool half = max(vm[0], vm[2]) <= kHalfMax;
    const uint2* inc = P.inc + ((size_t)i * g2 + q) * P.capI;
    const uint16_t* U = P.U + ((size_t)i * g2 + p) * P.TP * P.RP + m0;
    const uint16_t* R = P.R + ((size_t)i * g2 + q) * P.capI * P.RP + n0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t acc[RW][CP];
    fill_inf<RW, CP>(acc);
    if (threadIdx.x == 0) s_chg = 0;
    tile_minplus<RW, CP>(acc, [&](int k) { return U + (size_t)inc[k].y * P.RP; }, P.RP - m0, R, P.RP, P.RP - n0,
                         P.cnt[(size_t)i * (1 + g2) + 1 + q], half, nsm);
    uint16_t* D = node_mat(P, node);
    const int col = n0 + lane * 2 * CP;  // port of q; nP is a multiple of 4
    if (p == q) {
        const uint16_t* cm = child_mat(P, node, p);
        int ce[2 * CP];
#pragma unroll
        for (int c = 0; c < 2 * CP; ++c) ce[c] = P.cext[min(col + c, nP - 1)];
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            const uint16_t* crow = cm + (size_t)P.cext[min(m0 + warp * RW + r, nP - 1)] * P.C.NP;
#pragma unroll
            for (int c = 0; c < CP; ++c)
                acc[r][c] = min2(acc[r][c], (uint32_t)crow[ce[2 * c]] | ((uint32_t)crow[ce[2 * c + 1]] << 16));
        }
    }
    bool chg = false;
    if (col < nP) {
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            const int row = m0 + warp * RW + r;
            if (row >= nP) continue;
            uint32_t* d = reinterpret_cast<uint32_t*>(D + (size_t)(p * nP + row) * NP + q * nP + col);
            if (P.changed && P.isext[p * nP + row]) {
#pragma unroll
                for (int c = 0; c < CP; ++c) {
                    const uint32_t diff = d[c] ^ acc[r][c];
                    chg |= (diff & 0xffffu) && P.isext[q * nP + col + 2 * c];
                    chg |= (diff >> 16) && P.isext[q * nP + col + 2 * c + 1];
                }
            }
            if constexpr (CP == 2) *reinterpret_cast<uint2*>(d) = make_uint2(acc[r][0], acc[r][1]);
            else d[0] = acc[r][0];
        }
    }
    if (P.changed) {
        if (chg) s_chg = 1;
        __syncthreads();
        if (threadIdx.x == 0 && s_chg) P.changed[P.parent[i]] = 1;
    }
    if (p == q && I == J) return;
    uint16_t* Tt = reinterpret_cast<uint16_t*>(nsm);
    transpose_store<RW, CP>(Tt, acc);
    __syncthreads();
    for (int idx = threadIdx.x; idx < TN * (TM / 8); idx += kThreads) {
        const int j = idx / (TM / 8), c8 = idx % (TM / 8);
        if (n0 + j >= nP || m0 + c8 * 8 >= nP) continue;
        const uint4 v = transposed_chunk<TM, CP>(Tt, j, c8);
        uint2* d = reinterpret_cast<uint2*>(D + (size_t)(q * nP + n0 + j) * NP + p * nP + m0 + c8 * 8);
        d[0] = make_uint2(v.x, v.y);
        if (m0 + c8 * 8 + 4 < nP) d[1] = make_uint2(v.z, v.w);
    }
}

// ---------------------------------------------------------------------------
// Nodes with at most 64 seams and 64 ports per child (the lowest levels, of
// which there are thousands): one CTA does a whole node in shared memory.
// LC lanes hold the column pairs of a child (16 for up to 32 ports).
// ---------------------------------------------------------------------------
constexpr int kSmallSeams = 64, kSmallPorts = 64;

struct SmallLayout {
    int RP, ldU;  // row strides of R and U (multiples of 8)
    size_t o_inc, o_R, o_T, o_U, total;
};
__host__ __device__ inline SmallLayout small_layout(int g2, int nP, int capI) {
    SmallLayout L;
    L.RP = (nP + 7) / 8 * 8;
    L.ldU = (g2 * nP + 15) / 8 * 8;
    size_t o = kSmallSeams * sizeof(int4);
    L.o_inc = o;
    o += (size_t)g2 * capI * sizeof(uint2);
    o = (o + 15) / 16 * 16;
    L.o_R = o;
    o += (size_t)g2 * capI * L.RP * sizeof(uint16_t);
    L.o_T = o;
    o += (size_t)B * kTLD * sizeof(uint16_t);
    L.o_U = o;
    o += (size_t)kSmallSeams * L.ldU * sizeof(uint16_t);
    L.total = o;
    return L;
}

template <int LC>
__global__ void __launch_bounds__(kThreads) node_small_kernel(const NodeBuild P) {
    extern __shared__ __align__(16) unsigned char nsm[];
    __shared__ int q_cnt[256];
    __shared__ int s_w0, s_nE, s_chg;
    const int i = blockIdx.x, g2 = P.g * P.g, nP = P.nP, NP = P.N.NP;
    if (P.active && !P.active[i]) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const SmallLayout L = small_layout(g2, nP, P.capI);
    int4* edge = reinterpret_cast<int4*>(nsm);
    uint2* inc = reinterpret_cast<uint2*>(nsm + L.o_inc);
    uint16_t* R = reinterpret_cast<uint16_t*>(nsm + L.o_R);
    uint16_t (*T)[kTLD] = reinterpret_cast<uint16_t (*)[kTLD]>(nsm + L.o_T);
    uint16_t* U = reinterpret_cast<uint16_t*>(nsm + L.o_U);
    const int node = node_id(P, i);
    if (tid < g2) q_cnt[tid] = 0;
    if (tid == 0) s_chg = 0;
    uint16_t w = INF;
    unsigned bal = 0;
    if (tid < kSmallSeams) {
        if (tid < P.n_seams) w = seam_weight(P, node, tid);
        bal = __ballot_sync(FULL, w < INF);
        if (tid == 0) s_w0 = __popc(bal);
        if (tid == 32) s_nE = __popc(bal);
    }
    __syncthreads();
    if (w < INF) {
        const int e = (warp ? s_w0 : 0) + __popc(bal & ((1u << lane) - 1u));
        const int u = P.seams[6 * tid], v = P.seams[6 * tid + 1];
        const int qu = u / nP, qv = v / nP, xu = u - qu * nP, xv = v - qv * nP;
        const int iu = atomicAdd(&q_cnt[qu], 1), iv = atomicAdd(&q_cnt[qv], 1);
        edge[e] = make_int4(qu | (qv << 8), iu | (iv << 16), xu | (xv << 16), w);
        inc[qu * P.capI + iu] = make_uint2((unsigned)xu, (unsigned)e);
        inc[qv * P.capI + iv] = make_uint2((unsigned)xv | ((unsigned)w << 16), (unsigned)e);
    }
    __syncthreads();
    const int nE = s_w0 + s_nE;
    for (int q = 0; q < g2; ++q) {
        const uint16_t* cm = child_mat(P, node, q);
        for (int k = warp; k < q_cnt[q]; k += kWarps) {
            const uint2 rec = inc[q * P.capI + k];
            const uint16_t* crow = cm + (size_t)P.cext[rec.x & 0xffffu] * P.C.NP;
            for (int j = lane; j < L.RP; j += 32)
                R[(q * P.capI + k) * L.RP + j] = j < nP ? (uint16_t)sat_add(crow[P.cext[j]], rec.x >> 16) : INF;
        }
    }
    __syncthreads();
    for (int idx = tid; idx < B * B; idx += kThreads) {
        const int a = idx >> 6, c = idx & 63;
        uint32_t v = INF;
        if (a < nE && c < nE) {
            const int4 r = edge[a], k = edge[c];
            const int qr[2] = {r.x & 255, r.x >> 8}, qc[2] = {k.x & 255, k.x >> 8};
            const int ir[2] = {r.y & 0xffff, (int)((unsigned)r.y >> 16)};
            const int xc[2] = {k.z & 0xffff, (int)((unsigned)k.z >> 16)};
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int y = 0; y < 2; ++y)
                    if (qr[x] == qc[y])
                        v = min(v, sat_add(R[(qr[x] * P.capI + ir[x]) * L.RP + xc[y]], y ? (uint32_t)k.w : 0u));
        }
        T[a][c] = (uint16_t)v;
    }
    __syncthreads();
    close_pivot_block(T, nE);
    __syncthreads();
    // sub-warps of LC lanes; a lane holds one column pair of a child
    constexpr int kSub = 32 / LC, kSubs = kWarps * kSub;
    const int sub = warp * kSub + lane / LC, cl = lane % LC;
    const bool col_ok = 2 * cl < nP;
    {   // U: items of 4 edges x one child
        const int ng = (nE + 3) / 4;
        for (int it = sub; it < ng * g2; it += kSubs) {
            const int p = it / ng, e0 = (it - p * ng) * 4;
            uint32_t acc[4] = {INF2, INF2, INF2, INF2};
            for (int k = 0; k < q_cnt[p]; ++k) {
                const uint2 a = *reinterpret_cast<const uint2*>(&T[inc[p * P.capI + k].y][e0]);
                const uint32_t bv = reinterpret_cast<const uint32_t*>(R + (p * P.capI + k) * L.RP)[col_ok ? cl : 0];
                const uint32_t av[4] = {splat(a.x), splat(a.x >> 16), splat(a.y), splat(a.y >> 16)};
#pragma unroll
                for (int r = 0; r < 4; ++r) acc[r] = acc_clamp(acc[r], bv, av[r], INF2 - av[r]);
            }
            if (col_ok) {
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    reinterpret_cast<uint32_t*>(U + (e0 + r) * L.ldU + p * nP)[cl] = acc[r];
            }
        }
    }
    __syncthreads();
    // D: items of 8 rows i (children 0 .. q) x the columns of child q
    uint16_t* D = node_mat(P, node);
    bool chg = false;
    int q = 0, first = 0, ng = (nP + 7) / 8;  // items [first, first + ng) belong to q
    for (int it = sub;; it += kSubs) {
        while (q < g2 && it >= first + ng) {
            first += ng;
            ++q;
            ng = ((q + 1) * nP + 7) / 8;
        }
        if (q >= g2) break;
        const int i0 = (it - first) * 8;
        uint32_t acc[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) acc[r] = INF2;
        for (int k = 0; k < q_cnt[q]; ++k) {
            const uint4 a = *reinterpret_cast<const uint4*>(U + inc[q * P.capI + k].y * L.ldU + i0);
            const uint32_t bv = reinterpret_cast<const uint32_t*>(R + (q * P.capI + k) * L.RP)[col_ok ? cl : 0];
            const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
            for (int r2 = 0; r2 < 4; ++r2) {
                const uint32_t lo = splat(aw[r2]), hi = splat(aw[r2] >> 16);
                acc[2 * r2] = acc_clamp(acc[2 * r2], bv, lo, INF2 - lo);
                acc[2 * r2 + 1] = acc_clamp(acc[2 * r2 + 1], bv, hi, INF2 - hi);
            }
        }
        if (!col_ok) continue;
        const int lo = q * nP, hi = lo + nP, col = lo + 2 * cl;
        const uint16_t* cm = child_mat(P, node, q);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int row = i0 + r;
            if (row >= hi) continue;
            if (row >= lo) {
                const uint16_t* crow = cm + (size_t)P.cext[row - lo] * P.C.NP;
                acc[r] = min2(acc[r], (uint32_t)crow[P.cext[2 * cl]] | ((uint32_t)crow[P.cext[2 * cl + 1]] << 16));
            }
            uint32_t* d = reinterpret_cast<uint32_t*>(D + (size_t)row * NP + col);
            if (P.changed && P.isext[row]) {
                const uint32_t diff = *d ^ acc[r];
                chg |= (diff & 0xffffu) && P.isext[col];
                chg |= (diff >> 16) && P.isext[col + 1];
            }
            *d = acc[r];
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // the transposed entries of the other children (lo is a multiple of 4)
            if (i0 + 4 * h >= lo) continue;
#pragma unroll
            for (int x = 0; x < 2; ++x)
                *reinterpret_cast<uint2*>(D + (size_t)(col + x) * NP + i0 + 4 * h) =
                    make_uint2(__byte_perm(acc[4 * h], acc[4 * h + 1], x ? 0x7632 : 0x5410),
                               __byte_perm(acc[4 * h + 2], acc[4 * h + 3], x ? 0x7632 : 0x5410));
        }
    }
    if (P.changed) {
        if (chg) s_chg = 1;
        __syncthreads();
        if (tid == 0 && s_chg) P.changed[P.parent[i]] = 1;
    }
}

// INF in the padding of `count` matrices: rows and columns n .. NP - 1.
__global__ void pad_fill_kernel(MatSet M, int y0) {
    const int NP = M.NP, n = M.n, strip = NP - n;
    uint16_t* D = M.base + (size_t)(y0 + blockIdx.y) * NP * NP;
    const size_t side = (size_t)n * strip, total = side + (size_t)strip * NP;
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        if (e < side) D[(e / strip) * NP + n + e % strip] = INF;
        else D[(size_t)n * NP + (e - side)] = INF;
    }
}

constexpr int kMaxGridY = 65535;
inline unsigned blocks_for(size_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

template <class K>
void allow_smem(K kernel, size_t bytes) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

}  // namespace

void launch_pad_fill(MatSet M, int count, cudaStream_t st) {
    if (M.NP == M.n) return;
    const size_t e = (size_t)(M.NP - M.n) * (M.NP + M.n);
    for (int y0 = 0; y0 < count; y0 += kMaxGridY)
        pad_fill_kernel<<<dim3(std::min(64u, blocks_for(e, 256)), std::min(kMaxGridY, count - y0)), 256, 0, st>>>(M, y0);
}

bool node_build_small(const NodeBuild& P) {
    return P.n_seams <= kSmallSeams && P.nP <= kSmallPorts &&
           small_layout(P.g * P.g, P.nP, P.capI).total <= 100 * 1024;
}

size_t node_build_layout(NodeBuild& P, int n, unsigned char* base) {
    const size_t g2 = (size_t)P.g * P.g;
    P.n = n;
    P.TP = P.n_seams <= 64 ? 64 : (P.n_seams + 127) / 128 * 128;
    P.RP = (P.nP + 7) / 8 * 8;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        unsigned char* p = base + off;
        off += (bytes + 255) / 256 * 256;
        return p;
    };
    P.cnt = reinterpret_cast<int*>(take(n * (1 + g2) * sizeof(int)));
    P.vmax = reinterpret_cast<int*>(take((size_t)n * 4 * sizeof(int)));
    P.edge = reinterpret_cast<int4*>(take((size_t)n * P.TP * sizeof(int4)));
    P.inc = reinterpret_cast<uint2*>(take(n * g2 * P.capI * sizeof(uint2)));
    P.R = reinterpret_cast<uint16_t*>(take(n * g2 * P.capI * P.RP * sizeof(uint16_t)));
    P.T = reinterpret_cast<uint16_t*>(take((size_t)n * P.TP * P.TP * sizeof(uint16_t)));
    P.P = reinterpret_cast<uint16_t*>(take((size_t)2 * n * B * P.TP * sizeof(uint16_t)));
    P.U = reinterpret_cast<uint16_t*>(take(n * g2 * P.TP * P.RP * sizeof(uint16_t)));
    return off;
}

void launch_seam_count(const NodeBuild& P, int n, int* most, cudaStream_t st) {
    if (n > 0) seam_count_kernel<<<n, 128, 0, st>>>(P, most);
}

void launch_node_build(const NodeBuild& P, int n, int most_seams, cudaStream_t st) {
    if (n <= 0) return;
    const int g2 = P.g * P.g;
    if (node_build_small(P)) {
        const size_t smem = small_layout(g2, P.nP, P.capI).total;
        if (P.nP <= 32) {
            allow_smem(node_small_kernel<16>, smem);
            node_small_kernel<16><<<n, kThreads, smem, st>>>(P);
        } else {
            allow_smem(node_small_kernel<32>, smem);
            node_small_kernel<32><<<n, kThreads, smem, st>>>(P);
        }
        return;
    }
    seam_list_kernel<<<n, 256, 0, st>>>(P);
    const int cap = std::min(P.capI, most_seams);  // a child's incidences are distinct edges
    const int rounds = (most_seams + B - 1) / B;
    if (rounds > 0) {
        lift_rows_kernel<<<dim3(blocks_for(cap, kWarps), g2, n), kThreads, 0, st>>>(P);
        const unsigned tiles = P.TP / 64;
        seam_block_kernel<<<dim3(tiles * tiles, n), kThreads, 0, st>>>(P);
        const size_t smem = std::max(kStagePanelSmem, tile_smem_bytes<16, 2>());
        allow_smem(seam_stage_kernel, smem);
        const int nt = P.TP >= 128 ? (most_seams + 127) / 128 : 1;
        for (int t = 0; t <= rounds; ++t) {
            const int units = (t < rounds ? (P.TP >= 128 ? 2 * nt : 1) : 0) + (t > 0 ? nt * (nt + 1) / 2 : 0);
            seam_stage_kernel<<<dim3(units, n), kThreads, smem, st>>>(P, t);
        }
        seam_max_kernel<<<dim3(rounds, n), kThreads, 0, st>>>(P);
        // 64-wide tiles for children of up to 64 ports
        if (P.nP <= 64) {
            const size_t sm = tile_smem_bytes<8, 1>();
            lift_kernel<8, 1><<<dim3(blocks_for(most_seams, 64) * blocks_for(P.RP, 64), g2, n), kThreads, sm, st>>>(P);
        } else {
            const size_t sm = tile_smem_bytes<16, 2>();
            allow_smem(lift_kernel<16, 2>, sm);
            lift_kernel<16, 2><<<dim3(blocks_for(most_seams, 128) * blocks_for(P.RP, 128), g2, n), kThreads, sm, st>>>(P);
        }
    }
    const int TM = P.nP <= 64 ? 64 : 128;
    const int nt = (P.nP + TM - 1) / TM;
    const dim3 grid(g2 * nt * (nt + 1) / 2 + g2 * (g2 - 1) / 2 * nt * nt, n);
    if (P.nP <= 64) {
        node_tile_kernel<8, 1><<<grid, kThreads, tile_smem_bytes<8, 1>(), st>>>(P);
    } else {
        allow_smem(node_tile_kernel<16, 2>, tile_smem_bytes<16, 2>());
        node_tile_kernel<16, 2><<<grid, kThreads, tile_smem_bytes<16, 2>(), st>>>(P);
    }
}

}  // namespace hb
