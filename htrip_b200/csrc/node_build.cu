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
//   T  = closure of T0 (repeated squaring)
//   U_p[e][i]  = min_k T[e][e_k] (+) R_p[k][i]            (k over child p's)
//   D[i][j]    = min([p == q] S_p[i][j], min_k U_p[e_k][i] (+) R_q[k][j])
//                for i in child p, j in child q, p <= q, and transposed.
// Every sum is the exact clamped tropical product and the closure is unique,
// so D equals the reference's sequential relaxation over the seam endpoints
// bit for bit; each matrix is written once instead of once per 64 pivots.
// Measured against the blocked closure over the seam endpoints that it
// replaces (device time, B200): building a 1024 x 1024 street map, b = 8, 22.8 ->
// 4.6 ms; one weight change on a 256 x 256 map, b = 8, 2.45 -> 0.42 ms.
#include "closure.cuh"
#include "kernels.cuh"

#include <algorithm>
#include <type_traits>

namespace hb {

namespace {

constexpr unsigned FULL = 0xffffffffu;

// Half range (closure.cuh): distances of at most kHalfMax add up below kHalfInf, so
// with INF replaced by kHalfInf a sum needs no clamp: it never wraps (65534 at most)
// and a sum of kHalfInf or more means INF.

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

// Seam edge record: x = qu | qv << 8, y = iu | iv << 16 (incidence rows in the
// two children), z = xu | xv << 16 (ports in the two children), w = weight.
// Incidence record: x = port | offset << 16, y = edge.

// Active seams of every node: its edges and each child's incidences.
__global__ void __launch_bounds__(1024) seam_list_kernel(const NodeBuild P) {
    __shared__ int q_cnt[256];
    __shared__ int wtot[32];
    __shared__ int base;
    const int i = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
    if (P.active && !P.active[i]) return;
    const int node = node_id(P, i), g2 = P.g * P.g;
    for (int q = tid; q < g2; q += blockDim.x) q_cnt[q] = 0;
    if (tid == 0) base = 0;
    __syncthreads();
    int4* edge = P.edge + (size_t)i * P.TP;
    uint2* inc = P.inc + (size_t)i * g2 * P.capI;
    for (int s0 = 0; s0 < P.n_seams; s0 += blockDim.x) {
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
            for (int k = 0; k < nw; ++k) base += wtot[k];
        __syncthreads();
    }
    int* cnt = P.cnt + (size_t)i * (1 + g2);
    if (tid == 0) cnt[0] = base;
    for (int q = tid; q < g2; q += blockDim.x) cnt[1 + q] = q_cnt[q];
    if (tid < kNodeState) P.state[kNodeState * i + tid] = 0;
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
    if (threadIdx.x == 0 && s_max) atomicMax(P.state + kNodeState * i, s_max);
}

// T0 in 16 x 64 tiles (INF beyond the node's edges, up to the 128-tile edge)
// and its largest finite value.
__global__ void __launch_bounds__(kThreads) seam_block_kernel(const NodeBuild P) {
    __shared__ int4 er[16], ec[64];
    __shared__ int s_max;
    const int i = blockIdx.y, g2 = P.g * P.g, tid = threadIdx.x;
    if (P.active && !P.active[i]) return;
    const int nE = P.cnt[(size_t)i * (1 + g2)];
    const int tiles = P.TP / 64, I = blockIdx.x / tiles, J = blockIdx.x % tiles;
    const int used = min(P.TP, (nE + 127) / 128 * 128);
    if (I * 16 >= used || J * 64 >= used) return;
    const int4* edge = P.edge + (size_t)i * P.TP;
    if (tid < 16) {
        if (I * 16 + tid < nE) er[tid] = edge[I * 16 + tid];
    } else if (tid >= 64 && tid < 128) {
        if (J * 64 + tid - 64 < nE) ec[tid - 64] = edge[J * 64 + tid - 64];
    }
    if (tid == 0) s_max = 0;
    __syncthreads();
    const uint16_t* R = P.R + (size_t)i * g2 * P.capI * P.RP;
    uint16_t* T = P.T + (size_t)i * P.TP * P.TP;
    uint32_t mx = 0;
#pragma unroll
    for (int x4 = 0; x4 < 4; ++x4) {
        const int a = (tid >> 6) + 4 * x4, c = tid & 63;
        uint32_t v = INF;
        if (I * 16 + a < nE && J * 64 + c < nE) {
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
        T[(size_t)(I * 16 + a) * P.TP + J * 64 + c] = (uint16_t)v;
        if (v < INF) mx = max(mx, v);
    }
    mx = __reduce_max_sync(FULL, mx);
    if ((tid & 31) == 0 && mx) atomicMax(&s_max, (int)mx);
    __syncthreads();
    if (tid == 0 && s_max) atomicMax(P.state + kNodeState * i + 1, s_max);
}

// ---------------------------------------------------------------------------
// Min-plus product of one TM x TN tile (TM = W RW, TN = 64 CP, W warps):
//   acc[r][c] = min(acc[r][c], min_k A[arow(k)][row r] (+) Bp[k][column pair c]),  k < K
// (8-column chunks of an operand row from a_lim / b_lim on are taken from its
// start: their results are not used).  Warp w owns rows RW w .. RW w + RW - 1, a
// lane CP column pairs.  Steps come in chunks of kKC rows; kDepth chunks are in
// flight by cp.async (one chunk takes about 1000 cycles to use, less than its
// L2 round trip), and the gather index of a row is loaded a chunk before its row.
// Each thread splats the A values it copied itself, so that a row value is one
// broadcast word of 32 bits: no barrier between arrival and splat.
// half: every finite operand is <= kHalfMax, INF is taken as kHalfInf and no
// sum needs a clamp (results >= kHalfInf mean INF).  Otherwise each step of a
// warp is skipped (its rows all INF), unclamped (all <= INF_HEADROOM) or clamped.
// KS = 2: two groups of W warps take half of every chunk's steps each and trade
// halves of their rows at the end, so 64 x 64 tiles (of which there are few
// when a closure or a single node is all there is to do) have 8 warps to hide
// latencies: a closure pass over 390 seams, 16 nodes, 48 -> 44 us, over 195, 64 nodes, 33 -> 25 us.
// Ends with this warp's rows of the result in out: rows first_row() and on.
// ---------------------------------------------------------------------------
constexpr int kKC = 32;
constexpr int kDepth = 3;

template <int RW, int CP, int W>
constexpr size_t tile_smem_bytes() {
    return (size_t)kKC * (2 * W * RW * sizeof(uint32_t) + kDepth * (W * RW + 64 * CP) * sizeof(uint16_t) + 2 * W);
}

template <int RW, int W, int KS>
__device__ __forceinline__ int first_row() {
    const int warp = threadIdx.x >> 5;
    return (warp % W) * RW + (warp / W) * (RW / KS);
}

template <int RW, int CP, int W, int KS, class ARow>
__device__ __forceinline__ void tile_minplus(uint32_t (&out)[RW / KS][CP], ARow arow, const uint16_t* A, size_t lda,
                                             int a_lim, const uint16_t* Bp, size_t ldb, int b_lim, int K, bool half,
                                             unsigned char* smem) {
    constexpr int TM = W * RW, TN = 64 * CP, NT = 32 * W * KS;
    constexpr int NA = kKC * (TM / 8) / NT, NB = kKC * (TN / 8) / NT;
    static_assert(NA * NT == kKC * (TM / 8) && NB * NT == kKC * (TN / 8), "whole chunks per thread");
    uint32_t* As = reinterpret_cast<uint32_t*>(smem);                // [2][kKC][TM] splatted
    uint16_t* Ar = reinterpret_cast<uint16_t*>(As + 2 * kKC * TM);   // [kDepth][kKC][TM] as read
    uint16_t* Bs = Ar + kDepth * kKC * TM;                           // [kDepth][kKC][TN]
    uint8_t* cls = reinterpret_cast<uint8_t*>(Bs + kDepth * kKC * TN);  // [2][kKC][W]
    const int tid = threadIdx.x, warp = (tid >> 5) % W, lane = tid & 31, group = tid / (32 * W);
    const int n_c = (K + kKC - 1) / kKC;
    uint32_t acc[RW][CP];
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
        for (int c = 0; c < CP; ++c) acc[r][c] = INF2;
    int at[NA];  // rows of the next chunk to load
    auto index = [&](int c) {
#pragma unroll
        for (int x = 0; x < NA; ++x) {
            const int k = c * kKC + (tid + x * NT) / (TM / 8);
            at[x] = k < K ? arow(k) : 0;
        }
    };
    auto load = [&](int c) {
        if (c < n_c) {
            const int st = c % kDepth;
#pragma unroll
            for (int x = 0; x < NA; ++x) {
                const int idx = tid + x * NT, c8 = (idx % (TM / 8)) * 8;
                if (c * kKC + idx / (TM / 8) < K)
                    cp_async16(Ar + st * kKC * TM + idx * 8, A + (size_t)at[x] * lda + (c8 < a_lim ? c8 : 0));
            }
#pragma unroll
            for (int x = 0; x < NB; ++x) {
                const int idx = tid + x * NT, kk = idx / (TN / 8), c8 = (idx % (TN / 8)) * 8;
                if (c * kKC + kk < K)
                    cp_async16(Bs + st * kKC * TN + idx * 8, Bp + (size_t)(c * kKC + kk) * ldb + (c8 < b_lim ? c8 : 0));
            }
            index(c + 1);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    index(0);
#pragma unroll
    for (int c = 0; c < kDepth - 1; ++c) load(c);
    for (int c = 0; c < n_c; ++c) {
        uint32_t* Ab = As + (c & 1) * kKC * TM;
        uint8_t* cb = cls + (c & 1) * kKC * W;
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kDepth - 2) : "memory");
#pragma unroll
        for (int x = 0; x < NA; ++x) {  // rows beyond K: not read below
            const int idx = tid + x * NT, kk = idx / (TM / 8), c8 = idx % (TM / 8);
            const uint4 v = *reinterpret_cast<const uint4*>(Ar + (c % kDepth) * kKC * TM + idx * 8);
            uint32_t w[4] = {v.x, v.y, v.z, v.w};
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
                cb[kk * W + c8 / (RW / 8)] = mn >= INF ? 0 : (mx <= INF_HEADROOM ? 1 : 2);
            }
            uint4* dst = reinterpret_cast<uint4*>(Ab + idx * 8);
            dst[0] = make_uint4(splat(w[0]), splat(w[0] >> 16), splat(w[1]), splat(w[1] >> 16));
            dst[1] = make_uint4(splat(w[2]), splat(w[2] >> 16), splat(w[3]), splat(w[3] >> 16));
        }
        __syncthreads();  // chunk c is staged; every warp is done with chunk c - 1
        load(c + kDepth - 1);
        constexpr int KG = kKC / KS;
        const int k0 = group * KG, kn = min(k0 + KG, K - c * kKC);
        const uint32_t* bp = reinterpret_cast<const uint32_t*>(Bs + (c % kDepth) * kKC * TN) + lane * CP;
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
            for (int k = k0; k < kn; ++k) step(k, std::integral_constant<int, 0>());
        } else {
            for (int k = k0; k < kn; ++k) {
                const int cl = cb[k * W + warp];
                if (cl == 0) continue;  // uniform over the warp
                if (cl == 1) step(k, std::integral_constant<int, 1>());
                else step(k, std::integral_constant<int, 2>());
            }
        }
    }
    __syncthreads();  // the staging buffers are free
    if constexpr (KS == 1) {
#pragma unroll
        for (int r = 0; r < RW; ++r)
#pragma unroll
            for (int c = 0; c < CP; ++c) out[r][c] = acc[r][c];
    } else {
        static_assert(KS == 2, "two groups trade halves");
        constexpr int RH = RW / 2;
        uint32_t* ex = reinterpret_cast<uint32_t*>(smem) + (tid >> 5) * RH * CP * 32 + lane;
        const uint32_t* other =
            reinterpret_cast<const uint32_t*>(smem) + (warp + (1 - group) * W) * RH * CP * 32 + lane;
#pragma unroll
        for (int r = 0; r < RH; ++r)
#pragma unroll
            for (int c = 0; c < CP; ++c) ex[(r * CP + c) * 32] = group ? acc[r][c] : acc[RH + r][c];
        __syncthreads();
#pragma unroll
        for (int r = 0; r < RH; ++r)
#pragma unroll
            for (int c = 0; c < CP; ++c) out[r][c] = min2(group ? acc[RH + r][c] : acc[r][c], other[(r * CP + c) * 32]);
        __syncthreads();
    }
    if (half) {
#pragma unroll
        for (int r = 0; r < RW / KS; ++r)
#pragma unroll
            for (int c = 0; c < CP; ++c) out[r][c] = half_to_full(out[r][c]);
    }
}

// The tile transposed through shared memory: Tt[j][i] of TN x TM u16, in
// 16-byte chunks of 8 rows i.  Chunk q of row j sits at q ^ ((j / (2 CP)) & 7), so
// the 8 lanes of a 16-byte store phase (8 different rows) hit 8 different
// bank groups.  transposed_chunk reads chunk q of row j.
template <int TM, int RW, int CP>
__device__ __forceinline__ void transpose_store(uint16_t* Tt, const uint32_t (&acc)[RW][CP], int row0) {
    const int lane = threadIdx.x & 31;
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
                const int q = row0 / 8 + h;
                *reinterpret_cast<uint4*>(Tt + j * TM + ((q ^ key) * 8)) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
            }
        }
}
template <int TM, int CP>
__device__ __forceinline__ uint4 transposed_chunk(const uint16_t* Tt, int j, int q) {
    return *reinterpret_cast<const uint4*>(Tt + j * TM + ((q ^ ((j / (2 * CP)) & 7)) * 8));
}

// ---------------------------------------------------------------------------
// Closure of T by repeated squaring, in place: pass t takes T = min(T, T (x) T)
// over the upper-triangle 64 x 64 tiles, each also written transposed,
// so after t passes T holds every path of 2^t seam crossings.  A tile reads
// entries that other tiles of the pass may be lowering: an entry is the
// length of some path either way and at most its value before the pass, which is
// all a pass needs.  A node whose last pass changed nothing is closed and its later
// passes return at once: a street map needs 3 or 4 passes (few crossings
// on any shortest path), the worst case is log2 of the seams.  The blocked
// Floyd-Warshall this replaces needed a dependent launch per 64 seams at 25 us each
// whatever the map (1024 x 1024, b = 8: 56 launches, 1.46 ms); a pass over 280
// seams takes about as long as one of them.
// ---------------------------------------------------------------------------
constexpr int kSquareThreads = 256;

__global__ void __launch_bounds__(kSquareThreads) seam_square_kernel(const NodeBuild P, int t) {
    constexpr int TT = 64;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_max, s_chg, s_half;
    const int i = blockIdx.y;
    if (P.active && !P.active[i]) return;
    int* state = P.state + kNodeState * i;
    if (t > 0 && state[kNodeChanged + t - 1] == 0) return;  // closed
    const int nE = P.cnt[(size_t)i * (1 + P.g * P.g)], nt = (nE + TT - 1) / TT;
    if ((int)blockIdx.x >= nt * (nt + 1) / 2) return;
    int I, J;
    tri_pair(blockIdx.x, nt, I, J);
    const int tid = threadIdx.x, lane = tid & 31, row0 = first_row<16, 4, 2>(), TP = P.TP;
    uint16_t* T = P.T + (size_t)i * TP * TP;
    // values found in this pass may exceed the maximum read here: their entries
    // were INF before the pass, so taking a sum with one as INF loses nothing
    if (tid == 0) {
        s_max = s_chg = 0;
        s_half = *(volatile int*)(state + 1) <= kHalfMax;  // one value for the CTA: the pass raises it
    }
    __syncthreads();
    const bool half = s_half != 0;
    uint32_t acc[8][1], old[8];  // the old tile: no other CTA writes it
    uint32_t* d0 = reinterpret_cast<uint32_t*>(T + (size_t)(I * TT + row0) * TP + J * TT) + lane;
#pragma unroll
    for (int r = 0; r < 8; ++r) old[r] = __ldcg(d0 + (size_t)r * (TP / 2));
    tile_minplus<16, 1, 4, 2>(acc, [](int k) { return k; }, T + I * TT, TP, TP - I * TT, T + J * TT, TP, TP - J * TT, nE,
                           half, smem);
    bool chg = false;
    uint32_t mx = 0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        acc[r][0] = min2(acc[r][0], old[r]);
        if (acc[r][0] != old[r]) {
            d0[(size_t)r * (TP / 2)] = acc[r][0];
            chg = true;
            const uint32_t lo = acc[r][0] & 0xffffu, hi = acc[r][0] >> 16;
            if (lo < INF) mx = max(mx, lo);
            if (hi < INF) mx = max(mx, hi);
        }
    }
    mx = __reduce_max_sync(FULL, mx);
    if (lane == 0 && mx) atomicMax(&s_max, (int)mx);
    if (chg) s_chg = 1;
    __syncthreads();
    if (!s_chg) return;
    if (tid == 0) {
        atomicMax(state + 1, s_max);
        state[kNodeChanged + t] = 1;
    }
    if (I == J) return;
    uint16_t* Tt = reinterpret_cast<uint16_t*>(smem);
    transpose_store<TT, 8, 1>(Tt, acc, row0);
    __syncthreads();
    for (int idx = tid; idx < TT * (TT / 8); idx += kSquareThreads) {
        const int j = idx / (TT / 8), q = idx % (TT / 8);
        reinterpret_cast<uint4*>(T + (size_t)(J * TT + j) * TP + I * TT)[q] = transposed_chunk<TT, 1>(Tt, j, q);
    }
}

// U_p tiles: rows = edges, columns = ports of child p.
template <int RW, int CP, int W, int KS>
__global__ void __launch_bounds__(32 * W * KS, 2) lift_kernel(const NodeBuild P) {
    constexpr int TM = W * RW, TN = 64 * CP, NR = RW / KS;
    extern __shared__ __align__(16) unsigned char nsm[];
    __shared__ int s_max;
    const int i = blockIdx.z, p = blockIdx.y, g2 = P.g * P.g;
    if (P.active && !P.active[i]) return;
    const int* cnt = P.cnt + (size_t)i * (1 + g2);
    const int tn = (P.RP + TN - 1) / TN;
    const int m0 = (blockIdx.x / tn) * TM, n0 = (blockIdx.x % tn) * TN;
    if (m0 >= cnt[0]) return;
    const int* vm = P.state + kNodeState * i;
    const bool half = max(vm[0], vm[1]) <= kHalfMax;
    const uint2* inc = P.inc + ((size_t)i * g2 + p) * P.capI;
    const uint16_t* T = P.T + (size_t)i * P.TP * P.TP;
    const uint16_t* R = P.R + ((size_t)i * g2 + p) * P.capI * P.RP;
    const int row0 = first_row<RW, W, KS>(), lane = threadIdx.x & 31;
    uint32_t acc[NR][CP];
    if (threadIdx.x == 0) s_max = 0;
    tile_minplus<RW, CP, W, KS>(acc, [&](int k) { return (int)inc[k].y; }, T + m0, P.TP, P.TP - m0, R + n0, P.RP,
                            P.RP - n0, cnt[1 + p], half, nsm);
    uint16_t* U = P.U + ((size_t)i * g2 + p) * P.TP * P.RP;
    uint32_t mx = 0;
    const int col = n0 + lane * 2 * CP;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const int e = m0 + row0 + r;
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
    if (threadIdx.x == 0 && s_max) atomicMax(P.state + kNodeState * i + 2, s_max);
}

// D tiles: unit = (children p <= q, tile of p's ports x tile of q's ports).
template <int RW, int CP, int W, int KS>
__global__ void __launch_bounds__(32 * W * KS, 2) node_tile_kernel(const NodeBuild P) {
    constexpr int TM = W * RW, TN = 64 * CP, NR = RW / KS;
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
    const int* vm = P.state + kNodeState * i;
    const bool half = max(vm[0], vm[2]) <= kHalfMax;
    const uint2* inc = P.inc + ((size_t)i * g2 + q) * P.capI;
    const uint16_t* U = P.U + ((size_t)i * g2 + p) * P.TP * P.RP + m0;
    const uint16_t* R = P.R + ((size_t)i * g2 + q) * P.capI * P.RP + n0;
    const int row0 = first_row<RW, W, KS>(), lane = threadIdx.x & 31;
    uint32_t acc[NR][CP];
    if (threadIdx.x == 0) s_chg = 0;
    tile_minplus<RW, CP, W, KS>(acc, [&](int k) { return (int)inc[k].y; }, U, P.RP, P.RP - m0, R, P.RP, P.RP - n0,
                            P.cnt[(size_t)i * (1 + g2) + 1 + q], half, nsm);
    uint16_t* D = node_mat(P, node);
    const int col = n0 + lane * 2 * CP;  // port of q; nP is a multiple of 4
    if (p == q) {
        const uint16_t* cm = child_mat(P, node, p);
        int ce[2 * CP];
#pragma unroll
        for (int c = 0; c < 2 * CP; ++c) ce[c] = P.cext[min(col + c, nP - 1)];
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const uint16_t* crow = cm + (size_t)P.cext[min(m0 + row0 + r, nP - 1)] * P.C.NP;
#pragma unroll
            for (int c = 0; c < CP; ++c)
                acc[r][c] = min2(acc[r][c], (uint32_t)crow[ce[2 * c]] | ((uint32_t)crow[ce[2 * c + 1]] << 16));
        }
    }
    bool chg = false;
    if (P.changed && col < nP) {  // against the old matrix, before any store
        uint32_t cext[CP];
#pragma unroll
        for (int c = 0; c < CP; ++c)
            cext[c] = (P.isext[q * nP + col + 2 * c] ? 0xffffu : 0u) |
                      (P.isext[q * nP + col + 2 * c + 1] ? 0xffff0000u : 0u);
        uint32_t diff = 0;
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const int row = p * nP + min(m0 + row0 + r, nP - 1);
            const bool on = m0 + row0 + r < nP && P.isext[row];
            const uint32_t* d = reinterpret_cast<const uint32_t*>(D + (size_t)row * NP + q * nP + col);
#pragma unroll
            for (int c = 0; c < CP; ++c) diff |= on ? (d[c] ^ acc[r][c]) & cext[c] : 0u;
        }
        chg = diff != 0;
    }
    if (col < nP) {
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const int row = m0 + row0 + r;
            if (row >= nP) continue;
            uint32_t* d = reinterpret_cast<uint32_t*>(D + (size_t)(p * nP + row) * NP + q * nP + col);
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
    transpose_store<TM, NR, CP>(Tt, acc, row0);
    __syncthreads();
    for (int idx = threadIdx.x; idx < TN * (TM / 8); idx += 32 * W * KS) {
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
// LC lanes hold the column pairs of a child (16 for up to 32 ports); NT threads.
// Latency-bound, so global loads go out in batches (R rows four at a time, a
// row's child summary before the products) and the product loops are unrolled:
// one node of 64 seams 91 -> 56 us, 1024 of them 341 -> 285 us, 4096 of 32 seams
// 252 -> 217 us.
// ---------------------------------------------------------------------------
constexpr int kSmallSeams = 64, kSmallPorts = 64;
constexpr size_t kSmallSmem = 100 * 1024;  // two CTAs an SM

struct SmallLayout {
    int RP, ldU;  // row strides of R and U (multiples of 8)
    size_t o_inc, o_ext, o_R, o_T, o_U, total;
};
__host__ __device__ inline SmallLayout small_layout(int g2, int nP, int capI) {
    SmallLayout L;
    L.RP = (nP + 7) / 8 * 8;
    L.ldU = (g2 * nP + 15) / 8 * 8;
    size_t o = kSmallSeams * sizeof(int4);
    L.o_inc = o;
    o += (size_t)g2 * capI * sizeof(uint2);
    L.o_ext = o;
    o += kSmallPorts * sizeof(int);
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

template <int LC, int NT>
__global__ void __launch_bounds__(NT) node_small_kernel(const NodeBuild P) {
    constexpr int kW = NT / 32;
    extern __shared__ __align__(16) unsigned char nsm[];
    __shared__ int q_cnt[256];
    __shared__ int s_w0, s_nE, s_chg;
    const int i = blockIdx.x, g2 = P.g * P.g, nP = P.nP, NP = P.N.NP;
    if (P.active && !P.active[i]) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const SmallLayout L = small_layout(g2, nP, P.capI);
    int4* edge = reinterpret_cast<int4*>(nsm);
    uint2* inc = reinterpret_cast<uint2*>(nsm + L.o_inc);
    int* cext = reinterpret_cast<int*>(nsm + L.o_ext);
    uint16_t* R = reinterpret_cast<uint16_t*>(nsm + L.o_R);
    uint16_t (*T)[kTLD] = reinterpret_cast<uint16_t (*)[kTLD]>(nsm + L.o_T);
    uint16_t* U = reinterpret_cast<uint16_t*>(nsm + L.o_U);
    const int node = node_id(P, i);
    if (tid < g2) q_cnt[tid] = 0;
    if (tid == 0) s_chg = 0;
    for (int j = tid; j < nP; j += NT) cext[j] = P.cext[j];
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
    // R: the two incidences of every edge, one warp per row, four rows in flight
    for (int r0 = warp; r0 < 2 * nE; r0 += 4 * kW) {
        uint32_t v[4][2], off[4];
        int at[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int r = min(r0 + x * kW, 2 * nE - 1);
            const int4 e = edge[r >> 1];
            const int q = r & 1 ? e.x >> 8 : e.x & 255, k = r & 1 ? (int)((unsigned)e.y >> 16) : e.y & 0xffff;
            const int port = r & 1 ? (int)((unsigned)e.z >> 16) : e.z & 0xffff;
            const uint16_t* crow = child_mat(P, node, q) + (size_t)cext[port] * P.C.NP;
            at[x] = (q * P.capI + k) * L.RP;
            off[x] = r & 1 ? (uint32_t)e.w : 0u;
            v[x][0] = lane < nP ? __ldg(crow + cext[lane]) : INF;
            v[x][1] = lane + 32 < nP ? __ldg(crow + cext[lane + 32]) : INF;
        }
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            if (r0 + x * kW >= 2 * nE) continue;
            if (lane < L.RP) R[at[x] + lane] = (uint16_t)sat_add(v[x][0], off[x]);
            if (lane + 32 < L.RP) R[at[x] + lane + 32] = (uint16_t)sat_add(v[x][1], off[x]);
        }
    }
    __syncthreads();
    for (int idx = tid; idx < B * B; idx += NT) {
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
    if (tid < kThreads) close_pivot_block(T, nE);
    else
        for (int k = 0; k < nE; ++k) __syncthreads();  // its barriers
    __syncthreads();
    // sub-warps of LC lanes; a lane holds one column pair of a child
    constexpr int kSub = 32 / LC, kSubs = kW * kSub;
    const int sub = warp * kSub + lane / LC, cl = lane % LC;
    const bool col_ok = 2 * cl < nP;
    {   // U: items of 4 edges x one child
        const int ng = (nE + 3) / 4;
        for (int it = sub; it < ng * g2; it += kSubs) {
            const int p = it / ng, e0 = (it - p * ng) * 4;
            uint32_t acc[4] = {INF2, INF2, INF2, INF2};
            const int n = q_cnt[p];
#pragma unroll 4
            for (int k = 0; k < n; ++k) {
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
        const int lo = q * nP, hi = lo + nP, col = lo + 2 * cl;
        uint32_t acc[8], own[8];  // own: the rows' child summary (rows of child q)
#pragma unroll
        for (int r = 0; r < 8; ++r) acc[r] = own[r] = INF2;
        if (col_ok && i0 + 8 > lo) {
            const uint16_t* cm = child_mat(P, node, q);
            const int c0 = cext[2 * cl], c1 = cext[2 * cl + 1];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const int row = min(max(i0 + r - lo, 0), nP - 1);
                const uint16_t* crow = cm + (size_t)cext[row] * P.C.NP;
                if (i0 + r >= lo) own[r] = (uint32_t)__ldg(crow + c0) | ((uint32_t)__ldg(crow + c1) << 16);
            }
        }
        const int n = q_cnt[q];
#pragma unroll 4
        for (int k = 0; k < n; ++k) {
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
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int row = i0 + r;
            if (row >= hi) continue;
            acc[r] = min2(acc[r], own[r]);
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

// `bytes` is one value per kernel, whatever the index: the limit belongs to the kernel and the
// device, and another thread may be between its own limit and its launch.
template <class K>
void allow_smem(K kernel, size_t bytes) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// U, then D.
template <int RW, int CP, int W, int KS>
void launch_products(const NodeBuild& P, int n, cudaStream_t st) {
    constexpr int TM = W * RW, TN = 64 * CP;
    const size_t smem = tile_smem_bytes<RW, CP, W>();
    const int g2 = P.g * P.g, nt = (P.nP + TM - 1) / TM;
    allow_smem(lift_kernel<RW, CP, W, KS>, smem);
    allow_smem(node_tile_kernel<RW, CP, W, KS>, smem);
    lift_kernel<RW, CP, W, KS><<<dim3(blocks_for(P.n_seams, TM) * blocks_for(P.RP, TN), g2, n), 32 * W * KS, smem, st>>>(P);
    node_tile_kernel<RW, CP, W, KS>
        <<<dim3(g2 * nt * (nt + 1) / 2 + g2 * (g2 - 1) / 2 * nt * nt, n), 32 * W * KS, smem, st>>>(P);
}

// Fewer 128 x 128 tiles than two per SM (148 of them) leave SMs idle or with one CTA (8 warps),
// whose latencies show.  Whole builds, 128 x 128 tiles always / from one per SM / from two /
// from four / never: 256 x 256, b = 8: 472 / 457 / 453 / 453 / 451 us; 512 x 512:
// 1096 / 1097 / 1100 / 1134 / 1142; 1024 x 1024: 4729 / 4729 / 4731 / 4722 / 5440.
constexpr size_t kWideTiles = 2 * 148;

}  // namespace

void launch_pad_fill(MatSet M, int count, cudaStream_t st) {
    if (M.NP == M.n) return;
    const size_t e = (size_t)(M.NP - M.n) * (M.NP + M.n);
    for (int y0 = 0; y0 < count; y0 += kMaxGridY)
        pad_fill_kernel<<<dim3(std::min(64u, blocks_for(e, 256)), std::min(kMaxGridY, count - y0)), 256, 0, st>>>(M, y0);
}

bool node_build_small(const NodeBuild& P) {
    return P.n_seams <= kSmallSeams && P.nP <= kSmallPorts &&
           small_layout(P.g * P.g, P.nP, P.capI).total <= kSmallSmem;
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
    P.state = reinterpret_cast<int*>(take((size_t)n * kNodeState * sizeof(int)));
    P.edge = reinterpret_cast<int4*>(take((size_t)n * P.TP * sizeof(int4)));
    P.inc = reinterpret_cast<uint2*>(take(n * g2 * P.capI * sizeof(uint2)));
    P.R = reinterpret_cast<uint16_t*>(take(n * g2 * P.capI * P.RP * sizeof(uint16_t)));
    P.T = reinterpret_cast<uint16_t*>(take((size_t)n * P.TP * P.TP * sizeof(uint16_t)));
    P.U = reinterpret_cast<uint16_t*>(take(n * g2 * P.TP * P.RP * sizeof(uint16_t)));
    return off;
}

void launch_node_build(const NodeBuild& P, int n, cudaStream_t st) {
    if (n <= 0) return;
    const int g2 = P.g * P.g;
    if (node_build_small(P)) {
        const size_t smem = small_layout(g2, P.nP, P.capI).total;
        if (P.nP <= 32) {
            allow_smem(node_small_kernel<16, 256>, kSmallSmem);
            node_small_kernel<16, 256><<<n, 256, smem, st>>>(P);
        } else {
            allow_smem(node_small_kernel<32, 512>, kSmallSmem);
            node_small_kernel<32, 512><<<n, 512, smem, st>>>(P);
        }
        return;
    }
    // Grids cover every seam candidate: the active ones are counted on the device
    // (CTAs beyond them return at once), so the host waits for nothing.
    const int m = P.n_seams;
    seam_list_kernel<<<n, std::min(1024, (m + 31) / 32 * 32), 0, st>>>(P);
    lift_rows_kernel<<<dim3(blocks_for(P.capI, kWarps), g2, n), kThreads, 0, st>>>(P);
    const unsigned tiles = P.TP / 64;
    seam_block_kernel<<<dim3(4 * tiles * tiles, n), kThreads, 0, st>>>(P);
    const unsigned nq = blocks_for(m, 64);
    allow_smem(seam_square_kernel, tile_smem_bytes<16, 1, 4>());
    for (int t = 0; (1 << t) < m; ++t)  // paths of up to m crossings
        seam_square_kernel<<<dim3(nq * (nq + 1) / 2, n), kSquareThreads, tile_smem_bytes<16, 1, 4>(), st>>>(P, t);
    // 128 x 128 tiles where they fill the chip, else 64 x 64 ones (four times the CTAs)
    const int nt = (P.nP + 127) / 128;
    const bool wide = P.nP > 64 && (size_t)n * (g2 * nt * (nt + 1) / 2 + g2 * (g2 - 1) / 2 * nt * nt) >= kWideTiles;
    if (wide) launch_products<16, 2, 8, 1>(P, n, st);
    else launch_products<16, 1, 4, 2>(P, n, st);
}

}  // namespace hb
