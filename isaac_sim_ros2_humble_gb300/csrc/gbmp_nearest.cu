// gbmp_nearest.cu -- nearest neighbours of the state manager (gbmp_nearest).
//
// For every query the candidate of least squared distance over the robot's active joints,
// accumulated in joint order with fused multiply-adds (SingleArmStates.cu:1285-1300); the
// argmin key is (distance, candidate position).
#include <cooperative_groups.h>

#include <climits>

#include "gbmp_internal.h"

namespace cg = cooperative_groups;

namespace gbmp {

// k_nearest_tiles.  A warp holds 128 candidates in registers (four a lane, as two packed
// pairs, the active joints only) and passes the block's queries by them from shared
// memory; the warps of a cluster of up to eight blocks share the candidates of one tile of
// queries, and the blocks' results meet through distributed shared memory, so one launch
// without a workspace fills the GPU for one query as for thousands.
//
// What bounds it: 2 D operations on the FP32 pipe for each (query, candidate) pair (D
// active joints; they are issued as packed pairs, which leaves the issue slots to the
// rest).  A query's running best decides with one comparison of the four candidates'
// minimum whether anything more is to be done.  1,000 queries in 100,000 nodes of 7
// joints: 95 us (36 us at the FP32 pipe's rate; the rest is the latency of the query reads
// and of the candidate rows, 0.65 of the shared-memory / L1 wavefronts), 1,190 us with one
// warp for each query (k_nearest), which read every candidate row for every query, a row's
// stride between the lanes, on 1,000 of 9,728 warps; 7 queries in 190,000 nodes 16 against
// 1,120 us, 30 in 3,000 (a roadmap round) 5 against 64 us.
constexpr int kNearestDims = 16;      // instantiations 1 .. 16 active joints
constexpr int kNearestWarps = 8;      // a block; four blocks an SM at 64 registers
constexpr int kNearestPerWarp = 4 * kWarp;
constexpr int kNearestMaxTile = 128;  // queries of a block
constexpr int kNearestMaxCluster = 8;
constexpr unsigned kInfBits = 0x7f800000u;

__device__ __forceinline__ unsigned long long pack2(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float &x, float &y) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

template <int D>
__global__ void __launch_bounds__(kNearestWarps *kWarp, D <= 8 ? 4 : 2)
    k_nearest_tiles(const float *__restrict__ tree, const int *__restrict__ cand, long long ncand,
                    const float *__restrict__ queries, long long Q, int L, const unsigned char *__restrict__ active,
                    int tile, int *__restrict__ out) {
    // queries of the tile, each active joint twice (one packed operand), and their best
    // (distance bits, position)
    __shared__ __align__(16) unsigned long long s_q[kNearestMaxTile][D + (D & 1)];   // rows of whole 16-byte words
    __shared__ unsigned long long s_best[kNearestMaxTile];
    __shared__ int s_joint[kNearestDims];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), blocks = (int)cluster.num_blocks();
    const long long q0 = (long long)(blockIdx.x / blocks) * tile;
    const int nq = (int)min((long long)tile, Q - q0);
    const int warp = threadIdx.x / kWarp, lane = threadIdx.x & 31;
    if (threadIdx.x == 0)
        for (int j = 0, d = 0; j < L; ++j)
            if (active[j]) s_joint[d++] = j;
    for (int q = threadIdx.x; q < nq; q += blockDim.x) s_best[q] = ((unsigned long long)kInfBits << 32) | 0xffffffffu;
    __syncthreads();
    for (int e = threadIdx.x; e < nq * D; e += blockDim.x) {
        const float v = queries[(q0 + e / D) * L + s_joint[e % D]];
        s_q[e / D][e % D] = pack2(v, v);
    }
    __syncthreads();

    const long long step = (long long)blocks * kNearestWarps * kNearestPerWarp;
    for (long long c0 = (long long)(rank * kNearestWarps + warp) * kNearestPerWarp; c0 < ncand; c0 += step) {
        unsigned long long y[2][D];   // candidates (0, 1) and (2, 3) of this lane, negated
        {
            float v[4][D];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const long long c = c0 + u * kWarp + lane;
                const bool in = c < ncand;
                const float *row = tree + (in ? (cand ? (long long)cand[c] : c) : 0) * L;
                // past the end: NaN, which no comparison takes
#pragma unroll
                for (int d = 0; d < D; ++d) v[u][d] = in ? -row[s_joint[d]] : __int_as_float(0x7fffffff);
            }
#pragma unroll
            for (int d = 0; d < D; ++d) {
                y[0][d] = pack2(v[0][d], v[1][d]);
                y[1][d] = pack2(v[2][d], v[3][d]);
            }
        }
#pragma unroll 2
        for (int q = 0; q < nq; ++q) {
            unsigned long long a = 0ull, b = 0ull;
#pragma unroll
            for (int d = 0; d < D; d += 2) {
                const ulonglong2 qd = *reinterpret_cast<const ulonglong2 *>(&s_q[q][d]);
                const unsigned long long da = add2(qd.x, y[0][d]), db = add2(qd.x, y[1][d]);
                a = fma2(da, da, a);
                b = fma2(db, db, b);
                if (d + 1 < D) {
                    const unsigned long long ea = add2(qd.y, y[0][d + 1]), eb = add2(qd.y, y[1][d + 1]);
                    a = fma2(ea, ea, a);
                    b = fma2(eb, eb, b);
                }
            }
            float s[4];
            unpack2(a, s[0], s[1]);
            unpack2(b, s[2], s[3]);
            const float m = fminf(fminf(s[0], s[1]), fminf(s[2], s[3]));
            const unsigned cur = *(reinterpret_cast<volatile unsigned *>(&s_best[q]) + 1);   // distance bits
            // an equal distance may still win by its position
            if (__any_sync(kFull, m <= __uint_as_float(cur))) {
                float best = __uint_as_float(kInfBits);
                unsigned pos = 0xffffffffu;
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (s[u] < best) {
                        best = s[u];
                        pos = (unsigned)(c0 + u * kWarp + lane);
                    }
                const unsigned hi = __reduce_min_sync(kFull, __float_as_uint(best));   // distances are >= +0
                const unsigned lo = __reduce_min_sync(kFull, __float_as_uint(best) == hi ? pos : 0xffffffffu);
                if (lane == 0 && hi < kInfBits) atomicMin(&s_best[q], ((unsigned long long)hi << 32) | lo);
            }
        }
    }
    cluster.sync();
    if (rank == 0)
        for (int q = threadIdx.x; q < nq; q += blockDim.x) {
            unsigned long long best = s_best[q];
            for (int r = 1; r < blocks; ++r) best = min(best, cluster.map_shared_rank(s_best, r)[q]);
            const unsigned pos = (unsigned)best;
            out[q0 + q] = (best >> 32) >= kInfBits ? -1 : cand ? cand[pos] : (int)pos;
        }
    cluster.sync();   // the blocks stay until their results have been read
}

template <int D>
static cudaError_t nearest_launch(int dims, cudaLaunchConfig_t *cfg, void **args) {
    if constexpr (D <= kNearestDims) {
        if (dims == D) return cudaLaunchKernelExC(cfg, (const void *)k_nearest_tiles<D>, args);
        return nearest_launch<D + 1>(dims, cfg, args);
    }
    return cudaErrorInvalidValue;
}

// Nearest candidate per query, one warp per query: robots of more than kNearestDims active
// joints (or none), and candidate lists beyond 32-bit positions.  The
// squared distance is accumulated in joint order with fused multiply-adds
// (SingleArmStates.cu:1285-1300); the argmin key is (distance, candidate position).
__global__ void __launch_bounds__(256)
    k_nearest(const float *__restrict__ tree, const int *__restrict__ cand, long long ncand,
              const float *__restrict__ queries, long long Q, int L, const unsigned char *__restrict__ active,
              int *__restrict__ out) {
    __shared__ float qs[8][kMaxLinks];
    __shared__ unsigned char act[kMaxLinks];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int j = threadIdx.x; j < L; j += blockDim.x) act[j] = active[j];
    __syncthreads();
    const long long nw = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long q = blockIdx.x * (long long)(blockDim.x >> 5) + warp; q < Q; q += nw) {
        for (int j = lane; j < L; j += 32) qs[warp][j] = queries[q * L + j];
        __syncwarp();
        float best = __int_as_float(0x7f800000);
        long long bpos = LLONG_MAX;
        for (long long c = lane; c < ncand; c += 32) {
            const long long idx = cand ? cand[c] : c;
            const float *y = tree + idx * L;
            float s = 0.f;
            for (int j = 0; j < L; ++j)
                if (act[j]) {
                    const float d = __fadd_rn(qs[warp][j], -y[j]);
                    s = __fmaf_rn(d, d, s);
                }
            if (s < best) { best = s; bpos = c; }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const float ob = __shfl_xor_sync(kFull, best, off);
            const long long op = __shfl_xor_sync(kFull, bpos, off);
            if (ob < best || (ob == best && op < bpos)) { best = ob; bpos = op; }
        }
        if (lane == 0) out[q] = bpos == LLONG_MAX ? -1 : (int)(cand ? cand[bpos] : bpos);
        __syncwarp();
    }
}

}  // namespace gbmp

using namespace gbmp;

extern "C" gbmp_status gbmp_nearest(gbmp_robot r, const float *d_tree, int64_t M, const int32_t *d_cand, int64_t n_cand,
                                    const float *d_queries, int64_t Q, int32_t *d_out, void *stream) {
    GBMP_CHECK_ARG(r, "robot is NULL");
    GBMP_CHECK_ARG(M >= 0 && Q >= 0 && n_cand >= 0, "negative size");
    if (Q == 0) return GBMP_OK;
    GBMP_CHECK_ARG(d_queries && d_out, "queries/out is NULL");
    // SingleArmStates.cu:1359-1370: the manager and every candidate group must be non-empty.
    GBMP_CHECK_ARG(M > 0, "manager is empty");
    long long nc = d_cand ? n_cand : M;
    GBMP_CHECK_ARG(nc > 0, "candidate group is empty");
    GBMP_CHECK_ARG(d_tree, "tree is NULL");
    cudaStream_t s = (cudaStream_t)stream;
    ProfScope ps(GBMP_PROF_OTHER, s);
    const unsigned char *act = r->dev.active;
    // blocks a query tile: enough warps to hold the candidates at once, up to eight; then
    // queries a tile so that all tiles give four blocks for each SM (two: 113 us instead of 95
    // on the case above, one: 135; the query loop is bound by latency below that)
    int blocks = 1;
    while (blocks < kNearestMaxCluster && (long long)blocks * kNearestWarps * kNearestPerWarp < nc) blocks *= 2;
    const long long tiles = std::max(1, 4 * r->num_sms / blocks);
    int tile = (int)std::min<long long>(kNearestMaxTile, (Q + tiles - 1) / tiles);
    const long long grid = (Q + tile - 1) / tile * blocks;
    if (r->dim < 1 || r->dim > kNearestDims || nc >= INT_MAX || grid >= INT_MAX) {
        const long long nb = std::min<long long>((Q + 7) / 8, 64LL * r->num_sms);
        k_nearest<<<(unsigned)nb, 256, 0, s>>>(d_tree, d_cand, nc, d_queries, Q, r->L, act, d_out);
        GBMP_CUDA(cudaGetLastError());
        return GBMP_OK;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kNearestWarps * kWarp);
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)blocks;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    long long queries = Q;
    int L = r->L;
    void *args[] = {&d_tree, &d_cand, &nc, &d_queries, &queries, &L, &act, &tile, &d_out};
    GBMP_CUDA(nearest_launch<1>(r->dim, &cfg, args));
    return GBMP_OK;
}
