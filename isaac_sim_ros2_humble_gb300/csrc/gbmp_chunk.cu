// gbmp_chunk.cu -- the edge-validation kernel (edges cut into parts that warps take, their
// states in chunks of consecutive states; the chunk routines are in gbmp_chunk_device.cuh),
// its launch set-up, and FK alone by chunks of consecutive states (gbmp_fk).
#include "gbmp_order.h"
#include "gbmp_states_device.cuh"

namespace gbmp {

// Warps per block of the chunk kernel: three blocks of 8 warps per SM at 80 registers.
// The kernel is bound by instruction issue (0.72 of the issue slots at 65,536 edges), so
// more warps bring little: before scenes had a distance field, 2.46 ms with two blocks, 2.22
// with three, 2.21 with two blocks of 16 warps at 64 registers (65,536 edges of the 8-DOF
// arm, verdicts; 1.21 ms a call now).
constexpr int kChunkWarps = 8;

// Edge validation by chunks.  An edge's chunks, in their order, are cut into parts of
// consecutive chunks (EdgePlan, made by k_edge_order from the lengths); item i is part
// i / n_edges of edge order[i % n_edges], so part 0 of every edge comes first, the edges of
// each part longest first.  A warp takes `grab` items from a shared counter, drops those
// that are settled already (past the edge's end, or another part has recorded a hit that
// decides), one lane each, and walks the chunks of the others up to a chunk that holds a
// colliding state.  k_edge_order has written the outputs of a free edge (and of one too
// long to validate, which no warp walks); a hit clears ok and lowers the first hit (-1,
// the largest unsigned value, until then).
//
// Why parts: the free edges are few (18 % of the benchmark's) and long, so with one warp
// per edge most warps idled while some walked up to 56 chunks in a row: 64 edges 0.47 ms
// whole, 0.046 ms in parts; 3,001 edges of a 30-link robot with first hits 1.20 and 0.30
// ms; 65,536 edges (18 for each warp) 2.22 and 2.26 ms (all with the kernel of that time; now
// 0.035, 0.26 and 1.21 ms).
//
// The chunk orders are gbmp_order.h's: state order when the first hit is asked for,
// coarse to fine when only the verdict is.  On the 65,536 edges of the 8-DOF benchmark
// (uniform endpoints, 82 % colliding) the coarse-to-fine order checks 4.94 M states
// against 8.89 M, 4.19 M of them on the free edges; 8 passes give 4.97 M (5.01 M in plain
// order), 4 passes 5.06 M, a full bit-reversed order of the chunks 4.96 M.
//
// The chunk's states are tested side by side in the lanes (gbmp_chunk_device.cuh).
// When that came, 65,536 edges went from 3.79 ms (the states walked one by one, their spheres
// in the lanes) to 2.22 ms.

// A warp that holds a later part of an edge waits, at most kProbePolls looks, until the
// edge's probes are known or it has a hit (bits beside the state count).  The warp that holds
// them took them before this one took its item and does not wait before it has walked them.
// Without the wait a batch whose edges collide at once had every part of every edge walked: 161
// edges 180 us, 54 us with it (63 us with one warp an edge); 64 edges took 40 us with it, 35
// without.
constexpr int kProbed0 = 1 << 28, kProbed1 = 1 << 29, kHit = 1 << 30, kStepsMask = kProbed0 - 1;
constexpr int kProbePolls = 4096;
constexpr int kMaxGrab = 8;   // settled items taken at a time in a batch of few edges

template <int K, bool CNT>
__global__ void __launch_bounds__(kChunkWarps *kWarp, 3)
    k_edge_chunk(DevRobot R, DevEnv E, const float *__restrict__ from, const float *__restrict__ to,
                 int *nsteps, const float *__restrict__ dir, const int *__restrict__ order, int n_edges,
                 const EdgePlan *__restrict__ plan, unsigned long long *__restrict__ next, unsigned char *ok_out,
                 int *first_hit_out) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int nwords = env_words(E.ns, E.nb, E.nc);
    SmemTables t = carve_tables(smem, R, nwords);
    if (!stage_tables(R, E, t, nwords)) return;
    const int warp = threadIdx.x / kWarp;
    ChunkScratch cs;
    carve_chunk(smem + smem_tables_bytes(R, nwords), R, K, warp, cs);
    const int lane = threadIdx.x & 31;
    const bool any = first_hit_out == nullptr;
    // What is needed between chunks only lives in shared memory: the chunk routine takes
    // every register (80, three blocks an SM).
    __shared__ EdgePlan s_plan;
    __shared__ int4 s_item[kChunkWarps][kWarp];   // edge, states, first chunk, end
    if (threadIdx.x == 0) s_plan = *plan;
    __syncthreads();
    int grab = s_plan.grab;
    for (;;) {
        unsigned live;
        {
            const int parts = s_plan.parts;
            unsigned long long i0 = 0;
            if (lane == 0) i0 = atomicAdd(next, (unsigned long long)grab);
            i0 = __shfl_sync(kFull, i0, 0);
            const long long items = (long long)n_edges * parts, i = (long long)i0 + lane;
            if ((long long)i0 >= items) break;
            bool mine = false;
            if (lane < grab && i < items) {
                const int p = (int)(i / n_edges);
                const int e = order[i - (long long)p * n_edges];
                const int v = *(volatile int *)(nsteps + e), n = v & kStepsMask;
                if (n <= kMaxEdgeStates && !(any && (v & kHit))) {
                    const int nch = edge_chunk_count(n, K, any);
                    const int span = max(s_plan.span, (nch + parts - 1) / parts);
                    const int c0 = p * span, c1 = min(c0 + span, nch);
                    mine = c0 < c1 && (any || p == 0 ||
                                       *(volatile unsigned *)(first_hit_out + e) > (unsigned)edge_chunk_range(c0, n, K, any).x);
                    s_item[warp][lane] = make_int4(e, n, c0, c1);
                }
            }
            live = __ballot_sync(kFull, mine);   // also orders the items before their reads
            __syncwarp();
            // settled items go faster and faster in a batch of few edges
            grab = live || !s_plan.grow ? s_plan.grab : min(2 * grab, kMaxGrab);
        }
        for (; live; live &= live - 1u) {
            const int x = __ffs(live) - 1;
            if (s_plan.probing) {
                const int4 it = s_item[warp][x];
                // the probes (the first chunk, and for verdicts the last) come first: an edge
                // they settle is not walked by the warps that hold its other parts
                const int probes = any ? min(2, edge_chunk_count(it.y, K, any)) : 1;
                if (it.z >= probes) {
                    const int want = probes == 2 ? kProbed0 | kProbed1 : kProbed0;
                    bool hit = false;
                    for (int poll = 0; poll < kProbePolls; ++poll) {
                        const int v = *(volatile int *)(nsteps + it.x);
                        hit = any ? (v & kHit) != 0
                                  : *(volatile unsigned *)(first_hit_out + it.x) <= (unsigned)edge_chunk_range(it.z, it.y, K, any).x;
                        if (__any_sync(kFull, (v & want) == want || hit)) break;
                        __nanosleep(200);
                    }
                    if (__any_sync(kFull, hit)) continue;
                }
            }
            for (int c = s_item[warp][x].z;; ++c) {
                const int4 it = s_item[warp][x];
                if (c >= it.w) break;
                const StateRange r = edge_chunk_range(c, it.y, K, any);
                // the other warps' findings (relaxed: a late look costs a chunk, not the result)
                if (c > it.z) {
                    const bool settled = any ? (*(volatile int *)(nsteps + it.x) & kHit) != 0
                                             : *(volatile unsigned *)(first_hit_out + it.x) <= (unsigned)r.x;
                    if (__any_sync(kFull, settled)) break;
                }
                const long long off = (long long)it.x * R.L;
                const int h = warp_edge_chunk<K, CNT>(t, R, E, cs, lane, from + off, to + off, dir + off, r.x, r.y,
                                                      it.y, any);
                const int e = s_item[warp][x].x;
                if (lane == 0) {
                    if (h >= 0) {
                        if (ok_out) *(volatile unsigned char *)(ok_out + e) = 0;
                        if (first_hit_out) atomicMin(reinterpret_cast<unsigned *>(first_hit_out + e), (unsigned)h);
                    }
                    if (h >= 0 || (s_plan.probing && c < 2))
                        atomicOr(nsteps + e, (h >= 0 ? kHit : 0) | (c == 0 ? kProbed0 : c == 1 ? kProbed1 : 0));
                }
                if (h >= 0) break;
            }
        }
        __syncwarp();
    }
}

// The chunk kernel of K states a chunk (10 or 4), with or without work counting.
static const void *edge_chunk_kernel(int K, bool count) {
    if (K == 10) return count ? (const void *)k_edge_chunk<10, true> : (const void *)k_edge_chunk<10, false>;
    return count ? (const void *)k_edge_chunk<4, true> : (const void *)k_edge_chunk<4, false>;
}

// States per chunk: 10 (three pose-row lanes per state fill 30 of 32 lanes in the chunk
// FK; measured 8.22 ms against 8.43 for 8 on the 65,536-edge benchmark call), 4 for
// robots of more than 16 links, whose pose block per state is larger.
int edge_chunk_states(const DevRobot &R, int form) {
    if (!R.cull || form == 1) return 0;
    if (form == 4 || form == 10) return form;
    return R.L <= 16 ? 10 : 4;
}

gbmp_status edge_chunk_prepare(const DevRobot &R, const DevEnv &E, int num_sms, int K, size_t *smem, int *grid) {
    *smem = smem_tables_bytes(R, env_words(E.ns, E.nb, E.nc)) + smem_chunk_bytes(R, K) * kChunkWarps;
    const void *fn = edge_chunk_kernel(K, R.work != nullptr);
    const gbmp_status st = ensure_smem_optin(fn);
    if (st) return st;
    int per_sm = 0;
    GBMP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kChunkWarps * kWarp, *smem));
    if (per_sm < 1) {
        set_error("chunked edge kernel does not fit on an SM (%zu bytes of shared memory)", *smem);
        return GBMP_ERR_CAPACITY;
    }
    *grid = per_sm * num_sms;
    return GBMP_OK;
}

int edge_chunk_warps(int grid) { return grid * kChunkWarps; }

gbmp_status edge_chunk_launch(const DevRobot &R, const DevEnv &E, int K, int grid, size_t smem, cudaStream_t s,
                              const float *from, const float *to, int *nsteps, const float *dir,
                              const int *order, long long n_edges, const EdgePlan *plan, unsigned long long *next,
                              unsigned char *ok, int *first_hit) {
    // the grid is the resident blocks, at most one warp per item
    const long long need = (n_edges * kEdgeMaxParts + kChunkWarps - 1) / kChunkWarps;
    if (need < grid) grid = (int)need;
    int ne = (int)n_edges;
    DevRobot r = R;
    DevEnv e = E;
    void *args[] = {&r, &e, &from, &to, &nsteps, &dir, &order, &ne, &plan, &next, &ok, &first_hit};
    GBMP_CUDA(cudaLaunchKernel(edge_chunk_kernel(K, R.work != nullptr), dim3(grid), dim3(kChunkWarps * kWarp), args, smem,
                               s));
    GBMP_CUDA(cudaGetLastError());
    return GBMP_OK;
}

// ---------------------------------------------------------------------------------
// FK alone (gbmp_fk): chunks of up to kFkChunk consecutive states per warp, the chunk FK above,
// then the chunk's link poses and sphere centres written out.  The poses of consecutive
// states are consecutive in memory, so a chunk's poses are one block that the warp writes
// as 16-byte words, 512 contiguous bytes per store (float4 rows from shared memory, the
// constant last row 0 0 0 1 built in registers); the sphere centres of the chunk are
// likewise one block, written lane by lane in order.
// ---------------------------------------------------------------------------------
constexpr int kFkChunk = 10;
constexpr int kFkWarpBytes = 7680;

// States of a chunk: ten up to 16 links, then as many as keep a warp's poses within
// kFkWarpBytes (at least one).  More states a warp shorten the walk along the links per
// state, fewer leave room for more warps: 199,277 states of a robot of 30 links (60 spheres)
// take 210 us with 3, 194 with 4, 172 with 5, 179 with 7, 212 with 10; 314 us with a kernel
// of one state a warp, which robots of more than 16 links had.
inline int fk_chunk_states(const DevRobot &R) {
    return std::max(1, std::min(kFkChunk, kFkWarpBytes / (int)(sizeof(float) * 12 * std::max(R.L, 1))));
}
__host__ __device__ inline size_t smem_fk_chunk_warp(const DevRobot &R, int kc) {
    return align16(sizeof(float) * 12 * R.L * kc);
}

__global__ void __launch_bounds__(kChunkWarps *kWarp)
    k_fk_chunk(DevRobot R, const float *__restrict__ q, long long n, int kc, float *__restrict__ poses,
               float *__restrict__ centers, int vec) {
    extern __shared__ __align__(16) unsigned char smem[];
    const DevEnv E{};
    SmemTables t = carve_tables(smem, R, 0);
    if (!stage_tables(R, E, t, 0)) return;
    const int warp = threadIdx.x / kWarp, lane = threadIdx.x & 31;
    unsigned char *wbase = smem + smem_tables_bytes(R, 0) + smem_fk_chunk_warp(R, kc) * warp;
    float *lpK = reinterpret_cast<float *>(wbase);
    const int L = R.L, S = R.S;
    const long long nchunks = (n + kc - 1) / kc;
    const long long nw = (long long)gridDim.x * kChunkWarps;
    for (long long c = blockIdx.x * (long long)kChunkWarps + warp; c < nchunks; c += nw) {
        const long long s0 = c * kc;
        const int ks = (int)min((long long)kc, n - s0);
        const float *qc = q + s0 * L;
        warp_fk_chunk_q<kFkChunk, 4>(t, L, ks, [&](int k, int i) { return qc[k * L + i]; }, lpK, lane);
        store_fk_states(t, L, S, lpK, s0, ks, poses, centers, vec, lane);
        __syncwarp();
    }
}

gbmp_status fk_chunk_launch(const DevRobot &R, int num_sms, const float *q, long long n, float *poses,
                            float *centers, cudaStream_t s) {
    const int kc = fk_chunk_states(R);
    const size_t smem = smem_tables_bytes(R, 0) + smem_fk_chunk_warp(R, kc) * kChunkWarps;
    gbmp_status st = ensure_smem_optin((const void *)k_fk_chunk);
    if (st) return st;
    int per_sm = 0;
    GBMP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_fk_chunk, kChunkWarps * kWarp, smem));
    if (per_sm < 1) {
        set_error("FK kernel does not fit on an SM (%zu bytes of shared memory)", smem);
        return GBMP_ERR_CAPACITY;
    }
    long long grid = (long long)per_sm * num_sms;
    const long long need = ((n + kc - 1) / kc + kChunkWarps - 1) / kChunkWarps;
    if (need < grid) grid = need;
    const int vec = (reinterpret_cast<uintptr_t>(poses) & 15u) == 0;
    k_fk_chunk<<<(int)grid, kChunkWarps * kWarp, smem, s>>>(R, q, n, kc, poses, centers, vec);
    GBMP_CUDA(cudaGetLastError());
    return GBMP_OK;
}

}  // namespace gbmp
