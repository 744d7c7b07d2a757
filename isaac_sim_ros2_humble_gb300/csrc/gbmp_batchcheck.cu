// gbmp_batchcheck.cu -- state checks of many (robot, scene) requests in one launch.
//
// The reference checks one space's states per call (SingleArmSpace::checkStates,
// SingleArmSpace.cu:1572-1602): requests of different robots or scenes are separate
// launches.  Here a descriptor table lists the requests (robot tables, scene, inputs,
// outputs), and a second table splits their states into block-sized ranges; every block
// stages the tables of its own request into shared memory (bulk asynchronous copies) and
// checks its range with the routines of k_check_verdicts (several states a warp,
// check_verdicts) or k_check_costs (one, check_costs), so each request's outputs are
// bit-identical to a gbmp_check_states_fk call of its own.  Shared memory is sized for the
// largest request; the spheres-per-lane template of the costs covers the robot with the
// most spheres (smaller robots leave slots empty).
#include <algorithm>
#include <new>

#include "gbmp_states_device.cuh"

namespace gbmp {

struct CheckTask {
    DevRobot R;
    DevEnv E;
    const float *q;
    long long n;
    unsigned char *verdict;
    float *costs, *total, *poses, *centers;
};

struct CheckRange {
    int task, pad;
    long long lo, hi;
};

template <int SPL>
__global__ void __launch_bounds__(kWarpsPerBlock *kWarp, 4)
    k_batch_costs(const CheckTask *__restrict__ tasks, const CheckRange *__restrict__ ranges) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ CheckTask sT;
    __shared__ CheckRange sB;
    if (threadIdx.x == 0) {
        sB = ranges[blockIdx.x];
        sT = tasks[sB.task];
    }
    __syncthreads();
    const DevRobot &R = sT.R;
    const DevEnv &E = sT.E;
    const int nwords = env_words(E.ns, E.nb, E.nc);
    SmemTables t = carve_tables(smem, R, nwords);
    if (!stage_tables(R, E, t, nwords)) return;
    WarpScratch w = carve_warp(smem + smem_tables_bytes(R, nwords), R, threadIdx.x / kWarp);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (long long s = sB.lo + threadIdx.x / kWarp; s < sB.hi; s += kWarpsPerBlock)
        check_costs<SPL>(t, R, E, w, sT.q, s, sT.n, sT.verdict, sT.costs, sT.total, sT.poses, sT.centers, lane);
}

// `ks` states a warp at a time.  256 requests over 4 robots and 16 scenes, 1.57 million
// states: 5.38 ms with one warp for each state, 1.46 ms now.
template <bool CNT, bool TIGHT>
__global__ void __launch_bounds__(kStatesWarps *kWarp, kStatesResident / kStatesWarps)
    k_batch_verdicts(const CheckTask *__restrict__ tasks, const CheckRange *__restrict__ ranges, int ks) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ CheckTask sT;
    __shared__ CheckRange sB;
    if (threadIdx.x == 0) {
        sB = ranges[blockIdx.x];
        sT = tasks[sB.task];
    }
    __syncthreads();
    const DevRobot &R = sT.R;
    const DevEnv &E = sT.E;
    const int nwords = env_words(E.ns, E.nb, E.nc);
    SmemTables t = carve_tables(smem, R, nwords);
    if (!stage_tables(R, E, t, nwords)) return;
    const int warps = blockDim.x / kWarp, warp = threadIdx.x / kWarp, lane = threadIdx.x & 31;
    const StatesScratch sc = carve_states(smem + smem_tables_bytes(R, nwords), R, ks, warp);
    const int vec = (reinterpret_cast<unsigned long long>(sT.poses) & 15ull) == 0;
    for (long long s = sB.lo + warp * ks; s < sB.hi; s += warps * ks)
        check_verdicts<CNT, TIGHT>(t, R, E, sc, sT.q, s, (int)min((long long)ks, sB.hi - s), sT.verdict, sT.poses,
                                   sT.centers, vec, lane);
}

#define GBMP_BATCH_SPL_SWITCH(spl, ...)                    \
    switch (spl) {                                         \
    case 1: { constexpr int SPL = 1; __VA_ARGS__; } break; \
    case 2: { constexpr int SPL = 2; __VA_ARGS__; } break; \
    case 3: { constexpr int SPL = 3; __VA_ARGS__; } break; \
    case 4: { constexpr int SPL = 4; __VA_ARGS__; } break; \
    case 5: { constexpr int SPL = 5; __VA_ARGS__; } break; \
    case 6: { constexpr int SPL = 6; __VA_ARGS__; } break; \
    case 7: { constexpr int SPL = 7; __VA_ARGS__; } break; \
    default: { constexpr int SPL = 8; __VA_ARGS__; } break; \
    }

// Blocks per SM a launch may use: eight waves of the most blocks an SM can hold (eight
// of 256 threads), so that ranges of uneven requests even out across the SMs.
constexpr int kBatchBlocksPerSm = 64;

}  // namespace gbmp

using namespace gbmp;

struct gbmp_check_batch_s {
    int device = 0, num_sms = 0, max_requests = 0, max_ranges = 0;
    unsigned char *h_buf = nullptr;   // pinned: tasks, then ranges
    unsigned char *d_buf = nullptr;
    size_t bytes = 0;
    std::vector<int> order;           // the requests of a call that have states, as they are listed
    cudaEvent_t uploaded = nullptr;   // the last upload from h_buf has been read
    bool pending = false;
};

extern "C" {

gbmp_status gbmp_check_batch_create(int32_t max_requests, gbmp_check_batch *out) {
    GBMP_CHECK_ARG(out, "out is NULL");
    GBMP_CHECK_ARG(max_requests >= 1 && max_requests <= (1 << 20), "max_requests %d outside [1, 2^20]",
                   max_requests);
    *out = nullptr;
    auto *b = new gbmp_check_batch_s();
    b->max_requests = max_requests;
    gbmp_status st = GBMP_OK;
    do {
        if (cudaGetDevice(&b->device) != cudaSuccess ||
            cudaDeviceGetAttribute(&b->num_sms, cudaDevAttrMultiProcessorCount, b->device) != cudaSuccess) {
            set_error("no CUDA device");
            st = GBMP_ERR_CUDA;
            break;
        }
        b->max_ranges = max_requests + kBatchBlocksPerSm * b->num_sms;
        b->bytes = align16(sizeof(CheckTask) * (size_t)max_requests) + sizeof(CheckRange) * (size_t)b->max_ranges;
        if (cudaMallocHost(&b->h_buf, b->bytes) != cudaSuccess || cudaMalloc(&b->d_buf, b->bytes) != cudaSuccess ||
            cudaEventCreateWithFlags(&b->uploaded, cudaEventDisableTiming) != cudaSuccess) {
            set_error("check batch: allocation of %zu bytes failed", b->bytes);
            st = GBMP_ERR_OUT_OF_MEMORY;
            break;
        }
        try {   // so that a call allocates nothing
            b->order.reserve((size_t)max_requests);
        } catch (const std::bad_alloc &) {
            set_error("check batch: out of host memory for %d requests", max_requests);
            st = GBMP_ERR_OUT_OF_MEMORY;
        }
    } while (false);
    if (st) {
        gbmp_check_batch_destroy(b);
        return st;
    }
    *out = b;
    return GBMP_OK;
}

gbmp_status gbmp_check_batch_destroy(gbmp_check_batch b) {
    if (!b) return GBMP_OK;
    if (b->uploaded) {
        cudaEventSynchronize(b->uploaded);
        cudaEventDestroy(b->uploaded);
    }
    if (b->h_buf) cudaFreeHost(b->h_buf);
    if (b->d_buf) cudaFree(b->d_buf);
    delete b;
    return GBMP_OK;
}

gbmp_status gbmp_check_batch_run(gbmp_check_batch b, const gbmp_check_request *reqs, int32_t n_reqs, int32_t mode,
                                 void *stream) {
    GBMP_CHECK_ARG(b, "batch is NULL");
    GBMP_CHECK_ARG(n_reqs >= 0 && n_reqs <= b->max_requests, "%d requests, the batch holds %d", n_reqs,
                   b->max_requests);
    GBMP_CHECK_ARG(n_reqs == 0 || reqs, "requests is NULL");
    GBMP_CHECK_ARG(mode == GBMP_CHECK_VERDICT || mode == GBMP_CHECK_COST, "unknown mode %d", mode);
    int dev = 0;
    GBMP_CUDA(cudaGetDevice(&dev));
    GBMP_CHECK_ARG(dev == b->device, "the batch was created on device %d, current device is %d", b->device, dev);
    for (int i = 0; i < n_reqs; ++i) {
        const gbmp_check_request &q = reqs[i];
        GBMP_CHECK_ARG(q.robot && q.env, "request %d: robot/env is NULL", i);
        GBMP_CHECK_ARG(q.n >= 0, "request %d: n < 0", i);
        GBMP_CHECK_ARG(q.n == 0 || q.d_q, "request %d: q is NULL", i);
        GBMP_CHECK_ARG(q.robot->device == dev, "request %d: robot on device %d", i, q.robot->device);
    }
    // the previous call's upload must have been read before the pinned tables change
    if (b->pending) {
        GBMP_CUDA(cudaEventSynchronize(b->uploaded));
        b->pending = false;
    }
    auto *tasks = reinterpret_cast<CheckTask *>(b->h_buf);
    // requests of one robot and scene next to each other, so that the blocks the GPU
    // schedules together share their tables (in L2) and their path through the routine
    // (measured 5.74 against 6.05 ms on the 256-request benchmark mix); sorted by their
    // numbers, for a task is half a kilobyte
    b->order.clear();
    for (int i = 0; i < n_reqs; ++i)
        if (reqs[i].n) b->order.push_back(i);
    std::stable_sort(b->order.begin(), b->order.end(), [reqs](int x, int y) {
        const gbmp_check_request &p = reqs[x], &q = reqs[y];
        if (p.robot != q.robot) return p.robot->dev.stage < q.robot->dev.stage;
        return p.env->view.words < q.env->view.words;
    });
    const bool cost = mode == GBMP_CHECK_COST;
    int nt = 0, spl = 1;
    size_t smem = 0;   // of the costs' kernel, which also says which requests fit
    size_t tables = 0;
    DevRobot widest{};
    bool tight = true;   // every scene is
    long long total = 0;
    unsigned long long *work = work_counter();
    for (int i : b->order) {
        const gbmp_check_request &q = reqs[i];
        CheckTask &T = tasks[nt++];
        T.R = cost ? q.robot->dev : q.robot->dev_chunk;
        T.R.work = work;
        T.E = q.env->dev();
        T.q = q.d_q;
        T.n = q.n;
        T.verdict = q.d_verdict;
        T.costs = mode == GBMP_CHECK_COST ? q.d_costs : nullptr;
        T.total = mode == GBMP_CHECK_COST ? q.d_total : nullptr;
        T.poses = q.d_poses;
        T.centers = q.d_centers;
        spl = std::max(spl, T.R.spl);
        const int words = env_words(T.E.ns, T.E.nb, T.E.nc);
        smem = std::max(smem, smem_tables_bytes(q.robot->dev, words) + smem_warp_bytes(q.robot->dev) * kWarpsPerBlock);
        tables = std::max(tables, smem_tables_bytes(T.R, words));
        widest.L = std::max(widest.L, T.R.L);
        widest.G = std::max(widest.G, T.R.G);
        tight = tight && q.env->tight;
        total += q.n;
    }
    if (nt == 0) return GBMP_OK;
    int optin = 0;
    GBMP_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    if (smem + 1024 > (size_t)optin) {
        set_error("check batch: the largest request needs %zu bytes of shared memory", smem);
        return GBMP_ERR_CAPACITY;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const void *fn = nullptr;
    StatesShape sh{1, kWarpsPerBlock, 1, smem};
    if (cost) {
        GBMP_BATCH_SPL_SWITCH(spl, { fn = (const void *)k_batch_costs<SPL>; });
    } else {
        fn = work ? (tight ? (const void *)k_batch_verdicts<true, true> : (const void *)k_batch_verdicts<true, false>)
                  : (tight ? (const void *)k_batch_verdicts<false, true> : (const void *)k_batch_verdicts<false, false>);
    }
    gbmp_status st = ensure_smem_optin(fn);
    if (st) return st;
    if (cost) {
        GBMP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&sh.per_sm, fn, kWarpsPerBlock * kWarp, smem));
        if (sh.per_sm < 1) sh.per_sm = 1;
    } else {
        // one shape for all requests: the largest tables, and the scratch of a warp of as many
        // links and groups as any has
        const size_t limit = kSmemLimit - sizeof(CheckTask) - sizeof(CheckRange) - 16;
        const long long resident = (long long)kStatesResident * b->num_sms;
        const int want = (int)std::min<long long>(kStatesKs, (total + resident - 1) / resident);
        if (!states_shape(tables, [&](int ks) { return smem_states_bytes(widest, ks); }, want, limit, &sh)) {
            set_error("check batch: the largest request needs %zu bytes of shared memory", smem);
            return GBMP_ERR_CAPACITY;
        }
    }
    // states per block: about eight waves over all requests (when it was chosen, 1.53 ms on
    // the 256-request mix above; four: 1.57, sixteen: 1.52), at least one round of its warps
    const long long unit = (long long)sh.warps * sh.ks;
    const long long target = (long long)std::min(8 * sh.per_sm, kBatchBlocksPerSm) * b->num_sms;
    long long spb = (total + target - 1) / target;
    spb = std::max<long long>(spb, cost ? 4 * unit : unit);   // costs: at least four states a warp
    spb = (spb + unit - 1) / unit * unit;
    const size_t ranges_off = align16(sizeof(CheckTask) * (size_t)nt);   // the ranges follow the tasks: one copy
    auto *ranges = reinterpret_cast<CheckRange *>(b->h_buf + ranges_off);
    int nr = 0;
    for (int ti = 0; ti < nt; ++ti)
        for (long long lo = 0; lo < tasks[ti].n; lo += spb) {
            if (nr == b->max_ranges) {
                set_error("check batch: more than %d block ranges", b->max_ranges);
                return GBMP_ERR_CAPACITY;
            }
            ranges[nr++] = CheckRange{ti, 0, lo, std::min(lo + spb, tasks[ti].n)};
        }
    GBMP_CUDA(cudaMemcpyAsync(b->d_buf, b->h_buf, ranges_off + sizeof(CheckRange) * (size_t)nr,
                              cudaMemcpyHostToDevice, s));
    GBMP_CUDA(cudaEventRecord(b->uploaded, s));
    b->pending = true;
    const auto *d_tasks = reinterpret_cast<const CheckTask *>(b->d_buf);
    const auto *d_ranges = reinterpret_cast<const CheckRange *>(b->d_buf + ranges_off);
    ProfScope ps(GBMP_PROF_CHECK_STATES, s);
    void *args[] = {&d_tasks, &d_ranges, &sh.ks};   // the costs' kernel takes the first two
    GBMP_CUDA(cudaLaunchKernel(fn, dim3(nr), dim3(sh.warps * kWarp), args, sh.smem, s));
    return GBMP_OK;
}

}  // extern "C"
