// gbmp_project.cu -- projection of joint states onto a task-space region and the joint
// limits, replacing SingleArmSpace::projectStates (SingleArmSpace.cu:1631-1662) with
// TaskSpaceConstraint::computeGradientAndError / computeCost
// (TaskSpaceConstraint.cu:66-139, :167-396) and BoundaryConstraint
// (BoundaryConstraint.cu:36-155).
//
// One warp per state, all iterations in one launch (the reference launches FK, one
// gradient kernel per constraint, a gradient sum and an update kernel per iteration,
// each followed by a device synchronisation, and allocates the Jacobian buffers on
// every call).  Arithmetic is written with explicit rounding in the reference's operation
// order.
//
// What bounds it: the latency of one iteration's chain of dependent steps (a motion is
// hundreds of iterations, each needing the last; one warp issues an instruction every five
// cycles or so).  So the state lives in registers, joint j on lane j (and j + 32); sums that
// have an order are summed in it from shuffled registers, by every lane; the 21 sums of the
// damped 6 x 6 system stand one on a lane, its inversion has one column of [A | I] on each
// of twelve lanes with the rows in registers; the task frame's angles are computed side by
// side; recorded states of a motion are collision-checked eight at a time.  A pass takes
// 2.4 us alone: FK 0.7, task frame 0.4, the sums 0.2, the inversion 0.9.  Before, lane 0
// inverted the system element by element in shared memory and summed every norm alone:
// 200 motions of the 7-DOF arm took 16.2 ms, 4.3 ms now; 4,096 projections of 10 rounds
// 231 us, 82 us now.
#include <cmath>

#include "gbmp_states_device.cuh"

namespace gbmp {
namespace {

struct ProjParams {
    int task_link, use_boundary, iterations;
    float offset[16], reference[6], tolerance[6];
};

// A warp's scratch: link poses, joint-local transforms, the Jacobian (8 floats for each
// joint, up to a multiple of 4 joints) and the inverse (8 floats a column).
struct ProjScratch {
    float *lp, *loc, *J, *inv;
    // constrained motions: recorded states waiting for their check [kCheckStates][L], the
    // limits of the active joints [2][L] (none for the others), and the check's scratch
    float *rec, *lim;
    StatesScratch sc;
};

constexpr int kCheckStates = 8;   // recorded states checked together

__host__ __device__ inline size_t proj_warp_bytes(const DevRobot &R) {
    return 2 * align16(sizeof(float) * 12 * R.L) + sizeof(float) * 8 * (R.L + 3) + sizeof(float) * 48;
}
__host__ __device__ inline size_t cm_warp_bytes(const DevRobot &R) {
    return proj_warp_bytes(R) + align16(sizeof(float) * (kCheckStates + 2) * R.L) + smem_states_bytes(R, kCheckStates);
}

__device__ inline ProjScratch carve_proj(unsigned char *p, const DevRobot &R, bool checks) {
    ProjScratch c{};
    c.lp = reinterpret_cast<float *>(p); p += align16(sizeof(float) * 12 * R.L);
    c.loc = reinterpret_cast<float *>(p); p += align16(sizeof(float) * 12 * R.L);
    c.J = reinterpret_cast<float *>(p); p += sizeof(float) * 8 * (R.L + 3);
    c.inv = reinterpret_cast<float *>(p); p += sizeof(float) * 48;
    if (checks) {
        c.rec = reinterpret_cast<float *>(p);
        c.lim = c.rec + kCheckStates * R.L;
        p += align16(sizeof(float) * (kCheckStates + 2) * R.L);
        c.sc = carve_states(p, R, kCheckStates, 0);
    }
    return c;
}

__device__ __forceinline__ float dot3(float a0, float a1, float a2, float b0, float b1, float b2) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a0, b0), __fmul_rn(a1, b1)), __fmul_rn(a2, b2));
}

__device__ __forceinline__ float dead(float diff, float tol) {
    return copysignf(fmaxf(__fadd_rn(fabsf(diff), -tol), 0.0f), diff);
}

// What a lane keeps for the whole launch.  U: joints a lane (1 for up to 32 links, else 2).
// Lanes 0 .. 5 hold the components roll, pitch, yaw, x, y, z of the task frame's reference
// and tolerance; a lane's column of the frame's offset serves its element of the frame.
// Lanes 0 .. 20 hold the pairs row <= col of 0 .. 5 (pair_lane), the others (5, 5).
__host__ __device__ constexpr int pair_lane(int row, int col) { return row * 6 - row * (row - 1) / 2 + col - row; }

template <int U>
struct LaneConst {
    float off[4], ref, tol;
    int row, col;
    float lo[U], hi[U];
    bool act[U];
};

template <int U>
__device__ __forceinline__ LaneConst<U> lane_const(const DevRobot &R, const ProjParams &p, int lane) {
    LaneConst<U> c;
#pragma unroll
    for (int m = 0; m < 4; ++m) c.off[m] = p.offset[4 * m + (lane & 3)];
    const int k = lane < 3 ? lane + 3 : lane < 6 ? lane - 3 : 0;   // its place in x, y, z, roll, pitch, yaw
    c.ref = p.reference[k];
    c.tol = p.tolerance[k];
    c.row = c.col = 5;
    for (int i = 0; i < 6; ++i)
        for (int j = i; j < 6; ++j)
            if (pair_lane(i, j) == lane) { c.row = i; c.col = j; }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int j = lane + kWarp * u;
        c.act[u] = j < R.L && R.active[j] != 0;
        c.lo[u] = j < R.L ? R.lower[j] : 0.f;
        c.hi[u] = j < R.L ? R.upper[j] : 0.f;
    }
    return c;
}

// Sum over the joints in joint order of the lanes' values (rounded adds, from 0), on every
// lane.
template <int U>
__device__ __forceinline__ float ordered_sum(const float (&v)[U], int L) {
    float s = 0.f;
#pragma unroll
    for (int u = 0; u < U; ++u)
        for (int j = 0; j < min(L - kWarp * u, kWarp); ++j) s = __fadd_rn(s, __shfl_sync(kFull, v[u], j));
    return s;
}

// FK of the state in the lanes' registers into lp (warp_fk's arithmetic): the joint-local
// transforms, then lanes 0 .. 2 walk the chain, one pose row each, the next link's
// transform loaded a step ahead.
template <int U>
__device__ __forceinline__ void warp_fk_lanes(const SmemTables &t, int L, const float (&q)[U], float *loc, float *lp,
                                              int lane) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int i = lane + kWarp * u;
        if (i > 0 && i < L) joint_local(t, i, q[u], loc + 12 * i);
    }
    __syncwarp();
    if (lane < 3) {
        const float4 unit = make_float4(lane == 0 ? 1.f : 0.f, lane == 1 ? 1.f : 0.f, lane == 2 ? 1.f : 0.f, 0.f);
        float4 *rowp = reinterpret_cast<float4 *>(lp) + lane;
        const float4 *b = reinterpret_cast<const float4 *>(loc);
        float4 a = unit, b0, b1, b2;
        int ty = 0, par = 0;
        *rowp = a;
        if (L > 1) { b0 = b[3]; b1 = b[4]; b2 = b[5]; ty = t.type[1]; par = t.parent[1]; }
        for (int i = 1; i < L; ++i) {
            const int n = min(i + 1, L - 1);
            const float4 n0 = b[3 * n], n1 = b[3 * n + 1], n2 = b[3 * n + 2];
            const int nty = t.type[n], npar = t.parent[n];
            if (par != i - 1) a = rowp[3 * par];
            float4 o = unit;
            if (ty == 1 || ty == 2 || ty == 5) {
                o.x = __fmaf_rn(a.z, b2.x, __fmaf_rn(a.y, b1.x, __fmul_rn(a.x, b0.x)));
                o.y = __fmaf_rn(a.z, b2.y, __fmaf_rn(a.y, b1.y, __fmul_rn(a.x, b0.y)));
                o.z = __fmaf_rn(a.z, b2.z, __fmaf_rn(a.y, b1.z, __fmul_rn(a.x, b0.z)));
                o.w = __fadd_rn(__fmaf_rn(a.z, b2.w, __fmaf_rn(a.y, b1.w, __fmul_rn(a.x, b0.w))), a.w);
            }
            rowp[3 * i] = o;
            a = o;
            b0 = n0; b1 = n1; b2 = n2; ty = nty; par = npar;
        }
    }
    __syncwarp();
}

// The task frame, rows 0 .. 2 of (link pose, implicit last row 0 0 0 1) x offset
// (TaskSpaceConstraint.cu:47-63), one element a lane (lanes 0 .. 11), and its component on
// lanes 0 .. 5: roll, pitch, yaw, x, y, z.  pos: the frame's position, on every lane.
template <int U>
__device__ __forceinline__ float task_component(const float *lp, int link, const LaneConst<U> &c, float3 &pos, int lane) {
    const float4 T = reinterpret_cast<const float4 *>(lp + 12 * link)[lane < 12 ? lane >> 2 : 0];
    const float P = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(T.x, c.off[0]), __fmul_rn(T.y, c.off[1])),
                                        __fmul_rn(T.z, c.off[2])),
                              __fmul_rn(T.w, c.off[3]));
    pos = make_float3(__shfl_sync(kFull, P, 3), __shfl_sync(kFull, P, 7), __shfl_sync(kFull, P, 11));
    const float ay = __shfl_sync(kFull, P, lane == 0 ? 9 : 4), ax = __shfl_sync(kFull, P, lane == 0 ? 10 : 0);
    const float sp = __shfl_sync(kFull, P, 8);
    const float turn = atan2f(ay, ax);   // lane 0 the roll, the others the yaw
    const float pitch = asinf(-sp);
    return lane == 0 || lane == 2 ? turn : lane == 1 ? pitch : lane == 3 ? pos.x : lane == 4 ? pos.y : pos.z;
}

// One projection pass on the state in q (TaskSpaceConstraint::computeGradientAndError,
// TaskSpaceConstraint.cu:167-396; BoundaryConstraint.cu:36-155; update_with_grad, step 1):
// FK, the dead-banded task error and its damped pseudo-inverse step, the joint-limit
// pull, both added to the active joints.  Returns, on every lane, the total error the
// gradient kernels record for the state before the update: the norm of the dead-banded
// task error plus the norm of the limit violations (SingleArmStates.cu:847-871).
template <int U>
__device__ __forceinline__ float proj_pass(const SmemTables &t, const DevRobot &R, const ProjParams &p,
                                           const ProjScratch &w, const LaneConst<U> &lc, float (&q)[U], int lane) {
    const int L = R.L;
    const float *lp = w.lp;
    float gt[U], err = 0.f;
#pragma unroll
    for (int u = 0; u < U; ++u) gt[u] = 0.f;
    if (p.task_link >= 0) {
        warp_fk_lanes<U>(t, L, q, w.loc, w.lp, lane);
        float3 pos;
        const float val = task_component<U>(lp, p.task_link, lc, pos, lane);
        const float e = dead(__fadd_rn(lc.ref, -val), lc.tol);
        float E[6], e2 = 0.f;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            E[k] = __shfl_sync(kFull, e, k);
            e2 = __fadd_rn(e2, __fmul_rn(E[k], E[k]));
        }
        err = __fsqrt_rn(e2);
        float col[U][6];   // Jacobian columns of the lane's joints
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = lane + kWarp * u;
            float c0 = 0.f, c1 = 0.f, c2 = 0.f, c3 = 0.f, c4 = 0.f, c5 = 0.f;
            if (j <= p.task_link && lc.act[u]) {   // only the active joints' columns are used
                const float4 *T = reinterpret_cast<const float4 *>(lp + 12 * j);
                const float4 r0 = T[0], r1 = T[1], r2 = T[2];
                const float *a = t.axr + 4 * j;
                const float w0 = dot3(r0.x, r0.y, r0.z, a[0], a[1], a[2]);
                const float w1 = dot3(r1.x, r1.y, r1.z, a[0], a[1], a[2]);
                const float w2 = dot3(r2.x, r2.y, r2.z, a[0], a[1], a[2]);
                if (t.type[j] == 1) {
                    const float d0 = __fadd_rn(pos.x, -r0.w), d1 = __fadd_rn(pos.y, -r1.w), d2 = __fadd_rn(pos.z, -r2.w);
                    c0 = w0; c1 = w1; c2 = w2;
                    c3 = __fadd_rn(__fmul_rn(w1, d2), -__fmul_rn(w2, d1));
                    c4 = __fadd_rn(__fmul_rn(w2, d0), -__fmul_rn(w0, d2));
                    c5 = __fadd_rn(__fmul_rn(w0, d1), -__fmul_rn(w1, d0));
                } else if (t.type[j] == 2) {
                    c3 = w0; c4 = w1; c5 = w2;
                }
            }
            col[u][0] = c0; col[u][1] = c1; col[u][2] = c2; col[u][3] = c3; col[u][4] = c4; col[u][5] = c5;
            if (j < (p.task_link + 4) / 4 * 4) {   // rows of 0 up to a multiple of 4
                float4 *o = reinterpret_cast<float4 *>(w.J + 8 * j);
                o[0] = make_float4(c0, c1, c2, c3);
                o[1] = make_float4(c4, c5, 0.f, 0.f);
            }
        }
        __syncwarp();
        // J_a J_a^T in joint order (a joint that is not active adds 0), one of its 21 sums a
        // lane, then column `lane` of [J_a J_a^T + 1e-4 I | I] (lanes 0 .. 11)
        float sum = 0.f;
        for (int k0 = 0; k0 <= p.task_link; k0 += 4) {
            float x[4], y[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                x[u] = w.J[8 * (k0 + u) + lc.row];
                y[u] = w.J[8 * (k0 + u) + lc.col];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) sum = __fadd_rn(sum, __fmul_rn(x[u], y[u]));
        }
        if (lc.row == lc.col) sum = __fadd_rn(sum, 1e-4f);
        float A[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const float v = __shfl_sync(kFull, sum, pair_lane(min(i, min(lane, 5)), max(i, min(lane, 5))));
            A[i] = lane < 6 ? v : lane == 6 + i ? 1.f : 0.f;
        }
        // Gauss-Jordan without pivoting (TaskSpaceConstraint.cu:305-350): per pivot the
        // pivot column first (independent of the division), then the divided row
        bool invertible = true;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            float f[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) f[k] = __shfl_sync(kFull, A[k], i);
            invertible = invertible && !(fabsf(f[i]) < 1e-8f);
            A[i] = __fdiv_rn(A[i], f[i]);
#pragma unroll
            for (int k = 0; k < 6; ++k)
                if (k != i) A[k] = __fadd_rn(A[k], -__fmul_rn(f[k], A[i]));
        }
        if (lane >= 6 && lane < 12) {
            float4 *o = reinterpret_cast<float4 *>(w.inv + 8 * (lane - 6));
            o[0] = make_float4(A[0], A[1], A[2], A[3]);
            o[1] = make_float4(A[4], A[5], 0.f, 0.f);
        }
        __syncwarp();
        if (invertible) {
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                const float4 v0 = reinterpret_cast<const float4 *>(w.inv + 8 * i)[0];
                const float2 v1 = *reinterpret_cast<const float2 *>(w.inv + 8 * i + 4);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    float sum = __fadd_rn(0.0f, __fmul_rn(col[u][0], v0.x));
                    sum = __fadd_rn(sum, __fmul_rn(col[u][1], v0.y));
                    sum = __fadd_rn(sum, __fmul_rn(col[u][2], v0.z));
                    sum = __fadd_rn(sum, __fmul_rn(col[u][3], v0.w));
                    sum = __fadd_rn(sum, __fmul_rn(col[u][4], v1.x));
                    sum = __fadd_rn(sum, __fmul_rn(col[u][5], v1.y));
                    gt[u] = __fadd_rn(gt[u], __fmul_rn(sum, E[i]));
                }
            }
        }
    }
    // joint limits: the pull of each joint, and the norm of the violations in joint order
    float gb[U];
    bool out = false;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        gb[u] = 0.f;
        if (p.use_boundary && lc.act[u]) {
            if (q[u] < lc.lo[u]) gb[u] = __fadd_rn(lc.lo[u], -q[u]);
            else if (q[u] > lc.hi[u]) gb[u] = __fadd_rn(lc.hi[u], -q[u]);
        }
        out |= gb[u] != 0.f;
    }
    if (__any_sync(kFull, out)) {
        float v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = __fmul_rn(gb[u], gb[u]);
        err = __fadd_rn(err, __fsqrt_rn(ordered_sum<U>(v, L)));
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (lc.act[u]) q[u] = __fadd_rn(q[u], __fadd_rn(gt[u], gb[u]));
    return err;
}

// computeCost of the task-space constraint (TaskSpaceConstraint.cu:140-176, zero below
// 1e-4) and of the joint limits (BoundaryConstraint.cu:36-95, zero below 1e-4 before the
// square root) for the state in q whose FK is in lp, on every lane.
template <int U>
__device__ __forceinline__ void proj_costs(const DevRobot &R, const ProjParams &p, const float *lp,
                                           const LaneConst<U> &lc, const float (&q)[U], int lane, float &tc, float &bc) {
    tc = 0.f;
    bc = 0.f;
    if (p.task_link >= 0) {
        float3 pos;
        const float val = task_component<U>(lp, p.task_link, lc, pos, lane);
        const float d = __fadd_rn(val, -lc.ref);
        const float term = fmaxf(__fadd_rn(__fmul_rn(d, d), -__fmul_rn(lc.tol, lc.tol)), 0.f);
#pragma unroll
        for (int k = 0; k < 6; ++k) tc = __fadd_rn(tc, __shfl_sync(kFull, term, k < 3 ? k + 3 : k - 3));   // x first
        tc = __fsqrt_rn(tc);
        if (tc < 1e-4f) tc = 0.f;
    }
    if (p.use_boundary) {
        float v[U];
        bool out = false;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            v[u] = 0.f;
            if (lc.act[u]) {
                if (q[u] < lc.lo[u]) v[u] = __fmul_rn(__fadd_rn(lc.lo[u], -q[u]), __fadd_rn(lc.lo[u], -q[u]));
                else if (q[u] > lc.hi[u]) v[u] = __fmul_rn(__fadd_rn(q[u], -lc.hi[u]), __fadd_rn(q[u], -lc.hi[u]));
            }
            out |= v[u] != 0.f;
        }
        if (__any_sync(kFull, out)) {
            bc = ordered_sum<U>(v, R.L);
            bc = bc < 1e-4f ? 0.f : __fsqrt_rn(bc);
        }
    }
}

// checkStates on the nb recorded states in w.rec: true when every one is collision-free and
// has no task-space and no limit cost (proj_costs' arithmetic, one state a lane).
template <bool TIGHT>
__device__ __forceinline__ bool recorded_pass(const SmemTables &t, const DevRobot &R, const DevEnv &E,
                                              const ProjParams &p, const ProjScratch &w, int nb, int lane) {
    const int L = R.L;
    warp_fk_chunk_q<kStatesMax>(t, L, nb, [&](int k, int i) { return w.rec[k * L + i]; }, w.sc.lpK, lane);
    bool bad = false;
    if (lane < nb) {
        if (p.task_link >= 0) {
            const float4 *T = reinterpret_cast<const float4 *>(w.sc.lpK + 12 * (lane * L + p.task_link));
            const float4 r[3] = {T[0], T[1], T[2]};
            auto elem = [&](int row, int c) {
                return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(r[row].x, p.offset[c]), __fmul_rn(r[row].y, p.offset[4 + c])),
                                           __fmul_rn(r[row].z, p.offset[8 + c])),
                                 __fmul_rn(r[row].w, p.offset[12 + c]));
            };
            const float v[6] = {elem(0, 3), elem(1, 3), elem(2, 3), atan2f(elem(2, 1), elem(2, 2)), asinf(-elem(2, 0)),
                                atan2f(elem(1, 0), elem(0, 0))};
            float tc = 0.f;
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                const float d = __fadd_rn(v[k], -p.reference[k]), tl = p.tolerance[k];
                tc = __fadd_rn(tc, fmaxf(__fadd_rn(__fmul_rn(d, d), -__fmul_rn(tl, tl)), 0.f));
            }
            bad = !(__fsqrt_rn(tc) < 1e-4f);
        }
        if (p.use_boundary) {
            float bc = 0.f;
            for (int j = 0; j < L; ++j) {
                const float qv = w.rec[lane * L + j], lo = w.lim[j], hi = w.lim[L + j];
                const float d = qv < lo ? __fadd_rn(lo, -qv) : qv > hi ? __fadd_rn(qv, -hi) : 0.f;
                bc = __fadd_rn(bc, __fmul_rn(d, d));
            }
            bad = bad || !(bc < 1e-4f);
        }
    }
    if (__any_sync(kFull, bad)) return false;
    return warp_verdicts<false, TIGHT>(t, R, E, w.sc, nb, lane) == 0u;
}

template <int U>
__global__ void __launch_bounds__(kWarpsPerBlock *kWarp)
    k_project(DevRobot R, ProjParams p, float *__restrict__ qall, long long n, float *__restrict__ task_cost,
              float *__restrict__ bound_cost) {
    extern __shared__ __align__(16) unsigned char smem[];
    DevEnv E0{};
    SmemTables t = carve_tables(smem, R, 0);
    if (!stage_tables(R, E0, t, 0)) return;
    const int warps = blockDim.x / kWarp, warp = threadIdx.x / kWarp, lane = threadIdx.x & 31;
    const ProjScratch w = carve_proj(smem + smem_tables_bytes(R, 0) + proj_warp_bytes(R) * warp, R, false);
    const LaneConst<U> lc = lane_const<U>(R, p, lane);
    const int L = R.L;
    const long long nw = (long long)gridDim.x * warps;
    for (long long s = blockIdx.x * (long long)warps + warp; s < n; s += nw) {
        float *qs = qall + s * L;
        float q[U];
#pragma unroll
        for (int u = 0; u < U; ++u) q[u] = lane + kWarp * u < L ? qs[lane + kWarp * u] : 0.f;
        for (int it = 0; it < p.iterations; ++it) proj_pass<U>(t, R, p, w, lc, q, lane);
        if (p.task_link >= 0) warp_fk_lanes<U>(t, L, q, w.loc, w.lp, lane);
        float tc, bc;
        proj_costs<U>(R, p, w.lp, lc, q, lane, tc, bc);
        if (lane == 0) {
            if (task_cost) task_cost[s] = tc;
            if (bound_cost) bound_cost[s] = bc;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (lane + kWarp * u < L) qs[lane + kWarp * u] = q[u];
        __syncwarp();
    }
}

// Constrained motions (SingleArmSpace::computeConstrainedMotions, SingleArmSpace.cu:1049-1366),
// one warp per motion and every iteration in one launch (the reference runs a host loop of
// up to 10,000 iterations, each with an approach kernel, two projection passes of several
// kernels, three check kernels, device synchronisations and a copy of every state to the
// host, and then collision-checks the recorded states).  Per iteration: every joint moves
// `res` along the unit direction to the goal (approachKernel, :855-886); two projection
// passes (proj_pass); the motion stops approaching when the second pass's error exceeds
// 1e-3 (checkIfCostIsZero), when the state is farther from the goal than before or moved
// more than 5 res (checkValidOfApproaching); otherwise the state is recorded and checked
// as checkStates checks it (collision, task-space cost and limit cost all zero; checks
// end at the first failure), and reaching the goal within `res` ends the motion as
// achieved (checkAchieveGoal).  ok = achieved and every recorded state passed; cost = L2
// length over all joints of the recorded states; count = recorded states (the first
// `cap` are written to `states` when it is not null).
template <int U, bool TIGHT>
__global__ void __launch_bounds__(kWarpsPerBlock *kWarp)
    k_constrained_motion(DevRobot R, DevEnv E, ProjParams p, const float *__restrict__ from,
                         const float *__restrict__ to, long long n, float res, int max_iters,
                         unsigned char *__restrict__ ok_out, float *__restrict__ cost_out,
                         int *__restrict__ count_out, float *__restrict__ states, int cap) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int nwords = env_words(E.ns, E.nb, E.nc);
    SmemTables t = carve_tables(smem, R, nwords);
    if (!stage_tables(R, E, t, nwords)) return;
    const int warps = blockDim.x / kWarp, warp = threadIdx.x / kWarp, lane = threadIdx.x & 31;
    const ProjScratch w = carve_proj(smem + smem_tables_bytes(R, nwords) + cm_warp_bytes(R) * warp, R, true);
    const LaneConst<U> lc = lane_const<U>(R, p, lane);
    const int L = R.L;
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (lane + kWarp * u < L) {
            w.lim[lane + kWarp * u] = lc.act[u] ? lc.lo[u] : __int_as_float(0xff800000);
            w.lim[L + lane + kWarp * u] = lc.act[u] ? lc.hi[u] : __int_as_float(0x7f800000);
        }
    __syncwarp();
    const long long nw = (long long)gridDim.x * warps;
    for (long long s = blockIdx.x * (long long)warps + warp; s < n; s += nw) {
        float q[U], goal[U], prev[U], last[U], v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = lane + kWarp * u;
            q[u] = j < L ? from[s * L + j] : 0.f;
            goal[u] = j < L ? to[s * L + j] : 0.f;
            last[u] = 0.f;
        }
        bool achieved = false, feasible = true;
        int steps = 0, waiting = 0;
        double len = 0.0;
        for (int it = 0; it < max_iters; ++it) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                prev[u] = q[u];
                const float d = __fadd_rn(goal[u], -q[u]);
                v[u] = __fmul_rn(d, d);
            }
            const float nrm = __fsqrt_rn(ordered_sum<U>(v, L));
            if (nrm > 1e-6f)
#pragma unroll
                for (int u = 0; u < U; ++u)
                    q[u] = __fadd_rn(q[u], __fmul_rn(__fdiv_rn(__fadd_rn(goal[u], -q[u]), nrm), res));
            proj_pass<U>(t, R, p, w, lc, q, lane);
            const float err = proj_pass<U>(t, R, p, w, lc, q, lane);
            if (err > 1e-3f) break;
            // distances of the previous and the current state from the goal, and the step:
            // the first is the norm the approach started from (the same differences)
            float moved[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float b = __fadd_rn(q[u], -goal[u]), c = __fadd_rn(prev[u], -q[u]);
                v[u] = __fmul_rn(b, b);
                moved[u] = __fmul_rn(c, c);
            }
            const float to_goal = __fsqrt_rn(ordered_sum<U>(v, L)), step = __fsqrt_rn(ordered_sum<U>(moved, L));
            if (to_goal > nrm || step > __fmul_rn(res, 5.0f)) break;   // stopped approaching: not recorded
            if (steps > 0) {
                double s2 = 0.0;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const float d = __fadd_rn(q[u], -last[u]);
                    for (int j = 0; j < min(L - kWarp * u, kWarp); ++j) {
                        const double dj = (double)__shfl_sync(kFull, d, j);
                        if (lane == 0) s2 = fma(dj, dj, s2);
                    }
                }
                if (lane == 0) len += sqrt(s2);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int j = lane + kWarp * u;
                if (states && steps < cap && j < L) states[(s * cap + steps) * L + j] = q[u];
                last[u] = q[u];
            }
            ++steps;
            if (feasible) {   // its check, with those of the states recorded next
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (lane + kWarp * u < L) w.rec[waiting * L + lane + kWarp * u] = q[u];
                __syncwarp();
                if (++waiting == kCheckStates) {
                    feasible = recorded_pass<TIGHT>(t, R, E, p, w, waiting, lane);
                    waiting = 0;
                }
            }
            if (to_goal < res) {
                achieved = true;
                break;
            }
        }
        if (achieved && feasible && waiting) feasible = recorded_pass<TIGHT>(t, R, E, p, w, waiting, lane);
        if (lane == 0) {
            const bool ok = achieved && feasible;
            if (ok_out) ok_out[s] = ok;
            if (cost_out) cost_out[s] = ok ? (float)len : 0.f;
            if (count_out) count_out[s] = steps;
        }
        __syncwarp();
    }
}

// Shared memory that decides which scenes constrained motions accept, a warp's share
// besides smem_warp_bytes.
size_t cm_limit_bytes(const DevRobot &R) {
    return align16(sizeof(float) * 6 * R.L) + align16(sizeof(float) * 72) + align16(sizeof(float) * 24) +
           3 * sizeof(float) * kMaxLinks;
}

// Warps a block and blocks for n items of one warp each: few items go to as many SMs as
// there are.
void spread_warps(long long n, int num_sms, int *warps, long long *grid) {
    *warps = kWarpsPerBlock;
    while (*warps > 1 && (n + *warps - 1) / *warps < num_sms) *warps /= 2;
    *grid = (n + *warps - 1) / *warps;
}

}  // namespace
}  // namespace gbmp

using namespace gbmp;

// Space Jacobian of every link (SingleArmStates::calculateSpaceJacobian with
// kin_space_jacobian_per_link_kernel, SingleArmStates.cu:223-338, :793-817): for link i
// and joint j, w = R_j a_j (a_j the joint's axis as given, R_j the rotation of link j's
// pose) and p the pose positions; column j is (w, w x (p_i - p_j)) for a revolute
// joint, (0, w) for a prismatic one, and zero for link 0, joint 0, j > i and other joint
// types (joint order, not ancestry, as the reference has it).  Output [n][L][L][6]
// (state, link, joint, column).  One warp per state: FK, then the lanes over (i, j).
__global__ void __launch_bounds__(kWarpsPerBlock *kWarp)
    k_space_jacobian(DevRobot R, const float *__restrict__ q, long long n, float *__restrict__ jac) {
    extern __shared__ __align__(16) unsigned char smem[];
    DevEnv E0{};
    SmemTables t = carve_tables(smem, R, 0);
    if (!stage_tables(R, E0, t, 0)) return;
    const int warp = threadIdx.x / kWarp, lane = threadIdx.x & 31;
    WarpScratch w = carve_warp(smem + smem_tables_bytes(R, 0), R, warp);
    __syncthreads();
    const int L = R.L;
    const long long nw = (long long)gridDim.x * kWarpsPerBlock;
    for (long long s = blockIdx.x * (long long)kWarpsPerBlock + warp; s < n; s += nw) {
        for (int j = lane; j < L; j += kWarp) w.q[j] = q[s * L + j];
        __syncwarp();
        warp_fk(t, L, w, lane);
        float *out = jac + s * L * L * 6;
        for (int e = lane; e < L * L; e += kWarp) {
            const int i = e / L, j = e - i * L;
            float c[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            const int ty = t.type[j];
            if (i > 0 && j > 0 && j <= i && (ty == 1 || ty == 2)) {
                const float *Tj = w.lp + 12 * j, *Ti = w.lp + 12 * i;
                const float *a = t.axr + 4 * j;
                const float w0 = dot3(Tj[0], Tj[1], Tj[2], a[0], a[1], a[2]);
                const float w1 = dot3(Tj[4], Tj[5], Tj[6], a[0], a[1], a[2]);
                const float w2 = dot3(Tj[8], Tj[9], Tj[10], a[0], a[1], a[2]);
                if (ty == 1) {
                    const float d0 = __fadd_rn(Ti[3], -Tj[3]), d1 = __fadd_rn(Ti[7], -Tj[7]),
                                d2 = __fadd_rn(Ti[11], -Tj[11]);
                    c[0] = w0; c[1] = w1; c[2] = w2;
                    c[3] = __fadd_rn(__fmul_rn(w1, d2), -__fmul_rn(w2, d1));
                    c[4] = __fadd_rn(__fmul_rn(w2, d0), -__fmul_rn(w0, d2));
                    c[5] = __fadd_rn(__fmul_rn(w0, d1), -__fmul_rn(w1, d0));
                } else {
                    c[3] = w0; c[4] = w1; c[5] = w2;
                }
            }
#pragma unroll
            for (int k = 0; k < 6; ++k) out[6 * e + k] = c[k];
        }
        __syncwarp();
    }
}

extern "C" gbmp_status gbmp_space_jacobian(gbmp_robot r, const float *d_q, int64_t n, float *d_jac, void *stream) {
    GBMP_CHECK_ARG(r, "robot is NULL");
    GBMP_CHECK_ARG(n >= 0, "n < 0");
    if (n == 0) return GBMP_OK;
    GBMP_CHECK_ARG(d_q && d_jac, "q/jacobian is NULL");
    const size_t smem = smem_tables_bytes(r->dev, 0) + smem_warp_bytes(r->dev) * kWarpsPerBlock;
    gbmp_status so = ensure_smem_optin((const void *)k_space_jacobian);
    if (so) return so;
    int per_sm = 0;
    GBMP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_space_jacobian, kWarpsPerBlock * kWarp, smem));
    if (per_sm < 1) {
        set_error("Jacobian kernel does not fit on an SM (%zu bytes of shared memory)", smem);
        return GBMP_ERR_CAPACITY;
    }
    long long grid = (long long)per_sm * r->num_sms;
    const long long need = (n + kWarpsPerBlock - 1) / kWarpsPerBlock;
    if (need < grid) grid = need;
    ProfScope ps(GBMP_PROF_OTHER, (cudaStream_t)stream);
    k_space_jacobian<<<(unsigned)grid, kWarpsPerBlock * kWarp, smem, (cudaStream_t)stream>>>(r->dev, d_q, n, d_jac);
    GBMP_CUDA(cudaGetLastError());
    return GBMP_OK;
}

extern "C" gbmp_status gbmp_project_states(gbmp_robot r, const gbmp_projection *proj, float *d_q, int64_t n,
                                           float *d_task_cost, float *d_bound_cost, void *stream) {
    GBMP_CHECK_ARG(r && proj, "robot/projection is NULL");
    GBMP_CHECK_ARG(n >= 0, "n < 0");
    GBMP_CHECK_ARG(proj->task_link >= -1 && proj->task_link < r->L, "task_link %d outside [-1, %d)", proj->task_link,
                   r->L);
    GBMP_CHECK_ARG(proj->iterations >= 0 && proj->iterations <= 1000, "iterations %d outside [0, 1000]",
                   proj->iterations);
    GBMP_CHECK_ARG(r->L <= 2 * kWarp, "projection supports at most %d links", 2 * kWarp);
    if (n == 0) return GBMP_OK;
    GBMP_CHECK_ARG(d_q, "q is NULL");
    ProjParams p;
    p.task_link = proj->task_link;
    p.use_boundary = proj->use_boundary != 0;
    p.iterations = proj->iterations;
    for (int k = 0; k < 16; ++k) p.offset[k] = proj->offset[k];
    for (int k = 0; k < 6; ++k) {
        p.reference[k] = proj->reference[k];
        p.tolerance[k] = proj->tolerance[k];
    }
    const DevRobot &D = r->dev_chunk;
    const void *fn = r->L <= kWarp ? (const void *)k_project<1> : (const void *)k_project<2>;
    gbmp_status so = ensure_smem_optin(fn);
    if (so) return so;
    int warps = 0, per_sm = 0;
    long long grid = 0;
    spread_warps(n, r->num_sms, &warps, &grid);
    const size_t smem = smem_tables_bytes(D, 0) + proj_warp_bytes(D) * warps;
    GBMP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, warps * kWarp, smem));
    if (per_sm < 1) {
        set_error("projection kernel does not fit on an SM (%zu bytes of shared memory)", smem);
        return GBMP_ERR_CAPACITY;
    }
    grid = std::min<long long>(grid, (long long)per_sm * r->num_sms);
    long long ns = n;
    DevRobot R = D;
    void *args[] = {&R, &p, &d_q, &ns, &d_task_cost, &d_bound_cost};
    ProfScope ps(GBMP_PROF_OTHER, (cudaStream_t)stream);
    GBMP_CUDA(cudaLaunchKernel(fn, dim3((unsigned)grid), dim3(warps * kWarp), args, smem, (cudaStream_t)stream));
    return GBMP_OK;
}

extern "C" gbmp_status gbmp_constrained_motions(gbmp_robot r, gbmp_env env, const gbmp_projection *proj,
                                                const float *d_from, const float *d_to, int64_t n, float resolution,
                                                int32_t max_iterations, uint8_t *d_ok, float *d_cost,
                                                int32_t *d_num_states, float *d_states, int32_t states_cap,
                                                void *stream) {
    GBMP_CHECK_ARG(r && env && proj, "robot/env/projection is NULL");
    GBMP_CHECK_ARG(n >= 0, "n < 0");
    GBMP_CHECK_ARG(proj->task_link >= -1 && proj->task_link < r->L, "task_link %d outside [-1, %d)", proj->task_link,
                   r->L);
    GBMP_CHECK_ARG(max_iterations >= 1 && max_iterations <= 1000000, "max_iterations %d outside [1, 1e6]",
                   max_iterations);
    GBMP_CHECK_ARG(!d_states || states_cap >= 1, "states_cap < 1 with a states buffer");
    GBMP_CHECK_ARG(r->L <= 2 * kWarp, "constrained motions support at most %d links", 2 * kWarp);
    if (n == 0) return GBMP_OK;
    GBMP_CHECK_ARG(d_from && d_to, "from/to is NULL");
    const float res = resolution > 0.f ? resolution : r->resolution;
    GBMP_CHECK_ARG(std::isfinite(res), "resolution is not finite");
    ProjParams p;
    p.task_link = proj->task_link;
    p.use_boundary = proj->use_boundary != 0;
    p.iterations = 2;
    for (int k = 0; k < 16; ++k) p.offset[k] = proj->offset[k];
    for (int k = 0; k < 6; ++k) {
        p.reference[k] = proj->reference[k];
        p.tolerance[k] = proj->tolerance[k];
    }
    const DevEnv E = env->dev();
    DevRobot D = r->dev_chunk;
    D.work = nullptr;
    const int nwords = env_words(E.ns, E.nb, E.nc);
    const void *fn = env->tight ? r->L <= kWarp ? (const void *)k_constrained_motion<1, true>
                                                : (const void *)k_constrained_motion<2, true>
                     : r->L <= kWarp ? (const void *)k_constrained_motion<1, false>
                                     : (const void *)k_constrained_motion<2, false>;
    gbmp_status st = ensure_smem_optin(fn);
    if (st) return st;
    int warps = 0, per_sm = 0;
    long long grid = 0;
    spread_warps(n, r->num_sms, &warps, &grid);
    // what a block of eight warps took before is what a scene may take
    const size_t most = smem_tables_bytes(r->dev, nwords) + (smem_warp_bytes(r->dev) + cm_limit_bytes(r->dev)) * kWarpsPerBlock;
    size_t smem = smem_tables_bytes(D, nwords) + cm_warp_bytes(D) * warps;
    while (smem > kSmemLimit && warps > 1) {   // a large scene: fewer warps a block
        warps /= 2;
        smem = smem_tables_bytes(D, nwords) + cm_warp_bytes(D) * warps;
    }
    grid = (n + warps - 1) / warps;
    if (most <= kSmemLimit)
        GBMP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, warps * kWarp, smem));
    if (per_sm < 1) {
        set_error("constrained-motion kernel does not fit on an SM (%zu bytes of shared memory)", most);
        return GBMP_ERR_CAPACITY;
    }
    grid = std::min<long long>(grid, (long long)per_sm * r->num_sms);
    cudaStream_t s = (cudaStream_t)stream;
    ProfScope ps(GBMP_PROF_OTHER, s);
    DevEnv env_view = E;
    long long ns = n;
    float step = res;
    void *args[] = {&D, &env_view, &p, &d_from, &d_to, &ns, &step, &max_iterations, &d_ok, &d_cost, &d_num_states,
                    &d_states, &states_cap};
    GBMP_CUDA(cudaLaunchKernel(fn, dim3((unsigned)grid), dim3(warps * kWarp), args, smem, s));
    return GBMP_OK;
}
