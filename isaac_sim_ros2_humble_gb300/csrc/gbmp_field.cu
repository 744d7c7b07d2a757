// gbmp_field.cu -- the distance field of a scene (scene_far, gbmp_device.cuh), made once
// when the scene is created.
#include <algorithm>
#include <cmath>

#include "gbmp_internal.h"

namespace gbmp {

// The three least distances from every cell's centre to an obstacle (spheres |c - o| - r,
// cuboids the distance to the box, cylinders the signed distance) and the obstacles of the
// first two, every distance short by `slack` of what it was made from (kFieldSlack, and what
// rotations that are not quite orthonormal change distances by).
//
// One block for 4 x 4 x 4 cells.  First every obstacle's distance from the block's middle: with t
// the third least of them and w the way to its farthest cell centre, three obstacles lie within t +
// w of any of its cells, and one beyond t + 2 w of the middle is not among its three nearest.
// The others, listed, are what each cell tests, four lanes a cell.  What bounds it: the arithmetic
// of the distances, and for some tens of obstacles the launch.  With every obstacle tested for
// every cell a scene of 336 took 80 us to create and one of 2,260 obstacles 425 us; 68 and 295
// us with this (27 and 200 without a field).
constexpr int kFieldSide = 4, kFieldLanes = 4, kFieldThreads = kFieldSide * kFieldSide * kFieldSide * kFieldLanes;

struct Nearest3 {
    float d1 = 3.0e38f, d2 = 3.0e38f, d3 = 3.0e38f;
    int o1 = 0xffff, o2 = 0xffff;
    __device__ __forceinline__ void add(float d, int o) {
        if (!(d < d3)) return;   // (an obstacle beyond what a float squares is none)
        if (d < d2) {
            d3 = d2;
            const bool first = d < d1;
            d2 = first ? d1 : d;
            o2 = first ? o1 : o;
            if (first) { d1 = d; o1 = o; }
        } else {
            d3 = d;
        }
    }
    __device__ __forceinline__ void merge(int off) {   // with the lane `off` away
        const float e1 = __shfl_xor_sync(kFull, d1, off), e2 = __shfl_xor_sync(kFull, d2, off),
                    e3 = __shfl_xor_sync(kFull, d3, off);
        const int p1 = __shfl_xor_sync(kFull, o1, off), p2 = __shfl_xor_sync(kFull, o2, off);
        add(e1, p1);
        add(e2, p2);
        add(e3, 0xffff);   // below d1 and d2, so it ends as a third distance at most
    }
};

// Distance of (x, y, z) from obstacle o (the scene's numbering); `from`: the lengths it was
// made from, c1 = |x| + |y| + |z| among them.
__device__ __forceinline__ float field_distance(const DevEnv &E, int o, float x, float y, float z, float c1,
                                                float &from) {
    const float4 *w = E.words;
    float d;
    if (o < E.ns) {
        const float4 b = __ldg(w + o);
        d = sqrtf(sq3(x - b.x, y - b.y, z - b.z)) - b.w;
        from = fabsf(d) + c1 + fabsf(b.w);
        return d;
    }
    const bool box = o < E.ns + E.nb;
    w += box ? E.ns + 5 * (o - E.ns) : E.ns + 5 * E.nb + 4 * (o - E.ns - E.nb);
    const float4 r0 = __ldg(w), r1 = __ldg(w + 1), r2 = __ldg(w + 2), p = __ldg(w + 3);
    const float3 l = xform_rows(r0, r1, r2, x, y, z);
    if (box) {
        const float4 mx = __ldg(w + 4);
        const float dx = l.x - fminf(fmaxf(l.x, p.x), mx.x), dy = l.y - fminf(fmaxf(l.y, p.y), mx.y),
                    dz = l.z - fminf(fmaxf(l.z, p.z), mx.z);
        d = sqrtf(sq3(dx, dy, dz));
    } else {
        const float dx = sqrtf(l.x * l.x + l.y * l.y) - p.x, dz = fabsf(l.z) - p.y;
        const float ox = fmaxf(dx, 0.f), oz = fmaxf(dz, 0.f);
        d = sqrtf(ox * ox + oz * oz) + fminf(fmaxf(dx, dz), 0.f);
    }
    from = fabsf(d) + c1 + (fabsf(r0.w) + fabsf(r1.w) + fabsf(r2.w));
    return d;
}

__global__ void __launch_bounds__(kFieldThreads)
    k_scene_field(DevEnv E, float slack, int nbx, int nby, float4 *__restrict__ field) {
    __shared__ unsigned short s_list[kMaxEnvWords / 2];   // an obstacle takes more than two words
    __shared__ float s_third[kFieldThreads / kWarp][3];
    __shared__ int s_count[kFieldThreads / kWarp];
    const int tid = threadIdx.x, warp = tid / kWarp, lane = tid & 31, n = E.ns + E.nb + E.nc;
    const int bx = blockIdx.x % nbx, by = blockIdx.x / nbx % nby, bz = blockIdx.x / (nbx * nby);
    const int ix0 = kFieldSide * bx, iy0 = kFieldSide * by, iz0 = kFieldSide * bz;
    const int ix1 = min(ix0 + kFieldSide, E.nx) - 1, iy1 = min(iy0 + kFieldSide, E.ny) - 1,
              iz1 = min(iz0 + kFieldSide, E.nz) - 1;

    // --- the block's middle, and the obstacles that can be among the three nearest of a cell ---
    int count = 0;
    {
        const float x0 = cell_centre(E.ox, E.h, ix0), x1 = cell_centre(E.ox, E.h, ix1), y0 = cell_centre(E.oy, E.h, iy0),
                    y1 = cell_centre(E.oy, E.h, iy1), z0 = cell_centre(E.oz, E.h, iz0), z1 = cell_centre(E.oz, E.h, iz1);
        const float x = 0.5f * (x0 + x1), y = 0.5f * (y0 + y1), z = 0.5f * (z0 + z1);
        const float c1 = fabsf(x) + fabsf(y) + fabsf(z);
        // (and what rounding and rotations that are not quite orthonormal add)
        const float way = sqrtf(sq3(x1 - x, y1 - y, z1 - z)) * (1.f + 2.f * slack) + slack * c1;
        Nearest3 t;
        float from;
        for (int o = tid; o < n; o += kFieldThreads) {
            const float d = field_distance(E, o, x, y, z, c1, from);
            t.add(d + slack * from, 0);
        }
#pragma unroll
        for (int off = 1; off < kWarp; off <<= 1) t.merge(off);
        if (lane == 0) { s_third[warp][0] = t.d1; s_third[warp][1] = t.d2; s_third[warp][2] = t.d3; }
        __syncthreads();
        t = Nearest3();
#pragma unroll 1
        for (int v = 0; v < kFieldThreads / kWarp; ++v)
            for (int i = 0; i < 3; ++i) t.add(s_third[v][i], 0);
        const float limit = t.d3 + 2.f * way;
        for (int o0 = 0; o0 < n; o0 += kFieldThreads) {
            const int o = o0 + tid;
            bool on = false;
            if (o < n) {
                const float d = field_distance(E, o, x, y, z, c1, from);
                on = !(d - slack * from > limit);
            }
            const unsigned bal = __ballot_sync(kFull, on);
            if (lane == 0) s_count[warp] = __popc(bal);
            __syncthreads();
            int at = count;
            for (int v = 0; v < kFieldThreads / kWarp; ++v) {
                if (v < warp) at += s_count[v];
                count += s_count[v];
            }
            if (on) s_list[at + __popc(bal & ((1u << lane) - 1u))] = (unsigned short)o;
            __syncthreads();
        }
    }

    // --- the cells ---
    const int cell = tid / kFieldLanes, sub = tid % kFieldLanes;
    const int ix = ix0 + cell % kFieldSide, iy = iy0 + cell / kFieldSide % kFieldSide,
              iz = iz0 + cell / (kFieldSide * kFieldSide);
    const float x = cell_centre(E.ox, E.h, ix), y = cell_centre(E.oy, E.h, iy), z = cell_centre(E.oz, E.h, iz);
    const float c1 = fabsf(x) + fabsf(y) + fabsf(z);
    Nearest3 t;
#pragma unroll 2
    for (int i = sub; i < count; i += kFieldLanes) {
        float from;
        const int o = s_list[i];
        const float d = field_distance(E, o, x, y, z, c1, from);
        t.add(d - slack * from, o);
    }
#pragma unroll
    for (int off = 1; off < kFieldLanes; off <<= 1) t.merge(off);
    // A cell that no distance could be computed for names obstacle 0 and says nothing: a state
    // that is no number is tested against what its cell names.
    if (t.o1 == 0xffff) {
        t.d1 = t.d2 = t.d3 = -3.0e38f;
        t.o1 = 0;
    }
    if (sub == 0 && ix <= ix1 && iy <= iy1 && iz <= iz1)
        field[(iz * E.ny + iy) * E.nx + ix] = make_float4(t.d1, t.d2, t.d3, __int_as_float(t.o1 | t.o2 << 16));
}

// The field's region and cell size from the obstacles' bounding spheres (centre, radius:
// 4 doubles each): the box of the obstacles that span it, kFieldBorder wider on every side, in
// cubic cells, kFieldCells along its longest side.  A floor must not stretch the cells, nor an
// obstacle far from the rest: those that span it are at most kFieldLargest metres large (all,
// if there are none), and reach no farther from their centres' median than kFieldReach times
// what kFieldCore of them do (up to 1.6 in the scenes of the benchmarks, whose obstacles are
// in one place).  One sphere 20 m away among 336 obstacles in a 1.2 m cube made cells of 0.67 m
// instead of 0.07, and 70,000 states of the 8-DOF arm took 1,356 us; 57 us now.  But more than
// kFieldFew of the obstacles may be those around the robot: they stay in the grid unless its
// cells then exceed kFieldCoarse metres (34 obstacles by the robot and 316 in a pile 5 m away,
// cells of 0.2 m: 59 us, 122 with the grid over the pile alone; 30 m away 124 us with it).
// Queries outside the region go by its border cells, whose distances are to all obstacles.  The
// box of all obstacles bounds what lies outside.  False when a number is not finite: the scene
// then has no field, and every test runs.
constexpr double kFieldCore = 0.875, kFieldReach = 2.0, kFieldFew = 1.0 / 32, kFieldCoarse = 0.4;
constexpr size_t kFieldSample = 256;
bool scene_field_plan(const std::vector<double> &b, DevEnv &E, bool *tight) {
    const size_t n = b.size() / 4;
    if (n == 0) return false;
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    std::vector<size_t> span;
    span.reserve(n);
    for (size_t i = 0; i < n; ++i) {
        const double r = b[4 * i + 3];
        for (int a = 0; a < 3; ++a) {
            if (!std::isfinite(b[4 * i + a]) || !std::isfinite(r)) return false;
            lo[a] = std::min(lo[a], b[4 * i + a] - r);
            hi[a] = std::max(hi[a], b[4 * i + a] + r);
        }
        if (r <= kFieldLargest) span.push_back(i);
    }
    if (span.empty())
        for (size_t i = 0; i < n; ++i) span.push_back(i);
    // medians and the core's reach from at most kFieldSample of them, spread over the list
    const size_t all = span.size(), some = std::min(all, kFieldSample);
    auto sample = [&](size_t k) { return all == some ? k : k * 40503 % all; };
    std::vector<double> v(some), reach(all, 0.0);
    for (int a = 0; a < 3; ++a) {
        for (size_t k = 0; k < some; ++k) v[k] = b[4 * span[sample(k)] + a];
        std::nth_element(v.begin(), v.begin() + some / 2, v.end());
        const double mid = v[some / 2];
        for (size_t k = 0; k < all; ++k)
            reach[k] = std::max(reach[k], std::fabs(b[4 * span[k] + a] - mid) + b[4 * span[k] + 3]);
    }
    for (size_t k = 0; k < some; ++k) v[k] = reach[sample(k)];
    const size_t core = (size_t)std::ceil(kFieldCore * (double)some) - 1;
    std::nth_element(v.begin(), v.begin() + core, v.end());
    double farthest = kFieldReach * std::max(v[core], 0.0);
    double slo[3], shi[3], side;
    auto box = [&] {   // of the spanning obstacles within `farthest`
        side = 0.0;
        for (int a = 0; a < 3; ++a) {
            slo[a] = 1e300;
            shi[a] = -1e300;
            for (size_t k = 0; k < all; ++k)
                if (reach[k] <= farthest) {
                    slo[a] = std::min(slo[a], b[4 * span[k] + a] - b[4 * span[k] + 3]);
                    shi[a] = std::max(shi[a], b[4 * span[k] + a] + b[4 * span[k] + 3]);
                }
            slo[a] -= kFieldBorder;
            shi[a] += kFieldBorder;
            side = std::max(side, shi[a] - slo[a]);
        }
    };
    size_t beyond = 0;
    for (double r : reach) beyond += r > farthest;
    if ((double)beyond > kFieldFew * (double)all) {   // many: only where they would make the cells coarse
        const double within = farthest;
        farthest = 1e300;
        box();
        if (side > kFieldCoarse * kFieldCells) farthest = within;
        else beyond = 0;
    }
    box();
    for (int a = 0; a < 3; ++a)
        if (!(std::max(-slo[a], shi[a]) <= 2e6)) return false;
    if (!(side > 0.0)) return false;   // radii below 0
    const double h = side / kFieldCells;
    int cells[3];
    for (int a = 0; a < 3; ++a) cells[a] = std::max(1, std::min(kFieldCells, (int)std::ceil((shi[a] - slo[a]) / h - 1e-9)));
    E.nx = cells[0]; E.ny = cells[1]; E.nz = cells[2];
    E.ox = (float)slo[0]; E.oy = (float)slo[1]; E.oz = (float)slo[2];
    E.h = (float)h;
    E.inv_h = (float)(1.0 / h);
    *tight = h <= kFieldFine && beyond == 0 && all == n;
    for (int a = 0; a < 3; ++a) {   // outwards by more than single precision loses
        const double pad = 1e-5 + 1e-6 * std::max(std::fabs(lo[a]), std::fabs(hi[a]));
        (a == 0 ? E.lox : a == 1 ? E.loy : E.loz) = (float)(lo[a] - pad);
        (a == 0 ? E.hix : a == 1 ? E.hiy : E.hiz) = (float)(hi[a] + pad);
    }
    return true;
}

cudaError_t scene_field_build(const DevEnv &E, float slack, float4 *field, cudaStream_t s) {
    auto blocks = [](int n) { return (n + kFieldSide - 1) / kFieldSide; };
    // the launch's own result: cudaGetLastError would also report what an earlier call left
    DevEnv e = E;
    int nbx = blocks(E.nx), nby = blocks(E.ny);
    void *args[] = {&e, &slack, &nbx, &nby, &field};
    return cudaLaunchKernel((const void *)k_scene_field, dim3(nbx * nby * blocks(E.nz)), dim3(kFieldThreads), args, 0,
                            s);
}

}  // namespace gbmp
