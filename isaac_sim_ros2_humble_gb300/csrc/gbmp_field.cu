// gbmp_field.cu -- the distance field of a scene (scene_far, gbmp_device.cuh), made once
// when the scene is created.
#include <algorithm>
#include <cmath>

#include "gbmp_internal.h"

namespace gbmp {

// The three least distances from every cell's centre to an obstacle (spheres |c - o| - r,
// cuboids the distance to the box, cylinders the signed distance) and the obstacles of the
// first two, every distance short by `slack` of what it was made from (kFieldSlack, and what
// rotations that are not quite orthonormal change distances by): eight lanes a cell, each an eighth of the obstacles, then merged (one lane a
// cell leaves 32,768 threads with a chain over every obstacle: a scene of 336 took 75 us
// longer to create, 45 us with eight).
constexpr int kFieldLanes = 8;

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
};

__global__ void __launch_bounds__(256) k_scene_field(DevEnv E, float slack, float4 *__restrict__ field) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, cell = tid / kFieldLanes, o0 = tid % kFieldLanes;
    const bool in = cell < E.nx * E.ny * E.nz;
    const int ix = cell % E.nx, iy = cell / E.nx % E.ny, iz = cell / (E.nx * E.ny);
    const float x = cell_centre(E.ox, E.h, ix), y = cell_centre(E.oy, E.h, iy), z = cell_centre(E.oz, E.h, iz);
    const float c1 = fabsf(x) + fabsf(y) + fabsf(z);
    auto least = [&](float d, float size) { return d - slack * (fabsf(d) + c1 + size); };
    Nearest3 n;
    const float4 *w = E.words;
#pragma unroll 4
    for (int o = o0; o < E.ns; o += kFieldLanes) {
        const float4 b = __ldg(w + o);
        n.add(least(sqrtf(sq3(x - b.x, y - b.y, z - b.z)) - b.w, fabsf(b.w)), o);
    }
    w += E.ns;
#pragma unroll 2
    for (int o = o0; o < E.nb; o += kFieldLanes) {
        const float4 mn = __ldg(w + 5 * o + 3), mx = __ldg(w + 5 * o + 4);
        const float4 r0 = __ldg(w + 5 * o), r1 = __ldg(w + 5 * o + 1), r2 = __ldg(w + 5 * o + 2);
        const float3 l = xform_rows(r0, r1, r2, x, y, z);
        const float dx = l.x - fminf(fmaxf(l.x, mn.x), mx.x), dy = l.y - fminf(fmaxf(l.y, mn.y), mx.y),
                    dz = l.z - fminf(fmaxf(l.z, mn.z), mx.z);
        n.add(least(sqrtf(sq3(dx, dy, dz)), fabsf(r0.w) + fabsf(r1.w) + fabsf(r2.w)), E.ns + o);
    }
    w += 5 * E.nb;
#pragma unroll 2
    for (int o = o0; o < E.nc; o += kFieldLanes) {
        const float4 pr = __ldg(w + 4 * o + 3);
        const float4 r0 = __ldg(w + 4 * o), r1 = __ldg(w + 4 * o + 1), r2 = __ldg(w + 4 * o + 2);
        const float3 l = xform_rows(r0, r1, r2, x, y, z);
        const float dx = sqrtf(l.x * l.x + l.y * l.y) - pr.x, dz = fabsf(l.z) - pr.y;
        const float ox = fmaxf(dx, 0.f), oz = fmaxf(dz, 0.f);
        n.add(least(sqrtf(ox * ox + oz * oz) + fminf(fmaxf(dx, dz), 0.f), fabsf(r0.w) + fabsf(r1.w) + fabsf(r2.w)),
              E.ns + E.nb + o);
    }
#pragma unroll
    for (int off = 1; off < kFieldLanes; off <<= 1) {
        const float d1 = __shfl_xor_sync(kFull, n.d1, off), d2 = __shfl_xor_sync(kFull, n.d2, off),
                    d3 = __shfl_xor_sync(kFull, n.d3, off);
        const int o1 = __shfl_xor_sync(kFull, n.o1, off), o2 = __shfl_xor_sync(kFull, n.o2, off);
        n.add(d1, o1);
        n.add(d2, o2);
        n.add(d3, 0xffff);   // below d1 and d2, so it ends as a third distance at most
    }
    // A cell that no distance could be computed for names obstacle 0 and says nothing: a state
    // that is no number is tested against what its cell names.
    if (n.o1 == 0xffff) {
        n.d1 = n.d2 = n.d3 = -3.0e38f;
        n.o1 = 0;
    }
    if (in && o0 == 0) field[cell] = make_float4(n.d1, n.d2, n.d3, __int_as_float(n.o1 | n.o2 << 16));
}

// The field's region and cell size from the obstacles' bounding spheres (centre, radius:
// 4 doubles each): the box of the obstacles that span it, kFieldBorder wider on every side, in
// cubic cells, kFieldCells along its longest side.  A floor must not stretch the cells, nor an
// obstacle far from the rest: those that span it are at most kFieldLargest metres large (all,
// if there are none), and reach no farther from their centres' median than kFieldReach times
// what kFieldCore of them do (up to 1.6 in the scenes of the benchmarks, whose obstacles are
// in one place).  One sphere 20 m away among 336 obstacles in a 1.2 m cube made cells of 0.67 m
// instead of 0.07, and 70,000 states of the 8-DOF arm took 1,356 us; 57 us now.  Queries
// outside the region go by its border cells, whose distances are to all obstacles.  The box of
// all obstacles bounds what lies outside.  False when a number is not finite: the scene then
// has no field, and every test runs.
constexpr double kFieldCore = 0.875, kFieldReach = 2.0;
bool scene_field_plan(const std::vector<double> &b, DevEnv &E, bool *tight) {
    const size_t n = b.size() / 4;
    if (n == 0) return false;
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    std::vector<size_t> span;
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
    std::vector<double> v(span.size()), reach(span.size(), 0.0);
    for (int a = 0; a < 3; ++a) {
        for (size_t k = 0; k < span.size(); ++k) v[k] = b[4 * span[k] + a];
        std::nth_element(v.begin(), v.begin() + v.size() / 2, v.end());
        const double mid = v[v.size() / 2];
        for (size_t k = 0; k < span.size(); ++k)
            reach[k] = std::max(reach[k], std::fabs(b[4 * span[k] + a] - mid) + b[4 * span[k] + 3]);
    }
    v = reach;
    const size_t core = (size_t)std::ceil(kFieldCore * (double)v.size()) - 1;
    std::nth_element(v.begin(), v.begin() + core, v.end());
    const double farthest = kFieldReach * std::max(v[core], 0.0);
    double slo[3] = {1e300, 1e300, 1e300}, shi[3] = {-1e300, -1e300, -1e300}, side = 0.0;
    size_t outside = n - span.size();
    for (double r : reach) outside += r > farthest;
    for (int a = 0; a < 3; ++a) {
        for (size_t k = 0; k < span.size(); ++k)
            if (reach[k] <= farthest) {
                slo[a] = std::min(slo[a], b[4 * span[k] + a] - b[4 * span[k] + 3]);
                shi[a] = std::max(shi[a], b[4 * span[k] + a] + b[4 * span[k] + 3]);
            }
        slo[a] -= kFieldBorder;
        shi[a] += kFieldBorder;
        if (!(std::max(-slo[a], shi[a]) <= 2e6)) return false;
        side = std::max(side, shi[a] - slo[a]);
    }
    if (!(side > 0.0)) return false;   // radii below 0
    const double h = side / kFieldCells;
    int cells[3];
    for (int a = 0; a < 3; ++a) cells[a] = std::max(1, std::min(kFieldCells, (int)std::ceil((shi[a] - slo[a]) / h - 1e-9)));
    E.nx = cells[0]; E.ny = cells[1]; E.nz = cells[2];
    E.ox = (float)slo[0]; E.oy = (float)slo[1]; E.oz = (float)slo[2];
    E.h = (float)h;
    E.inv_h = (float)(1.0 / h);
    *tight = h <= kFieldFine && outside == 0;
    for (int a = 0; a < 3; ++a) {   // outwards by more than single precision loses
        const double pad = 1e-5 + 1e-6 * std::max(std::fabs(lo[a]), std::fabs(hi[a]));
        (a == 0 ? E.lox : a == 1 ? E.loy : E.loz) = (float)(lo[a] - pad);
        (a == 0 ? E.hix : a == 1 ? E.hiy : E.hiz) = (float)(hi[a] + pad);
    }
    return true;
}

cudaError_t scene_field_build(const DevEnv &E, float slack, float4 *field, cudaStream_t s) {
    const int cells = E.nx * E.ny * E.nz;
    // the launch's own result: cudaGetLastError would also report what an earlier call left
    DevEnv e = E;
    void *args[] = {&e, &slack, &field};
    return cudaLaunchKernel((const void *)k_scene_field, dim3((cells * kFieldLanes + 255) / 256), dim3(256), args, 0, s);
}

}  // namespace gbmp
