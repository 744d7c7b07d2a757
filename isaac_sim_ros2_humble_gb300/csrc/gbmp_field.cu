// gbmp_field.cu -- the distance field of a scene (scene_far, gbmp_device.cuh), made once
// when the scene is created.
#include <cmath>

#include "gbmp_internal.h"

namespace gbmp {

// Least distance of every cell's centre to an obstacle (spheres |c - o| - r, cuboids the
// distance to the box, cylinders the signed distance): eight lanes a cell, each an eighth
// of the obstacles (one lane a cell leaves 32,768 threads with a chain over every obstacle:
// a scene of 336 took 75 us longer to create, 42 us with eight).
constexpr int kFieldLanes = 8;

__global__ void __launch_bounds__(256) k_scene_field(DevEnv E, float *__restrict__ field) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, cell = tid / kFieldLanes, o0 = tid % kFieldLanes;
    const bool in = cell < E.nx * E.ny * E.nz;
    const int ix = cell % E.nx, iy = cell / E.nx % E.ny, iz = cell / (E.nx * E.ny);
    const float x = E.ox + ((float)ix + 0.5f) * E.h, y = E.oy + ((float)iy + 0.5f) * E.h,
                z = E.oz + ((float)iz + 0.5f) * E.h;
    float best = 3.0e38f;
    const float4 *w = E.words;
#pragma unroll 4
    for (int o = o0; o < E.ns; o += kFieldLanes) {
        const float4 b = __ldg(w + o);
        best = fminf(best, sqrtf(sq3(x - b.x, y - b.y, z - b.z)) - b.w);
    }
    w += E.ns;
#pragma unroll 2
    for (int o = o0; o < E.nb; o += kFieldLanes) {
        const float4 mn = __ldg(w + 5 * o + 3), mx = __ldg(w + 5 * o + 4);
        const float3 l = xform_rows(__ldg(w + 5 * o), __ldg(w + 5 * o + 1), __ldg(w + 5 * o + 2), x, y, z);
        const float dx = l.x - fminf(fmaxf(l.x, mn.x), mx.x), dy = l.y - fminf(fmaxf(l.y, mn.y), mx.y),
                    dz = l.z - fminf(fmaxf(l.z, mn.z), mx.z);
        best = fminf(best, sqrtf(sq3(dx, dy, dz)));
    }
    w += 5 * E.nb;
#pragma unroll 2
    for (int o = o0; o < E.nc; o += kFieldLanes) {
        const float4 pr = __ldg(w + 4 * o + 3);
        const float3 l = xform_rows(__ldg(w + 4 * o), __ldg(w + 4 * o + 1), __ldg(w + 4 * o + 2), x, y, z);
        const float dx = sqrtf(l.x * l.x + l.y * l.y) - pr.x, dz = fabsf(l.z) - pr.y;
        const float ox = fmaxf(dx, 0.f), oz = fmaxf(dz, 0.f);
        best = fminf(best, sqrtf(ox * ox + oz * oz) + fminf(fmaxf(dx, dz), 0.f));
    }
#pragma unroll
    for (int off = 1; off < kFieldLanes; off <<= 1) best = fminf(best, __shfl_xor_sync(kFull, best, off));
    if (in && o0 == 0) field[cell] = best;
}

// The field's region and cell size from the obstacles' bounding spheres (centre, radius:
// 4 doubles each): the box of the obstacles of at most kFieldLargest metres (of all, if
// there are no others: a floor must not stretch the cells), kFieldBorder wider on every
// side, in cubic cells, kFieldCells along its longest side.  The box of all obstacles
// bounds what lies outside.  False when a number is not finite: the scene then has no
// field, and every test runs.
bool scene_field_plan(const std::vector<double> &b, DevEnv &E) {
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300}, slo[3], shi[3];
    for (int a = 0; a < 3; ++a) { slo[a] = 1e300; shi[a] = -1e300; }
    for (size_t i = 0; i < b.size(); i += 4) {
        const double r = b[i + 3];
        for (int a = 0; a < 3; ++a) {
            if (!std::isfinite(b[i + a]) || !std::isfinite(r) || std::fabs(b[i + a]) > 1e6 || r > 1e6) return false;
            lo[a] = std::min(lo[a], b[i + a] - r);
            hi[a] = std::max(hi[a], b[i + a] + r);
            if (r <= kFieldLargest) {
                slo[a] = std::min(slo[a], b[i + a] - r);
                shi[a] = std::max(shi[a], b[i + a] + r);
            }
        }
    }
    if (b.empty()) return false;
    double side = 0.0;
    for (int a = 0; a < 3; ++a) {
        if (slo[a] > shi[a]) { slo[a] = lo[a]; shi[a] = hi[a]; }
        slo[a] -= kFieldBorder;
        shi[a] += kFieldBorder;
        side = std::max(side, shi[a] - slo[a]);
    }
    const double h = side / kFieldCells;
    int n[3];
    for (int a = 0; a < 3; ++a) n[a] = std::max(1, std::min(kFieldCells, (int)std::ceil((shi[a] - slo[a]) / h - 1e-9)));
    E.nx = n[0]; E.ny = n[1]; E.nz = n[2];
    E.ox = (float)slo[0]; E.oy = (float)slo[1]; E.oz = (float)slo[2];
    E.h = (float)h;
    E.inv_h = (float)(1.0 / h);
    for (int a = 0; a < 3; ++a) {   // outwards by more than single precision loses
        const double pad = 1e-5 + 1e-6 * std::max(std::fabs(lo[a]), std::fabs(hi[a]));
        (a == 0 ? E.lox : a == 1 ? E.loy : E.loz) = (float)(lo[a] - pad);
        (a == 0 ? E.hix : a == 1 ? E.hiy : E.hiz) = (float)(hi[a] + pad);
    }
    return true;
}

cudaError_t scene_field_build(const DevEnv &E, float *field, cudaStream_t s) {
    const int cells = E.nx * E.ny * E.nz;
    k_scene_field<<<(cells * kFieldLanes + 255) / 256, 256, 0, s>>>(E, field);
    return cudaGetLastError();
}

}  // namespace gbmp
