// gbmp_states_device.cuh -- collision verdicts of several unrelated states by one warp
// (state checks, gbmp_core.cu, gbmp_batchcheck.cu).
//
// The states of one warp (up to kStatesMax) are tested side by side in the lanes, like the
// chunks of gbmp_chunk_device.cuh, whose FK and sphere routines serve here too:
//   1. (state, group) items: the group's bounding sphere, kept for the self pairs, and
//      whether the scene's distance field clears it;
//   2. the spheres of the groups it does not clear, four (state, group) items at a time,
//      eight lanes each: the field again, now with the sphere's own radius, and for a
//      sphere it does not clear the exact tests against the two obstacles nearest to its
//      cell; the third distance says whether another could matter;
//   3. what is left open (a sphere with three obstacles close by, touching neither of the
//      two, or cells too coarse to say): in a tight scene, where this is rare, one sphere at a
//      time, the obstacles of the runs it touches one a lane (warp_sphere_hits); else all
//      such groups of a state at a time (warp_groups_hit);
//   4. the self pairs of the states that have not collided: (state, group pair) items,
//      then the overlapping ones four at a time, as in a chunk.
// Every test that decides is the per-pair formula of warp_collide, and what is left out
// lies kBroadMargin away, so the verdicts are warp_collide's.
#pragma once

#include "gbmp_chunk_device.cuh"

namespace gbmp {

constexpr int kStatesMax = 10;   // three pose-row lanes each

struct StatesScratch {
    float *lpK;    // link poses of the states [K][L*12]
    float4 *gb;    // group spheres of the states [K][G]
    int *it;       // (state, group) or (state, pair) items [max(K G, 32 K)]
};

__host__ __device__ inline size_t smem_states_bytes(const DevRobot &R, int K) {
    return align16(sizeof(float) * 12 * R.L * K) + align16(sizeof(float4) * R.G * K) +
           align16(sizeof(int) * (R.G > kWarp ? R.G : kWarp) * K);
}

__device__ inline StatesScratch carve_states(unsigned char *base, const DevRobot &R, int K, int warp) {
    unsigned char *p = base + smem_states_bytes(R, K) * warp;
    StatesScratch c;
    size_t off = 0;
    c.lpK = reinterpret_cast<float *>(p + off); off += align16(sizeof(float) * 12 * R.L * K);
    c.gb = reinterpret_cast<float4 *>(p + off); off += align16(sizeof(float4) * R.G * K);
    c.it = reinterpret_cast<int *>(p + off);
    return c;
}

// Exact test of the sphere (c, r) against obstacle o (the scene's numbering: spheres,
// cuboids, cylinders), the formulas of warp_collide.
__device__ __forceinline__ bool obstacle_hit(const SmemTables &t, const DevEnv &E, int o, float3 c, float r) {
    if (o < E.ns) {   // expanded form
        const float4 *sx = t.env + E.ns + 5 * E.nb + 4 * E.nc;
        const float4 b = sx[o];
        const float nb = reinterpret_cast<const float *>(sx + E.ns)[o];
        const float A = __fmaf_rn(c.z, c.z, __fmaf_rn(c.y, c.y, __fmaf_rn(c.x, c.x, -r * r)));
        return __fmaf_rn(c.x, b.x, __fmaf_rn(c.y, b.y, __fmaf_rn(c.z, b.z, __fmaf_rn(r, b.w, nb)))) > A;
    }
    if (o < E.ns + E.nb) {
        const float4 *bx = t.env + E.ns + 5 * (o - E.ns);
        const float4 mn = bx[3], mx = bx[4];
        const float3 l = xform_rows(bx[0], bx[1], bx[2], c.x, c.y, c.z);
        const float dx = l.x - fminf(fmaxf(l.x, mn.x), mx.x);
        const float dy = l.y - fminf(fmaxf(l.y, mn.y), mx.y);
        const float dz = l.z - fminf(fmaxf(l.z, mn.z), mx.z);
        return sq3(dx, dy, dz) < r * r;
    }
    const float4 *cy = t.env + E.ns + 5 * E.nb + 4 * (o - E.ns - E.nb);
    const float4 pr = cy[3];
    const float3 l = xform_rows(cy[0], cy[1], cy[2], c.x, c.y, c.z);
    const float dx = sqrtf(__fmaf_rn(l.y, l.y, __fmul_rn(l.x, l.x))) - pr.x;
    const float dz = fabsf(l.z) - pr.y;
    const float ox = dx > 0.f ? dx : 0.f, oz = dz > 0.f ? dz : 0.f;
    const float outside = sqrtf(__fmaf_rn(oz, oz, __fmul_rn(ox, ox)));
    const float inside = fminf(fmaxf(dx, dz), 0.f);
    return r - (outside + inside) > 0.f;
}

// One sphere against the scene by the field: false when it is settled, with h whether it
// touches an obstacle; true when obstacles are left that it might touch.
__device__ __forceinline__ bool sphere_open(const SmemTables &t, const DevEnv &E, float3 c, float r, bool &h) {
    const float rad = r + kBroadMargin;
    h = false;
    if (!E.field) return E.ns + E.nb + E.nc > 0;
    if (scene_outside(E, c.x, c.y, c.z, rad)) return false;
    float way;
    const float4 f = __ldg(scene_cell(E, c.x, c.y, c.z, way));
    if (f.x - way > rad) return false;
    const unsigned ids = __float_as_uint(f.w);   // the first always names an obstacle (k_scene_field)
    h = obstacle_hit(t, E, (int)(ids & 0xffffu), c, r);
    if (!h && !(f.y - way > rad)) {
        if ((ids >> 16) != 0xffffu) h = obstacle_hit(t, E, (int)(ids >> 16), c, r);
        return !h && !(f.z - way > rad);
    }
    return false;
}

// Whether the sphere (c, r), the same on every lane, touches an obstacle: the runs it
// touches, one a lane, then their obstacles, one a lane, type by type.
template <bool CNT>
__device__ __forceinline__ bool warp_sphere_hits(const SmemTables &t, const DevEnv &E, float3 c, float r, int lane,
                                                 unsigned long long &fl) {
    const int nrs = env_clusters(E.ns), nrb = env_clusters(E.nb), nrun = nrs + nrb + env_clusters(E.nc);
    const float4 *runs = t.env + env_cluster_base(E.ns, E.nb, E.nc);
    const float4 *sx = t.env + E.ns + 5 * E.nb + 4 * E.nc;
    const float *snb = reinterpret_cast<const float *>(sx + E.ns);
    const float A = __fmaf_rn(c.z, c.z, __fmaf_rn(c.y, c.y, __fmaf_rn(c.x, c.x, -r * r)));
    for (int c0 = 0; c0 < nrun; c0 += kWarp) {
        bool on = false;
        if (c0 + lane < nrun) {
            const float4 b = runs[c0 + lane];
            const float rr = r + kBroadMargin + b.w;
            on = !(sq3(c.x - b.x, c.y - b.y, c.z - b.z) >= rr * rr);   // NaN: as the tests below have it
        }
        unsigned bal = __ballot_sync(kFull, on);
        if (CNT) fl += (unsigned long long)min(kWarp, nrun - c0) * kFlGroupPair + (unsigned long long)__popc(bal) * kWarp * kFlSphereX;
        bool hit = false;
        for (; bal; bal &= bal - 1u) {
            const int run = c0 + __ffs(bal) - 1;
            if (run >= nrs) break;   // the sphere runs come first
            const int o = run * kWarp + lane;
            if (o < E.ns) {
                const float4 b = sx[o];
                hit |= __fmaf_rn(c.x, b.x, __fmaf_rn(c.y, b.y, __fmaf_rn(c.z, b.z, __fmaf_rn(r, b.w, snb[o])))) > A;
            }
        }
        for (; bal; bal &= bal - 1u) {
            const int run = c0 + __ffs(bal) - 1 - nrs;
            const bool box = run < nrb;
            const int o = (box ? run : run - nrb) * kWarp + lane;
            if (o < (box ? E.nb : E.nc)) hit |= obstacle_hit(t, E, E.ns + (box ? o : E.nb + o), c, r);
        }
        if (__any_sync(kFull, hit)) return true;
    }
    return false;
}

// Whether a sphere of the groups `groups` (bit q: group base + q) of one state touches an
// obstacle (lp: the state's link poses, gb: its group spheres from group base on): the groups,
// one a lane, against one run of 32 obstacles after another; the obstacles of a run that some
// touch, one a lane, against those groups; then each (obstacle, group) that touches, the
// group's spheres against the obstacle, four at a time, eight lanes each.  With it the cost of a
// state is bounded by that of testing every obstacle against every group; one open sphere at a
// time it was not: 70,000 states of a 30-link robot in 336 obstacles and a 20 m floor took 592
// us, 219 with this (536 with a warp a state and no field); in a room of six walls 951 and 267.
template <bool CNT>
__device__ __forceinline__ bool warp_groups_hit(const SmemTables &t, const DevEnv &E, const float *lp, const float4 *gb,
                                             int base, unsigned groups, int lane, unsigned long long &fl) {
    const int nrs = env_clusters(E.ns), nrb = env_clusters(E.nb), nrun = nrs + nrb + env_clusters(E.nc);
    const float4 *runs = t.env + env_cluster_base(E.ns, E.nb, E.nc);
    const int sub = lane >> 3, sl = lane & 7;
    const bool mine = (groups >> lane) & 1u;
    const float4 g = mine ? gb[lane] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float A = __fmaf_rn(g.z, g.z, __fmaf_rn(g.y, g.y, __fmaf_rn(g.x, g.x, -g.w * g.w)));
    if (CNT) fl += (unsigned long long)nrun * __popc(groups) * kFlGroupPair;
#pragma unroll 1
    for (int run = 0; run < nrun; ++run) {
        const float4 b = runs[run];
        const float rr = g.w + b.w;
        // NaN: as the tests below have it
        const bool on = mine && !(sq3(g.x - b.x, g.y - b.y, g.z - b.z) >= rr * rr);
        const unsigned gm = __ballot_sync(kFull, on);
        if (!gm) continue;
        const int type = run < nrs ? 0 : run < nrs + nrb ? 1 : 2;
        const int o0 = (run - (type == 0 ? 0 : type == 1 ? nrs : nrs + nrb)) * kWarp;   // within the type
        const int cnt = min(kWarp, (type == 0 ? E.ns : type == 1 ? E.nb : E.nc) - o0);
        const int o = o0 + min(lane, cnt - 1);
        unsigned mask = 0u;   // groups that this lane's obstacle touches
        if (type == 0) {   // expanded form, see warp_collide
            const float4 *sx = t.env + E.ns + 5 * E.nb + 4 * E.nc;
            const float4 w = sx[o];
            const float nb = reinterpret_cast<const float *>(sx + E.ns)[o];
#pragma unroll 2
            for (unsigned m = gm; m; m &= m - 1u) {
                const int q = __ffs(m) - 1;
                const float4 s = gb[q];
                const float v = __fmaf_rn(s.x, w.x, __fmaf_rn(s.y, w.y, __fmaf_rn(s.z, w.z, __fmaf_rn(s.w, w.w, nb))));
                if (v > __shfl_sync(kFull, A, q)) mask |= 1u << q;
            }
        } else {
            const int os = o + (type == 1 ? E.ns : E.ns + E.nb);   // in the scene's numbering
#pragma unroll 1
            for (unsigned m = gm; m; m &= m - 1u) {
                const int q = __ffs(m) - 1;
                const float4 s = gb[q];
                if (obstacle_hit(t, E, os, make_float3(s.x, s.y, s.z), s.w)) mask |= 1u << q;
            }
        }
        if (lane >= cnt) mask = 0u;
        const int flops = type == 0 ? kFlSphereX : type == 1 ? kFlCuboid : kFlCylinder;
        if (CNT) fl += (unsigned long long)cnt * __popc(gm) * flops;
        const int first = o0 + (type == 0 ? 0 : type == 1 ? E.ns : E.ns + E.nb);
        bool hit = false;
#pragma unroll 1
        for (unsigned left = __ballot_sync(kFull, mask != 0u); left; left = __ballot_sync(kFull, mask != 0u)) {
            const int q = __ffs(mask) - 1;   // one group of each obstacle that has one left
            mask &= mask - 1u;
#pragma unroll 1
            while (left) {
                unsigned c = left;   // the sub'th of them
                for (int i = 0; i < sub; ++i) c &= c - 1u;
                const int x = __ffs(c) - 1, xq = base + __shfl_sync(kFull, q, x & 31);
                if (c) {
                    const int j1 = t.gso[xq + 1];
                    const float *T = lp + 12 * t.glink[xq];
#pragma unroll 1
                    for (int j = t.gso[xq] + sl; j < j1; j += 8) {
                        float4 s;
                        const float3 p = sphere_centre(t, T, j, s);
                        hit |= obstacle_hit(t, E, first + x, p, s.w);
                    }
                }
                if (CNT)
                    fl += (unsigned long long)__reduce_add_sync(kFull, c && sl == 0 ? t.gso[xq + 1] - t.gso[xq] : 0) * (18 + flops);
                for (int i = 0; i < 4; ++i) left &= left - 1u;
            }
            if (__any_sync(kFull, hit)) return true;
        }
    }
    return false;
}

// Verdicts of the ks states whose link poses are in sc.lpK: bit k is set when state k
// collides.  TIGHT: the scene is (gbmp_env_s), few spheres stay open.
template <bool CNT, bool TIGHT>
__device__ inline unsigned warp_verdicts(const SmemTables &t, const DevRobot &R, const DevEnv &E,
                                         const StatesScratch &sc, int ks, int lane) {
    const unsigned all = (1u << ks) - 1u;
    const int sub = lane >> 3, sl = lane & 7, sh = lane & 24;
    const int G = R.G, pose = 12 * R.L;
    unsigned hit = 0u;
    unsigned long long fl = (unsigned long long)(R.base_flops - 24LL * R.S) * ks;

    // --- 1: group spheres of every state; the items that the field does not clear ---
    const int items = ks * G;
    const unsigned rG = (65536u + G - 1u) / (unsigned)max(G, 1);   // p / G = p * rG >> 16 (p < 10 * 64)
    int nit = 0;
    for (int p0 = 0; p0 < items; p0 += kWarp) {
        const int p = p0 + lane;
        bool on = false;
        int item = 0;
        if (p < items) {
            const int k = (int)(p * rG >> 16), g = p - k * G;
            const float4 s = group_sphere(t, sc.lpK + k * pose, g);
            sc.gb[p] = s;
            on = !scene_far(E, s.x, s.y, s.z, s.w);
            item = (g << 5) | k;
        }
        const unsigned bal = __ballot_sync(kFull, on);
        if (on) sc.it[nit + __popc(bal & ((1u << lane) - 1u))] = item;
        nit += __popc(bal);
    }
    if (CNT) fl += (unsigned long long)items * kFlField;
    __syncwarp();

    // --- 2: their spheres; the items left open move to the front of the list ---
    int left = TIGHT || E.field ? 0 : nit;
#pragma unroll 1
    for (int j0 = left; j0 < nit && hit != all; j0 += 4) {
        int v = 0, k = 0, g0 = 0, ng = 0;
        const float *T = sc.lpK;
        if (j0 + sub < nit) {
            v = sc.it[j0 + sub];
            k = v & 31;
            if (!((hit >> k) & 1u)) {
                g0 = t.gso[v >> 5];
                ng = t.gso[(v >> 5) + 1] - g0;
                T += k * pose + 12 * t.glink[v >> 5];
            }
        }
        const int ngw = __reduce_max_sync(kFull, ng);
        bool any_open = false;
        for (int jb = 0; jb < ngw; jb += 8) {
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
            float3 c = make_float3(0.f, 0.f, 0.f);
            bool open = false, h = false;
            if (jb + sl < ng) {
                c = sphere_centre(t, T, g0 + jb + sl, s);
                open = sphere_open(t, E, c, s.w, h);
            }
            hit |= __reduce_or_sync(kFull, h ? 1u << k : 0u);
            if (CNT) fl += (unsigned long long)__popc(__ballot_sync(kFull, jb + sl < ng)) * (18 + kFlField);
            if (!TIGHT) {
                any_open |= open;
                continue;
            }
            // --- 3, tight scenes: spheres left open, in states that have not collided ---
            for (unsigned ob = __ballot_sync(kFull, open && !((hit >> k) & 1u)); ob; ob &= ob - 1u) {
                const int x = __ffs(ob) - 1;
                const int kx = __shfl_sync(kFull, k, x);
                if ((hit >> kx) & 1u) continue;
                const float3 cx = make_float3(__shfl_sync(kFull, c.x, x), __shfl_sync(kFull, c.y, x),
                                              __shfl_sync(kFull, c.z, x));
                if (warp_sphere_hits<CNT>(t, E, cx, __shfl_sync(kFull, s.w, x), lane, fl)) hit |= 1u << kx;
            }
        }
        if (TIGHT) continue;
        const bool stays = (__ballot_sync(kFull, any_open) >> sh & 0xffu) && sl == 0 && !((hit >> k) & 1u);
        const unsigned bal = __ballot_sync(kFull, stays);
        if (stays) sc.it[left + __popc(bal & ((1u << lane) - 1u))] = v;
        left += __popc(bal);
        __syncwarp();
    }

    // --- 3, other scenes: the items left open, all groups of a state (within 32) at a time ---
#pragma unroll 1
    for (int i = 0; i < left;) {
        const int lead = sc.it[i], k = lead & 31, v = i + lane < left ? sc.it[i + lane] : -1;
        const bool same = v >= 0 && (v & 31) == k && v >> 10 == lead >> 10;   // items stand by state, then group
        const unsigned groups = __reduce_or_sync(kFull, same ? 1u << (v >> 5 & 31) : 0u);
        i += __popc(__ballot_sync(kFull, same));
        if ((hit >> k) & 1u) continue;
        const int base = lead >> 10 << 5;
        if (warp_groups_hit<CNT>(t, E, sc.lpK + k * pose, sc.gb + k * G + base, base, groups, lane, fl)) hit |= 1u << k;
    }
    __syncwarp();

    // --- 4: self pairs, 32 group pairs (one a lane) in every state, then the overlapping ones ---
#pragma unroll 1
    for (int q0 = 0; q0 < R.NPL && hit != all; q0 += kWarp) {
        unsigned on = 0u;   // states in which this lane's group pair overlaps
        if (q0 + lane < R.NPL) {
            const int4 pr = t.lpair[q0 + lane];
            const float4 *ga = sc.gb + pair_group(pr.x), *gb = sc.gb + pair_group(pr.y);
            for (int k = 0; k < ks; ++k) {
                const float4 a = ga[k * G], b = gb[k * G];
                const float rr = a.w + b.w;
                if (sq3(a.x - b.x, a.y - b.y, a.z - b.z) < rr * rr) on |= 1u << k;
            }
        }
        on &= ~hit;
        if (CNT) fl += (unsigned long long)min(kWarp, R.NPL - q0) * ks * kFlGroupPair;
        int n = 0;
        for (unsigned left = __reduce_or_sync(kFull, on); left; left &= left - 1u) {
            const int k = __ffs(left) - 1;
            const unsigned bal = __ballot_sync(kFull, (on >> k) & 1u);
            if ((on >> k) & 1u) sc.it[n + __popc(bal & ((1u << lane) - 1u))] = ((q0 + lane) << 5) | k;
            n += __popc(bal);
        }
        __syncwarp();
#pragma unroll 1
        for (int j0 = 0; j0 < n; j0 += 4) {
            int k = 0;
            int4 pr = make_int4(0, 0, 0, 0);
            float4 GA = make_float4(0.f, 0.f, 0.f, 0.f), GB = GA;
            const float *lp = sc.lpK;
            if (j0 + sub < n) {
                const int v = sc.it[j0 + sub];
                k = v & 31;
                if (!((hit >> k) & 1u)) {
                    pr = t.lpair[v >> 5];
                    lp += k * pose;
                    GA = sc.gb[k * G + pair_group(pr.x)];
                    GB = sc.gb[k * G + pair_group(pr.y)];
                }
            }
            const bool h = group_pair_hits<CNT>(t, R, lp, pr, GA, GB, sl, sh, fl);
            hit |= __reduce_or_sync(kFull, h ? 1u << k : 0u);
        }
        __syncwarp();
    }
    if (CNT && lane == 0) {
        atomicAdd(R.work, fl);
        atomicAdd(R.work + 1, (unsigned long long)ks);
    }
    return hit;
}

// Link poses (vec: 16-byte aligned) and sphere centres of the ks consecutive states from s0
// whose FK is in lpK, written as contiguous blocks.
__device__ inline void store_fk_states(const SmemTables &t, int L, int S, const float *lpK, long long s0, int ks,
                                       float *__restrict__ poses, float *__restrict__ centers, int vec, int lane) {
    if (poses) {
        if (vec) {
            float4 *P4 = reinterpret_cast<float4 *>(poses + s0 * L * 16);
            const float4 *rows = reinterpret_cast<const float4 *>(lpK);
            for (int f = lane; f < ks * L * 4; f += kWarp) {
                const int r = f & 3, kl = f >> 2;   // kl = k * L + link
                P4[f] = r < 3 ? rows[3 * kl + r] : make_float4(0.f, 0.f, 0.f, 1.f);
            }
        } else {
            float *P = poses + s0 * L * 16;
            for (int e = lane; e < ks * L * 16; e += kWarp) {
                const int kl = e >> 4, k = e & 15;
                P[e] = k < 12 ? lpK[12 * kl + k] : (k == 15 ? 1.f : 0.f);
            }
        }
    }
    if (centers) {
        float *Cc = centers + s0 * S * 3;
        for (int p = lane; p < ks * S; p += kWarp) {
            const int k = p / S, j = p - k * S;
            const int i = t.place[j];
            const float4 sp = t.sph[i];
            const float3 c3 = xform_point_a16(lpK + 12 * (k * L + t.slink[i]), sp.x, sp.y, sp.z);
            Cc[3 * p] = c3.x;
            Cc[3 * p + 1] = c3.y;
            Cc[3 * p + 2] = c3.z;
        }
    }
}

// States s0 .. s0 + ks - 1 of a verdict check, one warp: FK, poses / centres when asked for,
// verdicts.
template <bool CNT, bool TIGHT>
__device__ inline void check_verdicts(const SmemTables &t, const DevRobot &R, const DevEnv &E, const StatesScratch &sc,
                                      const float *__restrict__ q, long long s0, int ks,
                                      unsigned char *__restrict__ verdict, float *__restrict__ poses,
                                      float *__restrict__ centers, int vec, int lane) {
    const float *qs = q + s0 * R.L;
    warp_fk_chunk_q<kStatesMax>(t, R.L, ks, [&](int k, int i) { return qs[k * R.L + i]; }, sc.lpK, lane);
    if (poses || centers) store_fk_states(t, R.L, R.S, sc.lpK, s0, ks, poses, centers, vec, lane);
    const unsigned hit = warp_verdicts<CNT, TIGHT>(t, R, E, sc, ks, lane);
    if (verdict && lane < ks) verdict[s0 + lane] = (hit >> lane) & 1u;
    __syncwarp();
}

}  // namespace gbmp
