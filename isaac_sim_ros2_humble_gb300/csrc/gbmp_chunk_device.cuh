// gbmp_chunk_device.cuh -- validation of consecutive states of an edge by chunks
// (device routines shared by the edge-validation kernel, gbmp_chunk.cu, and the
// planner's edge checks, gbmp_rrtc_device.cuh).
//
// The interpolated states of one edge lie millimetres apart, so the obstacles near one
// state are the obstacles near its neighbours.  A warp takes K consecutive states of
// one edge (a chunk) and
//   A. runs the FK of all K states together (the joint-local transforms spread over the
//      lanes, then one lane per pose row of each state walking the chain), keeping the
//      link poses in shared memory, and bounds the centre of every sphere group (a
//      piece of a link's spheres) over the chunk by an axis-aligned box;
//   B. turns each box into a swept group sphere: centre = box centre, radius = half the
//      box diagonal + the group radius (which already carries kBroadMargin);
//   C. runs the broad phase ONCE for the chunk: the swept group spheres that the scene's
//      distance field does not clear (scene_far, one load a group, all groups at once)
//      against the bounding sphere of every run of 32 obstacles (scenes store obstacles
//      in spatially compact runs), then the obstacles of the runs some group touches against those
//      groups; an obstacle that touches any is tested exactly at once (D);
//   D. exact tests with the chunk's states side by side in the lanes: (state, sphere)
//      against an obstacle, (state, group pair) for the self pairs, whose overlapping
//      ones are settled four at a time, eight lanes each.  Sphere centres are computed
//      where they are tested; nothing is placed that no test reads.
// Because the swept spheres enclose every per-state group sphere, the tests cover every
// obstacle and pair any state of the chunk can touch, and they are the per-state
// kernel's (the same centres, rounded the same way): verdicts and first-hit indices
// equal the per-state kernel's.
//
// What bounds it: instruction issue and latency, not memory (the tables live in shared
// memory).  65,536 edges of the benchmark: 2.26 ms when every swept sphere was tested
// against every run, 1.25 ms with the field (most chunks then have no group left).
// Walking the states one after another left most lanes idle: per state of the benchmark's
// edges 0.3 obstacle candidates and 2.3 group pairs, each pair's test a chain of
// shared-memory loads over 7 spheres.  Side by side the chunk's 23 (state, pair) items fill
// a warp (3.8 -> 2.2 ms).  And the size of the code counts: the chunk kernel's loops are not unrolled
// (51 KB instead of 75 KB; 65,536 edges 1.21 against 1.25 ms a call), for the instruction cache
// holds about one such body.
#pragma once

#include "gbmp_internal.h"

namespace gbmp {

struct ChunkScratch {
    float *lpK;       // link poses of the chunk's states [K][L*12]
    float4 *sgb;      // swept group spheres (x, y, z, R) [G]
    float *sgA;       // |c|^2 - R^2 of each swept sphere
    int *pl;          // group pairs of one round whose swept spheres overlap [32]
    int *it;          // (state, pair) items of one round whose group spheres overlap [32]
};

// Per-warp shared memory of the chunk kernel: 4.9 KB for the 8-DOF benchmark arm at 10
// states (the joint-local transforms live where the poses replace them).
__host__ __device__ inline size_t smem_chunk_bytes(const DevRobot &R, int K) {
    return align16(sizeof(float) * 12 * R.L * K) + align16(sizeof(float4) * R.G) + align16(sizeof(float) * R.G) +
           2 * align16(sizeof(int) * kWarp);
}

__device__ inline void carve_chunk(unsigned char *base, const DevRobot &R, int K, int warp, ChunkScratch &c) {
    unsigned char *p = base + smem_chunk_bytes(R, K) * warp;
    size_t off = 0;
    c.lpK = reinterpret_cast<float *>(p + off); off += align16(sizeof(float) * 12 * R.L * K);
    c.sgb = reinterpret_cast<float4 *>(p + off); off += align16(sizeof(float4) * R.G);
    c.sgA = reinterpret_cast<float *>(p + off); off += align16(sizeof(float) * R.G);
    c.pl = reinterpret_cast<int *>(p + off); off += align16(sizeof(int) * kWarp);
    c.it = reinterpret_cast<int *>(p + off);
}

// FK of a chunk's ks states, all chains advancing together: first the ks x (L - 1)
// joint-local transforms of links 1.. spread over the lanes link-major (the lanes of one
// pass mostly share a joint type, so the type branches diverge little; link 0 is the
// identity and needs none), then the chains, one pose row a lane (below), each pose
// written over the joint-local transform it is made from.  qv(k, i) is joint i of state
// k.  The arithmetic is warp_fk's (joint_local, mul_elem), so poses are bit-identical.
template <int K, int UNROLL = 1, typename QV>
__device__ inline void warp_fk_chunk_q(const SmemTables &t, int L, int ks, QV qv, float *lpK, int lane) {
    const unsigned rks = (65536u + ks - 1u) / ks;   // idx / ks = idx * rks >> 16 (idx < 64 * 10)
#pragma unroll UNROLL
    for (int idx = lane; idx < ks * (L - 1); idx += kWarp) {
        const int i = 1 + (int)(idx * rks >> 16), k = idx - (i - 1) * ks;
        joint_local(t, i, qv(k, i), lpK + 12 * (k * L + i));
    }
    __syncwarp();
    // Composition: lane 3 k + r (k < ks) owns row r of state k's poses and walks the
    // links in order.  The parent's row is the lane's own: in registers while the parent
    // is the previous link, else its own earlier store.  The three lanes of a state read
    // a link's transform before any of them writes its pose there (the barrier).  Rows and
    // transforms are 16-byte aligned (48-byte poses in a block carved on 16 bytes) and
    // move as float4.
    static_assert(3 * K <= kWarp, "one lane per pose row of every state of a chunk");
    const int kr = lane / 3, rr = lane - 3 * kr;
    const bool own = lane < 3 * ks;
    float4 *base = reinterpret_cast<float4 *>(lpK + (own ? kr : 0) * 12 * L);
    float4 *rowp = base + rr;   // row rr of link 0
    const float4 unit = make_float4(rr == 0 ? 1.f : 0.f, rr == 1 ? 1.f : 0.f, rr == 2 ? 1.f : 0.f, 0.f);
    float4 a = unit;
    if (own) *rowp = a;
#pragma unroll UNROLL
    for (int i = 1; i < L; ++i) {
        const int ty = t.type[i], par = t.parent[i];
        float4 o = unit;
        if (own) {
            if (par != i - 1) a = rowp[3 * par];
            if (ty == 1 || ty == 2 || ty == 5) {
                const float4 b0 = base[3 * i], b1 = base[3 * i + 1], b2 = base[3 * i + 2];
                o.x = __fmaf_rn(a.z, b2.x, __fmaf_rn(a.y, b1.x, __fmul_rn(a.x, b0.x)));
                o.y = __fmaf_rn(a.z, b2.y, __fmaf_rn(a.y, b1.y, __fmul_rn(a.x, b0.y)));
                o.z = __fmaf_rn(a.z, b2.z, __fmaf_rn(a.y, b1.z, __fmul_rn(a.x, b0.z)));
                o.w = __fadd_rn(__fmaf_rn(a.z, b2.w, __fmaf_rn(a.y, b1.w, __fmul_rn(a.x, b0.w))), a.w);
            }
        }
        __syncwarp();
        if (own) rowp[3 * i] = o;
        a = o;
    }
    __syncwarp();
}

// FK of the chunk's ks states of one edge (state s = s0 + k from f towards t by d, the
// last state of the edge exactly t).
template <int K>
__device__ inline void warp_fk_chunk(const SmemTables &t, int L, int ks, const float *__restrict__ f,
                                     const float *__restrict__ to, const float *__restrict__ d, int s0, int n,
                                     float *lpK, int lane) {
    warp_fk_chunk_q<K>(
        t, L, ks,
        [&](int k, int i) {
            const int s = s0 + k;
            return (s == n - 1) ? to[i] : __fmaf_rn(d[i], (float)s, f[i]);
        },
        lpK, lane);
}

// Groups of `groups` (bit q) whose swept sphere touches the bounding sphere of run c0 +
// lane of an obstacle type with nruns runs; 0 for lanes past the last run.
__device__ __forceinline__ unsigned run_groups(const float4 *runs, int nruns, int c0, const ChunkScratch &cs,
                                               unsigned groups, int lane) {
    const int c = c0 + lane;
    unsigned gm = 0u;
    if (c < nruns) {
        const float4 b = runs[c];
#pragma unroll 1
        for (unsigned m = groups; m; m &= m - 1u) {
            const int q = __ffs(m) - 1;
            const float4 gs = cs.sgb[q];
            const float rr = gs.w + b.w;
            if (sq3(gs.x - b.x, gs.y - b.y, gs.z - b.z) < rr * rr) gm |= 1u << q;
        }
    }
    return gm;
}

// xform_point for a link pose in the chunk's pose block, which is 16-byte aligned (the
// block starts on 16 bytes and every pose is 48 bytes): three float4 loads, the same
// arithmetic.
__device__ __forceinline__ float3 xform_point_a16(const float *T, float x, float y, float z) {
    const float4 *T4 = reinterpret_cast<const float4 *>(T);
    const float4 r0 = T4[0], r1 = T4[1], r2 = T4[2];
    float3 o;
    o.x = __fadd_rn(__fmaf_rn(r0.z, z, __fmaf_rn(r0.y, y, __fmul_rn(r0.x, x))), r0.w);
    o.y = __fadd_rn(__fmaf_rn(r1.z, z, __fmaf_rn(r1.y, y, __fmul_rn(r1.x, x))), r1.w);
    o.z = __fadd_rn(__fmaf_rn(r2.z, z, __fmaf_rn(r2.y, y, __fmul_rn(r2.x, x))), r2.w);
    return o;
}

// Sphere j's centre in a state; T is the pose of its link.
__device__ __forceinline__ float3 sphere_centre(const SmemTables &t, const float *T, int j, float4 &s) {
    s = t.sph[j];
    return xform_point_a16(T, s.x, s.y, s.z);
}

// Group g's bounding sphere in the state whose link poses start at lp.
__device__ __forceinline__ float4 group_sphere(const SmemTables &t, const float *lp, int g) {
    const float4 s = t.grp[g];
    const float3 c = xform_point_a16(lp + 12 * t.glink[g], s.x, s.y, s.z);
    return make_float4(c.x, c.y, c.z, s.w);
}

// The states k < kmax of the chunk against one obstacle (TYPE 0 sphere, 1 cuboid, 2
// cylinder; o its index within the type), the spheres of the groups in `gm` only: the
// lanes take (state, sphere) pairs.  Returns the lane's lowest colliding state, or kmax.
template <int TYPE, bool CNT>
__device__ __forceinline__ int chunk_obstacle(const SmemTables &t, const DevRobot &R, const DevEnv &E,
                                              const float *lpK, int o, unsigned gm, int kmax, int lane,
                                              unsigned long long &fl) {
    float4 r0, r1, r2, p3, p4;
    float nb = 0.f;
    if (TYPE == 0) {
        const float4 *sx = t.env + E.ns + 5 * E.nb + 4 * E.nc;
        r0 = sx[o];
        nb = reinterpret_cast<const float *>(sx + E.ns)[o];
    } else if (TYPE == 1) {
        const float4 *bx = t.env + E.ns + 5 * o;
        r0 = bx[0]; r1 = bx[1]; r2 = bx[2]; p3 = bx[3]; p4 = bx[4];
    } else {
        const float4 *cy = t.env + E.ns + 5 * E.nb + 4 * o;
        r0 = cy[0]; r1 = cy[1]; r2 = cy[2]; p3 = cy[3];
    }
    int hk = kmax;
#pragma unroll 1
    for (; gm; gm &= gm - 1u) {
        const int g = __ffs(gm) - 1;
        const int g0 = t.gso[g], ng = t.gso[g + 1] - g0, total = ng * kmax;
        const float *T = lpK + 12 * t.glink[g];
        const float inv = 1.f / (float)ng;
#pragma unroll 1
        for (int idx = lane; idx < total; idx += kWarp) {
            const int k = (int)(((float)idx + 0.5f) * inv);   // idx / ng (idx < 2^12)
            float4 s;
            const float3 c = sphere_centre(t, T + k * 12 * R.L, g0 + idx - k * ng, s);
            bool h;
            if (TYPE == 0) {   // expanded form, see warp_collide
                const float A = __fmaf_rn(c.z, c.z, __fmaf_rn(c.y, c.y, __fmaf_rn(c.x, c.x, -s.w * s.w)));
                const float v = __fmaf_rn(c.x, r0.x, __fmaf_rn(c.y, r0.y, __fmaf_rn(c.z, r0.z, __fmaf_rn(s.w, r0.w, nb))));
                h = v > A;
            } else {
                const float3 l = xform_rows(r0, r1, r2, c.x, c.y, c.z);
                if (TYPE == 1) {
                    const float dx = l.x - fminf(fmaxf(l.x, p3.x), p4.x);
                    const float dy = l.y - fminf(fmaxf(l.y, p3.y), p4.y);
                    const float dz = l.z - fminf(fmaxf(l.z, p3.z), p4.z);
                    h = sq3(dx, dy, dz) < s.w * s.w;
                } else {
                    const float dx = sqrtf(__fmaf_rn(l.y, l.y, __fmul_rn(l.x, l.x))) - p3.x;
                    const float dz = fabsf(l.z) - p3.y;
                    const float ox = dx > 0.f ? dx : 0.f, oz = dz > 0.f ? dz : 0.f;
                    const float outside = sqrtf(__fmaf_rn(oz, oz, __fmul_rn(ox, ox)));
                    const float inside = fminf(fmaxf(dx, dz), 0.f);
                    h = s.w - (outside + inside) > 0.f;
                }
            }
            if (h) hk = min(hk, k);
        }
        if (CNT) fl += (unsigned long long)total * (24 + (TYPE == 0 ? kFlSphereX : TYPE == 1 ? kFlCuboid : kFlCylinder));
    }
    return hk;
}

// Whether a sphere of one group touches one of the other, eight lanes for a group pair
// (sl the lane's place among them, sh its first lane's number; every warp settles four
// pairs at once; pr: the pair's word of lpair, all 0 for none): the spheres of b against
// a's group sphere GA, and only where one touches it, a's spheres against GB and the
// touching pairs exactly, with the pair threshold (ri + rj)^2 rounded as the pair list's.
// A sphere that touches a sphere of the other group touches that group's enclosing sphere,
// so nothing is lost.  A group pair whose enabled sphere pairs are not all (sphere of a,
// sphere of b) pairs walks the pair list.  lp: the state's link poses.  True on the lanes
// that found a contact.
template <bool CNT>
__device__ __forceinline__ bool group_pair_hits(const SmemTables &t, const DevRobot &R, const float *lp, int4 pr,
                                                float4 GA, float4 GB, int sl, int sh, unsigned long long &fl) {
    bool hit = false;
    const int na = pair_count(pr.x), nb = pair_count(pr.y), b0 = pair_first(pr.y);
    const bool full = pr.w - pr.z == na * nb;
    const float *TA = lp + 12 * t.glink[pair_group(pr.x)], *TB = lp + 12 * t.glink[pair_group(pr.y)];
    const int nbw = __reduce_max_sync(kFull, full ? nb : 0);
#pragma unroll 1
    for (int jb = 0; jb < nbw; jb += 8) {
        bool ib = false;
        if (full && jb + sl < nb) {
            float4 s;
            const float3 c = sphere_centre(t, TB, b0 + jb + sl, s);
            const float rr = s.w + GA.w;
            ib = sq3(c.x - GA.x, c.y - GA.y, c.z - GA.z) < rr * rr;
        }
        const unsigned mb = (__ballot_sync(kFull, ib) >> sh) & 0xffu;
        if (mb) {
#pragma unroll 1
            for (int ja = sl; ja < na; ja += 8) {
                float4 s;
                const float3 c = sphere_centre(t, TA, pair_first(pr.x) + ja, s);
                const float rr = s.w + GB.w;
                if (sq3(c.x - GB.x, c.y - GB.y, c.z - GB.z) < rr * rr) {
#pragma unroll 1
                    for (unsigned m = mb; m; m &= m - 1u) {
                        float4 sb;
                        const float3 cb = sphere_centre(t, TB, b0 + jb + __ffs(m) - 1, sb);
                        const float sr = __fadd_rn(s.w, sb.w);
                        hit |= sq3(c.x - cb.x, c.y - cb.y, c.z - cb.z) < __fmul_rn(sr, sr);
                    }
                }
            }
        }
        if (CNT) {   // sphere centres and tests against the group spheres
            fl += (unsigned long long)__popc(__ballot_sync(kFull, full && jb + sl < nb)) * (18 + kFlSelf);
            fl += (unsigned long long)__reduce_add_sync(kFull, sl == 0 && mb ? na : 0) * (18 + kFlSelf);
        }
    }
    if (!full)
#pragma unroll 1
        for (int p = pr.z + sl; p < pr.w; p += 8) {
            const unsigned ij = __ldg(R.pairs + p);
            const float thr = __ldg(R.thr + p);
            float4 s;
            const float3 a = sphere_centre(t, lp + 12 * t.slink[ij & 0xffffu], ij & 0xffffu, s),
                         b = sphere_centre(t, lp + 12 * t.slink[ij >> 16], ij >> 16, s);
            hit |= sq3(a.x - b.x, a.y - b.y, a.z - b.z) < thr;
        }
    return hit;
}

// Self pairs of the group pairs cs.pl[0 .. npr) in the states k < kmax: the lanes first
// take (state, pair) items and keep those whose group spheres overlap; the kept items are
// settled four at a time (group_pair_hits).  Returns the lane's lowest colliding state, or
// kmax.
template <bool CNT>
__device__ __forceinline__ int chunk_self(const SmemTables &t, const DevRobot &R, const ChunkScratch &cs, int npr,
                                          int kmax, bool any, int lane, unsigned long long &fl) {
    const int total = npr * kmax;
    const float inv = 1.f / (float)npr;
    const int sub = lane >> 3, sl = lane & 7, sh = lane & 24;
    int hk = kmax;
#pragma unroll 1
    for (int i0 = 0; i0 < total; i0 += kWarp) {
        const int idx = i0 + lane;
        bool on = false;
        int item = 0;
        if (idx < total) {
            const int k = (int)(((float)idx + 0.5f) * inv), p = cs.pl[idx - k * npr];   // idx / npr (idx < 2^12)
            const int4 lp = t.lpair[p];
            const float *poses = cs.lpK + k * 12 * R.L;
            const float4 a = group_sphere(t, poses, pair_group(lp.x)), b = group_sphere(t, poses, pair_group(lp.y));
            const float rr = a.w + b.w;
            on = sq3(a.x - b.x, a.y - b.y, a.z - b.z) < rr * rr;
            item = (p << 5) | k;
        }
        const unsigned bal = __ballot_sync(kFull, on);
        if (CNT) fl += (unsigned long long)min(kWarp, total - i0) * (kFlGroupPair + 36);
        if (!bal) continue;
        if (on) cs.it[__popc(bal & ((1u << lane) - 1u))] = item;
        __syncwarp();
        const int nit = __popc(bal);
#pragma unroll 1
        for (int j0 = 0; j0 < nit; j0 += 4) {
            int k = 0;
            int4 pr = make_int4(0, 0, 0, 0);
            float4 GA = make_float4(0.f, 0.f, 0.f, 0.f), GB = GA;
            const float *lp = cs.lpK;
            if (j0 + sub < nit) {
                const int v = cs.it[j0 + sub];
                k = v & 31;
                pr = t.lpair[v >> 5];
                lp += k * 12 * R.L;
                GA = group_sphere(t, lp, pair_group(pr.x));
                GB = group_sphere(t, lp, pair_group(pr.y));
            }
            if (group_pair_hits<CNT>(t, R, lp, pr, GA, GB, sl, sh, fl)) hk = min(hk, k);
            if (any && __any_sync(kFull, hk < kmax)) return hk;
        }
        __syncwarp();
    }
    return hk;
}

// States [s0, s1) of one edge (from f to `to` with per-state step d, n states in all).
// Returns the lowest colliding state -- with `any`, some colliding state -- or -1.
template <int K, bool CNT>
__device__ inline int warp_edge_chunk(const SmemTables &t, const DevRobot &R, const DevEnv &E, const ChunkScratch &cs,
                                      int lane, const float *__restrict__ f, const float *__restrict__ to,
                                      const float *__restrict__ d, int s0, int s1, int n, bool any) {
    const int ks = s1 - s0;
    // FK and the group-centre transforms of every state; sphere centres are counted
    // where they are computed
    unsigned long long fl = (unsigned long long)(R.base_flops - 24LL * R.S) * ks;

    // --- A: FK of every state, box of each group centre ---
    warp_fk_chunk<K>(t, R.L, ks, f, to, d, s0, n, cs.lpK, lane);
    // lane = (part, group): the states are dealt to 32 / gw parts, gw >= G a power of two
    const int gw = R.G <= 8 ? 8 : R.G <= 16 ? 16 : 32;
    const int gq = lane & (gw - 1);
    float lox = 3.0e38f, loy = 3.0e38f, loz = 3.0e38f, hix = -3.0e38f, hiy = -3.0e38f, hiz = -3.0e38f;
    float gr = 0.f;
    if (gq < R.G) {
        const float4 g = t.grp[gq];
        const float *T = cs.lpK + 12 * t.glink[gq];
        gr = g.w;
#pragma unroll 1
        for (int k = lane / gw; k < ks; k += kWarp / gw) {
            const float3 c = xform_point_a16(T + k * 12 * R.L, g.x, g.y, g.z);
            lox = fminf(lox, c.x); loy = fminf(loy, c.y); loz = fminf(loz, c.z);
            hix = fmaxf(hix, c.x); hiy = fmaxf(hiy, c.y); hiz = fmaxf(hiz, c.z);
        }
    }
#pragma unroll 1
    for (int off = gw; off < kWarp; off <<= 1) {
        lox = fminf(lox, __shfl_xor_sync(kFull, lox, off));
        loy = fminf(loy, __shfl_xor_sync(kFull, loy, off));
        loz = fminf(loz, __shfl_xor_sync(kFull, loz, off));
        hix = fmaxf(hix, __shfl_xor_sync(kFull, hix, off));
        hiy = fmaxf(hiy, __shfl_xor_sync(kFull, hiy, off));
        hiz = fmaxf(hiz, __shfl_xor_sync(kFull, hiz, off));
    }

    // --- B: swept group spheres; those that the scene's distance field cannot clear ---
    bool is_near = false;
    if (lane < R.G) {
        const float cx = 0.5f * (lox + hix), cy = 0.5f * (loy + hiy), cz = 0.5f * (loz + hiz);
        const float hx = 0.5f * (hix - lox), hy = 0.5f * (hiy - loy), hz = 0.5f * (hiz - loz);
        const float rad = sqrtf(hx * hx + hy * hy + hz * hz) + gr;
        cs.sgb[lane] = make_float4(cx, cy, cz, rad);
        cs.sgA[lane] = __fmaf_rn(cz, cz, __fmaf_rn(cy, cy, __fmaf_rn(cx, cx, -rad * rad)));
        is_near = !scene_far(E, cx, cy, cz, rad);
    }
    const unsigned near_groups = __ballot_sync(kFull, is_near);
    if (CNT) fl += (unsigned long long)R.G * kFlField;
    __syncwarp();

    int kmax = ks;   // states below kmax are not yet known to collide (any: kmax == ks)
    auto settle = [&](int hk) {   // the lanes' lowest colliding states; true when done
        kmax = (int)__reduce_min_sync(kFull, (unsigned)hk);
        return any ? kmax < ks : kmax == 0;
    };

    // --- C: broad phase of the chunk, run spheres first ---
    // The bounding spheres of all runs (sphere runs, then box runs, then cylinder runs)
    // are tested in one pass, lane j taking run c0 + j against every swept group sphere;
    // only runs some group touches are visited, their obstacles are tested only against
    // the groups that touched the run, and an obstacle that touches a swept group sphere
    // is tested exactly (D).
    const float4 *sx = t.env + E.ns + 5 * E.nb + 4 * E.nc;
    const float *snb = reinterpret_cast<const float *>(sx + E.ns);
    const float4 *bx = t.env + E.ns;
    const float4 *cyl = t.env + E.ns + 5 * E.nb;
    const int nrs = env_clusters(E.ns), nrb = env_clusters(E.nb), nrun = nrs + nrb + env_clusters(E.nc);
    const float4 *runs_w = t.env + env_cluster_base(E.ns, E.nb, E.nc);
    bool done = false;
#pragma unroll 1
    for (int c0 = 0; c0 < nrun && near_groups && !done; c0 += kWarp) {
        const unsigned gmc = run_groups(runs_w, nrun, c0, cs, near_groups, lane);
        unsigned runs = __ballot_sync(kFull, gmc != 0u);
        if (CNT) fl += (unsigned long long)min(kWarp, nrun - c0) * __popc(near_groups) * kFlGroupPair;
        while (runs && !done) {
            const int j = __ffs(runs) - 1;
            runs &= runs - 1u;
            const unsigned gm = __shfl_sync(kFull, gmc, j);
            const int c = c0 + j;
            unsigned mask = 0u;
            if (c < nrs) {   // obstacle spheres (expanded form, see warp_collide)
                const int o = c * kWarp + lane;
                if (o < E.ns) {
                    const float4 b = sx[o];
                    const float nb = snb[o];
#pragma unroll 1
                    for (unsigned m = gm; m; m &= m - 1u) {
                        const int q = __ffs(m) - 1;
                        const float4 gs = cs.sgb[q];
                        const float v = __fmaf_rn(gs.x, b.x, __fmaf_rn(gs.y, b.y, __fmaf_rn(gs.z, b.z, __fmaf_rn(gs.w, b.w, nb))));
                        if (v > cs.sgA[q]) mask |= 1u << q;
                    }
                }
                if (CNT) fl += (unsigned long long)min(kWarp, E.ns - c * kWarp) * __popc(gm) * kFlSphereX;
            } else if (c < nrs + nrb) {   // cuboids
                const int o = (c - nrs) * kWarp + lane;
                if (o < E.nb) {
                    const float4 r0 = bx[5 * o], r1 = bx[5 * o + 1], r2 = bx[5 * o + 2], mn = bx[5 * o + 3], mx = bx[5 * o + 4];
#pragma unroll 1
                    for (unsigned m = gm; m; m &= m - 1u) {
                        const int q = __ffs(m) - 1;
                        const float4 gs = cs.sgb[q];
                        const float3 l = xform_rows(r0, r1, r2, gs.x, gs.y, gs.z);
                        const float dx = l.x - fminf(fmaxf(l.x, mn.x), mx.x);
                        const float dy = l.y - fminf(fmaxf(l.y, mn.y), mx.y);
                        const float dz = l.z - fminf(fmaxf(l.z, mn.z), mx.z);
                        if (sq3(dx, dy, dz) < gs.w * gs.w) mask |= 1u << q;
                    }
                }
                if (CNT) fl += (unsigned long long)min(kWarp, E.nb - (c - nrs) * kWarp) * __popc(gm) * kFlCuboid;
            } else {   // cylinders
                const int o = (c - nrs - nrb) * kWarp + lane;
                if (o < E.nc) {
                    const float4 r0 = cyl[4 * o], r1 = cyl[4 * o + 1], r2 = cyl[4 * o + 2], pr = cyl[4 * o + 3];
#pragma unroll 1
                    for (unsigned m = gm; m; m &= m - 1u) {
                        const int q = __ffs(m) - 1;
                        const float4 gs = cs.sgb[q];
                        const float3 l = xform_rows(r0, r1, r2, gs.x, gs.y, gs.z);
                        const float dx = sqrtf(__fmaf_rn(l.y, l.y, __fmul_rn(l.x, l.x))) - pr.x;
                        const float dz = fabsf(l.z) - pr.y;
                        const float ox = dx > 0.f ? dx : 0.f, oz = dz > 0.f ? dz : 0.f;
                        const float sdf = sqrtf(__fmaf_rn(oz, oz, __fmul_rn(ox, ox))) + fminf(fmaxf(dx, dz), 0.f);
                        if (gs.w - sdf > 0.f) mask |= 1u << q;
                    }
                }
                if (CNT) fl += (unsigned long long)min(kWarp, E.nc - (c - nrs - nrb) * kWarp) * __popc(gm) * kFlCylinder;
            }
            for (unsigned bal = __ballot_sync(kFull, mask != 0u); bal && !done; bal &= bal - 1u) {
                const int x = __ffs(bal) - 1;
                const unsigned om = __shfl_sync(kFull, mask, x);
                int hk;
                if (c < nrs) hk = chunk_obstacle<0, CNT>(t, R, E, cs.lpK, c * kWarp + x, om, kmax, lane, fl);
                else if (c < nrs + nrb) hk = chunk_obstacle<1, CNT>(t, R, E, cs.lpK, (c - nrs) * kWarp + x, om, kmax, lane, fl);
                else hk = chunk_obstacle<2, CNT>(t, R, E, cs.lpK, (c - nrs - nrb) * kWarp + x, om, kmax, lane, fl);
                done = settle(hk);
            }
        }
    }

    // --- self pairs: enabled group pairs whose swept spheres overlap, 32 at a time ---
#pragma unroll 1
    for (int k0 = 0; k0 < R.NPL && !done; k0 += kWarp) {
        const int k = k0 + lane;
        bool on = false;
        if (k < R.NPL) {
            const int4 lpr = t.lpair[k];
            const float4 a = cs.sgb[pair_group(lpr.x)], b = cs.sgb[pair_group(lpr.y)];
            const float rr = a.w + b.w;
            on = sq3(a.x - b.x, a.y - b.y, a.z - b.z) < rr * rr;
        }
        const unsigned bal = __ballot_sync(kFull, on);
        if (CNT) fl += (unsigned long long)min(kWarp, R.NPL - k0) * kFlGroupPair;
        if (!bal) continue;
        if (on) cs.pl[__popc(bal & ((1u << lane) - 1u))] = k;
        __syncwarp();
        done = settle(chunk_self<CNT>(t, R, cs, __popc(bal), kmax, any, lane, fl));
        __syncwarp();
    }
    if (CNT && lane == 0) {
        atomicAdd(R.work, fl);
        atomicAdd(R.work + 1, (unsigned long long)ks);
    }
    __syncwarp();
    return kmax < ks ? s0 + kmax : -1;
}

}  // namespace gbmp
