// Hemisphere rays of a patch of lumels, traced by one warp: the body of the
// ambient-occlusion and final-gather kernels.
//
// A lumel's rays share their origin and a half-space.  A walk from the root
// spends most of its visits on the boxes that hold the origin, which every
// ray of the lumel meets (17 of 22 on the terrain), and 80% of the terrain's
// rays hit nothing.  So a warp takes up to eight neighbouring lumels and
//   1. walks the tree once for all of them, opening every node whose box
//      meets the patch and dropping what lies behind every lumel's tangent
//      plane or out of reach: up to 32 subtrees remain (16 to 26 on the
//      terrain), which no ray has to find again;
//   2. takes the rays (lumel, sample) kChunk at a time: draws the directions
//      (each lane its rays one attempt after another, so that a lane that
//      accepted goes on to its next ray), tests the subtrees' boxes with all
//      lanes on the same box, and the triangles of the leaves at the origin;
//   3. walks the subtrees of the rays that met any (60%), lanes taking rays
//      from the chunk's queue, the rays that met most first;
//   4. adds the samples of each lumel in sample order.
// The hits are those of traverse() for each ray: the same boxes and triangles
// are tested except those that no ray of the patch can reach (kMargin), and
// the closest hit with the smaller-id tie-break does not depend on the order.
//
// What bounds it: the walk (14 of 25 ms on the terrain final gather) by the
// latency of its loads and by lanes whose walks differ; lists 0.6 ms, drawing
// 3, boxes 6.  Chunks of 256 rays: at 128 the warp waits longer for each
// chunk's last rays (27.7 ms), and half-chunks drawn while the last rays of
// the other half are walked spill (35 ms).  Patches of 4 and 2 lumels: 26.1
// and 27.2 ms.  Terrain final gather, 1024^2, 256 samples: 41.2 -> 25.0 ms
// (one lane per lumel, from the root, before); 97 x 75, 32 samples: 578 ->
// 115 us; terrain AO, 1024^2, 64 samples: 6.4 -> 3.8 ms.
#pragma once

#include "rl_device.cuh"

namespace rl {

constexpr int kPatch = 8;    // lumels that share a list, at most
constexpr int kChunk = 256;  // rays in flight per warp
constexpr int kList = 32;    // subtrees per patch, at most
constexpr unsigned kFull = 0xffffffffu;

// What the culling leaves out must be out of every ray's reach by far more
// than the rounding of the rays and of the triangle test: 2^-15 of the
// largest coordinate in play (the same order as the boxes' padding).
constexpr float kMargin = 1.0f / 32768.0f;

// One warp's shared memory.
template <bool kAny>
struct PatchMem {
    float4 xy[kList];     // centre x y, half-extent x y
    float4 zc[kList];     // centre z, half-extent z, node or leaf code, kOpen
    float pos[kPatch][3], nrm[kPatch][3], margin[kPatch];
    uint32_t item[kPatch];
    uint32_t own[kPatch];         // per lumel: list entries that are leaves whose box holds it
    float acc[kPatch][3];         // any hit: acc[p][0] counts (int bits)
    float v[3][kChunk];           // a ray's direction, then its sample's colour
    uint32_t mask[kChunk];        // subtrees that it met
    uint8_t queue[kChunk];        // rays to walk
};

constexpr int kOpen = 1;

struct PatchRays {
    uint2 key;
    uint32_t tag;
    int samples;
    float maxd;
};

// Slab test of one list entry, as slab2.
__device__ __forceinline__ bool slab1(float4 xy, float cz, float hz, const Slab& r, float iz, float oz, float az,
                                      float tnear, float tmax) {
    const f32x2 t = fma2(pack2(xy.x, xy.y), r.ixy, r.oxy), w = pack2(xy.z, xy.w);
    const float tz = __fmaf_rn(cz, iz, oz);
    const float2 a = unpack2(fma2(w, r.bxy, t)), b = unpack2(fma2(w, r.axy, t));
    const float lo = fmax3(a.x, a.y, fmaxf(__fmaf_rn(-hz, az, tz), tnear));
    const float hi = fmin3(b.x, b.y, fminf(__fmaf_rn(hz, az, tz), tmax));
    return lo <= hi * 1.0000003f;
}

// Whether rays of lumel p can reach the box: its farthest reach along the
// normal is not behind the tangent plane, and it is near enough.
template <bool kAny>
__device__ __forceinline__ bool in_reach(const PatchMem<kAny>& M, int p, float4 xy, float cz, float hz, float reach2) {
    const float nx = M.nrm[p][0], ny = M.nrm[p][1], nz = M.nrm[p][2];
    const float x = xy.x - M.pos[p][0], y = xy.y - M.pos[p][1], z = cz - M.pos[p][2];
    const float up = (nx * x + ny * y + nz * z) + (fabsf(nx) * xy.z + fabsf(ny) * xy.w + fabsf(nz) * hz);
    const float ex = fmaxf(fabsf(x) - xy.z, 0.f), ey = fmaxf(fabsf(y) - xy.w, 0.f), ez = fmaxf(fabsf(z) - hz, 0.f);
    return !(up < M.margin[p]) && !(ex * ex + ey * ey + ez * ez > reach2);
}

// The subtrees that rays of the patch's `lumels` lumels can reach, into
// M.xy / M.zc (returns their number), with the leaves that hold each lumel in
// M.own.  A list that would not fit keeps its nodes closed.
template <bool kAny>
__device__ __forceinline__ int patch_list(const DevScene& s, PatchMem<kAny>& M, int lumels, float maxd, int lane) {
    if (s.ntris == 0) {
        if (lane < kPatch) M.own[lane] = 0;
        __syncwarp();
        return 0;
    }
    float alo[3], ahi[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        alo[k] = ahi[k] = M.pos[0][k];
        for (int p = 1; p < lumels; p++) {
            alo[k] = fminf(alo[k], M.pos[p][k]);
            ahi[k] = fmaxf(ahi[k], M.pos[p][k]);
        }
    }
    // the largest coordinate in play; no culling where that is not a number or the rays run backwards
    float big = 0.f;
    {
        const float4 n0 = __ldg(s.nodes), n1 = __ldg(s.nodes + 1), n2 = __ldg(s.nodes + 2);
        const float c[12] = {fabsf(n0.x) + n0.z, fabsf(n0.y) + n0.w, fabsf(n1.x) + n1.z, fabsf(n1.y) + n1.w,
                             fabsf(n2.x) + n2.z, fabsf(n2.y) + n2.w, alo[0], alo[1], alo[2], ahi[0], ahi[1], ahi[2]};
#pragma unroll
        for (int k = 0; k < 12; k++) big = fmaxf(big, fabsf(c[k]));
    }
    const float m = maxd > 0.f ? kMargin * (big + maxd) : INFINITY;
    const float reach = maxd * (1.0f + 1.0f / 4096.0f) + m;
    const float reach2 = maxd > 0.f ? reach * reach : INFINITY;
    if (lane < lumels)
        M.margin[lane] = -m * (fabsf(M.nrm[lane][0]) + fabsf(M.nrm[lane][1]) + fabsf(M.nrm[lane][2]));
    __syncwarp();
    int count = 1, code = 0, flags = lane == 0 ? kOpen : 0;
    float4 xy = make_float4(0.f, 0.f, 0.f, 0.f);
    float cz = 0.f, hz = 0.f;
    const unsigned below = (1u << lane) - 1u;
    for (;;) {
        const bool open = lane < count && (flags & kOpen);
        if (!__any_sync(kFull, open)) break;
        float4 n0 = xy, n1 = xy, n2 = xy, n3 = xy;
        bool keep[2] = {false, false};
        int cflags[2] = {0, 0};
        if (open) {
            const float4* np = s.nodes + 4 * (size_t)code;
            n0 = __ldg(np);
            n1 = __ldg(np + 1);
            n2 = __ldg(np + 2);
            n3 = __ldg(np + 3);
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const float4 b = q == 0 ? n0 : n1;
                const float bc = q == 0 ? n2.x : n2.y, bh = q == 0 ? n2.z : n2.w;
                for (int p = 0; p < lumels && !keep[q]; p++) keep[q] = in_reach(M, p, b, bc, bh, reach2);
                const bool meets = b.x - b.z <= ahi[0] && b.x + b.z >= alo[0] && b.y - b.w <= ahi[1] &&
                                   b.y + b.w >= alo[1] && bc - bh <= ahi[2] && bc + bh >= alo[2];
                cflags[q] = meets && __float_as_int(q == 0 ? n3.x : n3.y) >= 0 ? kOpen : 0;
            }
        }
        const int kept = (keep[0] ? 1 : 0) + (keep[1] ? 1 : 0);
        const int out = open ? kept : (lane < count ? 1 : 0);
        const unsigned b1 = __ballot_sync(kFull, out >= 1), b2 = __ballot_sync(kFull, out == 2);
        const int total = __popc(b1) + __popc(b2);
        if (total > kList) break;  // stays closed
        const int at = __popc(b1 & below) + __popc(b2 & below);
        __syncwarp();
        if (open) {
            // the subtree at the origin last: it is walked first
            const bool swap = keep[1] && cflags[0] != 0 && cflags[1] == 0;
            if (keep[0]) {
                const int k = at + (swap ? 1 : 0);
                M.xy[k] = n0;
                M.zc[k] = make_float4(n2.x, n2.z, n3.x, __int_as_float(cflags[0]));
            }
            if (keep[1]) {
                const int k = at + (keep[0] && !swap ? 1 : 0);
                M.xy[k] = n1;
                M.zc[k] = make_float4(n2.y, n2.w, n3.y, __int_as_float(cflags[1]));
            }
        } else if (lane < count) {
            M.xy[at] = xy;
            M.zc[at] = make_float4(cz, hz, __int_as_float(code), __int_as_float(flags));
        }
        __syncwarp();
        count = total;
        if (lane < count) {
            xy = M.xy[lane];
            const float4 zc = M.zc[lane];
            cz = zc.x;
            hz = zc.y;
            code = __float_as_int(zc.z);
            flags = __float_as_int(zc.w);
        }
    }
    for (int p = 0; p < lumels; p++) {
        const float x = M.pos[p][0], y = M.pos[p][1], z = M.pos[p][2];
        const bool holds = lane < count && code < 0 && fabsf(x - xy.x) <= xy.z && fabsf(y - xy.y) <= xy.w &&
                           fabsf(z - cz) <= hz;
        const unsigned w = __ballot_sync(kFull, holds);
        if (lane == 0) M.own[p] = w;
    }
    __syncwarp();
    return count;
}

// One step of a walk: the next node is the nearer child met, else the top of
// the stack, else the next subtree of the ray's list mask.
struct Walk {
    V3 o, d;
    Slab slab;
    float best, hu, hv;
    int gid, sp, node;
    uint32_t mask;
};
template <bool kAny>
__device__ __forceinline__ void walk_pop(Walk& w, const PatchMem<kAny>& M, const int* stack) {
    if (w.sp > 0) {
        w.node = stack[--w.sp];
    } else if (w.mask) {
        const int e = 31 - __clz(w.mask);
        w.mask ^= 1u << e;
        w.node = __float_as_int(M.zc[e].z);
    } else {
        w.node = kNodeDone;
    }
}
template <bool kAny>
__device__ __forceinline__ void walk_node(const DevScene& s, Walk& w, const PatchMem<kAny>& M, int* stack,
                                          int* overflow) {
    const float4* np = s.nodes + 4 * (size_t)w.node;
    const float4 n0 = __ldg(np), n1 = __ldg(np + 1), n2 = __ldg(np + 2), n3 = __ldg(np + 3);
    bool h0, h1;
    float e0, e1;
    slab2(n0, n1, n2, w.slab, 0.01f, w.best, h0, h1, e0, e1);
    const int c0 = __float_as_int(n3.x), c1 = __float_as_int(n3.y);
    if (h0 && h1) {
        int nearc = c0, farc = c1;
        if (e1 < e0) { nearc = c1; farc = c0; }
        if (w.sp < kStackSize) stack[w.sp++] = farc;
        else if (overflow) *overflow = 1;
        w.node = nearc;
    } else if (h0 || h1) {
        w.node = h0 ? c0 : c1;
    } else {
        walk_pop(w, M, stack);
    }
}

// The rays of `lumels` lumels (M.pos, M.nrm, M.item set) of a patch.  `shade`
// turns a finished ray into its sample's colour: shade(dir, nrm, gid, u, v)
// -> V3 (gid -1: no hit); unused for any hit.  On return M.acc holds each
// lumel's colour sum in sample order (or its count of hits, int bits).
template <bool kAny, typename Shade>
__device__ __forceinline__ void patch_rays(const DevScene& s, PatchMem<kAny>& M, int lumels, const PatchRays& R,
                                           const Shade& shade, int refill, int* overflow) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const int nlist = patch_list(s, M, lumels, R.maxd, lane);
    if (lane < kPatch) M.acc[lane][0] = M.acc[lane][1] = M.acc[lane][2] = 0.f;  // int 0 as well
    __syncwarp();
    const unsigned S = (unsigned)R.samples;
    const unsigned total = (unsigned)lumels * S;  // the callers keep it below 2^31
    for (unsigned base = 0; base < total; base += kChunk) {
        const int n = (int)min((unsigned)kChunk, total - base);
        const unsigned p0 = base / S, edge = (p0 + 1) * S - base;  // lumel of ray 0; the first ray of the next one
        auto lumel_of = [&](unsigned r) {
            return (int)(S >= (unsigned)kChunk ? p0 + (r >= edge ? 1u : 0u) : (base + r) / S);
        };
        // directions: one attempt per step for each lane's current ray
        {
            int r = lane;
            unsigned p = (base + lane) / S, j = (base + lane) - p * S;
            uint32_t a = 0;
            while (r < n) {
                const uint4 w = philox(make_uint4(M.item[p], j, a, R.tag), R.key);
                const V3 v = mk3(u01(w.x) * 2.0f - 1.0f, u01(w.y) * 2.0f - 1.0f, u01(w.z) * 2.0f - 1.0f);
                if (!(len3(v) > 1.0f) || a == kMaxAttempts - 1) {
                    M.v[0][r] = v.x;
                    M.v[1][r] = v.y;
                    M.v[2][r] = v.z;
                    a = 0;
                    r += 32;
                    j += 32;
                    while (j >= S) {
                        j -= S;
                        p++;
                    }
                } else {
                    a++;
                }
            }
        }
        __syncwarp();
        // the list's boxes, and the triangles of the leaves that hold the lumel
        int queued = 0, light = kChunk;
        for (int r = lane; r - lane < n; r += 32) {
            uint32_t met = 0;
            if (r < n) {
                const int p = lumel_of(r);
                V3 dir = mk3(M.v[0][r], M.v[1][r], M.v[2][r]);
                const V3 nrm = mk3(M.nrm[p][0], M.nrm[p][1], M.nrm[p][2]);
                // random_hemisphere, segment_ray
                const float len = len3(dir);
                dir = mk3(dir.x / len, dir.y / len, dir.z / len);
                if (dot3(dir, nrm) < 0.0f) dir = neg3(dir);
                V3 o, d;
                float tnear, tfar;
                segment_ray(mk3(M.pos[p][0], M.pos[p][1], M.pos[p][2]), dir, R.maxd, o, d, tnear, tfar);
                const Slab slab = make_slab(o, d);
                const float iz = unpack2(slab.iz).x, oz = unpack2(slab.oz).x, az = unpack2(slab.az).x;
                const uint32_t own = M.own[p];
#pragma unroll 4
                for (int e = 0; e < nlist; e++) {
                    const float4 zc = M.zc[e];
                    if (slab1(M.xy[e], zc.x, zc.y, slab, iz, oz, az, tnear, tfar)) met |= 1u << e;
                }
                // a leaf that holds the lumel is met by every ray: look at its triangles
                for (uint32_t b = met & own; b; b &= b - 1) {
                    const int code = ~__float_as_int(M.zc[__ffs(b) - 1].z);
                    const int first = code >> 3, tris = (code & 7) + 1;
                    bool any = false;
                    for (int i = first; i < first + tris; i++) {
                        const float4* tp = s.tris + 3 * (size_t)i;
                        float t, u, v;
                        any |= tri_test(__ldg(tp), __ldg(tp + 1), __ldg(tp + 2), o, d, tnear, tfar, t, u, v);
                    }
                    if (!any) met ^= b & (0u - b);
                }
                if (kAny) {
                    if (met & own) {  // met already
                        atomicAdd(reinterpret_cast<int*>(&M.acc[p][0]), 1);
                        met = 0;
                    }
                } else if (met == 0) {
                    dir = shade(dir, nrm, -1, 0.f, 0.f);
                }
                M.v[0][r] = dir.x;
                M.v[1][r] = dir.y;
                M.v[2][r] = dir.z;
                M.mask[r] = met;
            }
            // rays that met several subtrees are walked first, so that the chunk does not end on them
            const bool heavy = __popc(met) > 2;
            const unsigned hv = __ballot_sync(kFull, heavy), lv = __ballot_sync(kFull, met != 0 && !heavy);
            if (heavy) M.queue[queued + __popc(hv & below)] = (uint8_t)r;
            else if (met) M.queue[light - 1 - __popc(lv & below)] = (uint8_t)r;
            queued += __popc(hv);
            light -= __popc(lv);
        }
        __syncwarp();
        // the queued rays' subtrees: entries [0, queued) and [light, kChunk)
        {
            const int waiting = queued + kChunk - light;
            Walk w;
            w.node = kNodeDone;
            w.sp = 0;
            int stack[kStackSize];
            int ray = -1, next = 0;
            for (;;) {
                const unsigned idle = __ballot_sync(kFull, w.node == kNodeDone);
                if (idle == kFull || (next < waiting && __popc(idle) >= refill)) {
                    if (w.node == kNodeDone) {
                        if (ray >= 0) {
                            const int p = lumel_of(ray);
                            if (kAny) {
                                if (w.gid >= 0) atomicAdd(reinterpret_cast<int*>(&M.acc[p][0]), 1);
                            } else {
                                const V3 c = shade(mk3(M.v[0][ray], M.v[1][ray], M.v[2][ray]),
                                                   mk3(M.nrm[p][0], M.nrm[p][1], M.nrm[p][2]), w.gid, w.hu, w.hv);
                                M.v[0][ray] = c.x;
                                M.v[1][ray] = c.y;
                                M.v[2][ray] = c.z;
                            }
                            ray = -1;
                        }
                        const int at = next + __popc(idle & below);
                        if (at < waiting) {
                            ray = M.queue[at < queued ? at : light + at - queued];
                            const int p = lumel_of(ray);
                            float tnear;
                            segment_ray(mk3(M.pos[p][0], M.pos[p][1], M.pos[p][2]),
                                        mk3(M.v[0][ray], M.v[1][ray], M.v[2][ray]), R.maxd, w.o, w.d, tnear, w.best);
                            w.slab = make_slab(w.o, w.d);
                            w.mask = M.mask[ray];
                            w.gid = -1;
                            w.sp = 0;
                            walk_pop(w, M, stack);
                        }
                    }
                    if (idle == kFull && next >= waiting) break;
                    next += __popc(idle);
                }
                // inner nodes, until none is left, many lanes wait at leaves or many for a ray
                for (;;) {
                    if (w.node >= 0) walk_node(s, w, M, stack, overflow);
                    if (w.node >= 0) walk_node(s, w, M, stack, overflow);
                    const int inner = __popc(__ballot_sync(kFull, w.node >= 0));
                    const int done = __popc(__ballot_sync(kFull, w.node == kNodeDone));
                    if (inner == 0 || (inner < 16 && 32 - inner - done >= 8) || (next < waiting && done >= refill)) break;
                }
                if (w.node >= 0 || w.node == kNodeDone) continue;
                const int code = ~w.node;
                const int first = code >> 3, tris = (code & 7) + 1;
                bool stop = false;
                for (int i = first; i < first + tris; i++) {
                    const float4* tp = s.tris + 3 * (size_t)i;
                    const float4 t0 = __ldg(tp), t1 = __ldg(tp + 1), t2 = __ldg(tp + 2);
                    float t, u, v;
                    // below best, which starts at the ray's end, or a tie with a smaller id
                    if (tri_test(t0, t1, t2, w.o, w.d, 0.01f, INFINITY, t, u, v) && t <= w.best) {
                        const int id = __float_as_int(t0.w);
                        if (t < w.best || (w.gid >= 0 && id < w.gid)) {
                            w.best = t;
                            w.gid = id;
                            w.hu = u;
                            w.hv = v;
                            if (kAny) { stop = true; break; }
                        }
                    }
                }
                if (stop) w.node = kNodeDone;
                else walk_pop(w, M, stack);
            }
        }
        __syncwarp();
        if (!kAny) {
            // each lumel's samples in order: one lane per lumel and channel
            const unsigned p = p0 + lane / 3;
            const int c = lane % 3;
            if (lane < 30 && p < (unsigned)lumels && p * S < base + n) {
                const int r0 = p * S > base ? (int)(p * S - base) : 0, r1 = (int)min((p + 1) * S - base, (unsigned)n);
                float sum = M.acc[p][c];
#pragma unroll 8
                for (int r = r0; r < r1; r++) sum = sum + M.v[c][r];
                M.acc[p][c] = sum;
            }
        }
        __syncwarp();
    }
}

// The valid lumels among the iteration's items [k0, k1) (at most kPatch) into
// M; lane l's item gives its lumel index i and its slot in M (-1: none).
template <bool kAny>
__device__ __forceinline__ int patch_load(PatchMem<kAny>& M, const DevMap& m, const Iter& it, long long k0,
                                          long long k1, long long& i, int& slot) {
    const int lane = threadIdx.x & 31;
    const bool valid = k0 + lane < k1 && iter_lumel(m, it, k0 + lane, i);
    const unsigned vote = __ballot_sync(kFull, valid);
    slot = -1;
    if (valid) {
        slot = __popc(vote & ((1u << lane) - 1u));
        const V3 p = ld3(m.position + 3 * i), n = ld3(m.normal + 3 * i);
        M.pos[slot][0] = p.x; M.pos[slot][1] = p.y; M.pos[slot][2] = p.z;
        M.nrm[slot][0] = n.x; M.nrm[slot][1] = n.y; M.nrm[slot][2] = n.z;
        M.item[slot] = (uint32_t)i;
    }
    __syncwarp();
    return __popc(vote);
}

}  // namespace rl
