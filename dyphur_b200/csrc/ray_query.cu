// Queries over the frame's products: batched ray casts against the LBVH and
// the per-shape contact filter.
//
//   dyph_ray_query      ray_query (core/src/ray_query.cpp:126-195): closest
//                       hit of each ray, LBVH walk over the fp16 node boxes,
//                       exact sphere / oriented-box test at the leaves.
//   dyph_contact_sensor ContactSensor::query (core/src/contact_sensor.cpp:6-59):
//                       the contacts whose body a or b has a given shape, in
//                       store order. The filter runs on the device (one pass,
//                       tile look-back compaction) and only the matches cross
//                       to the host.
//
// The ray walk keeps the reference's visiting order (a 64-entry stack, right
// child pushed before left, node box tested when popped) and its float
// expressions, so hits and tie-breaks are identical, not just close. In trees of
// some size it finds a bound on the hit first and then follows that order only
// among the leaves that can matter (ray_walk_kernel).
#include <algorithm>
#include <mutex>
#include <new>

#include "internal.cuh"

namespace dyph {
namespace {

constexpr int kRayThreads = 128;
constexpr int kRayStack = 64;  // ray_query.cpp:173

// Slab test against a node box (ray_query.cpp:14-33); tmin is where the ray
// enters it.
__device__ __forceinline__ bool ray_node_hit(float ox, float oy, float oz, float ix, float iy, float iz,
                                             float mnx, float mny, float mnz, float mxx, float mxy, float mxz,
                                             float best_t, float& tmin) {
    const float t1x = (mnx - ox) * ix, t2x = (mxx - ox) * ix;
    const float t1y = (mny - oy) * iy, t2y = (mxy - oy) * iy;
    const float t1z = (mnz - oz) * iz, t2z = (mxz - oz) * iz;
    tmin = t1x < t2x ? t1x : t2x;
    float tmax = t1x < t2x ? t2x : t1x;
    const float ylo = t1y < t2y ? t1y : t2y, yhi = t1y < t2y ? t2y : t1y;
    tmin = tmin > ylo ? tmin : ylo;
    tmax = tmax < yhi ? tmax : yhi;
    const float zlo = t1z < t2z ? t1z : t2z, zhi = t1z < t2z ? t2z : t1z;
    tmin = tmin > zlo ? tmin : zlo;
    tmax = tmax < zhi ? tmax : zhi;
    return tmax >= 0.f && tmax >= tmin && tmin < best_t;
}

// v rotated by the conjugate of (w, x, y, z): t = 2 (u x v), v + w t + u x t
// with u = (-x, -y, -z) (Quat::rotate, core/include/core/math/quat.hpp:39-42).
__device__ __forceinline__ void rotate_conj(float w, float x, float y, float z, float vx, float vy, float vz,
                                            float& rx, float& ry, float& rz) {
    const float ux = -x, uy = -y, uz = -z;
    const float tx = (uy * vz - uz * vy) * 2.f;
    const float ty = (uz * vx - ux * vz) * 2.f;
    const float tz = (ux * vy - uy * vx) * 2.f;
    rx = (vx + tx * w) + (uy * tz - uz * ty);
    ry = (vy + ty * w) + (uz * tx - ux * tz);
    rz = (vz + tz * w) + (ux * ty - uy * tx);
}

// Oriented box in the body frame; t or -1 (ray_query.cpp:37-73).
__device__ __forceinline__ float ray_box(float ox, float oy, float oz, float dx, float dy, float dz, float px,
                                         float py, float pz, float qw, float qx, float qy, float qz, float hx,
                                         float hy, float hz, float best_t) {
    float lox, loy, loz, ldx, ldy, ldz;
    rotate_conj(qw, qx, qy, qz, ox - px, oy - py, oz - pz, lox, loy, loz);
    rotate_conj(qw, qx, qy, qz, dx, dy, dz, ldx, ldy, ldz);
    const float ix = 1.f / ldx, iy = 1.f / ldy, iz = 1.f / ldz;
    const float t1x = (-hx - lox) * ix, t2x = (hx - lox) * ix;
    const float t1y = (-hy - loy) * iy, t2y = (hy - loy) * iy;
    const float t1z = (-hz - loz) * iz, t2z = (hz - loz) * iz;
    float tmin = t1x < t2x ? t1x : t2x;
    float tmax = t1x < t2x ? t2x : t1x;
    const float ylo = t1y < t2y ? t1y : t2y, yhi = t1y < t2y ? t2y : t1y;
    tmin = tmin > ylo ? tmin : ylo;
    tmax = tmax < yhi ? tmax : yhi;
    const float zlo = t1z < t2z ? t1z : t2z, zhi = t1z < t2z ? t2z : t1z;
    tmin = tmin > zlo ? tmin : zlo;
    tmax = tmax < zhi ? tmax : zhi;
    if (tmax < 0.f || tmin > tmax) return -1.f;
    const float t = tmin >= 0.f ? tmin : tmax;
    return (t >= 0.f && t < best_t) ? t : -1.f;
}

// Sphere by the quadratic; t or -1 (ray_query.cpp:76-91).
__device__ __forceinline__ float ray_sphere(float ox, float oy, float oz, float dx, float dy, float dz, float cx,
                                            float cy, float cz, float r, float best_t) {
    const float ocx = ox - cx, ocy = oy - cy, ocz = oz - cz;
    const float a = dx * dx + dy * dy + dz * dz;
    const float b = dx * ocx + dy * ocy + dz * ocz;
    const float c = ocx * ocx + ocy * ocy + ocz * ocz - r * r;
    const float disc = b * b - a * c;
    if (disc < 0.f) return -1.f;
    const float sq = __fsqrt_rn(disc);
    float t = (-b - sq) / a;
    if (t < 0.f) t = (-b + sq) / a;
    return (t >= 0.f && t < best_t) ? t : -1.f;
}

struct RayScene {
    dyph_bodies b;
    dyph_shapes sh;
};

__device__ __forceinline__ void ray_leaf(const RayScene& S, uint32_t bi, const dyph_ray& r, float& best_t,
                                         uint32_t& best_body) {
    const uint32_t shape = __ldg(&S.b.shape[bi]);
    const float hx = __ldg(&S.sh.half_x[shape]);
    float t;
    if (__ldg(&S.sh.type[shape]) == kShapeSphere) {
        t = ray_sphere(r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, S.b.pos_x[bi], S.b.pos_y[bi], S.b.pos_z[bi], hx, best_t);
    } else {
        // Every other shape type is cast as its box (ray_query.cpp:113-118).
        t = ray_box(r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, S.b.pos_x[bi], S.b.pos_y[bi], S.b.pos_z[bi], S.b.rot_w[bi],
                    S.b.rot_x[bi], S.b.rot_y[bi], S.b.rot_z[bi], hx, __ldg(&S.sh.half_y[shape]),
                    __ldg(&S.sh.half_z[shape]), best_t);
    }
    if (t >= 0.f) {
        best_t = t;
        best_body = bi;
    }
}

// The slab test against the six fp16 bounds of a NodeBox.
__device__ __forceinline__ bool ray_box_hit(const dyph_ray& r, float ix, float iy, float iz, const uint4& nb,
                                            float best_t, float& tmin) {
    return ray_node_hit(r.ox, r.oy, r.oz, ix, iy, iz, h2f_bits(nb.x & 0xFFFFu), h2f_bits(nb.x >> 16),
                        h2f_bits(nb.y & 0xFFFFu), h2f_bits(nb.y >> 16), h2f_bits(nb.z & 0xFFFFu),
                        h2f_bits(nb.z >> 16), best_t, tmin);
}

__global__ void __launch_bounds__(kRayThreads) ray_query_kernel(dyph_bvh_view bvh, RayScene S,
                                                                const dyph_ray* __restrict__ rays,
                                                                dyph_ray_hit* __restrict__ hits, uint32_t n_rays) {
    const uint32_t idx = blockIdx.x * kRayThreads + threadIdx.x;
    if (idx >= n_rays) return;
    const dyph_ray r = rays[idx];
    float best_t = r.t_max;
    uint32_t best_body = 0xFFFFFFFFu;
    const float ix = 1.f / r.dx, iy = 1.f / r.dy, iz = 1.f / r.dz;
    if (bvh.n == 1u) {
        // A one-body build has no tree (broadphase.cpp returns early): body 0.
        ray_leaf(S, 0u, r, best_t, best_body);
    } else if (bvh.n > 1u) {
        int32_t stack[kRayStack];
        int top = 0;
        stack[top++] = __ldg(bvh.root);
        const int32_t n_int = static_cast<int32_t>(bvh.n - 1u);
        const uint4* boxes = reinterpret_cast<const uint4*>(bvh.aabb);
        while (top > 0) {
            const int32_t node = stack[--top];
            float tmin;
            if (!ray_box_hit(r, ix, iy, iz, __ldg(&boxes[node]), best_t, tmin)) continue;
            if (node >= n_int) {
                ray_leaf(S, __ldg(&bvh.sorted_idx[node - n_int]), r, best_t, best_body);
            } else if (top + 1 < kRayStack) {
                stack[top++] = __ldg(&bvh.right[node]);
                stack[top++] = __ldg(&bvh.left[node]);
            }
        }
    }
    hits[idx] = dyph_ray_hit{best_t, best_body};
}

// ── the closest hit first ────────────────────────────────────────────────────
// The reference's walk visits the tree in leaf order and so passes most of a
// long ray's leaves before the near ones. Its result is a fold over the leaves
// in that order, best = t_max at first: leaf k is taken when its box test passes
// with an entry point m_k < best (its ancestors' tests then pass too: their boxes
// contain its box exactly and every operation of the slab test is monotone), and
// then best = t_k if t_k < best. For any leaf best ends at or below
// max(t_k, m_k), so a walk that goes to the nearer child first finds a bound U on
// the result quickly. With W >= U such that t_k <= W implies m_k <= W, leaves
// with t_k > W do not change the result: while best > W a leaf with t_k <= W is
// always taken, and afterwards t_k > W >= best is not. A second walk, in leaf
// order, therefore folds only the leaves with t_k <= W; it starts at W = U and
// begins again with W = m_k in the rare case that it meets one past W (the boxes
// are rounded to fp16 and may cut a body).
// The second walk needs a lower bound on t_k <= W at every node: the entry point
// into the node's box widened so far that it holds every point o + t_k d that the
// leaf tests can return. Such a point is at most L = W |d| from the origin o. The
// box test's lies within 5e-5 (L + size) of the body's box (rounding of rotation
// and slabs, quaternions within 1e-5 of unit length), the sphere test's within
// min(sqrt(20 eps) (L + 2 r), 10 eps (L + 2 r)^2 / r) of the sphere (the quadratic's
// cancellation). A leaf box holds its body's to within fp16 rounding, 2^-11 of
// each bound, and within the body's movement since the tree was built (a solve
// moves bodies). So each bound is widened by 5e-4 of itself and by the largest
// movement, with the terms in the bodies' sizes, over all leaves, found with the
// records, + 1e-4 L + min(2.5e-3 L, 1.5e-6 L^2 / the smallest sphere's radius).
// A body beyond fp16's range, as a pile that bursts throws out, has a leaf box
// that starts at +infinity or ends at -infinity on some axis: its entry point is
// infinite or behind the ray, so no ray with a finite t_max ever tests it.
// Rays with a zero or non-finite component, trees or bodies outside these
// assumptions, folds of more than kRayFoldSteps nodes (margins far beyond the
// leaves' sizes) and walks that reach the reference's stack limit take the
// reference's walk as it is (in_order).
//
// Records of the tree and its bodies, 16-byte words:
//   nodes  two per internal node, one sector: the left child's box and index,
//          the right child's box and index;
//   leaves four per leaf, in leaf order: position and body, rotation, half
//          extents and shape type, leaf box.
struct RayRecords {
    uint4* nodes;
    uint4* leaves;
    // [0] largest excess (float bits), [1] 1 when the tree or a body is outside the
    // assumptions, [2] complement of the smallest sphere radius's bits (0: no sphere),
    // [3] leaf boxes out of every finite ray's reach, [4] the bodies' hx + hy + hz
    // summed (float)
    uint32_t* words;
};
constexpr size_t kRayWords = 8;

// A tree of fewer bodies is walked as it is, and so is one by few rays, fewer than
// kRayRecordsWork over its bodies (8 into 16,384, 2 into 65,536): the scratch and two
// more launches cost 8 us at 16,385 bodies and 20 at 65,537 (a query whose rays all
// miss the pile at once, of 64 or 65,536 rays: 52 and 73, 60 and 94 us). The walk in
// leaf order and this one, in us by rays (random through the whole pile; short ones,
// three body lengths; downwards from 3 m above a body; a camera's) and bodies:
//            1 ray    4       8       64         4,096      65,536      a million
//   random   88>80    141>135 175>195 378>306    564>293    654>383     3,082>2,867  16,385 bodies
//            71>73    333>127 361>155 1,113>297  1,476>434  1,848>486   8,719>2,937  65,537
//   short    36>48    63>62   80>74   120>101    162>109    189>114       909>667    16,385
//            64>68    104>93  147>124 267>190    339>211    383>215     2,028>1,434  65,537
//   down     56>59    72>69   94>84   150>111    185>114    209>120     1,105>757    16,385
//            113>103  147>118 203>152 332>212    414>227    457>242     2,752>1,697  65,537
//   camera   37>47    49>56   49>58   186>148    224>148    257>204     1,282>1,091  16,385
// and at 8,193 bodies a million random rays took 1,852 and 2,474 us.
constexpr uint32_t kRayRecordsBodies = 16384;
constexpr uint64_t kRayRecordsWork = 1u << 17;  // rays times bodies
// Nodes that a ray visits in leaf order before it looks for a bound first. Leaf
// order is Morton order, which ascends in every coordinate: the more a ray does,
// the nearer it comes to meeting the near leaves first anyway. A million rays, random
// (up, across and down that order) and a camera's (across), into 16,385 bodies, and
// into the burst pile of 65,537:
//   384/96/24 2,804, 1,307 and 7,870 us; half of each 2,715, 1,804 and 7,110; twice
//   each 2,939, 1,046 and 7,730; 576 or 768 up as 384; across 192 2,891, 1,040 and
//   7,950; across 128 2,867, 1,091 and 7,870.
__device__ __forceinline__ uint32_t ray_steps(const dyph_ray& r) {
    const float s = (r.dx + r.dy + r.dz) / (fabsf(r.dx) + fabsf(r.dy) + fabsf(r.dz));
    return s > 0.25f ? 384u : (s > -0.25f ? 128u : 24u);
}
// A ray no longer than this many of the bodies' mean hx + hy + hz goes in leaf order
// to its end: few leaves lie along it, and the bound and the fold would each visit
// most of them again. A million short rays as above, all of them to the end and by
// steps: 667 and 1,315 us into 16,385 bodies, 1,434 and 2,443 into 65,537; with 10 in
// place of 16 the rays downwards (12 long) took 1,241 and 1,689 instead of 752 and 1,694.
constexpr float kRayShort = 16.f;

// The node index and the height of the reference's stack share a stack word.
constexpr uint32_t kRayNodeBits = 26;
constexpr uint32_t kRayMaxBodies = 1u << (kRayNodeBits - 1);  // nodes 0 .. 2 n - 2
constexpr uint32_t kRayNone = 0xFFFFFFFFu, kRayNodeMask = (1u << kRayNodeBits) - 1u;

// A ray past far bodies has a margin that grows with its length. A million rays
// into a pile that has thrown 10 % of its bodies 100 to 1e10 away: 8.6 ms with
// 128 steps, 7.8 with 512, 9.4 with 4096 (8.5 in leaf order alone).
constexpr uint32_t kRayFoldSteps = 512;

// A bound v moved by c of its magnitude (an infinite one stays). The margins are
// taken with fp16's 2^-11 and a little more, the fold's boxes with more still,
// which covers the rounding of far bodies' bounds.
constexpr float kRayHalf = 4.95e-4f, kRayWide = 5e-4f;
__device__ __forceinline__ float widen(float v, float c) { return v + c * fminf(fabsf(v), 1e5f); }
// Whether the box test never passes for a finite t_max, whatever the direction.
__device__ __forceinline__ bool out_of_reach(const BoxF& f) {
    return fmaxf(fmaxf(f.mnx, f.mny), f.mnz) == INFINITY || fminf(fminf(f.mxx, f.mxy), f.mxz) == -INFINITY;
}

__device__ __forceinline__ bool box_holds(const BoxF& a, const BoxF& b) {
    return a.mnx <= b.mnx && a.mny <= b.mny && a.mnz <= b.mnz && a.mxx >= b.mxx && a.mxy >= b.mxy && a.mxz >= b.mxz;
}

__global__ void __launch_bounds__(256) ray_records_kernel(dyph_bvh_view bvh, RayScene S, RayRecords R) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint4* boxes = reinterpret_cast<const uint4*>(bvh.aabb);
    float excess = 0.f, extent = 0.f;
    uint32_t small = 0u;
    bool odd = false, away = false;
    if (i < bvh.n) {
        if (i + 1u < bvh.n) {
            const int32_t l = bvh.left[i], r = bvh.right[i];
            uint4 lb = boxes[l], rb = boxes[r];
            const BoxF own = unpack_box(boxes[i]);
            odd = !box_holds(own, unpack_box(lb)) || !box_holds(own, unpack_box(rb));
            lb.w = static_cast<uint32_t>(l);
            rb.w = static_cast<uint32_t>(r);
            R.nodes[2ull * i] = lb;
            R.nodes[2ull * i + 1] = rb;
        }
        const uint32_t b = bvh.sorted_idx[i], sh = S.b.shape[b], type = S.sh.type[sh];
        const uint4 box = boxes[bvh.n - 1u + i];
        auto bits = [](float x) { return __float_as_uint(x); };
        const float px = S.b.pos_x[b], py = S.b.pos_y[b], pz = S.b.pos_z[b];
        const float qw = S.b.rot_w[b], qx = S.b.rot_x[b], qy = S.b.rot_y[b], qz = S.b.rot_z[b];
        const float hx = S.sh.half_x[sh], hy = S.sh.half_y[sh], hz = S.sh.half_z[sh];
        R.leaves[4ull * i] = make_uint4(bits(px), bits(py), bits(pz), b);
        R.leaves[4ull * i + 1] = make_uint4(bits(qw), bits(qx), bits(qy), bits(qz));
        R.leaves[4ull * i + 2] = make_uint4(bits(hx), bits(hy), bits(hz), type);
        R.leaves[4ull * i + 3] = box;
        const BoxF f = unpack_box(box);
        odd = odd || isnan(f.mnx) || isnan(f.mny) || isnan(f.mnz) || isnan(f.mxx) || isnan(f.mxy) || isnan(f.mxz);
        away = !odd && out_of_reach(f);
        if (!away) {
            // how far the body's present box leaves its leaf box
            float ex = hx, ey = hx, ez = hx;
            if (type != kShapeSphere) {
                ex = fabsf(1.f - 2.f * (qy * qy + qz * qz)) * hx + fabsf(2.f * (qx * qy - qz * qw)) * hy +
                     fabsf(2.f * (qx * qz + qy * qw)) * hz;
                ey = fabsf(2.f * (qx * qy + qz * qw)) * hx + fabsf(1.f - 2.f * (qx * qx + qz * qz)) * hy +
                     fabsf(2.f * (qy * qz - qx * qw)) * hz;
                ez = fabsf(2.f * (qx * qz - qy * qw)) * hx + fabsf(2.f * (qy * qz + qx * qw)) * hy +
                     fabsf(1.f - 2.f * (qx * qx + qy * qy)) * hz;
                const float q2 = qw * qw + qx * qx + qy * qy + qz * qz;
                odd = odd || !(fabsf(q2 - 1.f) <= 1e-5f) || !(hy >= 0.f) || !(hz >= 0.f);
            }
            const float over = fmaxf(
                fmaxf(fmaxf(widen(f.mnx, -kRayHalf) - (px - ex), (px + ex) - widen(f.mxx, kRayHalf)),
                      fmaxf(widen(f.mny, -kRayHalf) - (py - ey), (py + ey) - widen(f.mxy, kRayHalf))),
                fmaxf(widen(f.mnz, -kRayHalf) - (pz - ez), (pz + ez) - widen(f.mxz, kRayHalf)));
            // the sums above round: 1e-5 of the extents and of the excess, and of the
            // bounds what kRayWide leaves; and the leaf tests' terms in the size
            const float size = type == kShapeSphere ? 5e-3f * hx : 1e-4f * (hx + hy + hz);
            excess = 1.00001f * fmaxf(over, 0.f) + 1e-5f * (ex + ey + ez) + size + 1e-6f;
            extent = fminf(type == kShapeSphere ? 3.f * hx : hx + hy + hz, 1e6f);
            if (type == kShapeSphere) small = ~bits(fabsf(hx));
            odd = odd || !(hx >= 0.f) || !isfinite(fabsf(px) + fabsf(py) + fabsf(pz) + ex + ey + ez) ||
                  !(excess < 1e6f);
        }
    }
    const uint32_t e = __reduce_max_sync(0xffffffffu, odd ? 0u : __float_as_uint(excess));
    const bool any_odd = __any_sync(0xffffffffu, odd);
    const uint32_t n_away = __popc(__ballot_sync(0xffffffffu, away));
    small = __reduce_max_sync(0xffffffffu, small);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) extent += __shfl_xor_sync(0xffffffffu, extent, d);
    if ((threadIdx.x & 31u) == 0u) {
        if (small) atomicMax(&R.words[2], small);
        if (e) atomicMax(&R.words[0], e);
        if (any_odd) R.words[1] = 1u;
        if (n_away) atomicAdd(&R.words[3], n_away);
        atomicAdd(reinterpret_cast<float*>(&R.words[4]), extent);  // (a rounded sum only moves the rule's line)
    }
}

// One ray's walks over the records.
struct RayWalk {
    const dyph_bvh_view& bvh;
    const RayRecords& R;
    const dyph_ray& r;
    float ix, iy, iz;
    uint2* stack;  // [kRayStack] node | height << kRayNodeBits (of the reference's stack under the node), entry point
    float best_t;
    uint32_t best_body;
    bool deep;  // met the reference's stack limit, or the fold's own

    __device__ __forceinline__ bool box(const uint4& b, float best, float& tmin) const {
        return ray_box_hit(r, ix, iy, iz, b, best, tmin);
    }
    // t of a leaf if it is below `best`, else negative
    __device__ __forceinline__ float leaf(const uint4* l, float best, uint32_t& body) const {
        const uint4 p = __ldg(l), q = __ldg(l + 1), h = __ldg(l + 2);
        auto f = [](uint32_t x) { return __uint_as_float(x); };
        body = p.w;
        return h.w == kShapeSphere
                   ? ray_sphere(r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, f(p.x), f(p.y), f(p.z), f(h.x), best)
                   : ray_box(r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, f(p.x), f(p.y), f(p.z), f(q.x), f(q.y), f(q.z),
                             f(q.w), f(h.x), f(h.y), f(h.z), best);
    }
    // Whether the ray meets box b, widened by m (lo = o + m, hi = o - m), at or
    // before `most`; tlow: where it enters.
    __device__ __forceinline__ bool wide_box(const uint4& b, const float lo[3], const float hi[3], float most,
                                             float& tlow) const {
        const BoxF f = unpack_box(b);
        const float t1x = (widen(f.mnx, -kRayWide) - lo[0]) * ix, t2x = (widen(f.mxx, kRayWide) - hi[0]) * ix;
        const float t1y = (widen(f.mny, -kRayWide) - lo[1]) * iy, t2y = (widen(f.mxy, kRayWide) - hi[1]) * iy;
        const float t1z = (widen(f.mnz, -kRayWide) - lo[2]) * iz, t2z = (widen(f.mxz, kRayWide) - hi[2]) * iz;
        tlow = fmaxf(fmaxf(fminf(t1x, t2x), fminf(t1y, t2y)), fminf(t1z, t2z));
        const float thigh = fminf(fminf(fmaxf(t1x, t2x), fmaxf(t1y, t2y)), fmaxf(t1z, t2z));
        return thigh >= 0.f && thigh >= tlow && tlow <= most;
    }
    // A walk from `root`, of two children to the nearer or to the left one first:
    // test(box, entry) says whether a child is gone into, leaf_fn(leaf, entry) ends
    // the walk with true, keep(entry) whether a waiting node still is when its turn
    // comes. False when `steps` nodes did not end it.
    template <bool kNearFirst, class Test, class Leaf, class Keep>
    __device__ __forceinline__ bool walk(uint32_t root, float entry, uint32_t steps, Test&& test, Leaf&& leaf_fn,
                                         Keep&& keep) {
        const uint32_t n_int = bvh.n - 1u;
        uint32_t height = 0, node = root;
        int top = 0;
        while (true) {
            if (steps-- == 0u) return false;
            bool next = true;
            if (node < n_int) {
                const uint4 lb = __ldg(&R.nodes[2ull * node]), rb = __ldg(&R.nodes[2ull * node + 1]);
                float lt, rt;
                const bool room = height + 1u < static_cast<uint32_t>(kRayStack);
                deep = deep || !room;
                const bool lh = test(lb, lt) && room, rh = test(rb, rt) && room;
                if (lh || rh) {
                    const bool left = lh && (!kNearFirst || !rh || lt <= rt);
                    if (lh && rh)
                        stack[top++] = left ? make_uint2(rb.w | (height << kRayNodeBits), __float_as_uint(rt))
                                            : make_uint2(lb.w | ((height + 1u) << kRayNodeBits), __float_as_uint(lt));
                    node = left ? lb.w : rb.w;
                    entry = left ? lt : rt;
                    height += left ? 1u : 0u;
                    next = false;
                }
            } else if (leaf_fn(R.leaves + 4ull * (node - n_int), entry)) {
                return true;
            }
            while (next) {
                if (top == 0) return true;
                const uint2 e = stack[--top];
                entry = __uint_as_float(e.y);
                node = e.x & kRayNodeMask;
                height = e.x >> kRayNodeBits;
                next = !keep(entry);
            }
        }
    }

    // The reference's walk (ray_query_kernel), both children tested in one step:
    // a box test depends on the closest hit so far only through "enters before
    // it", which is tested again when the node's turn comes. False when it is not
    // done after `steps` nodes; best_t bounds the result from above then too.
    __device__ __forceinline__ bool in_order(uint32_t root, uint32_t steps) {
        best_t = r.t_max;
        best_body = kRayNone;
        float tmin;
        if (!box(__ldg(reinterpret_cast<const uint4*>(bvh.aabb) + root), best_t, tmin)) return true;
        return walk<false>(
            root, tmin, steps, [&](const uint4& b, float& t) { return box(b, best_t, t); },
            [&](const uint4* l, float) {
                uint32_t body;
                const float t = leaf(l, best_t, body);
                if (t >= 0.f) {
                    best_t = t;
                    best_body = body;
                }
                return false;
            },
            [&](float entry) { return entry < best_t; });
    }

    // A bound on the result that is at most U, nearer children first; U when
    // nothing below it is hit.
    __device__ __forceinline__ float bound(uint32_t root, float U) {
        float tmin;
        if (!box(__ldg(reinterpret_cast<const uint4*>(bvh.aabb) + root), U, tmin)) return U;
        walk<true>(
            root, tmin, ~0u, [&](const uint4& b, float& t) { return box(b, U, t); },
            [&](const uint4* l, float entry) {
                uint32_t body;
                const float t = leaf(l, U, body);
                if (t >= 0.f) U = fminf(U, fmaxf(t, entry));
                return false;
            },
            [&](float entry) { return entry < U; });
        return U;
    }

    // The fold over the leaves with t <= W in leaf order; returns W, or a larger
    // bound with which to begin again.
    __device__ __forceinline__ float fold(uint32_t root, float W, float slack, float inv_radius, float length) {
        const float past = nextafterf(W, INFINITY);  // t < past: t <= W
        const float L = W * length;
        const float m = slack + 1e-4f * L + fminf(2.5e-3f * L, 1.5e-6f * L * L * inv_radius);
        const float lo[3] = {r.ox + m, r.oy + m, r.oz + m}, hi[3] = {r.ox - m, r.oy - m, r.oz - m};
        float again = W;
        best_t = r.t_max;
        best_body = kRayNone;
        const bool ended = walk<false>(
            root, 0.f, kRayFoldSteps, [&](const uint4& b, float& t) { return wide_box(b, lo, hi, fminf(W, best_t), t); },
            [&](const uint4* l, float) {
                float tmin;
                if (!box(__ldg(l + 3), INFINITY, tmin)) return false;
                uint32_t body;
                const float t = leaf(l, fminf(past, best_t), body);
                if (!(t >= 0.f)) return false;
                if (tmin > W && best_t > W) {
                    again = tmin;
                    return true;
                }
                if (tmin < best_t) {
                    best_t = t;
                    best_body = body;
                }
                return false;
            },
            [&](float entry) { return entry <= fminf(W, best_t); });
        deep = deep || !ended;
        return again;
    }
};

// One thread per ray: ray_steps nodes of the reference's walk, which end most
// rays whose leaf order happens to be near first, then the bound and the fold.
// Bound by the latency of dependent loads in divergent lanes.
__global__ void __launch_bounds__(kRayThreads) ray_walk_kernel(dyph_bvh_view bvh, RayRecords R,
                                                               const dyph_ray* __restrict__ rays,
                                                               dyph_ray_hit* __restrict__ hits, uint32_t n_rays) {
    const uint32_t idx = blockIdx.x * kRayThreads + threadIdx.x;
    if (idx >= n_rays) return;
    const dyph_ray r = rays[idx];
    const uint32_t root = static_cast<uint32_t>(__ldg(bvh.root));
    uint2 stack[kRayStack];
    RayWalk w{bvh, R, r, 1.f / r.dx, 1.f / r.dy, 1.f / r.dz, stack};
    w.deep = false;
    const float d2 = r.dx * r.dx + r.dy * r.dy + r.dz * r.dz;
    const bool plain = R.words[1] != 0u || !isfinite(fabsf(r.ox) + fabsf(r.oy) + fabsf(r.oz)) ||
                       !isfinite(fabsf(w.ix) + fabsf(w.iy) + fabsf(w.iz)) || !(d2 > 1e-20f && d2 < 1e20f) ||
                       !(r.t_max > 0.f) || (R.words[3] != 0u && !isfinite(r.t_max));
    const float length = __fsqrt_rn(d2);
    const bool near = r.t_max * length * static_cast<float>(bvh.n) <= kRayShort * __uint_as_float(R.words[4]);
    if (!w.in_order(root, plain || near ? ~0u : ray_steps(r))) {
        float W = w.bound(root, w.best_t);
        bool done = !w.deep && W == r.t_max;  // nothing is entered and hit before t_max
        if (done) {
            w.best_t = r.t_max;
            w.best_body = kRayNone;
        }
        const float slack = __uint_as_float(R.words[0]);
        const uint32_t small = R.words[2];
        const float inv_radius = small ? 1.f / __uint_as_float(~small) : 0.f;
        for (int k = 0; k < 8 && !done && !w.deep; ++k) {
            const float W1 = w.fold(root, W, slack, inv_radius, length);
            done = W1 == W;
            W = W1;
        }
        if (!done || w.deep) w.in_order(root, ~0u);
    }
    hits[idx] = dyph_ray_hit{w.best_t, w.best_body};
}

// Stream-ordered scratch of the queries: a pool of its own per device that
// keeps at most kRayPoolKeep bytes between calls. Calls on any streams and
// threads take and return blocks through it.
constexpr int kRayMaxDevices = 64;
constexpr uint64_t kRayPoolKeep = 64ull << 20;
std::mutex g_ray_pool_mu;
cudaMemPool_t g_ray_pool[kRayMaxDevices] = {};

cudaMemPool_t ray_pool() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kRayMaxDevices) return nullptr;
    std::lock_guard<std::mutex> lock(g_ray_pool_mu);
    if (!g_ray_pool[dev]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        uint64_t keep = kRayPoolKeep;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) return nullptr;
        if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
            cudaMemPoolDestroy(pool);
            return nullptr;
        }
        g_ray_pool[dev] = pool;
    }
    return g_ray_pool[dev];
}

// A captured query takes no scratch: it would put an allocation into the caller's
// graph, which could then be instantiated only once at a time and not become part of
// another graph. A million random rays into a settled 65,537-body pile take 8.7 ms so
// instead of 2.9.
bool capturing(cudaStream_t s) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &status) == cudaSuccess) return status != cudaStreamCaptureStatusNone;
    cudaGetLastError();
    return true;
}

// ── contact sensor ──────────────────────────────────────────────────────────

constexpr int kSensorThreads = 256;
constexpr int kSensorRows = 9;  // body_a, body_b, pos xyz, normal xyz, depth

__global__ void __launch_bounds__(kSensorThreads) sensor_filter_kernel(dyph_contacts in,
                                                                       const uint32_t* __restrict__ body_shape,
                                                                       uint32_t n_bodies, uint32_t shape_idx,
                                                                       uint32_t* __restrict__ out, uint32_t cap,
                                                                       uint32_t* __restrict__ counts,
                                                                       uint32_t* __restrict__ status) {
    __shared__ uint32_t s_tile, s_excl;
    __shared__ uint32_t s_scan[kSensorThreads / 32];
    const uint32_t nc = min(*in.n, in.capacity);
    const uint32_t n_tiles = (nc + kSensorThreads - 1) / kSensorThreads;
    if (nc == 0u) {
        if (blockIdx.x == 0 && threadIdx.x == 0) counts[0] = 0u;
        return;
    }
    while (true) {
        if (threadIdx.x == 0) s_tile = atomicAdd(&counts[1], 1u);
        __syncthreads();
        const uint32_t tile = s_tile;
        if (tile >= n_tiles) break;
        const uint32_t i = tile * kSensorThreads + threadIdx.x;
        bool keep = false;
        uint32_t a = 0, b = 0;
        if (i < nc) {
            a = in.body_a[i];
            b = in.body_b[i];
            keep = (a < n_bodies && __ldg(&body_shape[a]) == shape_idx) ||
                   (b < n_bodies && __ldg(&body_shape[b]) == shape_idx);
        }
        uint32_t total;
        const uint32_t excl = block_exclusive_scan<kSensorThreads>(keep ? 1u : 0u, s_scan, total);
        if (threadIdx.x < 32) {
            const uint32_t e = lookback_warp(status, tile, total);
            if (threadIdx.x == 0) {
                s_excl = e;
                if (tile == n_tiles - 1) counts[0] = e + total;
            }
        }
        __syncthreads();
        if (keep) {
            const uint32_t pos = s_excl + excl;
            if (pos < cap) {
                const float row[7] = {in.pos_x[i], in.pos_y[i], in.pos_z[i], in.norm_x[i],
                                      in.norm_y[i], in.norm_z[i], in.depth[i]};
                out[pos] = a;
                out[static_cast<size_t>(cap) + pos] = b;
#pragma unroll
                for (int k = 0; k < 7; ++k) out[static_cast<size_t>(2 + k) * cap + pos] = __float_as_uint(row[k]);
            }
        }
        __syncthreads();
    }
}

int sensor_blocks() {
    static int blocks = 0;
    if (blocks == 0) {
        int dev = 0, sms = 148, per_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sensor_filter_kernel, kSensorThreads, 0);
        blocks = sms * std::max(1, std::min(per_sm, 8));
    }
    return blocks;
}

}  // namespace
}  // namespace dyph

struct dyph_contact_sensor {
    uint32_t shape_idx = 0;
    uint32_t cap = 0;             // rows of the device and host match buffers
    uint32_t* d_rows = nullptr;   // [9][cap] matches in store order
    uint32_t* counts = nullptr;   // [0] matches, [1] tile counter
    uint32_t* status = nullptr;   // look-back status per 256-contact tile
    uint32_t status_words = 0;
    uint32_t* h_rows = nullptr;   // pinned host copy of the matches
    uint32_t count = 0;           // matches of the last query
};

using namespace dyph;

extern "C" dyph_status dyph_ray_query(const dyph_bvh_view* bvh, const dyph_bodies* bodies, const dyph_shapes* shapes,
                                      const dyph_ray* d_rays, dyph_ray_hit* d_hits, uint32_t n_rays, dyph_stream s) {
    if (n_rays == 0) return DYPH_OK;
    if (!bvh || !bodies || !shapes || !d_rays || !d_hits) return DYPH_ERR_INVALID;
    if (bvh->n > 1u && (!bvh->root || !bvh->left || !bvh->right || !bvh->sorted_idx || !bvh->aabb))
        return DYPH_ERR_INVALID;
    if (bvh->n > bodies->n) return DYPH_ERR_INVALID;
    const uint32_t grid = (n_rays + kRayThreads - 1) / kRayThreads;
    cudaStream_t cs = reinterpret_cast<cudaStream_t>(s);
    if (bvh->n >= kRayRecordsBodies && bvh->n <= kRayMaxBodies &&
        static_cast<uint64_t>(n_rays) * bvh->n >= kRayRecordsWork && !capturing(cs)) {
        const RelaxedCapture relaxed;
        const size_t node_bytes = 32ull * bvh->n, leaf_bytes = 64ull * bvh->n;
        void* ws = nullptr;
        cudaMemPool_t pool = ray_pool();
        if (pool && cudaMallocFromPoolAsync(&ws, node_bytes + leaf_bytes + 4 * kRayWords, pool, cs) == cudaSuccess) {
            char* base = static_cast<char*>(ws);
            const RayRecords R{reinterpret_cast<uint4*>(base), reinterpret_cast<uint4*>(base + node_bytes),
                               reinterpret_cast<uint32_t*>(base + node_bytes + leaf_bytes)};
            cudaError_t e = cudaMemsetAsync(R.words, 0, 4 * kRayWords, cs);
            if (e == cudaSuccess) {
                ray_records_kernel<<<(bvh->n + 255) / 256, 256, 0, cs>>>(*bvh, RayScene{*bodies, *shapes}, R);
                ray_walk_kernel<<<grid, kRayThreads, 0, cs>>>(*bvh, R, d_rays, d_hits, n_rays);
                e = cudaGetLastError();
            }
            const cudaError_t fe = cudaFreeAsync(ws, cs);
            DYPH_CUDA_TRY(e);
            DYPH_CUDA_TRY(fe);
            return DYPH_OK;
        }
        cudaGetLastError();  // no scratch: the rays walk the view's own arrays
    }
    ray_query_kernel<<<grid, kRayThreads, 0, cs>>>(*bvh, RayScene{*bodies, *shapes}, d_rays, d_hits, n_rays);
    DYPH_CUDA_TRY(cudaGetLastError());
    return DYPH_OK;
}

extern "C" dyph_status dyph_contact_sensor_create(uint32_t shape_idx, dyph_contact_sensor** out) {
    if (!out) return DYPH_ERR_INVALID;
    auto* cs = new (std::nothrow) dyph_contact_sensor();
    if (!cs) return DYPH_ERR_NOMEM;
    cs->shape_idx = shape_idx;
    if (cudaMalloc(&cs->counts, 2 * sizeof(uint32_t)) != cudaSuccess) {
        delete cs;
        return DYPH_ERR_NOMEM;
    }
    *out = cs;
    return DYPH_OK;
}

extern "C" void dyph_contact_sensor_destroy(dyph_contact_sensor* cs) {
    if (!cs) return;
    if (cs->d_rows) cudaFree(cs->d_rows);
    if (cs->counts) cudaFree(cs->counts);
    if (cs->status) cudaFree(cs->status);
    if (cs->h_rows) cudaFreeHost(cs->h_rows);
    delete cs;
}

namespace {
dyph_status sensor_reserve(dyph_contact_sensor* cs, uint32_t capacity) {
    const uint32_t tiles = (capacity + kSensorThreads - 1) / kSensorThreads;
    if (tiles > cs->status_words) {
        if (cs->status) cudaFree(cs->status);
        cs->status = nullptr;
        cs->status_words = 0;
        if (cudaMalloc(&cs->status, std::max<size_t>(tiles, 1) * 4) != cudaSuccess) return DYPH_ERR_NOMEM;
        cs->status_words = tiles;
    }
    if (capacity > cs->cap) {
        if (cs->d_rows) cudaFree(cs->d_rows);
        if (cs->h_rows) cudaFreeHost(cs->h_rows);
        cs->d_rows = cs->h_rows = nullptr;
        cs->cap = 0;
        const size_t bytes = static_cast<size_t>(capacity) * kSensorRows * 4;
        if (cudaMalloc(&cs->d_rows, bytes) != cudaSuccess) return DYPH_ERR_NOMEM;
        if (cudaMallocHost(&cs->h_rows, bytes) != cudaSuccess) return DYPH_ERR_NOMEM;
        cs->cap = capacity;
    }
    return DYPH_OK;
}
}  // namespace

extern "C" dyph_status dyph_contact_sensor_filter(dyph_contact_sensor* cs, const dyph_contacts* contacts,
                                                  const uint32_t* d_body_shape, uint32_t n_bodies, dyph_stream s) {
    if (!cs || !contacts || !contacts->n || (n_bodies && !d_body_shape)) return DYPH_ERR_INVALID;
    const uint32_t capacity = std::max(contacts->capacity, 1u);
    dyph_status rs = sensor_reserve(cs, capacity);
    if (rs != DYPH_OK) return rs;
    cudaStream_t cs_ = reinterpret_cast<cudaStream_t>(s);
    const uint32_t tiles = (capacity + kSensorThreads - 1) / kSensorThreads;
    DYPH_CUDA_TRY(cudaMemsetAsync(cs->status, 0, static_cast<size_t>(tiles) * 4, cs_));
    DYPH_CUDA_TRY(cudaMemsetAsync(cs->counts, 0, 2 * sizeof(uint32_t), cs_));
    sensor_filter_kernel<<<sensor_blocks(), kSensorThreads, 0, cs_>>>(*contacts, d_body_shape, n_bodies,
                                                                       cs->shape_idx, cs->d_rows, cs->cap,
                                                                       cs->counts, cs->status);
    DYPH_CUDA_TRY(cudaGetLastError());
    return DYPH_OK;
}

extern "C" dyph_status dyph_contact_sensor_query(dyph_contact_sensor* cs, const dyph_contacts* contacts,
                                                 const uint32_t* d_body_shape, uint32_t n_bodies, dyph_stream s,
                                                 uint32_t* out_count) {
    dyph_status rs = dyph_contact_sensor_filter(cs, contacts, d_body_shape, n_bodies, s);
    if (rs != DYPH_OK) return rs;
    cudaStream_t cs_ = reinterpret_cast<cudaStream_t>(s);
    uint32_t m = 0;
    DYPH_CUDA_TRY(cudaMemcpyAsync(&m, cs->counts, sizeof(uint32_t), cudaMemcpyDeviceToHost, cs_));
    DYPH_CUDA_TRY(cudaStreamSynchronize(cs_));
    m = std::min(m, cs->cap);
    // Nine row copies of the matches only (one stream, one wait).
    for (int k = 0; k < kSensorRows && m > 0; ++k)
        DYPH_CUDA_TRY(cudaMemcpyAsync(cs->h_rows + static_cast<size_t>(k) * cs->cap,
                                      cs->d_rows + static_cast<size_t>(k) * cs->cap, static_cast<size_t>(m) * 4,
                                      cudaMemcpyDeviceToHost, cs_));
    DYPH_CUDA_TRY(cudaStreamSynchronize(cs_));
    cs->count = m;
    if (out_count) *out_count = m;
    return DYPH_OK;
}

extern "C" uint32_t dyph_contact_sensor_count(const dyph_contact_sensor* cs) { return cs ? cs->count : 0u; }
extern "C" uint32_t dyph_contact_sensor_shape_idx(const dyph_contact_sensor* cs) { return cs ? cs->shape_idx : 0u; }

namespace {
void sensor_view(uint32_t* rows, uint32_t cap, uint32_t* n, dyph_contacts* out) {
    auto row = [&](int k) { return rows ? rows + static_cast<size_t>(k) * cap : nullptr; };
    out->body_a = row(0);
    out->body_b = row(1);
    out->pos_x = reinterpret_cast<float*>(row(2));
    out->pos_y = reinterpret_cast<float*>(row(3));
    out->pos_z = reinterpret_cast<float*>(row(4));
    out->norm_x = reinterpret_cast<float*>(row(5));
    out->norm_y = reinterpret_cast<float*>(row(6));
    out->norm_z = reinterpret_cast<float*>(row(7));
    out->depth = reinterpret_cast<float*>(row(8));
    out->n = n;
    out->capacity = cap;
}
}  // namespace

extern "C" dyph_status dyph_contact_sensor_host_view(dyph_contact_sensor* cs, dyph_contacts* out) {
    if (!cs || !out) return DYPH_ERR_INVALID;
    sensor_view(cs->h_rows, cs->cap, &cs->count, out);
    return DYPH_OK;
}

extern "C" dyph_status dyph_contact_sensor_device_view(dyph_contact_sensor* cs, dyph_contacts* out) {
    if (!cs || !out) return DYPH_ERR_INVALID;
    sensor_view(cs->d_rows, cs->cap, cs->counts, out);
    return DYPH_OK;
}
