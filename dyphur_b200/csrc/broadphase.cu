// LBVH broadphase: Morton codes -> radix sort -> one-pass bottom-up Karras
// tree with fp16 boxes -> pair search over tiles of Morton-ordered leaves (tree
// walks for batched scenes) -> pairs written in ascending (a << 32 | b) order.
//
// Replaces Broadphase::build_and_query / sort_pairs (core/src/broadphase.cpp:
// 101-359). The tree is the reference's Karras tree node for node (same
// left / right / parent / NodeBox arrays, broadphase.cpp:158-288); it is built
// in a single kernel by letting each leaf walk up and the second child to
// arrive at a node merge the boxes (atomic rendezvous with release / acquire
// fences), instead of the reference's host-synchronised refit rounds.
#include <cuda_runtime.h>

#include <algorithm>
#include <new>
#include <vector>

#include "internal.cuh"

namespace dyph {
namespace {

constexpr int kBpThreads = 256;
constexpr int kMaxPartners = 32;  // per-thread sorted partner window (larger lists take extra passes)
constexpr int kFrontier = 128;     // pass 1a hands subtrees of at most this many leaves to pass 1b
constexpr int kFrontierItems = 16; // subtrees one query may hand on (more are walked in place)
constexpr int kQueuePerBody = 16;  // pass 1b queue capacity per body (overflow is walked in place)

// Single scene: 30-bit codes against the scene bounds. Batched scenes
// (codes64 != null): (scene << 30 | code) against each body's scene bounds,
// so every scene's leaves are contiguous after the sort.
__global__ void __launch_bounds__(kBpThreads) morton_kernel(GlobalBodies B, uint32_t n, dyph_aabb bounds,
                                                            uint32_t* __restrict__ codes,
                                                            uint32_t* __restrict__ sorted_idx,
                                                            uint32_t* __restrict__ counts,
                                                            uint32_t* __restrict__ tstatus, uint32_t n_tiles,
                                                            uint32_t* __restrict__ bucket_cnt,
                                                            uint64_t* __restrict__ codes64,
                                                            const uint32_t* __restrict__ scene_of,
                                                            const dyph_aabb* __restrict__ scene_bounds) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = tid; i < n; i += stride) {
        if (codes64) {
            const uint32_t sc = scene_of[i];
            codes64[i] = (static_cast<uint64_t>(sc) << 30) |
                         morton_code(B.px(i), B.py(i), B.pz(i), scene_bounds[sc]);
        } else {
            codes[i] = morton_code(B.px(i), B.py(i), B.pz(i), bounds);
        }
        sorted_idx[i] = i;
        bucket_cnt[i] = 0u;
    }
    for (uint32_t t = tid; t < n_tiles; t += stride) tstatus[t] = 0u;
    if (tid == 0) {
        counts[0] = 0u;
        counts[1] = 0u;
        counts[2] = 0u;
        counts[3] = 0u;  // pass 1b queue length, or wide leaves
        counts[4] = 0u;  // NaN seen
    }
}

// (code << 32 | body) as in the reference; batched: (scene << 52 | code << 22 | body).
__device__ __forceinline__ uint64_t key64(const uint32_t* codes, const uint64_t* codes64, const uint32_t* si, int i) {
    if (codes64) return (codes64[i] << 22) | static_cast<uint64_t>(si[i]);
    return (static_cast<uint64_t>(codes[i]) << 32) | static_cast<uint64_t>(si[i]);
}

// Common-prefix length between sorted positions i and i+1 (lbvh_delta,
// broadphase.cpp:38-41); -1 outside [0, n-1).
__device__ __forceinline__ int boundary_delta(const uint32_t* codes, const uint64_t* codes64, const uint32_t* si, int i,
                                              int n) {
    if (i < 0 || i >= n - 1) return -1;
    return __clzll(static_cast<long long>(key64(codes, codes64, si, i) ^ key64(codes, codes64, si, i + 1)));
}

// The tree bottom-up, one thread per leaf: the second child to arrive at a split
// merges the two and walks on. Bound by the chain of merges from the leaves to
// the root. Merges of subtrees inside a block's leaves, most of the chain, meet
// in shared memory and are written out together at the end; a child whose
// sibling did not come that way (it reaches into another block) then meets it in
// global memory, an atomic and two loads in L2 per merge.
constexpr int kBuildThreads = 1024;
__global__ void __launch_bounds__(kBuildThreads) build_kernel(GlobalBodies B, GlobalShapes S, uint32_t n_u,
                                                              const uint32_t* __restrict__ codes,
                                                              const uint32_t* __restrict__ si, BvhBuffers T) {
    // Split k0 + i: the children that arrived (three box words, far end | big << 31);
    // once merged, the node: box and first leaf | big << 31, last leaf and index.
    __shared__ uint4 s_child[2][kBuildThreads];
    __shared__ uint32_t s_flag[kBuildThreads];
    __shared__ int s_delta[kBuildThreads + 1];  // boundary_delta of k0 - 1 + i
    const int n = static_cast<int>(n_u);
    const int k0 = blockIdx.x * kBuildThreads, k1 = min(k0 + kBuildThreads, n);
    const int k = k0 + threadIdx.x;
    const uint64_t* codes64 = T.codes64;
    s_flag[threadIdx.x] = 0u;
    s_delta[threadIdx.x + 1] = boundary_delta(codes, codes64, si, k, n);
    if (threadIdx.x == 0) s_delta[0] = boundary_delta(codes, codes64, si, k0 - 1, n);
    uint4 box = make_uint4(0u, 0u, 0u, 0u);
    uint32_t big = 0u, body = 0u;
    int l = k, r = k;
    bool open = k < n;  // this thread carries a subtree [l, r] that has no parent yet
    if (open) {
        body = si[k];
        const uint32_t sh = B.shape(body);
        box = leaf_box(S.type(sh), B.px(body), B.py(body), B.pz(body), B.qw(body), B.qx(body), B.qy(body),
                       B.qz(body), S.hx(sh), S.hy(sh), S.hz(sh));
        // Static bodies (grounds, walls) are "large" to the tree walks: pairs with
        // them are found from the other body's side, so no thread walks the whole tree.
        big = B.im(body) == 0.f ? 1u : 0u;
        if (n == 1) open = false;
    }
    const uint4 own_box = box;
    const uint32_t own_big = big;
    __syncthreads();
    auto delta = [&](int i) {
        return i >= k0 - 1 && i < k1 ? s_delta[i - k0 + 1] : boundary_delta(codes, codes64, si, i, n);
    };
    // the index of node [L, R] (Karras): its end on the side of its parent's split
    auto node_index = [&](int L, int R) { return L == 0 && R == n - 1 ? 0 : (delta(R) > delta(L - 1) ? R : L); };
    auto child_index = [&](int L, int R, int end) { return L == R ? n - 1 + L : end; };
    auto write_node = [&](int s, int L, int R, int pidx, uint4 b, uint32_t bg) {
        const int lidx = child_index(L, s, s), ridx = child_index(s + 1, R, s + 1);
        T.big[pidx] = bg;
        T.aabb[pidx] = b;
        T.left[pidx] = lidx;
        T.right[pidx] = ridx;
        T.parent[lidx] = pidx;
        T.parent[ridx] = pidx;
        T.range_lo[pidx] = L;
        T.range_hi[pidx] = R;
        T.rsplit[s] = ridx;
    };
    // ── inside the block ──
    int parked = -1;  // the split where this thread arrived first
    while (open && !(l == 0 && r == n - 1)) {
        const bool is_left = delta(r) > delta(l - 1);  // merge across boundary r: we are the left child
        const int s = is_left ? r : l - 1;
        if (s < k0 || s + 1 >= k1) break;  // the sibling starts in another block
        s_child[is_left ? 0 : 1][s - k0] =
            make_uint4(box.x, box.y, box.z, static_cast<uint32_t>(is_left ? l : r) | (big << 31));
        __threadfence_block();
        if (atomicAdd(&s_flag[s - k0], 1u) == 0u) {
            parked = s - k0;
            break;
        }
        __threadfence_block();
        const volatile uint4* c = &s_child[is_left ? 1 : 0][s - k0];
        const uint4 sib = make_uint4(c->x, c->y, c->z, 0u);
        const uint32_t far = c->w;
        box = is_left ? merge_box(box, sib) : merge_box(sib, box);
        big |= far >> 31;
        if (is_left)
            r = static_cast<int>(far & 0x7FFFFFFFu);
        else
            l = static_cast<int>(far & 0x7FFFFFFFu);
        s_child[0][s - k0] = make_uint4(box.x, box.y, box.z, static_cast<uint32_t>(l) | (big << 31));
        s_child[1][s - k0] =
            make_uint4(static_cast<uint32_t>(r), static_cast<uint32_t>(node_index(l, r)), 0u, 0u);
    }
    __syncthreads();
    // (global writes wait until here: a fence above would wait for them)
    if (k < n) {
        T.sorted_keys[k] = key64(codes, codes64, si, k);
        T.inv_sorted[body] = static_cast<uint32_t>(k);
        T.aabb[n - 1 + k] = own_box;
        T.big[n - 1 + k] = own_big;
        if (k == 0) {
            T.parent[0] = -1;
            T.root[0] = 0;
        }
    }
    if (s_flag[threadIdx.x] == 2u) {
        const uint4 a = s_child[0][threadIdx.x], b = s_child[1][threadIdx.x];
        write_node(k, static_cast<int>(a.w & 0x7FFFFFFFu), static_cast<int>(b.x), static_cast<int>(b.y),
                   make_uint4(a.x, a.y, a.z, 0u), a.w >> 31);
    }
    if (parked >= 0 && s_flag[parked] == 2u) open = false;  // the sibling carried on
    __syncthreads();  // the nodes above are written before their parents are published
    // ── across blocks ──
    while (open && !(l == 0 && r == n - 1)) {
        const bool is_left = delta(r) > delta(l - 1);
        const int s = is_left ? r : l - 1;
        // Publish our far end (left child: slot 2s, right child: slot 2s+1), then
        // rendezvous at split s; the box and big word stand under our own index.
        T.slot[2 * s + (is_left ? 0 : 1)] = static_cast<uint32_t>(is_left ? l : r);
        // One acq_rel atomic: releases this child's slot / box / big writes and,
        // for the second arrival, acquires the sibling's.
        const uint32_t old = atom_add_acq_rel(&T.flags[s], 1u);
        if ((old & 1u) == 0u) return;  // first arrival: the sibling carries on
        // L2 loads (ld.global.cg): the sibling's writes were made on another SM.
        const int other = static_cast<int>(__ldcg(&T.slot[2 * s + (is_left ? 1 : 0)]));
        const int sidx = is_left ? child_index(s + 1, other, s + 1) : child_index(other, s, s);
        const uint4 sib = __ldcg(&T.aabb[sidx]);
        big |= __ldcg(&T.big[sidx]);
        box = is_left ? merge_box(box, sib) : merge_box(sib, box);
        if (is_left)
            r = other;
        else
            l = other;
        write_node(s, l, r, node_index(l, r), box, big);
    }
}

struct Partners {
    uint32_t v[kMaxPartners];
    int m;
};

__device__ __forceinline__ void partner_insert(Partners& p, uint32_t b) {
    int pos = p.m;
    if (pos == kMaxPartners) {
        if (b >= p.v[kMaxPartners - 1]) return;
        pos = kMaxPartners - 1;
    } else {
        p.m++;
    }
    while (pos > 0 && p.v[pos - 1] > b) {
        p.v[pos] = p.v[pos - 1];
        --pos;
    }
    p.v[pos] = b;
}

// Batched scenes: first and last sorted leaf of every scene.
__global__ void __launch_bounds__(kBpThreads) scene_range_kernel(uint32_t n, const uint64_t* __restrict__ codes64,
                                                                 uint32_t* __restrict__ first,
                                                                 uint32_t* __restrict__ last) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t sc = static_cast<uint32_t>(codes64[k] >> 30);
    if (k == 0 || static_cast<uint32_t>(codes64[k - 1] >> 30) != sc) first[sc] = k;
    if (k == n - 1 || static_cast<uint32_t>(codes64[k + 1] >> 30) != sc) last[sc] = k;
}

// A leaf is wide when it is longer than the whole scene's box over kWideShare:
// such a leaf would make its tile's box meet most others. Boxes that do not
// overlap leave room for few of them; they are tested against every leaf.
constexpr float kWideShare = 16.f;
constexpr uint32_t kWideBit = 1u << 31;  // body indices are below 2^30

__device__ __forceinline__ uint32_t min_half2(uint32_t a, uint32_t b) {
    const __half2 m = __hmin2(half2_bits(a), half2_bits(b));
    return static_cast<uint32_t>(__half_as_ushort(__low2half(m))) |
           (static_cast<uint32_t>(__half_as_ushort(__high2half(m))) << 16);
}

// Traversal record of every node (32 bytes): box + left child / body, then
// lo, hi and the escape node — the right child of the internal node whose
// split is hi (the next node in pre-order once this subtree is skipped), or -1
// when hi is the last leaf.
// The same launch prepares the tiled pair search (`tiles`): the leaves' pair
// boxes in leaf order, the box around each 32 of them, and the wide leaves.
__global__ void __launch_bounds__(kBpThreads) finalize_nodes_kernel(uint32_t n_u, BvhBuffers T, bool tiles,
                                                                    uint32_t* __restrict__ counts) {
    const int n = static_cast<int>(n_u);
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    // threads [0, n) leaves, [n, lead) fill up the last tile, then the internal nodes
    const int lead = (n + 31) & ~31;
    if (k < lead) {
        uint4 pb = make_uint4(0x7C007C00u, 0x7C007C00u, 0x7C007C00u, 0xFFFFFFFFu);  // +inf: overlaps nothing
        uint3 inner = make_uint3(0x7C007C00u, 0x7C007C00u, 0x7C007C00u);
        bool wide = false, nan = false;
        if (k < n) {
            const int j = n - 1 + k;
            const uint4 box = T.aabb[j];
            const uint32_t body = T.sorted_idx[k];
            T.trav[2 * j] = make_uint4(box.x, box.y, box.z, body);
            T.trav[2 * j + 1] = make_uint4(static_cast<uint32_t>(k), static_cast<uint32_t>(k),
                                           static_cast<uint32_t>(k >= n - 1 ? -1 : T.rsplit[k]), T.big[j]);
            if (tiles) {
                const BoxF b = unpack_box(box), r = unpack_box(T.aabb[T.root[0]]);
                const float ext = fmaxf(fmaxf(b.mxx - b.mnx, b.mxy - b.mny), b.mxz - b.mnz);
                const float all = fmaxf(fmaxf(r.mxx - r.mnx, r.mxy - r.mny), r.mxz - r.mnz);
                wide = !(ext <= all * (1.f / kWideShare));
                nan = isnan(b.mnx) || isnan(b.mny) || isnan(b.mnz) || isnan(b.mxx) || isnan(b.mxy) || isnan(b.mxz);
                pb = pair_box(box);
                if (!wide) inner = make_uint3(pb.x, pb.y, pb.z);
                pb.w = body | (wide ? kWideBit : 0u);
            }
        }
        if (tiles) {
            T.leaf_box[k] = pb;
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) {
                inner.x = min_half2(inner.x, __shfl_xor_sync(0xffffffffu, inner.x, d));
                inner.y = min_half2(inner.y, __shfl_xor_sync(0xffffffffu, inner.y, d));
                inner.z = min_half2(inner.z, __shfl_xor_sync(0xffffffffu, inner.z, d));
            }
            const unsigned wides = __ballot_sync(0xffffffffu, wide), nans = __ballot_sync(0xffffffffu, nan);
            const uint32_t lane = threadIdx.x & 31u;
            if (lane == 0u) T.tile_box[k >> 5] = make_uint4(inner.x, inner.y, inner.z, 0u);
            if (lane == 0u && nans) counts[4] = 1u;
            if (wides) {
                uint32_t at = 0;
                if (lane == 0u) at = atomicAdd(&counts[3], __popc(wides));
                at = __shfl_sync(0xffffffffu, at, 0);
                if (wide) T.wide[at + __popc(wides & ((1u << lane) - 1u))] = static_cast<uint32_t>(k);
            }
        }
        return;
    }
    const int j = k - lead;
    if (j >= n - 1) return;
    const uint4 box = T.aabb[j];
    const int lo = T.range_lo[j], hi = T.range_hi[j], w = T.left[j];
    const int esc = (hi >= n - 1) ? -1 : T.rsplit[hi];
    T.trav[2 * j] = make_uint4(box.x, box.y, box.z, static_cast<uint32_t>(w));
    T.trav[2 * j + 1] = make_uint4(static_cast<uint32_t>(lo), static_cast<uint32_t>(hi), static_cast<uint32_t>(esc),
                                   T.big[j]);
}

// Pair search of leaf k (pass 1). Every overlapping pair must be found exactly
// once: a pair of two small leaves from the larger leaf index, a pair with a
// large (static) leaf from the small side, a pair of two large leaves from the
// larger index. So a small query visits leaves i < k plus large leaves i > k,
// and a large query visits only large leaves i < k.
//
// The walk covers the subtree at `start` (pre-order: it ends at the first node
// whose leaf range starts past `end_leaf`). `frontier(node)` is offered every
// wanted, overlapping internal node covering at most kFrontier leaves; when it
// returns true the walk hands that subtree on instead of descending into it.
template <typename F, typename G>
__device__ __forceinline__ void walk_pairs(const BvhBuffers& T, int n, const BoxF& q, int k, bool me_big, int start,
                                           int begin_leaf, int end_leaf, F&& visit, G&& frontier) {
    int node = start;
    int budget = 2 * n;
    while (node >= 0) {
        if (node >= 2 * n - 1 || --budget < 0) {
            raise_error(DYPH_ERR_INVALID, 6u);
            return;
        }
        const uint4 r0 = __ldg(&T.trav[2 * node]);
        const uint4 r1 = __ldg(&T.trav[2 * node + 1]);
        if (static_cast<int>(r1.x) > end_leaf) return;
        if (static_cast<int>(r1.y) < begin_leaf) {  // subtree before the query's scene
            node = static_cast<int>(r1.z);
            continue;
        }
        const bool before = static_cast<int>(r1.x) < k;
        const bool has_big = r1.w != 0u;
        const bool wanted = me_big ? (has_big && before) : (before || has_big);
        if (!wanted) {
            if (me_big && !before) return;  // pre-order lo never decreases
            node = static_cast<int>(r1.z);
            continue;
        }
        if (box_overlap(unpack_box(r0), q)) {
            if (node >= n - 1) {
                visit(r0.w);
            } else if (!(static_cast<int>(r1.y - r1.x) < kFrontier && frontier(node))) {
                node = static_cast<int>(r0.w);
                continue;
            }
        }
        node = static_cast<int>(r1.z);
    }
}

// Stackless pre-order traversal over the traversal records: on a hit at an
// internal node go to its left child, otherwise take the escape link. Visits
// only nodes whose leaf range starts below `leaf_end` (pre-order lo values
// never decrease, so the walk stops at the first node that starts at or past
// it). `visit(body)` is called for every overlapping leaf.
template <typename F>
__device__ __forceinline__ void walk(const BvhBuffers& T, int n, const BoxF& q, int leaf_begin, int leaf_end,
                                     F&& visit) {
    int node = 0;
    // A well-formed tree visits each node at most once; anything longer (or an
    // index outside the tree) is reported instead of followed.
    int budget = 2 * n;
    while (node >= 0) {
        if (node >= 2 * n - 1 || --budget < 0) {
            raise_error(DYPH_ERR_INVALID, 7u);
            return;
        }
        const uint4 r0 = __ldg(&T.trav[2 * node]);
        const uint4 r1 = __ldg(&T.trav[2 * node + 1]);
        if (static_cast<int>(r1.x) >= leaf_end) return;
        if (static_cast<int>(r1.y) < leaf_begin) {
            node = static_cast<int>(r1.z);
            continue;
        }
        const BoxF nb = unpack_box(r0);
        if (box_overlap(nb, q)) {
            if (node >= n - 1) {
                visit(r0.w);
            } else {
                node = static_cast<int>(r0.w);
                continue;
            }
        }
        node = static_cast<int>(r1.z);
    }
}

// All overlapping partners b > lo of a query box, smallest kMaxPartners kept.
__device__ __forceinline__ uint32_t traverse(const BvhBuffers& T, int n, const BoxF& q, uint32_t a, uint32_t lo,
                                             Partners& p, int leaf_begin, int leaf_end) {
    uint32_t count = 0;
    p.m = 0;
    walk(T, n, q, leaf_begin, leaf_end, [&](uint32_t b) {
        if (b > lo && b != a) {
            ++count;
            partner_insert(p, b);
        }
    });
    return count;
}

// Sorted-leaf range [begin, end] of the scene of leaf k (the whole tree for a
// single scene).
__device__ __forceinline__ void scene_leaves(const BvhBuffers& T, int n, int k, int& begin, int& end) {
    if (!T.codes64) {
        begin = 0;
        end = n;
        return;
    }
    const uint32_t sc = static_cast<uint32_t>(T.codes64[k] >> 30);
    begin = static_cast<int>(T.scene_first[sc]);
    end = static_cast<int>(T.scene_last[sc]);
}

__device__ __forceinline__ void bucket_pair(const BvhBuffers& T, uint32_t me, uint32_t other) {
    const uint32_t a = me < other ? me : other;
    const uint32_t b = me < other ? other : me;
    const uint32_t slot = atomicAdd(&T.bucket_cnt[a], 1u);
    if (slot < static_cast<uint32_t>(kBucket)) T.bucket[static_cast<size_t>(a) * kBucket + slot] = b;
}

// Pass 1a for batched scenes, one thread per leaf in Morton order (neighbouring threads walk the
// same part of the tree): walk the tree above subtrees of at most kFrontier
// leaves and queue (leaf, subtree) items for pass 1b, so each query's work is
// spread over several threads. Leaf k tests only leaves i < k (plus static
// leaves from the small side), so every overlapping pair is found once; the
// pair goes to the bucket of its smaller body index.
__global__ void __launch_bounds__(kBpThreads) pair_find_kernel(uint32_t n_u, BvhBuffers T, uint2* __restrict__ queue,
                                                               uint32_t queue_cap, uint32_t* __restrict__ queue_len) {
    const int n = static_cast<int>(n_u);
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t items[kFrontierItems];
    uint32_t m = 0;
    if (k < n) {
        const uint4 r0 = __ldg(&T.trav[2 * (n - 1 + k)]);
        const uint4 r1 = __ldg(&T.trav[2 * (n - 1 + k) + 1]);
        const BoxF q = unpack_box(r0);
        const uint32_t me = r0.w;
        const bool me_big = r1.w != 0u;
        int sb, se;
        scene_leaves(T, n, k, sb, se);
        walk_pairs(
            T, n, q, k, me_big, 0, sb, se, [&](uint32_t other) { bucket_pair(T, me, other); },
            [&](int node) {
                if (m < static_cast<uint32_t>(kFrontierItems)) {
                    items[m++] = static_cast<uint32_t>(node);
                    return true;
                }
                return false;  // local list full: descend here instead
            });
    }
    // Warp-aggregated append of the items.
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t incl = m;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= static_cast<uint32_t>(d)) incl += y;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    uint32_t base = 0;
    if (lane == 31 && total) base = atomicAdd(queue_len, total);
    base = __shfl_sync(0xffffffffu, base, 31);
    if (m == 0) return;
    const uint32_t first = base + incl - m;
    const BoxF q = unpack_box(__ldg(&T.trav[2 * (n - 1 + k)]));
    const uint32_t me = __ldg(&T.trav[2 * (n - 1 + k)]).w;
    const bool me_big = __ldg(&T.trav[2 * (n - 1 + k) + 1]).w != 0u;
    int sb, se;
    scene_leaves(T, n, k, sb, se);
    for (uint32_t i = 0; i < m; ++i) {
        if (first + i < queue_cap) {
            queue[first + i] = make_uint2(static_cast<uint32_t>(k), items[i]);
        } else {  // queue full: walk the subtree here
            const int f = static_cast<int>(items[i]);
            const int end_leaf = min(static_cast<int>(__ldg(&T.trav[2 * f + 1]).y), se);
            walk_pairs(
                T, n, q, k, me_big, f, sb, end_leaf, [&](uint32_t other) { bucket_pair(T, me, other); },
                [](int) { return false; });
        }
    }
}

// Pass 1b, one thread per queued (leaf, subtree) item.
__global__ void __launch_bounds__(kBpThreads) pair_subtree_kernel(uint32_t n_u, BvhBuffers T,
                                                                  const uint2* __restrict__ queue, uint32_t queue_cap,
                                                                  const uint32_t* __restrict__ queue_len) {
    const int n = static_cast<int>(n_u);
    const uint32_t len = min(*queue_len, queue_cap);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < len; i += gridDim.x * blockDim.x) {
        const uint2 it = queue[i];
        const int k = static_cast<int>(it.x), f = static_cast<int>(it.y);
        const uint4 r0 = __ldg(&T.trav[2 * (n - 1 + k)]);
        const bool me_big = __ldg(&T.trav[2 * (n - 1 + k) + 1]).w != 0u;
        const BoxF q = unpack_box(r0);
        const uint32_t me = r0.w;
        int sb, se;
        scene_leaves(T, n, k, sb, se);
        const int end_leaf = min(static_cast<int>(__ldg(&T.trav[2 * f + 1]).y), se);
        walk_pairs(
            T, n, q, k, me_big, f, sb, end_leaf, [&](uint32_t other) { bucket_pair(T, me, other); },
            [](int) { return false; });
    }
}

// Pass 1 for a single scene of at most kTiledBodies bodies, one warp per tile of
// 32 leaves in Morton order and part of the tiles before it: a lane holds a leaf
// and meets 32 tile boxes as broadcasts (see pair_overlap), then the leaves of
// each tile that some lane's leaf met. Wide leaves are kept out of the tiles and
// meet every leaf. Every overlapping pair is found once, from its later leaf (or
// from the leaf that is not wide), and goes to the bucket of its smaller body
// index. The tests are
// dense and independent, where a walk of the tree per leaf waits for a node per
// step in divergent lanes; but tiles that straddle distant parts of the Morton
// order meet more tiles the more there are. Whole broadphase, tiles against tree
// walks: 52 and 67 us at 500 bodies of a pile, 89 and 122 at 2,000, 142 and 198 at
// 10,000, 209 and 274 at 32,000, 343 and 320 at 48,000.
// A NaN bound overlaps everything it is compared with, and a tree walk meets it
// only below ancestors that overlap: with one in the scene every leaf walks to the
// earlier leaves, as the reference's do (core/src/broadphase.cpp:290-345).
constexpr uint32_t kTiledBodies = 32768;
constexpr int kTileWarps = kBpThreads / 32;
__global__ void __launch_bounds__(kBpThreads) pair_tiles_kernel(uint32_t n_u, BvhBuffers T, uint32_t parts,
                                                                const uint32_t* __restrict__ counts) {
    __shared__ uint4 s_box[kTileWarps][32], s_tile[kTileWarps][32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t tiles = (n_u + 31u) >> 5;
    const uint32_t item = blockIdx.x * kTileWarps + warp;
    if (item >= tiles * parts) return;
    const uint32_t tile = tiles - 1u - item / parts, part = item % parts;  // the long rows first
    const uint32_t k = 32u * tile + lane;
    if (counts[4]) {
        if (part != 0u || k >= n_u) return;
        const int n = static_cast<int>(n_u), node = n - 1 + static_cast<int>(k);
        const uint4 r0 = __ldg(&T.trav[2 * node]);
        walk(T, n, unpack_box(r0), 0, static_cast<int>(k), [&](uint32_t other) { bucket_pair(T, r0.w, other); });
        return;
    }
    const uint4 mine = __ldg(&T.leaf_box[k]);
    const uint32_t me = mine.w & ~kWideBit;
    const bool i_am = k < n_u, wide = i_am && (mine.w & kWideBit) != 0u;
    const uint3 q = facing_box(mine);
    uint4* const other = s_box[warp];
    // the leaves of s_box that this lane's leaf meets, as bits
    auto meet = [&]() -> uint32_t {
        uint32_t w = 0;
#pragma unroll 8
        for (uint32_t j = 0; j < 32u; ++j) w |= pair_overlap(other[j], q) ? 1u << j : 0u;
        return i_am ? w : 0u;
    };
    auto emit = [&](uint32_t w) {
        for (; w; w &= w - 1u) bucket_pair(T, me, other[__ffs(static_cast<int>(w)) - 1].w & ~kWideBit);
    };
    const uint3 tq = facing_box(__ldg(&T.tile_box[tile]));
    uint4* const boxes = s_tile[warp];
    for (uint32_t t0 = part; t0 <= tile; t0 += 32u * parts) {  // every parts-th tile, 32 at a time
        // which of the 32 tiles' boxes this lane's leaf meets; a tile of leaves that
        // lie apart has a box that meets many tiles its leaves do not
        const uint32_t t = t0 + lane * parts;
        __syncwarp();
        boxes[lane] = t <= tile ? __ldg(&T.tile_box[t]) : make_uint4(0x7C007C00u, 0x7C007C00u, 0x7C007C00u, 0u);
        __syncwarp();
        uint32_t near = 0;
#pragma unroll 8
        for (uint32_t j = 0; j < 32u; ++j) near |= pair_overlap(boxes[j], q) ? 1u << j : 0u;
        const uint32_t there = (tile - t0) / parts;  // tiles of the 32 past the first
        if (there < 31u) near &= (2u << there) - 1u;
        if (!i_am || wide) near = 0u;
        uint32_t hits = __reduce_or_sync(0xffffffffu, near);
        uint4 o = make_uint4(0u, 0u, 0u, 0u);
        if (hits) o = __ldg(&T.leaf_box[32u * (t0 + (__ffs(static_cast<int>(hits)) - 1) * parts) + lane]);
        while (hits) {
            const uint32_t bit = static_cast<uint32_t>(__ffs(static_cast<int>(hits))) - 1u, u = t0 + bit * parts;
            hits &= hits - 1u;
            const uint4 cur = o;
            if (hits)  // the next tile's leaves, while this one's are tested
                o = __ldg(&T.leaf_box[32u * (t0 + (__ffs(static_cast<int>(hits)) - 1) * parts) + lane]);
            const bool mine_near = (near >> bit) & 1u, theirs = (cur.w & kWideBit) == 0u;
            unsigned others = __ballot_sync(0xffffffffu, theirs && pair_overlap(cur, tq));
            const unsigned nears = __ballot_sync(0xffffffffu, mine_near);
            if (!others) continue;
            __syncwarp();
            other[lane] = cur;
            uint32_t w = 0;
            if (__popc(nears) < __popc(others)) {
                // few leaves here: each met by the 32 there at once
                for (unsigned m = nears; m; m &= m - 1u) {
                    const int src = __ffs(static_cast<int>(m)) - 1;
                    const uint3 sq = make_uint3(__shfl_sync(0xffffffffu, q.x, src), __shfl_sync(0xffffffffu, q.y, src),
                                                __shfl_sync(0xffffffffu, q.z, src));
                    const unsigned met = __ballot_sync(0xffffffffu, theirs && pair_overlap(cur, sq));
                    if (static_cast<int>(lane) == src) w = met;
                }
                __syncwarp();
            } else {
                __syncwarp();
                for (; others; others &= others - 1u) {
                    const uint32_t j = static_cast<uint32_t>(__ffs(static_cast<int>(others))) - 1u;
                    w |= pair_overlap(other[j], q) ? 1u << j : 0u;
                }
                if (!mine_near) w = 0u;
            }
            if (u == tile) w &= (1u << lane) - 1u;  // earlier leaves only
            emit(w);
        }
    }
    const uint32_t n_wide = counts[3];
    for (uint32_t w0 = 32u * part; w0 < n_wide; w0 += 32u * parts) {
        const uint32_t leaf = w0 + lane < n_wide ? T.wide[w0 + lane] : 0xFFFFFFFFu;
        const uint4 o = leaf != 0xFFFFFFFFu ? __ldg(&T.leaf_box[leaf])
                                            : make_uint4(0x7C007C00u, 0x7C007C00u, 0x7C007C00u, 0xFFFFFFFFu);
        __syncwarp();
        other[lane] = o;
        __syncwarp();
        uint32_t w = meet();
        if (w0 + 32u > n_wide) w &= (1u << (n_wide - w0)) - 1u;
        // of two wide leaves the later one finds the pair
        for (uint32_t j = 0; j < 32u; ++j) {
            const uint32_t l = __shfl_sync(0xffffffffu, leaf, static_cast<int>(j));
            if (wide && l >= k) w &= ~(1u << j);
        }
        emit(w);
    }
}

// Whether a walk with query q reaches leaf k: its box and those above it overlap.
__device__ __forceinline__ bool reaches(const BvhBuffers& T, int n, int k, const BoxF& q) {
    int budget = n;
    for (int node = n - 1 + k; node >= 0 && budget-- > 0; node = T.parent[node])
        if (!box_overlap(unpack_box(T.aabb[node]), q)) return false;
    return true;
}

// Pass 2, one block per kWriteBodies bodies: place each body's pairs with a
// block scan + decoupled look-back (the counts are final after pass 1, so every
// tile publishes its aggregate at once), then write them sorted by b. Each warp
// ranks four buckets at a time, an element's place being the number of smaller
// partners (the partners are distinct): bound by the latency of a bucket's load,
// so a warp has four in flight and few in turn. A bucket that overflowed is
// rebuilt by a full traversal from the body's own leaf; with a NaN in the scene
// (counts[4], tiled search only), body by body, from the later leaf of each two.
constexpr int kWriteBodies = 64;
__global__ void __launch_bounds__(kBpThreads) pair_write_kernel(uint32_t n_u, BvhBuffers T, uint2* __restrict__ pairs,
                                                                uint32_t max_pairs, uint32_t* __restrict__ counts,
                                                                uint32_t* __restrict__ tstatus) {
    __shared__ uint32_t s_tile, s_excl;
    __shared__ uint32_t s_scan[kBpThreads / 32];
    __shared__ uint32_t s_off[kWriteBodies], s_cnt[kWriteBodies];
    const int n = static_cast<int>(n_u);
    if (threadIdx.x == 0) s_tile = atomicAdd(&counts[2], 1u);
    __syncthreads();
    const uint32_t tile = s_tile, a0 = tile * kWriteBodies, a = a0 + threadIdx.x;
    const bool mine = threadIdx.x < kWriteBodies && a < n_u;
    const uint32_t cnt = mine ? T.bucket_cnt[a] : 0u;
    uint32_t total;
    const uint32_t excl_block = block_exclusive_scan<kBpThreads>(cnt, s_scan, total);
    if (threadIdx.x < 32) {
        const uint32_t e = lookback_warp(tstatus, tile, total);
        if (threadIdx.x == 0) {
            s_excl = e;
            const uint32_t last_tile = (n_u - 1) / kWriteBodies;
            if (tile == last_tile) {
                const uint32_t all = e + total;
                counts[1] = all;
                counts[0] = all < max_pairs ? all : max_pairs;
            }
        }
    }
    __syncthreads();
    const uint32_t off = s_excl + excl_block;
    if (threadIdx.x < kWriteBodies) {
        s_off[threadIdx.x] = off;
        s_cnt[threadIdx.x] = cnt;
    }
    if (cnt > static_cast<uint32_t>(kBucket)) {
        Partners P;
        const uint32_t leaf = __ldg(&T.inv_sorted[a]);
        const BoxF q = unpack_box(__ldg(&T.trav[2 * (n - 1 + static_cast<int>(leaf))]));
        int sb, se;
        scene_leaves(T, n, static_cast<int>(leaf), sb, se);
        uint32_t written = 0;
        const bool nan = counts[4] != 0u;
        for (uint32_t b = a + 1u; nan && b < n_u; ++b) {
            const uint32_t other = __ldg(&T.inv_sorted[b]);
            const bool met = other < leaf ? reaches(T, n, static_cast<int>(other), q)
                                          : reaches(T, n, static_cast<int>(leaf), unpack_box(T.aabb[n_u - 1u + other]));
            if (!met) continue;
            if (off + written < max_pairs) pairs[off + written] = make_uint2(a, b);
            ++written;
        }
        if (!nan) traverse(T, n, q, a, a, P, sb, se + 1);
        while (!nan) {
            for (int i = 0; i < P.m; ++i) {
                const uint32_t pos = off + written + static_cast<uint32_t>(i);
                if (pos < max_pairs) pairs[pos] = make_uint2(a, P.v[i]);
            }
            written += static_cast<uint32_t>(P.m);
            if (written >= cnt || P.m == 0) break;
            traverse(T, n, q, a, P.v[P.m - 1], P, sb, se + 1);
        }
    }
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    constexpr int kPer = kBucket / 32;
    for (uint32_t q0 = (threadIdx.x >> 5) * 4u; q0 < static_cast<uint32_t>(kWriteBodies);
         q0 += kBpThreads / 32 * 4u) {
        uint32_t c[4], most = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            c[j] = s_cnt[q0 + j];
            most = max(most, c[j]);
        }
        if (most <= 32u) {
            uint32_t v[4], rank[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int j = 0; j < 4; ++j)
                v[j] = lane < c[j] ? T.bucket[static_cast<size_t>(a0 + q0 + j) * kBucket + lane] : 0xFFFFFFFFu;
            for (uint32_t t = 0; t < most; ++t) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    rank[j] += __shfl_sync(0xffffffffu, v[j], static_cast<int>(t)) < v[j] ? 1u : 0u;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t pos = s_off[q0 + j] + rank[j];
                if (lane < c[j] && pos < max_pairs) pairs[pos] = make_uint2(a0 + q0 + j, v[j]);
            }
            continue;
        }
        for (uint32_t q = q0; q < q0 + 4u; ++q) {
            // lane l holds elements l, l + 32, ...
            const uint32_t ab = a0 + q, base = s_off[q], mb = s_cnt[q];
            if (mb > static_cast<uint32_t>(kBucket)) continue;  // written above
            uint32_t v[kPer], rank[kPer];
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const uint32_t i = lane + 32u * j;
                v[j] = i < mb ? T.bucket[static_cast<size_t>(ab) * kBucket + i] : 0xFFFFFFFFu;
                rank[j] = 0u;
            }
#pragma unroll
            for (int jj = 0; jj < kPer; ++jj) {
                for (uint32_t l = 0; l < 32u; ++l) {
                    if (32u * jj + l >= mb) break;  // warp-uniform
                    const uint32_t w = __shfl_sync(0xffffffffu, v[jj], l);
#pragma unroll
                    for (int j = 0; j < kPer; ++j) rank[j] += (w < v[j]) ? 1u : 0u;
                }
            }
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const uint32_t i = lane + 32u * j;
                const uint32_t pos = base + rank[j];
                if (i < mb && pos < max_pairs) pairs[pos] = make_uint2(ab, v[j]);
            }
        }
    }
}

int subtree_blocks() {
    static int blocks = 0;
    if (blocks == 0) {
        int dev = 0, sms = 148;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        blocks = sms * 8;
    }
    return blocks;
}

template <typename T>
cudaError_t dev_alloc(T** p, size_t count) {
    return cudaMalloc(reinterpret_cast<void**>(p), std::max<size_t>(count, 1) * sizeof(T));
}

}  // namespace

dyph_status broadphase_build(dyph_broadphase* bp, const dyph_bodies* bodies, const dyph_shapes* shapes,
                             const dyph_aabb* bounds, cudaStream_t s) {
    if (!bp || !bodies || !shapes || !bounds) return DYPH_ERR_INVALID;
    const uint32_t n = bodies->n;
    if (n > bp->max_bodies) return DYPH_ERR_INVALID;
    const uint32_t n_tiles = (std::max(n, 1u) + kWriteBodies - 1) / kWriteBodies;
    GlobalBodies B{*bodies};
    GlobalShapes S{*shapes};
    const uint32_t mblocks = std::max(1u, std::min((n + kBpThreads - 1) / kBpThreads, 2048u));
    morton_kernel<<<mblocks, kBpThreads, 0, s>>>(B, n, *bounds, bp->codes, bp->bvh.sorted_idx, bp->counts,
                                                 bp->tstatus, n_tiles, bp->bvh.bucket_cnt, bp->bvh.codes64,
                                                 bp->bvh.scene_of, bp->scene_bounds);
    DYPH_CUDA_TRY(cudaGetLastError());
    bp->last_n = n;
    if (n < 2) return DYPH_OK;
    dyph_status st = bp->bvh.codes64
                         ? sort_u64_u32(bp->bvh.codes64, bp->bvh.sorted_idx, n, 30 + bp->scene_bits, bp->sort_ws,
                                        bp->sort_ws_bytes, s)
                         : sort_u32_u32(bp->codes, bp->bvh.sorted_idx, n, 30, bp->sort_ws, bp->sort_ws_bytes, s);
    if (st != DYPH_OK) return st;
    if (bp->bvh.codes64) {
        scene_range_kernel<<<(n + kBpThreads - 1) / kBpThreads, kBpThreads, 0, s>>>(
            n, bp->bvh.codes64, bp->bvh.scene_first, bp->bvh.scene_last);
        DYPH_CUDA_TRY(cudaGetLastError());
    }
    const uint32_t leaf_blocks = (n + kBpThreads - 1) / kBpThreads;
    build_kernel<<<(n + kBuildThreads - 1) / kBuildThreads, kBuildThreads, 0, s>>>(B, S, n, bp->codes, bp->bvh.sorted_idx, bp->bvh);
    DYPH_CUDA_TRY(cudaGetLastError());
    // Batched scenes pair inside each scene, by the tree walk; so do large single
    // ones, whose tiles more often straddle distant parts of the Morton order.
    const bool tiled = !bp->bvh.codes64 && n <= kTiledBodies;
    const uint32_t fin = ((n + 31u) & ~31u) + n - 1u;
    finalize_nodes_kernel<<<(fin + kBpThreads - 1) / kBpThreads, kBpThreads, 0, s>>>(n, bp->bvh, tiled, bp->counts);
    DYPH_CUDA_TRY(cudaGetLastError());
    if (tiled) {
        // few tiles: several warps to a tile's row
        const uint32_t tiles = (n + 31u) / 32u, parts = std::clamp(16384u / tiles, 1u, 16u);
        pair_tiles_kernel<<<(tiles * parts + kTileWarps - 1) / kTileWarps, kBpThreads, 0, s>>>(n, bp->bvh, parts,
                                                                                              bp->counts);
        DYPH_CUDA_TRY(cudaGetLastError());
    } else {
        const uint32_t queue_cap = bp->max_bodies * static_cast<uint32_t>(kQueuePerBody);
        pair_find_kernel<<<leaf_blocks, kBpThreads, 0, s>>>(n, bp->bvh, bp->queue, queue_cap, bp->counts + 3);
        DYPH_CUDA_TRY(cudaGetLastError());
        pair_subtree_kernel<<<subtree_blocks(), kBpThreads, 0, s>>>(n, bp->bvh, bp->queue, queue_cap,
                                                                    bp->counts + 3);
        DYPH_CUDA_TRY(cudaGetLastError());
    }
    pair_write_kernel<<<n_tiles, kBpThreads, 0, s>>>(n, bp->bvh, reinterpret_cast<uint2*>(bp->pairs), bp->max_pairs,
                                                     bp->counts, bp->tstatus);
    DYPH_CUDA_TRY(cudaGetLastError());
    return DYPH_OK;
}

dyph_status setup_done() {
    DYPH_CUDA_TRY(cudaStreamSynchronize(cudaStreamLegacy));
    return DYPH_OK;
}

dyph_status broadphase_create(uint32_t max_bodies, uint32_t max_pairs, dyph_broadphase** out) {
    if (!out || max_bodies == 0 || max_pairs == 0 || max_bodies >= (1u << 30)) return DYPH_ERR_INVALID;
    auto* bp = new (std::nothrow) dyph_broadphase();
    if (!bp) return DYPH_ERR_NOMEM;
    bp->max_bodies = max_bodies;
    bp->max_pairs = max_pairs;
    const size_t nb = max_bodies, ni = max_bodies > 1 ? max_bodies - 1 : 1, nn = 2 * nb - 1;
    bool ok = dev_alloc(&bp->codes, nb) == cudaSuccess && dev_alloc(&bp->bvh.sorted_idx, nb) == cudaSuccess &&
              dev_alloc(&bp->bvh.sorted_keys, nb) == cudaSuccess &&
              dev_alloc(&bp->bvh.inv_sorted, nb) == cudaSuccess && dev_alloc(&bp->bvh.left, ni) == cudaSuccess &&
              dev_alloc(&bp->bvh.right, ni) == cudaSuccess && dev_alloc(&bp->bvh.parent, nn) == cudaSuccess &&
              dev_alloc(&bp->bvh.root, 1) == cudaSuccess && dev_alloc(&bp->bvh.aabb, nn) == cudaSuccess &&
              dev_alloc(&bp->bvh.range_hi, ni) == cudaSuccess && dev_alloc(&bp->bvh.rsplit, ni) == cudaSuccess &&
              dev_alloc(&bp->bvh.slot, 2 * ni) == cudaSuccess && dev_alloc(&bp->bvh.flags, ni) == cudaSuccess &&
              dev_alloc(&bp->pairs, max_pairs) == cudaSuccess && dev_alloc(&bp->counts, 8) == cudaSuccess &&
              dev_alloc(&bp->tstatus, (nb + kWriteBodies - 1) / kWriteBodies) == cudaSuccess &&
              dev_alloc(&bp->bvh.range_lo, ni) == cudaSuccess && dev_alloc(&bp->bvh.trav, 2 * nn) == cudaSuccess &&
              dev_alloc(&bp->bvh.bucket_cnt, nb) == cudaSuccess && dev_alloc(&bp->bvh.big, nn) == cudaSuccess &&
              dev_alloc(&bp->bvh.bucket, nb * kBucket) == cudaSuccess &&
              dev_alloc(&bp->bvh.leaf_box, (nb + 31) / 32 * 32) == cudaSuccess &&
              dev_alloc(&bp->bvh.tile_box, (nb + 31) / 32) == cudaSuccess &&
              dev_alloc(&bp->bvh.wide, nb) == cudaSuccess &&
              (nb <= kTiledBodies || dev_alloc(&bp->queue, nb * kQueuePerBody) == cudaSuccess);
    if (ok) {
        bp->sort_ws_bytes = sort_workspace_bytes(nb, 4);
        ok = cudaMalloc(&bp->sort_ws, bp->sort_ws_bytes) == cudaSuccess;
    }
    // Arrival counters start even; every build adds none or two at a split.
    if (ok) ok = cudaMemset(bp->bvh.flags, 0, ni * sizeof(uint32_t)) == cudaSuccess;
    if (ok) ok = cudaMemset(bp->counts, 0, 8 * sizeof(uint32_t)) == cudaSuccess;
    if (ok) ok = sort_prepare() == DYPH_OK && setup_done() == DYPH_OK;
    if (!ok) {
        broadphase_destroy(bp);
        return DYPH_ERR_NOMEM;
    }
    *out = bp;
    return DYPH_OK;
}

dyph_status broadphase_set_scenes(dyph_broadphase* bp, uint32_t n_scenes, const uint32_t* h_body_offset,
                                  const dyph_aabb* h_scene_bounds) {
    if (!bp || n_scenes == 0 || !h_body_offset || !h_scene_bounds) return DYPH_ERR_INVALID;
    // Keys are (scene << 52 | code << 22 | body): at most 4096 scenes of a
    // tree of at most 2^22 bodies.
    if (n_scenes > 4096u || bp->max_bodies > (1u << 22) || h_body_offset[0] != 0u ||
        h_body_offset[n_scenes] > bp->max_bodies)
        return DYPH_ERR_INVALID;
    for (uint32_t i = 0; i < n_scenes; ++i)
        if (h_body_offset[i + 1] <= h_body_offset[i]) return DYPH_ERR_INVALID;  // every scene has a body
    const uint32_t n = h_body_offset[n_scenes];
    int bits = 0;
    while ((1u << bits) < n_scenes) ++bits;
    bool ok = true;
    if (!bp->bvh.codes64) ok = dev_alloc(&bp->bvh.codes64, bp->max_bodies) == cudaSuccess &&
                                 dev_alloc(&bp->bvh.scene_of, bp->max_bodies) == cudaSuccess &&
                                 (bp->queue || dev_alloc(&bp->queue, static_cast<size_t>(bp->max_bodies) *
                                                                         kQueuePerBody) == cudaSuccess);
    if (bp->scene_bounds) cudaFree(bp->scene_bounds);
    if (bp->bvh.scene_first) cudaFree(bp->bvh.scene_first);
    if (bp->bvh.scene_last) cudaFree(bp->bvh.scene_last);
    if (bp->body_offset) cudaFree(bp->body_offset);
    bp->scene_bounds = nullptr;
    bp->bvh.scene_first = bp->bvh.scene_last = bp->body_offset = nullptr;
    ok = ok && dev_alloc(&bp->scene_bounds, n_scenes) == cudaSuccess &&
         dev_alloc(&bp->bvh.scene_first, n_scenes) == cudaSuccess &&
         dev_alloc(&bp->bvh.scene_last, n_scenes) == cudaSuccess &&
         dev_alloc(&bp->body_offset, n_scenes + 1) == cudaSuccess;
    if (!ok) return DYPH_ERR_NOMEM;
    std::vector<uint32_t> scene_of(n);
    for (uint32_t sc = 0; sc < n_scenes; ++sc)
        for (uint32_t i = h_body_offset[sc]; i < h_body_offset[sc + 1]; ++i) scene_of[i] = sc;
    DYPH_CUDA_TRY(cudaMemcpy(bp->bvh.scene_of, scene_of.data(), n * 4, cudaMemcpyHostToDevice));
    DYPH_CUDA_TRY(cudaMemcpy(bp->scene_bounds, h_scene_bounds, n_scenes * sizeof(dyph_aabb), cudaMemcpyHostToDevice));
    DYPH_CUDA_TRY(cudaMemcpy(bp->body_offset, h_body_offset, (n_scenes + 1) * 4, cudaMemcpyHostToDevice));
    const size_t ws = sort_workspace_bytes(bp->max_bodies, 8);
    if (ws > bp->sort_ws_bytes) {
        if (bp->sort_ws) cudaFree(bp->sort_ws);
        bp->sort_ws = nullptr;
        bp->sort_ws_bytes = 0;
        if (cudaMalloc(&bp->sort_ws, ws) != cudaSuccess) return DYPH_ERR_NOMEM;
        bp->sort_ws_bytes = ws;
    }
    bp->n_scenes = n_scenes;
    bp->scene_bits = bits;
    return setup_done();
}

void broadphase_destroy(dyph_broadphase* bp) {
    if (!bp) return;
    void* ptrs[] = {bp->codes, bp->bvh.sorted_idx, bp->bvh.sorted_keys, bp->bvh.inv_sorted, bp->bvh.left,
                    bp->bvh.right, bp->bvh.parent, bp->bvh.root, bp->bvh.aabb, bp->bvh.range_hi, bp->bvh.rsplit,
                    bp->bvh.slot, bp->bvh.flags, bp->pairs, bp->counts, bp->tstatus, bp->sort_ws,
                    bp->bvh.range_lo, bp->bvh.trav, bp->bvh.bucket_cnt, bp->bvh.bucket, bp->bvh.big, bp->queue,
                    bp->bvh.leaf_box, bp->bvh.tile_box, bp->bvh.wide, bp->bvh.codes64, bp->bvh.scene_of, bp->bvh.scene_first, bp->bvh.scene_last,
                    bp->scene_bounds, bp->body_offset};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    delete bp;
}

}  // namespace dyph

using namespace dyph;

extern "C" dyph_status dyph_broadphase_create(uint32_t max_bodies, uint32_t max_pairs, dyph_broadphase** out) {
    return broadphase_create(max_bodies, max_pairs, out);
}

extern "C" void dyph_broadphase_destroy(dyph_broadphase* bp) { broadphase_destroy(bp); }

extern "C" dyph_status dyph_broadphase_build_and_query(dyph_broadphase* bp, const dyph_bodies* bodies,
                                                       const dyph_shapes* shapes, const dyph_aabb* bounds,
                                                       dyph_stream s) {
    return broadphase_build(bp, bodies, shapes, bounds, reinterpret_cast<cudaStream_t>(s));
}

extern "C" dyph_status dyph_broadphase_sort_pairs(dyph_broadphase* bp, uint32_t, dyph_stream) {
    return bp ? DYPH_OK : DYPH_ERR_INVALID;  // pairs are emitted in sorted order
}

extern "C" dyph_status dyph_broadphase_download_count(dyph_broadphase* bp, dyph_stream s, uint32_t* out) {
    if (!bp || !out) return DYPH_ERR_INVALID;
    cudaStream_t cs = reinterpret_cast<cudaStream_t>(s);
    DYPH_CUDA_TRY(cudaMemcpyAsync(out, bp->counts + 1, sizeof(uint32_t), cudaMemcpyDeviceToHost, cs));
    DYPH_CUDA_TRY(cudaStreamSynchronize(cs));
    return DYPH_OK;
}

extern "C" const dyph_pair* dyph_broadphase_pairs(const dyph_broadphase* bp) { return bp ? bp->pairs : nullptr; }
extern "C" const uint32_t* dyph_broadphase_count_ptr(const dyph_broadphase* bp) { return bp ? bp->counts : nullptr; }
extern "C" uint32_t dyph_broadphase_max_pairs(const dyph_broadphase* bp) { return bp ? bp->max_pairs : 0u; }

extern "C" dyph_status dyph_broadphase_bvh_view(const dyph_broadphase* bp, uint32_t n_active, dyph_bvh_view* out) {
    if (!bp || !out) return DYPH_ERR_INVALID;
    out->left = bp->bvh.left;
    out->right = bp->bvh.right;
    out->parent = bp->bvh.parent;
    out->root = bp->bvh.root;
    out->sorted_idx = bp->bvh.sorted_idx;
    out->aabb = reinterpret_cast<const dyph_node_box*>(bp->bvh.aabb);
    out->sorted_keys = bp->bvh.sorted_keys;
    out->n = n_active;
    return DYPH_OK;
}

extern "C" dyph_status dyph_broadphase_set_scenes(dyph_broadphase* bp, uint32_t n_scenes, const uint32_t* body_offset,
                                                  const dyph_aabb* scene_bounds) {
    return dyph::broadphase_set_scenes(bp, n_scenes, body_offset, scene_bounds);
}
