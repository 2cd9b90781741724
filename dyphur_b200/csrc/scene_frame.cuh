// Batched scenes, fused: one thread block runs whole frames of one scene —
// integrate, pair search, narrowphase and contact solve — on the scene's
// bodies in shared memory, frame after frame, and writes the bodies back once
// per launch. Included by
// world.cu (after solver.cu in the library's translation unit).
//
// Every stage is the single-scene stage restated for one block:
//   * integrate: integrate_body per dynamic, awake body (core/src/
//     integrator.cpp:18-68), all substeps in registers;
//   * pairs: the candidate-pair set is the set of body pairs whose fp16 leaf
//     boxes (core/src/broadphase.cpp:216-251) overlap under the traversal's
//     inclusive test (:322-325), because internal nodes merge the leaf boxes
//     exactly. So every (a, b) with a < b is tested directly and the pairs
//     come out in ascending (a << 32 | b) order, as Broadphase::sort_pairs
//     leaves them; a scene keeps the first max_pairs of them, as it does alone.
//     A NaN bound overlaps every other, where a tree walk meets it only below
//     ancestors that overlap: a single scene's frames follow the walk there
//     (reach_box), those of a batch take every such pair;
//   * narrowphase: process_pair (core/src/narrowphase.cpp:920-1001) per pair,
//     contacts compacted in pair order, the first max_contacts kept;
//   * solve: scene_solve (solver_scene.cuh).
// A scene's frame is therefore bit-identical to the frame of the scene
// stepped alone (of a batch, as long as no leaf box holds a NaN). The frame's pair and contact lists stay in per-scene slots
// and are compacted into the broadphase's / narrowphase's lists on request
// (scene_gather_*).
#pragma once

#include "solver_scene.cuh"

namespace dyph {
namespace {

// Per-body rows the fused frame adds after the solver's rows: shape type and
// flags, half extents (3), leaf box (4 words, see PairBox).
constexpr uint32_t kFrameBodyRows = 8;

__host__ __device__ __forceinline__ uint32_t frame_body_bytes(uint32_t nb) {
    const uint32_t ldb = (nb + 3u) & ~3u;
    return scene_body_bytes(nb) + kFrameBodyRows * 4u * ldb;
}

// Overlap bits of the candidate-pair search: bit j of word (c, a) says whether
// bodies a and b = 32 c + j > a overlap, for chunks c >= a / 32. Chunk c's words
// are consecutive in a (a warp's lanes take consecutive a), 32 (c + 1) of them.
__host__ __device__ __forceinline__ uint32_t overlap_chunks(uint32_t nb) { return (nb + 31u) >> 5; }
__host__ __device__ __forceinline__ uint32_t overlap_mask_base(uint32_t c) { return 16u * c * (c + 1u); }

struct FrameBufs {
    const uint32_t* pair_base;     // [n_scenes + 1] first pair slot of each scene (capacity 48 n + 64)
    const uint32_t* contact_base;  // [n_scenes + 1] first contact slot of each scene (capacity 16 n + 64)
    uint32_t* pair_raw;            // [total pair slots] a | b << 16 (local indices)
    uint32_t* contact_raw;         // [9][total contact slots] a, b (global), position, normal, depth
    uint32_t* color_raw;           // [total contact slots] colour (UINT32_MAX on the sequential order)
    uint32_t* counts;              // [4 n_scenes] stored pairs, true pairs, stored contacts, true contacts
    uint32_t* words;               // [kSceneWords][words_stride] contact words of scenes too big for shared memory
    uint32_t words_stride;         // total contact slots + n_scenes
    uint32_t contact_slots;        // total contact slots
};

// Shape rows of one scene in shared memory, indexed by local body (each body
// carries its own shape's type and half extents).
struct SceneShapes {
    const uint32_t* info;  // type | flags << 8
    const float* half;     // 3 rows
    uint32_t ld;
    __device__ __forceinline__ uint32_t type(uint32_t i) const { return info[i] & 0xFFu; }
    __device__ __forceinline__ float hx(uint32_t i) const { return half[i]; }
    __device__ __forceinline__ float hy(uint32_t i) const { return half[ld + i]; }
    __device__ __forceinline__ float hz(uint32_t i) const { return half[2 * ld + i]; }
};

struct SceneBodiesShaped : SceneBodies {
    __device__ __forceinline__ uint32_t shape(uint32_t i) const { return i; }
};

// Words a launch's last frame leaves for frame_run_stats_kernel, which moves
// them to the solver's meta words and clears them: largest colour + 1, JP
// rounds, some scene coloured, some scene solved.
constexpr int kAccMaxColor = 0, kAccRounds = 1, kAccColored = 2, kAccSolved = 3, kAccWords = 4;

// Frames of one launch at most (the per-frame count words), and words of each.
constexpr uint32_t kMaxRunFrames = 256, kRunRows = 5;

// Parameters of the fused kernels, one launch.
struct FrameParams {
    dyph_bodies gb;
    dyph_shapes gs;
    float gx, gy, gz, sub_dt, half_dt, mu, dt;
    int n_substeps, mode, n_iters;
    uint32_t* acc;     // [kAccWords]
    // [5][n_frames] stored / true pairs, stored / true contacts of every frame, over
    // all scenes; bit 0: a scene past its pair capacity, bit 1: past its contact capacity
    uint32_t* counts;
    unsigned long long* phase_ns;  // null, or [kFramePhases] device-clock ns summed over scenes
    uint32_t n_frames;             // frames of this launch
    uint32_t keep;                 // 1: the last frame's lists and statistics are kept (a call's last launch)
    // Poses after frame traj_first + j traj_every, j < traj_count: row j of traj, [n][7].
    float* traj;
    uint32_t traj_first, traj_every, traj_count;
    // State before frame ckpt_first + j ckpt_every: rows [13][n] at j of ckpt.
    float* ckpt;
    uint32_t ckpt_first, ckpt_every;
    dyph_aabb bounds;  // of a single scene (Morton codes of bodies with NaN boxes about)
};

// Phases of a scene's fused frame, timed per scene by its team leader when
// phase_ns is set: 0 staging + integrate + leaf boxes, 1 pair search,
// 2 narrowphase, 3 contact-solve set-up (lists, colours or levels, groups),
// 4 sweep + renormalisation, 5 write-back.
constexpr int kFramePhases = 6;

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void phase_mark(const Team& T, const FrameParams& P_, int k, uint64_t& t0) {
    if (P_.phase_ns && T.leader()) {
        const uint64_t t = global_ns();
        atomicAdd(&P_.phase_ns[k], static_cast<unsigned long long>(t - t0));
        t0 = t;
    }
}

// Recording for the adjoint pass (frame_scene with `adj`): the frame is
// recomputed from the given state, its branches and intermediates recorded,
// and nothing is reported; the end state goes to `store` when it is set (the
// given state is left as it was).
struct AdjRun {
    float* rec;          // [kRecWords][rec_stride] per-contact records, slot = contact slot of the scene
    uint32_t rec_stride;
    float* pose1;        // [7][n_stride] pose after integrate (x, q)
    float* qs;           // [4][n_stride] quaternions after the sweeps, before the renormalisations
    uint32_t n_stride;
    uint32_t* flag;      // unsupported paths
    float* store;        // [13][n_stride] the frame's end state (x, q, v, w), or null
};

// The 13 state rows of a scene's bodies into a [13][stride] buffer.
__device__ __forceinline__ void scene_store_state(const Team& T, float* out, uint32_t stride, uint32_t b0, uint32_t nb,
                                                  const SceneBodies& SB) {
    for (uint32_t i = T.rank(); i < nb; i += T.size()) {
        const float v[13] = {SB.px(i), SB.py(i), SB.pz(i), SB.qw(i), SB.qx(i), SB.qy(i), SB.qz(i),
                             SB.vx(i), SB.vy(i), SB.vz(i), SB.wx(i), SB.wy(i), SB.wz(i)};
#pragma unroll
        for (int r = 0; r < 13; ++r) out[static_cast<size_t>(r) * stride + b0 + i] = v[r];
    }
}

// The .trajectory rows (x, y, z, w, qx, qy, qz per body,
// examples/stress_test_blocks/main.cpp:191-197) of a scene's bodies.
__device__ __forceinline__ void scene_store_poses(const Team& T, float* out, uint32_t nb, const SceneBodies& SB) {
    for (uint32_t i = T.rank(); i < nb; i += T.size()) {
        const float v[7] = {SB.px(i), SB.py(i), SB.pz(i), SB.qw(i), SB.qx(i), SB.qy(i), SB.qz(i)};
#pragma unroll
        for (int r = 0; r < 7; ++r) out[7u * i + r] = v[r];
    }
}

// What the adjoint pass needs of a recomputed frame.
struct FrameOut {
    SceneContacts SC;
    uint32_t m, groups;
};

__device__ __forceinline__ bool pair_box_nan(uint4 b) {
    const __half2 x = half2_bits(b.x), y = half2_bits(b.y), z = half2_bits(b.z);
    return (__heq2_mask(x, x) & __heq2_mask(y, y) & __heq2_mask(z, z)) != 0xFFFFFFFFu;
}

// The pair box of leaf i as a walk of the tree meets it. The walk reaches a leaf
// below nodes that all overlap the query, and a node's box leaves out the NaN
// bounds among its leaves: a NaN bound of the leaf is held to the tightest bound of
// the nodes above it, the least (pair boxes negate the upper bounds) among the bodies
// whose keys share the longest prefix with the leaf's and whose bound is a number.
// The leaf's other bounds lie inside its ancestors'. code: Morton codes in the w
// words of `reach`.
__device__ __forceinline__ uint4 reach_box(const uint4* box, const uint4* reach, uint32_t nb, uint32_t i) {
    uint32_t out[3] = {box[i].x, box[i].y, box[i].z};
    const uint64_t key = (static_cast<uint64_t>(reach[i].w) << 32) | i;
#pragma unroll
    for (int h = 0; h < 6; ++h) {
        const int sh = 16 * (h & 1);
        if (!__hisnan(__ushort_as_half(static_cast<unsigned short>(out[h >> 1] >> sh)))) continue;
        int prefix = -1;
        float least = 0.f;
        for (uint32_t x = 0; x < nb; ++x) {
            const uint32_t w = h < 2 ? box[x].x : (h < 4 ? box[x].y : box[x].z);
            const float v = h2f_bits(static_cast<uint16_t>(w >> sh));
            if (isnan(v)) continue;
            const int c = __clzll(static_cast<long long>(key ^ ((static_cast<uint64_t>(reach[x].w) << 32) | x)));
            least = c > prefix ? v : (c == prefix ? fminf(least, v) : least);
            prefix = max(prefix, c);
        }
        if (prefix >= 0) out[h >> 1] = (out[h >> 1] & (0xFFFF0000u >> sh)) | (static_cast<uint32_t>(f2h_bits(least)) << sh);
    }
    return make_uint4(out[0], out[1], out[2], reach[i].w);
}

// Frame f of P_.n_frames of scene s by team T with `smem_bytes` of shared
// memory at smem. The first frame loads the scene's bodies, the next ones find
// them in shared memory as the frame before left them, and the last one writes
// them back; the lists in global memory and the solver's statistics are those
// of a call's last frame, so the frames before it do not write them.
// Returns false after raising an error. kRecord compiles the adjoint's
// recording in (`adj_in`, `out`); the forward frame is built without it.
// kPart: kFrameScene a frame of a batch's scene; kFrameSingle of a world's only
// scene, which returns false with sh.nan set when a leaf box holds a NaN; kFrameNan
// the rest of such a frame (see reach_box).
constexpr int kFrameScene = 0, kFrameSingle = 1, kFrameNan = 2;
template <bool kRecord, bool kAhead, int kPart = kFrameScene>
__device__ bool frame_scene(Team& T, uint32_t s, uint32_t f, unsigned char* smem, uint32_t smem_bytes,
                            SceneShared& sh, const SceneBufs& S, const FrameBufs& F, const FrameParams& P_,
                            const AdjRun* adj_in = nullptr, FrameOut* out = nullptr) {
    const bool end = f + 1u == P_.n_frames, last = end && P_.keep;
    const AdjRun* const adj = kRecord ? adj_in : nullptr;
    const GlobalBodies B{P_.gb};
    const uint32_t lane = threadIdx.x & 31u;
    uint64_t t0 = P_.phase_ns ? global_ns() : 0u;
    const uint32_t b0 = S.body_offset[s], nb = S.body_offset[s + 1] - b0;
    const uint32_t ldb = (nb + 3u) & ~3u;
    float* fb = reinterpret_cast<float*>(smem);
    const SceneSolverRows R = scene_solver_rows(fb, ldb);
    uint32_t* info = R.cnt + ldb;
    float* half = reinterpret_cast<float*>(info + ldb);
    uint4* box = reinterpret_cast<uint4*>(half + 3 * ldb);  // [ldb] pair boxes
    const SceneBodiesShaped SB{{fb, ldb}};
    const SceneShapes SS{info, half, ldb};
    const uint32_t pcap = F.pair_base[s + 1] - F.pair_base[s];
    const uint32_t ccap = F.contact_base[s + 1] - F.contact_base[s];
    // ── stage and integrate ──
    if (kPart != kFrameNan && f == 0u) {
        scene_load_bodies(T, B, b0, nb, fb, ldb);
        for (uint32_t i = T.rank(); i < nb; i += T.size()) {
            const uint32_t g = b0 + i, sh_i = P_.gb.shape[g];
            info[i] = P_.gs.type[sh_i] | (P_.gb.flags[g] << 8);
            half[i] = P_.gs.half_x[sh_i];
            half[ldb + i] = P_.gs.half_y[sh_i];
            half[2 * ldb + i] = P_.gs.half_z[sh_i];
        }
    }
    if (kPart != kFrameNan && !adj && P_.ckpt && f >= P_.ckpt_first && (f - P_.ckpt_first) % P_.ckpt_every == 0u) {
        const uint32_t j = (f - P_.ckpt_first) / P_.ckpt_every;
        scene_store_state(T, P_.ckpt + static_cast<size_t>(j) * 13u * P_.gb.n, P_.gb.n, b0, nb, SB);
    }
    for (uint32_t i = T.rank(); kPart != kFrameNan && i < nb; i += T.size()) {
        if (SB.im(i) != 0.f && !((info[i] >> 8) & kFlagSleeping)) {
            Pose p{SB.px(i), SB.py(i), SB.pz(i), SB.qw(i), SB.qx(i), SB.qy(i), SB.qz(i),
                   SB.vx(i), SB.vy(i), SB.vz(i)};
            const float ox = SB.wx(i), oy = SB.wy(i), oz = SB.wz(i);
            for (int k = 0; k < P_.n_substeps; ++k)
                integrate_body(p, ox, oy, oz, P_.gx, P_.gy, P_.gz, P_.sub_dt, P_.half_dt);
            SB.px(i) = p.px; SB.py(i) = p.py; SB.pz(i) = p.pz;
            SB.qw(i) = p.qw; SB.qx(i) = p.qx; SB.qy(i) = p.qy; SB.qz(i) = p.qz;
            SB.vx(i) = p.vx; SB.vy(i) = p.vy; SB.vz(i) = p.vz;
        }
        if (adj) {
            float* r = adj->pose1 + b0 + i;
            const float v[7] = {SB.px(i), SB.py(i), SB.pz(i), SB.qw(i), SB.qx(i), SB.qy(i), SB.qz(i)};
            for (int j = 0; j < 7; ++j) r[static_cast<size_t>(j) * adj->n_stride] = v[j];
        }
        box[i] = pair_box(leaf_box(SS.type(i), SB.px(i), SB.py(i), SB.pz(i), SB.qw(i), SB.qx(i), SB.qy(i), SB.qz(i),
                                   SS.hx(i), SS.hy(i), SS.hz(i)));
        if (kPart == kFrameSingle && pair_box_nan(box[i])) sh.nan = 1u;
        R.cnt[i] = 0u;
    }
    T.sync();
    phase_mark(T, P_, 0, t0);
    if (kPart == kFrameSingle && sh.nan != 0u) return false;
    uint4* reach = reinterpret_cast<uint4*>(R.mask);  // [ldb], over the masks and priorities of the solve
    if (kPart == kFrameNan) {
        for (uint32_t i = T.rank(); i < nb; i += T.size())
            reach[i] = make_uint4(box[i].x, box[i].y, box[i].z, morton_code(SB.px(i), SB.py(i), SB.pz(i), P_.bounds));
        T.sync();
        for (uint32_t i = T.rank(); i < nb; i += T.size())
            if (pair_box_nan(box[i])) reach[i] = reach_box(box, reach, nb, i);
        T.sync();
    }
    // ── candidate pairs: per body a, the partners b > a in ascending order ──
    // Every (a, b) is tested: a lane holds one body a and meets 32 partners one
    // after another, whose boxes the warp reads as broadcasts; the answers are
    // the bits of one word and nothing waits inside the 32. A warp takes 32
    // bodies and 32 partners at a time, so the triangle of pairs is split evenly
    // over the team. Alone on its SM a 512-body scene takes 30 us for this phase
    // and a 256-body one 10 us; with a warp on one body and a ballot per 32
    // partners, each waiting for six loads, they took 222 and 64 us.
    // The words go to the end of the team's shared memory when they fit there,
    // so the write pass reads them instead of testing the boxes again.
    const uint32_t chunks = overlap_chunks(nb), mask_words = overlap_mask_base(chunks);
    const uint32_t mask_off = (smem_bytes - 4u * mask_words) & ~15u;
    const bool keep_masks = 4u * mask_words <= smem_bytes && frame_body_bytes(nb) <= mask_off;
    uint32_t* masks = reinterpret_cast<uint32_t*>(smem + mask_off);
    // word (c, a) of this lane's a; partners past the scene's end do not overlap
    auto overlap_word = [&](uint32_t c, uint32_t a, const uint3& q) -> uint32_t {
        const uint32_t n_b = min(32u, nb - 32u * c);
        uint32_t w = 0;
        if (kPart == kFrameNan) {
            // the later leaf in Morton order (of equal codes the larger index) walks to the earlier one
            const uint32_t me = min(a, nb - 1u);
            const uint4 mine = reach[me];
            for (uint32_t j = 0; j < n_b; ++j) {
                const uint32_t b = 32u * c + j;
                const bool ov = mine.w > reach[b].w ? pair_overlap(reach[b], q) : pair_overlap(mine, facing_box(box[b]));
                w |= ov ? 1u << j : 0u;
            }
        } else if (n_b == 32u) {
#pragma unroll 8
            for (uint32_t j = 0; j < 32u; ++j) w |= pair_overlap(box[32u * c + j], q) ? 1u << j : 0u;
        } else {
#pragma unroll 4
            for (uint32_t j = 0; j < n_b; ++j) w |= pair_overlap(box[32u * c + j], q) ? 1u << j : 0u;
        }
        if ((a >> 5) == c) w &= ~((2u << lane) - 1u);  // b > a
        return a < nb ? w : 0u;
    };
    for (uint32_t c = 0, ga = T.warp();; ga += T.warps()) {
        while (c < chunks && ga > c) ga -= ++c;  // chunk c meets body groups 0..c
        if (c >= chunks) break;
        const uint32_t a = 32u * ga + lane;
        const uint32_t w = overlap_word(c, a, facing_box(box[min(a, nb - 1u)]));
        if (keep_masks) masks[overlap_mask_base(c) + a] = w;
        if (w) atomicAdd(&R.cnt[a], __popc(w));
    }
    T.sync();
    uint32_t p_true = 0;
    for (uint32_t base = 0; base < nb; base += T.size()) {
        const uint32_t i = base + T.rank();
        const uint32_t v = i < nb ? R.cnt[i] : 0u;
        uint32_t tot;
        const uint32_t ex = T.exclusive_scan(v, sh.scan, tot);
        if (i < nb) R.off[i] = p_true + ex;
        p_true += tot;
    }
    T.sync();
    const uint32_t P = min(p_true, pcap);
    // ── layout of the pairs and the contact words: shared memory if they fit ──
    const uint32_t cc = min(P, ccap);
    const uint32_t ldc = (cc + 4u) & ~3u;  // >= cc + 1: group offsets take m + 1 words
    const uint32_t pwords = (P + 3u) & ~3u;
    const uint32_t body_bytes = frame_body_bytes(nb);
    const bool in_smem = body_bytes + 4u * pwords + kSceneWords * 4u * ldc <= smem_bytes;
    uint32_t* pairs = in_smem ? reinterpret_cast<uint32_t*>(smem + body_bytes) : F.pair_raw + F.pair_base[s];
    const SceneContacts SC{in_smem ? reinterpret_cast<uint32_t*>(smem + body_bytes) + pwords
                                   : F.words + F.contact_base[s] + s,
                           in_smem ? ldc : F.words_stride};
    // the masks survive the write pass unless the pairs themselves reach them
    const bool use_masks = keep_masks && (!in_smem || body_bytes + 4u * pwords <= mask_off);
    // a lane writes its body's partners; a word with many (a ground that comes
    // first meets everything) is written by the whole warp
    for (uint32_t ga = T.warp(); ga < chunks; ga += T.warps()) {
        const uint32_t a = 32u * ga + lane;
        const uint3 q = facing_box(box[min(a, nb - 1u)]);
        uint32_t pos = a < nb ? R.off[a] : 0u;
        for (uint32_t c = ga; c < chunks; ++c) {
            uint32_t w = use_masks ? masks[overlap_mask_base(c) + a] : overlap_word(c, a, q);
            for (unsigned many = __ballot_sync(0xffffffffu, __popc(w) > 8); many; many &= many - 1u) {
                const int src = __ffs(static_cast<int>(many)) - 1;
                const uint32_t wa = __shfl_sync(0xffffffffu, w, src), at0 = __shfl_sync(0xffffffffu, pos, src);
                const uint32_t at = at0 + __popc(wa & ((1u << lane) - 1u));
                if (((wa >> lane) & 1u) && at < P) pairs[at] = (32u * ga + src) | ((32u * c + lane) << 16);
                if (static_cast<int>(lane) == src) {
                    pos += __popc(w);
                    w = 0u;
                }
            }
            for (; w; w &= w - 1u, ++pos)
                if (pos < P) pairs[pos] = a | ((32u * c + static_cast<uint32_t>(__ffs(static_cast<int>(w))) - 1u) << 16);
        }
    }
    T.sync();
    if (in_smem && !adj && last)
        for (uint32_t p = T.rank(); p < P; p += T.size()) F.pair_raw[F.pair_base[s] + p] = pairs[p];
    phase_mark(T, P_, 1, t0);
    // ── narrowphase: contacts in pair order ──
    for (uint32_t i = T.rank(); i < nb; i += T.size()) R.cnt[i] = 0u;
    if (kPart == kFrameNan && T.leader()) sh.nan = 0u;
    T.sync();
    uint32_t m_true = 0;
    const uint32_t cbase = F.contact_base[s];
    for (uint32_t base = 0; base < P; base += T.size()) {
        const uint32_t p = base + T.rank();
        Contact c{};
        bool hit = false;
        uint32_t br = 0u;
        if (p < P) {
            const uint32_t ab = pairs[p];
            hit = process_pair(SB, SS, ab & 0xFFFFu, ab >> 16, c, adj ? &br : nullptr);
        }
        uint32_t tot;
        const uint32_t k = m_true + T.count_before(hit, sh.scan, tot);
        m_true += tot;
        if (hit && k < cc) {
            SC.ab(k) = c.a | (c.b << 16);
            SC.lam(k) = 0.f;
            SC.pb(k) = kSceneNone;
            SC.g(0, k) = c.px; SC.g(1, k) = c.py; SC.g(2, k) = c.pz;
            SC.g(3, k) = c.nx; SC.g(4, k) = c.ny; SC.g(5, k) = c.nz;
            SC.g(6, k) = c.depth;
            if (SB.im(c.b) != 0.f) atomicAdd(&R.cnt[c.b], 1u);
            const uint32_t slot = cbase + k, st = F.contact_slots;
            if (adj) {
                adj->rec[27ull * adj->rec_stride + slot] = __uint_as_float(br);
            } else if (last) {
                F.contact_raw[slot] = b0 + c.a;
                F.contact_raw[st + slot] = b0 + c.b;
                F.contact_raw[2 * st + slot] = __float_as_uint(c.px);
                F.contact_raw[3 * st + slot] = __float_as_uint(c.py);
                F.contact_raw[4 * st + slot] = __float_as_uint(c.pz);
                F.contact_raw[5 * st + slot] = __float_as_uint(c.nx);
                F.contact_raw[6 * st + slot] = __float_as_uint(c.ny);
                F.contact_raw[7 * st + slot] = __float_as_uint(c.nz);
                F.contact_raw[8 * st + slot] = __float_as_uint(c.depth);
            }
        }
    }
    const uint32_t m = min(m_true, cc);
    T.sync();
    if (T.leader() && !adj) {
        if (last) {
            F.counts[4 * s + 0] = P;
            F.counts[4 * s + 1] = p_true;
            F.counts[4 * s + 2] = m;
            F.counts[4 * s + 3] = m_true;
        }
        atomicAdd(&P_.counts[f], P);
        atomicAdd(&P_.counts[P_.n_frames + f], p_true);
        atomicAdd(&P_.counts[2u * P_.n_frames + f], m);
        atomicAdd(&P_.counts[3u * P_.n_frames + f], m_true);
        // a scene past its own capacity keeps its ordered prefix, as it does alone
        const uint32_t over = (p_true > pcap ? 1u : 0u) | (m_true > ccap ? 2u : 0u);
        if (over) atomicOr(&P_.counts[4u * P_.n_frames + f], over);
    }
    phase_mark(T, P_, 2, t0);
    // ── contact solve (none without contacts, as the reference's solve returns) ──
    bool colored = false;
    uint32_t n_colors = 0, rounds = 0, groups = 0;
    if (m > 0) {
        SolveRecord rec{};
        if (adj) rec = SolveRecord{adj->rec, adj->rec_stride, cbase, adj->qs, adj->n_stride, b0, adj->flag};
        uint64_t t_sweep = 0;
        if (!scene_solve<kRecord, kAhead>(T, nb, m, SB, R, SC, P_.mode, P_.n_iters, P_.mu, P_.dt, sh, colored, n_colors, rounds,
                         adj ? &rec : nullptr, &groups, P_.phase_ns ? &t_sweep : nullptr))
            return false;
        if (P_.phase_ns && T.leader()) {
            atomicAdd(&P_.phase_ns[3], static_cast<unsigned long long>(t_sweep - t0));
            t0 = t_sweep;
        }
        if (!adj && last) {
            for (uint32_t k = T.rank(); k < m; k += T.size())
                F.color_raw[cbase + k] = colored ? SC.done(k) : kUncolored;
            if (T.leader()) {
                if (colored) {
                    atomicMax(&P_.acc[kAccMaxColor], n_colors);
                    P_.acc[kAccColored] = 1u;
                }
                atomicMax(&P_.acc[kAccRounds], rounds);
                P_.acc[kAccSolved] = 1u;
            }
        }
    }
    if (out) *out = FrameOut{SC, m, groups};
    phase_mark(T, P_, 4, t0);
    if (!adj) {
        if (P_.traj && f >= P_.traj_first && (f - P_.traj_first) % P_.traj_every == 0u) {
            const uint32_t j = (f - P_.traj_first) / P_.traj_every;
            if (j < P_.traj_count)
                scene_store_poses(T, P_.traj + (static_cast<size_t>(j) * P_.gb.n + b0) * 7u, nb, SB);
        }
        if (end) scene_store_bodies(T, B, b0, nb, SB);
    } else if (adj->store) {
        scene_store_state(T, adj->store, adj->n_stride, b0, nb, SB);
    }
    T.sync();
    phase_mark(T, P_, 5, t0);
    return true;
}

// All frames of the launch of scene s: scenes do not depend on one another, so
// a team takes its scene from frame to frame without waiting for the others.
template <bool kAhead>
__device__ __forceinline__ void run_scene(Team T, uint32_t s, unsigned char* smem, uint32_t smem_bytes,
                                          SceneShared& sh, const SceneBufs& S, const FrameBufs& F,
                                          const FrameParams& P_) {
    for (uint32_t f = 0; f < P_.n_frames; ++f)
        if (!frame_scene<false, kAhead>(T, s, f, smem, smem_bytes, sh, S, F, P_)) return;
}

// Work item i: items[4 i] a large scene solved by the whole block when
// items[4 i + 1] == kItemBlock; two mid-size scenes items[4 i] and
// items[4 i + 2], half the block and its shared memory each, when
// items[4 i + 1] == kItemHalf; otherwise up to four small scenes, a quarter of
// the block and its shared memory each. kItemEmpty marks an unused team.
constexpr uint32_t kItemEmpty = 0xFFFFFFFFu;
constexpr uint32_t kItemBlock = 0xFFFFFFFEu;
constexpr uint32_t kItemHalf = 0xFFFFFFFDu;

// The calling thread's team of a work item: its scene, its part of the block's
// shared memory and which of the block's SceneShared it uses.
struct ItemTeam {
    Team team;
    uint32_t scene, smem, bytes, shared;
};
__device__ __forceinline__ ItemTeam item_team(const uint32_t* item, uint32_t smem_bytes) {
    const uint32_t kind = item[1], share = (smem_bytes / 4u) & ~15u;
    if (kind == kItemBlock) return ItemTeam{Team{blockDim.x, 0u}, item[0], 0u, smem_bytes, 0u};
    const uint32_t quarter = threadIdx.x / (blockDim.x / 4u);
    if (kind == kItemHalf) {
        const uint32_t half = quarter >> 1;
        return ItemTeam{Team{blockDim.x / 2u, 1u + half}, item[2 * half], half * 2u * share, 2u * share, 2u * half};
    }
    return ItemTeam{Team{blockDim.x / 4u, 3u + quarter}, item[quarter], quarter * share, share, quarter};
}

// kMinBlocks is the register budget: 4 resident blocks of kSceneThreads per SM
// (128 registers a thread), 5 (96, 88 bytes of them spilled) or 6 (80, 112), or 2 of
// kSceneWideThreads (128). Which one runs best depends on the batch
// (dyph_world_autotune picks the budget with the shared memory cap; the wide
// form's rule is in setup_fused); all compute the same frames.
template <int kMinBlocks, int kThreads>
__global__ void __launch_bounds__(kThreads, kMinBlocks) scene_frame_kernel(SceneBufs S, FrameBufs F, FrameParams P_,
                                                                           const uint32_t* __restrict__ items,
                                                                           uint32_t n_items) {
    extern __shared__ __align__(16) unsigned char scene_smem[];
    __shared__ SceneShared sh[4];
    for (uint32_t it = blockIdx.x; it < n_items; it += gridDim.x) {
        const ItemTeam t = item_team(items + 4 * it, S.smem_bytes);
        if (t.scene != kItemEmpty)
            run_scene<kThreads == kSceneWideThreads>(t.team, t.scene, scene_smem + t.smem, t.bytes, sh[t.shared], S, F, P_);
        __syncthreads();
    }
}

// A single scene's frame with a NaN among its boxes, from the pairs on. Apart, so that
// the frames without one do not carry its code (they took 1.4 us longer with it, of 17
// on 9 boxes). Returns the team's turn, + 2 when the frame is done.
__device__ __noinline__ uint32_t nan_frame(Team T, uint32_t f, unsigned char* smem, uint32_t smem_bytes,
                                           SceneShared& sh, const SceneBufs& S, const FrameBufs& F,
                                           const FrameParams& P_) {
    const bool ok = frame_scene<false, true, kFrameNan>(T, 0u, f, smem, smem_bytes, sh, S, F, P_);
    return T.turn | (ok ? 2u : 0u);
}

// The frames of a world's only scene, on one block of kThreads.
template <int kThreads>
__global__ void __launch_bounds__(kThreads, 2) scene_single_kernel(const __grid_constant__ SceneBufs S,
                                                                   const __grid_constant__ FrameBufs F,
                                                                   const __grid_constant__ FrameParams P_) {
    extern __shared__ __align__(16) unsigned char scene_smem[];
    __shared__ SceneShared sh;
    if (threadIdx.x == 0) sh.nan = 0u;
    __syncthreads();
    Team T{kThreads, 0u};
    for (uint32_t f = 0; f < P_.n_frames; ++f) {
        if (frame_scene<false, true, kFrameSingle>(T, 0u, f, scene_smem, S.smem_bytes, sh, S, F, P_)) continue;
        if (sh.nan == 0u) return;
        const uint32_t r = nan_frame(T, f, scene_smem, S.smem_bytes, sh, S, F, P_);
        T.turn = r & 1u;
        if ((r & 2u) == 0u) return;
    }
}

// Exclusive scans of the scenes' stored pair / contact counts (one block):
// pos[2 s] / pos[2 s + 1] = first compacted pair / contact of scene s, and the
// totals into the broadphase / narrowphase stored-count words.
__global__ void __launch_bounds__(1024) scene_gather_scan_kernel(const uint32_t* __restrict__ counts,
                                                                 uint32_t n_scenes, uint32_t* __restrict__ pos,
                                                                 uint32_t* __restrict__ bp_counts,
                                                                 uint32_t* __restrict__ np_counts) {
    __shared__ uint32_t s_scan[32];
    __shared__ uint32_t carry[2];
    if (threadIdx.x < 2) carry[threadIdx.x] = 0u;
    __syncthreads();
    for (uint32_t base = 0; base < n_scenes; base += blockDim.x) {
        const uint32_t s = base + threadIdx.x;
        for (int w = 0; w < 2; ++w) {
            const uint32_t v = s < n_scenes ? counts[4 * s + 2 * w] : 0u;
            uint32_t tot;
            const uint32_t ex = block_exclusive_scan<1024>(v, s_scan, tot);
            if (s < n_scenes) pos[2 * s + w] = carry[w] + ex;
            __syncthreads();
            if (threadIdx.x == 0) carry[w] += tot;
            __syncthreads();
        }
    }
    if (threadIdx.x == 0) {
        bp_counts[0] = carry[0];
        np_counts[0] = carry[1];
    }
}

// Copy every scene's pairs (as global body indices), contacts and colours to
// their compacted positions (one block per scene).
__global__ void scene_gather_copy_kernel(SceneBufs S, FrameBufs F, const uint32_t* __restrict__ pos,
                                         dyph_pair* __restrict__ pairs, dyph_contacts cv,
                                         uint32_t* __restrict__ color) {
    const uint32_t s = blockIdx.x;
    if (s >= S.n_scenes) return;
    const uint32_t b0 = S.body_offset[s];
    const uint32_t np_ = F.counts[4 * s + 0], nc = F.counts[4 * s + 2];
    const uint32_t p0 = pos[2 * s], c0 = pos[2 * s + 1];
    for (uint32_t p = threadIdx.x; p < np_; p += blockDim.x) {
        const uint32_t ab = F.pair_raw[F.pair_base[s] + p];
        pairs[p0 + p] = dyph_pair{b0 + (ab & 0xFFFFu), b0 + (ab >> 16)};
    }
    const uint32_t st = F.contact_slots, cb = F.contact_base[s];
    float* rows[7] = {cv.pos_x, cv.pos_y, cv.pos_z, cv.norm_x, cv.norm_y, cv.norm_z, cv.depth};
    for (uint32_t k = threadIdx.x; k < nc; k += blockDim.x) {
        cv.body_a[c0 + k] = F.contact_raw[cb + k];
        cv.body_b[c0 + k] = F.contact_raw[st + cb + k];
#pragma unroll
        for (int r = 0; r < 7; ++r) rows[r][c0 + k] = __uint_as_float(F.contact_raw[(2 + r) * st + cb + k]);
        color[c0 + k] = F.color_raw[cb + k];
    }
}

}  // namespace
}  // namespace dyph
