// Batched scenes (included by solver.cu): one thread block solves one scene,
// the scene's bodies staged in shared memory.
//
// The reference solves one scene per XpbdSolver::solve (xpbd_solver.cpp:
// 603-733). A batch is many independent scenes, so each block takes one scene
// and runs exactly that solve on it:
//   * the scene's contacts are a contiguous run of the contact list (pairs are
//     sorted by body a and a scene's bodies are contiguous), local contact
//     index k = global index - first index;
//   * a scene without contacts is left alone (the reference returns before
//     any renormalisation when n_con == 0);
//   * sequential order (set_force_serial, or n_con <= 256 in the reference
//     mode, or a colouring that needs more than 64 colours or 256 rounds):
//     contacts are solved in waves, contact k as soon as the previous contact
//     of each of its dynamic bodies (in contact order) is solved — the serial
//     loop's per-body order, so the result is bit-identical to it;
//   * coloured order: Jones–Plassmann rounds with the priorities
//     hash(k) << 32 | k of the local index (:645-688), then colour by colour;
//   * every iteration renormalises every body of the scene (:579-584,
//     :726-731); a contact deferred at w_total < 1e-10 is retried by the next
//     iteration's sweep, as in the reference.
// Each scene therefore evolves bit for bit as it does stepped alone in the
// same mode. Waves and rounds are separated by block barriers; a scene whose
// chain of dependent contacts is d long takes d waves.
#pragma once

#include "solver_common.cuh"

namespace dyph {
namespace {

constexpr int kSceneThreads = 128;      // threads of a block
constexpr int kSceneWideThreads = 256;  // of the fused frame's larger form
constexpr uint32_t kSceneNone = 0xFFFFFFFFu;
constexpr uint32_t kSceneWords = 13;         // per-contact words (see SceneContacts)
constexpr uint32_t kSceneMaxBodies = 65535;  // local body indices are 16 bits

// Shared-memory bytes of a scene's body part (see the layout in scene_solve_kernel).
__host__ __device__ __forceinline__ uint32_t scene_body_bytes(uint32_t nb) {
    const uint32_t ldb = (nb + 3u) & ~3u;
    return 20u * 4u * ldb + 8u * ldb + 2u * 4u * ldb + 4u * (ldb + 4u) + 4u * ldb;
}

struct SceneBufs {
    const uint32_t* body_offset;  // [n_scenes + 1] first body of each scene
    const uint32_t* scene_of;     // [n] scene of each body
    const uint32_t* order;        // [n_scenes] scenes by descending body count (largest first)
    uint32_t* range;              // [2 n_scenes] first / one-past-last contact of each scene
    uint32_t* scratch;            // [kSceneWords][scratch_stride] per-contact words of scenes too big for shared memory
    uint32_t scratch_stride;      // max contacts + n_scenes (one extra word per scene)
    uint32_t n_scenes;
    uint32_t smem_bytes;          // dynamic shared memory of one block
};

// First and one-past-last contact of every scene (range cleared to 0 first).
__global__ void scene_range_kernel(dyph_contacts cv, SceneBufs S) {
    const uint32_t nc = contact_count(cv);
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < nc; c += gridDim.x * blockDim.x) {
        const uint32_t s = S.scene_of[cv.body_a[c]];
        if (c == 0 || S.scene_of[cv.body_a[c - 1]] != s) S.range[2 * s] = c;
        if (c + 1 == nc || S.scene_of[cv.body_a[c + 1]] != s) S.range[2 * s + 1] = c + 1;
    }
}

// Body rows of one scene in shared memory: row r of local body i at f[r * ld + i].
// Rows 0-12 state, 13 inverse mass, 14-19 inverse inertia.
struct SceneBodies {
    float* f;
    uint32_t ld;
    __device__ __forceinline__ float& px(uint32_t i) const { return f[0 * ld + i]; }
    __device__ __forceinline__ float& py(uint32_t i) const { return f[1 * ld + i]; }
    __device__ __forceinline__ float& pz(uint32_t i) const { return f[2 * ld + i]; }
    __device__ __forceinline__ float& qw(uint32_t i) const { return f[3 * ld + i]; }
    __device__ __forceinline__ float& qx(uint32_t i) const { return f[4 * ld + i]; }
    __device__ __forceinline__ float& qy(uint32_t i) const { return f[5 * ld + i]; }
    __device__ __forceinline__ float& qz(uint32_t i) const { return f[6 * ld + i]; }
    __device__ __forceinline__ float& vx(uint32_t i) const { return f[7 * ld + i]; }
    __device__ __forceinline__ float& vy(uint32_t i) const { return f[8 * ld + i]; }
    __device__ __forceinline__ float& vz(uint32_t i) const { return f[9 * ld + i]; }
    __device__ __forceinline__ float& wx(uint32_t i) const { return f[10 * ld + i]; }
    __device__ __forceinline__ float& wy(uint32_t i) const { return f[11 * ld + i]; }
    __device__ __forceinline__ float& wz(uint32_t i) const { return f[12 * ld + i]; }
    __device__ __forceinline__ float im(uint32_t i) const { return f[13 * ld + i]; }
    __device__ __forceinline__ float ixx(uint32_t i) const { return f[14 * ld + i]; }
    __device__ __forceinline__ float iyy(uint32_t i) const { return f[15 * ld + i]; }
    __device__ __forceinline__ float izz(uint32_t i) const { return f[16 * ld + i]; }
    __device__ __forceinline__ float ixy(uint32_t i) const { return f[17 * ld + i]; }
    __device__ __forceinline__ float ixz(uint32_t i) const { return f[18 * ld + i]; }
    __device__ __forceinline__ float iyz(uint32_t i) const { return f[19 * ld + i]; }
};

// Per-contact words of one scene (shared memory, or the global scratch for
// a scene with too many contacts): row r of local contact k at w[r * ld + k].
//   0 a | b << 16 (local body indices)   1 predecessor on a   2 predecessor on b
//   3 wave solved in / colour            4 b-side list entry   5 lambda
//   6-12 position xyz, normal xyz, depth (copied from the contact list)
struct SceneContacts {
    uint32_t* w;
    uint32_t ld;
    __device__ __forceinline__ uint32_t& ab(uint32_t k) const { return w[k]; }
    __device__ __forceinline__ uint32_t& pa(uint32_t k) const { return w[1 * ld + k]; }
    __device__ __forceinline__ uint32_t& pb(uint32_t k) const { return w[2 * ld + k]; }
    __device__ __forceinline__ uint32_t& done(uint32_t k) const { return w[3 * ld + k]; }
    __device__ __forceinline__ uint32_t& ent(uint32_t k) const { return w[4 * ld + k]; }
    __device__ __forceinline__ float& lam(uint32_t k) const { return reinterpret_cast<float*>(w)[5 * ld + k]; }
    __device__ __forceinline__ float& g(int r, uint32_t k) const { return reinterpret_cast<float*>(w)[(6 + r) * ld + k]; }
    __device__ __forceinline__ Contact contact(uint32_t k) const {
        Contact ct;
        const uint32_t ab_k = ab(k);
        ct.a = ab_k & 0xFFFFu;
        ct.b = ab_k >> 16;
        ct.px = g(0, k); ct.py = g(1, k); ct.pz = g(2, k);
        ct.nx = g(3, k); ct.ny = g(4, k); ct.nz = g(5, k);
        ct.depth = g(6, k);
        return ct;
    }
};

// A team of threads that runs one scene: the whole block (big scenes), half of
// it or a quarter (small scenes, several to a block). The size is a run-time
// value, so that a kernel holds one copy of a frame's code: the teams of an SM
// are in different phases of their frames, and a copy per kind of team pushed
// one another out of the instruction cache. Teams are aligned to their size;
// `bar` is the team's named barrier (0 the block's own, 1 and 2 the halves', 3
// to 6 the quarters'; immediate ids, so that a kernel reserves seven).
struct Team {
    uint32_t n, bar;
    uint32_t turn = 0;  // which scratch words the next scan takes
    __device__ __forceinline__ uint32_t rank() const { return threadIdx.x & (n - 1u); }
    __device__ __forceinline__ uint32_t size() const { return n; }
    __device__ __forceinline__ uint32_t warp() const { return rank() >> 5; }
    __device__ __forceinline__ uint32_t warps() const { return n >> 5; }
    __device__ __forceinline__ bool leader() const { return rank() == 0u; }
    __device__ __forceinline__ void sync() const {
        if (n == 32u) {
            __syncwarp();
            return;
        }
        switch (bar) {
            case 0: __syncthreads(); break;
            case 1: asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory"); break;
            case 2: asm volatile("bar.sync 2, %0;" ::"r"(n) : "memory"); break;
            case 3: asm volatile("bar.sync 3, %0;" ::"r"(n) : "memory"); break;
            case 4: asm volatile("bar.sync 4, %0;" ::"r"(n) : "memory"); break;
            case 5: asm volatile("bar.sync 5, %0;" ::"r"(n) : "memory"); break;
            default: asm volatile("bar.sync 6, %0;" ::"r"(n) : "memory");
        }
    }
    // The exclusive prefix of v over the team and its total. A scan takes one
    // barrier: two halves of the scratch alternate, and a thread that writes a
    // half again has passed the barrier after everyone's reads of it.
    __device__ __forceinline__ uint32_t exclusive_scan(uint32_t v, uint32_t* scratch, uint32_t& total) {
        const uint32_t lane = threadIdx.x & 31u;
        uint32_t x = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= static_cast<uint32_t>(d)) x += y;
        }
        return finish_scan(x, x - v, scratch, total);
    }
    // The same of one bit per thread.
    __device__ __forceinline__ uint32_t count_before(bool p, uint32_t* scratch, uint32_t& total) {
        const uint32_t lane = threadIdx.x & 31u;
        const unsigned m = __ballot_sync(0xffffffffu, p);
        return finish_scan(__popc(m), __popc(m & ((1u << lane) - 1u)), scratch, total);
    }

private:
    // last: the warp's total in its last lane; before: the prefix inside the warp
    __device__ __forceinline__ uint32_t finish_scan(uint32_t last, uint32_t before, uint32_t* scratch,
                                                    uint32_t& total) {
        if (n == 32u) {
            total = __shfl_sync(0xffffffffu, last, 31);
            return before;
        }
        uint32_t* w = scratch + turn * (kSceneWideThreads / 32);
        turn ^= 1u;
        if ((threadIdx.x & 31u) == 31u) w[warp()] = last;
        sync();
        total = 0u;
        for (uint32_t i = 0; i < warps(); ++i) {
            if (i == warp()) before += total;
            total += w[i];
        }
        return before;
    }
};

// Levels of the sequential order on one scene: level(k) = 1 + the larger
// level of k's predecessors on its two dynamic bodies. Contacts of one level
// share no dynamic body, and solving the levels in ascending order gives
// every body its contacts in contact order: the serial loop's result, bit for
// bit. Levels go to SC.done (1-based); returns the level count, or 0 if the
// predecessor links were inconsistent (they cannot be: every predecessor has a
// lower index).
// A warp takes 32 consecutive contacts at a time and polls their predecessors'
// levels until it has them all; the warps of a team work on neighbouring
// contacts at once and meet at no barrier. The lowest unfinished contact can
// always be finished, and each warp goes through its contacts in ascending
// order, so the polls end. A pass over all contacts between barriers took a pass
// per level (25 us of set-up on a 256-body stack, 22 with polls); links inside a
// warp's 32 contacts go by shuffles (set-up of a push scene 12.6 -> 9.8 us).
__device__ uint32_t scene_levels(const Team& T, uint32_t m, const SceneContacts& SC, uint32_t* s_max) {
    for (uint32_t k = T.rank(); k < m; k += T.size()) SC.done(k) = 0u;
    if (T.leader()) *s_max = 0u;
    T.sync();
    uint32_t my_max = 0, spins = 0;
    volatile uint32_t* done = &SC.done(0);
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t k0 = T.rank() & ~31u; k0 < m; k0 += T.size()) {
        // a predecessor among the warp's 32 is read by a shuffle, an earlier one from its word
        const uint32_t k = k0 + lane;
        const bool mine = k < m;
        const uint32_t pa = mine ? SC.pa(k) : kSceneNone, pb = mine ? SC.pb(k) : kSceneNone;
        const bool in_a = pa != kSceneNone && pa >= k0, in_b = pb != kSceneNone && pb >= k0;
        bool wait_a = pa != kSceneNone && !in_a, wait_b = pb != kSceneNone && !in_b, open = mine;
        uint32_t level = 0, la = 0, lb = 0;
        while (__any_sync(0xffffffffu, open)) {
            if (wait_a) wait_a = (la = done[pa]) == 0u;
            if (wait_b) wait_b = (lb = done[pb]) == 0u;
            const uint32_t sa = __shfl_sync(0xffffffffu, level, static_cast<int>(in_a ? pa - k0 : lane));
            const uint32_t sb = __shfl_sync(0xffffffffu, level, static_cast<int>(in_b ? pb - k0 : lane));
            if (open && !wait_a && !wait_b && (!in_a || sa != 0u) && (!in_b || sb != 0u)) {
                level = max(in_a ? sa : la, in_b ? sb : lb) + 1u;
                done[k] = level;
                open = false;
            }
            if (++spins > kSpinLimit) break;
        }
        my_max = max(my_max, level);
        __syncwarp();
    }
    my_max = __reduce_max_sync(0xffffffffu, spins > kSpinLimit ? kSceneNone : my_max);
    if ((threadIdx.x & 31u) == 0u) atomicMax(s_max, my_max);
    T.sync();
    const uint32_t levels = *s_max;
    T.sync();
    return levels == kSceneNone ? 0u : levels;
}

// Counting sort of the scene's contacts by group done(k) - base (a level or a
// colour) into SC.ent; group g is SC.ent[SC.pa(g), SC.pa(g + 1)). The
// predecessor rows are free once the groups are known. *s_passes receives the
// groups' sixteens (see scene_sweep).
__device__ void scene_group(Team& T, uint32_t m, uint32_t groups, uint32_t base, const SceneContacts& SC,
                            uint32_t* s_scan, uint32_t* s_passes) {
    for (uint32_t g = T.rank(); g <= groups; g += T.size()) SC.pa(g) = 0u;
    if (T.leader()) *s_passes = 0u;
    T.sync();
    for (uint32_t k = T.rank(); k < m; k += T.size()) atomicAdd(&SC.pa(SC.done(k) - base), 1u);
    T.sync();
    uint32_t passes = 0;
    for (uint32_t g0 = 0, carry = 0; g0 <= groups; g0 += T.size()) {
        const uint32_t g = g0 + T.rank();
        const uint32_t v = g <= groups ? SC.pa(g) : 0u;
        passes += (v + 15u) >> 4;
        uint32_t tot;
        const uint32_t ex = T.exclusive_scan(v, s_scan, tot);
        if (g <= groups) {
            SC.pa(g) = carry + ex;
            SC.pb(g) = carry + ex;  // fill cursor
        }
        carry += tot;
    }
    passes = __reduce_add_sync(0xffffffffu, passes);
    if ((threadIdx.x & 31u) == 0u && passes) atomicAdd(s_passes, passes);
    T.sync();
    for (uint32_t k = T.rank(); k < m; k += T.size()) SC.ent(atomicAdd(&SC.pb(SC.done(k) - base), 1u)) = k;
    T.sync();
}

// What the adjoint pass records of a scene's solve (solve_record): for every
// contact that acts, both bodies' state before its solve and lambda; the
// quaternions before the renormalisations.
constexpr int kRecWords = 36;  // per-contact record rows (see SolveRecord)
struct SolveRecord {
    // rows r of contact k at rec[r * stride + base + k]: 0-12 body a state,
    // 13-25 body b state, 26 lambda before, 27 narrowphase branch word,
    // 28-34 contact geometry adjoint (point, normal, depth), 35 the solve's
    // branch flags (bits of a float; 0 when the contact did not act)
    float* rec;
    uint32_t stride, base;
    float* qs;           // [4][qs_stride] quaternions after the sweeps, at body b0 + i
    uint32_t qs_stride, b0;
    uint32_t* flag;      // set when the solve took a path the adjoint does not cover
};

__device__ __forceinline__ void record_state(float* r, uint32_t stride, const SideBody& S, int row0) {
    const float v[13] = {S.px, S.py, S.pz, S.qw, S.qx, S.qy, S.qz, S.vx, S.vy, S.vz, S.wx, S.wy, S.wz};
#pragma unroll
    for (int j = 0; j < 13; ++j) r[static_cast<size_t>(row0 + j) * stride] = v[j];
}

// One sweep over the groups in ascending order, one contact per lane pair at a
// time inside a group (no two of a group share a dynamic body): groups are
// narrow and their chain bounds the frame (see solve_contact_side). A sweep and
// its renormalisation took 70 us with a contact per lane on a 256-body stack
// alone on its SM, 44 us with a contact per lane pair; 41.6 and 27.9 us on the
// 66-body push scenes. kRecord compiles the recording in; without it `rec` is
// ignored. kAhead, for kernels whose warps have their scheduler to themselves:
// what does not depend on the group before (the next group's bounds, contact and
// constant body rows) is loaded ahead of the barrier, and when almost every
// group fits one warp (`passes`, the groups' sixteens, are hardly more than the
// groups) the first warp sweeps alone. On full SMs the extra registers and
// instructions cost more than they hide (455 against 440 us a frame on 4096
// stacks; 76 against 80 us on two 256-body stacks).
template <bool kRecord, bool kAhead>
__device__ void scene_sweep(const Team& T, uint32_t groups, uint32_t passes, const SceneBodies& SB,
                            const SceneContacts& SC, float mu, float dt, int* s_flag,
                            const SolveRecord* rec_in = nullptr, int iter = 0) {
    const SolveRecord* const rec = kRecord ? rec_in : nullptr;
    const bool is_b = T.rank() & 1u, alone = kAhead && T.size() > 32u && passes - groups <= groups / 16u;
    const uint32_t first = alone ? 0u : (T.rank() & ~31u) >> 1, step = alone ? 16u : T.size() >> 1;
    if (!alone || T.warp() == 0u) {
        uint32_t k = 0, bi = 0;
        Contact ct{};
        SideBody S{};
        float lc = 0.f;
        // contact i0 + lane / 2 of a group that ends at `end`, and its body's constant rows
        auto fetch = [&](uint32_t i0, uint32_t end) {
            const uint32_t i = i0 + ((T.rank() & 31u) >> 1);
            k = SC.ent(i < end ? i : i0);
            ct = SC.contact(k);
            lc = SC.lam(k);
            bi = is_b ? ct.b : ct.a;
            S.m = SB.im(bi);
            S.ixx = SB.ixx(bi); S.iyy = SB.iyy(bi); S.izz = SB.izz(bi);
            S.ixy = SB.ixy(bi); S.ixz = SB.ixz(bi); S.iyz = SB.iyz(bi);
        };
        uint32_t start = SC.pa(0), end = SC.pa(1);
        if (kAhead && start + first < end) fetch(start + first, end);
        for (uint32_t g = 0; g < groups; ++g) {
            bool fetched = kAhead;
            for (uint32_t i0 = start + first; i0 < end; i0 += step) {  // warp-uniform
                if (!fetched) fetch(i0, end);
                fetched = false;
                const bool valid = i0 + ((T.rank() & 31u) >> 1) < end;
                S.px = SB.px(bi); S.py = SB.py(bi); S.pz = SB.pz(bi);
                S.qw = SB.qw(bi); S.qx = SB.qx(bi); S.qy = SB.qy(bi); S.qz = SB.qz(bi);
                S.vx = SB.vx(bi); S.vy = SB.vy(bi); S.vz = SB.vz(bi);
                S.wx = SB.wx(bi); S.wy = SB.wy(bi); S.wz = SB.wz(bi);
                int res;
                if (rec) {
                    // The pre-solve state of the first sweep, the one the adjoint
                    // differentiates, marked as acted only if it did. A later sweep
                    // (after a deferral) must not overwrite it: it re-solves only the
                    // deferred contacts, and one of those that acts there is
                    // reported as a path the adjoint does not cover.
                    float* r = rec->rec + rec->base + k;
                    const float lc0 = lc;
                    if (iter == 0 && valid) record_state(r, rec->stride, S, is_b ? 13 : 0);
                    uint32_t fl = 0u;
                    res = solve_contact_side<kAhead>(valid, is_b, S, ct, mu, lc, dt, &fl);
                    if (valid && !is_b) {
                        if (fl & kSfActive) {
                            r[26ull * rec->stride] = lc0;
                            r[35ull * rec->stride] = __uint_as_float(fl);
                            if (iter > 0) atomicOr(rec->flag, 1u);  // acted after a renormalisation
                        } else if (iter == 0) {
                            r[35ull * rec->stride] = 0.f;
                        }
                    }
                } else {
                    res = solve_contact_side<kAhead>(valid, is_b, S, ct, mu, lc, dt);
                }
                if (res == kSolveDone) {
                    if (S.m != 0.f) store_side(SB, bi, S);
                    if (!is_b) SC.lam(k) = lc;
                } else if (res == kSolveDeferred) {
                    *s_flag = 1;
                }
            }
            start = end;
            if (g + 1u < groups) {
                end = SC.pa(g + 2u);
                if (kAhead && start + first < end) fetch(start + first, end);
            }
            if (alone)
                __syncwarp();
            else
                T.sync();
        }
    }
    if (alone) T.sync();
}

// Block-shared scalars of one scene's solve.
struct SceneShared {
    uint32_t scan[2 * (kSceneWideThreads / 32)];
    uint32_t rem, over, maxcol, passes;
    uint32_t nan;  // a leaf box of a single scene's frame holds a NaN (frame_scene)
    int flag;
};

// The solver's per-body rows after the 20 body rows (see scene_body_bytes).
struct SceneSolverRows {
    uint64_t* mask;  // [ldb] JP colour masks
    uint32_t* pri;   // [2][ldb] JP priorities of even and odd rounds
    uint32_t* off;   // [ldb + 4] b-side list offsets
    uint32_t* cnt;   // [ldb] counts / fill cursors / last b-side contact
};

__device__ __forceinline__ SceneSolverRows scene_solver_rows(float* fb, uint32_t ldb) {
    SceneSolverRows R;
    R.mask = reinterpret_cast<uint64_t*>(fb + 20 * ldb);
    R.pri = reinterpret_cast<uint32_t*>(R.mask + ldb);
    R.off = R.pri + 2 * ldb;
    R.cnt = R.off + ldb + 4;
    return R;
}

__device__ __forceinline__ void scene_load_bodies(const Team& T, const GlobalBodies& B, uint32_t b0, uint32_t nb,
                                                  float* fb, uint32_t ldb) {
    const SceneBodies SB{fb, ldb};
    for (uint32_t i = T.rank(); i < nb; i += T.size()) {
        const uint32_t g = b0 + i;
        SB.px(i) = B.px(g); SB.py(i) = B.py(g); SB.pz(i) = B.pz(g);
        SB.qw(i) = B.qw(g); SB.qx(i) = B.qx(g); SB.qy(i) = B.qy(g); SB.qz(i) = B.qz(g);
        SB.vx(i) = B.vx(g); SB.vy(i) = B.vy(g); SB.vz(i) = B.vz(g);
        SB.wx(i) = B.wx(g); SB.wy(i) = B.wy(g); SB.wz(i) = B.wz(g);
        fb[13 * ldb + i] = B.im(g);
        fb[14 * ldb + i] = B.ixx(g); fb[15 * ldb + i] = B.iyy(g); fb[16 * ldb + i] = B.izz(g);
        fb[17 * ldb + i] = B.ixy(g); fb[18 * ldb + i] = B.ixz(g); fb[19 * ldb + i] = B.iyz(g);
    }
}

__device__ __forceinline__ void scene_store_bodies(const Team& T, const GlobalBodies& B, uint32_t b0, uint32_t nb,
                                                   const SceneBodies& SB) {
    for (uint32_t i = T.rank(); i < nb; i += T.size()) {
        const uint32_t g = b0 + i;
        B.px(g) = SB.px(i); B.py(g) = SB.py(i); B.pz(g) = SB.pz(i);
        B.qw(g) = SB.qw(i); B.qx(g) = SB.qx(i); B.qy(g) = SB.qy(i); B.qz(g) = SB.qz(i);
        B.vx(g) = SB.vx(i); B.vy(g) = SB.vy(i); B.vz(g) = SB.vz(i);
        B.wx(g) = SB.wx(i); B.wy(g) = SB.wy(i); B.wz(g) = SB.wz(i);
    }
}

// Jones–Plassmann colouring of a scene's contacts into SC.done: the rounds taken
// in `rounds`, what is left uncoloured in sh.rem, sh.over when a body needs a 65th
// colour, the largest colour in sh.maxcol.
__device__ __forceinline__ void scene_color(const Team& T, uint32_t nb, uint32_t m, const SceneBodies& SB,
                                      const SceneSolverRows& R, const SceneContacts& SC, SceneShared& sh,
                                      uint32_t& rounds) {
    // A contact's priority is hash(k) << 32 | k; the hash (murmur3's
    // finaliser) is a bijection, so its 32 bits alone are distinct and in
    // the same order, and shared memory has a native 32-bit maximum. A
    // winner is the only one on its bodies, so it updates their masks
    // without atomics. Each thread keeps its uncoloured contacts as bits
    // (up to 64 of them, the rest by their colour word); priorities
    // alternate between two rows, one cleared while the other is used.
    // Set-up of a 512-body mixed scene alone: 80 us, 137 with 64-bit
    // maxima over all contacts in every round.
    // The bodies of a contact, 0xFFFF for a static one, wait in its list entry's
    // word (free until the groups are made).
    T.sync();  // the lists' last reads
    for (uint32_t k = T.rank(); k < m; k += T.size()) {
        const uint32_t ab = SC.ab(k);
        SC.done(k) = kUncolored;
        SC.ent(k) = ab | (SB.im(ab & 0xFFFFu) == 0.f ? 0xFFFFu : 0u) | (SB.im(ab >> 16) == 0.f ? 0xFFFF0000u : 0u);
    }
    for (uint32_t i = T.rank(); i < nb; i += T.size()) {
        R.mask[i] = 0ull;
        R.pri[i] = 0u;
    }
    if (T.leader()) {
        sh.rem = m;
        sh.over = 0u;
        sh.maxcol = 0u;
    }
    const uint32_t mine = m > T.rank() ? (m - T.rank() + T.size() - 1u) / T.size() : 0u;
    uint64_t open = mine >= 64u ? ~0ull : (1ull << mine) - 1ull;
    // fn(k, bodies) for each of this thread's uncoloured contacts, four loads ahead
    auto for_open = [&](auto&& fn) {
        for (uint64_t o = open; o;) {
            uint32_t j[4], ab[4];
            int c = 0;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                j[u] = o ? static_cast<uint32_t>(__ffsll(static_cast<long long>(o))) - 1u : 0u;
                c += o ? 1 : 0;
                o &= o - 1ull;
                ab[u] = SC.ent(T.rank() + j[u] * T.size());
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (u < c && fn(T.rank() + j[u] * T.size(), ab[u])) open &= ~(1ull << j[u]);
        }
        for (uint32_t j = 64u; j < mine; ++j) {
            const uint32_t k = T.rank() + j * T.size();
            if (SC.done(k) == kUncolored) fn(k, SC.ent(k));
        }
    };
    uint32_t my_max = 0u;
    T.sync();
    while (sh.rem > 0u && rounds < kMaxRounds) {
        uint32_t* pri = R.pri + (rounds & 1u) * ((nb + 3u) & ~3u);
        uint32_t* next = R.pri + (~rounds & 1u) * ((nb + 3u) & ~3u);
        for_open([&](uint32_t k, uint32_t ab) {
            const uint32_t a = ab & 0xFFFFu, b = ab >> 16, pk = hash_u32(k);
            if (a != 0xFFFFu) atomicMax(&pri[a], pk);
            if (b != 0xFFFFu) atomicMax(&pri[b], pk);
            return false;
        });
        for (uint32_t i = T.rank(); i < nb; i += T.size()) next[i] = 0u;
        T.sync();
        uint32_t won = 0u;
        for_open([&](uint32_t k, uint32_t ab) {
            const uint32_t a = ab & 0xFFFFu, b = ab >> 16, pk = hash_u32(k);
            const bool da = a != 0xFFFFu, db = b != 0xFFFFu;
            if ((da && pri[a] != pk) || (db && pri[b] != pk)) return false;  // not a local maximum
            const uint64_t used = (da ? R.mask[a] : 0ull) | (db ? R.mask[b] : 0ull);
            if (~used == 0ull) {  // > 64 colours: the reference falls back to the serial order
                sh.over = 1u;
                return false;
            }
            const uint32_t col = static_cast<uint32_t>(__ffsll(static_cast<long long>(~used)) - 1);
            SC.done(k) = col;
            if (da) R.mask[a] |= 1ull << col;
            if (db) R.mask[b] |= 1ull << col;
            my_max = max(my_max, col);
            ++won;
            return true;
        });
        won = __reduce_add_sync(0xffffffffu, won);
        if ((threadIdx.x & 31u) == 0u && won) atomicSub(&sh.rem, won);
        T.sync();
        ++rounds;
    }
    my_max = __reduce_max_sync(0xffffffffu, my_max);
    if ((threadIdx.x & 31u) == 0u) atomicMax(&sh.maxcol, my_max);
    T.sync();
}

// XpbdSolver::solve on one scene whose m >= 1 contacts sit in SC (rows ab,
// lambda = 0, geometry; pb = none) with R.cnt[b] = the b-side contact count of
// every dynamic body b. Leaves the bodies solved and renormalised in SB and
// the colours (or UINT32_MAX) in SC.done. Returns false after raising an error.
template <bool kRecord = false, bool kAhead = false>
__device__ bool scene_solve(Team& T, uint32_t nb, uint32_t m, const SceneBodies& SB, const SceneSolverRows& R,
                            const SceneContacts& SC, int mode, int n_iters, float mu, float dt, SceneShared& sh,
                            bool& colored_out, uint32_t& n_colors_out, uint32_t& rounds_out,
                            const SolveRecord* rec_in = nullptr, uint32_t* groups_out = nullptr,
                            uint64_t* sweep_start = nullptr) {
    const SolveRecord* const rec = kRecord ? rec_in : nullptr;
    // ── predecessors in contact order: b-side lists (scan, fill, sort) ──
    if (T.leader()) sh.flag = 0;
    uint32_t entries = 0;
    for (uint32_t base = 0; base < nb; base += T.size()) {
        const uint32_t i = base + T.rank();
        const uint32_t v = i < nb ? R.cnt[i] : 0u;
        uint32_t tot;
        const uint32_t ex = T.exclusive_scan(v, sh.scan, tot);
        if (i < nb) {
            R.off[i] = entries + ex;
            R.cnt[i] = 0u;
        }
        entries += tot;
    }
    if (T.leader()) R.off[nb] = entries;
    T.sync();
    for (uint32_t k = T.rank(); k < m; k += T.size()) {
        const uint32_t b = SC.ab(k) >> 16;
        if (SB.im(b) != 0.f) SC.ent(R.off[b] + atomicAdd(&R.cnt[b], 1u)) = k;
    }
    T.sync();
    for (uint32_t x = T.rank(); x < nb; x += T.size()) {
        const uint32_t lo = R.off[x], hi = R.off[x + 1];
        for (uint32_t i = lo + 1; i < hi; ++i) {
            const uint32_t v = SC.ent(i);
            uint32_t j = i;
            while (j > lo && SC.ent(j - 1) > v) {
                SC.ent(j) = SC.ent(j - 1);
                --j;
            }
            SC.ent(j) = v;
        }
        for (uint32_t i = lo + 1; i < hi; ++i) SC.pb(SC.ent(i)) = SC.ent(i - 1);
        R.cnt[x] = hi > lo ? SC.ent(hi - 1) : kSceneNone;  // last b-side contact of x
    }
    T.sync();
    for (uint32_t k = T.rank(); k < m; k += T.size()) {
        const uint32_t a = SC.ab(k) & 0xFFFFu;
        uint32_t p = kSceneNone;
        if (SB.im(a) != 0.f) p = (k > 0 && (SC.ab(k - 1) & 0xFFFFu) == a) ? k - 1 : R.cnt[a];
        SC.pa(k) = p;
    }
    // ── colouring (reference mode above 256 contacts, coloured mode always) ──
    bool colored = mode == DYPH_SOLVER_COLORED ||
                   ((mode == DYPH_SOLVER_REFERENCE || mode == DYPH_SOLVER_REFERENCE_ROUNDS) && m > kSerialThreshold);
    uint32_t n_colors = 0, rounds = 0;
    if (colored) {
        scene_color(T, nb, m, SB, R, SC, sh, rounds);
        colored = sh.rem == 0u && sh.over == 0u;
        n_colors = sh.maxcol + 1u;
        T.sync();
    }
    // ── groups: colours, or the levels of the sequential order ──
    uint32_t groups = n_colors, base = 0u;
    if (!colored) {
        groups = scene_levels(T, m, SC, &sh.maxcol);
        base = 1u;
        if (groups == 0u) {
            if (T.leader()) raise_error(DYPH_ERR_TIMEOUT, 11u);
            return false;
        }
    }
    scene_group(T, m, groups, base, SC, sh.scan, &sh.passes);
    if (sweep_start && T.leader()) {
        uint64_t t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        *sweep_start = t;
    }
    // ── sweeps and renormalisation ──
    bool deferred = false;
    if (groups_out) *groups_out = groups;
    for (int iter = 0; iter < n_iters; ++iter) {
        if (iter == 0 || deferred) {
            scene_sweep<kRecord, kAhead>(T, groups, sh.passes, SB, SC, mu, dt, &sh.flag, rec, iter);
            deferred = sh.flag != 0;
        }
        if (rec && iter == 0)
            for (uint32_t i = T.rank(); i < nb; i += T.size()) {
                float* q = rec->qs + rec->b0 + i;
                q[0] = SB.qw(i);
                q[rec->qs_stride] = SB.qx(i);
                q[2ull * rec->qs_stride] = SB.qy(i);
                q[3ull * rec->qs_stride] = SB.qz(i);
            }
        const int times = deferred ? 1 : n_iters - iter;
        for (uint32_t i = T.rank(); i < nb; i += T.size()) {
            float qw = SB.qw(i), qx = SB.qx(i), qy = SB.qy(i), qz = SB.qz(i);
            // a quaternion that renormalises to itself stays: the rest of the passes are skipped
            for (int t = 0; t < times; ++t) {
                const float pw = qw, px = qx, py = qy, pz = qz;
                renormalize(qw, qx, qy, qz);
                if (qw == pw && qx == px && qy == py && qz == pz) break;
            }
            SB.qw(i) = qw; SB.qx(i) = qx; SB.qy(i) = qy; SB.qz(i) = qz;
        }
        T.sync();
        if (!deferred) break;
    }
    colored_out = colored;
    n_colors_out = n_colors;
    rounds_out = rounds;
    return true;
}

__device__ __forceinline__ void scene_stats(const Team& T, uint32_t* meta, bool colored, uint32_t n_colors,
                                            uint32_t rounds) {
    if (T.leader()) {
        if (colored) {
            atomicMax(&meta[kMetaMaxColor], n_colors - 1u);
            meta[kMetaSceneColored] = 1u;
        }
        atomicMax(&meta[kMetaRounds], rounds);
        meta[kMetaDecision] = kDecisionScenes;
    }
}

__global__ void __launch_bounds__(kSceneThreads, 4) scene_solve_kernel(dyph_contacts cv, dyph_bodies gb,
                                                                       SceneBufs S, int mode, int n_iters,
                                                                       float mu, float dt,
                                                                       uint32_t* __restrict__ color,
                                                                       uint32_t* __restrict__ meta) {
    extern __shared__ __align__(16) unsigned char scene_smem[];
    __shared__ SceneShared sh;
    const GlobalBodies B{gb};
    Team T{kSceneThreads, 0u};
    for (uint32_t t = blockIdx.x; t < S.n_scenes; t += gridDim.x) {
        const uint32_t s = S.order[t];
        const uint32_t b0 = S.body_offset[s], nb = S.body_offset[s + 1] - b0;
        const uint32_t k0 = S.range[2 * s], m = S.range[2 * s + 1] - k0;
        if (m == 0) continue;  // no contacts: the reference's solve returns at once
        // ── layout: bodies, then (if they fit) the contact words ──
        const uint32_t ldb = (nb + 3u) & ~3u;
        float* fb = reinterpret_cast<float*>(scene_smem);
        const SceneSolverRows R = scene_solver_rows(fb, ldb);
        const uint32_t body_bytes = scene_body_bytes(nb);
        const uint32_t ldc = (m + 4u) & ~3u;  // >= m + 1: group offsets take m + 1 words
        const bool in_smem = body_bytes + kSceneWords * 4u * ldc <= S.smem_bytes;
        const SceneBodies SB{fb, ldb};
        // (in the scratch, scene s owns words [k0 + s, k0 + s + m] of each row: m + 1 words)
        const SceneContacts SC{in_smem ? reinterpret_cast<uint32_t*>(scene_smem + body_bytes) : S.scratch + k0 + s,
                               in_smem ? ldc : S.scratch_stride};
        // ── stage the scene's bodies and contacts ──
        scene_load_bodies(T, B, b0, nb, fb, ldb);
        for (uint32_t i = threadIdx.x; i < nb; i += blockDim.x) R.cnt[i] = 0u;
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < m; k += blockDim.x) {
            const uint32_t a = cv.body_a[k0 + k] - b0, b = cv.body_b[k0 + k] - b0;
            SC.ab(k) = a | (b << 16);
            SC.lam(k) = 0.f;
            const uint32_t c = k0 + k;
            SC.g(0, k) = cv.pos_x[c]; SC.g(1, k) = cv.pos_y[c]; SC.g(2, k) = cv.pos_z[c];
            SC.g(3, k) = cv.norm_x[c]; SC.g(4, k) = cv.norm_y[c]; SC.g(5, k) = cv.norm_z[c];
            SC.g(6, k) = cv.depth[c];
            SC.pb(k) = kSceneNone;
            if (SB.im(b) != 0.f) atomicAdd(&R.cnt[b], 1u);
        }
        __syncthreads();
        bool colored = false;
        uint32_t n_colors = 0, rounds = 0;
        if (!scene_solve(T, nb, m, SB, R, SC, mode, n_iters, mu, dt, sh, colored, n_colors, rounds)) return;
        // ── write back, colours and statistics ──
        scene_store_bodies(T, B, b0, nb, SB);
        for (uint32_t k = threadIdx.x; k < m; k += blockDim.x) color[k0 + k] = colored ? SC.done(k) : kUncolored;
        scene_stats(T, meta, colored, n_colors, rounds);
        __syncthreads();
    }
}

}  // namespace
}  // namespace dyph
