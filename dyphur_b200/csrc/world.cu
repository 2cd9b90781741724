// The whole frame step behind one handle.
//
// One frame is the reference's loop body (examples/stress_test_blocks/
// main.cpp:264-279): integrate, build_and_query, sort_pairs (already sorted),
// Narrowphase::run, XpbdSolver::solve. Every count stays on the device, so a
// frame has no host round trip. A single scene's first step captures one frame
// into a CUDA graph and every later frame replays it; a batch whose scenes fit
// a block's shared memory runs on fused kernels, and so do the frames of a
// small single scene but a call's last. A small kernel at the end folds the
// pair / contact counts into peak and overflow words.
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <new>
#include <vector>

#include "internal.cuh"
#include "scene_frame.cuh"
#include "scene_adjoint.cuh"

struct dyph_world {
    dyph_world_desc desc{};
    dyph_broadphase* bp = nullptr;
    dyph_narrowphase* np = nullptr;
    dyph_xpbd* sv = nullptr;
    uint32_t* stats = nullptr;  // [0] last pairs, [1] last contacts, [2] peak pairs, [3] peak contacts, [4] status
    cudaStream_t stream = nullptr;
    cudaEvent_t ev_in = nullptr, ev_out = nullptr;
    cudaGraphExec_t graph = nullptr;
    cudaGraphExec_t episode = nullptr;  // n_frames frames in one graph (dyph_world_capture_episode)
    int32_t episode_frames = 0;
    uint64_t* scene_hash = nullptr;  // [n_scenes] per-scene FNV-1a results
    // Trajectory recording (dyph_world_set_trajectory): pose rows packed on
    // the frame's stream into one of two device staging buffers, copied to the
    // caller's pinned host buffer on a side stream.
    float* traj_host = nullptr;
    uint32_t traj_every = 0, traj_max = 0;
    uint64_t traj_frame = 0;              // frames stepped by dyph_world_step since the last set-up
    float* traj_stage[2] = {nullptr, nullptr};  // [traj_slots][7 n] records each
    uint32_t traj_slots = 0;
    uint64_t traj_chunk = 0;              // staging buffers filled by fused steps since the last set-up
    cudaStream_t traj_stream = nullptr;
    cudaEvent_t traj_packed[2] = {nullptr, nullptr};
    cudaEvent_t traj_copied[2] = {nullptr, nullptr};
    bool traj_pending = false;            // a copy on the side stream not yet joined
    bool traj_live[2] = {false, false};   // traj_copied[k] was last recorded outside a capture
    // Batched scenes with the whole frame fused into one kernel (one block per scene).
    bool fused = false;
    uint32_t frame_smem = 0;
    uint32_t* f_pair_base = nullptr;     // [n_scenes + 1]
    uint32_t* f_contact_base = nullptr;  // [n_scenes + 1]
    uint32_t* f_pair_raw = nullptr;
    uint32_t* f_contact_raw = nullptr;
    uint32_t* f_color_raw = nullptr;
    uint32_t* f_counts = nullptr;        // [4 n_scenes]
    uint32_t* f_run = nullptr;           // [kAccWords] + [kRunRows kMaxRunFrames] a launch's statistics (zero between launches)
    uint32_t* f_words = nullptr;
    uint32_t* f_pos = nullptr;           // [2 n_scenes] gather positions
    uint32_t* f_items = nullptr;         // [4 f_n_items] work items of the fused kernel
    uint32_t f_n_items = 0;
    unsigned long long* f_phase = nullptr;  // [kFramePhases] phase timing of fused frames (null = off)
    // A small single scene's frames but a call's last (solo_frames): one block of
    // the fused frame's code (scene_single_kernel). Device words: body, pair and
    // contact ranges and counts; then the pair slots and the contact words. Null when
    // the scene is not small.
    uint32_t* s_buf = nullptr;
    uint32_t s_smem = 0, s_pairs = 0, s_contacts = 0;
    dyph_solver_mode graph_mode = DYPH_SOLVER_REFERENCE;  // the solver mode that the captured frame holds
    // Adjoint of fused frames (dyph_world_rollout_backward), allocated on first use.
    // Record sets, one per frame of two checkpoint segments: contact records,
    // poses after integrate, quaternions before renormalisation, contact
    // words, counts.
    std::vector<float*> a_rec;       // [kRecWords][f_contact_slots]
    std::vector<float*> a_pose1;     // [7][n]
    std::vector<float*> a_qs;        // [4][n]
    std::vector<uint32_t*> a_words;  // [kSceneWords][f_words_stride]
    std::vector<uint32_t*> a_mg;     // [2 n_scenes]
    AdjSet* a_sets = nullptr;        // [a_sets_n] the record sets, for the kernels
    size_t a_sets_n = 0;
    float* a_g = nullptr;            // [13][n] the state's adjoint
    float* a_seg[2] = {nullptr, nullptr};  // [a_seg_frames][13][n] states of frames 1.. of a segment (double buffer)
    uint32_t a_seg_frames = 0;
    uint32_t* a_pairs = nullptr;         // pair slots of spilled scenes, the recording's own
    cudaStream_t a_stream = nullptr;     // records the next checkpoint segment while this one is reversed
    cudaEvent_t a_seg_ready = nullptr, a_rtail = nullptr, a_rev_done = nullptr;
    uint32_t* a_flag = nullptr;
    uint32_t a_sized[4] = {0, 0, 0, 0};  // contact slots, words stride, pair slots, scenes the sets were made for
    uint32_t f_words_stride = 0, f_contact_slots = 0, f_pair_slots = 0;
    // Knobs of the fused kernel (dyph_world_set_fused_config / dyph_world_autotune).
    std::vector<uint32_t> h_body_offset;  // host copy of the scenes' body ranges
    uint32_t f_smem_cap = 0;              // shared memory cap per block (0 = what the largest scene needs)
    uint32_t f_teams = 2;                 // 0 blocks only, 1 + small scenes a quarter, 2 + mid-size half a block
    uint32_t f_threads = kSceneThreads;   // threads of a block (rule in setup_fused)
    bool f_resident = false;              // all blocks of the batch fit the device at once
    uint32_t f_variant = 0;               // register budget: 4 (0), 5 (1) or 6 (2) blocks per SM
    uint32_t f_warp_scenes = 0, f_half_scenes = 0, f_block_scenes = 0;
    // Work items of the adjoint's reverse kernel, laid out on their own: its
    // levels are long dependent chains with a barrier each, which favours
    // smaller teams than the forward frame's choice.
    uint32_t* r_items = nullptr;
    uint32_t r_n_items = 0, r_smem = 0;
    uint32_t r_smem_cap = 0;              // 0: a third of an SM's shared memory
    uint32_t r_teams = 2;
    uint32_t r_warp_scenes = 0, r_half_scenes = 0, r_block_scenes = 0;
    float f_tuned_ms = 0.f;
    uint32_t f_tuned_candidates = 0;
};

namespace dyph {
namespace {

constexpr uint32_t kHistory = 4096;

// The recomputation with recording of a segment's frames (record_scene), on the
// fused kernel's work items.
template <int kMinBlocks, int kThreads>
__global__ void __launch_bounds__(kThreads, kMinBlocks) scene_frame_record_kernel(SceneBufs S, FrameBufs F,
                                                                                  FrameParams P_, AdjSegment D,
                                                                                  const uint32_t* __restrict__ items,
                                                                                  uint32_t n_items) {
    for_each_item(items, n_items, S.smem_bytes,
                  [&](Team& T, uint32_t s, unsigned char* smem, uint32_t bytes, SceneShared& sh) {
                      for (uint32_t f = 0; f < P_.n_frames; ++f) {
                          const AdjSet& k = D.sets[f];
                          FrameBufs Ff = F;
                          Ff.words = k.words;
                          record_scene<kThreads == kSceneWideThreads>(T, s, f, smem, bytes, sh, S, Ff, P_, segment_run(D, f, P_.n_frames),
                                       AdjKeep{k.words, k.mg});
                      }
                  });
}
constexpr size_t kStatsWords = 8 + 2 * kHistory;

__global__ void frame_stats_kernel(const uint32_t* __restrict__ bp_counts, const uint32_t* __restrict__ np_counts,
                                   uint32_t max_pairs, uint32_t max_contacts, uint32_t* __restrict__ stats) {
    const uint32_t p = bp_counts[1], c = np_counts[1];
    stats[0] = p;
    stats[1] = c;
    stats[2] = max(stats[2], p);
    stats[3] = max(stats[3], c);
    // per-frame history ring: [8 + 2 k] pairs, [9 + 2 k] contacts of frame k mod kHistory
    const uint32_t f = stats[5]++;
    stats[8 + 2 * (f % kHistory)] = p;
    stats[9 + 2 * (f % kHistory)] = c;
    if (p > max_pairs) atomicCAS(&stats[4], 0u, static_cast<uint32_t>(DYPH_ERR_PAIR_OVERFLOW));
    if (c > max_contacts) atomicCAS(&stats[4], 0u, static_cast<uint32_t>(DYPH_ERR_CONTACT_OVERFLOW));
}

// The statistics of a fused launch of n_frames <= kMaxRunFrames frames (one
// block): the world's history, peaks and status as frame_stats_kernel keeps
// them frame by frame, the stored-count words and the solver's meta words of
// the last frame. Clears the launch's words for the next one.
__global__ void __launch_bounds__(kMaxRunFrames) frame_run_stats_kernel(uint32_t* __restrict__ run, uint32_t n_frames,
                                                                        uint32_t* __restrict__ bp_counts,
                                                                        uint32_t* __restrict__ np_counts,
                                                                        uint32_t* __restrict__ meta,
                                                                        uint32_t max_pairs, uint32_t max_contacts,
                                                                        uint32_t* __restrict__ stats) {
    const uint32_t f = threadIdx.x;
    uint32_t* counts = run + kAccWords;
    const uint32_t total = stats[5];
    uint32_t p = 0, c = 0;
    if (f < n_frames) {
        p = counts[n_frames + f];
        c = counts[3u * n_frames + f];
        stats[8 + 2 * ((total + f) % kHistory)] = p;
        stats[9 + 2 * ((total + f) % kHistory)] = c;
        atomicMax(&stats[2], p);
        atomicMax(&stats[3], c);
        if (f + 1u == n_frames) {
            stats[0] = p;
            stats[1] = c;
            bp_counts[0] = counts[f];
            bp_counts[1] = p;
            np_counts[0] = counts[2u * n_frames + f];
            np_counts[1] = c;
        }
    }
    // the earliest frame past a capacity sets the status: a scene's capacity before
    // the world's, pairs before contacts
    __shared__ uint32_t s_first;
    if (f == 0) s_first = kMaxRunFrames;
    const uint32_t over = f < n_frames ? counts[4u * n_frames + f] : 0u;
    __syncthreads();
    if (over || p > max_pairs || c > max_contacts) atomicMin(&s_first, f);
    __syncthreads();
    if (f == s_first) {
        const bool pairs = over ? (over & 1u) != 0u : p > max_pairs;
        atomicCAS(&stats[4], 0u, static_cast<uint32_t>(pairs ? DYPH_ERR_PAIR_OVERFLOW : DYPH_ERR_CONTACT_OVERFLOW));
    }
    if (f < 16u) {
        uint32_t v = 0u;
        if (f == kMetaMaxColor && run[kAccMaxColor]) v = run[kAccMaxColor] - 1u;
        if (f == kMetaRounds) v = run[kAccRounds];
        if (f == kMetaSceneColored) v = run[kAccColored];
        if (f == kMetaDecision) v = run[kAccSolved] ? kDecisionScenes : 0u;
        meta[f] = v;
    }
    __syncthreads();
    if (f == 0) stats[5] = total + n_frames;
    if (f < static_cast<uint32_t>(kAccWords)) run[f] = 0u;
    for (uint32_t i = f; i < kRunRows * n_frames; i += kMaxRunFrames) counts[i] = 0u;
}

// Pose rows of every body, interleaved per body as the .trajectory row
// (x, y, z, w, qx, qy, qz), examples/stress_test_blocks/main.cpp:191-197.
__global__ void pack_pose_kernel(GlobalBodies B, float* __restrict__ out) {
    const uint32_t n = B.v.n;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float* r = out + 7ull * i;
        r[0] = B.px(i); r[1] = B.py(i); r[2] = B.pz(i);
        r[3] = B.qw(i); r[4] = B.qx(i); r[5] = B.qy(i); r[6] = B.qz(i);
    }
}

// Queue trajectory record `rec` (the pose rows after the frame just queued on
// s): pack into staging buffer rec % 2 once that buffer's previous copy is
// done (when `wait_prev`), then copy it to the host on the side stream.
dyph_status enqueue_trajectory_record(dyph_world* w, cudaStream_t s, uint64_t rec, bool wait_prev) {
    const uint32_t n = w->desc.bodies.n;
    const int k = static_cast<int>(rec & 1u);
    if (wait_prev) DYPH_CUDA_TRY(cudaStreamWaitEvent(s, w->traj_copied[k], 0));
    pack_pose_kernel<<<(n + 255) / 256, 256, 0, s>>>(GlobalBodies{w->desc.bodies}, w->traj_stage[k]);
    DYPH_CUDA_TRY(cudaGetLastError());
    DYPH_CUDA_TRY(cudaEventRecord(w->traj_packed[k], s));
    DYPH_CUDA_TRY(cudaStreamWaitEvent(w->traj_stream, w->traj_packed[k], 0));
    DYPH_CUDA_TRY(cudaMemcpyAsync(w->traj_host + rec * 7ull * n, w->traj_stage[k], 7ull * n * sizeof(float),
                                  cudaMemcpyDeviceToHost, w->traj_stream));
    DYPH_CUDA_TRY(cudaEventRecord(w->traj_copied[k], w->traj_stream));
    w->traj_pending = true;
    return DYPH_OK;
}

// Order every queued trajectory copy, the last one out of staging buffer
// `last`, before the work that follows on s.
dyph_status join_trajectory(dyph_world* w, cudaStream_t s, uint64_t last) {
    if (!w->traj_pending) return DYPH_OK;
    DYPH_CUDA_TRY(cudaStreamWaitEvent(s, w->traj_copied[last & 1u], 0));
    w->traj_pending = false;
    return DYPH_OK;
}

bool trajectory_frame(const dyph_world* w, uint64_t frame) {
    return w->traj_host && frame % w->traj_every == 0 && frame / w->traj_every < w->traj_max;
}

// Records an event inside a stream capture as a real timestamp node.
dyph_status probe_record(void* ev, cudaStream_t s) {
    if (!ev) return DYPH_OK;
    DYPH_CUDA_TRY(cudaEventRecordWithFlags(static_cast<cudaEvent_t>(ev), s, cudaEventRecordExternal));
    return DYPH_OK;
}

// What a fused launch does besides stepping: its frames' numbers, the
// trajectory rows and the checkpoints it writes (see FrameParams).
struct FusedRun {
    uint32_t n_frames;  // <= kMaxRunFrames
    bool keep = true;   // the last launch of a call
    float* traj = nullptr;
    uint32_t traj_first = 0, traj_count = 0;
    float* ckpt = nullptr;
    uint32_t ckpt_first = 0, ckpt_every = 1;
};

// The fused kernel's form that the world's settings ask for.
struct FusedForm {
    const void* kernel;
    uint32_t threads;
};
FusedForm fused_form(const dyph_world* w) {
    if (w->f_threads == static_cast<uint32_t>(kSceneWideThreads))
        return {reinterpret_cast<const void*>(scene_frame_kernel<2, kSceneWideThreads>), kSceneWideThreads};
    switch (w->f_variant) {
        case 1: return {reinterpret_cast<const void*>(scene_frame_kernel<5, kSceneThreads>), kSceneThreads};
        case 2: return {reinterpret_cast<const void*>(scene_frame_kernel<6, kSceneThreads>), kSceneThreads};
        default: return {reinterpret_cast<const void*>(scene_frame_kernel<4, kSceneThreads>), kSceneThreads};
    }
}

constexpr uint32_t kSoloHead = 16;  // words before a solo scene's pair slots

// n_frames frames of every scene (of the one scene, for a world that is not a
// batch) in one launch, and their statistics.
dyph_status launch_run(dyph_world* w, const FusedRun& r, cudaStream_t s) {
    const dyph_world_desc& d = w->desc;
    const dyph_integrator_params& ip = d.integrator;
    const float sub_dt = ip.dt / static_cast<float>(ip.n_substeps);
    const bool solo = !w->fused;
    SceneBufs S{w->bp->body_offset, w->bp->bvh.scene_of, w->sv->scene_order, nullptr, nullptr, 0, w->bp->n_scenes,
                w->frame_smem};
    FrameBufs F{w->f_pair_base, w->f_contact_base, w->f_pair_raw, w->f_contact_raw, w->f_color_raw,
                w->f_counts, w->f_words, w->f_words_stride, w->f_contact_slots};
    if (solo) {
        uint32_t* h = w->s_buf;
        S = SceneBufs{h, nullptr, nullptr, nullptr, nullptr, 0, 1u, w->s_smem};
        F = FrameBufs{h + 2, h + 4, h + kSoloHead, nullptr, nullptr, h + 8, h + kSoloHead + w->s_pairs,
                      w->s_contacts + 1u, w->s_contacts};
    }
    FrameParams P{d.bodies, d.shapes, ip.gravity[0], ip.gravity[1], ip.gravity[2], sub_dt, 0.5f * sub_dt,
                  w->sv->friction, ip.dt, ip.n_substeps, static_cast<int>(solo ? w->graph_mode : w->sv->mode),
                  w->sv->n_iters, w->f_run, w->f_run + kAccWords, w->f_phase, r.n_frames,
                  r.keep ? 1u : 0u, r.traj, r.traj_first, std::max(w->traj_every, 1u), r.traj_count, r.ckpt,
                  r.ckpt_first, r.ckpt_every, d.scene_bounds};
    if (solo) {
        scene_single_kernel<kSceneWideThreads><<<1, kSceneWideThreads, w->s_smem, s>>>(S, F, P);
    } else {
        const FusedForm form = fused_form(w);
        void* args[] = {&S, &F, &P, &w->f_items, &w->f_n_items};
        DYPH_CUDA_TRY(cudaLaunchKernel(form.kernel, dim3(w->f_n_items), dim3(form.threads), args, w->frame_smem, s));
    }
    frame_run_stats_kernel<<<1, kMaxRunFrames, 0, s>>>(w->f_run, r.n_frames, w->bp->counts, w->np->counts, w->sv->meta,
                                                      w->bp->max_pairs, w->np->max_contacts, w->stats);
    DYPH_CUDA_TRY(cudaGetLastError());
    return DYPH_OK;
}

// Frames [frame0, frame0 + n_frames) of a fused batch, frame numbers as the
// trajectory counts them, in as few launches as the per-frame words and the
// trajectory's staging buffers allow when all of the batch's blocks are
// resident at once (no scene waits for the slowest of a frame: 67 against 79 us
// a frame on 256 push scenes, 51 against 60 on 64 stacks). With more blocks than
// that a frame is a launch: the queue's order, longest first, then balances
// every frame (421 us against 480 on 4096 stacks). Records go to one of the two staging
// buffers, traj_slots of them per launch, and from there to the host on the
// side stream while the next launch runs; chunk counts the buffers filled,
// live says whether a buffer's last copy has to be waited for (a capture may
// only wait for events of its own). ckpt receives the state before every
// ckpt_every-th frame of this call.
dyph_status enqueue_run(dyph_world* w, cudaStream_t s, uint64_t frame0, uint32_t n_frames, uint64_t& chunk,
                        bool live[2], float* ckpt = nullptr, uint32_t ckpt_every = 1) {
    const size_t n = w->desc.bodies.n;
    for (uint32_t done = 0; done < n_frames;) {
        FusedRun r{std::min(n_frames - done, w->f_resident ? kMaxRunFrames : 1u)};
        uint64_t rec0 = 0;
        if (w->traj_host) {
            const uint64_t every = w->traj_every, f = frame0 + done;
            rec0 = (f + every - 1) / every;  // the first record at or after frame f
            if (rec0 < w->traj_max) {
                const uint64_t most = std::min<uint64_t>(w->traj_slots, w->traj_max - rec0);
                // the launch ends with the record that fills the buffer
                r.n_frames = static_cast<uint32_t>(
                    std::min<uint64_t>(r.n_frames, rec0 * every - f + (most - 1) * every + 1));
                const uint64_t past = (f + r.n_frames - 1) / every + 1;  // one past the last record
                if (past > rec0) {
                    r.traj = w->traj_stage[chunk & 1u];
                    r.traj_first = static_cast<uint32_t>(rec0 * every - f);
                    r.traj_count = static_cast<uint32_t>(past - rec0);
                }
            }
        }
        if (ckpt) {
            const uint32_t c = (done + ckpt_every - 1) / ckpt_every;
            r.ckpt = ckpt + static_cast<size_t>(c) * 13 * n;
            r.ckpt_first = c * ckpt_every - done;
            r.ckpt_every = ckpt_every;
        }
        r.keep = done + r.n_frames == n_frames;
        const int k = static_cast<int>(chunk & 1u);
        if (r.traj && live[k]) DYPH_CUDA_TRY(cudaStreamWaitEvent(s, w->traj_copied[k], 0));
        const dyph_status st = launch_run(w, r, s);
        if (st != DYPH_OK) return st;
        if (r.traj) {
            DYPH_CUDA_TRY(cudaEventRecord(w->traj_packed[k], s));
            DYPH_CUDA_TRY(cudaStreamWaitEvent(w->traj_stream, w->traj_packed[k], 0));
            DYPH_CUDA_TRY(cudaMemcpyAsync(w->traj_host + rec0 * 7 * n, w->traj_stage[k],
                                          r.traj_count * 7 * n * sizeof(float), cudaMemcpyDeviceToHost,
                                          w->traj_stream));
            DYPH_CUDA_TRY(cudaEventRecord(w->traj_copied[k], w->traj_stream));
            w->traj_pending = true;
            live[k] = true;
            ++chunk;
        }
        done += r.n_frames;
    }
    return DYPH_OK;
}

// One frame; when probe_stage matches a stage (0 integrate, 1 broadphase,
// 2 narrowphase, 3 solver) the events are recorded around it; probe_stage 4
// records them around the solver's dataflow kernel alone. keep: the last frame of a
// call (a fused batch stores no lists before it).
dyph_status enqueue_frame(dyph_world* w, cudaStream_t s, int probe_stage = -1, void* ev0 = nullptr,
                          void* ev1 = nullptr, bool keep = true) {
    const dyph_world_desc& d = w->desc;
    dyph_status st;
    if (w->fused) {
        if (probe_stage >= 0 && (st = probe_record(ev0, s)) != DYPH_OK) return st;
        if ((st = launch_run(w, FusedRun{1u, keep}, s)) != DYPH_OK) return st;
        return probe_stage >= 0 ? probe_record(ev1, s) : DYPH_OK;
    }
    w->sv->probe_flow[0] = probe_stage == 4 ? ev0 : nullptr;
    w->sv->probe_flow[1] = probe_stage == 4 ? ev1 : nullptr;
    for (int stage = 0; stage < 4; ++stage) {
        if (stage == probe_stage && (st = probe_record(ev0, s)) != DYPH_OK) return st;
        switch (stage) {
            case 0: st = integrate_launch(&d.bodies, &d.integrator, s); break;
            case 1: st = broadphase_build(w->bp, &d.bodies, &d.shapes, &d.scene_bounds, s); break;
            case 2:
                st = narrowphase_run(w->np, w->bp->pairs, w->bp->counts, w->bp->max_pairs, &d.bodies, &d.shapes, s);
                break;
            default: st = xpbd_solve(w->sv, &w->np->view, &d.bodies, d.integrator.dt, s); break;
        }
        if (st != DYPH_OK) break;
        if (stage == probe_stage && (st = probe_record(ev1, s)) != DYPH_OK) break;
    }
    w->sv->probe_flow[0] = w->sv->probe_flow[1] = nullptr;
    if (st != DYPH_OK) return st;
    frame_stats_kernel<<<1, 1, 0, s>>>(w->bp->counts, w->np->counts, w->bp->max_pairs, w->np->max_contacts,
                                       w->stats);
    DYPH_CUDA_TRY(cudaGetLastError());
    return DYPH_OK;
}

}  // namespace
}  // namespace dyph

using namespace dyph;

extern "C" void dyph_world_destroy(dyph_world* w) {
    if (!w) return;
    if (w->graph) cudaGraphExecDestroy(w->graph);
    if (w->episode) cudaGraphExecDestroy(w->episode);
    if (w->ev_in) cudaEventDestroy(w->ev_in);
    if (w->ev_out) cudaEventDestroy(w->ev_out);
    if (w->stream) cudaStreamDestroy(w->stream);
    if (w->stats) cudaFree(w->stats);
    if (w->scene_hash) cudaFree(w->scene_hash);
    if (w->traj_stream) cudaStreamSynchronize(w->traj_stream);
    for (int k = 0; k < 2; ++k) {
        if (w->traj_stage[k]) cudaFree(w->traj_stage[k]);
        if (w->traj_packed[k]) cudaEventDestroy(w->traj_packed[k]);
        if (w->traj_copied[k]) cudaEventDestroy(w->traj_copied[k]);
    }
    if (w->traj_stream) cudaStreamDestroy(w->traj_stream);
    void* fb[] = {w->f_pair_base, w->f_contact_base, w->f_pair_raw, w->f_contact_raw, w->f_color_raw, w->f_counts, w->f_run, w->s_buf,
                  w->f_words, w->f_pos, w->f_items, w->r_items, w->f_phase, w->a_g, w->a_sets, w->a_seg[0],
                  w->a_seg[1], w->a_flag, w->a_pairs};
    for (void* p : fb)
        if (p) cudaFree(p);
    for (size_t k = 0; k < w->a_rec.size(); ++k) {
        void* pk[] = {w->a_rec[k], w->a_pose1[k], w->a_qs[k], w->a_words[k], w->a_mg[k]};
        for (void* p : pk)
            if (p) cudaFree(p);
    }
    if (w->a_stream) cudaStreamDestroy(w->a_stream);
    if (w->a_seg_ready) cudaEventDestroy(w->a_seg_ready);
    if (w->a_rtail) cudaEventDestroy(w->a_rtail);
    if (w->a_rev_done) cudaEventDestroy(w->a_rev_done);
    broadphase_destroy(w->bp);
    narrowphase_destroy(w->np);
    xpbd_destroy(w->sv);
    delete w;
}

namespace {
dyph_status run_words(dyph_world* w);
uint32_t fused_smem_need(uint32_t max_nb);
uint32_t fused_smem_floor(uint32_t max_nb);
dyph_status fused_smem_prepare();

// A single scene of at most this many bodies steps the frames of a call but the
// last on one block (scene_single_kernel), in one launch: a frame is then one
// block's work instead of a dozen launches that a scene of this size cannot
// fill. The last frame runs the stage kernels, so the tree, the lists, the
// colours and the statistics that a program reads after a call are theirs.
// A frame in us, one block against the stage kernels, on stacks of boxes and on loose
// piles, whose few contacts leave the levels short:
//   reference order   16 / 61 (9)  102 / 138 (201)  148 / 148 (289)  168 / 145 (344)
//                     pile: 13 / 62 (61)  15 / 68 (201)  25 / 71 (401)  31 / 73 (506)
//   sequential        128 / 198 (201)  174 / 226 (289)  294 / 291 (433)  280 / 267 (505)
//                     pile: 25 / 69 (401)  31 / 74 (506)
// The limits lie where a dense stack breaks even: the count of bodies is all that is
// known ahead of the frames. A little past it the sequential order still has the pile's
// gain against 5 % of a stack's time.
constexpr uint32_t kSoloBodies = 256, kSoloSequentialBodies = 512;
bool solo_size(const dyph_world* w) {
    return w->desc.bodies.n <= (w->sv->mode == DYPH_SOLVER_SEQUENTIAL ? kSoloSequentialBodies : kSoloBodies);
}

// The one block's buffers, made with the world: a step allocates nothing, since
// another stream may be in a capture meanwhile. Without them the world steps every
// frame on the stage kernels.
void solo_reserve(dyph_world* w) {
    if (!solo_size(w)) return;
    const uint32_t n = w->desc.bodies.n;
    // no more pairs than there are, so that the slots stay small whatever the capacities
    const uint32_t pairs = std::min(w->bp->max_pairs, n * (n - 1u) / 2u), contacts = std::min(w->np->max_contacts, pairs);
    const size_t words = kSoloHead + pairs + static_cast<size_t>(kSceneWords) * (contacts + 1u);
    const uint32_t head[kSoloHead] = {0u, n, 0u, pairs, 0u, contacts};
    if (fused_smem_prepare() != DYPH_OK || run_words(w) != DYPH_OK ||
        cudaMalloc(&w->s_buf, words * sizeof(uint32_t)) != cudaSuccess ||
        cudaMemcpy(w->s_buf, head, sizeof(head), cudaMemcpyHostToDevice) != cudaSuccess || setup_done() != DYPH_OK) {
        cudaGetLastError();
        if (w->s_buf) cudaFree(w->s_buf);
        w->s_buf = nullptr;
        return;
    }
    w->s_pairs = pairs;
    w->s_contacts = contacts;
    w->s_smem = fused_smem_need(n);
}

// Whether the frames of a call but the last run on one block.
bool solo_frames(const dyph_world* w) {
    return w->s_buf && !w->fused && w->bp->n_scenes == 0u && !w->traj_host && solo_size(w);
}
}  // namespace

extern "C" dyph_status dyph_world_create(const dyph_world_desc* desc, dyph_stream, dyph_world** out) {
    if (!desc || !out || desc->bodies.n == 0 || desc->integrator.n_substeps <= 0) return DYPH_ERR_INVALID;
    dyph_status dc = dyph_device_check();
    if (dc != DYPH_OK) return dc;
    auto* w = new (std::nothrow) dyph_world();
    if (!w) return DYPH_ERR_NOMEM;
    w->desc = *desc;
    dyph_status st = broadphase_create(desc->bodies.n, desc->max_pairs, &w->bp);
    if (st == DYPH_OK) st = narrowphase_create(desc->max_contacts, &w->np);
    if (st == DYPH_OK) st = narrowphase_reserve(w->np, desc->max_pairs);
    if (st == DYPH_OK) st = narrowphase_reserve_bodies(w->np, desc->bodies.n);
    if (st == DYPH_OK) st = xpbd_create(desc->n_iters, desc->max_contacts, desc->bodies.n, desc->friction, &w->sv);
    if (st == DYPH_OK) {
        w->sv->mode = desc->mode;
        if (cudaMalloc(&w->stats, kStatsWords * sizeof(uint32_t)) != cudaSuccess ||
            cudaMemset(w->stats, 0, kStatsWords * sizeof(uint32_t)) != cudaSuccess || setup_done() != DYPH_OK ||
            cudaStreamCreateWithFlags(&w->stream, cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&w->ev_in, cudaEventDisableTiming) != cudaSuccess ||
            cudaEventCreateWithFlags(&w->ev_out, cudaEventDisableTiming) != cudaSuccess)
            st = DYPH_ERR_CUDA;
    }
    if (st != DYPH_OK) {
        dyph_world_destroy(w);
        return st;
    }
    solo_reserve(w);
    *out = w;
    return DYPH_OK;
}

namespace {
// The frames of a solo scene before a call's last one.
dyph_status enqueue_solo(dyph_world* w, cudaStream_t s, uint32_t n_frames) {
    for (uint32_t done = 0; done < n_frames; done += kMaxRunFrames) {
        FusedRun r{std::min(n_frames - done, kMaxRunFrames)};
        r.keep = false;
        const dyph_status st = launch_run(w, r, s);
        if (st != DYPH_OK) return st;
    }
    return DYPH_OK;
}

// dyph_world_step; a fused batch also writes checkpoints (dyph_world_rollout).
dyph_status world_step(dyph_world* w, int32_t n_frames, dyph_stream s, float* ckpt = nullptr, uint32_t ckpt_every = 1) {
    cudaStream_t cs = reinterpret_cast<cudaStream_t>(s);
    // Not in a caller's capture: the host counts the frames of each call, and a new
    // layout gives back the buffers that recorded launches would go on using.
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    DYPH_CUDA_TRY(cudaStreamIsCapturing(cs, &capture));
    if (capture != cudaStreamCaptureStatusNone) DYPH_CUDA_TRY(cudaErrorStreamCaptureUnsupported);
    DYPH_CUDA_TRY(cudaEventRecord(w->ev_in, cs));
    DYPH_CUDA_TRY(cudaStreamWaitEvent(w->stream, w->ev_in, 0));
    uint64_t last = 0;
    if (w->fused) {
        const dyph_status st = enqueue_run(w, w->stream, w->traj_frame, static_cast<uint32_t>(n_frames), w->traj_chunk,
                                           w->traj_live, ckpt, ckpt_every);
        if (st != DYPH_OK) return st;
        w->traj_frame += static_cast<uint64_t>(n_frames);
        last = w->traj_chunk - 1;
    } else {
        if (!w->graph) {
            cudaGraph_t g = nullptr;
            DYPH_CUDA_TRY(cudaStreamBeginCapture(w->stream, cudaStreamCaptureModeThreadLocal));
            dyph_status st = enqueue_frame(w, w->stream);
            cudaError_t ce = cudaStreamEndCapture(w->stream, &g);
            if (st != DYPH_OK) {
                if (g) cudaGraphDestroy(g);
                return st;
            }
            if (ce != cudaSuccess) return DYPH_ERR_CUDA;
            ce = cudaGraphInstantiate(&w->graph, g, 0);
            cudaGraphDestroy(g);
            if (ce != cudaSuccess) {
                w->graph = nullptr;
                return DYPH_ERR_CUDA;
            }
            w->graph_mode = w->sv->mode;
        }
        int32_t f = 0;
        if (n_frames > 1 && solo_frames(w)) {
            const dyph_status st = enqueue_solo(w, w->stream, static_cast<uint32_t>(n_frames - 1));
            if (st != DYPH_OK) return st;
            f = n_frames - 1;
            w->traj_frame += static_cast<uint64_t>(f);
        }
        for (; f < n_frames; ++f) {
            DYPH_CUDA_TRY(cudaGraphLaunch(w->graph, w->stream));
            if (trajectory_frame(w, w->traj_frame)) {
                last = w->traj_frame / w->traj_every;
                const int k = static_cast<int>(last & 1u);
                dyph_status st = enqueue_trajectory_record(w, w->stream, last, w->traj_live[k]);
                if (st != DYPH_OK) return st;
                w->traj_live[k] = true;
            }
            ++w->traj_frame;
        }
    }
    dyph_status jst = join_trajectory(w, w->stream, last);
    if (jst != DYPH_OK) return jst;
    DYPH_CUDA_TRY(cudaEventRecord(w->ev_out, w->stream));
    DYPH_CUDA_TRY(cudaStreamWaitEvent(cs, w->ev_out, 0));
    return DYPH_OK;
}
}  // namespace

extern "C" dyph_status dyph_world_step(dyph_world* w, int32_t n_frames, dyph_stream s) {
    if (!w || n_frames < 0) return DYPH_ERR_INVALID;
    return n_frames == 0 ? DYPH_OK : world_step(w, n_frames, s);
}

extern "C" dyph_status dyph_world_capture_episode(dyph_world* w, int32_t n_frames, int32_t probe_stage,
                                                  void* const* ev_start, void* const* ev_end) {
    if (!w || n_frames <= 0 || probe_stage < -1 || probe_stage > 4) return DYPH_ERR_INVALID;
    if (probe_stage >= 0 && (!ev_start || !ev_end)) return DYPH_ERR_INVALID;
    if (w->episode) {
        cudaGraphExecDestroy(w->episode);
        w->episode = nullptr;
    }
    const bool solo = probe_stage < 0 && n_frames > 1 && solo_frames(w);
    cudaGraph_t g = nullptr;
    DYPH_CUDA_TRY(cudaStreamBeginCapture(w->stream, cudaStreamCaptureModeThreadLocal));
    dyph_status st = DYPH_OK;
    uint64_t last = 0;
    if (w->fused && probe_stage < 0) {
        uint64_t chunk = 0;
        bool live[2] = {false, false};
        st = enqueue_run(w, w->stream, 0, static_cast<uint32_t>(n_frames), chunk, live);
        last = chunk - 1;
    } else {
        int32_t f0 = 0;
        if (solo) {
            const dyph_solver_mode mode = w->graph_mode;
            w->graph_mode = w->sv->mode;
            st = enqueue_solo(w, w->stream, static_cast<uint32_t>(n_frames - 1));
            w->graph_mode = mode;
            f0 = n_frames - 1;
        }
        for (int32_t f = f0; f < n_frames && st == DYPH_OK; ++f) {
            // a probed fused frame is a launch of its own between the events
            st = enqueue_frame(w, w->stream, probe_stage, probe_stage >= 0 ? ev_start[f] : nullptr,
                               probe_stage >= 0 ? ev_end[f] : nullptr, f + 1 == n_frames);
            if (st == DYPH_OK && trajectory_frame(w, static_cast<uint64_t>(f))) {
                last = static_cast<uint64_t>(f) / w->traj_every;
                st = enqueue_trajectory_record(w, w->stream, last, last >= 2);
            }
        }
    }
    if (st == DYPH_OK) st = join_trajectory(w, w->stream, last);
    w->traj_pending = false;
    cudaError_t ce = cudaStreamEndCapture(w->stream, &g);
    if (st != DYPH_OK) {
        if (g) cudaGraphDestroy(g);
        return st;
    }
    if (ce != cudaSuccess) return DYPH_ERR_CUDA;
    ce = cudaGraphInstantiate(&w->episode, g, 0);
    cudaGraphDestroy(g);
    if (ce != cudaSuccess) {
        w->episode = nullptr;
        return DYPH_ERR_CUDA;
    }
    w->episode_frames = n_frames;
    return DYPH_OK;
}

extern "C" dyph_status dyph_world_run_episode(dyph_world* w, dyph_stream s) {
    if (!w || !w->episode) return DYPH_ERR_INVALID;
    cudaStream_t cs = reinterpret_cast<cudaStream_t>(s);
    DYPH_CUDA_TRY(cudaEventRecord(w->ev_in, cs));
    DYPH_CUDA_TRY(cudaStreamWaitEvent(w->stream, w->ev_in, 0));
    DYPH_CUDA_TRY(cudaGraphLaunch(w->episode, w->stream));
    DYPH_CUDA_TRY(cudaEventRecord(w->ev_out, w->stream));
    DYPH_CUDA_TRY(cudaStreamWaitEvent(cs, w->ev_out, 0));
    return DYPH_OK;
}

extern "C" dyph_status dyph_event_create(void** out) {
    if (!out) return DYPH_ERR_INVALID;
    cudaEvent_t e = nullptr;
    DYPH_CUDA_TRY(cudaEventCreate(&e));
    *out = e;
    return DYPH_OK;
}

extern "C" void dyph_event_destroy(void* ev) {
    if (ev) cudaEventDestroy(static_cast<cudaEvent_t>(ev));
}

extern "C" dyph_status dyph_event_record(void* ev, dyph_stream s) {
    if (!ev) return DYPH_ERR_INVALID;
    DYPH_CUDA_TRY(cudaEventRecord(static_cast<cudaEvent_t>(ev), reinterpret_cast<cudaStream_t>(s)));
    return DYPH_OK;
}

extern "C" dyph_status dyph_event_elapsed_ms(void* start, void* end, float* ms) {
    if (!start || !end || !ms) return DYPH_ERR_INVALID;
    DYPH_CUDA_TRY(cudaEventSynchronize(static_cast<cudaEvent_t>(end)));
    DYPH_CUDA_TRY(cudaEventElapsedTime(ms, static_cast<cudaEvent_t>(start), static_cast<cudaEvent_t>(end)));
    return DYPH_OK;
}

extern "C" dyph_status dyph_world_check_finite(dyph_world* w, dyph_stream s, uint32_t* out_first_bad) {
    if (!w) return DYPH_ERR_INVALID;
    return dyph_bodies_check_finite(&w->desc.bodies, s, out_first_bad);
}

extern "C" dyph_status dyph_world_download_stats(dyph_world* w, dyph_stream s, uint32_t* last_pairs,
                                                 uint32_t* last_contacts, uint32_t* peak_pairs,
                                                 uint32_t* peak_contacts, uint32_t* status) {
    if (!w) return DYPH_ERR_INVALID;
    cudaStream_t cs = reinterpret_cast<cudaStream_t>(s);
    uint32_t h[5] = {0, 0, 0, 0, 0};
    DYPH_CUDA_TRY(cudaMemcpyAsync(h, w->stats, sizeof(h), cudaMemcpyDeviceToHost, cs));
    DYPH_CUDA_TRY(cudaStreamSynchronize(cs));
    if (last_pairs) *last_pairs = h[0];
    if (last_contacts) *last_contacts = h[1];
    if (peak_pairs) *peak_pairs = h[2];
    if (peak_contacts) *peak_contacts = h[3];
    if (status) *status = h[4];
    return DYPH_OK;
}

extern "C" dyph_status dyph_world_download_history(dyph_world* w, dyph_stream s, uint32_t* pairs,
                                                   uint32_t* contacts, uint32_t cap, uint32_t* frames_total) {
    if (!w) return DYPH_ERR_INVALID;
    cudaStream_t cs = reinterpret_cast<cudaStream_t>(s);
    static thread_local uint32_t h[kStatsWords];
    DYPH_CUDA_TRY(cudaMemcpyAsync(h, w->stats, sizeof(h), cudaMemcpyDeviceToHost, cs));
    DYPH_CUDA_TRY(cudaStreamSynchronize(cs));
    const uint32_t total = h[5];
    if (frames_total) *frames_total = total;
    // most recent min(cap, total, kHistory) frames, oldest first
    uint32_t m = total < kHistory ? total : kHistory;
    if (m > cap) m = cap;
    for (uint32_t i = 0; i < m; ++i) {
        const uint32_t f = total - m + i;
        if (pairs) pairs[i] = h[8 + 2 * (f % kHistory)];
        if (contacts) contacts[i] = h[9 + 2 * (f % kHistory)];
    }
    return DYPH_OK;
}

extern "C" dyph_status dyph_world_broadphase(dyph_world* w, dyph_broadphase** out) {
    if (!w || !out) return DYPH_ERR_INVALID;
    *out = w->bp;
    return DYPH_OK;
}
extern "C" dyph_status dyph_world_narrowphase(dyph_world* w, dyph_narrowphase** out) {
    if (!w || !out) return DYPH_ERR_INVALID;
    *out = w->np;
    return DYPH_OK;
}
extern "C" dyph_status dyph_world_solver(dyph_world* w, dyph_xpbd** out) {
    if (!w || !out) return DYPH_ERR_INVALID;
    *out = w->sv;
    return DYPH_OK;
}

namespace {

// Fused frames for batched scenes: per-scene pair / contact slots sized as the
// scene's own capacities when stepped alone (48 n + 64 pairs, 16 n + 64
// contacts), and one block's shared memory for the largest scene's bodies
// plus about two contacts per body.
// Shared memory a block needs for the largest scene's bodies plus its pair
// and contact words, and the least it can run with (bodies plus 64 contacts'
// words; pair and contact lists then live in global memory).
constexpr uint32_t kMaxSmem = 200u * 1024u;

uint32_t fused_smem_need(uint32_t max_nb) {
    return std::min(kMaxSmem, frame_body_bytes(max_nb) + (4u + kSceneWords * 4u) * 2u * std::max(64u, max_nb));
}
uint32_t fused_smem_floor(uint32_t max_nb) { return frame_body_bytes(max_nb) + 56u * 64u; }

// Work items, largest scenes first: a scene whose estimated shared-memory
// need fits a quarter of the block's (`share`) runs on a quarter of the block,
// four such scenes to a block (teams >= 1); one that fits half of it on half the
// block (teams == 2); larger scenes take the whole block.
template <class Est>
void build_items(const uint32_t* body_offset, uint32_t n_scenes, uint32_t share, uint32_t teams, Est est,
                 std::vector<uint32_t>& items, uint32_t& n_small, uint32_t& n_mid) {
    std::vector<uint32_t> order(n_scenes);
    for (uint32_t i = 0; i < n_scenes; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [body_offset](uint32_t x, uint32_t y) {
        return body_offset[x + 1] - body_offset[x] > body_offset[y + 1] - body_offset[y];
    });
    items.clear();
    std::vector<uint32_t> small, mid;
    for (uint32_t s : order) {
        const uint32_t e = est(body_offset[s + 1] - body_offset[s]);
        if (teams >= 1 && e <= share) {
            small.push_back(s);
        } else if (teams >= 2 && e <= 2u * share) {
            mid.push_back(s);
        } else {
            items.insert(items.end(), {s, kItemBlock, kItemEmpty, kItemEmpty});
        }
    }
    for (size_t i = 0; i < mid.size(); i += 2)
        items.insert(items.end(), {mid[i], kItemHalf, i + 1 < mid.size() ? mid[i + 1] : kItemEmpty, kItemHalf});
    for (size_t i = 0; i < small.size(); i += 4)
        for (size_t j = 0; j < 4; ++j) items.push_back(i + j < small.size() ? small[i + j] : kItemEmpty);
    n_small = static_cast<uint32_t>(small.size());
    n_mid = static_cast<uint32_t>(mid.size());
}

// The fused kernels may take up to kMaxSmem of dynamic shared memory, set
// once per device: the attribute belongs to the kernel, not to a world, so a
// world that lowered it would make another world's launches fail.
constexpr int kFusedMaxDevices = 64;
std::mutex g_fused_smem_mu;
bool g_fused_smem[kFusedMaxDevices] = {};

dyph_status fused_smem_prepare() {
    int dev = 0;
    DYPH_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kFusedMaxDevices) return DYPH_ERR_INVALID;
    std::lock_guard<std::mutex> lock(g_fused_smem_mu);
    if (g_fused_smem[dev]) return DYPH_OK;
    for (const void* k : {reinterpret_cast<const void*>(scene_frame_kernel<4, kSceneThreads>),
                          reinterpret_cast<const void*>(scene_frame_kernel<5, kSceneThreads>),
                          reinterpret_cast<const void*>(scene_frame_kernel<6, kSceneThreads>),
                          reinterpret_cast<const void*>(scene_frame_kernel<2, kSceneWideThreads>),
                          reinterpret_cast<const void*>(scene_single_kernel<kSceneWideThreads>),
                          reinterpret_cast<const void*>(scene_frame_record_kernel<4, kSceneThreads>),
                          reinterpret_cast<const void*>(scene_frame_record_kernel<2, kSceneWideThreads>),
                          reverse_kernel()})
        DYPH_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kMaxSmem)));
    g_fused_smem[dev] = true;
    return DYPH_OK;
}

// Dynamic shared memory per block with which `blocks` blocks of `kernel`
// share an SM, as the occupancy calculator counts it (static shared memory
// and the per-block reservation included): the SM's share for one block,
// lowered in 128-byte steps until that many blocks fit.
uint32_t smem_for_blocks(const void* kernel, int threads, int blocks) {
    int dev = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess) {
        cudaGetLastError();
        return 0u;
    }
    uint32_t bytes = std::min(kMaxSmem, static_cast<uint32_t>(per_sm / blocks)) & ~127u;
    for (; bytes >= 128u; bytes -= 128u) {
        int fit = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kernel, threads, bytes) != cudaSuccess) {
            cudaGetLastError();
            return 0u;
        }
        if (fit >= blocks) return bytes;
    }
    return 0u;
}

// Dynamic shared memory per block when `blocks` blocks of `kernel` split an
// SM's shared memory (its static shared memory and the per-block reservation
// counted), whatever its registers allow.
uint32_t smem_share(const void* kernel, uint32_t blocks) {
    int dev = 0, per_sm = 0, reserved = 0;
    cudaFuncAttributes fa{};
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev) != cudaSuccess ||
        cudaFuncGetAttributes(&fa, kernel) != cudaSuccess) {
        cudaGetLastError();
        return 0u;
    }
    const int64_t bytes = static_cast<int64_t>(per_sm) / blocks - reserved - static_cast<int64_t>(fa.sharedSizeBytes);
    return bytes > 0 ? std::min(kMaxSmem, static_cast<uint32_t>(bytes) & ~127u) : 0u;
}

// The reverse kernel's items and shared memory: per scene its bodies' rows
// plus the contact words and records of about 2.5 contacts per body (a scene
// with more reads them from global memory).
dyph_status setup_reverse(dyph_world* w) {
    const uint32_t n_scenes = static_cast<uint32_t>(w->h_body_offset.size() - 1);
    const uint32_t* off = w->h_body_offset.data();
    uint32_t max_nb = 0;
    for (uint32_t i = 0; i < n_scenes; ++i) max_nb = std::max(max_nb, off[i + 1] - off[i]);
    // Default: a third of an SM's shared memory. The kernel's registers allow
    // two blocks per SM; the smaller blocks leave shared memory to the
    // recording kernel that runs beside it. At least the largest scene's
    // bodies plus 64 contacts' words.
    uint32_t smem = w->r_smem_cap ? std::min(kMaxSmem, w->r_smem_cap & ~15u) : smem_share(reverse_kernel(), 3u);
    smem = std::max(smem, frame_body_bytes(max_nb) + kSceneWords * 4u * 64u);
    if (smem > kMaxSmem) return DYPH_ERR_TOO_LARGE;
    std::vector<uint32_t> items;
    uint32_t n_small = 0, n_mid = 0;
    build_items(off, n_scenes, (smem / 4u) & ~15u, w->r_teams,
                [](uint32_t nb) { return frame_body_bytes(nb) + (kSceneWords + kRecWords) * 10u * nb; }, items,
                n_small, n_mid);
    if (w->r_items) cudaFree(w->r_items);
    w->r_items = nullptr;
    if (cudaMalloc(&w->r_items, items.size() * 4) != cudaSuccess) return DYPH_ERR_NOMEM;
    DYPH_CUDA_TRY(cudaMemcpy(w->r_items, items.data(), items.size() * 4, cudaMemcpyHostToDevice));
    w->r_n_items = static_cast<uint32_t>(items.size() / 4);
    w->r_smem = smem;
    w->r_warp_scenes = n_small;
    w->r_half_scenes = n_mid;
    w->r_block_scenes = n_scenes - n_small - n_mid;
    return setup_done();
}

// The words of a launch's statistics.
dyph_status run_words(dyph_world* w) {
    if (w->f_run) return DYPH_OK;
    const size_t bytes = (kAccWords + static_cast<size_t>(kRunRows) * kMaxRunFrames) * sizeof(uint32_t);
    if (cudaMalloc(&w->f_run, bytes) != cudaSuccess) return DYPH_ERR_NOMEM;
    DYPH_CUDA_TRY(cudaMemset(w->f_run, 0, bytes));
    return DYPH_OK;
}

dyph_status setup_fused(dyph_world* w, uint32_t n_scenes, const uint32_t* body_offset) {
    w->fused = false;
    w->h_body_offset.assign(body_offset, body_offset + n_scenes + 1);
    uint32_t max_nb = 0;
    std::vector<uint32_t> pb(n_scenes + 1, 0u), cb(n_scenes + 1, 0u);
    for (uint32_t i = 0; i < n_scenes; ++i) {
        const uint32_t nb = body_offset[i + 1] - body_offset[i];
        max_nb = std::max(max_nb, nb);
        pb[i + 1] = pb[i] + std::max(64u, 48u * nb + 64u);
        cb[i + 1] = cb[i] + std::max(64u, 16u * nb + 64u);
    }
    if (fused_smem_floor(max_nb) > kMaxSmem) return DYPH_ERR_TOO_LARGE;
    dyph_status prep = fused_smem_prepare();
    if (prep != DYPH_OK) return prep;
    uint32_t smem = fused_smem_need(max_nb);
    if (w->f_smem_cap) {
        smem = std::max(fused_smem_floor(max_nb), std::min(smem, w->f_smem_cap & ~15u));
    } else {
        // With more scenes than SMs, a block that leaves room for a second one
        // on its SM beats one that holds the largest scene whole.
        int dev = 0, sms = 0;
        DYPH_CUDA_TRY(cudaGetDevice(&dev));
        DYPH_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        const uint32_t two = smem_for_blocks(reinterpret_cast<const void*>(scene_frame_kernel<4, kSceneThreads>),
                                             kSceneThreads, 2);
        if (n_scenes > static_cast<uint32_t>(sms) && smem > two && two >= fused_smem_floor(max_nb)) smem = two;
    }
    uint32_t** bufs[] = {&w->f_pair_base, &w->f_contact_base, &w->f_pair_raw, &w->f_contact_raw, &w->f_color_raw,
                         &w->f_counts, &w->f_words, &w->f_pos};
    for (uint32_t** b : bufs) {
        if (*b) cudaFree(*b);
        *b = nullptr;
    }
    if (w->f_items) cudaFree(w->f_items);
    w->f_items = nullptr;
    const size_t pslots = pb[n_scenes], cslots = cb[n_scenes];
    w->f_contact_slots = static_cast<uint32_t>(cslots);
    w->f_pair_slots = static_cast<uint32_t>(pslots);
    w->f_words_stride = static_cast<uint32_t>(cslots + n_scenes);
    const size_t sizes[] = {n_scenes + 1ull, n_scenes + 1ull, pslots, 9 * cslots, cslots, 4ull * n_scenes,
                            static_cast<size_t>(kSceneWords) * w->f_words_stride, 2ull * n_scenes};
    for (int k = 0; k < 8; ++k)
        if (cudaMalloc(bufs[k], sizes[k] * sizeof(uint32_t)) != cudaSuccess) return DYPH_ERR_NOMEM;
    // Work items: a scene's frame is expected to need its bodies' rows plus
    // about 4 pairs and 2.5 contacts per body.
    std::vector<uint32_t> items;
    uint32_t n_small = 0, n_mid = 0;
    build_items(body_offset, n_scenes, (smem / 4u) & ~15u, w->f_teams,
                [](uint32_t nb) { return frame_body_bytes(nb) + 146u * nb; }, items, n_small, n_mid);
    w->f_n_items = static_cast<uint32_t>(items.size() / 4);
    if (cudaMalloc(&w->f_items, items.size() * 4) != cudaSuccess) return DYPH_ERR_NOMEM;
    DYPH_CUDA_TRY(cudaMemcpy(w->f_items, items.data(), items.size() * 4, cudaMemcpyHostToDevice));
    DYPH_CUDA_TRY(cudaMemcpy(w->f_pair_base, pb.data(), pb.size() * 4, cudaMemcpyHostToDevice));
    DYPH_CUDA_TRY(cudaMemcpy(w->f_contact_base, cb.data(), cb.size() * 4, cudaMemcpyHostToDevice));
    DYPH_CUDA_TRY(cudaMemset(w->f_counts, 0, 4ull * n_scenes * sizeof(uint32_t)));
    prep = run_words(w);
    if (prep != DYPH_OK) return prep;
    w->frame_smem = smem;
    {
        int dev = 0, sms = 0, per_sm = 0;
        DYPH_CUDA_TRY(cudaGetDevice(&dev));
        DYPH_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        w->f_threads = kSceneThreads;
        FusedForm form = fused_form(w);
        DYPH_CUDA_TRY(
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, form.kernel, static_cast<int>(form.threads), smem));
        // Blocks of twice the threads where the chip would otherwise hold at most
        // half the warps the registers allow: shared memory for two blocks an SM
        // at most, or at most two blocks per SM in all. A frame with 256 against
        // 128 threads: 220 and 297 us on 1024 mixed scenes (115 KB a block), 64
        // and 67 on 256 push scenes, 46 and 50 on 64 stacks.
        if (w->f_variant == 0 && (per_sm <= 2 || w->f_n_items <= 2u * static_cast<uint32_t>(sms))) {
            w->f_threads = kSceneWideThreads;
            form = fused_form(w);
            DYPH_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, form.kernel,
                                                                        static_cast<int>(form.threads), smem));
        }
        w->f_resident = w->f_n_items <= static_cast<uint32_t>(per_sm) * static_cast<uint32_t>(sms);
    }
    w->f_warp_scenes = n_small;
    w->f_half_scenes = n_mid;
    w->f_block_scenes = n_scenes - n_small - n_mid;
    dyph_status st = setup_reverse(w);
    if (st != DYPH_OK) return st;
    w->fused = true;
    return DYPH_OK;
}

void drop_graphs(dyph_world* w) {
    if (w->graph) cudaGraphExecDestroy(w->graph);
    if (w->episode) cudaGraphExecDestroy(w->episode);
    w->graph = w->episode = nullptr;
    w->episode_frames = 0;
}

void fused_report(const dyph_world* w, dyph_fused_config* out) {
    *out = dyph_fused_config{};
    if (!w->fused) return;
    int per_sm = 0;
    const FusedForm form = fused_form(w);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, form.kernel, static_cast<int>(form.threads), w->frame_smem);
    out->smem_bytes = w->frame_smem;
    out->teams = w->f_teams;
    out->warp_scenes = w->f_warp_scenes;
    out->half_scenes = w->f_half_scenes;
    out->block_scenes = w->f_block_scenes;
    out->blocks = w->f_n_items;
    out->blocks_per_sm = static_cast<uint32_t>(per_sm);
    out->register_blocks = 4u + w->f_variant;
    out->ms_per_frame = w->f_tuned_ms;
    out->candidates = w->f_tuned_candidates;
}

// Tuned configurations, per device and batch profile (scene sizes, solver
// settings), for the life of the process.
struct TunedConfig {
    uint32_t smem_cap;
    uint32_t teams;
    uint32_t variant;
    float ms;
};
std::mutex g_tuned_mu;
std::map<uint64_t, TunedConfig> g_tuned;

uint64_t tune_key(const dyph_world* w) {
    int dev = 0;
    cudaGetDevice(&dev);
    uint64_t h = 0xcbf29ce484222325ull;
    auto mix = [&h](uint64_t v) {
        for (int b = 0; b < 8; ++b) {
            h ^= (v >> (8 * b)) & 0xFFu;
            h *= 0x100000001b3ull;
        }
    };
    mix(static_cast<uint64_t>(dev));
    mix(static_cast<uint64_t>(w->sv->mode));
    mix(static_cast<uint64_t>(w->sv->n_iters));
    mix(static_cast<uint64_t>(w->desc.integrator.n_substeps));
    for (uint32_t v : w->h_body_offset) mix(v);
    return h;
}

}  // namespace

extern "C" dyph_status dyph_world_sync_lists(dyph_world* w, dyph_stream s) {
    if (!w) return DYPH_ERR_INVALID;
    if (!w->fused) return DYPH_OK;
    cudaStream_t cs = reinterpret_cast<cudaStream_t>(s);
    DYPH_CUDA_TRY(cudaEventRecord(w->ev_in, cs));
    DYPH_CUDA_TRY(cudaStreamWaitEvent(w->stream, w->ev_in, 0));
    const uint32_t n = w->bp->n_scenes;
    scene_gather_scan_kernel<<<1, 1024, 0, w->stream>>>(w->f_counts, n, w->f_pos, w->bp->counts, w->np->counts);
    SceneBufs S{w->bp->body_offset, w->bp->bvh.scene_of, w->sv->scene_order, nullptr, nullptr, 0, n, 0};
    FrameBufs F{w->f_pair_base, w->f_contact_base, w->f_pair_raw, w->f_contact_raw, w->f_color_raw, w->f_counts,
                w->f_words, w->f_words_stride, w->f_contact_slots};
    scene_gather_copy_kernel<<<n, 256, 0, w->stream>>>(S, F, w->f_pos, w->bp->pairs, w->np->view, w->sv->color);
    DYPH_CUDA_TRY(cudaGetLastError());
    DYPH_CUDA_TRY(cudaEventRecord(w->ev_out, w->stream));
    DYPH_CUDA_TRY(cudaStreamWaitEvent(cs, w->ev_out, 0));
    return DYPH_OK;
}

extern "C" dyph_status dyph_world_fused_config(dyph_world* w, dyph_fused_config* out) {
    if (!w || !out) return DYPH_ERR_INVALID;
    fused_report(w, out);
    return DYPH_OK;
}

extern "C" dyph_status dyph_world_set_fused_config(dyph_world* w, uint32_t smem_cap, uint32_t teams,
                                                   uint32_t register_blocks) {
    if (!w || !w->fused || teams > 2u || (register_blocks != 0 && (register_blocks < 4 || register_blocks > 6)))
        return DYPH_ERR_INVALID;
    DYPH_CUDA_TRY(cudaStreamSynchronize(w->stream));
    w->f_smem_cap = smem_cap;
    w->f_teams = teams;
    w->f_variant = register_blocks ? register_blocks - 4u : 0u;
    const std::vector<uint32_t> off = w->h_body_offset;
    dyph_status st = setup_fused(w, static_cast<uint32_t>(off.size() - 1), off.data());
    drop_graphs(w);
    return st;
}

extern "C" dyph_status dyph_world_adjoint_config(dyph_world* w, dyph_fused_config* out) {
    if (!w || !out) return DYPH_ERR_INVALID;
    *out = dyph_fused_config{};
    if (!w->fused) return DYPH_OK;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, reverse_kernel(), kSceneThreads, w->r_smem);
    out->smem_bytes = w->r_smem;
    out->teams = w->r_teams;
    out->warp_scenes = w->r_warp_scenes;
    out->half_scenes = w->r_half_scenes;
    out->block_scenes = w->r_block_scenes;
    out->blocks = w->r_n_items;
    out->blocks_per_sm = static_cast<uint32_t>(per_sm);
    out->register_blocks = 2u;
    return DYPH_OK;
}

extern "C" dyph_status dyph_world_set_adjoint_config(dyph_world* w, uint32_t smem_bytes, uint32_t teams) {
    if (!w || !w->fused || teams > 2u) return DYPH_ERR_INVALID;
    DYPH_CUDA_TRY(cudaStreamSynchronize(w->stream));
    w->r_smem_cap = smem_bytes;
    w->r_teams = teams;
    return setup_reverse(w);
}

extern "C" dyph_status dyph_world_autotune(dyph_world* w, int32_t frames, dyph_stream s, dyph_fused_config* out) {
    if (!w || !w->fused || frames <= 0) return DYPH_ERR_INVALID;
    cudaStream_t cs = reinterpret_cast<cudaStream_t>(s);
    DYPH_CUDA_TRY(cudaStreamSynchronize(w->stream));
    DYPH_CUDA_TRY(cudaStreamSynchronize(cs));
    const uint64_t key = tune_key(w);
    {
        std::lock_guard<std::mutex> lock(g_tuned_mu);
        auto it = g_tuned.find(key);
        if (it != g_tuned.end()) {
            dyph_status st =
                dyph_world_set_fused_config(w, it->second.smem_cap, it->second.teams, 4u + it->second.variant);
            w->f_tuned_ms = it->second.ms;
            w->f_tuned_candidates = 0;  // taken from the cache
            if (out) fused_report(w, out);
            return st;
        }
    }
    const size_t n = w->desc.bodies.n;
    uint32_t max_nb = 0;
    for (size_t k = 0; k + 1 < w->h_body_offset.size(); ++k)
        max_nb = std::max(max_nb, w->h_body_offset[k + 1] - w->h_body_offset[k]);
    // The state, the statistics and the phase timer are put back after the trials.
    float* saved = nullptr;
    uint32_t saved_stats[5];
    if (cudaMalloc(&saved, 13 * n * sizeof(float)) != cudaSuccess) return DYPH_ERR_NOMEM;
    float* rows[13] = {w->desc.bodies.pos_x, w->desc.bodies.pos_y, w->desc.bodies.pos_z, w->desc.bodies.rot_w,
                       w->desc.bodies.rot_x, w->desc.bodies.rot_y, w->desc.bodies.rot_z, w->desc.bodies.vel_x,
                       w->desc.bodies.vel_y, w->desc.bodies.vel_z, w->desc.bodies.ang_x, w->desc.bodies.ang_y,
                       w->desc.bodies.ang_z};
    auto copy_rows = [&](bool save) -> cudaError_t {
        for (int r = 0; r < 13; ++r) {
            cudaError_t e = save ? cudaMemcpyAsync(saved + r * n, rows[r], n * 4, cudaMemcpyDeviceToDevice, w->stream)
                                 : cudaMemcpyAsync(rows[r], saved + r * n, n * 4, cudaMemcpyDeviceToDevice, w->stream);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    };
    dyph_status st = DYPH_OK;
    unsigned long long* phase = w->f_phase;
    w->f_phase = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    const uint32_t need = fused_smem_need(max_nb), floor_ = fused_smem_floor(max_nb);
    // caps below the need down to the floor itself (the least a block can hold)
    std::vector<uint32_t> caps = {need};
    for (uint32_t c : {96u << 10, 72u << 10, 56u << 10, 48u << 10, 44u << 10, 40u << 10, 32u << 10})
        if (c < need && c >= floor_) caps.push_back(c);
    if (floor_ < need && std::find(caps.begin(), caps.end(), floor_) == caps.end()) caps.push_back(floor_);
    TunedConfig best{need, 2u, 0u, 1e30f};
    uint32_t tried = 0;
    const uint32_t cap0 = w->f_smem_cap, variant0 = w->f_variant;
    const uint32_t teams0 = w->f_teams;
    do {
        if (cudaMemcpyAsync(saved_stats, w->stats, sizeof(saved_stats), cudaMemcpyDeviceToHost, w->stream) !=
                cudaSuccess ||
            copy_rows(true) != cudaSuccess || cudaEventCreate(&e0) != cudaSuccess ||
            cudaEventCreate(&e1) != cudaSuccess) {
            st = DYPH_ERR_CUDA;
            break;
        }
        for (uint32_t cap : caps) {
            for (uint32_t combo = 0; combo < 9u && st == DYPH_OK; ++combo) {
                const uint32_t teams = 2u - combo / 3u;
                const uint32_t variant = combo % 3u;
                w->f_smem_cap = cap;
                w->f_teams = teams;
                w->f_variant = variant;
                st = setup_fused(w, static_cast<uint32_t>(w->h_body_offset.size() - 1), w->h_body_offset.data());
                if (st != DYPH_OK) break;
                // one untimed frame, then the timed ones launched as a call's, each trial from the saved state
                st = launch_run(w, FusedRun{1u, false}, w->stream);
                if (st == DYPH_OK && cudaEventRecord(e0, w->stream) != cudaSuccess) st = DYPH_ERR_CUDA;
                const uint32_t all = static_cast<uint32_t>(frames), run = w->f_resident ? kMaxRunFrames : 1u;
                for (uint32_t f = 0; f < all && st == DYPH_OK; f += run)
                    st = launch_run(w, FusedRun{std::min(all - f, run), all - f <= run}, w->stream);
                if (st == DYPH_OK && cudaEventRecord(e1, w->stream) != cudaSuccess) st = DYPH_ERR_CUDA;
                if (st == DYPH_OK && (copy_rows(false) != cudaSuccess || cudaStreamSynchronize(w->stream) != cudaSuccess))
                    st = DYPH_ERR_CUDA;
                float ms = 0.f;
                if (st == DYPH_OK && cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess) st = DYPH_ERR_CUDA;
                if (st != DYPH_OK) break;
                ++tried;
                ms /= static_cast<float>(frames);
                if (ms < best.ms) best = TunedConfig{cap, teams, variant, ms};
            }
            if (st != DYPH_OK) break;
        }
    } while (false);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    w->f_phase = phase;
    if (st == DYPH_OK) {
        w->f_smem_cap = best.smem_cap;
        w->f_teams = best.teams;
        w->f_variant = best.variant;
    } else {
        w->f_smem_cap = cap0;
        w->f_teams = teams0;
        w->f_variant = variant0;
    }
    const dyph_status st2 = setup_fused(w, static_cast<uint32_t>(w->h_body_offset.size() - 1), w->h_body_offset.data());
    drop_graphs(w);
    if (st == DYPH_OK && st2 == DYPH_OK) {
        if (cudaMemcpyAsync(w->stats, saved_stats, sizeof(saved_stats), cudaMemcpyHostToDevice, w->stream) !=
                cudaSuccess ||
            cudaStreamSynchronize(w->stream) != cudaSuccess)
            st = DYPH_ERR_CUDA;
        w->f_tuned_ms = best.ms;
        w->f_tuned_candidates = tried;
        std::lock_guard<std::mutex> lock(g_tuned_mu);
        g_tuned[key] = best;
    }
    cudaFree(saved);
    if (out) fused_report(w, out);
    return st != DYPH_OK ? st : st2;
}

extern "C" dyph_status dyph_world_set_scenes(dyph_world* w, uint32_t n_scenes, const uint32_t* body_offset,
                                             const dyph_aabb* scene_bounds) {
    if (!w || !body_offset || n_scenes == 0 || body_offset[n_scenes] != w->desc.bodies.n) return DYPH_ERR_INVALID;
    DYPH_CUDA_TRY(cudaStreamSynchronize(w->stream));
    dyph_status st = broadphase_set_scenes(w->bp, n_scenes, body_offset, scene_bounds);
    if (st != DYPH_OK) return st;
    // One block per scene when the largest scene fits a block; otherwise the
    // whole-batch kernels solve the batch.
    st = xpbd_set_scenes(w->sv, n_scenes, body_offset, w->bp->body_offset, w->bp->bvh.scene_of);
    if (st != DYPH_OK && st != DYPH_ERR_TOO_LARGE) return st;
    if (st == DYPH_OK) {
        st = setup_fused(w, n_scenes, body_offset);
        if (st != DYPH_OK && st != DYPH_ERR_TOO_LARGE) return st;
    }
    if (w->s_buf) cudaFree(w->s_buf);  // a batch has no use for it
    w->s_buf = nullptr;
    // Captured frames launch the single-scene form: record them again.
    if (w->graph) cudaGraphExecDestroy(w->graph);
    if (w->episode) cudaGraphExecDestroy(w->episode);
    w->graph = nullptr;
    w->episode = nullptr;
    w->episode_frames = 0;
    if (w->scene_hash) cudaFree(w->scene_hash);
    w->scene_hash = nullptr;
    if (cudaMalloc(&w->scene_hash, n_scenes * sizeof(uint64_t)) != cudaSuccess) return DYPH_ERR_NOMEM;
    return DYPH_OK;
}

extern "C" dyph_status dyph_world_scene_hashes(dyph_world* w, dyph_stream s, uint64_t* host_out, uint32_t cap) {
    if (!w || !host_out) return DYPH_ERR_INVALID;
    cudaStream_t cs = reinterpret_cast<cudaStream_t>(s);
    const uint32_t n = w->bp->n_scenes ? w->bp->n_scenes : 1u;
    if (cap < n) return DYPH_ERR_INVALID;
    if (!w->scene_hash && cudaMalloc(&w->scene_hash, sizeof(uint64_t)) != cudaSuccess) return DYPH_ERR_NOMEM;
    dyph_status st = fnv_state(&w->desc.bodies, w->bp->n_scenes ? w->bp->body_offset : nullptr, n, w->scene_hash, cs);
    if (st != DYPH_OK) return st;
    DYPH_CUDA_TRY(cudaMemcpyAsync(host_out, w->scene_hash, n * sizeof(uint64_t), cudaMemcpyDeviceToHost, cs));
    DYPH_CUDA_TRY(cudaStreamSynchronize(cs));
    return DYPH_OK;
}

extern "C" dyph_status dyph_world_set_trajectory(dyph_world* w, float* host_dst, uint32_t every,
                                                 uint32_t max_records) {
    if (!w || (host_dst && (every == 0 || max_records == 0))) return DYPH_ERR_INVALID;
    DYPH_CUDA_TRY(cudaStreamSynchronize(w->stream));
    if (w->traj_stream) DYPH_CUDA_TRY(cudaStreamSynchronize(w->traj_stream));
    // A captured episode has the old recording baked in.
    if (w->episode) {
        cudaGraphExecDestroy(w->episode);
        w->episode = nullptr;
        w->episode_frames = 0;
    }
    w->traj_host = host_dst;
    w->traj_every = every;
    w->traj_max = max_records;
    w->traj_frame = 0;
    w->traj_chunk = 0;
    w->traj_pending = false;
    w->traj_live[0] = w->traj_live[1] = false;
    if (!host_dst) return DYPH_OK;
    cudaPointerAttributes attr{};
    if (cudaPointerGetAttributes(&attr, host_dst) != cudaSuccess || attr.type != cudaMemoryTypeHost) {
        cudaGetLastError();
        w->traj_host = nullptr;
        return DYPH_ERR_INVALID;  // pageable memory: the copies could not run asynchronously or be captured
    }
    // A single scene's frames are recorded one by one, a fused batch's a few to
    // a launch: staging buffers of at most 64 MiB and 8 records.
    const size_t bytes = 7ull * w->desc.bodies.n * sizeof(float);
    const uint32_t slots =
        w->fused ? static_cast<uint32_t>(std::clamp<size_t>((size_t(64) << 20) / bytes, 1, 8)) : 1u;
    for (int k = 0; k < 2; ++k) {
        if (w->traj_stage[k] && slots > w->traj_slots) {
            cudaFree(w->traj_stage[k]);
            w->traj_stage[k] = nullptr;
        }
        if (!w->traj_stage[k] && cudaMalloc(&w->traj_stage[k], slots * bytes) != cudaSuccess) {
            w->traj_host = nullptr;
            w->traj_slots = 0;
            return DYPH_ERR_NOMEM;
        }
        if (!w->traj_packed[k]) DYPH_CUDA_TRY(cudaEventCreateWithFlags(&w->traj_packed[k], cudaEventDisableTiming));
        if (!w->traj_copied[k]) DYPH_CUDA_TRY(cudaEventCreateWithFlags(&w->traj_copied[k], cudaEventDisableTiming));
    }
    if (!w->traj_stream) DYPH_CUDA_TRY(cudaStreamCreateWithFlags(&w->traj_stream, cudaStreamNonBlocking));
    w->traj_slots = std::max(w->traj_slots, slots);
    return DYPH_OK;
}

extern "C" dyph_status dyph_world_set_phase_timing(dyph_world* w, int on) {
    if (!w) return DYPH_ERR_INVALID;
    if (!w->fused) return on ? DYPH_ERR_INVALID : DYPH_OK;
    DYPH_CUDA_TRY(cudaStreamSynchronize(w->stream));
    // captured frames hold the old setting
    if (w->graph) cudaGraphExecDestroy(w->graph);
    if (w->episode) cudaGraphExecDestroy(w->episode);
    w->graph = w->episode = nullptr;
    w->episode_frames = 0;
    if (!on) {
        if (w->f_phase) cudaFree(w->f_phase);
        w->f_phase = nullptr;
        return DYPH_OK;
    }
    if (!w->f_phase && cudaMalloc(&w->f_phase, kFramePhases * sizeof(unsigned long long)) != cudaSuccess)
        return DYPH_ERR_NOMEM;
    DYPH_CUDA_TRY(cudaMemset(w->f_phase, 0, kFramePhases * sizeof(unsigned long long)));
    return setup_done();
}

extern "C" dyph_status dyph_world_download_phase_ns(dyph_world* w, dyph_stream s, uint64_t* out, uint32_t cap) {
    if (!w || !out || cap < static_cast<uint32_t>(kFramePhases) || !w->f_phase) return DYPH_ERR_INVALID;
    cudaStream_t cs = reinterpret_cast<cudaStream_t>(s);
    DYPH_CUDA_TRY(cudaMemcpyAsync(out, w->f_phase, kFramePhases * sizeof(uint64_t), cudaMemcpyDeviceToHost, cs));
    DYPH_CUDA_TRY(cudaMemsetAsync(w->f_phase, 0, kFramePhases * sizeof(uint64_t), cs));
    DYPH_CUDA_TRY(cudaStreamSynchronize(cs));
    return DYPH_OK;
}

namespace dyph {
namespace {

// A BodyView over a [13][n] state buffer, with the world's constant rows.
dyph_bodies state_view(const dyph_world* w, float* st) {
    dyph_bodies v = w->desc.bodies;
    const size_t n = v.n;
    float** rows[13] = {&v.pos_x, &v.pos_y, &v.pos_z, &v.rot_w, &v.rot_x, &v.rot_y, &v.rot_z,
                        &v.vel_x, &v.vel_y, &v.vel_z, &v.ang_x, &v.ang_y, &v.ang_z};
    for (int r = 0; r < 13; ++r) *rows[r] = st + r * n;
    return v;
}

// Frames per recorded segment of a backward pass with a checkpoint at every
// frame: enough to record the next segment while one is reversed, with one
// wait between the two streams per segment; fewer when the two segments'
// record sets would pass kRecordBudget bytes.
constexpr int32_t kRecordGroup = 4;
constexpr size_t kRecordBudget = size_t(2) << 30;

// Bytes of one record set (records, poses after integrate, quaternions before
// renormalisation, contact words, counts).
size_t record_set_bytes(const dyph_world* w) {
    return 4 * (static_cast<size_t>(kRecWords) * w->f_contact_slots + 11ull * w->desc.bodies.n +
                static_cast<size_t>(kSceneWords) * w->f_words_stride + 2ull * std::max(w->bp->n_scenes, 1u));
}

// The adjoint's buffers: `sets` record sets and two segment buffers of
// `seg_states` states each. The record sets and the recording's pair slots
// are sized by the scenes' slots, so they are made again after the scenes
// change (dyph_world_set_scenes).
dyph_status adjoint_buffers(dyph_world* w, uint32_t sets, uint32_t seg_states) {
    const size_t n = w->desc.bodies.n;
    const uint32_t n_sc = std::max(w->bp->n_scenes, 1u);
    if (!w->a_g) {
        const bool ok =
            cudaMalloc(&w->a_g, 13 * n * 4) == cudaSuccess && cudaMalloc(&w->a_flag, 4) == cudaSuccess;
        if (!ok) return DYPH_ERR_NOMEM;
        DYPH_CUDA_TRY(cudaStreamCreateWithFlags(&w->a_stream, cudaStreamNonBlocking));
        for (cudaEvent_t* e : {&w->a_seg_ready, &w->a_rtail, &w->a_rev_done})
            DYPH_CUDA_TRY(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
    }
    const uint32_t sized[4] = {w->f_contact_slots, w->f_words_stride, w->f_pair_slots, n_sc};
    if (!std::equal(sized, sized + 4, w->a_sized)) {
        for (size_t k = 0; k < w->a_rec.size(); ++k) {
            void* pk[] = {w->a_rec[k], w->a_pose1[k], w->a_qs[k], w->a_words[k], w->a_mg[k]};
            for (void* p : pk)
                if (p) cudaFree(p);
        }
        w->a_rec.clear();
        w->a_pose1.clear();
        w->a_qs.clear();
        w->a_words.clear();
        w->a_mg.clear();
        if (w->a_sets) cudaFree(w->a_sets);
        w->a_sets = nullptr;
        w->a_sets_n = 0;
        if (w->a_pairs) cudaFree(w->a_pairs);
        w->a_pairs = nullptr;
        std::fill(w->a_sized, w->a_sized + 4, 0u);
        if (cudaMalloc(&w->a_pairs, static_cast<size_t>(std::max(w->f_pair_slots, 1u)) * 4) != cudaSuccess)
            return DYPH_ERR_NOMEM;
        std::copy(sized, sized + 4, w->a_sized);
    }
    while (w->a_rec.size() < sets) {
        float *rec = nullptr, *pose1 = nullptr, *qs = nullptr;
        uint32_t *words = nullptr, *mg = nullptr;
        const bool ok =
            cudaMalloc(&rec, static_cast<size_t>(kRecWords) * w->f_contact_slots * 4) == cudaSuccess &&
            cudaMalloc(&pose1, 7 * n * 4) == cudaSuccess && cudaMalloc(&qs, 4 * n * 4) == cudaSuccess &&
            cudaMalloc(&words, static_cast<size_t>(kSceneWords) * w->f_words_stride * 4) == cudaSuccess &&
            cudaMalloc(&mg, 2ull * n_sc * 4) == cudaSuccess;
        if (!ok) {
            void* pk[] = {rec, pose1, qs, words, mg};
            for (void* p : pk)
                if (p) cudaFree(p);
            return DYPH_ERR_NOMEM;
        }
        w->a_rec.push_back(rec);
        w->a_pose1.push_back(pose1);
        w->a_qs.push_back(qs);
        w->a_words.push_back(words);
        w->a_mg.push_back(mg);
    }
    // (a call that ran out of memory may have left sets that the table does not have)
    if (w->a_sets_n != w->a_rec.size()) {
        std::vector<AdjSet> table(w->a_rec.size());
        for (size_t k = 0; k < table.size(); ++k)
            table[k] = AdjSet{w->a_rec[k], w->a_pose1[k], w->a_qs[k], w->a_words[k], w->a_mg[k]};
        if (w->a_sets) cudaFree(w->a_sets);
        w->a_sets = nullptr;
        w->a_sets_n = 0;
        if (cudaMalloc(&w->a_sets, table.size() * sizeof(AdjSet)) != cudaSuccess) return DYPH_ERR_NOMEM;
        // read by the recordings on a_stream and by the reversals that wait for them
        DYPH_CUDA_TRY(cudaMemcpyAsync(w->a_sets, table.data(), table.size() * sizeof(AdjSet), cudaMemcpyHostToDevice,
                                      w->a_stream));
        w->a_sets_n = table.size();
    }
    if (seg_states > w->a_seg_frames) {
        for (float*& b : w->a_seg) {
            if (b) cudaFree(b);
            b = nullptr;
        }
        w->a_seg_frames = 0;
        for (float*& b : w->a_seg)
            if (cudaMalloc(&b, static_cast<size_t>(seg_states) * 13 * n * 4) != cudaSuccess) return DYPH_ERR_NOMEM;
        w->a_seg_frames = seg_states;
    }
    return DYPH_OK;
}

}  // namespace
}  // namespace dyph

extern "C" dyph_status dyph_world_rollout(dyph_world* w, int32_t n_frames, int32_t every, float* d_ckpt,
                                          dyph_stream s) {
    if (!w || !w->fused || n_frames <= 0 || every <= 0 || !d_ckpt) return DYPH_ERR_INVALID;
    return world_step(w, n_frames, s, d_ckpt, static_cast<uint32_t>(every));
}

extern "C" dyph_status dyph_world_rollout_backward(dyph_world* w, int32_t n_frames, int32_t every,
                                                   const float* d_ckpt, const float* d_grad_final,
                                                   float* d_grad_init, float* d_grad_inv_mass, dyph_stream s) {
    if (!w || !w->fused || n_frames <= 0 || every <= 0 || !d_ckpt || !d_grad_final || !d_grad_init ||
        !d_grad_inv_mass)
        return DYPH_ERR_INVALID;
    // Frames are recorded in segments on a_stream, one launch a segment and one
    // record set per frame; sets alternate between two segments, so segment
    // seg - 1 is recorded while segment seg is reversed on the caller's stream,
    // last frame first. With checkpoints every `every` > 1 frames a segment is a
    // checkpoint's frames; with a checkpoint at every frame it is up to
    // kRecordGroup frames (one frame when that many sets do not fit). The
    // recording loads the segment's first checkpoint and goes on from there.
    int32_t group = every;
    if (every == 1) {
        const size_t sets = kRecordBudget / (2 * record_set_bytes(w));
        group = static_cast<int32_t>(std::max<size_t>(1, std::min<size_t>(kRecordGroup, sets)));
    }
    dyph_status st = DYPH_ERR_NOMEM;
    for (;;) {
        const uint32_t seg_frames = static_cast<uint32_t>(std::min(group, n_frames));
        st = adjoint_buffers(w, 2u * seg_frames, every > 1 ? seg_frames - 1u : 0u);
        if (st == DYPH_ERR_NOMEM) cudaGetLastError();  // the failed allocation
        if (st != DYPH_ERR_NOMEM || every > 1 || group == 1) break;
        group = 1;
    }
    if (st != DYPH_OK) return st;
    const int32_t seg_frames = std::min(group, n_frames);
    const int32_t n_seg = (n_frames + group - 1) / group;
    const size_t n = w->desc.bodies.n;
    cudaStream_t cs = reinterpret_cast<cudaStream_t>(s);
    DYPH_CUDA_TRY(cudaMemsetAsync(w->a_flag, 0, 4, cs));
    DYPH_CUDA_TRY(cudaMemsetAsync(d_grad_inv_mass, 0, n * 4, cs));
    DYPH_CUDA_TRY(cudaMemcpyAsync(w->a_g, d_grad_final, 13 * n * 4, cudaMemcpyDeviceToDevice, cs));
    const dyph_world_desc& d = w->desc;
    const dyph_integrator_params& ip = d.integrator;
    const float sub_dt = ip.dt / static_cast<float>(ip.n_substeps);
    SceneBufs S{w->bp->body_offset, w->bp->bvh.scene_of, w->sv->scene_order, nullptr, nullptr, 0, w->bp->n_scenes,
                w->frame_smem};
    SceneBufs S_rev = S;
    S_rev.smem_bytes = w->r_smem;
    auto seg_len = [&](int32_t seg) { return std::min(group, n_frames - seg * group); };
    auto ckpt = [&](int32_t c) { return d_ckpt + static_cast<size_t>(c) * 13 * n; };
    // Segment seg's frames. The state that the reversal of frame f starts from is
    // its segment's checkpoint, or what its predecessor's recording stored (with a
    // checkpoint at every frame, its own checkpoint, the same bits). The kernels
    // only read a checkpoint.
    auto segment = [&](int32_t seg) {
        float* state1 = every > 1 ? w->a_seg[seg & 1] : const_cast<float*>(ckpt(seg * group)) + 13 * n;
        const float* state0 = ckpt(every > 1 ? seg : seg * group);
        return AdjSegment{w->a_sets + static_cast<size_t>(seg & 1) * seg_frames, w->f_contact_slots,
                          static_cast<uint32_t>(n), w->a_flag, state0, state1, every > 1 ? 1u : 0u};
    };
    auto params = [&](int32_t seg) {
        FrameParams p{};
        p.gb = state_view(w, const_cast<float*>(segment(seg).state0));
        p.gs = d.shapes;
        p.gx = ip.gravity[0];
        p.gy = ip.gravity[1];
        p.gz = ip.gravity[2];
        p.sub_dt = sub_dt;
        p.half_dt = 0.5f * sub_dt;
        p.mu = w->sv->friction;
        p.dt = ip.dt;
        p.n_substeps = ip.n_substeps;
        p.mode = static_cast<int>(w->sv->mode);
        p.n_iters = w->sv->n_iters;
        p.n_frames = static_cast<uint32_t>(seg_len(seg));
        return p;
    };
    // The recordings spill into their own pair slots; the contact words are a set's.
    FrameBufs fb{w->f_pair_base, w->f_contact_base, w->a_pairs, w->f_contact_raw, w->f_color_raw,
                 w->f_counts, nullptr, w->f_words_stride, w->f_contact_slots};
    auto record_segment = [&](int32_t seg) -> dyph_status {
        const bool wide = w->f_threads == static_cast<uint32_t>(kSceneWideThreads);
        const void* kernel =
            wide ? reinterpret_cast<const void*>(scene_frame_record_kernel<2, kSceneWideThreads>)
                 : reinterpret_cast<const void*>(scene_frame_record_kernel<4, kSceneThreads>);
        FrameParams p = params(seg);
        AdjSegment ds = segment(seg);
        void* args[] = {&S, &fb, &p, &ds, &w->f_items, &w->f_n_items};
        DYPH_CUDA_TRY(cudaLaunchKernel(kernel, dim3(w->f_n_items), dim3(w->f_threads), args, w->frame_smem,
                                       w->a_stream));
        DYPH_CUDA_TRY(cudaEventRecord(w->a_seg_ready, w->a_stream));
        return DYPH_OK;
    };
    // everything below starts after the caller's stream
    DYPH_CUDA_TRY(cudaEventRecord(w->a_rtail, cs));
    DYPH_CUDA_TRY(cudaStreamWaitEvent(w->a_stream, w->a_rtail, 0));
    if ((st = record_segment(n_seg - 1)) != DYPH_OK) return st;
    for (int32_t seg = n_seg - 1; seg >= 0; --seg) {
        DYPH_CUDA_TRY(cudaStreamWaitEvent(cs, w->a_seg_ready, 0));
        if (seg > 0) {
            // segment seg - 1's sets and states were last read by segment
            // seg + 1's reverse passes, queued on cs before this point
            if (seg + 1 < n_seg) DYPH_CUDA_TRY(cudaStreamWaitEvent(w->a_stream, w->a_rev_done, 0));
            if ((st = record_segment(seg - 1)) != DYPH_OK) return st;
        }
        AdjFrame G{w->a_g, d_grad_inv_mass};
        FrameParams ps = params(seg);
        AdjSegment ds = segment(seg);
        void* args[] = {&S_rev, &fb, &ps, &ds, &G, &w->r_items, &w->r_n_items};
        DYPH_CUDA_TRY(cudaLaunchKernel(reverse_kernel(), dim3(w->r_n_items), dim3(kSceneThreads), args, w->r_smem, cs));
        DYPH_CUDA_TRY(cudaEventRecord(w->a_rev_done, cs));
    }
    // the side stream ends before the caller's stream goes on
    DYPH_CUDA_TRY(cudaEventRecord(w->a_rtail, w->a_stream));
    DYPH_CUDA_TRY(cudaStreamWaitEvent(cs, w->a_rtail, 0));
    DYPH_CUDA_TRY(cudaMemcpyAsync(d_grad_init, w->a_g, 13 * n * 4, cudaMemcpyDeviceToDevice, cs));
    uint32_t flag = 0;
    DYPH_CUDA_TRY(cudaMemcpyAsync(&flag, w->a_flag, 4, cudaMemcpyDeviceToHost, cs));
    DYPH_CUDA_TRY(cudaStreamSynchronize(cs));
    return flag ? DYPH_ERR_UNSUPPORTED : DYPH_OK;
}
