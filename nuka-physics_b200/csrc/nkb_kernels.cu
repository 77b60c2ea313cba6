// Host side of the kernels: picks the step-kernel variant of a world, and the small reset / observation kernels.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdio>
#include "nkb_launch.h"

namespace nkb {

// Per-env reset from the creation snapshot (reference ops/readout.cu:771-776 RestoreState semantics).
__global__ void reset_kernel(ResetParams r) {
    const uint32_t slot = blockIdx.x;
    const uint32_t env = r.env_ids != nullptr ? r.env_ids[slot] : slot;
    if (env >= r.env_count) return;
    if (r.env_ids == nullptr && r.env_mask != nullptr && r.env_mask[env] == 0u) return;
    for (uint32_t f = 0u; f < r.field_count; ++f) {
        const ResetField fd = r.fields[f];
        uint32_t* dst = reinterpret_cast<uint32_t*>(fd.dst) + (size_t)env * fd.words;
        const uint32_t* src = reinterpret_cast<const uint32_t*>(fd.src);
        for (uint32_t k = threadIdx.x; k < fd.words; k += blockDim.x) dst[k] = fd.per_env_src ? src[(size_t)env * fd.words + k] : (fd.src != nullptr ? src[k] : fd.fill);
    }
}

extern const StepVariant kStepBodies, kStepBare, kStepBareSlim, kStepBareControl, kStepNarrow, kStepNarrowSlim, kStepNarrowRigid, kStepWide, kStepWideRigid;
extern const StepVariant kStepNarrowControl, kStepNarrowRigidControl, kStepWideControl, kStepWideRigidControl;

extern const StepVariant kStagesNarrow, kSolveNarrow, kStagesNarrowRigid, kSolveNarrowRigid, kStagesWide, kSolveWide;

bool step_kernel_has_slim(const TemplateView& t) {
    return t.ndof <= 32u && t.n_free == 0u && t.cfg.control_mode != 3u && t.cfg.control_mode != 4u;
}

static bool has_contacts(const TemplateView& t) { return t.B != 0u && t.cfg.max_contacts != 0u; }

// no articulation, up to 32 or up to 64 coordinates per articulation; with or without free rigid bodies; the slim
// (128-register) build exists for articulations of up to 32 without bodies only
static const StepVariant& step_variant(const TemplateView& t, bool slim) {
    // control modes 3 and 4 run the builds that hold the controllers
    const bool control = t.cfg.control_mode == 3u || t.cfg.control_mode == 4u;
    if (t.L == 0u && t.n_free != 0u) return kStepBodies;
    if (!has_contacts(t) && t.n_free == 0u && t.ndof <= 32u) return control ? kStepBareControl : slim ? kStepBareSlim : kStepBare;
    if (control) return t.ndof > 32u ? (t.n_free != 0u ? kStepWideRigidControl : kStepWideControl) : (t.n_free != 0u ? kStepNarrowRigidControl : kStepNarrowControl);
    if (t.ndof > 32u) return t.n_free != 0u ? kStepWideRigid : kStepWide;
    if (t.n_free != 0u) return kStepNarrowRigid;
    return slim ? kStepNarrowSlim : kStepNarrow;
}

int step_kernel_registers(const TemplateView& t, bool slim) { return step_variant(t, slim).registers(); }

int step_kernel_resident_blocks(const TemplateView& t, bool slim, uint32_t warps_per_block, size_t shared_bytes) {
    return step_variant(t, slim).resident_blocks(warps_per_block, shared_bytes);
}

cudaError_t launch_step(const StepParams& p, uint32_t warps_per_block, bool slim, cudaStream_t stream) {
    return step_variant(p.t, slim).launch(p, warps_per_block, stream);
}

const StepVariant* split_variant(uint32_t ndof, uint32_t n_free, bool control, StepPart part) {
    if (control || (ndof > 32u && n_free != 0u)) return nullptr;
    if (ndof > 32u) return part == kPartStages ? &kStagesWide : &kSolveWide;
    if (n_free != 0u) return part == kPartStages ? &kStagesNarrowRigid : &kSolveNarrowRigid;
    return part == kPartStages ? &kStagesNarrow : &kSolveNarrow;
}

// Value k of an env's observation record (the reference's gym layer builds the record with a chain of torch ops on the field views,
// python/nuka/tasks/go2_obs.py:282-305).  `action` is the env's last action of the value's joint.
static __device__ float observation_value(const StateView& s, uint32_t L, const ObservationParams& o, uint32_t env, uint32_t k, float action) {
    const uint32_t nj = L - 1u;
    const float* twist = s.link_vel + (size_t)env * L * 6u;              // root link: angular (3) then linear (3), base frame
    float v;
    if (k < 3u) v = twist[3u + k] * o.lin_vel_scale;
    else if (k < 6u) v = twist[k - 3u] * o.ang_vel_scale;
    else if (k < 9u) {
        // world (0, 0, -1) in the base frame: R(q)^T g = (w^2 - |u|^2) g - 2 w (u x g) + 2 u (u . g), python/nuka/tasks/go2_obs.py:96-112
        const float* pose = s.link_pose + (size_t)env * L * 7u;
        const float w = pose[3], x = pose[4], y = pose[5], z = pose[6];
        const float a = w * w - (x * x + y * y + z * z);
        const float cross[3] = {-y, x, 0.f};                             // u x g with g = (0, 0, -1)
        const float u[3] = {x, y, z};
        const float g[3] = {0.f, 0.f, -1.f};
        const uint32_t c = k - 6u;
        v = a * g[c] - 2.0f * w * cross[c] + 2.0f * u[c] * (-z);
    } else if (k < 12u) {
        const uint32_t c = k - 9u;
        v = o.command[(size_t)env * o.command_stride + c] * o.command_scale[c];
    } else if (k < 12u + 2u * nj) {
        const bool vel = k >= 12u + nj;
        const uint32_t i = k - 12u - (vel ? nj : 0u);
        const uint32_t slot = o.joint_order != nullptr ? o.joint_order[i] : i;
        const size_t src = (size_t)env * L + 1u + slot;
        v = vel ? s.qdot[src] * o.dof_vel_scale
                : (s.q[src] - (o.default_position != nullptr ? o.default_position[i] : 0.f)) * o.dof_pos_scale;
    } else v = action;
    return fminf(fmaxf(v, -o.clip), o.clip);
}

// One observation record per env, composed from the state arrays in one pass.  One thread per output value; the record is short, so
// consecutive threads write consecutive floats.
__global__ void pack_observations_kernel(const __grid_constant__ StateView s, uint32_t L, const __grid_constant__ ObservationParams o, float* out) {
    const uint32_t nj = L - 1u, record = 12u + 3u * nj, width = record + (o.reward != nullptr ? 1u : 0u);
    const size_t total = (size_t)s.env_count * width;
    for (size_t at = (size_t)blockIdx.x * blockDim.x + threadIdx.x; at < total; at += (size_t)gridDim.x * blockDim.x) {
        const uint32_t env = (uint32_t)(at / width), k = (uint32_t)(at % width);
        float v;
        if (k == record) v = o.reward[env];                              // the reward rides along unclipped
        else v = observation_value(s, L, o, env, k, k >= record - nj && o.last_action != nullptr ? o.last_action[(size_t)env * nj + (k - (record - nj))] : 0.f);
        out[(size_t)env * o.row_stride + k] = v;
    }
}

// ---- an episode loop's work around the step, in the caller's place (nuka/vec_env.py) ------------------------------------------
// Three launches for what takes about thirty tensor operations (a pass of 4 steps of 1 quadruped 646 us with those, 585 so; of 1000
// 1203 and 1084).  Products and sums round one by one, as the tensor operations do.

// Actions, clipped, become drive targets in the library's joint order and the last action of the observations.
__global__ void apply_actions_kernel(const __grid_constant__ StateView s, uint32_t L, const __grid_constant__ EpisodeParams p) {
    const uint32_t nj = L - 1u;
    const size_t total = (size_t)s.env_count * nj;
    for (size_t at = (size_t)blockIdx.x * blockDim.x + threadIdx.x; at < total; at += (size_t)gridDim.x * blockDim.x) {
        const uint32_t env = (uint32_t)(at / nj), i = (uint32_t)(at % nj);
        float a = p.actions[at];
        a = a < -p.action_clip ? -p.action_clip : a > p.action_clip ? p.action_clip : a;           // NaN stays
        p.last_action[at] = a;
        s.drive_target[(size_t)env * L + 1u + p.joint_order[i]] = __fadd_rn(p.default_position[i], __fmul_rn(p.action_scale, a));
    }
}

// Reward, termination and truncation of every env after the step; lane = env.
__global__ void judge_episodes_kernel(const __grid_constant__ StateView s, uint32_t L, const __grid_constant__ EpisodeParams p) {
    const uint32_t env = blockIdx.x * blockDim.x + threadIdx.x;
    if (env >= s.env_count) return;
    const int32_t steps = p.episode_steps[env] + 1;
    p.episode_steps[env] = steps;
    const float* base = s.base_pose + (size_t)env * 7u;
    const float z = base[2], off = __fsub_rn(s.link_vel[(size_t)env * L * 6u + 3u], p.command[0]);
    const float low = __fsub_rn(0.25f, z);
    p.reward[env] = __fsub_rn(expf(__fmul_rn(-4.0f, __fmul_rn(off, off))), __fmul_rn(2.0f, low < 0.f ? 0.f : low));
    const float up = __fsub_rn(1.0f, __fmul_rn(2.0f, __fadd_rn(__fmul_rn(base[4], base[4]), __fmul_rn(base[5], base[5]))));
    const bool fallen = z < p.termination_height || up < p.min_up || s.status[env] != 0u, late = steps >= p.max_episode_length;
    p.terminated[env] = fallen; p.truncated[env] = late && !fallen; p.done[env] = fallen || late;
    p.done_mask[env] = fallen || late ? 1u : 0u;
}

// After the reset of the finished envs: their targets, last actions and step counts begin again; every env's observation record goes
// to `out` and to `copy`.
__global__ void observe_episodes_kernel(const __grid_constant__ StateView s, uint32_t L, const __grid_constant__ ObservationParams o,
                                        const __grid_constant__ EpisodeParams p, float* out, float* copy) {
    const uint32_t nj = L - 1u, width = 12u + 3u * nj;
    const size_t total = (size_t)s.env_count * width;
    for (size_t at = (size_t)blockIdx.x * blockDim.x + threadIdx.x; at < total; at += (size_t)gridDim.x * blockDim.x) {
        const uint32_t env = (uint32_t)(at / width), k = (uint32_t)(at % width);
        const bool fresh = p.done_mask[env] != 0u;
        float action = 0.f;
        if (k >= width - nj) {
            float* last = p.last_action + (size_t)env * nj + (k - (width - nj));
            action = *last;
            if (fresh) { action = __fmul_rn(action, 0.f); *last = action; }
        }
        if (fresh && k < L) s.drive_target[(size_t)env * L + k] = p.default_targets[(size_t)env * L + k];
        if (fresh && k == 0u) p.episode_steps[env] = 0;
        const float v = observation_value(s, L, o, env, k, action);
        out[at] = v;
        copy[at] = v;
    }
}

static uint32_t stride_blocks(size_t total) { return (uint32_t)std::min<size_t>((total + 255u) / 256u, 148u * 8u); }

cudaError_t launch_apply_actions(const StateView& s, uint32_t L, const EpisodeParams& p, cudaStream_t stream) {
    apply_actions_kernel<<<stride_blocks((size_t)s.env_count * (L - 1u)), 256, 0, stream>>>(s, L, p);
    return cudaGetLastError();
}

cudaError_t launch_judge_episodes(const StateView& s, uint32_t L, const EpisodeParams& p, cudaStream_t stream) {
    judge_episodes_kernel<<<(s.env_count + 127u) / 128u, 128, 0, stream>>>(s, L, p);
    return cudaGetLastError();
}

cudaError_t launch_observe_episodes(const StateView& s, uint32_t L, const ObservationParams& o, const EpisodeParams& p, float* out, float* copy, cudaStream_t stream) {
    observe_episodes_kernel<<<stride_blocks((size_t)s.env_count * (12u + 3u * (L - 1u))), 256, 0, stream>>>(s, L, o, p, out, copy);
    return cudaGetLastError();
}

cudaError_t launch_pack_observations(const StateView& s, uint32_t L, const ObservationParams& o, float* out, cudaStream_t stream) {
    if (s.env_count == 0u || L < 2u) return cudaSuccess;
    const size_t total = (size_t)s.env_count * (12u + 3u * (L - 1u) + (o.reward != nullptr ? 1u : 0u));
    pack_observations_kernel<<<stride_blocks(total), 256, 0, stream>>>(s, L, o, out);
    return cudaGetLastError();
}

cudaError_t launch_reset(const ResetParams& r, uint32_t count, cudaStream_t stream) {
    if (count == 0u) return cudaSuccess;
    reset_kernel<<<count, 128, 0, stream>>>(r);
    return cudaGetLastError();
}

}  // namespace nkb
