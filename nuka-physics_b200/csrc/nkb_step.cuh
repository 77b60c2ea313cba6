// Device code of the fused step kernel: one warp advances one env through the whole pipeline (kinematics, drives,
// dynamics, collision, row assembly, block-descent solve, integration) with every intermediate in the warp's
// shared-memory slice; global memory sees only the env's state.
// The stage order is the reference's nk::Pipeline::BuildInterval (src/nk/pipeline/pipeline.cpp:367-986).
// Each instantiation of step_kernel is compiled in a translation unit of its own (nkb_step_*.cu) so that the
// variants build in parallel; NKB_STEP_VARIANT defines the host-side handle of one.
#pragma once
#include <cuda_runtime.h>
#include <cstdlib>
#include <mutex>
#include "nkb_solver.cuh"
#include "nkb_lbvh.cuh"
#include "nkb_manifold.cuh"
#include "nkb_launch.h"

namespace nkb {

// Torque-free rotation of a free rigid body over one step, in its principal frame (the quantity of the reference's
// SolveFreeRotation, ops/rigid_types.cuh:39-122, used by ops/articulation.cu:1059-1116): the implicit-midpoint form of
// Euler's equations for the scaled angular momentum u,
//     g(u) = u - u0 + c * (m_y m_z, m_z m_x, m_x m_y) = 0,   m = (u0 + u) / 2,   c = dt (a_y - a_z, a_z - a_x, a_x - a_y),
// with a the scaled inverse principal inertias.  Newton's method: the Jacobian is the identity plus three off-diagonal
// pairs, small enough to invert through its column triple products; a step is halved (at most 8 times) until the
// residual's largest component drops; at most 12 steps to 1e-6.  `mid_out` is the midpoint angular velocity.
struct FreeRotation {
    V3 u0, c;
    NKB_DEV V3 midpoint(V3 u) const { return (u0 + u) * 0.5f; }
    NKB_DEV V3 residual(V3 u) const {
        const V3 m = midpoint(u);
        return mk3(u.x - u0.x + c.x * m.y * m.z, u.y - u0.y + c.y * m.z * m.x, u.z - u0.z + c.z * m.x * m.y);
    }
    NKB_DEV static float largest(V3 r) { return fmaxf(fabsf(r.x), fmaxf(fabsf(r.y), fabsf(r.z))); }
    // Newton direction d with (dg/du) d = r at midpoint m, by Cramer's rule on the Jacobian's columns; false when singular
    NKB_DEV bool direction(V3 m, V3 r, V3& d) const {
        const V3 col0 = mk3(1.0f, 0.5f * c.y * m.z, 0.5f * c.z * m.y);
        const V3 col1 = mk3(0.5f * c.x * m.z, 1.0f, 0.5f * c.z * m.x);
        const V3 col2 = mk3(0.5f * c.x * m.y, 0.5f * c.y * m.x, 1.0f);
        const V3 c12 = cross(col1, col2);
        const float det = dot(col0, c12);
        if (!isfinite(det) || fabsf(det) < 1.0e-12f) return false;
        d = mk3(dot(r, c12), dot(col0, cross(r, col2)), dot(col0, cross(col1, r))) * (1.0f / det);
        return true;
    }
};

NKB_DEV bool solve_free_rotation(V3 w0, V3 inv_i, float dt, V3& mid_out) {
    mid_out = mk3(0.f, 0.f, 0.f);
    const V3 momentum = mk3(w0.x / inv_i.x, w0.y / inv_i.y, w0.z / inv_i.z);
    const float scale = FreeRotation::largest(momentum);
    if (scale == 0.0f) return true;                     // at rest
    const V3 a = inv_i * scale;
    FreeRotation eq;
    eq.u0 = momentum * (1.0f / scale);
    eq.c = mk3(dt * (a.y - a.z), dt * (a.z - a.x), dt * (a.x - a.y));
    V3 u = eq.u0;
    for (int newton = 0; newton <= 12; ++newton) {
        const V3 r = eq.residual(u);
        const float size = FreeRotation::largest(r);
        if (!isfinite(size)) return false;
        if (size <= 1.0e-6f) {
            const V3 m = eq.midpoint(u);
            mid_out = mk3(a.x * m.x, a.y * m.y, a.z * m.z);
            return true;
        }
        V3 d;
        if (newton == 12 || !eq.direction(eq.midpoint(u), r, d)) return false;
        float fraction = 1.0f;
        bool improved = false;
        for (int halving = 0; halving < 8 && !improved; ++halving, fraction *= 0.5f) {
            const V3 trial = u - d * fraction;
            const float trial_size = FreeRotation::largest(eq.residual(trial));
            if (isfinite(trial_size) && trial_size < size) { u = trial; improved = true; }
        }
        if (!improved) return false;
    }
    return false;
}

NKB_DEV void stage_integrate_bodies(Env& e, bool use_pseudo) {
    const TemplateView& t = *e.t;
    const float dt = t.cfg.dt;
#pragma unroll 1
    for (uint32_t b = e.lane; b < t.B; b += 32u) {
        if (!(__ldg(t.inv_mass + b) > 0.f) || __ldg(t.body_to_link + b) != kNoLink) continue;
        float* pose = sm_bpose(e, b);
        float* bv = sm_bvel(e, b);
        const V3 inv_i = ld3(t.inv_inertia + 3u * b);
        const Q4 iq = ldq(t.inertial_quat + 4u * b);
        const Q4 principal = qnorm_le(qmul(ldq(pose + 3), iq), 1.0e-12f);
        const V3 w0 = qrot(mkq(principal.w, -principal.x, -principal.y, -principal.z), ld3(bv + 3));
        V3 midpoint;
        if (!solve_free_rotation(w0, inv_i, dt, midpoint)) { e.status |= kStatusGyroFailure; continue; }
        const V3 momentum = qrot(principal, mk3(w0.x / inv_i.x, w0.y / inv_i.y, w0.z / inv_i.z));
        V3 v = ld3(bv);
        const V3 w = qrot(principal, midpoint);
        const V3 ipos = ld3(t.inertial_pos + 3u * b);
        const V3 center = ld3(pose) + qrot(ldq(pose + 3), ipos);
        Q4 q = qnorm_le(qmul(mkq(1.0f, 0.5f * dt * w.x, 0.5f * dt * w.y, 0.5f * dt * w.z), ldq(pose + 3)), 1.0e-12f);
        if (use_pseudo) {
            const float* ps = sm_bpseudo(e, b);
            v = v + ld3(ps);
            q = qnorm_le(qmul(mkq(1.0f, 0.5f * dt * ps[3], 0.5f * dt * ps[4], 0.5f * dt * ps[5]), q), 1.0e-12f);
        }
        stq(pose + 3, q);
        st3(pose, center + v * dt - qrot(q, ipos));
        float winv[6];
        world_inv_inertia(q, iq, inv_i, winv);
        st3(bv + 3, sym_mulv(winv, momentum));
    }
    __syncwarp();
}

// Applied drive efforts from the drives' impulses (ops/articulation.cu:999-1016).
NKB_DEV void stage_readout_drives(Env& e, uint32_t nheads) {
    const TemplateView& t = *e.t;
#pragma unroll 1
    for (uint32_t h = e.lane; h < nheads; h += 32u) {
        // a limit row's slot keeps the multiplier of the velocity solve for the next step (block_descent_tile.cuh:2556)
        if (hu(e, HF_FLAGS, h) & kHeadLimit) e.s->limit_lambda[((size_t)e.env * t.L + hu(e, HF_REF, h)) * 2u + (hf(e, HF_UNITV, h) < 0.f ? 1u : 0u)] = hf(e, HF_LAMX, h);
    }
    float applied = 0.f;
    if (e.lane < t.L && joint_dofs(e.jtype) == 1u) {
        const float impulse = sm_fixed(e)[e.link_dof];
        if (impulse != 0.f) { applied = impulse / t.cfg.dt - e.drive_dissipation * e.qd; e.tau += applied; }
    }
    if (e.lane < t.L) e.s->actuator[(size_t)e.env * t.L + e.lane] = applied;
    __syncwarp();
}

NKB_DEV void stage_store_bodies(Env& e, bool velocities) {
    const TemplateView& t = *e.t;
    float* gp = e.s->body_pose + (size_t)e.env * t.B * 7u;
    const float* sp = e.sm + e.lay->bpose;
#pragma unroll 1
    for (uint32_t k = e.lane; k < t.B * 7u; k += 32u) gp[k] = sp[k];
    if (!velocities) return;
#pragma unroll 1
    for (uint32_t b = e.lane; b < t.B; b += 32u) {
        if (__ldg(t.body_to_link + b) != kNoLink || !(__ldg(t.inv_mass + b) > 0.f)) continue;     // only free dynamic bodies move
        const size_t gb = (size_t)e.env * t.B + b;
        st3(e.s->body_linvel + gb * 3u, ld3(sm_bvel(e, b)));
        st3(e.s->body_angvel + gb * 3u, ld3(sm_bvel(e, b) + 3));
    }
}

// Register cap of the regular builds: one coordinate per lane settles at 167 registers without spills, two at the cap with 16 bytes;
// three warps to a scheduler partition.  Which worlds are worth a build of 128 registers and four warps is the slim build's question
// below.
// NR = coordinates per lane: 1 for articulations of up to 32 coordinates, 2 for up to 64, 0 for worlds without one.
// kRigid = the world has free rigid bodies; without them the rigid-block solver code is compiled out.
// Whole steps with free bodies are held to fewer resident warps by shared memory than by registers, so they take a wider cap: no
// spills, and a team of 8 warps still fits the register file.
#ifndef NKB_MAXNREG
#define NKB_MAXNREG 176
#endif
#ifndef NKB_MAXNREG_RIGID
#define NKB_MAXNREG_RIGID 224
#endif
// The slim build of the same kernel: at 128 registers a fourth warp fits each scheduler partition, so small envs (14 KB
// of shared memory) reach 16 resident warps per SM instead of 12.  It spills about 250 bytes; a world takes it only where the
// extra residency is really there (World::BuildLayout).  The stages of split steps fit 128 registers without spills, the solve
// with 8 bytes (one coordinate per lane, no free bodies).
// Worlds of bodies only run in teams, two piles to an SM: 168 registers for 12 warps, teams of 6 (1024
// piles of 48 boxes, 2 steps: 14.5 ms; 128 registers, teams of 8 and 400 bytes of spills, 15.5; 700 of 24 4.82 and 5.85).
#ifndef NKB_MAXNREG_BODIES
#define NKB_MAXNREG_BODIES 168
#endif
// The parts of split steps, where slices are small: three warps to a partition (solves of quadrupeds with boxes at 224 registers and
// no spills, two: 5.97 ms; at 168, three: 5.41).
#ifndef NKB_MAXNREG_SPLIT
#define NKB_MAXNREG_SPLIT 168
#endif
#ifndef NKB_MAXNREG_SLIM
#define NKB_MAXNREG_SLIM 128
#endif
// Warps that wait for one another after their solves and then go through the straight-line stages (the end of a step, the
// start of the next) side by side, so that they share the fetches of their instructions: about 230 KB of code per step against
// the 128 KB an SM keeps at hand.  Warps at 15 different places of it are stalled on instruction fetch more than half of the
// time (ncu: no_instruction 6.6 of 12.4 cycles per issue; 16 384 quadrupeds, 4 steps: 20.9 ms without any meeting).
// Solves differ by a factor of three between envs, so a fixed group (a block-wide barrier) waits for its slowest member: 40 %
// of the solve time (11.7 ms).  Here the next `group` warps of the block to finish their solves go on together, whoever they
// are, and a warp whose env is done takes the next env of the launch's queue.
// One shared word carries the number of waiting warps (low byte) and a generation; a warp goes on when the generation moves.
// Whoever completes a group moves it, and so does a warp that leaves for good when those that wait are all that are left.  A
// wait that outlasts its cycle budget just ends: who walks with whom changes no result.
struct Rally { uint32_t word, alive; };
constexpr long long kRallyPatience = 100000000ll;        // cycles: about 50 ms
NKB_DEV uint32_t rally_peek(const uint32_t* w) { return *reinterpret_cast<const volatile uint32_t*>(w); }
NKB_DEV void rally_wait(Rally* r, uint32_t group, uint32_t lane) {
    if (group <= 1u) return;
    __syncwarp();
    uint32_t generation = 0u;
    if (lane == 0u) {
        const uint32_t before = atomicAdd(&r->word, 1u);
        generation = before >> 8;
        __threadfence_block();
        if ((before & 0xffu) + 1u >= min(group, rally_peek(&r->alive)))
            for (uint32_t seen = rally_peek(&r->word), found; (seen >> 8) == generation; seen = found)
                if ((found = atomicCAS(&r->word, seen, (generation + 1u) << 8)) == seen) break;
    }
    generation = __shfl_sync(NKB_FULL, generation, 0);
    const long long begin = clock64();
    while ((rally_peek(&r->word) >> 8) == generation) {            // every lane polls the same word: the warp stays together
        if (clock64() - begin > kRallyPatience) break;
        __nanosleep(64);
    }
    __syncwarp();
}
NKB_DEV void rally_leave(Rally* r, uint32_t group, uint32_t lane) {
    if (group <= 1u || lane != 0u) return;
    const uint32_t left = atomicSub(&r->alive, 1u) - 1u;
    __threadfence_block();
    for (uint32_t seen = rally_peek(&r->word), found; (seen & 0xffu) != 0u && (seen & 0xffu) >= min(group, left); seen = found)
        if ((found = atomicCAS(&r->word, seen, ((seen >> 8) + 1u) << 8)) == seen) break;
}

// ---- a step split over launches -------------------------------------------------------------------------------------------
// The straight-line stages of a step are about 170 KB of code that every env runs once, the solve about 60 KB that envs run a
// different number of times.  In one kernel the two fight: warps that run the stages together share the instruction fetches
// (an SM keeps 128 KB at hand; apart from one another they fetch everything again, one instruction in six cycles for the whole
// SM), but then they wait for the longest solve among them.  Split, the stages run in blocks whose warps stay together, and
// the solves run one warp to a block, each SM taking the next env as one finishes.  In between an env's slice of shared memory
// waits in global memory (L2 for the usual batches): only what the other side reads, heads and rows up to the live count.
template <bool kLoad>
NKB_DEV void image_words(float* img, uint32_t at, float* sm, uint32_t to, uint32_t words, uint32_t lane) {
    // regions start on 16-byte boundaries and are padded to them
    float4* g = reinterpret_cast<float4*>(img + at);
    float4* s = reinterpret_cast<float4*>(sm + to);
#pragma unroll 4
    for (uint32_t k = lane; k < (words + 3u) >> 2; k += 32u) { if (kLoad) s[k] = __ldcg(g + k); else __stcg(g + k, s[k]); }
}
// Keeps the warps of a stages block side by side (each passes the same barriers; warps without an env have left).
template <int kPart> NKB_DEV void stay_together() { if constexpr (kPart == kPartStages) __syncthreads(); }
// What crosses: kBefore from the stages to the solve, kAfter from the solve back to the stages, kAside past the solve.
enum ImageSet : int { kBefore = 0, kAfter = 1, kAside = 2 };
template <bool kLoad, int kSet>
NKB_DEV void image_move(Env& e, const StepParams& p, float* img, uint32_t nheads) {
    const TemplateView& t = p.t;
    const SmemLayout &a = p.im, &b = p.sm;
    const uint32_t l = e.lane, slots = t.B != 0u ? t.n_free + 1u : 0u, n4 = (t.ndof + 3u) & ~3u;
    auto move = [&](uint32_t from, uint32_t to, uint32_t words) { if (words != 0u) image_words<kLoad>(img, from, e.sm, to, words, l); };
    if (kSet == kAside) {
        move(a.bpose, b.bpose, 7u * t.B);
        move(a.pairs, b.pairs, t.slot_cap); move(a.cnormal, b.cnormal, 12u * t.slot_cap); move(a.cfeat, b.cfeat, 8u * t.slot_cap);
        return;
    }
    if (kLoad || kSet == kBefore) move(a.fixed, b.fixed, t.ndof);      // the stages' own
    move(a.vel, b.vel, t.L != 0u ? 6u : 0u);
    move(a.bvel, b.bvel, 6u * slots);
    move(a.heads, b.heads, kHeadStride * nheads);
    if (kSet == kBefore) {
        move(a.mass, b.mass, t.ndof * b.ld); move(a.factor, b.factor, b.factor_words);
        move(a.bwinv, b.bwinv, 6u * slots);
        move(a.cdepth, b.cdepth, 4u * t.slot_cap);
        if (kLoad) move(a.jpool, b.jpool, 3u * n4 * e.reach);            // the stages write it in place
    } else {
        move(a.vecs + b.vstride * kVecPseudo, b.vecs + b.vstride * kVecPseudo, t.ndof);
        move(a.bpseudo, b.bpseudo, 6u * slots);
    }
}

template <int NR, bool kRigid, bool kControl, int kPart>
NKB_DEV void advance_env(const StepParams& p, float* sm, uint32_t env, uint32_t lane, Rally* rally) {
    const TemplateView& t = p.t;
    constexpr int K = NR > 0 ? NR : 1;
    const bool has_artic = NR > 0 && t.L != 0u, has_bodies = t.B != 0u;
    const bool has_collidables = kPart != kPartBare && has_bodies && t.cfg.max_contacts != 0u;
    const bool use_pseudo = t.cfg.pos_iters != 0u && (t.cfg.max_contacts != 0u || t.L != 0u);
    Env e;
    env_begin<NR>(e, p, sm, env, lane);
    uint32_t nheads = 0u;
    float* img = nullptr;
    float4* lanes = nullptr;
    uint32_t* tail = nullptr;
    bool resumed = kPart == kPartSolve;                 // the first trip starts behind the stages that lead to the solve
    if constexpr (kSplitPart<kPart>) {
        resumed = resumed || p.resume != 0u;
        img = p.image + (size_t)(env - p.image_first) * p.image_stride;
        lanes = reinterpret_cast<float4*>(img + p.image_stride - kImageLaneWords);
        tail = reinterpret_cast<uint32_t*>(lanes + 32);
        if (kPart == kPartStages) e.pool = img + p.im.jpool;            // nothing here reads the rows
        if (resumed) {
            const float4 mine = __ldcg(lanes + lane);
            const uint4 words = __ldcg(reinterpret_cast<const uint4*>(tail));
            e.qd = mine.x; e.qdd = mine.y; e.tau = mine.z; e.drive_dissipation = mine.w;
            e.status = lane == 0u ? words.x : 0u; nheads = words.y; e.branching = words.z != 0u; e.reach = words.w;
            image_move<true, kPart == kPartSolve ? kBefore : kAfter>(e, p, img, nheads);
            if (kPart == kPartStages) image_move<true, kAside>(e, p, img, nheads);
            __syncwarp();
        }
    }
    // A step ends where the next begins, with the kinematics of the new coordinates: one pass over them serves both.
#pragma unroll 1
    for (uint32_t step = resumed ? 1u : 0u;; ++step) {
      if (kPart != kPartSolve && !resumed) {
        stay_together<kPart>();
        float E[9];
        V3 r = mk3(0.f, 0.f, 0.f);
        if (has_artic) {
            if (lane < t.L) joint_xform(e, E, r);
            stage_kinematics(e, E, r, step == 0u);
            tick(e, 1);
            if (step != 0u) stage_store_links(e);
        }
        if (has_bodies) {
            stage_body_poses(e, step == 0u);
            if (step != 0u) stage_store_bodies(e, true);
        }
        if (step != 0u) {
            uint32_t st = __reduce_or_sync(NKB_FULL, e.status);
            // The gyro bit describes the latest step only (the reference clears it before every body integration,
            // ops/articulation.cu:1053-1056, 1810-1812); every other bit stays until the env is reset.
            if (lane == 0u && (st != 0u || has_bodies)) {
                const uint32_t before = p.s.status[env];
                const uint32_t after = (has_bodies ? before & ~kStatusGyroFailure : before) | st;
                if (after != before) p.s.status[env] = after;
            }
            __syncwarp();
            tick(e, 13);
            if (kPart == kPartStages ? p.last != 0u : step == p.steps) return;
        }
        e.status = 0u; e.branching = false; e.merged = kMergeUntried; e.by_rows = kRowsNone; e.reach = 0u;
        if (p.mode == kModeRefresh) {
            if (has_bodies) stage_store_bodies(e, false);
            if (has_artic) {
                float* gp = p.s.link_pose + (size_t)env * t.L * 7u;
#pragma unroll 1
                for (uint32_t k = lane; k < t.L * 7u; k += 32u) gp[k] = sm[p.sm.pose + k];
            }
            return;
        }
        if (has_artic) {
            stage_drives(e);
            float bias[K];
            stage_dynamics<K>(e, E, r, bias);
            // Computed torque and operational-space control (pipeline.cpp:406-426) take the accelerations twice, force-free for
            // the controller and then under its feedforward effort; the mass matrix and the bias are the same.  The controllers
            // are compiled into the kControl builds of the kernel only (they would cost every other world registers).
            const bool two_passes = kControl && (t.cfg.control_mode == 3u || t.cfg.control_mode == 4u) && p.mode != kModeDynamicsOnly;
            const int first = two_passes ? 0 : 1;
#pragma unroll 1
            for (int pass = first; pass < 2; ++pass) {
                stage_accelerations<K>(e, bias, pass == first, pass == 1 && p.mode != kModeDynamicsOnly);
                if constexpr (kControl) { if (pass == 0) stage_computed_torque<K>(e); }
            }
            tick(e, 2);
        }
        if (p.mode == kModeDynamicsOnly) {
            if (lane < t.L) p.s.qddot[(size_t)env * t.L + lane] = e.qdd;
            return;
        }
        uint32_t pair_count = 0u;
        stay_together<kPart>();
        if (has_bodies) stage_body_kick(e);
        if (has_collidables) {
            stage_aabbs(e);
            pair_count = t.broadphase_tree != 0u ? stage_pairs_lbvh(e) : stage_pairs(e);
            tick(e, 3);
            narrowphase_frames(e);
            if constexpr (kRigid) team_fork(e, kTeamNarrowphase, pair_count, [&](uint32_t first, uint32_t stride) { narrowphase_range(e, pair_count, first, stride); });
            else narrowphase_range(e, pair_count, 0u, 1u);
            tick(e, 4);
            stage_store_contacts(e, pair_count);
            tick(e, 5);
        }
        if (p.mode == kModeCollideOnly) {
            if (has_bodies) stage_store_bodies(e, false);
            const uint32_t st = __reduce_or_sync(NKB_FULL, e.status);
            if (lane == 0u) p.s.status[env] |= st;
            return;
        }
        stay_together<kPart>();
        nheads = stage_rows<NR, kPart != kPartBare>(e, pair_count);
        tick(e, 6);
        if constexpr (kRigid) team_fork(e, kTeamWarmStart, nheads, [&](uint32_t first, uint32_t stride) { warm_start_range(e, nheads, first, stride); });
        else if constexpr (kPart != kPartBare) warm_start_range(e, nheads, 0u, 1u);
        __syncwarp();
        tick(e, 7);
        if constexpr (kPart == kPartStages) {
            image_move<false, kBefore>(e, p, img, nheads); image_move<false, kAside>(e, p, img, nheads);
            __stcg(lanes + lane, make_float4(e.qd, e.qdd, e.tau, e.drive_dissipation));
            const uint32_t st = __reduce_or_sync(NKB_FULL, e.status);
            if (lane == 0u) __stcg(reinterpret_cast<uint4*>(tail), make_uint4(st, nheads, e.branching ? 1u : 0u, e.reach));
            return;
        }
      }
        if constexpr (kPart != kPartStages) stage_solve<NR, kRigid, NR == 2 && kPart != kPartBare>(e, nheads);
        if constexpr (kPart == kPartSolve) {
            image_move<false, kAfter>(e, p, img, nheads);
            __stcg(reinterpret_cast<float*>(lanes + lane), e.qd);
            const uint32_t st = __reduce_or_sync(NKB_FULL, e.status);
            if (lane == 0u) tail[0] = st;
            return;
        }
        resumed = false;
        if constexpr (!kSplitPart<kPart>) { rally_wait(rally, p.group, lane); tick(e, 29); }
        if (has_collidables) {
            stage_cache_commit(e, nheads, [&](uint32_t ncontact) {
                if constexpr (kRigid) team_fork(e, kTeamCacheOwners, ncontact, [&](uint32_t first, uint32_t stride) { cache_owners_range(e, ncontact, first, stride); });
                else cache_owners_range(e, ncontact, 0u, 1u);
            });
        }
        if (has_artic) stage_readout_drives(e, nheads);
        tick(e, 12);
        if (has_artic) { stage_integrate_links(e, use_pseudo); }
        if (has_bodies) stage_integrate_bodies(e, use_pseudo);
        __syncwarp();
    }
}

// A helper warp's life: wait for a command, do its share (rigid blocks of a colour, or a slice of
// a stage's outer loop), answer, until told to leave (or until a wait runs out).
template <int NR>
NKB_DEV void team_helper(float* sm, const SmemLayout& shared_layout, const TemplateView& t, const StateView& state, uint32_t env,
                         uint32_t member, uint32_t lane, uint32_t vstride) {
    const TeamCommand* cmd = team_command(sm, shared_layout);
    uint32_t* answer = reinterpret_cast<uint32_t*>(team_result(sm, shared_layout, member));
    uint32_t last = 0u;
#pragma unroll 1
    for (uint32_t trips = 0u; trips < (1u << 24); ++trips) {
        // every lane polls the same word, so the warp never splits over the wait
        uint32_t seq = last;
        {
            const long long begin = clock64();
#pragma unroll 1
            while ((seq = team_peek(&cmd->seq)) == last) {
                if (clock64() - begin > kTeamPatience) break;
                __nanosleep(100);
            }
        }
        seq = __shfl_sync(NKB_FULL, seq, 0);
        __syncwarp();
        if (seq == last) {                                   // the lead never called: leave, and say so
            if (lane == 0u) atomicOr(state.status + env, kStatusTeamTimeout);
            return;
        }
        __threadfence_block();
        last = seq;
        const uint32_t op = team_peek(&cmd->op);
        if (op == kTeamExit) return;
        if ((shared_layout.team_drill & 2u) != 0u) continue;          // drill: a helper that never answers
        RigidResult r = {0.f, 0.f, 0u};
        const uint32_t k_begin = cmd->k_begin, k_end = cmd->k_end, nblocks = cmd->nblocks;
        if (op == kTeamDescend && k_begin < k_end && k_end <= nblocks && nblocks <= t.B + 1u) {
            RigidRun run;
            run.sm = sm; run.lay = &shared_layout; run.t = &t; run.lane = lane; run.vstride = vstride;
            run.nheads = cmd->nheads; run.nblocks = nblocks; run.tol = cmd->tol;
#ifdef NKB_STAGE_TAPS
            const long long tap0 = clock64();
#endif
            r = descend_share<NR>(run, k_begin, k_end, member, shared_layout.team, cmd->position != 0u);
#ifdef NKB_STAGE_TAPS
            if (state.dbg_cycles != nullptr && lane == 0u && member == 1u) {
                uint32_t* cyc = state.dbg_cycles + (size_t)env * 32u;
                cyc[30] += (uint32_t)(clock64() - tap0); cyc[31] += 1u;
            }
#endif
        }
        else if (op == kTeamNarrowphase || op == kTeamWarmStart || op == kTeamCacheOwners) {
            Env e = bare_env(sm, &shared_layout, &t, &state, env, lane, vstride);
            if (op == kTeamNarrowphase) narrowphase_range(e, k_begin, member, shared_layout.team);
            else if (op == kTeamWarmStart) warm_start_range(e, k_begin, member, shared_layout.team);
            else cache_owners_range(e, k_begin, member, shared_layout.team);
            r.status = e.status;
        }
        __syncwarp();
        if (lane == 0u) {
            float* out = team_result(sm, shared_layout, member);
            out[0] = r.momentum; out[1] = r.residual; answer[2] = r.status;
            __threadfence_block();
            team_poke(answer + 3, seq);
        }
        __syncwarp();
    }
}

// Block layout: blockDim.x / 32 warps, `team` consecutive warps per env (one unless the world runs in team mode); an
// env's shared-memory slice is shared by its team.
template <int NR, bool kRigid, bool kSlim, bool kControl, int kPart>
__global__ void __maxnreg__(NR == 0 ? NKB_MAXNREG_BODIES : kSlim ? NKB_MAXNREG_SLIM : kSplitPart<kPart> ? NKB_MAXNREG_SPLIT : kRigid ? NKB_MAXNREG_RIGID : NKB_MAXNREG) step_kernel(const __grid_constant__ StepParams p) {
    extern __shared__ __align__(16) float smem[];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t team = kRigid ? p.sm.team : 1u;
    const uint32_t slot = warp / team, member = warp - slot * team;
    uint32_t env = blockIdx.x * ((blockDim.x >> 5) / team) + slot;
    if constexpr (kSplitPart<kPart>) env = p.first + env < p.end ? p.first + env : 0xffffffffu;
    if constexpr (kPart == kPartSolve) {
        if (p.tier != kTierAll && env != 0xffffffffu) {
            const uint4 words = __ldcg(reinterpret_cast<const uint4*>(p.image + (size_t)(env - p.image_first + 1u) * p.image_stride - 4u));
            if ((words.y <= p.tier_heads && words.w <= p.tier_reach) != (p.tier == kTierSmall)) return;
        }
    }
    float* sm = smem + (size_t)slot * p.sm.words;
    if constexpr (kRigid) {
        // team mode: every lead zeroes its team's sequence numbers before any helper looks (a block-wide barrier, passed by
        // every thread before any leaves)
        if (team > 1u) {
            if (member == 0u) team_open(sm, p.sm, lane);
            __syncthreads();
        }
    }
    if (p.sel_ids != nullptr) env = env < p.sel_count ? p.sel_ids[env] : 0xffffffffu;
    __shared__ Rally rally;
    if (p.group > 1u) {
        if (threadIdx.x == 0u) { rally.word = 0u; rally.alive = min(blockDim.x >> 5, p.s.env_count - min(p.s.env_count, env)); }
        __syncthreads();
    }
    if (env >= p.s.env_count) return;                       // the whole team leaves together
    if (p.sel_mask != nullptr && p.sel_mask[env] == 0u) return;
    if constexpr (kRigid) {
        if (member != 0u) { team_helper<NR>(sm, p.sm, p.t, p.s, env, member, lane, 32u * (NR > 0 ? NR : 1)); return; }
    }
#pragma unroll 1
    for (;;) {
        advance_env<NR, kRigid, kControl, kPart>(p, sm, env, lane, &rally);
        if (p.queue == nullptr) break;
        uint32_t next = 0u;
        if (lane == 0u) next = atomicAdd(p.queue, 1u);
        env = gridDim.x * (blockDim.x >> 5) + __shfl_sync(NKB_FULL, next, 0);
        if (env >= p.s.env_count) break;
    }
    rally_leave(&rally, p.group, lane);
    if (p.queue != nullptr && lane == 0u) {
        // the launch's last warp leaves the queue zeroed for the next launch
        __threadfence();
        const uint32_t warps = gridDim.x * (blockDim.x >> 5);
        if (atomicInc(p.queue + 1, warps - 1u) == warps - 1u) *reinterpret_cast<volatile uint32_t*>(p.queue) = 0u;
    }
    if constexpr (kRigid) { if ((p.sm.team_drill & 1u) == 0u) team_dismiss(sm, p.sm, lane); }
}

// Raises the kernel's dynamic shared-memory limit to `bytes` if it is not there yet.  The limit is per function and
// per device and only ever grows, so worlds of different sizes stepped from different threads cannot undo each other's
// setting between the attribute call and the launch.
template <int NR, bool kRigid, bool kSlim, bool kControl, int kPart>
static cudaError_t variant_reserve_shared(size_t bytes) {
    static std::mutex lock;
    static size_t reserved[64] = {0};
    if (bytes <= 48u * 1024u) return cudaSuccess;
    int device = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err != cudaSuccess) return err;
    if (device < 0 || device >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> hold(lock);
    if (bytes <= reserved[device]) return cudaSuccess;
    err = cudaFuncSetAttribute(step_kernel<NR, kRigid, kSlim, kControl, kPart>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (err == cudaSuccess) reserved[device] = bytes;
    return err;
}

template <int NR, bool kRigid, bool kSlim, bool kControl, int kPart>
static int variant_resident_blocks(uint32_t warps_per_block, size_t shared_bytes) {
    if (variant_reserve_shared<NR, kRigid, kSlim, kControl, kPart>(shared_bytes) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, step_kernel<NR, kRigid, kSlim, kControl, kPart>, (int)(warps_per_block * 32u), shared_bytes) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return blocks;
}

template <int NR, bool kRigid, bool kSlim, bool kControl, int kPart>
static int variant_registers() {
    cudaFuncAttributes attr{};
    if (cudaFuncGetAttributes(&attr, step_kernel<NR, kRigid, kSlim, kControl, kPart>) != cudaSuccess) { cudaGetLastError(); return 0; }
    return attr.numRegs;
}

template <int NR, bool kRigid, bool kSlim, bool kControl, int kPart>
static cudaError_t variant_launch(const StepParams& p, uint32_t warps_per_block, cudaStream_t stream) {
    const uint32_t team = kRigid ? p.sm.team : 1u;
    const uint32_t envs_per_block = warps_per_block / team;
    if (envs_per_block == 0u || envs_per_block * team != warps_per_block || envs_per_block > kWarpsPerBlockMax) return cudaErrorInvalidConfiguration;
    const size_t bytes = (size_t)envs_per_block * p.sm.words * sizeof(float);
    const cudaError_t err = variant_reserve_shared<NR, kRigid, kSlim, kControl, kPart>(bytes);
    if (err != cudaSuccess) return err;
    const uint32_t envs = kSplitPart<kPart> ? p.end - p.first : p.sel_ids != nullptr ? p.sel_count : p.s.env_count;
    if (envs == 0u) return cudaSuccess;
    const uint32_t needed = (envs + envs_per_block - 1u) / envs_per_block;
    const uint32_t blocks = p.queue != nullptr ? p.grid : needed;       // a persistent launch's grid is smaller than the batch
    step_kernel<NR, kRigid, kSlim, kControl, kPart><<<blocks, warps_per_block * 32u, bytes, stream>>>(p);
    return cudaGetLastError();
}

#define NKB_STEP_VARIANT(name, NR, RIGID, SLIM, CONTROL, PART) \
    extern const StepVariant name = {variant_resident_blocks<NR, RIGID, SLIM, CONTROL, PART>, variant_registers<NR, RIGID, SLIM, CONTROL, PART>, \
                                     variant_launch<NR, RIGID, SLIM, CONTROL, PART>};

}  // namespace nkb
