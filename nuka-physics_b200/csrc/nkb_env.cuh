// Per-warp view of one env and its shared-memory accessors, shared by every stage of the step kernel.
#pragma once
#include "nkb_math.cuh"
#include "nkb_types.h"

namespace nkb {

// Whether the articulation's multipliers are known: not in use, before the first descent of a step, after it.
constexpr uint32_t kMergeUntried = 0xffffffffu;
enum RowsState : uint32_t { kRowsNone = 0, kRowsFresh = 1, kRowsSettled = 2 };

// Per-warp view of one env: template, state, shared-memory slice and this lane's registers.
struct Env {
    const TemplateView* t;
    const StateView* s;
    const SmemLayout* lay;
    float* sm;
    uint32_t env, lane;
    // lane = link
    uint32_t parent, jtype, depth, link_dof;
    float q, qd, qdd, tau;
    V3 axis;                 // unit joint axis in the link frame
    float drive_command, drive_dissipation, drive_lower, drive_upper;
    // lane = dof: a lane owns coordinates lane and lane + 32 (the second only when the articulation has more than 32)
    uint32_t dof_link[2], dof_comp[2];   // comp == kNoLink for scalar joints
    uint32_t status;
    bool branching;          // a contact of this step acts on two branches of the articulation's tree
    uint32_t merged;         // then: depth of the tree with those branches joined, 0 where that is deeper than the solve's levels, kMergeUntried before a descent asks
    uint32_t by_rows, rows;  // the articulation descends in the space of its rows (RowsState), how many there are
    float* pool;             // where stage_rows leaves the contact rows' Jacobians
    uint32_t reach;          // contact heads that act on the articulation; the others have no rows there
    uint32_t vstride;        // words per shared-memory vector: 32 x coordinates per lane
#ifdef NKB_STAGE_TAPS
    uint32_t* cyc;           // stage cycle counters of this env, or null
    long long t0;
#endif
};

// Stage cycle counters are a build-time instrument (-DNKB_STAGE_TAPS); the shipped kernel carries none of it.
#ifdef NKB_STAGE_TAPS
// Adds the cycles since the last tick to stage counter k.
NKB_DEV void tick(Env& e, int k) {
    if (e.cyc == nullptr) return;
    const long long now = clock64();
    if (e.lane == 0u) e.cyc[k] += (uint32_t)(now - e.t0);
    e.t0 = now;
}
NKB_DEV void tick_count(Env& e, int k) { if (e.cyc != nullptr && e.lane == 0u) e.cyc[k] += 1u; }
#else
NKB_DEV void tick(Env&, int) {}
NKB_DEV void tick_count(Env&, int) {}
#endif

NKB_DEV float* sm_pose(const Env& e, uint32_t l) { return e.sm + e.lay->pose + 7u * l; }
NKB_DEV float* sm_xrot(const Env& e, uint32_t l) { return e.sm + e.lay->xrot + 9u * l; }
NKB_DEV float* sm_xtr(const Env& e, uint32_t l) { return e.sm + e.lay->xtr + 3u * l; }
NKB_DEV float* sm_vel(const Env& e, uint32_t l) { return e.sm + e.lay->vel + 6u * l; }
NKB_DEV float* sm_acc(const Env& e, uint32_t l) { return e.sm + e.lay->acc + 6u * l; }
NKB_DEV float* sm_pbias(const Env& e, uint32_t l) { return e.sm + e.lay->pbias + 6u * l; }
NKB_DEV float* sm_ic(const Env& e, uint32_t l) { return e.sm + e.lay->ic + 10u * l; }
NKB_DEV float* sm_mass(const Env& e) { return e.sm + e.lay->mass; }
NKB_DEV float* sm_factor(const Env& e) { return e.sm + e.lay->factor; }
NKB_DEV float* sm_vec(const Env& e, uint32_t k) { return e.sm + e.lay->vecs + e.vstride * k; }   // 32 or 64 words per vector
// value of coordinate j from per-lane registers x[r] (coordinate lane + 32 r)
template <int NR>
NKB_DEV float coord_bcast(const float (&x)[NR], uint32_t j) {
    if (NR == 1) return __shfl_sync(NKB_FULL, x[0], j);
    return __shfl_sync(NKB_FULL, j < 32u ? x[0] : x[NR - 1], j & 31u);
}
// vector slots
enum { kVecAcc = 0, kVecFree = 1, kVecU = 2, kVecPseudo = 3, kVecTmp = 4, kVecTmp2 = 5,
       // Newton-loop scratch shares slots whose other users run before or after the solve
       kVecS0 = kVecTmp, kVecS1 = kVecTmp2, kVecS2 = kVecAcc,
       // the Newton direction is staged after the last read of S0 in an iteration and consumed before the next write
       kVecD = kVecS0, kVecCount = 6 };
NKB_DEV float* sm_fixed(const Env& e) { return e.sm + e.lay->fixed; }

NKB_DEV uint32_t joint_dofs(uint32_t t) { return (t == kRevolute || t == kPrismatic) ? 1u : t == kFloating ? 6u : t == kSpherical ? 3u : 0u; }

template <int NR>
NKB_DEV void env_begin(Env& e, const StepParams& p, float* sm, uint32_t env, uint32_t lane) {
    e.t = &p.t; e.s = &p.s; e.lay = &p.sm; e.sm = sm; e.env = env; e.lane = lane;
    const TemplateView& t = p.t;
    const bool link = lane < t.L;
    e.parent = link ? __ldg(t.parent + lane) : kNoLink;
    e.jtype = link ? __ldg(t.jtype + lane) : (uint32_t)kFixed;
    e.depth = link ? __ldg(t.depth + lane) : 0xffffu;
    e.link_dof = link ? __ldg(t.link_dof + lane) : 0u;
    e.axis = mk3(0.f, 0.f, 0.f);
    if (link) {
        V3 a = ld3(t.axis + 3u * lane);
        const float ls = dot(a, a);
        e.axis = ls > 1.0e-12f ? a * rsqrtf(ls) : mk3(0.f, 0.f, 0.f);
    }
    const size_t at = (size_t)env * t.L + lane;
    e.q = link ? p.s.q[at] : 0.f;
    e.qd = link ? p.s.qdot[at] : 0.f;
    e.qdd = 0.f; e.tau = 0.f;
    e.drive_command = e.drive_dissipation = e.drive_lower = e.drive_upper = 0.f;
    e.vstride = 32u * (NR > 0 ? NR : 1);
    e.dof_link[1] = 0u; e.dof_comp[1] = kNoLink;
#pragma unroll
    for (uint32_t r = 0u; r < (uint32_t)NR; ++r) {
        const uint32_t c = lane + 32u * r;
        const bool dof = c < t.ndof;
        e.dof_link[r] = dof ? __ldg(t.dof_link + c) : 0u;
        e.dof_comp[r] = kNoLink;
        if (dof && __ldg(t.jtype + e.dof_link[r]) == kFloating) e.dof_comp[r] = c - __ldg(t.link_dof + e.dof_link[r]);
    }
    e.status = 0u; e.branching = false; e.merged = kMergeUntried; e.by_rows = kRowsNone; e.rows = 0u; e.reach = 0u; e.pool = sm + p.sm.jpool;
#ifdef NKB_STAGE_TAPS
    e.cyc = p.s.dbg_cycles != nullptr ? p.s.dbg_cycles + (size_t)env * 32u : nullptr;
    e.t0 = clock64();
#endif
}

}  // namespace nkb
