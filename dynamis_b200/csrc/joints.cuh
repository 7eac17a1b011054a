// joints.cuh - ball joints: the warm start, velocity and position passes, the jointed-pair filter
// and the island coupling of constraints.
//
// Joints are solved Gauss-Seidel within a component (a connected set of joints), layer by layer in
// the order of the host planner (plan_joints, crates/dynamis-world/src/schedule.rs:105-296), with a
// forward and a backward sweep per pass (joint_velocity.wgsl:24-54, joint_position.wgsl:30-61).
// The joints of one layer share no body, and components share none either, so a layer's joints run
// in parallel and components run independently. The device packs components into 32-lane warps
// (JointPlan::groups): a component owns `lanes` lanes, steps through its layers, and the warp meets
// at __syncwarp after every layer, which also orders the body rows one layer writes before the next
// layer reads them (a layer's data that is loaded ahead holds nothing that the sweep writes before). Body rows are read and written in place, as the reference's joint passes do:
// these passes run as kernels of their own, between the contact kernels of the same iteration.
#pragma once

#include <cstddef>

#include "step.cuh"

namespace dyn {

enum JointPass : int { JP_WARM = 0, JP_SOLVE = 1, JP_POSITION = 2 };

// ---- what the passes ask of a joint, in solve order ----
// A pass is a chain of dependent solves (64 for a chain of 32 joints: a forward and a backward
// sweep), so its time is the latency of one solve times the chain's length. Two lanes run a joint,
// one per body: each keeps its body's half of every row and they exchange the point velocities (the
// anchors, in the position pass) by shuffles. What does not change while a substep's passes run (the
// arms, the rows' masses, the flags) is computed once per substep and laid out in solve order, and
// the next layer's is loaded while the current one is solved. One lane per joint that derived it all
// in every solve took 2.5 us a solve in the velocity pass and 3.1 us in the position pass (131,072
// joints in chains of 32); this takes 1.7 and 2.5 us.
constexpr uint32_t kJointFirstInert = 1u << 30, kJointSecondInert = 1u << 31;

__global__ void __launch_bounds__(128) k_joint_prepare(DeviceWorld w) {
    GRID_STRIDE(at, w.jcount) {
        const uint32_t j = w.jrows[at];
        const uint4 meta = w.jmeta[j];
        const float4 aa4 = w.janchor_a[j], ab4 = w.janchor_b[j];
        DBody first = load_dbody(w.hot, meta.z), second = load_dbody(w.hot, meta.w);
        const bool inert_a = dbody_inert(first), inert_b = dbody_inert(second);
        if (inert_a) first = dbody_frozen(first);
        if (inert_b) second = dbody_frozen(second);
        const f3 anchor_a = arm(first, xyz(aa4)), anchor_b = arm(second, xyz(ab4));
        float k[3];
#pragma unroll
        for (uint32_t i = 0; i < 3; ++i) {
            const f3 axis = mk3(i == 0 ? 1.0f : 0.0f, i == 1 ? 1.0f : 0.0f, i == 2 ? 1.0f : 0.0f);
            k[i] = momentum_mass(first, second, anchor_a, anchor_b, axis);
        }
        w.jo_meta[at] = make_uint4(j, meta.z, meta.w, meta.y | (inert_a ? kJointFirstInert : 0u) | (inert_b ? kJointSecondInert : 0u));
        w.jo_mass[at] = make_float4(k[0], k[1], k[2], 0.0f);
        w.jo_arm[2u * at] = mk4(anchor_a - dbody_com(first), first.inverse_mass);
        w.jo_arm[2u * at + 1u] = mk4(anchor_b - dbody_com(second), second.inverse_mass);
        w.jo_anchor[2u * at] = aa4;
        w.jo_anchor[2u * at + 1u] = ab4;
    }
}

// One lane's side of a joint, as far as it can be loaded ahead of the solve: nothing in it changes
// between the start of a sweep and the joint's turn in it.
struct JointSide {
    uint4 meta;     // joint, first row, second row, flags
    float4 mass;    // velocity passes: the rows' masses
    float4 arm;     // this side's arm and inverse mass (0 when inert)
    float4 anchor;  // this side's anchor and break limit (force on the first side, torque on the second)
    float4 other;   // position pass: the other side's arm record (its inverse mass)
    float acc[3];
    uint32_t broken;
    float4 rot, ii0;  // velocity passes: this side's body
    float2 ii1;
    uint32_t row;
};
template <int kPass>
__device__ __forceinline__ JointSide load_joint(const DeviceWorld& w, uint32_t at, uint32_t side) {
    JointSide s;
    s.meta = __ldg(w.jo_meta + at);
    s.arm = __ldg(w.jo_arm + 2u * at + side);
    s.anchor = __ldg(w.jo_anchor + 2u * at + side);
    s.row = side ? s.meta.z : s.meta.y;
    const dyn_constraint_runtime_record& rt = w.jruntime[s.meta.x];
    s.broken = rt.broken;
    if (kPass == JP_POSITION) {
        s.other = __ldg(w.jo_arm + 2u * at + 1u - side);
    } else {
        s.mass = __ldg(w.jo_mass + at);
        for (uint32_t i = 0; i < 3u; ++i) s.acc[i] = rt.accumulated[i];
        const BodyHot& h = w.hot[s.row];
        const bool inert = (s.meta.w & (side ? kJointSecondInert : kJointFirstInert)) != 0u;
        s.rot = h.rot;
        s.ii0 = inert ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : h.ii0;
        s.ii1 = inert ? make_float2(0.0f, 0.0f) : make_float2(h.ii1.x, h.ii1.y);
    }
    return s;
}
__device__ __forceinline__ f3 from_partner(f3 v) {
    return mk3(__shfl_xor_sync(0xFFFFFFFFu, v.x, 1), __shfl_xor_sync(0xFFFFFFFFu, v.y, 1), __shfl_xor_sync(0xFFFFFFFFu, v.z, 1));
}
// This side's half of a pair impulse: the first body takes -j, the second +j.
__device__ __forceinline__ void side_impulse(const JointSide& s, uint32_t side, f3 j, f3* v, f3* av) {
    const f3 dv = j * s.arm.w, da = inv_inertia_world(s.ii0, s.ii1, s.rot, cross(xyz(s.arm), j));
    *v = side ? *v + dv : *v - dv;
    *av = side ? *av + da : *av - da;
}
__device__ __forceinline__ f3 joint_axis(uint32_t i) {
    return mk3(i == 0 ? 1.0f : 0.0f, i == 1 ? 1.0f : 0.0f, i == 2 ? 1.0f : 0.0f);
}

// joint_solve.wgsl:803-832 (warm_joint) for a ball joint (warm_constraint_rows :754-766).
__device__ __forceinline__ void joint_warm(const DeviceWorld& w, const JointSide& s, uint32_t side, bool active) {
    if (!active || s.broken != 0u) return;
    BodyHot& h = w.hot[s.row];
    f3 v = xyz(h.vel), av = xyz(h.ang);
    if (s.meta.w & DYN_CONSTRAINT_WARM_START) {
#pragma unroll
        for (uint32_t i = 0; i < 3; ++i) side_impulse(s, side, joint_axis(i) * s.acc[i], &v, &av);
    }
    h.vel = mk4(v, 0.0f);
    h.ang = mk4(av, 0.0f);
}

// joint_solve.wgsl:236-267 and 419-430 (solve_joint for a ball joint: three point rows along the
// world axes, solve_point_row :96-128), then the break test (:679-686) and the write-back. Every lane
// of the warp runs it (the shuffles); only the active ones store.
__device__ __forceinline__ void joint_solve(const DeviceWorld& w, const dyn_step_params& p, const JointSide& s, uint32_t side,
                                            bool active, bool residual) {
    active = active && s.broken == 0u && (s.meta.w & (kJointFirstInert | kJointSecondInert)) != (kJointFirstInert | kJointSecondInert);
    const bool warm = (s.meta.w & DYN_CONSTRAINT_WARM_START) != 0u;
    f3 v = s3(0.0f), av = s3(0.0f);
    if (active) {
        v = xyz(w.hot[s.row].vel);
        av = xyz(w.hot[s.row].ang);
    }
    const f3 v0 = v, av0 = av, r = xyz(s.arm);
    const float k[3] = {s.mass.x, s.mass.y, s.mass.z};
    float acc[3];
#pragma unroll
    for (uint32_t i = 0; i < 3; ++i) acc[i] = warm ? s.acc[i] : 0.0f;
    f3 linear = s3(0.0f), angular = s3(0.0f);  // FrameForces of this side (joint_solve.wgsl:1-6)
#pragma unroll
    for (uint32_t i = 0; i < 3; ++i) {
        const f3 axis = joint_axis(i);
        const f3 mine = v + cross(av, r), theirs = from_partner(mine);
        if (k[i] > 0.0f) {
            const float speed = dot(side ? mine - theirs : theirs - mine, axis);
            const float next = acc[i] - speed / k[i];
            const float applied = next - acc[i];  // row_impulse with no cap
            side_impulse(s, side, axis * applied, &v, &av);
            acc[i] = next;
            // point_reaction (joint_solve.wgsl:58-69) over the bodies the row started from
            const f3 impulse = side ? axis * acc[i] : -(axis * acc[i]);
            linear = linear + impulse;
            angular = angular + cross(r, impulse);
        }
    }
    if (residual) {
        const float lin = length(v - v0), ang = length(av - av0);
        const float lin2 = __shfl_xor_sync(0xFFFFFFFFu, lin, 1), ang2 = __shfl_xor_sync(0xFFFFFFFFu, ang, 1);
        if (active && side == 0u) {
            max_counter(&w.counters[DYN_COUNTER_SOLVE_LINEAR_RESIDUAL], (uint32_t)solver_word(wmax(lin, lin2), DYN_SOLVER_VELOCITY_SCALE));
            max_counter(&w.counters[DYN_COUNTER_SOLVE_ANGULAR_RESIDUAL], (uint32_t)solver_word(wmax(ang, ang2), DYN_SOLVER_VELOCITY_SCALE));
        }
    }
    const float force_limit = __shfl_xor_sync(0xFFFFFFFFu, s.anchor.w, 1);  // on the second side: the first's
    if (!active) return;
    dyn_constraint_runtime_record& rt = w.jruntime[s.meta.x];
    if (side && (s.meta.w & DYN_CONSTRAINT_HAS_BREAK)) {
        const float force = length(linear) / p.dt;
        const float torque = length(angular) / p.dt;
        if ((force_limit > 0.0f && force > force_limit) || (s.anchor.w > 0.0f && torque > s.anchor.w)) rt.broken = 1u;
    }
    if (side == 0u) {
#pragma unroll
        for (uint32_t i = 0; i < 3; ++i) rt.accumulated[i] = acc[i];
        if (!warm) {
            for (uint32_t i = 3; i < DYN_CONSTRAINT_ACCUMULATOR_SLOTS; ++i) rt.accumulated[i] = 0.0f;
        }
    }
    float4* reaction = reinterpret_cast<float4*>(&rt.reaction) + 2u * side;
    reaction[0] = mk4(linear, 0.0f);
    reaction[1] = mk4(angular, 0.0f);
    BodyHot& h = w.hot[s.row];
    h.vel = mk4(v, 0.0f);
    h.ang = mk4(av, 0.0f);
}
static_assert(offsetof(dyn_constraint_reaction_record, angular_first) == 16 &&
                  offsetof(dyn_constraint_reaction_record, linear_second) == 32 &&
                  offsetof(dyn_constraint_reaction_record, angular_second) == 48 &&
                  sizeof(dyn_constraint_runtime_record) % 16 == 0,
              "a side's reaction is two float4");

// joint_position.wgsl:18-36 (project) over joint_correction.wgsl:5-27, 85-90 for a ball joint:
// three point rows on the world axes (correction.wgsl:48-66, 93-104), each applied to working
// copies of the bodies (a shift, and the orientation renormalised), then the summed correction applied
// once to the stored rows. The correction carries no angular part, so the stored orientation ends as
// the first row's renormalisation of it.
__device__ __forceinline__ void joint_project(const DeviceWorld& w, const dyn_step_params& p, const JointSide& s, uint32_t side,
                                              bool active) {
    active = active && s.broken == 0u;
    float4 pos0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), rot = make_float4(0.0f, 0.0f, 0.0f, 1.0f), res = pos0;
    if (active) {
        pos0 = w.hot[s.row].pos;
        rot = w.hot[s.row].rot;
        res = w.resolution[s.row];
    }
    const f3 local = xyz(s.anchor);
    const float k = side ? s.other.w + s.arm.w : s.arm.w + s.other.w;
    f3 position = xyz(pos0), total = s3(0.0f);
    float4 turned = rot;
#pragma unroll
    for (uint32_t i = 0; i < 3; ++i) {
        const f3 axis = joint_axis(i);
        const f3 mine = quat_rotate(rot, local) + position, theirs = from_partner(mine);
        f3 lin = s3(0.0f);
        if (k > 0.0f) {
            const float magnitude = p.relaxation * (dot(side ? mine - theirs : theirs - mine, axis) - 0.0f) / k;
            lin = axis * (side ? -magnitude * s.arm.w : magnitude * s.arm.w);
        }
        position = position + lin;
        if (i < 2u) rot = normalize4(quat_mul(mk4(s3(0.0f) * 0.5f, 1.0f), rot));  // the last one is read by nothing
        if (i == 0u) turned = rot;
        total = total + lin;
    }
    const float moved = dot(total, total);
    const float moved2 = __shfl_xor_sync(0xFFFFFFFFu, moved, 1);
    if (!active || !(moved > 0.0f || moved2 > 0.0f)) return;
    BodyHot& h = w.hot[s.row];
    h.pos = mk4(xyz(pos0) + total, pos0.w);
    h.rot = turned;
    w.resolution[s.row] = make_float4(res.x + total.x, res.y + total.y, res.z + total.z, 0.0f);
}

// One warp per group of components (joint_velocity.wgsl:24-54 with a warp for a workgroup). A
// component owns g.z lanes, two per joint it solves side by side.
template <int kPass>
__global__ void __launch_bounds__(32) k_joints(DeviceWorld w, dyn_step_params p) {
    const uint32_t group = blockIdx.x;
    if (group >= w.jgroup_count) return;
    const uint32_t lane = threadIdx.x & 31u;
    const uint4 g = w.jgroups[group];
    const uint32_t lanes = g.z, slot = lane / lanes, li = lane % lanes;
    const uint32_t side = li & 1u, joint = li >> 1, stride = lanes >> 1;
    uint32_t layer_offset = 0, layer_count = 0;
    if (slot < g.y) {
        const uint2 c = w.jcomps[g.x + slot];
        layer_offset = c.x;
        layer_count = c.y;
    }
    const bool residual = kPass == JP_SOLVE && w.ctl[CTL_ROUNDS] == p.solve_iterations;
    auto layer = [&](uint32_t sweep, uint32_t step) {
        if (step >= layer_count) return make_uint2(0u, 0u);
        return __ldg(w.jlayers + (sweep == 0u ? layer_offset + step : layer_offset + layer_count - 1u - step));
    };
    JointSide idle{};
    idle.broken = 1u;
    for (uint32_t sweep = 0; sweep < 2u; ++sweep) {
        uint2 range = layer(sweep, 0u), next = layer(sweep, 1u);
        JointSide s = joint < range.y ? load_joint<kPass>(w, range.x + joint, side) : idle;
        for (uint32_t step = 0; step < g.w; ++step) {
            // the next layer's joint and the range of the one after it, on their way during this solve
            const JointSide ahead = joint < next.y ? load_joint<kPass>(w, next.x + joint, side) : idle;
            const uint2 later = layer(sweep, step + 2u);
            const uint32_t trips = __reduce_max_sync(0xFFFFFFFFu, (range.y + stride - 1u) / stride);
            for (uint32_t trip = 0; trip < trips; ++trip) {
                const uint32_t index = joint + trip * stride;
                const bool active = index < range.y;
                if (trip > 0u) s = active ? load_joint<kPass>(w, range.x + index, side) : idle;
                if (kPass == JP_WARM) {
                    joint_warm(w, s, side, active);
                } else if (kPass == JP_SOLVE) {
                    joint_solve(w, p, s, side, active, residual);
                } else {
                    joint_project(w, p, s, side, active);
                }
            }
            __syncwarp();
            s = ahead;
            range = next;
            next = later;
        }
    }
}

// COUNTER_JOINTS: the jointed pairs the narrowphase filters this step (joint_filter.wgsl:9-24).
__global__ void k_joint_count(DeviceWorld w) {
    GRID_STRIDE(i, w.jfilter_count) {
        if (w.jruntime[w.jfilter_joint[i]].broken == 0u) add_counter(&w.counters[DYN_COUNTER_JOINTS], 1u);
    }
}

// island_link_constraints.wgsl: every unbroken joint couples its two rows.
__global__ void k_island_link_joints(DeviceWorld w) {
    GRID_STRIDE(j, w.jcount) {
        if (w.jruntime[j].broken != 0u) continue;
        const uint4 meta = w.jmeta[j];
        if (!island_couple(w, meta.z, meta.w)) add_counter(&w.counters[DYN_COUNTER_ISLAND_FAULTS], 1u);
    }
}

}  // namespace dyn
