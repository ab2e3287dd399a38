// arc_step_warps.cuh - the warp-per-leg step (FP32): one group of 32 worlds.
//
// A CTA of four warps steps 32 worlds: lane j of warp k is leg k of world j.
// The reference's Gauss-Seidel order (csrc/arc_phys.c:729-735) couples the
// legs only through the torso: joint 3k (torso -> coxa of leg k) must see
// the torso as joint 3(k-1) left it. So warp k solves its torso joint after
// warp k-1 solved its own (a named barrier between the two warps, one
// arrive and one sync), and everything else of leg k - its two other
// joints, its five spheres, its three bodies' velocities - runs without
// waiting. Warp 0 also owns the torso's own work (its integration, its
// sphere, its contact velocities), so the torso sphere's contacts lead warp
// 0's list as sphere 0 leads the reference's, and the four warps' lists in
// warp order are the reference's contact list.
//
// Code size decides this kernel's speed. With 16 warps of 4 CTAs per SM in
// different phases of the step, a kernel whose code does not fit the SM's
// instruction cache spends most cycles waiting for instructions. Every
// phase is therefore one generic routine, run by a small interpreter over a
// per-warp list of operations (integrate bodies a..b, solve joints a..b,
// collide spheres a..b, ...): one copy of each routine, whatever the body.
// The bodies live in shared memory ([field][world], conflict-free); a
// routine loads the few it works on, recomputes their rotation and world
// inverse inertia from q (the same function of q as the reference's
// body_sync, so the same values), and stores them back.
//
// Rotations the reference leaves stale: update_velocities (csrc/arc_phys.c:
// 674-687) normalises q without re-syncing, so the velocity pass and the
// next substep's gyroscopic term use the rotation of the un-normalised q of
// the position pass. Each body therefore keeps two quaternions: field Q, the
// position-pass q the rotation comes from, and field QP, the substep-start
// q (and, after the velocity update, the normalised q the next substep
// starts from).
//
// This header holds the step of one group, `step_group`, which the control
// step kernel of arc_task.cu runs in FP32, alone (the physics step) or
// followed by the task layer on the group's worlds (the fused control step),
// and arc_step_warps64.cu's kernel runs in FP64 (ARC_WARPS_FP64). Everything
// here has internal linkage: each including translation unit has its own
// copy, its operation lists in its own constant bank.
#pragma once

#include "arc_kernels.cuh"

namespace arc {
namespace wl {
namespace {

constexpr int kWarps = 4;   // one per leg
constexpr int kWorlds = 32; // one per lane
constexpr int kThreads = kWarps * kWorlds;
constexpr int kOnChip = kWarpsOnChipContacts;

// the precision of the step: FP32 (arc_task.cu's control-step kernel) or,
// where the including file defines ARC_WARPS_FP64, FP64 (arc_step_warps64.cu)
#ifdef ARC_WARPS_FP64
using F = double;
#else
using F = float;
#endif
using V = V3<F>;
using Q = Q4<F>;
using P = Pose<F>;

// body fields: x, q (position pass), v, w, x_prev, q_prev / normalised q
constexpr int kX = 0, kQ = 3, kV = 7, kW = 10, kXP = 13, kQP = 16, kBodyF = 20;
constexpr int kTorso = 3;  // body slot of the torso; 0..2: the lane's coxa, femur, tibia

// The model constants stay in the kernel's parameter space: all lanes of a
// warp read the same body, joint or sphere, a broadcast from the constant
// cache.
template <int OnChip, int Warps> struct SmemOf {
    static constexpr int kOnChipRecords = OnChip;
    F leg[kWarps][3 * kBodyF][kWorlds];   // the lane's three bodies
    F anch[kWarps][5 * 6][kWorlds];       // anchor, anchor normal of the lane's five spheres
    F con[Warps][OnChip * 7][kWorlds];    // on-chip contact records: local3 n3 body
    F torso[kBodyF + 6][kWorlds];     // each world's torso, then its sphere's anchor
    int nc[2][kWarps][kWorlds];       // contact counts (capped lists), by substep parity
    int bad[Warps][kWorlds];
};
using Smem = SmemOf<kOnChip, kWarps>;
// of a split group (SplitSync): a foot's contacts, one or two, stay on chip
using SplitSmem = SmemOf<2, 2 * kWarps>;

// A field array in shared memory: element f at p[f * kWorlds]. Every
// per-world array has the same row length, so fields are constant offsets
// from the pointer whichever body it points at.
struct Ref {
    F* p;
    __device__ __forceinline__ F& operator[](int f) const { return p[f * kWorlds]; }
};
__device__ __forceinline__ V getv(Ref r, int f) { return V{r[f], r[f + 1], r[f + 2]}; }
__device__ __forceinline__ void setv(Ref r, int f, V v)
{
    r[f] = v.x;
    r[f + 1] = v.y;
    r[f + 2] = v.z;
}
__device__ __forceinline__ Q getq(Ref r, int f) { return Q{r[f], r[f + 1], r[f + 2], r[f + 3]}; }
__device__ __forceinline__ void setq(Ref r, int f, Q q)
{
    r[f] = q.w;
    r[f + 1] = q.x;
    r[f + 2] = q.y;
    r[f + 3] = q.z;
}
__device__ __forceinline__ void load_pose(Ref r, const BodyK<F>& k, P& b)
{
    b.x = getv(r, kX);
    b.q = getq(r, kQ);
    body_sync(b, k);
}
__device__ __forceinline__ void store_pose(Ref r, const P& b)
{
    setv(r, kX, b.x);
    setq(r, kQ, b.q);
}

// named barriers between two warps (ids 1..8; 0 is __syncthreads). The
// producer's arrive orders its earlier shared-memory writes before the
// consumer's sync returns.
__device__ __forceinline__ void bar_arrive(int id) { asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void bar_sync(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

// csrc/arc_phys.c:413-457 for a joint with a parent: the drive (solve_rot,
// :353-371), the limit and the axis alignment (solve_rot_block, :328-346)
// and the attachment (solve_point, :308-320), in that order, with one site
// that applies the impulse (+p on the parent, -p on the child, :196-211).
__device__ __forceinline__ void joint_positions(P& bp, const BodyK<F>& kp, P& bc, const BodyK<F>& kc,
                                                const JointK<F>& j, F target, F& torque_acc, F hh)
{
#pragma unroll 1
    for (int stage = 0; stage < 4; ++stage) {
        const V a1 = mul(bp.rot, j.a1);
        S3<F> K{F(0), F(0), F(0), F(0), F(0), F(0)};
        V rhs{F(0), F(0), F(0)}, p{F(0), F(0), F(0)}, r1{F(0), F(0), F(0)}, r2{F(0), F(0), F(0)};
        bool positional = false;
        if (stage < 2) {
            if (stage == 0 ? !(j.kp > F(0)) : !(j.lo <= j.hi))
                continue;
            const V b1 = mul(bp.rot, j.b1), b2 = mul(bc.rot, j.b2);
            const F s = dot(cross(b1, b2), a1), c = dot(b1, b2);
            // the limit needs the angle only outside [lo, hi]
            if (stage == 1 &&
                !(j.hi - j.lo > F(kPi) || s * j.lim[0] - c * j.lim[1] < F(0) || j.lim[3] * c - j.lim[2] * s < F(0)))
                continue;
            const F phi = r_atan2(s, c);
            if (stage == 0) {
                const V rot = scale(a1, phi - target);
                const F theta = len(rot);
                if (theta < F(1e-12))
                    continue;
                const V n = scale(rot, F(1) / theta);
                const F denom = dot(n, mul(bp.iiw, n)) + dot(n, mul(bc.iiw, n)) + j.alpha_hh;
                if (denom <= F(0))
                    continue;
                F dl = theta / denom;
                if (dl > j.max_dl)
                    dl = j.max_dl;
                p = scale(n, dl);
                torque_acc -= dot(p, a1) / hh;
            } else {
                if (phi < j.lo)
                    rhs = scale(a1, phi - j.lo);
                else if (phi > j.hi)
                    rhs = scale(a1, phi - j.hi);
                else
                    continue;
            }
        } else if (stage == 2) {
            rhs = cross(a1, mul(bc.rot, j.a2));
        } else {
            r1 = mul(bp.rot, j.r1);
            r2 = mul(bc.rot, j.r2);
            rhs = (bc.x + r2) - (bp.x + r1);
            positional = true;
        }
        if (stage > 0) {
            if (len2(rhs) < F(1e-24))
                continue;
            if (positional) {
                add_point_mass(K, bp.iiw, kp.inv_mass, r1);
                add_point_mass(K, bc.iiw, kc.inv_mass, r2);
            } else {
                K.xx = bp.iiw.xx + bc.iiw.xx; K.xy = bp.iiw.xy + bc.iiw.xy; K.xz = bp.iiw.xz + bc.iiw.xz;
                K.yy = bp.iiw.yy + bc.iiw.yy; K.yz = bp.iiw.yz + bc.iiw.yz; K.zz = bp.iiw.zz + bc.iiw.zz;
            }
            if (!solve3_sym(K, rhs, p))
                continue;
        }
        const V pn = -p;
        if (positional) {
            bp.x = madd(bp.x, p, kp.inv_mass);
            bc.x = madd(bc.x, pn, kc.inv_mass);
        }
        const V tp = mul(bp.iiw, positional ? cross(r1, p) : p);
        const V tc = mul(bc.iiw, positional ? cross(r2, pn) : pn);
        bp.q = q_turn(bp.q, tp);
        bc.q = q_turn(bc.q, tc);
        if (positional)  // the last stage: the caller keeps x and q only
            break;
        body_sync(bp, kp);
        body_sync(bc, kc);
    }
}

// One sphere against the column grid (csrc/arc_phys.c:542-610) with its
// contacts (solve_contact, :488-500) and the closing friction correction
// (solve_friction, :512-539). The scan and the friction share one site of
// the positional correction against the static world (solve_pos with no
// second body and alpha = 0, :226-242). Returns 1 when the sphere touched.
template <class Rec>
__device__ __forceinline__ int collide(P& b, const BodyK<F>& k, Ref body, const SphereK<F>& sk,
                                       SphereState<F>& ss, const TerrainView<F>& t, F inv_cell, const StepK<F>& st,
                                       Rec&& record)
{
    const F rad = sk.radius;
    V c = b.x + mul(b.rot, sk.pos);
    // a blown-up state must not reach the int conversions
    if (!(r_fabs(c.x) < F(1e6) && r_fabs(c.y) < F(1e6))) {
        ss.anchored = 0;
        return 0;
    }
    // the columns under the sphere's box (csrc/arc_phys.c:557-560), scaled by
    // 1/cell instead of divided by cell: the two differ only when a box edge
    // lies within an ulp of a column edge, where that column's face is the
    // sphere's radius away and cannot make a contact either way
    const int ix0 = (int)r_floor(((c.x - rad) - t.ox) * inv_cell);
    const int ix1 = (int)r_floor(((c.x + rad) - t.ox) * inv_cell);
    const int iy0 = (int)r_floor(((c.y - rad) - t.oy) * inv_cell);
    const int iy1 = (int)r_floor(((c.y + rad) - t.oy) * inv_cell);
    // the heights of the box's first 2 x 2 columns, loaded together: a
    // sphere narrower than a column spans at most that many, and the
    // buried-edge test's neighbours of one of them are the others
    F h00 = F(0), h10 = F(0), h01 = F(0), h11 = F(0);
    h00 = terrain_cell(t, ix0, iy0);
    if (ix1 > ix0)
        h10 = terrain_cell(t, ix0 + 1, iy0);
    if (iy1 > iy0) {
        h01 = terrain_cell(t, ix0, iy0 + 1);
        if (ix1 > ix0)
            h11 = terrain_cell(t, ix0 + 1, iy0 + 1);
    }
    auto height = [&](int cx, int cy) {
        const int dx = cx - ix0, dy = cy - iy0;
        if (dx >= 0 && dy >= 0 && dx < 2 && dy < 2 && cx <= ix1 && cy <= iy1)
            return dy ? (dx ? h11 : h01) : (dx ? h10 : h00);
        return terrain_cell(t, cx, cy);
    };
    F ln = F(0), depth_max = F(0);
    V n_max{F(0), F(0), F(1)};
    int touched = 0, ix = ix0, iy = iy0;
    // a box of at most 2 x 2 columns is scanned through the bits of `left`
    // (column dx + 2 dy), a wider one column by column. The bits give the
    // columns higher than the sphere's bottom at once: of the 9 columns that
    // a lane's spheres span in a substep 0.6 are, and testing one per
    // iteration cost a warp 22 iterations where 6 find them all (4,096
    // worlds in CTAs of four warps: 504 us against 527)
    const bool wide = ix1 - ix0 > 1 || iy1 - iy0 > 1;
    int left = 1 | (ix1 > ix0 ? 2 : 0) | (iy1 > iy0 ? 4 : 0) | (ix1 > ix0 && iy1 > iy0 ? 8 : 0);
#pragma unroll 1
    for (;;) {
        V r, d, n{F(0), F(0), F(1)};
        F depth = F(0);
        bool contact = false;
#pragma unroll 1
        while (!contact) {
            int cx, cy;
            F top;
            if (wide) {
                if (iy > iy1)
                    break;
                cx = ix;
                cy = iy;
                if (++ix > ix1) {
                    ix = ix0;
                    ++iy;
                }
                top = height(cx, cy);
                if (c.z - rad >= top)
                    continue;
            } else {
                const F low = c.z - rad;
                const int below = left & ((low >= h00 ? 0 : 1) | (low >= h10 ? 0 : 2) | (low >= h01 ? 0 : 4) | (low >= h11 ? 0 : 8));
                if (!below)
                    break;
                const int bit = below & -below;
                left &= ~(2 * bit - 1);
                const int dx = (bit & 10) ? 1 : 0, dy = (bit & 12) ? 1 : 0;
                cx = ix0 + dx;
                cy = iy0 + dy;
                top = dy ? (dx ? h11 : h01) : (dx ? h10 : h00);
            }
            const F x0 = t.ox + F(cx) * t.cell, x1 = x0 + t.cell;
            const F y0 = t.oy + F(cy) * t.cell, y1 = y0 + t.cell;
            // edges and corners buried by an equal or higher neighbour
            const int sx = c.x > x1 ? 1 : (c.x < x0 ? -1 : 0);
            const int sy = c.y > y1 ? 1 : (c.y < y0 ? -1 : 0);
            bool buried = false;
#pragma unroll 1
            for (int m = 1; m < 4 && !buried; ++m) {
                if (((m & 1) && !sx) || ((m & 2) && !sy))
                    continue;
                buried = height(cx + ((m & 1) ? sx : 0), cy + ((m & 2) ? sy : 0)) >= top;
            }
            if (buried)
                continue;
            const V q{r_clamp(c.x, x0, x1), r_clamp(c.y, y0, y1), r_min(c.z, top)};
            const V diff = c - q;
            const F dist = len(diff);
            if (dist > F(1e-9)) {
                if (dist >= rad)
                    continue;
                n = scale(diff, F(1) / dist);
                depth = rad - dist;
            } else {
                depth = top - c.z + rad;  // centre inside the column: out through the top
            }
            r = madd(c, n, -rad) - b.x;
            d = scale(n, depth);
            contact = true;
        }
        if (!contact) {
            if (!touched)
                break;
            // friction, once, after the scan; c is the current centre
            const V p = madd(c, n_max, -rad);
            if (!ss.anchored || dot(n_max, ss.anchor_n) < F(0.9)) {
                const V c0 = getv(body, kXP) + qrotate(getq(body, kQP), sk.pos);
                ss.anchor = madd(c0, n_max, -rad);
                ss.anchor_n = n_max;
                ss.anchored = 1;
            }
            V e = p - ss.anchor;
            e = madd(e, n_max, -dot(e, n_max));
            const F l = len(e);
            if (l < F(1e-12))
                break;
            r = p - b.x;
            const F lt = l / w_pos(b, k, r, scale(e, F(1) / l));
            F frac = F(1);
            if (lt > st.mu_s * ln) {
                frac = r_min(st.mu_d * ln / lt, F(1));
                ss.anchor = madd(ss.anchor, e, F(1) - frac);
            }
            d = scale(e, -frac);
        }
        F dl = F(0);
        const F cl = len(d);
        if (cl >= F(1e-12)) {
            const V nn = scale(d, F(1) / cl);
            const F denom = w_pos(b, k, r, nn);
            if (denom > F(0)) {
                dl = cl / denom;
                pos_impulse(b, k, r, scale(nn, dl));
            }
        }
        if (!contact)
            break;  // the friction correction closes the sphere
        ln += dl;
        record(tmul(b.rot, r), n);
        c = b.x + mul(b.rot, sk.pos);
        if (depth > depth_max) {
            depth_max = depth;
            n_max = n;
        }
        touched = 1;
    }
    if (!touched)
        ss.anchored = 0;
    return touched;
}

// per-warp operation lists: kind | a << 4 | b << 8 | wait << 12 | arrive << 16
// | align << 20. An op with a wait first syncs on that named barrier; one with
// an arrive arrives on it when done; one with align starts with its sibling
// warps (AlignedSync).
enum : uint32_t { OP_END = 0, OP_INT, OP_JNT, OP_COL, OP_UPD, OP_DMP, OP_CVL, OP_CNT };
// INT/UPD a..b: body ordinals (0 torso, 1..3 coxa, femur, tibia)
// JNT/DMP a..b: the leg's joints (0 torso->coxa, 1 coxa->femur, 2 femur->tibia)
// COL a..b: sphere ordinals on one body (0 torso sphere, 1 femur, 2..5 tibia)
// CVL a: contact velocities of the leg's bodies (0) or of the torso (1)
// CNT: publish the contact count, then __syncthreads (capped lists only)
#define ARC_OP(kind, a, b, w, r) ((kind) | (a) << 4 | (b) << 8 | (w) << 12 | (r) << 16)
// Uncapped lists. Warp 0 owns the torso's own work, and each substep's
// chain of torso hand-offs starts and ends in it: it integrates the torso
// and solves joint 0 at once (no hand-off), collides the torso's sphere
// after joint 9 (barrier 4), and applies the torso's contact velocities
// after joint 9's drive damping (barrier 8), before the next substep. Warp
// k > 0 solves joint 3k after warp k-1's (barrier k) and damping joint 3k
// after warp k-1's (barrier 4+k). Each warp solves what the next hand-off
// needs first (its coxa's velocity right after joint 3k+1, the only other
// joint that moves the coxa) and the rest of its leg while the chain runs
// elsewhere; work on different bodies commutes, so this is the reference's
// order. Warp 0 runs ahead of the others in issue priority: the torso's
// work there makes the step 5% faster than the same lists with the torso
// on warp 3.
//
// Two such lists, the same work in another order. While the chain is with
// the later legs, a leg that is done with its torso joint has time to spare:
// joints 3, 6 and 9 take 3.7k cycles each, a leg's third joint 3.9k, its
// femur sphere 2.1k and its tibia's four spheres 13k (32 worlds, one CTA on
// the SM, of 47k cycles a substep). kListLatency fills that wait: legs 0 and
// 1 solve their third joint and collide the femur before their damping
// joint, leg 2 its third joint, leg 3, whose damping joint comes at once,
// nothing. It pays while an SM holds one or two CTAs of four warps (the step
// of robots thrown about by random actions, 4,096 worlds: 405 us against 450;
// 9,400: 508 against 533; FP64 with one, 4,096: 625 against 670, and not with
// two, 8,000: 776 against 730); with more the other groups fill the waits and
// the damping chain's earlier start wins (a control step of 65,536 standing
// robots: 3.19 ms against 2.99 in aligned CTAs, 3.75 against 3.43 in CTAs of
// one group), so kListThroughput leaves all of it for later. Most launches
// that small are split and have lists of their own (below): kListLatency is
// for those that cannot be (recorded contacts, tiles), for the small fused
// ones and for the last groups of an aligned launch.
#define ARC_LEG_HEAD(k)                                                                                        \
    ARC_OP(OP_INT, 1, 4, 0, 0), ARC_OP(OP_JNT, 0, 1, k, (k) + 1), ARC_OP(OP_JNT, 1, 2, 0, 0),                   \
        ARC_OP(OP_UPD, 1, 2, 0, 0)
#define ARC_TORSO_HEAD                                                                                         \
    ARC_OP(OP_INT, 0, 4, 0, 0), ARC_OP(OP_JNT, 0, 1, 0, 1), ARC_OP(OP_JNT, 1, 2, 0, 0), ARC_OP(OP_UPD, 1, 2, 0, 0)
#define ARC_TORSO_DAMP ARC_OP(OP_COL, 0, 1, 4, 0), ARC_OP(OP_UPD, 0, 1, 0, 0), ARC_OP(OP_DMP, 0, 1, 0, 5)
#define ARC_LEG_DAMP(k) ARC_OP(OP_DMP, 0, 1, 4 + (k), 5 + (k))
#define ARC_JOINT3 (ARC_OP(OP_JNT, 2, 3, 0, 0) | 1 << 20)
#define ARC_FEMUR ARC_OP(OP_COL, 1, 2, 0, 0)
#define ARC_LEG_TAIL                                                                                           \
    ARC_OP(OP_COL, 2, 6, 0, 0), ARC_OP(OP_UPD, 2, 4, 0, 0), ARC_OP(OP_DMP, 1, 3, 0, 0), ARC_OP(OP_CVL, 0, 0, 0, 0)
#define ARC_TORSO_TAIL ARC_OP(OP_CVL, 1, 0, 8, 0)
// Capped lists: warp 0 owns the torso, whose sphere's contacts lead the
// list as sphere 0 leads the reference's, and every lane's count is
// published before any contact velocity.
#define ARC_CAPPED_OPS(k)                                                                                           \
    {ARC_OP(OP_INT, 1, 4, 0, 0), ARC_OP(OP_JNT, 0, 1, k, k + 1), ARC_OP(OP_JNT, 1, 3, 0, 0),                        \
     ARC_OP(OP_COL, 1, 2, 0, 0), ARC_OP(OP_COL, 2, 6, 0, 0), ARC_OP(OP_UPD, 1, 4, 0, 0), ARC_OP(OP_CNT, 0, 0, 0, 0), \
     ARC_OP(OP_DMP, 0, 1, 4 + k, 5 + k), ARC_OP(OP_DMP, 1, 3, 0, 0), ARC_OP(OP_CVL, 0, 0, 0, 0), OP_END}

constexpr int kMaxOps = 20;
enum : int { kListThroughput = 0, kListLatency = 1, kListCapped = 2 };
__constant__ uint32_t kOps[3][kWarps][kMaxOps] = {
    {{ARC_TORSO_HEAD, ARC_TORSO_DAMP, ARC_JOINT3, ARC_FEMUR, ARC_LEG_TAIL, ARC_TORSO_TAIL, OP_END},
     {ARC_LEG_HEAD(1), ARC_LEG_DAMP(1), ARC_JOINT3, ARC_FEMUR, ARC_LEG_TAIL, OP_END},
     {ARC_LEG_HEAD(2), ARC_LEG_DAMP(2), ARC_JOINT3, ARC_FEMUR, ARC_LEG_TAIL, OP_END},
     {ARC_LEG_HEAD(3), ARC_LEG_DAMP(3), ARC_JOINT3, ARC_FEMUR, ARC_LEG_TAIL, OP_END}},
    {{ARC_TORSO_HEAD, ARC_JOINT3, ARC_FEMUR, ARC_TORSO_DAMP, ARC_LEG_TAIL, ARC_TORSO_TAIL, OP_END},
     {ARC_LEG_HEAD(1), ARC_JOINT3, ARC_FEMUR, ARC_LEG_DAMP(1), ARC_LEG_TAIL, OP_END},
     {ARC_LEG_HEAD(2), ARC_JOINT3, ARC_LEG_DAMP(2), ARC_FEMUR, ARC_LEG_TAIL, OP_END},
     {ARC_LEG_HEAD(3), ARC_LEG_DAMP(3), ARC_JOINT3, ARC_FEMUR, ARC_LEG_TAIL, OP_END}},
    {{ARC_OP(OP_INT, 0, 2, 0, 0), ARC_OP(OP_JNT, 0, 1, 0, 1), ARC_OP(OP_INT, 2, 4, 0, 0), ARC_OP(OP_JNT, 1, 3, 0, 0),
      ARC_OP(OP_COL, 0, 1, 4, 0), ARC_OP(OP_UPD, 0, 1, 0, 0), ARC_OP(OP_COL, 1, 2, 0, 0), ARC_OP(OP_COL, 2, 6, 0, 0),
      ARC_OP(OP_UPD, 1, 4, 0, 0), ARC_OP(OP_CNT, 0, 0, 0, 0), ARC_OP(OP_DMP, 0, 1, 0, 5), ARC_OP(OP_DMP, 1, 3, 0, 0),
      ARC_OP(OP_CVL, 0, 0, 0, 0), ARC_OP(OP_CVL, 1, 0, 8, 0), OP_END},
     ARC_CAPPED_OPS(1), ARC_CAPPED_OPS(2), ARC_CAPPED_OPS(3)}};
// Split lists (SplitSync): two warps a leg. Warps 0..3 have the torso, the
// coxas and the femurs' spheres, warps 4..7 joint 3k+2 and the tibias.
// Barriers 1..4: the torso's hand-offs around the ring of the first four, for
// joints and damping joints in turn (AlignedSync); 5+k: leg k's upper to its
// lower warp (after joint 3k+1, after damping joint 3k+1); 9+k: back (the femur
// integrated; joint 3k+2 solved). A leg's two barriers take turns: neither warp
// signals again before it was signalled to. Leg 1's femur collides before its
// damping joint, which comes late, leg 2's and 3's after theirs.
#define ARC_UPPER_HEAD(k)                                                                                      \
    ARC_OP(OP_INT, 1, 2, 0, 0), ARC_OP(OP_JNT, 0, 1, k, (k) + 1), ARC_OP(OP_JNT, 1, 2, 9 + (k), 5 + (k)),       \
        ARC_OP(OP_UPD, 1, 2, 0, 0)
#define ARC_UPPER_DAMP(k) ARC_OP(OP_DMP, 0, 1, k, (k) + 1)
#define ARC_UPPER_FEMUR(k) ARC_OP(OP_COL, 1, 2, 9 + (k), 0), ARC_OP(OP_UPD, 2, 3, 0, 0)
#define ARC_UPPER_TAIL(k) ARC_OP(OP_DMP, 1, 2, 0, 5 + (k)), OP_END
#define ARC_LOWER(k)                                                                                           \
    {ARC_OP(OP_INT, 2, 4, 0, 9 + (k)), ARC_OP(OP_JNT, 2, 3, 5 + (k), 9 + (k)), ARC_OP(OP_COL, 2, 6, 0, 0),      \
     ARC_OP(OP_UPD, 3, 4, 0, 0), ARC_OP(OP_DMP, 2, 3, 5 + (k), 0), ARC_OP(OP_CVL, 0, 0, 0, 0), OP_END}
__constant__ uint32_t kSplitOps[2 * kWarps][kMaxOps] = {
    {ARC_OP(OP_INT, 0, 2, 0, 0), ARC_OP(OP_JNT, 0, 1, 0, 1), ARC_OP(OP_JNT, 1, 2, 9, 5), ARC_OP(OP_UPD, 1, 2, 0, 0),
     ARC_UPPER_FEMUR(0), ARC_OP(OP_COL, 0, 1, 4, 0), ARC_OP(OP_UPD, 0, 1, 0, 0), ARC_OP(OP_DMP, 0, 1, 0, 1),
     ARC_OP(OP_DMP, 1, 2, 0, 5), ARC_OP(OP_CVL, 1, 0, 4, 0), OP_END},
    {ARC_UPPER_HEAD(1), ARC_UPPER_FEMUR(1), ARC_UPPER_DAMP(1), ARC_UPPER_TAIL(1)},
    {ARC_UPPER_HEAD(2), ARC_UPPER_DAMP(2), ARC_UPPER_FEMUR(2), ARC_UPPER_TAIL(2)},
    {ARC_UPPER_HEAD(3), ARC_UPPER_DAMP(3), ARC_UPPER_FEMUR(3), ARC_UPPER_TAIL(3)},
    ARC_LOWER(0), ARC_LOWER(1), ARC_LOWER(2), ARC_LOWER(3)};
#undef ARC_UPPER_HEAD
#undef ARC_UPPER_DAMP
#undef ARC_UPPER_FEMUR
#undef ARC_UPPER_TAIL
#undef ARC_LOWER
#undef ARC_LEG_HEAD
#undef ARC_TORSO_HEAD
#undef ARC_TORSO_DAMP
#undef ARC_LEG_DAMP
#undef ARC_JOINT3
#undef ARC_FEMUR
#undef ARC_LEG_TAIL
#undef ARC_TORSO_TAIL
#undef ARC_CAPPED_OPS
#undef ARC_OP

// ---------------------------------------------------------------------------


// How the warps of a group wait for one another, by the kernel that runs it.
// CtaSync: the CTA is the group.
struct CtaSync {
    static constexpr bool kSplit = false;
    static constexpr int half = 0;
    __device__ __forceinline__ void group() const { __syncthreads(); }
    __device__ __forceinline__ void wait(int id) const { bar_sync(id); }
    __device__ __forceinline__ void arrive(int id) const { bar_arrive(id); }
    __device__ __forceinline__ void align(int, int) const {}
};

// AlignedSync: the CTA holds several groups that start their third joints
// together. The step's loop is larger than the SM's instruction cache, and in
// four CTAs of one group each the 16 warps stream through it at 16 places.
// Warps of the same leg run the same code in the same order; where they run
// it at the same time they fetch it once (16,384 worlds: 97.6 % of the fetches
// hit, not 94.4; waiting for instructions 0.35 per issue, not 0.52). A control
// step of standing robots, in CTAs of one group / four to a CTA without the
// aligning / aligned: 65,536 worlds 3,430 / 3,550 / 2,990 us, 16,384 of many
// terrain sizes 984 / 1,030 / 853, FP64 16,384 2,100 / 2,020 / 1,790. Robots
// thrown about by random actions differ too much to stay together: the step of
// 65,536 takes 2,455 / 2,518 / 2,469 us. Once a substep is enough, and the third
// joint is the best place for it (65,536 worlds 3.16 ms; at leg 0's substep
// start 3.24, before the tibia's spheres 3.20, at both 3.30; not aligned 3.64).
// Warps that share a scheduler then have it to themselves in turns, so each
// group's legs start at another warp (step_aligned).
//
// Each group has four of the sixteen named barriers, one per neighbouring
// pair of warps around the ring (0-1, 1-2, 2-3, 3-0). A pair's joint and
// damping hand-offs take turns on it: the second cannot be signalled before
// the first was received, as each follows from the last around the ring. The
// whole group's barrier is the first pair's, used only where every warp has
// passed the substeps' last hand-off.
//
// The aligned start is a schedule, not an exchange: no result depends on it,
// and a wait for it ends by itself after a while.
struct AlignedSync {
    static constexpr bool kSplit = false;
    static constexpr int half = 0;
    int base;        // the group's first barrier
    unsigned* word;  // per leg: groups running | arrived << 8 | starts so far << 16
    __device__ __forceinline__ void group() const
    {
        asm volatile("bar.sync %0, %1;" ::"r"(base), "n"(kThreads) : "memory");
    }
    __device__ __forceinline__ void wait(int id) const { bar_sync(((id - 1) & 3) + base); }
    __device__ __forceinline__ void arrive(int id) const { bar_arrive(((id - 1) & 3) + base); }
    // one lane: arrives (+1) or leaves (-1); the last one starts the others
    __device__ __forceinline__ unsigned change(unsigned* w, bool leaving) const
    {
        unsigned old = *(volatile unsigned*)w;
        for (;;) {
            const unsigned running = (old & 255u) - (leaving ? 1u : 0u), here = ((old >> 8) & 255u) + (leaving ? 0u : 1u);
            const unsigned go = here > 0 && here >= running ? 1u : 0u;
            const unsigned next = running | (go ? 0u : here << 8) | (((old >> 16) + go) & 0xffffu) << 16;
            const unsigned seen = atomicCAS(w, old, next);
            if (seen == old)
                return go ? ~0u : old >> 16;  // ~0: started
            old = seen;
        }
    }
    __device__ __forceinline__ void align(int leg, int lane) const
    {
        if (lane == 0) {
            const unsigned starts = change(word + leg, false);
            if (starts != ~0u)
                for (int spin = 0; spin < (1 << 16) && *(volatile unsigned*)(word + leg) >> 16 == starts; ++spin)
                    ;
        }
        __syncwarp();
    }
    __device__ __forceinline__ void join(int leg) const { atomicAdd(word + leg, 1u); }
    __device__ __forceinline__ void leave(int leg) const { change(word + leg, true); }
};

// SplitSync: the CTA is one group, with two warps a leg (the split lists). A
// group alone on an SM waits: its four warps are busy for 33k of a substep's
// 47k cycles, and the tail of a leg, its tibia's spheres above all (10k), holds
// back the next substep's first joint. With the tibias on warps of their own the
// next substep's torso joints, which need the coxas only, run beside that tail.
// A substep is then 27k cycles: the ring of four torso joints (4.1k each), the
// torso's sphere and the damping ring on one side, and on the other a leg's
// joints, spheres, damping and contact velocities in turn (27k too), so a third
// warp a leg would not help. Tried on top and slower or not the same bits: the
// tibia's spheres looked at together before (+0..13 %), the joints' four stages
// unrolled (-5..10 %, but rounded otherwise than the rolled loop of large
// batches, and a world must not depend on its batch).
struct SplitSync {
    static constexpr bool kSplit = true;
    int half;  // 0: the torso's and the coxas' warps, 1: the femurs' and tibias'
    __device__ __forceinline__ void group() const { __syncthreads(); }
    __device__ __forceinline__ void wait(int id) const { bar_sync(id); }
    __device__ __forceinline__ void arrive(int id) const { bar_arrive(id); }
    __device__ __forceinline__ void align(int, int) const {}
};

// Groups that share an SM's memory and registers, and so an aligned CTA.
constexpr int kAligned = sizeof(F) == 4 ? 4 : 2;
constexpr int kSplitTo = sizeof(F) == 4 ? 2 : 1;      // groups per SM

struct AlignedSmem {
    Smem step[kAligned];
    int next[kAligned];    // each slot's next group
    unsigned word[kWarps];
};

// How a launch over n_items worlds is split: worlds per group (one CTA's
// lanes) and the operation list.
//   Worlds per group. A group's time is that of the longest path over its
// worlds' contacts, so with fewer groups than SMs smaller groups are faster,
// up to about half as many groups as SMs (split groups, FP32: 64 worlds one
// per group 272 us, as two groups of 32 283; 1,000 worlds in groups of 14 294,
// of 32 305, of 7 on nearly every SM 324; FP64 399 and 408, then 438, 433 and
// 533; in CTAs of four warps 64: 322 and 353, 1,000: 367 and 386). More also
// crowd out what runs beside the step, so the split stops there; and a launch
// that shares the GPU with others (`alone` false) keeps groups of 32.
//   Operation list: kListLatency up to two groups per SM in FP32, up to one
// in FP64, whose SMs hold two (the figures are at the lists above).
//   Split groups (SplitSync) up to two groups per SM in FP32, one in FP64
// (FP32, CTAs of four warps and split: 1 world 292 and 257 us, 64: 322 and
// 272, 1,000: 367 and 294, 4,096: 405 and 349, 6,000: 459 and 437, 9,400: 504
// and 485; FP64, 1: 445 and 377, 4,096: 632 and 565), where a whole control
// step runs in one launch, no list can reach the reference's cap and nobody
// records contacts.
//   Aligned CTAs (AlignedSync) take a work queue and a whole SM each, so not
// beside others, and all that is more than split groups take (a training step
// of 10,007 standing robots: 843 us in CTAs of their own, 828 aligned; FP64,
// thrown-about robots, 7,000: 781 and 733, 9,400: 832 and 762; larger ones at
// AlignedSync). They run kListThroughput.
struct GroupPlan {
    int per_group, groups, list;
    bool aligned, split;
};
// splittable: a whole control step with uncapped lists that nobody records
inline GroupPlan group_plan(int n_items, int sms, bool alone, bool queue, bool splittable)
{
    const int spread = sms / 2 > 0 ? sms / 2 : 1;
    GroupPlan p;
    p.per_group = kWorlds;
    if (alone && n_items < spread * kWorlds)
        p.per_group = (n_items + spread - 1) / spread;
    p.groups = (n_items + p.per_group - 1) / p.per_group;
    p.list = alone && p.groups <= (sizeof(F) == 4 ? 2 : 1) * sms ? kListLatency : kListThroughput;
    p.aligned = alone && queue && p.groups > kSplitTo * sms;
    p.split = alone && splittable && p.groups <= kSplitTo * sms;
    return p;
}

// One control step of a group's worlds (items first .. first + per_group - 1,
// at most 32: worlds ids[item], or item itself without ids) by the group's
// warps, lane j of warp `leg` here, in the order of the operation list `list`. On return the
// worlds' records, flags, time and unstable marks are written and every
// thread of the CTA has passed the group's last barrier.
//
// Substeps sub0 .. sub1 - 1 of the control step (0 .. M.substeps - 1: the
// whole step). A control step in several such tiles, one launch each, gives
// the worlds of one launch bit for bit: between tiles the record holds the
// bodies (with the normalised q), anchors, touch counts and the summed drive
// torques, and tile_q (13 x 4 floats per world) the position-pass q whose
// rotation the next substep's gyroscopic term uses; the joint outputs, time
// and stability come at the end of the last tile.
template <class Sync, class Mem>
__device__ __forceinline__ void step_group(const Sync& sync, Mem& sm, const DevModel<F>& M, const Worlds<F>& W, const Actuation& A,
                                           F* __restrict__ spill, int spill_per_lane, int lane_cap,
                                           const int* __restrict__ ids, int n_items, int first, int leg, int j,
                                           int sub0, int sub1, F* __restrict__ tile_q, int per_group, int list)
{
    // a split group steps whole control steps with uncapped lists only
    const bool first_tile = Sync::kSplit || sub0 == 0, last_tile = Sync::kSplit || sub1 >= M.substeps;
    // what this warp has of the leg: the coxa (leg 0: and the torso), the femur
    // and tibia, or both; its contact list
    const bool upper = !Sync::kSplit || sync.half == 0, lower = !Sync::kSplit || sync.half == 1;
    const int body0 = upper ? 0 : 1, body1 = lower ? 3 : 1, warp = kWarps * sync.half + leg;
    auto has_sphere = [&](int s) { return s == 0 ? upper : lower; };  // of the leg's: the femur's, the tibia's
    const int item = first + j;
    const int world = j < per_group && item < n_items ? (ids ? ids[item] : item) : -1;
    const bool valid = world >= 0 && world < W.n;
    const int wi = valid ? world : 0;

    F* rec = W.rec + (size_t)wi * W.stride;
    F* sr = rec + W.off_sphere;
    F* jr = rec + W.off_joint;
    const int b_c = 1 + 3 * leg, b_f = 2 + 3 * leg, b_t = 3 + 3 * leg;  // coxa, femur, tibia
    const int j0 = 3 * leg;
    const Ref torso{&sm.torso[0][j]};
    auto body_ref = [&](int slot) {
        return slot == kTorso ? torso : Ref{&sm.leg[leg][slot * kBodyF][j]};
    };
    // actuation (csrc/arc_sim.c:132-136)
    F target0 = F(0), target1 = F(0), target2 = F(0);
    if (valid && upper) {
        target0 = actuate(M, A, world, j0);
        target1 = actuate(M, A, world, j0 + 1);
        jr[j0 * kJointRec] = target0;
        jr[(j0 + 1) * kJointRec] = target1;
    }
    if (valid && lower) {
        target2 = actuate(M, A, world, j0 + 2);
        jr[(j0 + 2) * kJointRec] = target2;
    }
    F tacc0 = F(0), tacc1 = F(0), tacc2 = F(0);
    if (!first_tile) {
        tacc0 = jr[j0 * kJointRec + 3];
        tacc1 = jr[(j0 + 1) * kJointRec + 3];
        tacc2 = jr[(j0 + 2) * kJointRec + 3];
    }
    const bool active = valid && W.unstable[wi] == 0;
    auto stage_body = [&](Ref r, const F* src) {
        setv(r, kX, V{src[0], src[1], src[2]});
        setq(r, kQ, Q{src[3], src[4], src[5], src[6]});
        setq(r, kQP, Q{src[3], src[4], src[5], src[6]});
        setv(r, kV, V{src[7], src[8], src[9]});
        setv(r, kW, V{src[10], src[11], src[12]});
    };
    // the position-pass q of a tile's predecessor
    auto stage_q = [&](Ref r, int body) {
        const F* tq = tile_q + ((size_t)wi * 13 + body) * 4;
        setq(r, kQ, Q{tq[0], tq[1], tq[2], tq[3]});
    };
#pragma unroll 1
    for (int i = body0; i < body1; ++i) {
        stage_body(body_ref(i), rec + (b_c + i) * kBodyRec);
        if (!first_tile)
            stage_q(body_ref(i), b_c + i);
    }
    uint32_t anch = 0;
    const uint32_t* sphr = W.sph + (size_t)wi * 21;
#pragma unroll
    for (int s = 0; s < 5; ++s) {
        if (has_sphere(s)) {
            const F* a = sr + (5 * leg + 1 + s) * kSphereRec;
#pragma unroll
            for (int c = 0; c < 6; ++c)
                sm.anch[leg][6 * s + c][j] = a[c];
            anch |= ((sphr[5 * leg + 1 + s] >> 16) & 1u) << s;
        }
    }
    // warp 0 collides the torso's sphere and keeps its flags
    const bool capped = !Sync::kSplit && kWarps * lane_cap > kMaxContacts;
    if (leg == 0 && upper) {
        stage_body(torso, rec);
        if (!first_tile)
            stage_q(torso, 0);
#pragma unroll
        for (int c = 0; c < 6; ++c)
            torso[kBodyF + c] = sr[c];
        anch |= ((sphr[0] >> 16) & 1u) << 5;
    }
    const TerrainView<F> T = terrain_of(W, wi);
    const F inv_cell = F(1) / T.cell;
    const StepK<F>& st = M.step;
    unsigned long long touches = 0;  // 10 bits per sphere: leg spheres 0..4, torso sphere at 50
    if (!first_tile) {
#pragma unroll
        for (int s = 0; s < 5; ++s)
            touches |= (unsigned long long)(sphr[5 * leg + 1 + s] & 1023u) << (10 * s);
        if (leg == 0)
            touches |= (unsigned long long)(sphr[0] & 1023u) << 50;
    }
    const uint32_t* ops = Sync::kSplit ? &kSplitOps[warp][0] : &kOps[capped ? (int)kListCapped : list][leg][0];
    // a warp's contact records of this lane beyond the on-chip ones; the upper
    // list of a split group's leg fills the room, which holds both, from its end
    constexpr int kOn = Mem::kOnChipRecords;
    auto spill_at = [&](int list_warp, int c) {
        const int slot = Sync::kSplit && list_warp < kWarps ? spill_per_lane - 1 - (c - kOn) : c - kOn;
        return spill + (((size_t)wi * kWarps + leg) * (size_t)spill_per_lane + slot) * 8;
    };
    int last_nc = 0;  // this lane's contact records in the last substep
    sync.group();

    for (int sub = sub0; sub < sub1; ++sub) {
        int nc = 0;
        auto record = [&](int body, V local, V n) {
            if (nc < kOn) {
                const Ref d{&sm.con[warp][nc * 7][j]};
                setv(d, 0, local);
                setv(d, 3, n);
                d[6] = (F)body;
            } else if (nc < lane_cap && ARC_IN_BOUNDS(nc - kOn, spill_per_lane, kCheckSpillWrite)) {
                F* d = spill_at(warp, nc);
                d[0] = local.x; d[1] = local.y; d[2] = local.z;
                d[3] = n.x; d[4] = n.y; d[5] = n.z;
                d[6] = (F)body;
            }
            ++nc;
        };
#pragma unroll 1
        for (int i = 0;; ++i) {
            const uint32_t op = ops[i];
            const uint32_t kind = op & 15u;
            if (kind == OP_END)
                break;
            const int a = (op >> 4) & 15, b = (op >> 8) & 15, wait = (op >> 12) & 15, arrive = (op >> 16) & 15;
            if (op >> 20)
                sync.align(leg, j);
            if (wait)
                sync.wait(wait);
            if (kind == OP_CNT) {
                // double-buffered: a warp may record substep s+1 while
                // another still reads the counts of substep s
                sm.nc[sub & 1][leg][j] = nc;
                sync.group();
            } else if (active) {
                switch (kind) {
                case OP_INT:
                    // csrc/arc_phys.c:658-672
#pragma unroll 1
                    for (int o = a; o < b; ++o) {
                        const Ref r = body_ref(o == 0 ? kTorso : o - 1);
                        const BodyK<F>& k = M.body[o == 0 ? 0 : b_c + o - 1];
                        V x = getv(r, kX), v = getv(r, kV), w = getv(r, kW);
                        const Q q0 = getq(r, kQP);
                        setv(r, kXP, x);
                        v = madd(v, st.gravity, st.h);
                        x = madd(x, v, st.h);
                        if (!k.iso) {
                            const M3<F> rot = m3_from_quat(getq(r, kQ));
                            w = mul(rot, gyroscopic(k, tmul(rot, w), st.h));
                        }
                        setv(r, kX, x);
                        setq(r, kQ, q_turn(q0, scale(w, st.h)));
                        setv(r, kV, v);
                        setv(r, kW, w);
                    }
                    break;
                case OP_JNT:
#pragma unroll 1
                    for (int c = a; c < b; ++c) {
                        const Ref rp = body_ref(c == 0 ? kTorso : c - 1), rc = body_ref(c);
                        const BodyK<F>& kp = M.body[c == 0 ? 0 : b_c + c - 1];
                        const BodyK<F>& kc = M.body[b_c + c];
                        P bp, bc;
                        load_pose(rp, kp, bp);
                        load_pose(rc, kc, bc);
                        F acc = c == 0 ? tacc0 : (c == 1 ? tacc1 : tacc2);
                        const F tgt = c == 0 ? target0 : (c == 1 ? target1 : target2);
                        joint_positions(bp, kp, bc, kc, M.joint[j0 + c], tgt, acc, st.hh);
                        if (c == 0)
                            tacc0 = acc;
                        else if (c == 1)
                            tacc1 = acc;
                        else
                            tacc2 = acc;
                        store_pose(rp, bp);
                        store_pose(rc, bc);
                    }
                    break;
                case OP_COL: {
                    // csrc/arc_phys.c:542-610, spheres a..b-1 of one body
                    const int slot = a == 0 ? kTorso : (a == 1 ? 1 : 2);
                    const int bid = a == 0 ? 0 : (a == 1 ? b_f : b_t);
                    const Ref r = body_ref(slot);
                    const BodyK<F>& k = M.body[bid];
                    P pose;
                    load_pose(r, k, pose);
#pragma unroll 1
                    for (int s = a; s < b; ++s) {
                        const int bit = s == 0 ? 5 : s - 1;
                        const Ref ra{s == 0 ? &sm.torso[kBodyF][j] : &sm.anch[leg][6 * (s - 1)][j]};
                        SphereState<F> ss{getv(ra, 0), getv(ra, 3), (int)((anch >> bit) & 1u)};
                        const int t = collide(pose, k, r, M.sphere[s == 0 ? 0 : 5 * leg + s], ss, T, inv_cell, st,
                                                     [&](V l, V n) { record(bid, l, n); });
                        touches += (unsigned long long)t << (10 * bit);
                        anch = (anch & ~(1u << bit)) | ((uint32_t)(ss.anchored != 0) << bit);
                        setv(ra, 0, ss.anchor);
                        setv(ra, 3, ss.anchor_n);
                    }
                    store_pose(r, pose);
                    if (Sync::kSplit && a == 1)
                        sm.nc[0][leg][j] = nc;  // the femur's, for the lower warp
                    break;
                }
                case OP_UPD:
                    // csrc/arc_phys.c:674-687; the rotation stays that of the
                    // un-normalised q (field Q)
#pragma unroll 1
                    for (int o = a; o < b; ++o) {
                        const Ref r = body_ref(o == 0 ? kTorso : o - 1);
                        Q q = getq(r, kQ);
                        V v, w;
                        update_velocity(q, getv(r, kX), v, w, getv(r, kXP), getq(r, kQP), st);
                        setq(r, kQP, q);
                        setv(r, kV, v);
                        setv(r, kW, w);
                    }
                    break;
                case OP_DMP: {
                    // csrc/arc_phys.c:459-481; the child of joint c is the
                    // parent of joint c+1 (rotation of the position pass)
                    P bp, bc;
                    Ref rp = body_ref(a == 0 ? kTorso : a - 1);
                    bp.q = getq(rp, kQ);
                    body_sync(bp, M.body[a == 0 ? 0 : b_c + a - 1]);
                    V wp = getv(rp, kW);
#pragma unroll 1
                    for (int c = a; c < b; ++c) {
                        const Ref rc = body_ref(c);
                        bc.q = getq(rc, kQ);
                        body_sync(bc, M.body[b_c + c]);
                        V wc = getv(rc, kW);
                        const JointK<F>& J = M.joint[j0 + c];
                        F acc = c == 0 ? tacc0 : (c == 1 ? tacc1 : tacc2);
                        joint_velocities<F, true>(bp.rot, bp.iiw, wp, bc.iiw, wc, J, joint_step_k(J, st), st.h,
                                                  acc);
                        if (c == 0)
                            tacc0 = acc;
                        else if (c == 1)
                            tacc1 = acc;
                        else
                            tacc2 = acc;
                        setv(rp, kW, wp);
                        rp = rc;
                        bp = bc;
                        wp = wc;
                    }
                    setv(rp, kW, wp);
                    break;
                }
                case OP_CVL: {
                    // csrc/arc_phys.c:612-626, the reference's (sphere-major)
                    // list order under its cap
                    int base = 0;
                    if (capped)
                        for (int l = 0; l < leg; ++l)
                            base += sm.nc[sub & 1][l][j];
                    // a split leg's lower warp takes the femur's contacts too,
                    // from its upper warp's list
                    int list_warp = Sync::kSplit && lower ? leg : warp;
                    int count = Sync::kSplit && lower ? sm.nc[0][leg][j] : nc;
#pragma unroll 1
                    for (;; list_warp = warp, count = nc) {
                        const int ncl = count < lane_cap ? count : lane_cap;
#pragma unroll 1
                        for (int c = 0; c < ncl && base + c < kMaxContacts; ++c) {
                            F rc[7];
                            if (c < kOn) {
#pragma unroll
                                for (int f = 0; f < 7; ++f)
                                    rc[f] = sm.con[list_warp][c * 7 + f][j];
                            } else {
                                if (!ARC_IN_BOUNDS(c - kOn, spill_per_lane, kCheckSpillRead))
                                    continue;
                                const F* src = spill_at(list_warp, c);
#pragma unroll
                                for (int f = 0; f < 7; ++f)
                                    rc[f] = src[f];
                            }
                            const int bid = (int)rc[6];
                            if ((bid == 0) != (a == 1))
                                continue;
                            const Ref r = body_ref(bid == 0 ? kTorso : (bid == b_f ? 1 : 2));
                            const BodyK<F>& k = M.body[bid];
                            P pose;
                            pose.q = getq(r, kQ);
                            body_sync(pose, k);
                            V v = getv(r, kV), w = getv(r, kW);
                            contact_velocity(pose.rot, pose.iiw, k.inv_mass, v, w,
                                             ContactRec<F>{V{rc[0], rc[1], rc[2]}, V{rc[3], rc[4], rc[5]}});
                            setv(r, kV, v);
                            setv(r, kW, w);
                        }
                        if (!Sync::kSplit || list_warp == warp)
                            break;
                    }
                    break;
                }
                default:
                    break;
                }
            }
            if (arrive)
                sync.arrive(arrive);
        }
        last_nc = nc;
    }
    sync.group();

    if (!Sync::kSplit && last_tile && W.lastc) {
        // the last substep's contact list in the reference's order
        // (csrc/arc_phys.c:493-499): sphere by sphere, the torso's first,
        // which is the four warps' lists in warp order (the torso's records
        // lead warp 0's). Counts go through the (now free) count array.
        sm.nc[0][leg][j] = last_nc < lane_cap ? last_nc : lane_cap;
        sync.group();
        if (active) {
            int before = 0, total = 0;  // records of the warps listed ahead of this one; of all
            for (int l = 0; l < kWarps; ++l) {
                total += sm.nc[0][l][j];
                if (l < leg)
                    before += sm.nc[0][l][j];
            }
            const int mine = sm.nc[0][leg][j];
            F* dst = W.lastc + (size_t)world * kMaxContacts * kContactRec;
#pragma unroll 1
            for (int c = 0; c < mine; ++c) {
                const int at = before + c;
                if (at >= kMaxContacts)
                    continue;
                F rc[7];
                if (c < kOn) {
#pragma unroll
                    for (int f = 0; f < 7; ++f)
                        rc[f] = sm.con[warp][c * 7 + f][j];
                } else {
                    if (!ARC_IN_BOUNDS(c - kOn, spill_per_lane, kCheckSpillRead))
                        continue;
                    const F* src = spill_at(warp, c);
#pragma unroll
                    for (int f = 0; f < 7; ++f)
                        rc[f] = src[f];
                }
                F* d = dst + (size_t)at * kContactRec;
                d[0] = rc[6];
                for (int f = 0; f < 6; ++f)
                    d[1 + f] = rc[f];
            }
            if (leg == 0)
                W.lastn[world] = total < kMaxContacts ? total : kMaxContacts;
        }
    }

    if (!last_tile) {
        // hand the state to the next tile
        if (active) {
            auto keep = [&](Ref r, int body) {
                F* d = rec + body * kBodyRec;
                const V x = getv(r, kX), v = getv(r, kV), w = getv(r, kW);
                const Q q = getq(r, kQP), qa = getq(r, kQ);
                d[0] = x.x; d[1] = x.y; d[2] = x.z;
                d[3] = q.w; d[4] = q.x; d[5] = q.y; d[6] = q.z;
                d[7] = v.x; d[8] = v.y; d[9] = v.z;
                d[10] = w.x; d[11] = w.y; d[12] = w.z;
                F* tq = tile_q + ((size_t)wi * 13 + body) * 4;
                tq[0] = qa.w; tq[1] = qa.x; tq[2] = qa.y; tq[3] = qa.z;
            };
#pragma unroll 1
            for (int i = 0; i < 3; ++i)
                keep(body_ref(i), b_c + i);
            if (leg == 0)
                keep(torso, 0);
            jr[j0 * kJointRec + 3] = tacc0;
            jr[(j0 + 1) * kJointRec + 3] = tacc1;
            jr[(j0 + 2) * kJointRec + 3] = tacc2;
            uint32_t* sphw = W.sph + (size_t)world * 21;
#pragma unroll
            for (int s = 0; s < 5; ++s) {
                F* a = sr + (5 * leg + 1 + s) * kSphereRec;
#pragma unroll
                for (int c = 0; c < 6; ++c)
                    a[c] = sm.anch[leg][6 * s + c][j];
                sphw[5 * leg + 1 + s] = (uint32_t)((touches >> (10 * s)) & 1023u) | (((anch >> s) & 1u) << 16);
            }
            if (leg == 0) {
#pragma unroll
                for (int c = 0; c < 6; ++c)
                    sr[c] = torso[kBodyF + c];
                sphw[0] = (uint32_t)((touches >> 50) & 1023u) | (((anch >> 5) & 1u) << 16);
            }
        }
        sync.group();
        return;
    }

    // epilogue (csrc/arc_phys.c:739-746), from the normalised quaternions
    int bad = 0;
    if (active) {
        const Ref r0 = body_ref(0), r1 = body_ref(1), r2 = body_ref(2);
        const Q tq = getq(torso, kQP), q0 = getq(r0, kQP), q1 = getq(r1, kQP), q2 = getq(r2, kQP);
        const V tw = getv(torso, kW), w0 = getv(r0, kW), w1 = getv(r1, kW), w2 = getv(r2, kW);
        const JointK<F>& J0 = M.joint[j0];
        const JointK<F>& J1 = M.joint[j0 + 1];
        const JointK<F>& J2 = M.joint[j0 + 2];
        if (upper) {
            jr[(j0 + 0) * kJointRec + 1] = joint_angle(tq, q0, J0);
            jr[(j0 + 0) * kJointRec + 2] = joint_rate(tq, tw, w0, J0);
            jr[(j0 + 1) * kJointRec + 1] = joint_angle(q0, q1, J1);
            jr[(j0 + 1) * kJointRec + 2] = joint_rate(q0, w0, w1, J1);
            jr[(j0 + 0) * kJointRec + 3] = tacc0 / F(M.substeps);
            jr[(j0 + 1) * kJointRec + 3] = tacc1 / F(M.substeps);
        }
        if (lower) {
            jr[(j0 + 2) * kJointRec + 1] = joint_angle(q1, q2, J2);
            jr[(j0 + 2) * kJointRec + 2] = joint_rate(q1, w1, w2, J2);
            jr[(j0 + 2) * kJointRec + 3] = tacc2 / F(M.substeps);
        }
        auto put = [&](Ref r, F* d) {
            const V x = getv(r, kX), v = getv(r, kV), w = getv(r, kW);
            const Q q = getq(r, kQP);
            bad |= body_unstable(x, v, w);
            d[0] = x.x; d[1] = x.y; d[2] = x.z;
            d[3] = q.w; d[4] = q.x; d[5] = q.y; d[6] = q.z;
            d[7] = v.x; d[8] = v.y; d[9] = v.z;
            d[10] = w.x; d[11] = w.y; d[12] = w.z;
        };
#pragma unroll 1
        for (int i = body0; i < body1; ++i)
            put(body_ref(i), rec + (b_c + i) * kBodyRec);
        uint32_t* sphw = W.sph + (size_t)world * 21;
#pragma unroll
        for (int s = 0; s < 5; ++s) {
            if (has_sphere(s)) {
                F* a = sr + (5 * leg + 1 + s) * kSphereRec;
#pragma unroll
                for (int c = 0; c < 6; ++c)
                    a[c] = sm.anch[leg][6 * s + c][j];
                sphw[5 * leg + 1 + s] = (uint32_t)((touches >> (10 * s)) & 1023u) | (((anch >> s) & 1u) << 16);
            }
        }
        if (leg == 0 && upper)
            put(torso, rec);
        if (leg == 0 && upper) {
#pragma unroll
            for (int c = 0; c < 6; ++c)
                sr[c] = torso[kBodyF + c];
            sphw[0] = (uint32_t)((touches >> 50) & 1023u) | (((anch >> 5) & 1u) << 16);
        }
    }
    sm.bad[warp][j] = bad;
    sync.group();
    if (active && leg == 0 && upper) {
        W.time[world] += M.step_dt;
        int any = 0;
#pragma unroll
        for (int w = 0; w < (Sync::kSplit ? 2 : 1) * kWarps; ++w)
            any |= sm.bad[w][j];
        if (any)
            W.unstable[world] = 1;
    }
}

template <class W> inline bool splittable(const W& w, int lane_cap, int sub0, int sub1, int substeps)
{
    return kWarps * lane_cap <= kMaxContacts && !w.lastc && sub0 == 0 && sub1 >= substeps;
}

// One group per CTA of 2 * kThreads threads, split (SplitSync).
__device__ __forceinline__ void step_split(SplitSmem& sm, const DevModel<F>& M, const Worlds<F>& W,
                                           const Actuation& A, F* __restrict__ spill, int spill_per_lane,
                                           int lane_cap, const int* __restrict__ ids, int n_items, int per_group)
{
    const int tid = threadIdx.x % kThreads;
    step_group(SplitSync{(int)threadIdx.x / kThreads}, sm, M, W, A, spill, spill_per_lane, lane_cap, ids, n_items,
               blockIdx.x * per_group, tid / kWorlds, tid % kWorlds, 0, M.substeps, nullptr, per_group, 0);
}

// The groups of a launch in CTAs of kAligned groups, one CTA per SM: slot g of
// CTA b takes group b + g * gridDim.x first (so that few groups spread over
// the SMs) and then what the queue hands out. All threads of the CTA call it.
//
// What is left over from whole waves of slots runs on SMs that are emptying:
// up to kAligned / 2 groups per SM it takes the latency list, and fewer worlds
// than one group per SM are split into as many groups as SMs (the step of
// 20,000 thrown-about robots, 33 groups more than one wave: 1,160 us without
// either, 1,145 with; 25,000: 1,260 and 1,231; 65,536: 2,505 and 2,469).
__device__ __forceinline__ void step_aligned(AlignedSmem& as, const DevModel<F>& M, const Worlds<F>& W,
                                             const Actuation& A, F* __restrict__ spill, int spill_per_lane,
                                             int lane_cap, const int* __restrict__ ids, int n_items, int* queue,
                                             int sub0, int sub1, F* __restrict__ tile_q, int list)
{
    // each group's legs start at another warp: warps 4 apart share a scheduler,
    // and with leg k of every group on the same one, that scheduler had the
    // chain's four joints to issue at once while the others waited (thrown-about
    // robots, 16,384 worlds 740 -> 674 us, 65,536 2,694 -> 2,475; FP64 16,384
    // 1,505 -> 1,398)
    const int tid = threadIdx.x % kThreads, slot = threadIdx.x / kThreads, j = tid % kWorlds;
    const int leg = (tid / kWorlds + slot * (kWarps / kAligned)) % kWarps;
    const int grid = gridDim.x, whole = n_items / (kAligned * grid * kWorlds) * kAligned * grid;  // groups
    const int rest = n_items - whole * kWorlds;
    const bool tail = whole > 0 && rest <= kAligned / 2 * grid * kWorlds;
    const int rest_per = tail && rest < grid * kWorlds ? (rest + grid - 1) / grid : kWorlds;
    const int n_groups = whole + (rest > 0 ? (rest + rest_per - 1) / rest_per : 0);
    if (threadIdx.x < kWarps)
        as.word[threadIdx.x] = 0u;
    __syncthreads();  // the only barrier of the whole CTA: its barrier 0 is slot 0's from here on
    const AlignedSync sync{kWarps * slot, as.word};
    int group = blockIdx.x + slot * grid;
#pragma unroll 1
    while (group < n_groups) {
        if (j == 0)
            sync.join(leg);
        const bool over = group >= whole;
        step_group(sync, as.step[slot], M, W, A, spill, spill_per_lane, lane_cap, ids, n_items,
                   over ? whole * kWorlds + (group - whole) * rest_per : group * kWorlds, leg, j, sub0, sub1,
                   tile_q, over ? rest_per : kWorlds, over && tail ? (int)kListLatency : list);
        if (j == 0)
            sync.leave(leg);
        if (tid == 0)
            as.next[slot] = kAligned * grid + atomicAdd(queue, 1);
        sync.group();
        group = as.next[slot];
        sync.group();
    }
    // the last slot to leave zeroes the queue for the next launch
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(queue + 1, 1) == kAligned * grid - 1) {
            queue[0] = 0;
            queue[1] = 0;
            __threadfence();
        }
    }
}

}  // namespace
}  // namespace wl
}  // namespace arc
