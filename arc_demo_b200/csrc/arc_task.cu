// arc_task.cu - task layer kernels (arc/task.py on the device) and the
// cooperative world reset (csrc/arc_sim.c:88-110).
#include "arc_task.cuh"
#include "arc_step_warps.cuh"

namespace arc {

namespace {

// ---------------------------------------------------------------------------
// reference RNG (csrc/arc_rng.h:14-53), integer exact

struct Xorshift {
    uint32_t s[4];
    __device__ __forceinline__ uint32_t next()
    {
        uint32_t t = s[3], v = s[0];
        s[3] = s[2];
        s[2] = s[1];
        s[1] = v;
        t = t ^ (t << 11);
        t ^= t >> 8;
        s[0] = t ^ v ^ (v >> 19);
        return s[0];
    }
    __device__ __forceinline__ void seed(uint32_t seed)
    {
        for (int i = 0; i < 4; ++i) {
            uint32_t x = seed + 0x9e3779b9U * (uint32_t)(i + 1);
            x = (x ^ (x >> 16)) * 0x7feb352dU;
            x = (x ^ (x >> 15)) * 0x846ca68bU;
            seed = x ^ (x >> 16);
            s[i] = seed ? seed : 1U;
        }
    }
};

// Jumping ahead in the stream. xorshift128 is linear over GF(2): one step
// is a 128 x 128 bit matrix M acting on the state (s0 s1 s2 s3). A reset's
// draws are cut into 32 slices of kSlice, one per lane of a warp, and row b
// of g_skip holds column b of M^(kSlice * lane) for every lane (built once
// per device by k_skip_init), so all lanes jump to their slices by XORing the
// rows of the state bits that are set: the same rows for every lane, 512
// coalesced bytes each, sixteen loads in flight. Row 128 is zero. The draws
// that follow are the stream's own, bit for bit. (Skipping each lane by
// powers of two, M^(2^k), took three times the loads and diverged.)
constexpr int kSlice = 149;  // 32 slices hold the 4,742 draws of a 64 x 64 terrain and its stance
__device__ uint4 g_skip[129][32];

__global__ void k_skip_init()
{
    const int lane = blockIdx.x, b = threadIdx.x;
    Xorshift r;
    for (int w = 0; w < 4; ++w)
        r.s[w] = (b >> 5) == w ? 1u << (b & 31) : 0u;
    for (int it = 0; it < kSlice * lane; ++it)
        r.next();
    g_skip[b][lane] = make_uint4(r.s[0], r.s[1], r.s[2], r.s[3]);
}

// Moves a state that all lanes of a warp share to the start of the lane's
// slice. rows: kSkipRows bytes of shared memory for the warp.
constexpr int kSkipRows = 128 + 16;
__device__ __forceinline__ void rng_to_slice(Xorshift& r, int lane, unsigned char* rows)
{
    // the rows of the set bits, listed by the lanes: lane l looks at bits 4l .. 4l + 3
    const int word = lane >> 3, bit0 = 4 * lane;
    const uint32_t mine = (word == 0 ? r.s[0] : word == 1 ? r.s[1] : word == 2 ? r.s[2] : r.s[3]) >> (bit0 & 31) & 15u;
    int at = 0, n = 0;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        at += w < word ? __popc(r.s[w]) : (w == word ? __popc(r.s[w] & ((1u << (bit0 & 31)) - 1u)) : 0);
        n += __popc(r.s[w]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
        if ((mine >> u) & 1u)
            rows[at++] = (unsigned char)(bit0 + u);
    if (lane < 16)
        rows[n + lane] = 128;
    __syncwarp();
    uint4 o = make_uint4(0u, 0u, 0u, 0u);
    for (int k = 0; k < n; k += 16) {
        uint4 c[16];
#pragma unroll
        for (int u = 0; u < 16; ++u)
            c[u] = g_skip[rows[k + u]][lane];
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            o.x ^= c[u].x;
            o.y ^= c[u].y;
            o.z ^= c[u].z;
            o.w ^= c[u].w;
        }
    }
    r.s[0] = o.x;
    r.s[1] = o.y;
    r.s[2] = o.z;
    r.s[3] = o.w;
}

// rng_range(lo, hi) of a raw draw u (csrc/arc_rng.h:45-53)
__device__ __forceinline__ double range_of(uint32_t u, double lo, double hi)
{
    return lo + (hi - lo) * (u * (1.0 / 4294967296.0));
}

// ---------------------------------------------------------------------------
// device RNG of the task layer (checkpoints, reset seeds): a counter-based
// splitmix64 stream per (seed, world, kind). The reference draws these from
// numpy's PCG64 on the host (arc/task.py:117,138-139); the device cannot
// reproduce that stream, so it draws the same distributions from its own.

__device__ __forceinline__ uint64_t splitmix64(uint64_t x)
{
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

__device__ __forceinline__ uint64_t stream_u64(uint64_t seed, int world, uint32_t kind, uint32_t counter)
{
    return splitmix64(splitmix64(seed ^ (((uint64_t)(uint32_t)world << 32) | kind)) + counter);
}

__device__ __forceinline__ double unit(uint64_t x) { return (double)(x >> 11) * (1.0 / 9007199254740992.0); }

// the identity of world i's streams: its index, or the key its tenant gave it
__device__ __forceinline__ int key_of(const TaskState& S, int i) { return S.key ? (int)S.key[i] : i; }

// ---------------------------------------------------------------------------
// world read-outs in FP64 (what arc_sim_observe returns, csrc/arc_sim.c:140-183)

// The largest touch share of the spheres of one contact channel.
template <class R>
__device__ __forceinline__ double contact_of(const DevModel<R>& M, const uint32_t* sph, int channel)
{
    const double inv = 1.0 / M.substeps;
    double c = 0.0;
    for (int s = 0; s < M.ns; ++s) {
        const double v = (int)(sph[s] & 0xffffu) * inv;
        if (M.channel[s] == channel)
            c = c > v ? c : v;
    }
    return c;
}

template <class R> __device__ __forceinline__ double height_at(const Worlds<R>& W, int i, double x, double y)
{
    const TerrainGeomD g = W.tgd[i];
    double fx = floor((x - g.ox) / g.cell), fy = floor((y - g.oy) / g.cell);
    if (!(fx >= 0.0 && fy >= 0.0 && fx < g.nx && fy < g.ny))
        return g.outside;
    if (!terrain_column_ok(W, i, (int)fx + (long long)(int)fy * g.nx, kCheckHeightsRead))
        return g.outside;
    return (double)W.th[W.toff[i] + (int)fx + (int)fy * g.nx];
}

// |angle| between the gaze (body +x on the ground) and the target (arc/task.py:79-85)
__device__ __forceinline__ double gaze_error(const M3<double>& rot, V3<double> pos, const double* target)
{
    double fx = rot.m[0][0], fy = rot.m[1][0];
    double dx = target[0] - pos.x, dy = target[1] - pos.y;
    return fabs(atan2(fx * dy - fy * dx, fx * dx + fy * dy));
}

// R^T a, summed like numpy's a @ R for a row vector
__device__ __forceinline__ V3<double> rt_mul(const M3<double>& r, V3<double> a)
{
    return V3<double>{a.x * r.m[0][0] + a.y * r.m[1][0] + a.z * r.m[2][0],
                      a.x * r.m[0][1] + a.y * r.m[1][1] + a.z * r.m[2][1],
                      a.x * r.m[0][2] + a.y * r.m[1][2] + a.z * r.m[2][2]};
}

constexpr int kHeightsAt = 9 + 3 * kNumJoints + 3;  // offset of the heights in an observation row

__device__ __forceinline__ float obs_value(double v)
{
    float f = (float)v;
    return isfinite(f) ? f : 0.0f;
}

// The heading frame of the terrain heights (csrc/arc_sim.c:185-203).
__device__ __forceinline__ void heading_of(Q4<double> q, double& cy, double& sy)
{
    const V3<double> f = qrotate(q, V3<double>{1.0, 0.0, 0.0});
    const double yaw = atan2(f.y, f.x);
    cy = cos(yaw);
    sy = sin(yaw);
}

// Where a world's terrain heights are sampled (csrc/arc_sim.c:185-203): its
// heading, position and columns.
template <class R> struct HeightFrame {
    double cy, sy, x, y;
    double z;  // height of the standing torso's ground: x.z - stand_height
    double cell, inv_cell, ox, oy, outside, nx, ny;
    const R* th;
    int pitch, world;
};

template <class R>
__device__ __forceinline__ HeightFrame<R> height_frame(const TaskParams& P, const Worlds<R>& W, int i, V3<double> x,
                                                       Q4<double> q)
{
    const TerrainGeomD g = W.tgd[i];
    HeightFrame<R> f;
    heading_of(q, f.cy, f.sy);
    f.x = x.x;
    f.y = x.y;
    f.z = x.z - P.stand_height;
    f.cell = g.cell;
    f.inv_cell = 1.0 / g.cell;
    f.ox = g.ox;
    f.oy = g.oy;
    f.outside = g.outside;
    f.nx = g.nx;
    f.ny = g.ny;
    f.th = W.th + W.toff[i];
    f.pitch = g.nx;
    f.world = i;
    return f;
}

// The height at (fo, lo) in the frame.
template <class R>
__device__ __forceinline__ double sample_height(const Worlds<R>& W, const HeightFrame<R>& f, double fo, double lo)
{
    const double px = f.x + f.cy * fo - f.sy * lo, py = f.y + f.sy * fo + f.cy * lo;
    // csrc/arc_terrain.h:42-50: floor((p - o) / cell) in 0 .. n - 1, which
    // the quotient itself decides
    const double qx = divide(px - f.ox, f.cell, f.inv_cell), qy = divide(py - f.oy, f.cell, f.inv_cell);
    const bool in = qx >= 0.0 && qy >= 0.0 && qx < f.nx && qy < f.ny &&
                    terrain_column_ok(W, f.world, (int)qx + (long long)(int)qy * f.pitch, kCheckHeightsRead);
    const int idx = in ? (int)qx + (int)qy * f.pitch : 0;
    const double top = (double)f.th[idx];
    return in ? top : f.outside;
}

// The observation's entry of a terrain height.
template <class R> __device__ __forceinline__ float height_value(const HeightFrame<R>& f, double h)
{
    const double rel = f.z - h;
    return obs_value(rel < -1.0 ? -1.0 : (rel > 1.0 ? 1.0 : rel));
}

// The parts of an observation row (arc/task.py:231-259): entries 0..8 the
// torso's, 9..44 the joints', 45..47 the checkpoint's, then the heights and
// the feet's contacts.
__device__ __forceinline__ void obs_torso(const M3<double>& r, V3<double> v, V3<double> w, float* row)
{
    row[0] = obs_value(-r.m[2][0]);
    row[1] = obs_value(-r.m[2][1]);
    row[2] = obs_value(-r.m[2][2]);
    const V3<double> lin = rt_mul(r, v), ang = rt_mul(r, w);
    row[3] = obs_value(lin.x);
    row[4] = obs_value(lin.y);
    row[5] = obs_value(lin.z);
    row[6] = obs_value(0.25 * ang.x);
    row[7] = obs_value(0.25 * ang.y);
    row[8] = obs_value(0.25 * ang.z);
}

__device__ __forceinline__ void obs_joint(const TaskParams& P, int j, double angle, double rate, double action,
                                          float* row)
{
    row[9 + j] = obs_value(angle - P.default_angles[j]);
    row[9 + kNumJoints + j] = obs_value(0.1 * rate);
    row[9 + 2 * kNumJoints + j] = obs_value(action);
}

// c, s: cosine and sine of the heading
__device__ __forceinline__ void obs_target(double c, double s, double dx, double dy, float* row)
{
    const double fwd = c * dx + s * dy, left = -s * dx + c * dy;
    double dist = hypot(fwd, left);
    dist = dist > 1e-6 ? dist : 1e-6;
    row[kHeightsAt - 3] = obs_value(fwd / dist);
    row[kHeightsAt - 2] = obs_value(left / dist);
    row[kHeightsAt - 1] = obs_value((dist < 6.0 ? dist : 6.0) / 6.0);
}

// Checkpoint 3-6 m away inside the terrain (arc/task.py:127-151), drawn
// from the device stream; also refreshes target_z, prev_dist, prev_gaze.
template <class R>
__device__ void place_target(const TaskParams& P, const Worlds<R>& W, const TaskState& S, int i, V3<double> pos,
                             const M3<double>& rot)
{
    const double limit = P.half_extent - P.border;
    double tx = 0.5 * pos.x, ty = 0.5 * pos.y;
    for (int t = 0; t < 20; ++t) {
        const unsigned k = S.draws[i]++;
        const double ang = -kPi + 2.0 * kPi * unit(stream_u64(P.seed, key_of(S, i), 1u, 2u * k));
        const double dist = P.checkpoint_min_dist +
                            (P.checkpoint_max_dist - P.checkpoint_min_dist) *
                                unit(stream_u64(P.seed, key_of(S, i), 1u, 2u * k + 1u));
        const double cx = pos.x + dist * cos(ang), cy = pos.y + dist * sin(ang);
        if (fabs(cx) < limit && fabs(cy) < limit) {
            tx = cx;
            ty = cy;
            break;
        }
    }
    S.target[2 * i] = tx;
    S.target[2 * i + 1] = ty;
    S.target_z[i] = height_at(W, i, tx, ty);
    const double dx = tx - pos.x, dy = ty - pos.y;
    S.prev_dist[i] = sqrt(dx * dx + dy * dy);
    S.prev_gaze[i] = gaze_error(rot, pos, S.target + 2 * i);
    S.in_view[i] = S.prev_gaze[i] < P.fov_rad;
}

// ---------------------------------------------------------------------------
// arc/task.py:155-220, and 231-259 for the observation: 32 worlds per CTA

__device__ __forceinline__ double clip_action(float action)
{
    const double a = (double)action;
    return a < -1.0 ? -1.0 : (a > 1.0 ? 1.0 : a);
}

// One world's step of the task layer but its observation and stored action;
// returns whether its episode ended. jr, sph: its joints' and spheres' records.
template <class R>
__device__ __forceinline__ bool task_step_world(const DevModel<R>& M, const Worlds<R>& W, const TaskParams& P,
                                                const TaskState& S, const TaskOut& O, const R* jr,
                                                const uint32_t* sph, const float* action, const float* prev_action,
                                                V3<double> x, Q4<double> q, V3<double> v, V3<double> w,
                                                const M3<double>& rot, int i)
{
    const int steps = S.steps[i] + 1;
    S.steps[i] = steps;
    const double* tgt = S.target + 2 * i;
    const double dist = hypot(tgt[0] - x.x, tgt[1] - x.y);
    const double gaze = gaze_error(rot, x, tgt);
    double view = (cos(gaze) - P.cos_fov) / (1.0 - P.cos_fov);
    view = view < 0.0 ? 0.0 : (view > 1.0 ? 1.0 : view);
    const bool in_view = gaze < P.fov_rad;
    double progress = S.prev_dist[i] - dist;
    progress = progress < P.max_speed * P.dt ? progress : P.max_speed * P.dt;
    if (progress > 0)
        progress = progress * view;
    const double turn = S.prev_gaze[i] - gaze;
    const bool reached = dist < P.checkpoint_radius && in_view;
    const V3<double> br = rt_mul(rot, w);
    const bool torso = contact_of(M, sph, kNumLegs) > 0;
    const int torso_steps = torso ? S.torso_steps[i] + 1 : 0;
    S.torso_steps[i] = torso_steps;
    double power = 0.0, rate = 0.0;
    for (int j = 0; j < kNumJoints; ++j) {
        power += fabs((double)jr[j * kJointRec + 2] * (double)jr[j * kJointRec + 3]);
        const double d = clip_action(action[j]) - (double)prev_action[j];
        rate += d * d;
    }
    double reward = P.w_progress * progress + P.w_turn * turn + P.w_checkpoint * (reached ? 1.0 : 0.0) - P.w_time -
                    P.w_energy * power * P.dt - P.w_action_rate * rate -
                    P.w_body_contact * (contact_of(M, sph, kNumLegs + 1) > 0 ? 1.0 : 0.0) -
                    P.w_torso_contact * (torso ? 1.0 : 0.0) - P.w_body_rate * (br.x * br.x + br.y * br.y) -
                    P.w_bounce * (v.z * v.z);
    bool finite = true;
    {
        const double r13[13] = {x.x, x.y, x.z, q.w, q.x, q.y, q.z,
                                v.x, v.y, v.z, w.x, w.y, w.z};
        for (int c = 0; c < 13; ++c)
            finite = finite && isfinite(r13[c]);
    }
    const bool bad = W.unstable[i] != 0 || !finite;
    const bool vd = fabs(x.x) > P.half_extent || fabs(x.y) > P.half_extent || x.z < P.void_z;
    const bool flip = rot.m[2][2] < P.flip_up_z;
    const bool beached = torso_steps > P.beached_steps;
    const bool fell = flip || beached || vd || bad;
    const int cause = bad ? 1 : (vd ? 2 : (flip ? 3 : (beached ? 4 : 0)));
    if (fell)
        reward = reward - P.w_fall;
    if (bad)
        reward = -P.w_fall;
    S.prev_dist[i] = dist;
    S.prev_gaze[i] = gaze;
    S.in_view[i] = in_view;
    const int checkpoints = S.checkpoints[i] + (reached ? 1 : 0);
    S.checkpoints[i] = checkpoints;
    if (reached && !fell)
        place_target(P, W, S, i, x, rot);
    const bool truncated = steps >= P.max_steps && !fell;
    O.reward[i] = (float)reward;
    O.terminated[i] = fell;
    O.truncated[i] = truncated;
    O.cause[i] = (signed char)cause;
    const bool done = fell || truncated;
    if (done) {
        O.ended_checkpoints[i] = checkpoints;
        O.ended_difficulty[i] = S.difficulty[i];
        O.ended_steps[i] = steps;
        if (P.curriculum) {
            // arc/task.py:222-227
            const bool up = checkpoints >= P.level_up_checkpoints;
            const bool down = fell && checkpoints == 0 && steps < P.level_down_steps;
            double lvl = S.level[i] + P.level_step * ((up ? 1.0 : 0.0) - (down ? 1.0 : 0.0));
            lvl = rint(lvl * 1e6) / 1e6;
            S.level[i] = lvl < 0.0 ? 0.0 : (lvl > P.max_difficulty ? P.max_difficulty : lvl);
        }
        if (O.done_list)
            O.done_list[atomicAdd(O.done_count, 1)] = i;
    }
    return done;
}

// What the task layer does with a group of worlds.
enum : int {
    kTaskStep = 0,     // the step, no observation
    kTaskStepObs = 1,  // the step and the observation
    kTaskObserve = 2,  // the observation alone
};

constexpr int kTaskWorlds = 32;
constexpr int kTaskThreads = 128;

constexpr int kTaskSpheres = 21;  // the quadruped's

template <class R> struct TaskSmem {
    HeightFrame<R> frame[kTaskWorlds];
    double head_c[kTaskWorlds], head_s[kTaskWorlds];
    double off[kNumOffsets][2];
    int world[kTaskWorlds];
    int done[kTaskWorlds];  // the world's episode ended in this step
    // the worlds' records, copied in (odd row lengths: no bank conflicts)
    R rec[kTaskWorlds][kBodyRec + kNumJoints * kJointRec];
    uint32_t sph[kTaskWorlds][kTaskSpheres];
    float action[kTaskWorlds][kNumJoints + 1], prev[kTaskWorlds][kNumJoints + 1];
    // their observation rows but the heights: entries 0..47, the feet's contacts
    float row[kTaskWorlds][kHeightsAt + kNumLegs + 1];
};

// The task layer on up to 32 worlds by the four warps of a CTA: lane j of
// every warp has the same world (< 0: none). Warp 0 does the step (rewards,
// terminations, the next checkpoint), warp 1 the torso's and the
// checkpoint's entries, warp 2 the feet's and the frame the heights are
// sampled in, warp 3 the joints'; then all threads sample the heights, on
// consecutive entries of a row. Compiled once per mode (not inlined): the
// task kernels and the fused control step run the same code. On return every
// thread has passed a barrier after the last read of ts but done.
//
// Latency bound: a chain of FP64 functions per world, then scattered terrain
// loads. One thread per world did all but the heights in 35 us whatever the
// batch, each lane reading its own record and writing its own row 32 sectors
// at a time; here the records come in and the rows go out through shared
// memory, a lane per word, and the chain's parts run side by side. The
// heights took another 79-102 us per 65,536 worlds in a kernel whose nine
// threads per world each took the heading's arctangent, sine and cosine anew,
// read the sample offsets from the constant bank at another address in every
// lane, and divided twice; a warp per world keeps its offsets in registers
// and has five samples in flight per lane (a thread per sample, with the
// frame read from shared memory for each, took 70k cycles against 25k). Both
// together: 65,536 worlds 205 -> 98 us, 4,096 48 -> 18 us, FP64 16,384 78 ->
// 33 us; the observation alone of one world 42 -> 9 us.
template <class R, int kMode>
__device__ __noinline__ void task_group(TaskSmem<R>& ts, const DevModel<R>& M, const Worlds<R>& W, const TaskParams& P,
                                        const TaskState& S, const TaskOut& O, const float* __restrict__ actions,
                                        int i)
{
    const int tid = threadIdx.x, role = tid / 32, lane = tid & 31;
    if (role == 0)
        ts.world[lane] = i;
    if (kMode != kTaskStep)
        for (int c = tid; c < 2 * kNumOffsets; c += kTaskThreads)
            ts.off[c / 2][c % 2] = P.offsets[c / 2][c % 2];
    __syncthreads();
    // each warp copies eight worlds, four at a time: a lane per word
    constexpr int kRec = kBodyRec + kNumJoints * kJointRec, kEach = kTaskWorlds / (kTaskThreads / 32);
    static_assert(kRec > 32 && kRec <= 64 && kTaskSpheres <= 32 && kNumJoints <= 16, "words of a world per lane");
#pragma unroll 1
    for (int k0 = role * kEach; k0 < (role + 1) * kEach; k0 += 4) {
        R lo[4], hi[4];
        uint32_t sph[4];
        float act[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int w = ts.world[k0 + u] < 0 ? 0 : ts.world[k0 + u];
            const R* rec = W.rec + (size_t)w * W.stride;
            const int c = lane + 32;
            lo[u] = rec[lane < kBodyRec ? lane : W.off_joint + lane - kBodyRec];
            hi[u] = c < kRec ? rec[W.off_joint + c - kBodyRec] : R(0);
            sph[u] = lane < kTaskSpheres ? W.sph[(size_t)w * kTaskSpheres + lane] : 0u;
            // lanes 0 .. 11: the stored action; 16 .. 27: the new one
            act[u] = 0.0f;
            if ((lane & 15) < kNumJoints && (lane < 16 || kMode != kTaskObserve))
                act[u] = (lane < 16 ? S.prev_action : actions)[(size_t)w * kNumJoints + (lane & 15)];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            ts.rec[k0 + u][lane] = lo[u];
            if (lane + 32 < kRec)
                ts.rec[k0 + u][lane + 32] = hi[u];
            if (lane < kTaskSpheres)
                ts.sph[k0 + u][lane] = sph[u];
            if ((lane & 15) < kNumJoints)
                (lane < 16 ? ts.prev : ts.action)[k0 + u][lane & 15] = act[u];
        }
    }
    __syncthreads();
    V3<double> x{0.0, 0.0, 0.0};
    if (i >= 0) {
        const R* rec = ts.rec[lane];
        const R* jr = rec + kBodyRec;
        float* row = ts.row[lane];
        x = V3<double>{(double)rec[0], (double)rec[1], (double)rec[2]};
        const Q4<double> q{(double)rec[3], (double)rec[4], (double)rec[5], (double)rec[6]};
        if (role <= 1) {
            const V3<double> v{(double)rec[7], (double)rec[8], (double)rec[9]};
            const V3<double> w{(double)rec[10], (double)rec[11], (double)rec[12]};
            const M3<double> rot = m3_from_quat(q);
            if (role == 0) {
                if (kMode != kTaskObserve)
                    ts.done[lane] = task_step_world(M, W, P, S, O, jr, ts.sph[lane], ts.action[lane], ts.prev[lane],
                                                    x, q, v, w, rot, i);
            } else if (kMode != kTaskStep) {
                obs_torso(rot, v, w, row);
                const double heading = atan2(rot.m[1][0], rot.m[0][0]);
                ts.head_c[lane] = cos(heading);
                ts.head_s[lane] = sin(heading);
            }
        } else if (kMode != kTaskStep) {
            if (role == 2) {
                ts.frame[lane] = height_frame(P, W, i, x, q);
                for (int l = 0; l < kNumLegs; ++l)
                    row[kHeightsAt + l] = obs_value(contact_of(M, ts.sph[lane], l));
            } else {
                for (int j = 0; j < kNumJoints; ++j)  // the action as the step stores it
                    obs_joint(P, j, (double)jr[j * kJointRec + 1], (double)jr[j * kJointRec + 2],
                              kMode == kTaskObserve ? (double)ts.prev[lane][j]
                                                    : (double)(float)clip_action(ts.action[lane][j]),
                              row);
            }
        }
    } else if (role == 0) {
        ts.done[lane] = 0;
    }
    __syncthreads();
    if (kMode != kTaskObserve)
        for (int t = tid; t < kTaskWorlds * kNumJoints; t += kTaskThreads) {
            const int k = t / kNumJoints, c = t % kNumJoints, w = ts.world[k];
            if (w >= 0)
                S.prev_action[(size_t)w * kNumJoints + c] = (float)clip_action(ts.action[k][c]);
        }
    if (kMode == kTaskStep)
        return;
    if (role == 1 && i >= 0)
        obs_target(ts.head_c[lane], ts.head_s[lane], S.target[2 * i] - x.x, S.target[2 * i + 1] - x.y, ts.row[lane]);
    // the heights: a warp per world, a lane's five samples (the last of some
    // lanes is none) side by side
    constexpr int kEachLane = (kNumOffsets + 31) / 32;
    double fo[kEachLane], lo[kEachLane];
#pragma unroll
    for (int u = 0; u < kEachLane; ++u) {
        const int m = lane + 32 * u < kNumOffsets ? lane + 32 * u : kNumOffsets - 1;
        fo[u] = ts.off[m][0];
        lo[u] = ts.off[m][1];
    }
#pragma unroll 1
    for (int k = role; k < kTaskWorlds; k += kTaskThreads / 32) {
        if (ts.world[k] < 0)
            continue;
        const HeightFrame<R> f = ts.frame[k];
        float* dst = O.obs + (size_t)ts.world[k] * kObsSize + kHeightsAt + lane;
        double h[kEachLane];
#pragma unroll
        for (int u = 0; u < kEachLane; ++u)
            h[u] = sample_height(W, f, fo[u], lo[u]);
#pragma unroll
        for (int u = 0; u < kEachLane; ++u)
            if (lane + 32 * u < kNumOffsets)
                dst[32 * u] = height_value(f, h[u]);
    }
    __syncthreads();
    for (int t = tid; t < kTaskWorlds * (kHeightsAt + kNumLegs); t += kTaskThreads) {
        const int k = t / (kHeightsAt + kNumLegs), c = t % (kHeightsAt + kNumLegs);
        if (ts.world[k] >= 0)
            O.obs[(size_t)ts.world[k] * kObsSize + (c < kHeightsAt ? c : c + kNumOffsets)] = ts.row[k][c];
    }
    __syncthreads();
    if (kMode == kTaskStepObs && O.terminal_obs) {
        // the ended worlds' rows, a warp each
        for (int k = role; k < kTaskWorlds; k += kTaskThreads / 32)
            if (ts.done[k]) {
                const size_t at = (size_t)ts.world[k] * kObsSize;
                for (int c = lane; c < kObsSize; c += 32)
                    O.terminal_obs[at + c] = O.obs[at + c];
            }
        __syncthreads();
    }
}

// Worlds first + k (or ids[k]; neither: k) for k < count.
template <class R, int kMode>
__global__ void __launch_bounds__(kTaskThreads)
k_task(const __grid_constant__ DevModel<R> M, Worlds<R> W, const __grid_constant__ TaskParams P, TaskState S,
       TaskOut O, const float* __restrict__ actions, int first, int count, const int* __restrict__ ids)
{
    __shared__ TaskSmem<R> ts;
    const int k = blockIdx.x * kTaskWorlds + (threadIdx.x & 31);
    task_group<R, kMode>(ts, M, W, P, S, O, actions, k < count ? (ids ? ids[k] : first + k) : -1);
}

// ---------------------------------------------------------------------------
// cooperative reset (csrc/arc_sim.c:88-110, csrc/arc_terrain.c:35-71): a CTA
// of four warps resets one world at a time. Warp 0 draws the world's RNG
// stream (each lane one slice) into shared memory while the others tabulate
// the lattice coordinates; the warps build the terrain in blocks of 32 x 8
// cells, a lane walking down eight cells of a column, while warp 0 first
// turns the joints (a lane per leg), which needs no ground; then the bodies
// are placed on the ground, and the warps share the task state, the
// checkpoint and the observation.
//
// In a control step a few worlds end and the step waits for the slowest of
// them, so one world's latency counts as much as the throughput of a whole
// batch. One warp per world spent 200 us on a world: 128 columns a lane with
// both noises' four lattice values and two FP64 divisions each, 143 heights
// and the stance in one lane. Here a thread walks down its column of cells
// and keeps the two x-interpolations of each noise until the lattice row
// changes (3 FP64 operations a noise and cell instead of 10), the division by
// the constant step is a multiplication with a correcting FMA pair, and
// no lane is left with more than a leg's joints or the checkpoint. (Code that
// one lane runs once costs most in fetching it: the task state and
// observation of a new world by one thread took 46k cycles.) The reset of
// the 470 worlds that end in a step of 65,536: 217 -> 33 us; of 26 in one of
// 4,096: 200 -> 26 us; of 16,384 worlds at once 2,001 -> 514 us (268 MB of
// terrain written: 41 us at the copy rate), bound by instruction issue (57 %
// of cycles) and the barriers between the phases.

constexpr int kResetThreads = 128;
constexpr int kResetWarps = kResetThreads / 32;
constexpr int kResetPerSm = 8;                                   // 26 KB of shared memory each
constexpr int kLat1 = (kGridMax / 8 + 2) * (kGridMax / 8 + 2);   // 100
constexpr int kLat2 = (kGridMax / 3 + 2) * (kGridMax / 3 + 2);   // 529
constexpr int kMaxDraws = kLat1 + kLat2 + kGridMax * kGridMax + kMaxJoints + 1;
static_assert(kMaxDraws <= 32 * kSlice, "a world's draws fit 32 slices");

struct ResetSmem {
    double lat[kLat1 + kLat2];
    // lattice coordinates of column index i for the two spacings (8, 3):
    // integer part and smoothed fraction (csrc/arc_terrain.c:41-45)
    double frac[2][kGridMax];
    int whole[2][kGridMax];
    uint32_t draw[kMaxDraws];       // the raw draws: lattices, jitter, stance noise and yaw
    double top[kResetWarps];        // highest column under the robot, per warp
    unsigned long long under;       // columns (of either axis) under the robot
    int outside;                    // the robot's footprint leaves the grid
    int next;                       // the next block of cells
    uint32_t seed;
    unsigned char rows[kSkipRows];
    double angle[kMaxJoints];
    V3<double> up[kMaxJoints], down[kMaxJoints];  // parent -> joint, joint -> child, in the world
    V3<double> x[kMaxBodies];
    Q4<double> q[kMaxBodies];
};

// The generator's arithmetic is written with explicitly rounded FP64
// operations (no FMA contraction): the quantisation to 0.03 m steps and the
// base shift must see the reference's roundings bit for bit
// (csrc/arc_terrain.c:84-123 evaluates each operation separately).
__device__ __forceinline__ double smooth(double t)
{
    return __dmul_rn(__dmul_rn(t, t), __dsub_rn(3.0, __dmul_rn(2.0, t)));
}

__device__ __forceinline__ void lattice_coord(int spacing, int i, int& g, double& t)
{
    const double f = __ddiv_rn((double)i, (double)spacing);
    g = (int)f;
    t = smooth(__dsub_rn(f, (double)g));
}

__device__ __forceinline__ double noise_at(const double* lat, int m, const double* frac, const int* whole, int ix,
                                           int iy)
{
    const int gx = whole[ix], gy = whole[iy];
    const double tx = frac[ix], ty = frac[iy];
    double a = lat[gx + gy * m], b = lat[gx + 1 + gy * m];
    double c = lat[gx + (gy + 1) * m], d = lat[gx + 1 + (gy + 1) * m];
    double top = __dadd_rn(a, __dmul_rn(__dsub_rn(b, a), tx));
    double bot = __dadd_rn(c, __dmul_rn(__dsub_rn(d, c), tx));
    return __dadd_rn(__dmul_rn(top, __dsub_rn(1.0, ty)), __dmul_rn(bot, ty));
}

// one column: hills + bumps + jitter, quantised (csrc/arc_terrain.c:93-118)
__device__ __forceinline__ double column_height(const ResetSmem& sm, const double* lat1, int m1, const double* lat2,
                                                int m2, int ix, int iy, double amp1, double amp2, double ampj,
                                                uint32_t draw)
{
    double v = __dadd_rn(0.0, __dmul_rn(amp1, noise_at(lat1, m1, sm.frac[0], sm.whole[0], ix, iy)));
    v = __dadd_rn(v, __dmul_rn(amp2, noise_at(lat2, m2, sm.frac[1], sm.whole[1], ix, iy)));
    const double u = __dmul_rn((double)draw, 1.0 / 4294967296.0);
    const double jitter = __dadd_rn(-1.0, __dmul_rn(2.0, u));
    const double hj = __dadd_rn(v, __dmul_rn(ampj, jitter));
    return __dmul_rn(0.03, floor(__dadd_rn(__ddiv_rn(hj, 0.03), 0.5)));
}

__device__ __forceinline__ unsigned long long scan_cells(double reach, double step, double o, double cell, int n,
                                                         bool& outside)
{
    unsigned long long mask = 0;
    for (double x = -reach; x <= reach; x += step) {
        double f = floor((x - o) / cell);
        if (f >= 0.0 && f < n)
            mask |= 1ull << (int)f;
        else
            outside = true;
    }
    return mask;
}

// A lattice's interpolation along x at row gy, and between two rows: the
// operations of noise_at.
__device__ __forceinline__ double noise_row(const double* lat, int m, int gy, double tx)
{
    const double a = lat[gy * m], b = lat[gy * m + 1];
    return __dadd_rn(a, __dmul_rn(__dsub_rn(b, a), tx));
}
__device__ __forceinline__ double noise_between(double top, double bot, double ty)
{
    return __dadd_rn(__dmul_rn(top, __dsub_rn(1.0, ty)), __dmul_rn(bot, ty));
}

// Forward kinematics of joints j0 .. j1 - 1, whose parents are turned
// (csrc/arc_phys.c:749-782, with the stance noise of csrc/arc_sim.c:99-103):
// everything but the positions, which wait for the ground.
__device__ __forceinline__ void turn_joints(ResetSmem& sm, const ResetModel& RM, const uint32_t* draw, int j0, int j1)
{
#pragma unroll 1
    for (int j = j0; j < j1; ++j) {
        double a = RM.default_angles[j] + range_of(draw[j], -0.1, 0.1);
        a = a < RM.lo[j] ? RM.lo[j] : (a > RM.hi[j] ? RM.hi[j] : a);
        sm.angle[j] = a;
        const int p = RM.parent[j];
        const Q4<double> qp = p >= 0 ? sm.q[p] : q_identity<double>();
        sm.up[j] = qrotate(qp, RM.r1[j]);
        const double s = sin(0.5 * a), ca = cos(0.5 * a);
        const Q4<double> qa{ca, RM.a1[j].x * s, RM.a1[j].y * s, RM.a1[j].z * s};
        const Q4<double> qc = qnormalize(qmul(qp, qmul(qa, RM.q_rel0[j])));
        sm.q[RM.child[j]] = qc;
        sm.down[j] = qrotate(qc, RM.r2[j]);
    }
}

__device__ __forceinline__ void place_joints(ResetSmem& sm, const ResetModel& RM, int j0, int j1)
{
    for (int j = j0; j < j1; ++j) {
        const int p = RM.parent[j];
        const V3<double> anchor = (p >= 0 ? sm.x[p] : V3<double>{0.0, 0.0, 0.0}) + sm.up[j];
        sm.x[RM.child[j]] = anchor - sm.down[j];
    }
}

// Resets world i; called by all kResetThreads threads of a CTA. When it
// returns every thread has passed a barrier after the world's last write.
template <class R>
__device__ __forceinline__ void reset_world(ResetSmem& sm, const ResetModel& RM, const Worlds<R>& W,
                                            TerrainGeom<R>* tg, TerrainGeomD* tgd, int i, uint32_t seed, double diff,
                                            int n, double cell)
{
    const int tid = threadIdx.x, lane = tid & 31;
    n = n < kGridMax ? n : kGridMax;
    const bool rough = diff > 0.0;
    const int m1 = n / 8 + 2, m2 = n / 3 + 2;
    const int L = rough ? m1 * m1 + m2 * m2 : 0;
    const int J = rough ? n * n : 0;
    R* h = W.th + W.toff[i];
    if (!terrain_column_ok(W, i, (long long)n * n - 1, kCheckTerrainWrite))
        return;  // the whole CTA: n and the slice are the world's
    TerrainGeomD g;
    g.nx = g.ny = n;
    g.cell = cell;
    g.ox = -0.5 * n * cell;
    g.oy = -0.5 * n * cell;
    g.outside = -100.0;
    if (tid < 32) {
        const int total = L + J + RM.nj + 1;
        const int first = lane * kSlice, last = first + kSlice < total ? first + kSlice : total;
        Xorshift rng;
        rng.seed(seed);
        rng_to_slice(rng, lane, sm.rows);
        for (int k = first; k < last; ++k)
            sm.draw[k] = rng.next();
    } else {
        for (int c = tid - 32; c < 2 * kGridMax; c += kResetThreads - 32)
            lattice_coord(c < kGridMax ? 8 : 3, c % kGridMax, sm.whole[c / kGridMax][c % kGridMax],
                          sm.frac[c / kGridMax][c % kGridMax]);
        if (tid == 32) {
            // the grid is square and centred: x and y scan the same columns
            bool out = false;
            sm.under = scan_cells(RM.footprint + 0.1, 0.5 * cell, g.ox, cell, n, out);
            sm.outside = out;
            sm.next = 0;
            tgd[i] = g;
            tg[i] = TerrainGeom<R>{n, n, (R)g.cell, (R)g.ox, (R)g.oy, (R)g.outside};
        }
    }
    __syncthreads();
    for (int k = tid; k < L; k += kResetThreads)
        sm.lat[k] = __fma_rn((double)sm.draw[k], 2.0 / 4294967296.0, -1.0);  // -1 + 2 u: the product is exact
    __syncthreads();

    // the joints, a lane per leg
    const int lanes = RM.legs > 0 ? RM.legs : 1, per = RM.nj / lanes;
    if (tid < 32) {
        const uint32_t* draw = sm.draw + L + J;
        if (lane == 0) {
            const double yaw = range_of(draw[RM.nj], -kPi, kPi);
            const double sy = sin(0.5 * yaw), cyw = cos(0.5 * yaw);
            sm.q[0] = qnormalize(Q4<double>{cyw, 0.0 * sy, 0.0 * sy, 1.0 * sy});
        }
        __syncwarp();
        if (lane < lanes)
            turn_joints(sm, RM, draw, lane * per, (lane + 1) * per);
        __syncwarp();
    }
    const unsigned long long under = sm.under;
    double gmax = rough ? -1e300 : 0.0;
    if (!rough) {
        for (int c = tid; c < n * n; c += kResetThreads)
            h[c] = R(0);
    } else {
        const double amp1 = __dmul_rn(0.45, diff), amp2 = __dmul_rn(0.12, diff), ampj = __dmul_rn(0.06, diff);
        const double* lat1 = sm.lat;
        const double* lat2 = sm.lat + m1 * m1;
        const uint32_t* draw = sm.draw + L;
        const double f0x = floor((0.0 - g.ox) / g.cell), f0y = floor((0.0 - g.oy) / g.cell);
        double base = g.outside;
        if (f0x >= 0.0 && f0y >= 0.0 && f0x < n && f0y < n) {
            const int ix = (int)f0x, iy = (int)f0y;
            base = column_height(sm, lat1, m1, lat2, m2, ix, iy, amp1, amp2, ampj, draw[ix + iy * n]);
        }
        // blocks of 32 x 8 cells (two of 16 x 4 for at most 16 columns) to the
        // warps as they come: a lane walks down its column. The rows of a
        // block share the coarse noise's lattice row.
        const int wide = n > 16 ? 32 : 16, rows = n > 16 ? 8 : 4, over = (n + wide - 1) / wide;
        const int blocks = over * ((n + 7) / 8);
        for (;;) {
            int block = 0;
            if (lane == 0)
                block = atomicAdd(&sm.next, 1);
            block = __shfl_sync(0xffffffffu, block, 0);
            if (block >= blocks)
                break;
            const int ix = block % over * wide + (lane & (wide - 1));
            const int iy0 = block / over * 8 + (n > 16 ? 0 : lane / 16 * 4);
            if (ix >= n || iy0 >= n)
                continue;
            const double* c1 = lat1 + sm.whole[0][ix];
            const double* c2 = lat2 + sm.whole[1][ix];
            const double tx1 = sm.frac[0][ix], tx2 = sm.frac[1][ix];
            const int g1 = sm.whole[0][iy0];
            const double top1 = noise_row(c1, m1, g1, tx1), bot1 = noise_row(c1, m1, g1 + 1, tx1);
            int g2 = sm.whole[1][iy0];
            double top2 = noise_row(c2, m2, g2, tx2), bot2 = noise_row(c2, m2, g2 + 1, tx2);
            const uint32_t below = ((under >> ix) & 1) ? (uint32_t)(under >> iy0) : 0u;
            const int count = n - iy0 < rows ? n - iy0 : rows;
            const uint32_t* dr = draw + ix + iy0 * n;
            R* col = h + ix + iy0 * n;
#pragma unroll 1
            for (int k = 0; k < count; ++k, dr += n, col += n) {
                if (sm.whole[1][iy0 + k] != g2) {
                    ++g2;
                    top2 = bot2;
                    bot2 = noise_row(c2, m2, g2 + 1, tx2);
                }
                // column_height, operation by operation
                const double v = __dadd_rn(__dmul_rn(amp1, noise_between(top1, bot1, sm.frac[0][iy0 + k])),
                                           __dmul_rn(amp2, noise_between(top2, bot2, sm.frac[1][iy0 + k])));
                const double jitter = __fma_rn((double)*dr, 2.0 / 4294967296.0, -1.0);
                const double hj = __dadd_rn(v, __dmul_rn(ampj, jitter));
                const double top = __dmul_rn(0.03, floor(__dadd_rn(divide(hj, 0.03, 1.0 / 0.03), 0.5)));
                const double hf = __dsub_rn(top, base);
                *col = (R)hf;
                if ((below >> k) & 1)
                    gmax = gmax > hf ? gmax : hf;
            }
        }
        for (int off = 16; off > 0; off >>= 1) {
            const double o = __shfl_xor_sync(0xffffffffu, gmax, off);
            gmax = gmax > o ? gmax : o;
        }
    }
    if (lane == 0)
        sm.top[tid / 32] = gmax;
    __syncthreads();

    R* rec = W.rec + (size_t)i * W.stride;
    R* sr = rec + W.off_sphere;
    R* jr = rec + W.off_joint;
    if (tid < 32) {
        // on the ground (csrc/arc_sim.c:104-109)
        double ground = sm.outside ? g.outside : -1e30;
        if (under)
            for (int w = 0; w < kResetWarps; ++w)
                ground = ground > sm.top[w] ? ground : sm.top[w];
        if (lane == 0)
            sm.x[0] = V3<double>{0.0, 0.0, ground + RM.stand_height + 0.03};
        __syncwarp();
        if (lane < lanes)
            place_joints(sm, RM, lane * per, (lane + 1) * per);
    } else {
        for (int c = tid - 32; c < RM.ns * kSphereRec; c += kResetThreads - 32)
            sr[c] = R(0);
        for (int c = tid - 32; c < RM.ns; c += kResetThreads - 32)
            W.sph[(size_t)i * RM.ns + c] = 0;
        for (int j = tid - 32; j < RM.nj; j += kResetThreads - 32) {
            jr[j * kJointRec + 0] = (R)sm.angle[j];
            jr[j * kJointRec + 1] = (R)sm.angle[j];
            jr[j * kJointRec + 2] = R(0);
            jr[j * kJointRec + 3] = R(0);
        }
        if (tid == 32) {
            W.unstable[i] = 0;
            W.time[i] = 0.0;
        }
    }
    __syncthreads();
    for (int b = tid; b < RM.nb; b += kResetThreads) {
        R* r = rec + b * kBodyRec;
        const V3<double> x = sm.x[b];
        const Q4<double> q = sm.q[b];
        r[0] = (R)x.x; r[1] = (R)x.y; r[2] = (R)x.z;
        r[3] = (R)q.w; r[4] = (R)q.x; r[5] = (R)q.y; r[6] = (R)q.z;
        for (int c = 7; c < 13; ++c)
            r[c] = R(0);
    }
    __syncthreads();
}

template <class R>
__global__ void __launch_bounds__(kResetThreads, kResetPerSm)
k_reset(const __grid_constant__ ResetModel RM, Worlds<R> W, TerrainGeom<R>* tg, TerrainGeomD* tgd,
        const int* __restrict__ ids, int n_ids, const unsigned* __restrict__ seeds,
        const double* __restrict__ difficulty, const int* __restrict__ grid_of, double cell)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ResetSmem& sm = *reinterpret_cast<ResetSmem*>(smem_raw);
    for (int k = blockIdx.x; k < n_ids; k += gridDim.x) {
        const int i = ids[k];
        reset_world(sm, RM, W, tg, tgd, i, seeds[k], difficulty[k], grid_of ? grid_of[i] : kGridMax, cell);
    }
}

// ArcTask.reset (arc/task.py:113-125) + the observation of the new episode,
// by the kResetThreads threads of a CTA (compiled once, as task_step_world).
template <class R>
__device__ __noinline__ void task_reset_world(ResetSmem& sm, const DevModel<R>& M, const ResetModel& RM, const Worlds<R>& W,
                                 TerrainGeom<R>* tg, TerrainGeomD* tgd, const int* __restrict__ grid_of, double cell,
                                 const TaskParams& P, const TaskState& S, float* obs, int i)
{
    const int tid = threadIdx.x;
    if (tid == 0) {
        const unsigned e = S.episode[i]++;
        sm.seed = (uint32_t)stream_u64(P.seed, key_of(S, i), 2u, e);
        S.difficulty[i] = S.level[i];
    }
    __syncthreads();
    reset_world(sm, RM, W, tg, tgd, i, sm.seed, S.level[i], grid_of ? grid_of[i] : kGridMax, cell);
    // warp 0: the checkpoint; warp 1: the task state and the rest of the row
    // but the heights; warps 2, 3: the heights
    float* row = obs ? obs + (size_t)i * kObsSize : nullptr;
    const R* b0 = W.rec + (size_t)i * W.stride;
    const V3<double> x{(double)b0[0], (double)b0[1], (double)b0[2]};
    const Q4<double> q{(double)b0[3], (double)b0[4], (double)b0[5], (double)b0[6]};
    if (tid < 32) {
        const M3<double> rot = m3_from_quat(q);
        if (tid == 0)
            place_target(P, W, S, i, x, rot);
        __syncwarp();
        if (tid == 0 && row) {
            const double heading = atan2(rot.m[1][0], rot.m[0][0]);
            obs_target(cos(heading), sin(heading), S.target[2 * i] - x.x, S.target[2 * i + 1] - x.y, row);
        }
    } else if (tid < 64) {
        const int j = tid - 32;
        const R* jr = b0 + W.off_joint;
        if (j < kNumJoints) {
            S.prev_action[(size_t)i * kNumJoints + j] = 0.0f;
            if (row)
                obs_joint(P, j, (double)jr[j * kJointRec + 1], (double)jr[j * kJointRec + 2], 0.0, row);
        } else if (j < kNumJoints + kNumLegs) {
            if (row)  // no sphere has touched yet
                row[kHeightsAt + kNumOffsets + j - kNumJoints] = 0.0f;
        } else if (j == kNumJoints + kNumLegs) {
            S.torso_steps[i] = 0;
            S.steps[i] = 0;
            S.checkpoints[i] = 0;
            if (row)
                obs_torso(m3_from_quat(q), V3<double>{(double)b0[7], (double)b0[8], (double)b0[9]},
                          V3<double>{(double)b0[10], (double)b0[11], (double)b0[12]}, row);
        }
    } else if (row) {
        const HeightFrame<R> f = height_frame(P, W, i, x, q);
        for (int m = tid - 64; m < kNumOffsets; m += kResetThreads - 64)
            row[kHeightsAt + m] = height_value(f, sample_height(W, f, P.offsets[m][0], P.offsets[m][1]));
    }
    __syncthreads();  // the next world's reset reuses sm
}

template <class R>
__global__ void __launch_bounds__(kResetThreads, kResetPerSm)
k_task_reset(const __grid_constant__ DevModel<R> M, const __grid_constant__ ResetModel RM, Worlds<R> W,
             TerrainGeom<R>* tg, TerrainGeomD* tgd, const int* __restrict__ grid_of, double cell,
             const __grid_constant__ TaskParams P, TaskState S, float* obs, const int* __restrict__ ids,
             const int* __restrict__ count_dev, int max_n)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ResetSmem& sm = *reinterpret_cast<ResetSmem*>(smem_raw);
    const int n = count_dev ? min(*count_dev, max_n) : max_n;
    for (int k = blockIdx.x; k < n; k += gridDim.x)
        task_reset_world(sm, M, RM, W, tg, tgd, grid_of, cell, P, S, obs, ids[k]);
}

template <class R>
__global__ void k_task_set_targets(Worlds<R> W, const __grid_constant__ TaskParams P, TaskState S,
                                   const int* __restrict__ ids, const double* __restrict__ xy, int n)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n)
        return;
    const int i = ids[k];
    const R* rec = W.rec + (size_t)i * W.stride;
    V3<double> pos{(double)rec[0], (double)rec[1], (double)rec[2]};
    Q4<double> q{(double)rec[3], (double)rec[4], (double)rec[5], (double)rec[6]};
    M3<double> rot = m3_from_quat(q);
    const double tx = xy[2 * k], ty = xy[2 * k + 1];
    S.target[2 * i] = tx;
    S.target[2 * i + 1] = ty;
    S.target_z[i] = height_at(W, i, tx, ty);
    const double dx = tx - pos.x, dy = ty - pos.y;
    S.prev_dist[i] = sqrt(dx * dx + dy * dy);
    S.prev_gaze[i] = gaze_error(rot, pos, S.target + 2 * i);
    S.in_view[i] = S.prev_gaze[i] < P.fov_rad;
}

// A warp per world, a lane per column (arc_env_get_task_state).
__global__ void __launch_bounds__(256)
k_task_rows(TaskState S, TaskOut O, const int* __restrict__ ids, int first, int n, double* __restrict__ rows,
            float* __restrict__ reward, unsigned char* __restrict__ bytes)
{
    const int k = (blockIdx.x * 256 + threadIdx.x) / 32, lane = threadIdx.x & 31;
    if (k >= n)
        return;
    const int i = ids ? ids[k] : first + k;
    double v = 0.0;
    switch (lane) {
    case 0: case 1: v = S.target[2 * i + lane]; break;
    case 2: v = S.target_z[i]; break;
    case 3: v = S.prev_dist[i]; break;
    case 4: v = S.prev_gaze[i]; break;
    case 17: v = S.torso_steps[i]; break;
    case 18: v = S.steps[i]; break;
    case 19: v = S.checkpoints[i]; break;
    case 20: v = S.level[i]; break;
    case 21: v = S.difficulty[i]; break;
    case 22: v = S.in_view[i]; break;
    case 23: v = S.episode[i]; break;
    case 24: v = S.draws[i]; break;
    default:
        if (lane < 17)
            v = S.prev_action[(size_t)i * 12 + lane - 5];
    }
    if (lane < 25)
        rows[(size_t)k * 25 + lane] = v;
    if (!reward)
        return;
    if (lane == 25)
        reward[k] = O.reward[i];
    else if (lane == 26)
        bytes[k] = O.terminated[i];
    else if (lane == 27)
        bytes[(size_t)n + k] = O.truncated[i];
    else if (lane == 28)
        bytes[2 * (size_t)n + k] = (unsigned char)O.cause[i];
}

// ---------------------------------------------------------------------------
// The warp-per-leg step (FP32, the quadruped) and, fused with it, the task
// layer of ArcVecEnv.step_wait (arc/env.py:99-117). One kernel template
// serves every form, instantiated per form:
//   kPhysics      the step alone (arc_sim_step, the separate env step, tiles
//                 of substeps);
//   kWithTask     each CTA steps a group of 32 worlds, then, before its next
//                 group, runs the task layer on them (task_group); the ended
//                 worlds go to the ended-world list, which a separate reset
//                 launch then takes;
//   kWithResets   the same, and the group's ended worlds are reset in the
//                 kernel too, one after the other by the whole CTA.
// The task functions are compiled once (not inlined) and called both from
// the fused forms and from the separate task kernels, so their outputs do
// not depend on the form. The physics is inlined into each instantiation:
// the physics-only one then holds no task code and gets the registers it needs
// without spills (127; one kernel for every form took 128 with spills and
// stepped 6 % slower); the fused instantiations compile the same
// physics source in another context and agree with it to FP32 rounding
// rather than bit for bit, and are 9-10 % slower (65,536 worlds, policy
// included: 3.03 ms, 3.34 with the task, 3.31 with the resets too). The
// ended-world list is filled in completion order, as the separate task kernel
// fills it.
static_assert(kResetThreads == wl::kThreads, "the fused form's CTA resets worlds");
enum : int { kPhysics = 0, kWithTask = 1, kWithResets = 2 };

struct ControlSmem {
    union {
        wl::Smem step;
        TaskSmem<float> task;  // after the group's step
        ResetSmem reset;       // after the task layer
    };
    int ended[wl::kWorlds];  // worlds of the group whose episode ended
    int n_ended;
    int next;  // the next group from the work queue
};

template <int kMode>
__global__ void __launch_bounds__(wl::kThreads, 4)
k_control_step(const __grid_constant__ DevModel<float> M, const __grid_constant__ ResetModel RM, Worlds<float> W,
               TerrainGeom<float>* tg, TerrainGeomD* tgd, const int* __restrict__ grid_of, double cell,
               const __grid_constant__ TaskParams P, TaskState S, TaskOut O, Actuation A,
               float* __restrict__ spill, int spill_per_lane, int lane_cap, const int* __restrict__ ids, int n_items,
               int* queue, int sub0, int sub1, float* __restrict__ tile_q, int per_group, int list)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ControlSmem& cs = *reinterpret_cast<ControlSmem*>(smem_raw);
    const int tid = threadIdx.x, leg = tid / wl::kWorlds, j = tid % wl::kWorlds;
    const int n_groups = (n_items + per_group - 1) / per_group;
    // with a queue every group, the first included, is taken from it: a CTA
    // that becomes resident only when others leave finds the queue empty
    // instead of holding back a group of its own
    int first = blockIdx.x;
    if (queue) {
        if (tid == 0)
            cs.next = atomicAdd(queue, 1);
        __syncthreads();
        first = cs.next;
    }
#pragma unroll 1
    for (int group = first; group < n_groups;) {
        wl::step_group(wl::CtaSync{}, cs.step, M, W, A, spill, spill_per_lane, lane_cap, ids, n_items,
                       group * per_group, leg, j, sub0, sub1, tile_q, per_group, list);
        if constexpr (kMode != kPhysics) {
            // arc/task.py:155-259
            const int at = group * wl::kWorlds + j, item = at < n_items ? (ids ? ids[at] : at) : -1;
            const int world = item < W.n ? item : -1;
            __syncthreads();  // warp 0 has read the step's shared memory for the last time
            task_group<float, kTaskStepObs>(cs.task, M, W, P, S, O, A.actions32, world);
            if (tid == 0)
                cs.n_ended = 0;
            __syncthreads();
            if (tid < wl::kWorlds && cs.task.done[j])
                cs.ended[atomicAdd(&cs.n_ended, 1)] = world;
            if constexpr (kMode == kWithResets) {
                __syncthreads();
#pragma unroll 1
                for (int e = 0; e < cs.n_ended; ++e)
                    task_reset_world(cs.reset, M, RM, W, tg, tgd, grid_of, cell, P, S, O.obs, cs.ended[e]);
            }
        }
        if (!queue)
            break;
        __syncthreads();  // this group's task and reset work is done with the shared memory
        if (tid == 0)
            cs.next = atomicAdd(queue, 1);
        __syncthreads();
        group = cs.next;
    }
    if (queue) {
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            if (atomicAdd(queue + 1, 1) == (int)gridDim.x - 1) {
                queue[0] = 0;
                queue[1] = 0;
                __threadfence();
            }
        }
    }
}

// The physics of many groups, in CTAs of four that run aligned.
__global__ void __launch_bounds__(wl::kThreads * wl::kAligned, 1)
k_step_aligned(const __grid_constant__ DevModel<float> M, Worlds<float> W, Actuation A, float* __restrict__ spill,
               int spill_per_lane, int lane_cap, const int* __restrict__ ids, int n_items, int* queue, int sub0,
               int sub1, float* __restrict__ tile_q, int list)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    wl::step_aligned(*reinterpret_cast<wl::AlignedSmem*>(smem_raw), M, W, A, spill, spill_per_lane, lane_cap, ids,
                     n_items, queue, sub0, sub1, tile_q, list);
}

// The physics of few groups, each split over eight warps.
__global__ void __launch_bounds__(2 * wl::kThreads, 2)
k_step_split(const __grid_constant__ DevModel<float> M, Worlds<float> W, Actuation A, float* __restrict__ spill,
             int spill_per_lane, int lane_cap, const int* __restrict__ ids, int n_items, int per_group)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    wl::step_split(*reinterpret_cast<wl::SplitSmem*>(smem_raw), M, W, A, spill, spill_per_lane, lane_cap, ids, n_items,
                   per_group);
}

// One launch of k_control_step<kMode> over the n_items worlds ids[0 .. n_items).
template <int kMode>
cudaError_t launch_form(const DevModel<float>& M, const ResetModel& RM, const Worlds<float>& W,
                        TerrainGeom<float>* tg, TerrainGeomD* tgd, const int* grid_of, double cell,
                        const TaskParams& P, const TaskState& S, const TaskOut& O, const Actuation& A, float* spill,
                        int spill_per_lane, int lane_cap, const int* ids, int n_items, int* queue, int sub0, int sub1,
                        float* tile_q, cudaStream_t stream, bool alone)
{
    const int smem = (int)sizeof(ControlSmem);
    // per device and form: the shared-memory attribute, and how many CTAs are
    // resident at once (the work queue's wave)
    static std::atomic<unsigned long long> configured{0};
    static int resident[64] = {}, sm_count[64] = {};
    cudaError_t e = once_per_device(configured, [&](int dev) {
        cudaError_t r = cudaFuncSetAttribute(k_control_step<kMode>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (r == cudaSuccess && kMode == kPhysics)
            r = cudaFuncSetAttribute(k_step_aligned, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(wl::AlignedSmem));
        if (r == cudaSuccess && kMode == kPhysics)
            r = cudaFuncSetAttribute(k_step_split, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(wl::SplitSmem));
        int sms = 0, per_sm = 0;
        if (r == cudaSuccess)
            r = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (r == cudaSuccess)
            r = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_control_step<kMode>, wl::kThreads, smem);
        if (r == cudaSuccess)
            resident[dev] = sms * (per_sm > 0 ? per_sm : 1), sm_count[dev] = sms;
        return r;
    });
    if (e != cudaSuccess)
        return e;
    int dev = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess)
        return e;
    wl::GroupPlan plan = wl::group_plan(n_items, sm_count[dev], alone, queue != nullptr,
                                        wl::splittable(W, lane_cap, sub0, sub1, M.substeps));
    if (kMode != kPhysics)  // the fused forms' task work takes whole groups of 32
        plan = wl::GroupPlan{wl::kWorlds, (n_items + wl::kWorlds - 1) / wl::kWorlds, plan.list, false,
                             false};
    if (plan.split) {
        k_step_split<<<plan.groups, 2 * wl::kThreads, sizeof(wl::SplitSmem), stream>>>(
            M, W, A, spill, spill_per_lane, lane_cap, ids, n_items, plan.per_group);
        return cudaGetLastError();
    }
    if (plan.aligned) {
        k_step_aligned<<<sm_count[dev], wl::kThreads * wl::kAligned, sizeof(wl::AlignedSmem), stream>>>(
            M, W, A, spill, spill_per_lane, lane_cap, ids, n_items, queue, sub0, sub1, tile_q, plan.list);
        return cudaGetLastError();
    }
    // with a queue, one wave of resident CTAs
    const int grid = queue && plan.groups > resident[dev] ? resident[dev] : plan.groups;
    k_control_step<kMode><<<grid, wl::kThreads, smem, stream>>>(M, RM, W, tg, tgd, grid_of, cell, P, S, O, A, spill,
                                                                spill_per_lane, lane_cap, ids, n_items, queue, sub0,
                                                                sub1, tile_q, plan.per_group, plan.list);
    return cudaGetLastError();
}

cudaError_t control_launch(const DevModel<float>& M, const ResetModel& RM, const Worlds<float>& W,
                           TerrainGeom<float>* tg, TerrainGeomD* tgd, const int* grid_of, double cell,
                           const TaskParams& P, const TaskState& S, const TaskOut& O, const Actuation& A,
                           float* spill, int spill_per_lane, int lane_cap, const int* ids, int n_items, int* queue,
                           int mode, int sub0, int sub1, float* tile_q, cudaStream_t stream, bool alone)
{
    switch (mode) {
    case kPhysics:
        return launch_form<kPhysics>(M, RM, W, tg, tgd, grid_of, cell, P, S, O, A, spill, spill_per_lane, lane_cap,
                                     ids, n_items, queue, sub0, sub1, tile_q, stream, alone);
    case kWithTask:
        return launch_form<kWithTask>(M, RM, W, tg, tgd, grid_of, cell, P, S, O, A, spill, spill_per_lane, lane_cap,
                                      ids, n_items, queue, sub0, sub1, tile_q, stream, alone);
    case kWithResets:
        return launch_form<kWithResets>(M, RM, W, tg, tgd, grid_of, cell, P, S, O, A, spill, spill_per_lane,
                                        lane_cap, ids, n_items, queue, sub0, sub1, tile_q, stream, alone);
    default:
        return cudaErrorInvalidValue;
    }
}

template <class R>
__global__ void k_env_admit(TaskState S, const int* __restrict__ ids, const double* __restrict__ difficulty,
                            const unsigned* __restrict__ keys, int n)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n)
        return;
    const int i = ids[k];
    S.level[i] = difficulty[k];
    S.difficulty[i] = difficulty[k];
    S.key[i] = keys[k];
    S.episode[i] = 0;
    S.draws[i] = 0;
}

int reset_grid(int n)
{
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int cap = sms * kResetPerSm;
    return n < cap ? (n > 0 ? n : 1) : cap;
}

}  // namespace

template <class R>
cudaError_t launch_task_step(const DevModel<R>& M, const Worlds<R>& W, const TaskParams& P, const TaskState& S,
                             const TaskOut& O, const float* actions, bool write_obs, cudaStream_t stream, int first,
                             int count, const int* ids)
{
    if (count < 0)
        count = W.n - first;
    if (count <= 0 || (!ids && (first < 0 || first + count > W.n)))
        return count == 0 ? cudaSuccess : cudaErrorInvalidValue;
    const int grid = (count + kTaskWorlds - 1) / kTaskWorlds;
    if (write_obs && O.obs)
        k_task<R, kTaskStepObs><<<grid, kTaskThreads, 0, stream>>>(M, W, P, S, O, actions, first, count, ids);
    else
        k_task<R, kTaskStep><<<grid, kTaskThreads, 0, stream>>>(M, W, P, S, O, actions, first, count, ids);
    return cudaGetLastError();
}

template <class R>
cudaError_t launch_task_observe(const DevModel<R>& M, const Worlds<R>& W, const TaskParams& P, const TaskState& S,
                                float* obs, const int* ids, int n_ids, cudaStream_t stream)
{
    if (n_ids <= 0)
        return cudaSuccess;
    TaskOut O{};
    O.obs = obs;
    k_task<R, kTaskObserve><<<(n_ids + kTaskWorlds - 1) / kTaskWorlds, kTaskThreads, 0, stream>>>(
        M, W, P, S, O, nullptr, 0, n_ids, ids);
    return cudaGetLastError();
}

template <class R>
cudaError_t launch_task_reset(const DevModel<R>& M, const ResetModel& RM, const Worlds<R>& W, TerrainGeom<R>* tg,
                              TerrainGeomD* tgd, const int* grid_of, double cell, const TaskParams& P,
                              const TaskState& S, float* obs, const int* ids, const int* count_dev, int max_n,
                              cudaStream_t stream)
{
    if (max_n <= 0)
        return cudaSuccess;
    static std::atomic<unsigned long long> configured{0};
    cudaError_t e = once_per_device(configured, [](int) {
        return cudaFuncSetAttribute(k_task_reset<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ResetSmem));
    });
    if (e != cudaSuccess)
        return e;
    k_task_reset<R><<<reset_grid(max_n), kResetThreads, sizeof(ResetSmem), stream>>>(M, RM, W, tg, tgd, grid_of, cell, P,
                                                                                  S, obs, ids, count_dev, max_n);
    return cudaGetLastError();
}

template <class R>
cudaError_t launch_task_set_targets(const Worlds<R>& W, const TaskParams& P, const TaskState& S, const int* ids,
                                    const double* xy, int n, cudaStream_t stream)
{
    if (n <= 0)
        return cudaSuccess;
    k_task_set_targets<R><<<(n + 127) / 128, 128, 0, stream>>>(W, P, S, ids, xy, n);
    return cudaGetLastError();
}

cudaError_t init_reset_tables(cudaStream_t stream)
{
    k_skip_init<<<32, 128, 0, stream>>>();
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? cudaStreamSynchronize(stream) : e;
}

template <class R>
cudaError_t launch_reset_warp(const ResetModel& RM, const Worlds<R>& W, TerrainGeom<R>* tg, TerrainGeomD* tgd,
                              const int* ids, int n_ids, const unsigned* seeds, const double* difficulty,
                              const int* grid_of, double cell, cudaStream_t stream)
{
    if (n_ids <= 0)
        return cudaSuccess;
    static std::atomic<unsigned long long> configured{0};
    cudaError_t e = once_per_device(configured, [](int) {
        return cudaFuncSetAttribute(k_reset<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ResetSmem));
    });
    if (e != cudaSuccess)
        return e;
    k_reset<R><<<reset_grid(n_ids), kResetThreads, sizeof(ResetSmem), stream>>>(RM, W, tg, tgd, ids, n_ids, seeds,
                                                                                 difficulty, grid_of, cell);
    return cudaGetLastError();
}

template <class R>
cudaError_t launch_env_admit(const DevModel<R>& M, const ResetModel& RM, const Worlds<R>& W, TerrainGeom<R>* tg,
                             TerrainGeomD* tgd, const int* grid_of, double cell, const TaskParams& P,
                             const TaskState& S, float* obs, const int* ids, const double* difficulty,
                             const unsigned* keys, int n, cudaStream_t stream)
{
    if (n <= 0)
        return cudaSuccess;
    if (!S.key)
        return cudaErrorInvalidValue;
    k_env_admit<R><<<(n + 127) / 128, 128, 0, stream>>>(S, ids, difficulty, keys, n);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return e;
    return launch_task_reset<R>(M, RM, W, tg, tgd, grid_of, cell, P, S, obs, ids, nullptr, n, stream);
}

cudaError_t launch_task_rows(const TaskState& S, const TaskOut& O, const int* ids, int first, int n, double* rows,
                             float* reward, unsigned char* bytes, cudaStream_t stream)
{
    if (n <= 0)
        return cudaSuccess;
    k_task_rows<<<(n + 7) / 8, 256, 0, stream>>>(S, O, ids, first, n, rows, reward, bytes);
    return cudaGetLastError();
}

cudaError_t launch_control_step(const DevModel<float>& M, const ResetModel& RM, const Worlds<float>& W,
                                TerrainGeom<float>* tg, TerrainGeomD* tgd, const int* grid_of, double cell,
                                const TaskParams& P, const TaskState& S, const TaskOut& O, const float* actions,
                                float* spill, int spill_per_lane, int lane_cap, const int* ids, int n_items, int* queue,
                                bool resets, cudaStream_t stream, bool alone)
{
    if (W.n <= 0 || n_items <= 0)
        return cudaSuccess;
    if (!M.leaper)
        return cudaErrorInvalidValue;
    return control_launch(M, RM, W, tg, tgd, grid_of, cell, P, S, O, Actuation{nullptr, actions}, spill,
                          spill_per_lane, lane_cap, ids, n_items, queue, resets ? kWithResets : kWithTask, 0,
                          M.substeps, nullptr, stream, alone);
}

cudaError_t launch_step_warps(const DevModel<float>& M, const Worlds<float>& W, const Actuation& A, float* spill,
                              int spill_per_lane, int lane_cap, const int* ids, int n_items, int* queue,
                              cudaStream_t stream, bool alone, int tile, float* tile_q)
{
    if (W.n <= 0 || n_items <= 0)
        return cudaSuccess;
    if (!M.leaper)
        return cudaErrorInvalidValue;
    // the task layer's parameters, which the physics alone does not read
    static const ResetModel RM{};
    static const TaskParams P{};
    if (tile <= 0 || tile >= M.substeps || !tile_q)
        tile = M.substeps;
    for (int sub0 = 0; sub0 < M.substeps; sub0 += tile) {
        const int sub1 = sub0 + tile < M.substeps ? sub0 + tile : M.substeps;
        cudaError_t e = control_launch(M, RM, W, nullptr, nullptr, nullptr, 0.0, P, TaskState{}, TaskOut{}, A, spill,
                                       spill_per_lane, lane_cap, ids, n_items, queue, kPhysics, sub0, sub1, tile_q,
                                       stream, alone);
        if (e != cudaSuccess)
            return e;
    }
    return cudaSuccess;
}

#define ARC_INSTANTIATE_TASK(R)                                                                                    \
    template cudaError_t launch_task_step<R>(const DevModel<R>&, const Worlds<R>&, const TaskParams&,            \
                                             const TaskState&, const TaskOut&, const float*, bool, cudaStream_t, \
                                             int, int, const int*);                                              \
    template cudaError_t launch_task_observe<R>(const DevModel<R>&, const Worlds<R>&, const TaskParams&,         \
                                                const TaskState&, float*, const int*, int, cudaStream_t);        \
    template cudaError_t launch_task_reset<R>(const DevModel<R>&, const ResetModel&, const Worlds<R>&,           \
                                              TerrainGeom<R>*, TerrainGeomD*, const int*, double,                \
                                              const TaskParams&, const TaskState&, float*, const int*,           \
                                              const int*, int, cudaStream_t);                                    \
    template cudaError_t launch_task_set_targets<R>(const Worlds<R>&, const TaskParams&, const TaskState&,       \
                                                    const int*, const double*, int, cudaStream_t);               \
    template cudaError_t launch_env_admit<R>(const DevModel<R>&, const ResetModel&, const Worlds<R>&,            \
                                             TerrainGeom<R>*, TerrainGeomD*, const int*, double, const TaskParams&, \
                                             const TaskState&, float*, const int*, const double*, const unsigned*, \
                                             int, cudaStream_t);                                                  \
    template cudaError_t launch_reset_warp<R>(const ResetModel&, const Worlds<R>&, TerrainGeom<R>*,              \
                                              TerrainGeomD*, const int*, int, const unsigned*, const double*,    \
                                              const int*, double, cudaStream_t);

ARC_INSTANTIATE_TASK(float)
ARC_INSTANTIATE_TASK(double)

}  // namespace arc
