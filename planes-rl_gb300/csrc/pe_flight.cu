// pe_flight.cu -- the 600 Hz 6DOF flight of every (plane, scenario) pair (src/sim.cu:55-212) in the
// reference's arithmetic: panels rotated to the world frame, sums in its 128-thread order.
//
// Mapping.  A block of four warps flies four flights.  A flight's panels are staged once into shared
// memory with the print-warp normal already applied (it is constant over a flight: it depends on the
// panel, the CG shift and the scenario only).  The reference sums panels with 128 threads, panel t on
// thread t % 128, then a shuffle-down tree inside each warp, then a serial sum of the 4 warp totals
// (src/sim.cu:134-176); here warp (k + flight) % 4 of the block stands for the reference's warp k, so
// the short last round of a flight's panels falls on another warp for each of the four.  The sums of
// four flights over a warp go through one transposed exchange along the same tree.
//
// Bound by register reads: a step's 308 FFMA of three registers take two cycles of a scheduler each, its other
// 685 instructions one, 1,300 of the 1,310 cycles measured with 20 flights per SM (issue slots 76 % busy).
// What is not panels is the point of the split: eight lanes hold one flight's integrator, so one warp
// advances the rotation of the block's four flights and another their translation and gusts, other warps
// each step; state and constants stay in shared memory and leave the registers to the panels.  With a warp
// for each flight a step took 1,150 warp instructions, here 990.  Flights of pop x 8, warp per flight ->
// this: 45.9 -> 38.8 ms at 16,384, 6.89 -> 5.58 at 2,048, 2.38 -> 1.60 at 256, 1.59 -> 0.80 at 8.  Pairs of
// panels in f32x2 (740 instructions, FFMA2 of three cycles) gave 39.8, 5.77, 1.96, 0.91; attitude rows as
// uniform operands (by REDUX) 41.3 and 5.91.
//
// Rounding.  The fused operations of the step are spelled out (dot_exact, cross_exact and the like), so
// results do not hang on how the compiler pairs them.
//
// Chunking.  A launch advances flights by at most `step_end - step_begin` steps; flights still
// airborne are appended to the next launch's list and their state is saved (64 B).  The clock
// restarts at every multiple of 600 steps, as the reference's 600-step launches do
// (src/sim.cu:113), whatever launch length is chosen here.
#include <algorithm>

#include "pe_internal.cuh"

namespace pe {

// Per-flight constants held in registers for the whole flight.
struct FlightConst {
    float mass, invmass;
    float I[6];
    float invI[9];
    float air_rho, skin_cf;
    float phase, gust, base_x, base_y;
    vec3 cg;
    float warp_pitch, warp_roll;
};

__device__ __forceinline__ int flight_env_seed(const FlightArgs& a, int p, int s) {
    return (int)((uint32_t)a.seeds[s] + (a.vary ? (uint32_t)p * 7919u : 0u));
}

__device__ __forceinline__ void flight_setup(const FlightArgs& a, int p, int s, FlightConst* fc,
                                             MassProps* pmp_out, Scenario* sc_out) {
    const int env_seed = flight_env_seed(a, p, s);
    Scenario sc;
    scenario_desc(env_seed, &sc);
    MassProps src;
    const float* m = a.plane_mp + (size_t)p * kMpN;
    src.mass = m[0]; src.invmass = m[1]; src.com = mk3(m[2], m[3], m[4]);
    for (int k = 0; k < 6; k++) src.I[k] = m[5 + k];
    for (int k = 0; k < 9; k++) src.invI[k] = m[11 + k];
    MassProps pmp; vec3 cg;
    printed_mass_props(src, sc, &pmp, &cg);
    fc->mass = pmp.mass; fc->invmass = pmp.invmass;
    for (int k = 0; k < 6; k++) fc->I[k] = pmp.I[k];
    for (int k = 0; k < 9; k++) fc->invI[k] = pmp.invI[k];
    fc->air_rho = sc.v[S_AIR_RHO]; fc->skin_cf = sc.v[S_SKIN_CF];
    fc->phase = seed_phase(env_seed);
    fc->gust = sc.v[S_GUST]; fc->base_x = sc.v[S_BASE_X]; fc->base_y = sc.v[S_BASE_Y];
    fc->cg = cg;
    fc->warp_pitch = sc.v[S_WARP_PITCH]; fc->warp_roll = sc.v[S_WARP_ROLL];
    if (pmp_out) *pmp_out = pmp;
    if (sc_out) *sc_out = sc;
}

constexpr int kRefSlots = 4;                         // flights of a block, and its warps
constexpr int kRefThreads = 32 * kRefSlots;
constexpr int kRefPad = (kNtMax + 31) / 32 * 32;     // staged panels, filled up with empty ones

// A block's flights.  Arrays of [slot] are read by the eight lanes of each slot at once.
struct RefBlock {
    float4 pos_t[kRefSlots], q[kRefSlots], vel[kRefSlots], wb[kRefSlots];
    float4 cst[6][kRefSlots];                        // RefConst
    float4 pre[kRefSlots][5];                        // rows of the rotation | spin in the world, velocity | half the
                                                     // density, wind | skin friction
    float4 part[kRefSlots][2 * kRefSlots + 1];       // by virtual warp: force, torque
    int nt[kRefSlots], flight[kRefSlots], step[kRefSlots];
    float4 rb[kRefSlots][kRefPad];                   // centroid, area
    float2 nxy[kRefSlots][kRefPad];                  // normal
    float nz[kRefSlots][kRefPad];
};

// What the integrator needs of FlightConst, next to the panels'.
struct alignas(16) RefConst {
    float I[6], invI[9], pad0;                                      // the rotation's: four float4
    float mass, invmass, phase, gust, base_x, base_y, pad1, pad2;   // the translation's: two
};
static_assert(sizeof(RefConst) == 6 * sizeof(float4), "RefConst is six float4");

__device__ __forceinline__ vec3 xyz(float4 v) { return mk3(v.x, v.y, v.z); }

__device__ __forceinline__ FlightState ref_state(const RefBlock& b, int m) {
    const float4 p = b.pos_t[m], q = b.q[m];
    FlightState st;
    st.pos = xyz(p); st.t = p.w;
    st.q = mkq(q.x, q.y, q.z, q.w);
    st.vel = xyz(b.vel[m]); st.wb = xyz(b.wb[m]);
    st.step = b.step[m];
    st.pad = 0;
    return st;
}

__device__ __forceinline__ void ref_store(RefBlock& b, int m, const FlightState& st) {
    b.pos_t[m] = make_float4(st.pos.x, st.pos.y, st.pos.z, st.t);
    b.q[m] = make_float4(st.q.w, st.q.x, st.q.y, st.q.z);
    b.vel[m] = make_float4(st.vel.x, st.vel.y, st.vel.z, 0.0f);
    b.wb[m] = make_float4(st.wb.x, st.wb.y, st.wb.z, 0.0f);
    b.step[m] = st.step;
}

// Put flight (p, s) in slot m, by a whole warp: constants, state (from *st0, or released) and panels with
// the print-warped unit normal (src/sim.cu:135-143), the last round of 32 filled up with empty ones.
__device__ __noinline__ void ref_fill(const FlightArgs& a, RefBlock& b, int m, int flight, const FlightState* st0) {
    const int lane = threadIdx.x & 31;
    const int p = flight / a.nseeds, s = flight - p * a.nseeds;
    const int nt = a.plane_nt[p];
    FlightConst fc;
    MassProps pmp;
    Scenario sc;
    flight_setup(a, p, s, &fc, &pmp, &sc);
    FlightState st;
    if (st0) st = *st0;
    else release(sc, pmp, fc.cg, &st);
    if (lane == 0) {
        ref_store(b, m, st);
        b.nt[m] = nt;
        b.flight[m] = flight;
        RefConst c;
        for (int k = 0; k < 6; k++) c.I[k] = fc.I[k];
        for (int k = 0; k < 9; k++) c.invI[k] = fc.invI[k];
        c.mass = fc.mass;
        c.invmass = fc.invmass;
        c.phase = fc.phase; c.gust = fc.gust; c.base_x = fc.base_x; c.base_y = fc.base_y;
        c.pad0 = c.pad1 = c.pad2 = 0.0f;
        const float4* o = reinterpret_cast<const float4*>(&c);
        for (int k = 0; k < 6; k++) b.cst[k][m] = o[k];
        b.pre[m][3].w = __fmul_rn(0.5f, fc.air_rho);
        b.pre[m][4].w = fc.skin_cf;
    }
    const int off = a.plane_off[p];
    for (int i = lane; i - lane < nt; i += 32) {
        float4 rbA = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        vec3 nb = mk3(0.0f, 0.0f, 0.0f);
        if (i < nt) {
            float4 c4 = a.pc[off + i], n4 = a.pn[off + i];
            vec3 rb = vsub(mk3(c4.x, c4.y, c4.z), fc.cg);
            nb = mk3(n4.x, n4.y, n4.z);
            float ar = fc.warp_roll * fmaxf(-1.f, fminf(1.f, rb.y / 0.125f));
            float ap = fc.warp_pitch * fmaxf(-1.f, fminf(1.f, rb.x / 0.125f));
            vec3 nr = mk3(nb.x, nb.y - ar * nb.z, nb.z + ar * nb.y);
            nb = vnorm(mk3(nr.x + ap * nr.z, nr.y, nr.z - ap * nr.x));
            rbA = make_float4(rb.x, rb.y, rb.z, c4.w);
        }
        b.rb[m][i] = rbA;
        b.nxy[m][i] = make_float2(nb.x, nb.y);
        b.nz[m][i] = nb.z;
    }
}

// The order in which vdot and vcross are fused here.
__device__ __forceinline__ float dot_exact(vec3 a, vec3 b) {
    return __fmaf_rn(a.z, b.z, __fmaf_rn(a.x, b.x, __fmul_rn(a.y, b.y)));
}
__device__ __forceinline__ vec3 cross_exact(vec3 a, vec3 b) {
    return mk3(__fmaf_rn(a.y, b.z, -__fmul_rn(a.z, b.y)), __fmaf_rn(a.z, b.x, -__fmul_rn(a.x, b.z)),
               __fmaf_rn(a.x, b.y, -__fmul_rn(a.y, b.x)));
}

// What the panels of slot m's next step need of the rotation: its rows and the spin in the world.
__device__ __forceinline__ void ref_publish_rotation(RefBlock& b, int m, bool write, quat4 q, vec3 wb) {
    const float w = q.w, x = q.x, y = q.y, z = q.z;
    const float yy = __fmul_rn(y, y), zz = __fmul_rn(z, z), xz = __fmul_rn(x, z);
    const vec3 r0 = mk3(1 - 2 * __fadd_rn(yy, zz), 2 * __fmaf_rn(x, y, -__fmul_rn(w, z)), 2 * __fmaf_rn(w, y, xz));
    const vec3 r1 = mk3(2 * __fmaf_rn(x, y, __fmul_rn(w, z)), 1 - 2 * __fmaf_rn(x, x, zz), 2 * __fmaf_rn(y, z, -__fmul_rn(w, x)));
    const vec3 r2 = mk3(2 * __fmaf_rn(-w, y, xz), 2 * __fmaf_rn(y, z, __fmul_rn(w, x)), 1 - 2 * __fmaf_rn(x, x, yy));
    const vec3 ww = mk3(__fmaf_rn(r0.z, wb.z, __fmaf_rn(r0.y, wb.y, __fmul_rn(r0.x, wb.x))),
                        dot_exact(r1, wb), dot_exact(r2, wb));
    if (!write) return;
    b.q[m] = make_float4(q.w, q.x, q.y, q.z);
    b.wb[m] = make_float4(wb.x, wb.y, wb.z, 0.0f);
    b.pre[m][0] = make_float4(r0.x, r0.y, r0.z, ww.x);
    b.pre[m][1] = make_float4(r1.x, r1.y, r1.z, ww.y);
    b.pre[m][2] = make_float4(r2.x, r2.y, r2.z, ww.z);
}

// wind_at with its fused operations spelled out: a * p + b * t + c * phase, and the sums of the sines.
__device__ __forceinline__ vec3 ref_wind(vec3 p, float t, float s, float gust, float base_x, float base_y) {
    auto gs = [&](float a, float x, float b, float c) { return sinf(__fmaf_rn(c, s, __fmaf_rn(a, x, __fmul_rn(b, t)))); };
    float gx = __fmaf_rn(0.55f, gs(0.9f, p.x, 1.3f, 1.0f), __fmul_rn(0.35f, gs(2.3f, p.z, 2.1f, 1.7f)));
    gx = __fmaf_rn(0.25f, gs(4.1f, p.y, 3.3f, 0.4f), gx);
    float gy = __fmaf_rn(0.50f, gs(1.1f, p.x, 1.7f, 2.2f), __fmul_rn(0.30f, gs(3.1f, p.z, 2.9f, 0.9f)));
    float gz = __fmaf_rn(0.30f, gs(1.4f, p.x, 2.3f, 3.1f), __fmul_rn(0.20f, gs(2.7f, p.y, 1.9f, 1.2f)));
    return mk3(__fmaf_rn(gust, gx, base_x), __fmaf_rn(gust, gy, base_y), gust * gz);
}

// And of the translation: velocity and wind.
__device__ __forceinline__ void ref_publish_translation(RefBlock& b, int m, bool write, vec3 pos, vec3 vel, float t, int step) {
    if (step > 0 && step % kChunk == 0) t = step * PE_DT;
    const float4 c0 = b.cst[4][m], c1 = b.cst[5][m];
    vec3 wind = ref_wind(pos, t, c0.z, c0.w, c1.x, c1.y);
    if (!write) return;
    b.pos_t[m] = make_float4(pos.x, pos.y, pos.z, t);
    b.vel[m] = make_float4(vel.x, vel.y, vel.z, 0.0f);
    b.step[m] = step;
    float* o = reinterpret_cast<float*>(&b.pre[m][3]);  // the fourth of each is the flight's own
    o[0] = vel.x; o[1] = vel.y; o[2] = vel.z;
    o[4] = wind.x; o[5] = wind.y; o[6] = wind.z;
}

// Aerodynamic force and torque of one panel, added to acc (FIRST: written to it; src/sim.cu:135-158).  A panel
// without flow adds zeros.
template <bool FIRST>
__device__ __forceinline__ void panel_exact(const float4* rbA, const float2* nxy, const float* nz, vec3 r0, vec3 r1,
                                            vec3 r2, vec3 ww, vec3 vel, vec3 wind, float half_rho, float skin_cf,
                                            float* acc) {
    const float4 c = *rbA;
    const float2 n = *nxy;
    const vec3 rb = xyz(c), nb = mk3(n.x, n.y, *nz);
    const vec3 rw = mk3(dot_exact(r0, rb), dot_exact(r1, rb), dot_exact(r2, rb));
    const vec3 nw = mk3(dot_exact(r0, nb), dot_exact(r1, nb), dot_exact(r2, nb));
    const vec3 vr = vsub(vadd(vel, cross_exact(ww, rw)), wind);
    const float V2 = dot_exact(vr, vr);
    float iv = 1.0f / sqrtf(V2);
    iv = V2 < 1e-6f ? 0.0f : iv;
    const vec3 vh = vscl(vr, iv);
    const float s = dot_exact(vh, nw);
    const float qd = half_rho * V2 * c.w;
    const float cn = __fmaf_rn(PE_CN_SLOPE * s, sqrtf(fmaxf(0.f, __fmaf_rn(-s, s, 1.f))), 2.0f * s * fabsf(s));
    const float kn = -qd * cn, kt = -qd * skin_cf;
    const vec3 tang = mk3(__fmaf_rn(-nw.x, s, vh.x), __fmaf_rn(-nw.y, s, vh.y), __fmaf_rn(-nw.z, s, vh.z));
    const vec3 f = mk3(__fmaf_rn(nw.x, kn, __fmul_rn(tang.x, kt)), __fmaf_rn(nw.y, kn, __fmul_rn(tang.y, kt)),
                       __fmaf_rn(nw.z, kn, __fmul_rn(tang.z, kt)));
    const vec3 tq = cross_exact(rw, f);
    const float add[6] = {f.x, f.y, f.z, tq.x, tq.y, tq.z};
#pragma unroll
    for (int k = 0; k < 6; k++) acc[k] = FIRST ? add[k] : __fadd_rn(acc[k], add[k]);
}

// The panels of every slot and their sums over this warp, by all warps.
__device__ __forceinline__ void ref_panels(RefBlock& b, int warp, int lane) {
    float v[6 * kRefSlots];
    static_assert(kRefPad <= 3 * 128, "three rounds of 128 panels");
#pragma unroll
    for (int m = 0; m < kRefSlots; m++) {
        float* acc = v + 6 * m;
        const int nt = b.nt[m];
        const int i0 = 32 * ((warp - m) & 3);
        if (i0 < nt) {
            const float4 p0 = b.pre[m][0], p1 = b.pre[m][1], p2 = b.pre[m][2], p3 = b.pre[m][3], p4 = b.pre[m][4];
            const vec3 r0 = xyz(p0), r1 = xyz(p1), r2 = xyz(p2), ww = mk3(p0.w, p1.w, p2.w), vel = xyz(p3), wind = xyz(p4);
            const float4* rb = b.rb[m] + i0 + lane;
            const float2* nxy = b.nxy[m] + i0 + lane;
            const float* nz = b.nz[m] + i0 + lane;
            panel_exact<true>(rb, nxy, nz, r0, r1, r2, ww, vel, wind, p3.w, p4.w, acc);
            if (i0 + 128 < nt) {
                panel_exact<false>(rb + 128, nxy + 128, nz + 128, r0, r1, r2, ww, vel, wind, p3.w, p4.w, acc);
                if (i0 + 256 < nt)
                    panel_exact<false>(rb + 256, nxy + 256, nz + 256, r0, r1, r2, ww, vel, wind, p3.w, p4.w, acc);
            }
        } else {
#pragma unroll
            for (int k = 0; k < 6; k++) acc[k] = 0.0f;
        }
    }
    // transposed: a level halves the values a lane carries; lane 8 m + 4 h + q (q < 3) ends with
    // component 3 h + q of slot m, summed along the tree of offsets 16, 8, 4, 2, 1
    auto fold = [&](int off, int half) {
        const bool up = (lane & off) != 0;
#pragma unroll
        for (int k = 0; k < half; k++) {
            const float send = up ? v[k] : v[k + half];
            const float keep = up ? v[k + half] : v[k];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    };
    fold(16, 12);
    fold(8, 6);
    fold(4, 3);
    v[3] = 0.0f;
    fold(2, 2);
    fold(1, 1);
    const int m = lane >> 3;
    if ((lane & 3) != 3) {
        float* part = reinterpret_cast<float*>(&b.part[m][2 * ((warp - m) & 3)]);
        part[lane & 7] = v[0];
    }
}

// The sum of slot m's force (k = 0) or torque (k = 1): ((0 + W0) + W1) + W2) + W3, thread 0's serial order.
__device__ __forceinline__ vec3 ref_sum(const RefBlock& b, int m, int k) {
    vec3 t = mk3(0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int w = 0; w < 4; w++) t = vadd(t, xyz(b.part[m][2 * w + k]));
    return t;
}

// The integrator (src/sim.cu:177-196) in two halves that need nothing of each other: rotation,
__device__ __forceinline__ void ref_rotate(const RefBlock& b, int m, vec3 Ts, quat4* q_out, vec3* wb_out) {
    RefConst fc;
    float4* o = reinterpret_cast<float4*>(&fc);
#pragma unroll
    for (int k = 0; k < 4; k++) o[k] = b.cst[k][m];
    const float4 q4 = b.q[m];
    const vec3 r0 = xyz(b.pre[m][0]), r1 = xyz(b.pre[m][1]), r2 = xyz(b.pre[m][2]);
    vec3 wb = xyz(b.wb[m]);
    vec3 tb = mk3(dot_exact(mk3(r0.x, r1.x, r2.x), Ts), dot_exact(mk3(r0.y, r1.y, r2.y), Ts), dot_exact(mk3(r0.z, r1.z, r2.z), Ts));
    vec3 Iw = mk3(dot_exact(mk3(fc.I[0], fc.I[3], fc.I[4]), wb), dot_exact(mk3(fc.I[3], fc.I[1], fc.I[5]), wb),
                  __fmaf_rn(fc.I[2], wb.z, __fmaf_rn(fc.I[5], wb.y, __fmul_rn(fc.I[4], wb.x))));
    vec3 tq = vsub(tb, cross_exact(wb, Iw));
    vec3 dw = mk3(dot_exact(mk3(fc.invI[0], fc.invI[1], fc.invI[2]), tq), dot_exact(mk3(fc.invI[3], fc.invI[4], fc.invI[5]), tq),
                  dot_exact(mk3(fc.invI[6], fc.invI[7], fc.invI[8]), tq));
    wb = vadd(wb, vscl(dw, PE_DT));
    float wl = vlen(wb);
    if (wl > 150.f) wb = vscl(wb, 150.f / wl);
    quat4 q = mkq(q4.x, q4.y, q4.z, q4.w);
    quat4 dq = qmul(q, mkq(0, wb.x, wb.y, wb.z));
    dq.z = __fmaf_rn(-q.y, wb.x, __fmaf_rn(q.w, wb.z, __fmul_rn(q.x, wb.y)));
    *q_out = qnormalize(mkq(q.w + 0.5f * dq.w * PE_DT, q.x + 0.5f * dq.x * PE_DT,
                            q.y + 0.5f * dq.y * PE_DT, q.z + 0.5f * dq.z * PE_DT));
    *wb_out = wb;
}

// and translation.  Returns 1 when the flight ends at `step` (src/sim.cu:197-204).
__device__ __forceinline__ int ref_translate(const RefBlock& b, int m, vec3 Fs, vec3* pos_out, vec3* vel_out, int step,
                                             int max_steps, float* fit) {
    const float4 c = b.cst[4][m];  // mass, 1 / mass
    Fs.z -= c.x * PE_GRAV;
    vec3 vel = xyz(b.vel[m]), pos = xyz(b.pos_t[m]);
    vel = vadd(vel, vscl(Fs, c.y * PE_DT));
    float vl = vlen(vel);
    if (vl > 60.f) vel = vscl(vel, 60.f / vl);
    pos = vadd(pos, vscl(vel, PE_DT));
    *pos_out = pos;
    *vel_out = vel;
    int bad = !(pos.x == pos.x && vel.x == vel.x);
    *fit = bad ? -10.0f : pos.x;
    return pos.z <= 0.0f || bad || fabsf(pos.y) > 300.f || pos.x < -50.f || step == max_steps - 1;
}

// The next flight of the queue into slot m, by a whole warp; none left: the slot stays empty.
__device__ __forceinline__ void ref_next(const FlightArgs& a, RefBlock& b, int m, int n_work) {
    const int lane = threadIdx.x & 31;
    for (;;) {
        int f = 0;
        if (lane == 0) f = atomicAdd(a.work, 1);
        f = __shfl_sync(0xffffffffu, f, 0);
        if (f >= n_work) {
            if (lane == 0) b.nt[m] = 0;
            break;
        }
        const int flight = a.active_in ? a.active_in[f] : f;
        if (a.step_begin == 0 && a.plane_nt[flight / a.nseeds] <= 0) {  // oversize: hard negative, no steps
            if (lane == 0) { a.dist[flight] = -100.0f; a.steps[flight] = 0; }  // (src/sim.cu:108-109)
            continue;
        }
        ref_fill(a, b, m, flight, a.step_begin == 0 ? nullptr : a.state + flight);
        break;
    }
    __syncwarp();
}

// Persistent flight kernel: each block's slots (the first `slots` of them) take flights until the list is
// exhausted.  nt[slot]: panels of its flight; 0 empty; kEnded and kPaused ask for the next flight.
constexpr int kEnded = -1, kPaused = -2;
__global__ void __launch_bounds__(kRefThreads, 5) k_flight(FlightArgs a, int slots) {
    extern __shared__ float4 smem[];
    RefBlock& b = *reinterpret_cast<RefBlock*>(smem);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    int lane;
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));
    const int m = lane >> 3;  // the slot this lane integrates
    const bool leads = (lane & 7) == 0;
    const int n_work = a.active_in ? *a.n_active_in : a.n_flights;
    const int end = min(a.step_end, a.max_steps);
    if (lane == 0) b.nt[warp] = warp < slots ? kEnded : 0;
    __syncthreads();
    for (int turn = 0;; turn = (turn + 1) & 3) {
        if ((b.nt[0] | b.nt[1] | b.nt[2] | b.nt[3]) < 0) {
            __syncthreads();  // every warp has seen it
            const int k = warp;
            if (b.nt[k] < 0) {
                if (lane == 0 && b.nt[k] == kPaused && a.active_out) {
                    const int flight = b.flight[k];
                    a.state[flight] = ref_state(b, k);
                    a.active_out[atomicAdd(a.n_active_out, 1)] = flight;
                }
                __syncwarp();
                ref_next(a, b, k, n_work);
                if (b.nt[k] > 0) {
                    const FlightState st = ref_state(b, k);
                    __syncwarp();
                    ref_publish_rotation(b, k, lane == 0, st.q, st.wb);
                    ref_publish_translation(b, k, lane == 0, st.pos, st.vel, st.t, st.step);
                }
            }
            __syncthreads();
        }
        if ((b.nt[0] | b.nt[1] | b.nt[2] | b.nt[3]) == 0) break;
        ref_panels(b, warp, lane);
        __syncthreads();
        if (warp == turn) {
            quat4 q;
            vec3 wb;
            ref_rotate(b, m, ref_sum(b, m, 1), &q, &wb);
            __syncwarp();
            ref_publish_rotation(b, m, leads, q, wb);
        } else if (warp == ((turn + 1) & 3)) {
            vec3 pos, vel;
            float fit;
            int step = b.step[m];
            const float t = b.pos_t[m].w + PE_DT;
            const bool live = b.nt[m] > 0;
            const int ended = ref_translate(b, m, ref_sum(b, m, 0), &pos, &vel, step, a.max_steps, &fit);
            __syncwarp();
            if (ended) {
                if (leads && live) {
                    const int flight = b.flight[m];
                    a.dist[flight] = fit;
                    a.steps[flight] = step + 1;
                    b.nt[m] = kEnded;
                }
            } else {
                step++;
                if (step < end) {
                    ref_publish_translation(b, m, leads, pos, vel, t, step);
                } else if (leads && live) {  // the clock restarts in the next launch
                    b.pos_t[m] = make_float4(pos.x, pos.y, pos.z, t);
                    b.vel[m] = make_float4(vel.x, vel.y, vel.z, 0.0f);
                    b.step[m] = step;
                    b.nt[m] = kPaused;
                }
            }
        }
        __syncthreads();
    }
}

// Teacher-forced single step (parity tests): flight f from state_in[f].
__global__ void __launch_bounds__(kRefThreads) k_debug_step(FlightArgs a, const FlightState* state_in,
                                                            FlightState* state_out, float* FT, int* done_out,
                                                            float* fit_out, int step) {
    extern __shared__ float4 smem[];
    RefBlock& b = *reinterpret_cast<RefBlock*>(smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int flight = blockIdx.x * kRefSlots + warp;
    const bool mine = flight < a.n_flights;
    FlightState st;
    if (mine) {
        st = state_in[flight];
        ref_fill(a, b, warp, flight, state_in + flight);
        __syncwarp();
        ref_publish_rotation(b, warp, lane == 0, st.q, st.wb);
        ref_publish_translation(b, warp, lane == 0, st.pos, st.vel, st.t, step);
    } else if (lane == 0) {
        b.nt[warp] = 0;
    }
    __syncthreads();
    ref_panels(b, warp, lane);
    __syncthreads();
    if (!mine || lane) return;
    const vec3 F = ref_sum(b, warp, 0), T = ref_sum(b, warp, 1);
    float fit = 0.0f;
    const int done = ref_translate(b, warp, F, &st.pos, &st.vel, step, a.max_steps, &fit);
    ref_rotate(b, warp, T, &st.q, &st.wb);
    st.t = b.pos_t[warp].w + PE_DT;
    state_out[flight] = st;
    const float ft[6] = {F.x, F.y, F.z, T.x, T.y, T.z};
    for (int k = 0; k < 6; k++) FT[flight * 6 + k] = ft[k];
    done_out[flight] = done;
    fit_out[flight] = done ? fit : 0.0f;
}

__global__ void k_debug_release(FlightArgs a, FlightState* out) {
    const int flight = blockIdx.x * blockDim.x + threadIdx.x;
    if (flight >= a.n_flights) return;
    const int p = flight / a.nseeds, s = flight - p * a.nseeds;
    FlightConst fc; MassProps pmp; Scenario sc;
    flight_setup(a, p, s, &fc, &pmp, &sc);
    FlightState st;
    release(sc, pmp, fc.cg, &st);
    out[flight] = st;
}

// ---------------------------------------------------------------- host-side launch helpers
int flight_blocks_per_sm() {
    cudaFuncSetAttribute((const void*)k_flight, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RefBlock));
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_flight, kRefThreads, sizeof(RefBlock)) != cudaSuccess) return 0;
    return nb;
}

cudaError_t launch_flight(const FlightArgs& a, int grid, cudaStream_t s) {
    cudaError_t e = cudaFuncSetAttribute((const void*)k_flight, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RefBlock));
    if (e != cudaSuccess) return e;
    // few flights spread over the blocks: fewer of them in each, none idle
    const int slots = (int)std::min<long long>(kRefSlots, ((long long)a.n_flights + grid - 1) / grid);
    k_flight<<<grid, kRefThreads, sizeof(RefBlock), s>>>(a, slots);
    return cudaGetLastError();
}

cudaError_t launch_debug_step(const FlightArgs& a, const FlightState* state_in, FlightState* state_out,
                              float* FT, int* done, float* fit, int step, cudaStream_t s) {
    cudaError_t e = cudaFuncSetAttribute((const void*)k_debug_step, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RefBlock));
    if (e != cudaSuccess) return e;
    const int grid = (a.n_flights + kRefSlots - 1) / kRefSlots;
    k_debug_step<<<grid, kRefThreads, sizeof(RefBlock), s>>>(a, state_in, state_out, FT, done, fit, step);
    return cudaGetLastError();
}

cudaError_t launch_debug_release(const FlightArgs& a, FlightState* out, cudaStream_t s) {
    k_debug_release<<<(a.n_flights + 127) / 128, 128, 0, s>>>(a, out);
    return cudaGetLastError();
}

}  // namespace pe
