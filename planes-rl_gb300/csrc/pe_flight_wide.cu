// pe_flight_wide.cu -- the body-frame flight (pe_flight_fast.cuh) with a block of three warps per
// flight, for batches whose time is their longest flights' chains of steps.
//
// A flight of 32 lanes walks its step's chain alone, 0.6 to 0.7 us of it: up to six pair passes one
// after the other, a five-level shuffle tree for six sums, the integrator.  Here the chain is spread:
//   * a lane holds its one or two pairs in registers for the whole flight (pass n on warp n % 3), so the
//     panel part is one pair's chain with no loads;
//   * the pair forces cross through shared memory, and warp w adds components w of force and torque over
//     the passes in their fixed order, its own passes from registers;
//   * the lane totals cross once more, and the fold takes sixteen totals per lane (four levels of the tree
//     without a shuffle);
//   * warp 0 turns the plane while warp 1 moves it and takes its gusts, one sine per lane; warp 2 stores
//     what pe_grad keeps.  Attitude rows, rates and air velocity cross through shared memory.
// Three barriers of three warps per step.  The step's code is instantiated for each warp: its own values stay
// in registers, all lanes store what one would (no branch), the rates cross once and are doubled by the
// readers.  Bound: that chain, 0.38 us a step alone, a fifth of it shared-memory wavefronts, and from six
// flights per SM on the 800 warp instructions of a flight-step, twice the other kernels', so the dispatch
// gives it small batches and the last flights of large ones (pe_internal.cuh).
// Measured, flights of 64 x 8 (longest 1,368 steps): 0.96 ms at 32 lanes; here 0.84 ms with every warp
// integrating, 0.76 ms with the integrator split, 0.63 ms with its branches and clamps off the chain and
// the sines spread, 0.53 ms with the code by warp and the shorter fold.  (Six warps of a pass each: 0.64;
// the two pairs of a lane overlap.  Five blocks per SM at 128 registers: 0.56.)  The sums run in the fixed
// order of pe_flight_fast.cuh: every distance and step count is bit-identical to the other kernels'.
#include <type_traits>

#include "pe_flight_fast.cuh"

namespace pe {

namespace {

constexpr int kWideWarps = 3;
constexpr int kWidePasses = 6;  // pair v + 32 n of pass n: 192 pairs hold the largest plane's 172
static_assert(32 * kWidePasses >= (kNtMax + 1) / 2, "every pair has a pass");

struct WideSmem {
    // -force of each pair, packed (even, odd panel): x and y, z
    ulonglong2 nf_xy[kWidePasses][32];
    f2 nf_z[kWidePasses][32];
    alignas(16) float tot[6][36];           // lane totals of the six sums, lane v at (v % 4) * 8 + v / 4
    float4 rows[3];             // attitude rows and body rates, from warp 0
    float4 air;                 // air velocity; as an int 1 once the flight is over, 2 at the launch's last step; warp 1
    int next;
};

// The block's barrier; the three warps meet it at different places of the step.
__device__ __forceinline__ void block_sync() { asm volatile("bar.sync 0;" ::: "memory"); }

// Staged pair q: its seven packed values.
struct WidePair {
    f2 rbx, rby, rbz, ak, nbx, nby, nbz;
};
__device__ __forceinline__ WidePair wide_stage(const FlightArgs& a, int off, int nt, int q, vec3 cg, float half_rho,
                                               float wp, float wr) {
    float4 oa[2], ob[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        oa[h] = ob[h] = make_float4(0, 0, 0, 0);
        if (2 * q + h < nt)
            fast_stage_one(a.pc[off + 2 * q + h], a.pn[off + 2 * q + h], cg, half_rho, wp, wr, &oa[h], &ob[h]);
    }
    WidePair p;
    p.rbx = pk(oa[0].x, oa[1].x); p.rby = pk(oa[0].y, oa[1].y); p.rbz = pk(oa[0].z, oa[1].z); p.ak = pk(oa[0].w, oa[1].w);
    p.nbx = pk(ob[0].x, ob[1].x); p.nby = pk(ob[0].y, ob[1].y); p.nbz = pk(ob[0].z, ob[1].z);
    return p;
}

__device__ __forceinline__ f2 axis(f2 x, f2 y, f2 z, int i) { return i == 0 ? x : (i == 1 ? y : z); }

// Three of the six sums on every lane: lanes 2c + r fold the totals of lanes r and r + 2, r + 4, ... of sum
// first + c by bits 16, 8, 4 and 2; the last level takes both results of a sum at once.  (Four lanes per sum
// and twelve shuffles: 3 % more per step; one lane and three: 2 %.)
__device__ __forceinline__ vec3 wide_fold(const WideSmem& sm, int first, int lane) {
    const ulonglong2* row = reinterpret_cast<const ulonglong2*>(&sm.tot[first + min(lane >> 1, 2)][(lane & 1) * 8]);
    const ulonglong2 lo = row[0], hi = row[1], lo2 = row[4], hi2 = row[5];
    float t0, t1, u0, u1;
    upk(add2(add2(lo.x, hi.x), add2(lo.y, hi.y)), t0, t1);
    upk(add2(add2(lo2.x, hi2.x), add2(lo2.y, hi2.y)), u0, u1);
    const float t = add_(add_(t0, t1), add_(u0, u1));
    float o[3];
#pragma unroll
    for (int c = 0; c < 3; c++) o[c] = add_(__shfl_sync(0xffffffffu, t, 2 * c), __shfl_sync(0xffffffffu, t, 2 * c + 1));
    return mk3(o[0], o[1], o[2]);
}

// Attitude rows and body rates for every warp, one vector per lane.
__device__ __forceinline__ void wide_put_rot(WideSmem& sm, vec3 r0, vec3 r1, vec3 r2, vec3 w) {
    sm.rows[0] = make_float4(r0.x, r0.y, r0.z, r1.x);
    sm.rows[1] = make_float4(r1.y, r1.z, r2.x, r2.y);
    sm.rows[2] = make_float4(r2.z, w.x, w.y, w.z);
}

template <bool GRAD>
__global__ void __launch_bounds__(32 * kWideWarps, 4) k_flight_wide(FlightArgs a) {
    __shared__ WideSmem sm;
    int tid;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));  // kept in a register: read anew it costs a chain 20 cycles
    const int lane = tid & 31;
    const int w = (int)__reduce_or_sync(0xffffffffu, (unsigned)tid >> 5);  // provably the same on a warp's lanes
    const int w1 = w == 2 ? 0 : w + 1, w2 = w == 0 ? 2 : w - 1;  // the axes after w, cyclically
    const int n_work = a.active_in ? *a.n_active_in : a.n_flights;
    while (true) {
        if (tid == 0) sm.next = atomicAdd(a.work, 1);
        block_sync();
        const int f = sm.next;
        block_sync();
        if (f >= n_work) break;
        const int flight = a.active_in ? a.active_in[f] : f;
        const int p = flight / a.nseeds, s = flight - p * a.nseeds;
        const int nt = a.plane_nt[p];
        if (nt <= 0) {
            if (tid == 0) {
                a.dist[flight] = -100.0f;
                a.steps[flight] = 0;
                if (GRAD) a.grad_kind[flight] = 0;
            }
            continue;
        }
        FastConst fc;
        vec3 cg;
        float air_rho, wp, wr;
        FlightState st;
        if (GRAD) {
            grad_record(a, flight, &fc, &cg, &air_rho, &wp, &wr, &st);
            if (a.active_in) st = a.state[flight];
        } else {
            MassProps pmp;
            Scenario sc;
            fast_setup(a, p, s, &fc, &cg, &air_rho, &wp, &wr, &pmp, &sc);
            if (!a.active_in)
                release(sc, pmp, cg, &st);
            else
                st = a.state[flight];
        }
        float* ck = nullptr;
        float* fsum = nullptr;
        if (GRAD) {
            ck = a.grad_ck + (size_t)flight * a.grad_nck * 16;
            fsum = a.grad_fsum ? a.grad_fsum + (size_t)flight * a.max_steps * 8 : nullptr;
            if (tid == 0 && !a.active_in) *reinterpret_cast<FlightState*>(ck) = st;  // the release state
        }
        const int off = a.plane_off[p];
        const float half_rho = mul_(0.5f, air_rho);
        const bool two = nt > 2 * 32 * kWideWarps;
        const WidePair q0 = wide_stage(a, off, nt, lane + 32 * w, cg, half_rho, wp, wr);
        WidePair q1 = {};
        if (two) q1 = wide_stage(a, off, nt, lane + 32 * (w + kWideWarps), cg, half_rho, wp, wr);
        // the arms that warp w's torque sums multiply: rb along the axes w + 2 and w + 1
        f2 arm2[kWidePasses], arm1[kWidePasses];
#pragma unroll
        for (int n = 0; n < kWidePasses; n++) {
            float r[2][3] = {{0, 0, 0}, {0, 0, 0}};
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int i = 2 * (lane + 32 * n) + h;
                if (i < nt) {
                    const float4 c4 = a.pc[off + i];
                    r[h][0] = sub_(c4.x, cg.x); r[h][1] = sub_(c4.y, cg.y); r[h][2] = sub_(c4.z, cg.z);
                }
            }
            const f2 x = pk(r[0][0], r[1][0]), y = pk(r[0][1], r[1][1]), z = pk(r[0][2], r[1][2]);
            arm2[n] = axis(x, y, z, w2);
            arm1[n] = axis(x, y, z, w1);
        }
        // Warp 0 turns the plane, warp 1 moves it, warp 2 stores what pe_grad keeps.  What every warp needs
        // of the state -- attitude rows, body rates, air velocity -- crosses through shared memory.
        const int end = min(a.step_end, a.max_steps);
        int step = st.step, over = 0;
        const WindLane wind_of = wind_lane(lane, fc.phase);
        if (w == 0) {
            vec3 r0, r1, r2;
            fast_rows(st.q, &r0, &r1, &r2);
            wide_put_rot(sm, r0, r1, r2, st.wb);
        } else if (w == 1) {
            if (step > 0 && step % kChunk == 0) st.t = mul_((float)step, PE_DT);
            const vec3 wind = wind_lanes(st.pos, mul_(wind_of.ct, st.t), wind_of, fc.gust, fc.base_x, fc.base_y);
            if (lane == 0)
                sm.air = make_float4(sub_(st.vel.x, wind.x), sub_(st.vel.y, wind.y), sub_(st.vel.z, wind.z), 0.0f);
        }
        vec3 before = st.pos;                       // the position one step back (warp 1)
        // steps to the next checkpoint, the last one's index
        int to_ck = GRAD ? a.grad_K - step % a.grad_K : 0, ck_i = GRAD ? step / a.grad_K : 0;
        int to_clock = kChunk - step % kChunk;      // steps to the clock's restart
        const int at = (lane & 3) * 8 + (lane >> 2);
        auto fly = [&](auto two_passes, auto warp_of) {
            constexpr bool TWO = decltype(two_passes)::value;
            constexpr int w = decltype(warp_of)::value, w1 = (w + 1) % 3, w2 = (w + 2) % 3;
            constexpr int NP = TWO ? kWidePasses : kWideWarps;
            for (;; step++) {
                block_sync();
                const float4 air = sm.air, m0 = sm.rows[0], m1 = sm.rows[1], m2 = sm.rows[2];
                over = __float_as_int(air.w);
                const vec3 r0 = mk3(m0.x, m0.y, m0.z), r1 = mk3(m0.w, m1.x, m1.y), r2 = mk3(m1.z, m1.w, m2.x);
                const vec3 vb = fast_body(r0, r1, r2, mk3(air.x, air.y, air.z));
                PairConst k;
                k.vbx = bc(vb.x); k.vby = bc(vb.y); k.vbz = bc(vb.z);
                k.wbx = bc(m2.y); k.wby = bc(m2.z); k.wbz = bc(m2.w);
                k.nwbx = bc(-m2.y); k.nwby = bc(-m2.z); k.nwbz = bc(-m2.w);
                k.k19 = c_k19; k.cf = bc(fc.skin_cf); k.tiny = c_tiny; k.mone = c_mone;
                f2 nx, ny, nz, mx, my, mz;
                pair_force(q0.rbx, q0.rby, q0.rbz, q0.ak, q0.nbx, q0.nby, q0.nbz, k, fc.skin_cf, nx, ny, nz);
                sm.nf_xy[w][lane] = make_ulonglong2(nx, ny); sm.nf_z[w][lane] = nz;
                if (TWO) {
                    pair_force(q1.rbx, q1.rby, q1.rbz, q1.ak, q1.nbx, q1.nby, q1.nbz, k, fc.skin_cf, mx, my, mz);
                    sm.nf_xy[w + kWideWarps][lane] = make_ulonglong2(mx, my); sm.nf_z[w + kWideWarps][lane] = mz;
                }
                if (over) break;  // tested here, off the chain: the state is one step too far on
                block_sync();
                f2 fn, tq, tp;
#pragma unroll
                for (int n = 0; n < NP; n++) {  // this warp's own passes from its registers
                    f2 x, y, z;
                    if (n == w) { x = nx; y = ny; z = nz; }
                    else if (n == w + kWideWarps) { x = mx; y = my; z = mz; }
                    else { const ulonglong2 xy = sm.nf_xy[n][lane]; x = xy.x; y = xy.y; z = sm.nf_z[n][lane]; }
                    fn = n ? add2(fn, axis(x, y, z, w)) : axis(x, y, z, w);
                    tq = n ? fma2(arm2[n], axis(x, y, z, w1), tq) : mul2(arm2[0], axis(x, y, z, w1));
                    tp = n ? fma2(arm1[n], axis(x, y, z, w2), tp) : mul2(arm1[0], axis(x, y, z, w2));
                }
                float e, o, e2, o2;
                upk(fn, e, o);
                sm.tot[w][at] = -add_(e, o);
                upk(tq, e, o); upk(tp, e2, o2);
                sm.tot[3 + w][at] = sub_(add_(e, o), add_(e2, o2));
                const bool mark = GRAD && --to_ck == 0;
                if (mark) { to_ck = a.grad_K; ++ck_i; }
                FlightState* at_ck = GRAD ? reinterpret_cast<FlightState*>(ck + (size_t)ck_i * 16) : nullptr;
                if constexpr (w == 0) {
                    const vec3 gyro = fast_gyro(fc, st.wb);
                    block_sync();
                    fast_rotate<true>(fc, gyro, wide_fold(sm, 3, lane), st.wb, st.q);
                    vec3 n0, n1, n2;
                    fast_rows(st.q, &n0, &n1, &n2);
                    wide_put_rot(sm, n0, n1, n2, st.wb);
                    // a flight that ends here leaves its checkpoint unread
                    if (mark && lane == 0) { at_ck->q = st.q; at_ck->wb = st.wb; }
                } else if constexpr (w == 1) {
                    st.t = add_(st.t, PE_DT);
                    if (--to_clock == 0) {  // as the next step starts: the clock restarts every 600 steps
                        to_clock = kChunk;
                        st.t = mul_((float)(step + 1), PE_DT);
                    }
                    const float tt = mul_(wind_of.ct, st.t);
                    before = st.pos;
                    block_sync();
                    const vec3 Fb = wide_fold(sm, 0, lane);
                    fast_translate<true>(fc, mk3(dot_(r0, Fb), dot_(r1, Fb), dot_(r2, Fb)), st.vel, st.pos);
                    const vec3 wind = wind_lanes(st.pos, tt, wind_of, fc.gust, fc.base_x, fc.base_y);
                    const int now = fast_over(st.pos, st.vel, step, a.max_steps) ? 1 : (step + 1 >= end ? 2 : 0);
                    sm.air = make_float4(sub_(st.vel.x, wind.x), sub_(st.vel.y, wind.y), sub_(st.vel.z, wind.z),
                                         __int_as_float(now));
                    if (lane == 0) {
                        if (mark) {
                            at_ck->pos = st.pos; at_ck->vel = st.vel; at_ck->t = st.t;
                            at_ck->step = 0; at_ck->pad = 0;
                        }
                    }
                } else {
                    block_sync();
                    if (GRAD && fsum) {
                        const vec3 F = wide_fold(sm, 0, lane), T = wide_fold(sm, 3, lane);
                        if (lane == 0) {
                            float4* d4 = reinterpret_cast<float4*>(fsum + (size_t)step * 8);
                            d4[0] = make_float4(F.x, F.y, F.z, T.x);
                            d4[1] = make_float4(T.y, T.z, 0.0f, 0.0f);
                        }
                    }
                }
            }
        };
        auto as_warp = [&](auto two_passes) {
            if (w == 0) fly(two_passes, std::integral_constant<int, 0>{});
            else if (w == 1) fly(two_passes, std::integral_constant<int, 1>{});
            else fly(two_passes, std::integral_constant<int, 2>{});
        };
        if (two) as_warp(std::true_type{}); else as_warp(std::false_type{});
        float fit = 0.0f;
        int kind = 0;
        if (over == 1 && w == 1)
            kind = fast_end(before, st.pos, st.vel, step - 1, a.max_steps, GRAD ? 1 : a.smooth, &fit);
        // The flight ended in step - 1, or it goes on in a later launch at `step`.  Every caller flies the whole
        // horizon; without the second, or without `end` in the step loop, the compiler orders a step's chain
        // worse (1 x 8 220 -> 226 us, 8 x 128 722 -> 729), so the kernel keeps what it can do.
        if (lane == 0) {
            if (over == 1) {
                if (w == 1) {
                    if (GRAD) a.grad_kind[flight] = kind;
                    a.dist[flight] = fit;
                    a.steps[flight] = step;
                }
            } else if (a.active_out) {
                FlightState* keep = a.state + flight;
                if (w == 0) { keep->q = st.q; keep->wb = st.wb; }
                if (w == 1) {
                    keep->pos = st.pos; keep->vel = st.vel; keep->t = st.t; keep->step = step; keep->pad = 0;
                    a.active_out[atomicAdd(a.n_active_out, 1)] = flight;
                }
            }
        }
    }
}

}  // namespace

cudaError_t flight_wide_configure(int* bps) {
    int n = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_flight_wide<false>, 32 * kWideWarps, 0);
    *bps = n > 0 ? n : 1;
    return e;
}

cudaError_t launch_flight_wide(const FlightArgs& a, int nsm, int bps, cudaStream_t s) {
    if (a.rec || a.spread > 0.f) return cudaErrorInvalidValue;
    const int grid = a.n_flights < bps * nsm ? a.n_flights : bps * nsm;
    if (a.grad_setup)
        k_flight_wide<true><<<grid, 32 * kWideWarps, 0, s>>>(a);
    else
        k_flight_wide<false><<<grid, 32 * kWideWarps, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace pe
