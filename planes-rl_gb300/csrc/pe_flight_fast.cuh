// pe_flight_fast.cuh -- the flight step in the body frame (the throughput formulation), shared by the
// kernels that fly it: pe_flight_fast.cu (a flight per 16 or 32 lanes of a warp), pe_flight_quad.cu
// (four flights per warp) and pe_flight_wide.cu (a flight per block).
//
// Same physics as src/sim.cu:129-204, rearranged for fewer operations per panel:
//   * the air velocity is rotated into the body frame once per step,
//       v_b = R^T (vel - wind),  and per panel  vr = v_b + wb x rb
//     instead of rotating every panel's position and normal into the world frame
//     (R^T (ww x R rb) = wb x rb for a rotation R);
//   * with vh = vr / |vr| and s = vh . nb the panel force
//       f = -qd cn nb - qd cf (vh - s nb) = a nb + b vr,
//       a = -qd (cn - cf s),  b = -qd cf / |vr|,
//     so neither vh nor the tangential vector is formed; 1/|vr| is one rsqrt;
//   * 0.5 rho A is folded into the staged panel once per flight;
//   * force and torque sums stay in the body frame: the integrator needs the body torque and
//     rotates only the total force to the world frame;
//   * two panels share every FP32 instruction (packed f32x2 add/mul/fma of sm_103a), read from
//     a pair-interleaved shared-memory layout so each 128-bit load yields two packed operands;
//     torque is accumulated as the two halves of the cross product and subtracted once per step,
//     so no packed negation is needed.
// About 25 instructions per panel-step against about 80 in the reference's form.  A panel whose
// relative flow is below 1e-3 m/s adds its (vanishing, < 1e-9 of the weight) force instead of
// being skipped.  Results differ from the reference arithmetic in rounding only; the parity
// tests bound the flight-level effect.
//
// Summation order is fixed by panel index, not by the execution shape: panel i belongs to pair
// q = i / 2 (even panels in the low half, odd in the high half), pair q to virtual lane
// v = q % 32; each virtual lane sums its pairs in order, adds its odd to its even partial sum, and
// the 32 virtual lanes reduce along one xor tree, so every shape (16 or 32 lanes per flight, any
// chunk length or grid) is bit-identical.  Every lane of a flight makes the same number of pair
// passes, ceil(ceil(nt / 2) / lanes): 11 for a 344-panel plane at 16 lanes (12 in a layout of
// 64-panel rows).  Passes beyond the plane's pairs read zero panels, whose force and torque are
// exact zeros; the partial sums start at +0 and in round-to-nearest a sum is -0 only when both
// terms are, so adding them changes no bit and the shapes still agree.
#pragma once
#include "pe_f32x2.cuh"
#include "pe_internal.cuh"

namespace pe {

struct FastConst {
    float mass, invmass;
    float I[6];
    float invI[9];
    float skin_cf;
    float phase, gust, base_x, base_y;
};

__device__ __forceinline__ void fast_setup(const FlightArgs& a, int p, int s, FastConst* fc, vec3* cg_out,
                                           float* air_rho, float* warp_pitch, float* warp_roll, MassProps* pmp_out,
                                           Scenario* sc_out) {
    const int env_seed = (int)((uint32_t)a.seeds[s] + (a.vary ? (uint32_t)p * 7919u : 0u));
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
    fc->skin_cf = sc.v[S_SKIN_CF];
    fc->phase = seed_phase(env_seed);
    fc->gust = sc.v[S_GUST]; fc->base_x = sc.v[S_BASE_X]; fc->base_y = sc.v[S_BASE_Y];
    *cg_out = cg;
    *air_rho = sc.v[S_AIR_RHO];
    *warp_pitch = sc.v[S_WARP_PITCH];
    *warp_roll = sc.v[S_WARP_ROLL];
    if (pmp_out) *pmp_out = pmp;
    if (sc_out) *sc_out = sc;
}

// The gradient model's set-up of a flight (FlightArgs.grad_setup), for pe_grad's forward pass.
__device__ __forceinline__ void grad_record(const FlightArgs& a, int flight, FastConst* fc, vec3* cg, float* air_rho,
                                            float* warp_pitch, float* warp_roll, FlightState* st) {
    const float* r = a.grad_setup + (size_t)flight * kGradSetupFloats;
    fc->mass = r[0]; fc->invmass = r[1];
    for (int c = 0; c < 6; c++) fc->I[c] = r[2 + c];
    for (int c = 0; c < 9; c++) fc->invI[c] = r[8 + c];
    fc->skin_cf = r[17]; fc->phase = r[18]; fc->gust = r[19]; fc->base_x = r[20]; fc->base_y = r[21];
    *cg = mk3(r[22], r[23], r[24]);
    *air_rho = r[25]; *warp_pitch = r[26]; *warp_roll = r[27];
    *st = *reinterpret_cast<const FlightState*>(r + 32);
}

// Explicitly rounded arithmetic: the compiler may neither contract nor reorder these, so the
// step is bit-identical in every template instance and execution shape.
__device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float mul_(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add_(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub_(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float dot_(vec3 a, vec3 b) { return fma_(a.z, b.z, fma_(a.y, b.y, mul_(a.x, b.x))); }
__device__ __forceinline__ float len_(vec3 a) { return __fsqrt_rn(dot_(a, a)); }

// Staged panel: (rb xyz, 0.5 rho A), (print-warped unit normal xyz, 0); src/sim.cu:135-143.
static __device__ __noinline__ void fast_stage_one(float4 c4, float4 n4, vec3 cg, float half_rho, float warp_pitch,
                                                   float warp_roll, float4* oa, float4* ob) {
    const vec3 rb = mk3(sub_(c4.x, cg.x), sub_(c4.y, cg.y), sub_(c4.z, cg.z));
    const float ar = mul_(warp_roll, fmaxf(-1.f, fminf(1.f, mul_(rb.y, 8.0f))));
    const float ap = mul_(warp_pitch, fmaxf(-1.f, fminf(1.f, mul_(rb.x, 8.0f))));
    const vec3 nr = mk3(n4.x, fma_(-ar, n4.z, n4.y), fma_(ar, n4.y, n4.z));
    vec3 nb = mk3(fma_(ap, nr.z, nr.x), nr.y, fma_(-ap, nr.x, nr.z));
    const float l = len_(nb);
    nb = l > 1e-12f ? mk3(__fdiv_rn(nb.x, l), __fdiv_rn(nb.y, l), __fdiv_rn(nb.z, l)) : mk3(0, 0, 1);
    *oa = make_float4(rb.x, rb.y, rb.z, mul_(half_rho, c4.w));
    *ob = make_float4(nb.x, nb.y, nb.z, 0.0f);
}

// Pair-interleaved panel layout of one flight: pair q holds panels 2q (low half) and 2q + 1 (high
// half); virtual lane v owns pairs v, v + 32, v + 64, ...  Slots from panel nt up to the flight's
// last pass are zero panels.
struct PairedPanels {
    float4* a;  // (rbx0, rbx1, rby0, rby1)
    float4* b;  // (rbz0, rbz1, ak0, ak1)   ak = 0.5 rho A
    float4* c;  // (nbx0, nbx1, nby0, nby1)
    float2* d;  // (nbz0, nbz1)
};
// Pair slots of one flight: every pair the passes of LPF lanes read, 176 at 16 lanes, 192 at 32.
template <int LPF>
__host__ __device__ constexpr int slot_pairs() { return LPF * ((kNtMax / 2 + LPF - 1) / LPF); }
template <int LPF>
__host__ __device__ constexpr size_t paired_bytes() {
    return (size_t)slot_pairs<LPF>() * (3 * sizeof(float4) + sizeof(float2));
}
template <int LPF>
__device__ __forceinline__ PairedPanels paired_view(char* base) {
    constexpr int kPairs = slot_pairs<LPF>();
    PairedPanels pp;
    pp.a = (float4*)base;
    pp.b = pp.a + kPairs;
    pp.c = pp.b + kPairs;
    pp.d = (float2*)(pp.c + kPairs);
    return pp;
}

template <int LPF>
__device__ __forceinline__ void fast_stage(const FlightArgs& a, int p, int nt, int j, vec3 cg, float air_rho,
                                           float warp_pitch, float warp_roll, PairedPanels pp) {
    const int off = a.plane_off[p];
    const float half_rho = mul_(0.5f, air_rho);
    const int slots = 2 * LPF * (((nt + 1) / 2 + LPF - 1) / LPF);  // every pair the passes read
    for (int i = j; i < slots; i += LPF) {
        float4 oa = make_float4(0, 0, 0, 0), ob = make_float4(0, 0, 0, 0);
        if (i < nt) fast_stage_one(a.pc[off + i], a.pn[off + i], cg, half_rho, warp_pitch, warp_roll, &oa, &ob);
        const int q = i >> 1, h = i & 1;
        float* pa = (float*)&pp.a[q];
        float* pb = (float*)&pp.b[q];
        float* pc = (float*)&pp.c[q];
        float* pd = (float*)&pp.d[q];
        pa[h] = oa.x; pa[2 + h] = oa.y;
        pb[h] = oa.z; pb[2 + h] = oa.w;
        pc[h] = ob.x; pc[2 + h] = ob.y;
        pd[h] = ob.z;
    }
}

// Gust field (src/common.h:459-467) with explicit rounding, from its phases' clock terms tt and seed
// terms ss.
struct WindTerms { float v[7]; };
__device__ __forceinline__ WindTerms wind_clock(float t) {
    return {{mul_(1.3f, t), mul_(2.1f, t), mul_(3.3f, t), mul_(1.7f, t), mul_(2.9f, t), mul_(2.3f, t), mul_(1.9f, t)}};
}
__device__ __forceinline__ WindTerms wind_seed(float s) {
    return {{s, mul_(1.7f, s), mul_(0.4f, s), mul_(2.2f, s), mul_(0.9f, s), mul_(3.1f, s), mul_(1.2f, s)}};
}
__device__ __forceinline__ vec3 wind_sum(const float v[7], float gust, float bx, float by) {
    const float gx = mul_(gust, fma_(0.25f, v[2], fma_(0.35f, v[1], mul_(0.55f, v[0]))));
    const float gy = mul_(gust, fma_(0.30f, v[4], mul_(0.50f, v[3])));
    const float gz = mul_(gust, fma_(0.20f, v[6], mul_(0.30f, v[5])));
    return mk3(add_(bx, gx), add_(by, gy), gz);
}
__device__ __forceinline__ vec3 wind_field(vec3 p, const WindTerms& tt, const WindTerms& ss, float gust, float bx, float by) {
    const float v[7] = {__sinf(add_(fma_(0.9f, p.x, tt.v[0]), ss.v[0])), __sinf(add_(fma_(2.3f, p.z, tt.v[1]), ss.v[1])),
                        __sinf(add_(fma_(4.1f, p.y, tt.v[2]), ss.v[2])), __sinf(add_(fma_(1.1f, p.x, tt.v[3]), ss.v[3])),
                        __sinf(add_(fma_(3.1f, p.z, tt.v[4]), ss.v[4])), __sinf(add_(fma_(1.4f, p.x, tt.v[5]), ss.v[5])),
                        __sinf(add_(fma_(2.7f, p.y, tt.v[6]), ss.v[6]))};
    return wind_sum(v, gust, bx, by);
}
// The same with one sine per lane: lane i (mod 8) holds phase i's factors of its axis, the clock and the
// seed; lanes 7 repeat phase 6.
struct WindLane {
    float cp, ct, ss;
    int axis;
};
__device__ __forceinline__ WindLane wind_lane(int lane, float s) {
    const int i = min(lane & 7, 6);
    const float cp[7] = {0.9f, 2.3f, 4.1f, 1.1f, 3.1f, 1.4f, 2.7f}, ct[7] = {1.3f, 2.1f, 3.3f, 1.7f, 2.9f, 2.3f, 1.9f};
    const WindTerms t = wind_seed(s);
    WindLane w = {cp[0], ct[0], t.v[0], 0};
#pragma unroll
    for (int k = 1; k < 7; k++)
        if (i == k) { w.cp = cp[k]; w.ct = ct[k]; w.ss = t.v[k]; }
    w.axis = i == 1 || i == 4 ? 2 : (i == 2 || i == 6 ? 1 : 0);
    return w;
}
__device__ __forceinline__ vec3 wind_lanes(vec3 p, float tt, const WindLane& w, float gust, float bx, float by) {
    const float q = w.axis == 0 ? p.x : (w.axis == 1 ? p.y : p.z);
    const float x = __sinf(add_(fma_(w.cp, q, tt), w.ss));
    float v[7];
#pragma unroll
    for (int i = 0; i < 7; i++) v[i] = __shfl_sync(0xffffffffu, x, i, 8);
    return wind_sum(v, gust, bx, by);
}
__device__ __forceinline__ vec3 fast_wind(vec3 p, float t, float s, float gust, float bx, float by) {
    return wind_field(p, wind_clock(t), wind_seed(s), gust, bx, by);
}

// Body->world rotation rows of a unit quaternion (src/common.h:38-43) with explicit rounding.
__device__ __forceinline__ void fast_rows(quat4 q, vec3* r0, vec3* r1, vec3* r2) {
    const float w = q.w, x = q.x, y = q.y, z = q.z;
    const float xx = mul_(x, x), yy = mul_(y, y), zz = mul_(z, z);
    const float xy = mul_(x, y), xz = mul_(x, z), yz = mul_(y, z);
    const float wx = mul_(w, x), wy = mul_(w, y), wz = mul_(w, z);
    *r0 = mk3(fma_(-2.0f, add_(yy, zz), 1.0f), mul_(2.0f, sub_(xy, wz)), mul_(2.0f, add_(xz, wy)));
    *r1 = mk3(mul_(2.0f, add_(xy, wz)), fma_(-2.0f, add_(xx, zz), 1.0f), mul_(2.0f, sub_(yz, wx)));
    *r2 = mk3(mul_(2.0f, sub_(xz, wy)), mul_(2.0f, add_(yz, wx)), fma_(-2.0f, add_(xx, yy), 1.0f));
}

// Packed constants as constant-bank operands: 1.9 (PE_CN_SLOPE), 1e-30 and -1, each twice.  As
// immediates every use takes two moves into a register pair (28 of a flight-step's 400 instructions).
static __constant__ unsigned long long c_k19 = 0x3ff333333ff33333ull, c_tiny = 0x0da242600da24260ull, c_mone = 0xbf800000bf800000ull;
// Per-step constants of the packed panel pass (both halves equal).
struct PairConst {
    f2 vbx, vby, vbz;     // body-frame air velocity
    f2 wbx, wby, wbz;     // body rates
    f2 nwbx, nwby, nwbz;  // negated body rates
    f2 k19, cf, tiny, mone;
};
// Packed partial sums of one virtual lane: even panels in the low half, odd in the high half.
//   fn = sum of -f;  tq = the positive half of rb x f's products, tp = the subtracted half
struct PairAcc {
    f2 fnx, fny, fnz, tqx, tqy, tqz, tpx, tpy, tpz;
};
__device__ __forceinline__ void pair_acc_zero(PairAcc& z) {
    z.fnx = z.fny = z.fnz = z.tqx = z.tqy = z.tqz = z.tpx = z.tpy = z.tpz = 0ull;
}

// -force of two panels (one pair) in the body frame.
__device__ __forceinline__ void pair_force(f2 rbx, f2 rby, f2 rbz, f2 ak, f2 nbx, f2 nby, f2 nbz, const PairConst& k,
                                           float k_cf_scalar, f2& nfx, f2& nfy, f2& nfz) {
    // vr = v_b + wb x rb
    const f2 vx = fma2(k.wby, rbz, fma2(k.nwbz, rby, k.vbx));
    const f2 vy = fma2(k.wbz, rbx, fma2(k.nwbx, rbz, k.vby));
    const f2 vz = fma2(k.wbx, rby, fma2(k.nwby, rbx, k.vbz));
    // |vr|^2 + 1e-30: finite 1/|vr| at rest, and below half an ulp of any |vr|^2 above ~1e-23
    const f2 V2 = fma2(vz, vz, fma2(vy, vy, fma2(vx, vx, k.tiny)));
    float v2a, v2b;
    upk(V2, v2a, v2b);
    const f2 inv = pk(rsqrtf(v2a), rsqrtf(v2b));
    const f2 vn = fma2(vz, nbz, fma2(vy, nby, mul2(vx, nbx)));
    const f2 s = mul2(vn, inv);
    const f2 qd = mul2(V2, ak);
    float sa, sb;
    upk(s, sa, sb);
    // s^2 - 1 for both panels in one packed FMA; its negation rounds exactly as 1 - s^2 would
    float ua, ub;
    upk(fma2(s, s, k.mone), ua, ub);
    const f2 sq = pk(sqrtf(fmaxf(0.0f, -ua)), sqrtf(fmaxf(0.0f, -ub)));
    // cn - cf s = s (1.9 sqrt(1 - s^2) + 2 |s| - cf)
    const f2 g = fma2(sq, k.k19, pk(__fmaf_rn(2.0f, fabsf(sa), -k_cf_scalar), __fmaf_rn(2.0f, fabsf(sb), -k_cf_scalar)));
    // -f = na nb + nb_ vr with na = qd (cn - cf s), nb_ = qd cf / |vr|
    const f2 na = mul2(mul2(qd, s), g);
    const f2 nv = mul2(mul2(qd, k.cf), inv);
    nfx = fma2(na, nbx, mul2(nv, vx));
    nfy = fma2(na, nby, mul2(nv, vy));
    nfz = fma2(na, nbz, mul2(nv, vz));
}

// Force and torque of a pair, added to the partial sums.  INIT writes them as the sums' first terms
// instead of adding them to +0: the two agree unless every term so far is -0, and then differ only in
// the sign of a zero sum.
template <bool INIT = false>
__device__ __forceinline__ void pair_eval(f2 rbx, f2 rby, f2 rbz, f2 ak, f2 nbx, f2 nby, f2 nbz, const PairConst& k,
                                          float k_cf_scalar, PairAcc& acc) {
    f2 nfx, nfy, nfz;
    pair_force(rbx, rby, rbz, ak, nbx, nby, nbz, k, k_cf_scalar, nfx, nfy, nfz);
    if (INIT) {  // the first pair of a virtual lane: the sums start from it, not from +0 + it
        acc.fnx = nfx; acc.fny = nfy; acc.fnz = nfz;
        acc.tqx = mul2(rbz, nfy); acc.tpx = mul2(rby, nfz);
        acc.tqy = mul2(rbx, nfz); acc.tpy = mul2(rbz, nfx);
        acc.tqz = mul2(rby, nfx); acc.tpz = mul2(rbx, nfy);
        return;
    }
    acc.fnx = add2(acc.fnx, nfx);
    acc.fny = add2(acc.fny, nfy);
    acc.fnz = add2(acc.fnz, nfz);
    // rb x f = (rbz nfy - rby nfz, rbx nfz - rbz nfx, rby nfx - rbx nfy)
    acc.tqx = fma2(rbz, nfy, acc.tqx);
    acc.tpx = fma2(rby, nfz, acc.tpx);
    acc.tqy = fma2(rbx, nfz, acc.tqy);
    acc.tpy = fma2(rbz, nfx, acc.tpy);
    acc.tqz = fma2(rby, nfx, acc.tqz);
    acc.tpz = fma2(rbx, nfy, acc.tpz);
}

// The same for pair q of a flight's staged panels.
template <bool INIT = false>
__device__ __forceinline__ void fast_pair(const PairedPanels& pp, int q, const PairConst& k, float k_cf_scalar, PairAcc& acc) {
    const float4 A = pp.a[q], B = pp.b[q], C = pp.c[q];
    const float2 D = pp.d[q];
    pair_eval<INIT>(pk(A.x, A.y), pk(A.z, A.w), pk(B.x, B.y), pk(B.z, B.w), pk(C.x, C.y), pk(C.z, C.w), pk(D.x, D.y), k,
                    k_cf_scalar, acc);
}

// Totals of one virtual lane: force and torque, even + odd partial sums.
__device__ __forceinline__ void pair_acc_total(const PairAcc& a, float out[6]) {
    float e, o, e2, o2;
    upk(a.fnx, e, o); out[0] = -add_(e, o);
    upk(a.fny, e, o); out[1] = -add_(e, o);
    upk(a.fnz, e, o); out[2] = -add_(e, o);
    upk(a.tqx, e, o); upk(a.tpx, e2, o2); out[3] = sub_(add_(e, o), add_(e2, o2));
    upk(a.tqy, e, o); upk(a.tpy, e2, o2); out[4] = sub_(add_(e, o), add_(e2, o2));
    upk(a.tqz, e, o); upk(a.tpz, e2, o2); out[5] = sub_(add_(e, o), add_(e2, o2));
}

// Sum over the 32 virtual lanes along one xor tree, identical on every lane of the group.
// The six components (+2 zero slots) are reduced transposed: each of the first three cross-lane
// levels halves the values a lane carries (4 + 2 + 1 shuffles), the last levels are plain
// butterflies, and six shuffles broadcast the totals: 19 shuffles instead of 30.
template <int LPF>
__device__ __forceinline__ void fast_reduce(float (&acc)[32 / LPF][6], unsigned mask, int j, float out[6]) {
    constexpr int NV = 32 / LPF;
    float v[8];
#pragma unroll
    for (int c = 0; c < 6; c++) v[c] = NV == 2 ? add_(acc[0][c], acc[NV - 1][c]) : acc[0][c];
    v[6] = 0.0f;
    v[7] = 0.0f;
#pragma unroll
    for (int lv = 0; lv < 3; lv++) {
        const int m = (LPF / 2) >> lv;
        const int half = 4 >> lv;
        const bool up = (j & m) != 0;
#pragma unroll
        for (int i = 0; i < half; i++) {
            const float send = up ? v[i] : v[i + half];
            const float keep = up ? v[i + half] : v[i];
            v[i] = add_(keep, __shfl_xor_sync(mask, send, m, LPF));
        }
    }
#pragma unroll
    for (int m = LPF / 16; m >= 1; m >>= 1) v[0] = add_(v[0], __shfl_xor_sync(mask, v[0], m, LPF));
#pragma unroll
    for (int c = 0; c < 6; c++) {
        const int src = ((c >> 2) & 1) * (LPF / 2) + ((c >> 1) & 1) * (LPF / 4) + (c & 1) * (LPF / 8);
        out[c] = __shfl_sync(mask, v[0], src, LPF);
    }
}

// What the forward pass of pe_grad keeps of a step: the body-frame aerodynamic force and torque,
// and at the last step how the flight ended (1 ground, 2 other bound or horizon, 3 NaN).
struct StepOut {
    float fb[6];
    int kind;
};

// What a step derives from its state before the panels: the attitude rows and the body-frame air
// velocity.
struct StepPre {
    vec3 r0, r1, r2;
    vec3 vb;
};

// R^T v: column k of R is (r0[k], r1[k], r2[k]).
__device__ __forceinline__ vec3 fast_body(vec3 r0, vec3 r1, vec3 r2, vec3 v) {
    return mk3(fma_(r2.x, v.z, fma_(r1.x, v.y, mul_(r0.x, v.x))), fma_(r2.y, v.z, fma_(r1.y, v.y, mul_(r0.y, v.x))),
               fma_(r2.z, v.z, fma_(r1.z, v.y, mul_(r0.z, v.x))));
}

// LANES: the gusts with one sine per lane (wl, of lane i mod 8 of the flight).
template <bool LANES = false>
__device__ __forceinline__ StepPre fast_pre(const FastConst& fc, FlightState& st, int step, const WindLane* wl = nullptr) {
    if (step > 0 && step % kChunk == 0) st.t = mul_((float)step, PE_DT);
    StepPre pre;
    fast_rows(st.q, &pre.r0, &pre.r1, &pre.r2);
    const vec3 wind = LANES ? wind_lanes(st.pos, mul_(wl->ct, st.t), *wl, fc.gust, fc.base_x, fc.base_y)
                            : fast_wind(st.pos, st.t, fc.phase, fc.gust, fc.base_x, fc.base_y);
    const vec3 va = mk3(sub_(st.vel.x, wind.x), sub_(st.vel.y, wind.y), sub_(st.vel.z, wind.z));
    pre.vb = fast_body(pre.r0, pre.r1, pre.r2, va);
    return pre;
}

__device__ __forceinline__ PairConst pair_const(const FastConst& fc, vec3 vb, vec3 wb) {
    PairConst k;
    k.vbx = bc(vb.x); k.vby = bc(vb.y); k.vbz = bc(vb.z);
    k.wbx = bc(wb.x); k.wby = bc(wb.y); k.wbz = bc(wb.z);
    k.nwbx = bc(-wb.x); k.nwby = bc(-wb.y); k.nwbz = bc(-wb.z);
    k.k19 = c_k19; k.cf = bc(fc.skin_cf); k.tiny = c_tiny; k.mone = c_mone;
    return k;
}

// The integrator's rotation: the gyroscopic torque of body rates w, then the next rates and attitude
// from the aerodynamic torque tb.
__device__ __forceinline__ vec3 fast_gyro(const FastConst& fc, vec3 w) {
    const vec3 Iw = mk3(fma_(fc.I[4], w.z, fma_(fc.I[3], w.y, mul_(fc.I[0], w.x))),
                        fma_(fc.I[5], w.z, fma_(fc.I[1], w.y, mul_(fc.I[3], w.x))),
                        fma_(fc.I[2], w.z, fma_(fc.I[5], w.y, mul_(fc.I[4], w.x))));
    return mk3(fma_(w.y, Iw.z, -mul_(w.z, Iw.y)), fma_(w.z, Iw.x, -mul_(w.x, Iw.z)), fma_(w.x, Iw.y, -mul_(w.y, Iw.x)));
}
// LATE: the limit on the rates is asked for after the attitude, so that a lone chain does not wait for the
// branch (3 % of a step of pe_flight_wide.cu; kernels that others' warps keep busy lose 4 % by it).
// A squared length safely below the limit's needs no root (a NaN takes the long way).
__device__ __forceinline__ bool fast_limit(vec3& v, float safe, float limit) {
    const float v2 = dot_(v, v);
    if (v2 < safe) return false;
    const float l = sqrtf(v2);
    if (!(l > limit)) return false;
    const float k = __fdiv_rn(limit, l);
    v = mk3(mul_(v.x, k), mul_(v.y, k), mul_(v.z, k));
    return true;
}
template <bool LATE = false>
__device__ __forceinline__ void fast_rotate(const FastConst& fc, vec3 gyro, vec3 tb, vec3& w, quat4& q) {
    const vec3 tq = mk3(sub_(tb.x, gyro.x), sub_(tb.y, gyro.y), sub_(tb.z, gyro.z));
    const vec3 dw = mk3(fma_(fc.invI[2], tq.z, fma_(fc.invI[1], tq.y, mul_(fc.invI[0], tq.x))),
                        fma_(fc.invI[5], tq.z, fma_(fc.invI[4], tq.y, mul_(fc.invI[3], tq.x))),
                        fma_(fc.invI[8], tq.z, fma_(fc.invI[7], tq.y, mul_(fc.invI[6], tq.x))));
    w = mk3(fma_(dw.x, PE_DT, w.x), fma_(dw.y, PE_DT, w.y), fma_(dw.z, PE_DT, w.z));
    if (!LATE) fast_limit(w, 22499.f, 150.f);
    // q += 0.5 dt q (0, w); normalize
    auto turn = [&](vec3 v) {
        const float h = mul_(0.5f, PE_DT);
        const float dqw = -fma_(q.z, v.z, fma_(q.y, v.y, mul_(q.x, v.x)));
        const float dqx = fma_(q.y, v.z, fma_(-q.z, v.y, mul_(q.w, v.x)));
        const float dqy = fma_(q.z, v.x, fma_(-q.x, v.z, mul_(q.w, v.y)));
        const float dqz = fma_(q.x, v.y, fma_(-q.y, v.x, mul_(q.w, v.z)));
        const quat4 qn = mkq(fma_(h, dqw, q.w), fma_(h, dqx, q.x), fma_(h, dqy, q.y), fma_(h, dqz, q.z));
        const float il = rsqrtf(fma_(qn.z, qn.z, fma_(qn.y, qn.y, fma_(qn.x, qn.x, mul_(qn.w, qn.w)))));
        return mkq(mul_(qn.w, il), mul_(qn.x, il), mul_(qn.y, il), mul_(qn.z, il));
    };
    quat4 next = turn(w);
    if (LATE && fast_limit(w, 22499.f, 150.f)) next = turn(w);
    q = next;
}
// The integrator's translation from the world-frame aerodynamic force Fs.
template <bool LATE = false>
__device__ __forceinline__ void fast_translate(const FastConst& fc, vec3 Fs, vec3& vel, vec3& pos) {
    Fs.z = fma_(-fc.mass, PE_GRAV, Fs.z);
    const float kv = mul_(fc.invmass, PE_DT);
    vel = mk3(fma_(Fs.x, kv, vel.x), fma_(Fs.y, kv, vel.y), fma_(Fs.z, kv, vel.z));
    if (!LATE) fast_limit(vel, 3599.f, 60.f);
    const vec3 from = pos;
    auto move = [&]() { pos = mk3(fma_(vel.x, PE_DT, from.x), fma_(vel.y, PE_DT, from.y), fma_(vel.z, PE_DT, from.z)); };
    move();
    if (LATE && fast_limit(vel, 3599.f, 60.f)) move();
}
// Whether the flight ends at `step`.
__device__ __forceinline__ bool fast_over(vec3 pos, vec3 vel, int step, int max_steps) {
    return !(pos.x == pos.x && vel.x == vel.x) | (pos.z <= 0.0f) | (fabsf(pos.y) > 300.f) | (pos.x < -50.f) |
           (step == max_steps - 1);
}
// How the flight ends at `step` (0: it goes on; 1 ground, 2 other bound or horizon, 3 NaN) and its
// distance.
__device__ __forceinline__ int fast_end(vec3 p0, vec3 pos, vec3 vel, int step, int max_steps, int smooth, float* fit) {
    const int bad = !(pos.x == pos.x && vel.x == vel.x);
    if (pos.z <= 0.0f || bad || fabsf(pos.y) > 300.f || pos.x < -50.f) {
        *fit = bad ? -10.0f : pos.x;
        if (smooth && !bad && pos.z <= 0.0f) {  // the z = 0 crossing between the last two states
            const float a = __fdiv_rn(p0.z, sub_(p0.z, pos.z));
            *fit = fma_(sub_(pos.x, p0.x), a, p0.x);
        }
        return bad ? 3 : (pos.z <= 0.0f ? 1 : 2);
    }
    if (step == max_steps - 1) {
        *fit = pos.x;
        return 2;
    }
    return 0;
}

// The integrator and the end of the flight, from the step's body-frame force and torque sum[6].
// Returns 1 when the flight ends at `step`.
__device__ __forceinline__ int fast_post(const FastConst& fc, const StepPre& pre, const float sum[6], FlightState& st,
                                         int step, int max_steps, int smooth, float* fit, float sumw[6], StepOut* so) {
    const vec3 r0 = pre.r0, r1 = pre.r1, r2 = pre.r2;
    const vec3 Fb = mk3(sum[0], sum[1], sum[2]);
    const vec3 tb = mk3(sum[3], sum[4], sum[5]);
    if (so) {
#pragma unroll
        for (int c = 0; c < 6; c++) so->fb[c] = sum[c];
    }
    // world force for the translational update; the rotational update takes the body torque
    const vec3 Fs = mk3(dot_(r0, Fb), dot_(r1, Fb), dot_(r2, Fb));
    if (sumw) {
        sumw[0] = Fs.x; sumw[1] = Fs.y; sumw[2] = Fs.z;
        sumw[3] = dot_(r0, tb); sumw[4] = dot_(r1, tb); sumw[5] = dot_(r2, tb);
    }
    const vec3 p0 = st.pos;
    fast_rotate(fc, fast_gyro(fc, st.wb), tb, st.wb, st.q);
    fast_translate(fc, Fs, st.vel, st.pos);
    st.t = add_(st.t, PE_DT);
    const int kind = fast_end(p0, st.pos, st.vel, step, max_steps, smooth, fit);
    if (so && kind) so->kind = kind;
    return kind != 0;
}

template <int LPF>
__device__ __forceinline__ int fast_step(const FastConst& fc, const PairedPanels& pp, int nt, int j,
                                         unsigned mask, FlightState& st, int step, int max_steps, int smooth,
                                         float* fit, float sumw[6], StepOut* so = nullptr) {
    const StepPre pre = fast_pre(fc, st, step);
    const PairConst k = pair_const(fc, pre.vb, st.wb);
    constexpr int NV = 32 / LPF;
    // pass n reads pair j + LPF n, of virtual lane j + LPF (n % NV); the same count on every lane
    const int passes = ((nt + 1) / 2 + LPF - 1) / LPF;
    float acc[NV][6];
    if constexpr (NV == 2) {
        PairAcc p0, p1;
        int n = 0;
        if (passes >= 2) {
            fast_pair<true>(pp, j, k, fc.skin_cf, p0);
            fast_pair<true>(pp, j + LPF, k, fc.skin_cf, p1);
            n = 2;
        } else {
            pair_acc_zero(p0);
            pair_acc_zero(p1);
        }
        for (; n + 1 < passes; n += 2) {
            fast_pair(pp, j + LPF * n, k, fc.skin_cf, p0);
            fast_pair(pp, j + LPF * (n + 1), k, fc.skin_cf, p1);
        }
        if (n < passes) fast_pair(pp, j + LPF * n, k, fc.skin_cf, p0);
        pair_acc_total(p0, acc[0]);
        pair_acc_total(p1, acc[NV - 1]);
    } else {
        PairAcc p0;
        int n = 0;
        if (passes >= 1) {
            fast_pair<true>(pp, j, k, fc.skin_cf, p0);
            n = 1;
        } else {
            pair_acc_zero(p0);
        }
#pragma unroll 2
        for (; n < passes; n++) fast_pair(pp, j + LPF * n, k, fc.skin_cf, p0);
        pair_acc_total(p0, acc[0]);
    }
    float sum[6];
    fast_reduce<LPF>(acc, mask, j, sum);
    return fast_post(fc, pre, sum, st, step, max_steps, smooth, fit, sumw, so);
}

template <int LPF>
__device__ __forceinline__ unsigned fast_mask(int lane) {
    return LPF == 32 ? 0xffffffffu : (0xffffu << (lane & 16));
}

}  // namespace pe
