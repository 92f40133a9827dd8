// pe_grad_common.cuh -- what the gradient's kernels share: a flight's constants, states and per-step
// entries in memory (pe_grad.cu: the forward set-up, the serial reverse passes and the genome
// contraction; pe_grad_time.cu: the reverse pass parallel in time).
#pragma once
#include <cuda_runtime.h>

#include "pe_grad_model.h"
#include "pe_internal.cuh"

namespace pe {

namespace {

using F3 = pg::V3<float>;
using FSt = pg::St<float>;

constexpr int kPanelFloats = 7 * kNtMax;  // rbx rby rbz nbx nby nbz ak (SoA)
constexpr int kSegFloats = 20;            // state (14) + body force (3) + body torque (3)
constexpr int kCkFloats = 16;             // one checkpointed state

__device__ __forceinline__ float warp_sum(float v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ FSt zero_state() {
    FSt z;
    z.pos = pg::v3(0.f, 0.f, 0.f);
    z.vel = z.pos;
    z.w = z.pos;
    z.q[0] = z.q[1] = z.q[2] = z.q[3] = 0.f;
    z.t = 0.f;
    return z;
}

// Constants of one flight: scenario draw, print variation, gust phase.
struct FlightCtx {
    pg::FlightP<float> P;
    F3 cg;
    float sigma, beta[6];
    float sc[kScenN];
    int nt, off;
};

__device__ __forceinline__ void flight_setup(const GradArgs& a, int f, FlightCtx& c) {
    const int p = f / a.nseeds, s = f - p * a.nseeds;
    const int seed = a.seeds[s] + (a.vary ? p * 7919 : 0);
    Scenario S;
    scenario_desc(seed, &S);
#pragma unroll
    for (int k = 0; k < kScenN; k++) c.sc[k] = S.v[k];
    const float* mp = a.plane_mp + (size_t)p * kMpN;
    float I[6];
#pragma unroll
    for (int k = 0; k < 6; k++) I[k] = mp[5 + k];
    pg::printed(c.sc, mp[0], I, c.P, &c.cg, &c.sigma, c.beta);
    c.P.phase = seed_phase(seed);
    c.nt = a.plane_nt[p];
    c.off = a.plane_off[p];
}

// A flight's constants as k_grad_setup wrote them: the forward pass flew with these, and every
// reverse kernel takes them from here rather than from its own flight_setup, whose rounding may
// differ in the last place with how the compiler fuses it into each kernel.
__device__ __forceinline__ pg::FlightP<float> setup_flightp(const GradArgs& a, int f) {
    const float* r = a.setup + (size_t)f * kGradSetupFloats;
    pg::FlightP<float> P;
    P.mass = r[0];
    P.invmass = r[1];
#pragma unroll
    for (int k = 0; k < 6; k++) P.I[k] = r[2 + k];
#pragma unroll
    for (int k = 0; k < 9; k++) P.invI[k] = r[8 + k];
    P.cf = r[17];
    P.phase = r[18];
    P.gust = r[19];
    P.base_x = r[20];
    P.base_y = r[21];
    return P;
}

__device__ __forceinline__ void store_state16(float* dst, const FSt& s) {
    float4* d4 = reinterpret_cast<float4*>(dst);
    d4[0] = make_float4(s.pos.x, s.pos.y, s.pos.z, s.q[0]);
    d4[1] = make_float4(s.q[1], s.q[2], s.q[3], s.vel.x);
    d4[2] = make_float4(s.vel.y, s.vel.z, s.w.x, s.w.y);
    d4[3] = make_float4(s.w.z, s.t, 0.f, 0.f);
}
__device__ __forceinline__ FSt load_state16(const float* src) {
    const float4* s4 = reinterpret_cast<const float4*>(src);
    const float4 a = s4[0], b = s4[1], c = s4[2], d = s4[3];
    FSt s;
    s.pos = pg::v3(a.x, a.y, a.z);
    s.q[0] = a.w; s.q[1] = b.x; s.q[2] = b.y; s.q[3] = b.z;
    s.vel = pg::v3(b.w, c.x, c.y);
    s.w = pg::v3(c.z, c.w, d.x);
    s.t = d.y;
    return s;
}
// A step's body force and torque as the forward pass stores them (2 float4).
__device__ __forceinline__ void store_fsum(float* dst, F3 F, F3 T) {
    float4* d4 = reinterpret_cast<float4*>(dst);
    d4[0] = make_float4(F.x, F.y, F.z, T.x);
    d4[1] = make_float4(T.y, T.z, 0.f, 0.f);
}
__device__ __forceinline__ void load_fsum(const float* src, F3* F, F3* T) {
    const float4* s4 = reinterpret_cast<const float4*>(src);
    const float4 a = s4[0], b = s4[1];
    *F = pg::v3(a.x, a.y, a.z);
    *T = pg::v3(a.w, b.x, b.y);
}
__device__ __forceinline__ void put3(float* d, F3 v) { d[0] = v.x; d[1] = v.y; d[2] = v.z; }
__device__ __forceinline__ F3 get3(const float* d) { return pg::v3(d[0], d[1], d[2]); }
}  // namespace

}  // namespace pe
