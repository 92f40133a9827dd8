// pe_grad_time.cu -- pe_grad's reverse pass with the panel work parallel in time.
//
// A flight's adjoint is a chain back over its steps, and the serial kernels of pe_grad.cu carry the
// panels' adjoint inside it: two block barriers and a panel pass per step, 1.3 us a step, 1.8 ms for the
// longest of 256 x 8 flights.  But the panels enter the chain only through the step's (force, torque) as
// a function of the body air velocity and body rates, whose 6 x 6 Jacobian depends on the forward flight
// alone.  So:
//   k_adj_states    thread per segment: the state before every step, from the checkpoint and the stored
//                   forces through this model's integrator (as the serial kernels rebuild them);
//   k_adj_jacobian  lane per step: the sum over the panels of that Jacobian, then the adjoint of the whole
//                   step as a 13 x 10 matrix, column by column through the model's own adjoint functions;
//   k_adj_chain     a warp per flight, a component per lane: ten shuffles and ten FMAs a step, no barrier;
//                   leaves the adjoint of every state;
//   k_adj_panels    block per 128 steps of a flight, a pair or two per lane: the panels' own adjoints and the
//                   mass properties', sums over steps that no longer feed the chain.
// With v = vb + w x r, B = [I; [r]x] and the panel force f = -(na n + nv v), na and nv functions of v,
//   d(na)/dv = alpha n + beta v,  d(nv)/dv = gamma v,
//   (Lvb; Lw) = -G (LF; LT),  G = sum of (alpha N + beta V) N^T + gamma V V^T + nv B B^T
// over the panels, N = B n, V = B v.
//
// The records take 633 bytes per flight-step (kAdjEnt floats, and kAdjChunk per 32 steps) for the first
// kAdjSteps steps of every flight; longer flights take the serial kernel, and so do all where the records and
// the adjoints' parts do not fit kAdjBytes, and most calls of horizons below 96 steps (pe_grad).
// Built without fast math, as pe_grad.cu.
//
// Measured (GB300, 256 x 8 x 3600 / 64 x 8 x 7200): states 0.05 / 0.04 ms, Jacobians 0.94 / 0.29, chain
// 0.10 / 0.08 (with the model's adjoint in the chain, eight lanes a flight: 0.74 / 0.66), panels 0.77 /
// 0.27 (512 steps a block: 0.81 / 0.46, for want of blocks); the call 4.03 -> 3.25 ms and 2.63 -> 1.40 ms, and 3.06 and 1.30 since parts of 128 steps and
// k_grad_genome's corner adjoints.  The Jacobians and the panels are bound by register reads (a scalar FMA of
// three registers takes two cycles of the two banks, a packed one three), not by the pipe: 163 instructions
// per panel and 32 steps take 224 cycles.
#include <cuda_runtime.h>

#include <type_traits>

#include "pe_f32x2.cuh"
#include "pe_grad_common.cuh"

namespace pe {

namespace {

// A step's entry: [0..13] the state before it, [16..21] its force and torque, vb at [15] [22] [23].
__device__ __forceinline__ float* adj_ent(const GradArgs& a, int f, int j) {
    return a.rec + ((size_t)f * a.rec_steps + j) * kAdjEnt;
}
// Matrices of 32 steps: element (row i, column c) of step j at [(13 c + i) * 33 + j % 32]; a lane per step
// writes rows of 32, a lane per component reads without bank conflicts.  The chain replaces the first
// 16 floats per step by the adjoint of the state after the step: pos, vel + dt pos, w, q.
constexpr int kMatRows = 13, kMatCols = 10, kMatElems = kMatRows * kMatCols;
static_assert(kAdjChunk >= 33 * kMatElems && kAdjChunk % 4 == 0, "a chunk holds its matrices in whole vectors");
__device__ __forceinline__ float* adj_chunk(const GradArgs& a, int f, int chunk) {
    return a.rec + (size_t)a.n_flights * a.rec_steps * kAdjEnt + ((size_t)f * (a.rec_steps / 32) + chunk) * kAdjChunk;
}
__device__ __forceinline__ void load_ent(const float* e, FSt& s, F3* F, F3* T, F3* vb) {
    const float4* e4 = reinterpret_cast<const float4*>(e);
    const float4 d = e4[3], f0 = e4[4], f1 = e4[5];
    s = load_state16(e);
    *F = pg::v3(f0.x, f0.y, f0.z);
    *T = pg::v3(f0.w, f1.x, f1.y);
    if (vb) *vb = pg::v3(d.w, f1.z, f1.w);
}
// Whether this pass differentiates flight f (the serial kernel takes the longer ones).
__device__ __forceinline__ bool adj_takes(const GradArgs& a, int f) {
    const int kind = a.kind[f];
    return (kind == 1 || kind == 2) && a.steps[f] <= a.rec_steps;
}
__device__ __forceinline__ float fast_rsqrt(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// ------------------------------------------------------------------ states
__global__ void __launch_bounds__(64) k_adj_states(GradArgs a, int nseg) {
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int f = (int)(id / nseg), seg = (int)(id - (long long)f * nseg);
    if (f >= a.n_flights) return;
    const int k = a.steps[f] - 1, j0 = seg * a.K;
    if (j0 > k || !adj_takes(a, f)) return;
    const int j1 = min(j0 + a.K - 1, k);
    const pg::FlightP<float> P = setup_flightp(a, f);
    FSt cur = load_state16(a.ck + ((size_t)f * a.nck + seg) * kCkFloats);
    int to_chunk = kChunk - j0 % kChunk;
    const float* fs = a.fsum + (size_t)f * a.max_steps * 8;
    F3 Fn, Tn;  // the next step's, asked for a step ahead
    load_fsum(fs + (size_t)j0 * 8, &Fn, &Tn);
    for (int j = j0; j <= j1; j++) {
        float* e = adj_ent(a, f, j);
        const F3 Fb = Fn, Tb = Tn;
        load_fsum(fs + (size_t)min(j + 1, j1) * 8, &Fn, &Tn);
        store_state16(e, cur);
        store_fsum(e + 16, Fb, Tb);
        pg::M3<float> R;
        pg::rot_rows(cur.q, R);
        pg::PostF<float> pf;
        const FSt nx = pg::step_post_f(P, cur, R, Fb, Tb, pf);
        if (j == k) {
            store_state16(a.after + (size_t)f * 16, nx);
        } else {
            cur = nx;
            if (--to_chunk == 0) { cur.t = (float)(j + 1) * pg::kDt; to_chunk = kChunk; }  // src/sim.cu:113
        }
    }
}

// ------------------------------------------------------------------ work items
constexpr int kJacSteps = 64;  // steps (threads) per item of the Jacobians
static_assert(kAdjSteps % kAdjPart == 0 && kAdjPart % 32 == 0 && kAdjSteps % kJacSteps == 0 && kAdjSteps / kJacSteps <= 64,
              "an item is flight * 64 + part");

// items[] = flight * 64 + part for every kJacSteps steps of every flight to differentiate, longest
// flights first, and behind cap for every kAdjPart steps (at least one: constant distances are zeroed
// there); their counts to work[5] and work[7].
__global__ void __launch_bounds__(1024) k_adj_items(GradArgs a, long long cap) {
    __shared__ int warp_tot[32][2];
    __shared__ int s_base[2];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tid < 2) s_base[tid] = 0;
    __syncthreads();
    for (int i0 = 0; i0 < a.n_flights; i0 += 1024) {
        int f = 0, n[2] = {0, 0}, x[2];
        if (i0 + tid < a.n_flights) {
            f = a.order[i0 + tid];
            const int kind = a.kind[f], steps = a.steps[f];
            const bool takes = adj_takes(a, f);
            n[0] = takes ? (steps + kJacSteps - 1) / kJacSteps : 0;
            n[1] = takes ? (steps + kAdjPart - 1) / kAdjPart : (kind == 0 || kind == 3 ? 1 : 0);
        }
#pragma unroll
        for (int q = 0; q < 2; q++) {
            x[q] = n[q];
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x[q], o);
                if (lane >= o) x[q] += y;
            }
            if (lane == 31) warp_tot[w][q] = x[q];
        }
        __syncthreads();
        if (w < 2) {
            int t = warp_tot[lane][w];
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= o) t += y;
            }
            warp_tot[lane][w] = t;
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int at = s_base[q] + x[q] - n[q] + (w > 0 ? warp_tot[w - 1][q] : 0);
            for (int i = 0; i < n[q]; i++) a.items[q * cap + at + i] = f * 64 + i;
        }
        __syncthreads();
        if (tid < 2) s_base[tid] += warp_tot[31][tid];
        __syncthreads();
    }
    if (tid < 2) a.work[5 + 2 * tid] = s_base[tid];
}

// ------------------------------------------------------------------ Jacobians
constexpr int kJacBlocks = 8;  // per SM
struct JacPanel {
    float4 r, n, m;  // (rb, 0.5 rho A), (normal, skin friction x 0.5 rho A), (rb x normal, -)
};

__global__ void __launch_bounds__(kJacSteps, kJacBlocks) k_adj_jacobian(GradArgs a) {
    __shared__ JacPanel sp[kNtMax];
    __shared__ int s_item;
    const int tid = threadIdx.x;
    const int count = a.work[5];
    for (;;) {
        __syncthreads();
        if (tid == 0) s_item = atomicAdd(&a.work[6], 1);
        __syncthreads();
        if (s_item >= count) break;
        const int item = a.items[s_item];
        const int f = item >> 6, part = item & 63;
        const int p = f / a.nseeds;
        const int nt = a.plane_nt[p], off = a.plane_off[p], k = a.steps[f] - 1;
        const float* rec = a.setup + (size_t)f * kGradSetupFloats;
        const F3 cg = pg::v3(rec[22], rec[23], rec[24]);
        for (int i = tid; i < nt; i += kJacSteps) {
            const float4 c4 = a.pc[off + i], n4 = a.pn[off + i];
            F3 rb, nb;
            float ak;
            pg::stage(pg::v3(c4.x, c4.y, c4.z), c4.w, pg::v3(n4.x, n4.y, n4.z), cg, rec[25], rec[26], rec[27], &rb, &nb, &ak);
            const F3 m = pg::cross(rb, nb);
            sp[i].r = make_float4(rb.x, rb.y, rb.z, ak);
            sp[i].n = make_float4(nb.x, nb.y, nb.z, rec[17] * ak);
            sp[i].m = make_float4(m.x, m.y, m.z, 0.f);
        }
        __syncthreads();
        const int j = part * kJacSteps + tid;
        const bool on = j <= k;
        if (!__any_sync(0xffffffffu, on)) continue;  // a warp past the flight's end
        float* e = adj_ent(a, f, on ? j : k);
        F3 vb, w;
        {
            const pg::FlightP<float> P = setup_flightp(a, f);
            const FSt st = load_state16(e);
            pg::Pre<float> q;
            pg::step_pre(P, st, q);
            if (on) { e[15] = q.vb.x; e[22] = q.vb.y; e[23] = q.vb.z; }
            vb = q.vb;
            w = q.w;
        }
        const float cf = rec[17];
        // P N^T in full, V V^T's upper triangle, and the moments of nv
        float A[6][6], S[21], E0 = 0.f, E1[3] = {0.f, 0.f, 0.f}, E2[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int r = 0; r < 6; r++)
#pragma unroll
            for (int c = 0; c < 6; c++) A[r][c] = 0.f;
#pragma unroll
        for (int r = 0; r < 21; r++) S[r] = 0.f;
#pragma unroll 1
        for (int i = 0; i < nt; i++) {
            const float4 r = sp[i].r, n = sp[i].n, m = sp[i].m;
            const float vx = fmaf(w.y, r.z, fmaf(-w.z, r.y, vb.x));
            const float vy = fmaf(w.z, r.x, fmaf(-w.x, r.z, vb.y));
            const float vz = fmaf(w.x, r.y, fmaf(-w.y, r.x, vb.z));
            const float V2 = fmaf(vz, vz, fmaf(vy, vy, fmaf(vx, vx, 1e-30f)));
            const float inv = fast_rsqrt(V2);
            const float V1 = V2 * inv;
            const float s = fmaf(vz, n.z, fmaf(vy, n.y, vx * n.x)) * inv;
            const float u = fmaf(-s, s, 1.f);
            // sqrt(u) and s^2 / sqrt(u), the latter dropped where the root's slope is not taken
            const float rs = fast_rsqrt(fmaxf(u, 1e-12f));
            const bool in = u > 1e-12f;
            const float sq = in ? u * rs : 0.f;
            const float as2 = 2.f * fabsf(s);
            const float gf = fmaf(1.9f, sq, as2 - cf);
            const float x = in ? 1.9f * s * s * rs : 0.f;  // D = gf + 2 |s| - x
            const float akV = r.w * V1;
            const float al = akV * (gf + as2 - x);
            const float be = r.w * s * (gf - as2 + x);     // ak s (2 gf - D)
            const float ga = n.w * inv, nv = cf * akV;
            const float V[6] = {vx, vy, vz, fmaf(r.y, vz, -r.z * vy), fmaf(r.z, vx, -r.x * vz), fmaf(r.x, vy, -r.y * vx)};
            const float N[6] = {n.x, n.y, n.z, m.x, m.y, m.z};
            float Q[6];
#pragma unroll
            for (int q = 0; q < 6; q++) {
                const float Pq = fmaf(be, V[q], al * N[q]);
                Q[q] = ga * V[q];
#pragma unroll
                for (int c = 0; c < 6; c++) A[q][c] = fmaf(Pq, N[c], A[q][c]);
            }
            int at = 0;
#pragma unroll
            for (int q = 0; q < 6; q++)
#pragma unroll
                for (int c = q; c < 6; c++, at++) S[at] = fmaf(Q[q], V[c], S[at]);
            E0 += nv;
            const float nx = nv * r.x, ny = nv * r.y, nz = nv * r.z;
            E1[0] += nx; E1[1] += ny; E1[2] += nz;
            E2[0] = fmaf(nx, r.x, E2[0]); E2[1] = fmaf(ny, r.y, E2[1]); E2[2] = fmaf(nz, r.z, E2[2]);
            E2[3] = fmaf(nx, r.y, E2[3]); E2[4] = fmaf(nx, r.z, E2[4]); E2[5] = fmaf(ny, r.z, E2[5]);
        }
        {
            int at = 0;
#pragma unroll
            for (int q = 0; q < 6; q++)
#pragma unroll
                for (int c = q; c < 6; c++, at++) {
                    A[q][c] += S[at];
                    if (c != q) A[c][q] += S[at];
                }
            // nv B B^T: [I, -[r]x; [r]x, |r|^2 - r r^T]
#pragma unroll
            for (int q = 0; q < 3; q++) A[q][q] += E0;
            A[3][1] -= E1[2]; A[3][2] += E1[1]; A[4][0] += E1[2]; A[4][2] -= E1[0]; A[5][0] -= E1[1]; A[5][1] += E1[0];
            A[1][3] -= E1[2]; A[2][3] += E1[1]; A[0][4] += E1[2]; A[2][4] -= E1[0]; A[0][5] -= E1[1]; A[1][5] += E1[0];
            A[3][3] += E2[1] + E2[2]; A[4][4] += E2[0] + E2[2]; A[5][5] += E2[0] + E2[1];
            A[3][4] -= E2[3]; A[4][3] -= E2[3]; A[3][5] -= E2[4]; A[5][3] -= E2[4]; A[4][5] -= E2[5]; A[5][4] -= E2[5];
        }
        // The step's adjoint, one column per unit vector of (vel + dt pos, w, q) after the step; the
        // position's own adjoint passes through and is the chain's to add.
        const pg::FlightP<float> P = setup_flightp(a, f);
        FSt st;
        F3 Fb, Tb;
        load_ent(e, st, &Fb, &Tb, nullptr);
        pg::Pre<float> pr;
        float Jw[3][3];
        pg::step_pre(P, st, pr, Jw);
        pg::PostF<float> pf;
        (void)pg::step_post_f(P, st, pr.R, Fb, Tb, pf);
        float* out = adj_chunk(a, f, j >> 5) + (tid & 31);
#pragma unroll 1
        for (int c = 0; c < kMatCols; c++) {
            FSt L1 = zero_state(), L0 = zero_state();
            L1.vel = pg::v3(c == 0 ? 1.f : 0.f, c == 1 ? 1.f : 0.f, c == 2 ? 1.f : 0.f);
            L1.w = pg::v3(c == 3 ? 1.f : 0.f, c == 4 ? 1.f : 0.f, c == 5 ? 1.f : 0.f);
#pragma unroll
            for (int q = 0; q < 4; q++) L1.q[q] = c == 6 + q ? 1.f : 0.f;
            pg::M3<float> LR;
#pragma unroll
            for (int r = 0; r < 3; r++)
#pragma unroll
                for (int q = 0; q < 3; q++) LR.a[r][q] = 0.f;
            pg::LamP<float> LP = {};
            F3 LF, LT;
            pg::step_post_adj_f(P, st, pr.R, Fb, pf, L1, L0, &LF, &LT, LR, LP);
            float z[6];
#pragma unroll
            for (int q = 0; q < 6; q++)
                z[q] = -(A[q][0] * LF.x + A[q][1] * LF.y + A[q][2] * LF.z + A[q][3] * LT.x + A[q][4] * LT.y + A[q][5] * LT.z);
            pg::step_pre_adj(P, st, pr, pg::v3(z[0], z[1], z[2]), pg::v3(z[3], z[4], z[5]), LR, L0, Jw);
            const float v[kMatRows] = {L0.pos.x, L0.pos.y, L0.pos.z,
                                       fmaf(pg::kDt, L0.pos.x, L0.vel.x), fmaf(pg::kDt, L0.pos.y, L0.vel.y),
                                       fmaf(pg::kDt, L0.pos.z, L0.vel.z),
                                       L0.w.x, L0.w.y, L0.w.z, L0.q[0], L0.q[1], L0.q[2], L0.q[3]};
#pragma unroll
            for (int i = 0; i < kMatRows; i++) out[(kMatRows * c + i) * 33] = v[i];
        }
    }
}

// ------------------------------------------------------------------ the chain
__device__ __forceinline__ void copy16(float* dst, const float* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// Lane i < 13 carries component i of the state's adjoint: position (0..2), velocity + dt position (3..5),
// body rates (6..8), attitude (9..12).  Chunks of 32 steps' matrices arrive one ahead.
__global__ void __launch_bounds__(32) k_adj_chain(GradArgs a) {
    extern __shared__ __align__(16) float buf[];  // [2][kAdjChunk]
    const int lane = threadIdx.x, row = min(lane, kMatRows - 1);
    const int f = a.order[blockIdx.x];
    if (!adj_takes(a, f)) return;
    const int k = a.steps[f] - 1, kind = a.kind[f];
    auto fetch = [&](int c) {
        if (c >= 0) {
            const float* src = adj_chunk(a, f, c);
            float* dst = buf + (c & 1) * kAdjChunk;
            for (int q = lane; q < kAdjChunk / 4; q += 32) copy16(dst + 4 * q, src + 4 * q);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int last = k >> 5;
    fetch(last);
    fetch(last - 1);
    float lam = 0.f, lb = 0.f;  // lb: the distance's adjoint of the state before the last step
    {
        FSt Lb = zero_state(), L = Lb;
        const FSt before = load_state16(adj_ent(a, f, k)), after = load_state16(a.after + (size_t)f * 16);
        pg::terminate_adj(before, after, kind, Lb, L);
        const int x = lane % 3;
        const float p = x == 0 ? L.pos.x : (x == 1 ? L.pos.y : L.pos.z);
        const float q = x == 0 ? Lb.pos.x : (x == 1 ? Lb.pos.y : Lb.pos.z);
        lam = lane < 3 ? p : (lane < 6 ? pg::kDt * p : 0.f);
        lb = lane < 3 ? q : (lane < 6 ? pg::kDt * q : 0.f);
    }
    for (int c = last; c >= 0; c--) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        const float* m = buf + (c & 1) * kAdjChunk + row * 33;
        float* keep = adj_chunk(a, f, c);
        for (int t = min(k - 32 * c, 31); t >= 0; t--) {
            if (lane < 16) keep[16 * t + lane] = lam;
            // the position's adjoint passes through, into vel + dt pos too
            const float p = __shfl_sync(0xffffffffu, lam, lane >= 3 && lane < 6 ? lane - 3 : lane);
            float s0 = lane < 3 ? lam : (lane < 6 ? pg::kDt * p : 0.f), s1 = 0.f;
#pragma unroll
            for (int q = 0; q < kMatCols; q += 2) {
                s0 = fmaf(m[(kMatRows * q) * 33 + t], __shfl_sync(0xffffffffu, lam, 3 + q), s0);
                s1 = fmaf(m[(kMatRows * (q + 1)) * 33 + t], __shfl_sync(0xffffffffu, lam, 4 + q), s1);
            }
            lam = s0 + s1 + lb;
            lb = 0.f;
        }
        __syncwarp();  // every lane has read the chunk's buffer
        fetch(c - 2);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (lane < 16) a.after[(size_t)f * 16 + lane] = lam;  // the adjoint of the release state
}

// ------------------------------------------------------------------ panels
constexpr int kPanWarps = 3, kPanThreads = 32 * kPanWarps;
constexpr int kPanSteps = 32 * kPanWarps;  // steps staged at a time, 32 by each warp
constexpr int kPanValues = 18;  // vb, w, -w, -LF, LT, -LT, each twice

struct PanPair {
    f2 rx, ry, rz, nx, ny, nz, ak;
};
struct PanAcc {
    f2 rx, ry, rz, nx, ny, nz, ak;
};

// The adjoints of a pair's panels at one step, added to acc.
__device__ __forceinline__ void pan_pair(const PanPair& p, const f2* k, f2 cf, PanAcc& acc) {
    const f2 vx = fma2(k[4], p.rz, fma2(k[8], p.ry, k[0]));
    const f2 vy = fma2(k[5], p.rx, fma2(k[6], p.rz, k[1]));
    const f2 vz = fma2(k[3], p.ry, fma2(k[7], p.rx, k[2]));
    const f2 V2 = fma2(vz, vz, fma2(vy, vy, fma2(vx, vx, bc(1e-30f))));
    float a, b;
    upk(V2, a, b);
    const f2 inv = pk(fast_rsqrt(a), fast_rsqrt(b));
    const f2 V1 = mul2(V2, inv);
    const f2 s = mul2(fma2(vz, p.nz, fma2(vy, p.ny, mul2(vx, p.nx))), inv);
    float sa, sb, ua, ub;
    upk(s, sa, sb);
    upk(fma2(s, s, bc(-1.f)), ua, ub);
    ua = -ua;
    ub = -ub;
    const float ra = fast_rsqrt(fmaxf(ua, 1e-12f)), rb = fast_rsqrt(fmaxf(ub, 1e-12f));
    const bool ia = ua > 1e-12f, ib = ub > 1e-12f;
    const f2 sq = pk(ia ? ua * ra : 0.f, ib ? ub * rb : 0.f);
    const f2 as2 = pk(2.f * fabsf(sa), 2.f * fabsf(sb));
    const f2 gf = fma2(bc(1.9f), sq, sub2(as2, cf));
    const f2 D = sub2(add2(gf, as2), pk(ia ? 1.9f * sa * sa * ra : 0.f, ib ? 1.9f * sb * sb * rb : 0.f));
    const f2 h1 = mul2(mul2(V2, s), gf), h2 = mul2(V1, cf);
    const f2 na = mul2(p.ak, h1), nv = mul2(p.ak, h2);
    const f2 al = mul2(mul2(p.ak, V1), D);
    const f2 be = mul2(mul2(p.ak, s), sub2(add2(gf, gf), D));
    const f2 ga = mul2(mul2(p.ak, cf), inv);
    const f2 fx = fma2(na, p.nx, mul2(nv, vx)), fy = fma2(na, p.ny, mul2(nv, vy)), fz = fma2(na, p.nz, mul2(nv, vz));
    // L = -(LF + LT x r)
    const f2 Lx = fma2(p.ry, k[14], fma2(p.rz, k[16], k[9]));
    const f2 Ly = fma2(p.rz, k[12], fma2(p.rx, k[17], k[10]));
    const f2 Lz = fma2(p.rx, k[13], fma2(p.ry, k[15], k[11]));
    const f2 x = fma2(Lz, p.nz, fma2(Ly, p.ny, mul2(Lx, p.nx)));
    const f2 y = fma2(Lz, vz, fma2(Ly, vy, mul2(Lx, vx)));
    const f2 px = mul2(al, x), q = fma2(be, x, mul2(ga, y));
    const f2 Lvx = fma2(q, vx, fma2(px, p.nx, mul2(nv, Lx)));
    const f2 Lvy = fma2(q, vy, fma2(px, p.ny, mul2(nv, Ly)));
    const f2 Lvz = fma2(q, vz, fma2(px, p.nz, mul2(nv, Lz)));
    // r: LT x (-f) + Lv x w
    acc.rx = fma2(Lvy, k[5], fma2(Lvz, k[7], fma2(k[13], fz, fma2(k[17], fy, acc.rx))));
    acc.ry = fma2(Lvz, k[3], fma2(Lvx, k[8], fma2(k[14], fx, fma2(k[15], fz, acc.ry))));
    acc.rz = fma2(Lvx, k[4], fma2(Lvy, k[6], fma2(k[12], fy, fma2(k[16], fx, acc.rz))));
    acc.nx = fma2(vx, px, fma2(Lx, na, acc.nx));
    acc.ny = fma2(vy, px, fma2(Ly, na, acc.ny));
    acc.nz = fma2(vz, px, fma2(Lz, na, acc.nz));
    acc.ak = fma2(x, h1, fma2(y, h2, acc.ak));
}

// The mass properties' adjoints of one step, by lane, summed over the warp into smem lp[17].
__device__ __forceinline__ void pan_params(const pg::LamP<float>& LP, int lane, float* lp) {
    const float v[17] = {LP.mass, LP.invmass, LP.I[0], LP.I[1], LP.I[2], LP.I[3], LP.I[4], LP.I[5],
                         LP.invI[0], LP.invI[1], LP.invI[2], LP.invI[3], LP.invI[4], LP.invI[5], LP.invI[6], LP.invI[7],
                         LP.invI[8]};
#pragma unroll
    for (int q = 0; q < 17; q++) {
        const float t = warp_sum(v[q]);
        if (lane == 0) lp[q] += t;
    }
}

__global__ void __launch_bounds__(kPanThreads, 5) k_adj_panels(GradArgs a, long long cap) {
    __shared__ __align__(16) f2 sk[2][kPanSteps][kPanValues];
    __shared__ float lp[kPanWarps][17];
    __shared__ int s_item;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int count = a.work[7];
    for (;;) {
    __syncthreads();
    if (tid == 0) s_item = atomicAdd(&a.work[8], 1);
    if (lane < 17) lp[warp][lane] = 0.f;
    __syncthreads();
    if (s_item >= count) break;
    const int item = a.items[cap + s_item];
    const int f = item >> 6, part = item & 63;
    float* out = a.adj + ((size_t)f * a.adj_parts + part) * kAdjStride;
    if (!adj_takes(a, f)) {  // oversize or NaN flight: constant distance
        for (int i = tid; i < kAdjStride; i += kPanThreads) out[i] = 0.f;
        continue;
    }
    const int first = part * kAdjPart;
    const int p = f / a.nseeds, nt = a.plane_nt[p], off = a.plane_off[p], n = min(a.steps[f], first + kAdjPart);
    const float* rec = a.setup + (size_t)f * kGradSetupFloats;
    const F3 cg = pg::v3(rec[22], rec[23], rec[24]);
    const float rho = rec[25], wp = rec[26], wr = rec[27];
    const f2 cf = bc(rec[17]);
    PanPair pp[2];
    PanAcc acc[2];
#pragma unroll
    for (int c = 0; c < 2; c++) {
        float v[2][7];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int i = 2 * (tid + c * kPanThreads) + h;
            F3 rb = pg::v3(0.f, 0.f, 0.f), nb = rb;
            float ak = 0.f;
            if (i < nt) {
                const float4 c4 = a.pc[off + i], n4 = a.pn[off + i];
                pg::stage(pg::v3(c4.x, c4.y, c4.z), c4.w, pg::v3(n4.x, n4.y, n4.z), cg, rho, wp, wr, &rb, &nb, &ak);
            }
            v[h][0] = rb.x; v[h][1] = rb.y; v[h][2] = rb.z; v[h][3] = nb.x; v[h][4] = nb.y; v[h][5] = nb.z; v[h][6] = ak;
        }
        pp[c] = {pk(v[0][0], v[1][0]), pk(v[0][1], v[1][1]), pk(v[0][2], v[1][2]), pk(v[0][3], v[1][3]),
                 pk(v[0][4], v[1][4]), pk(v[0][5], v[1][5]), pk(v[0][6], v[1][6])};
        acc[c] = {0ull, 0ull, 0ull, 0ull, 0ull, 0ull, 0ull};
    }
    // What the panels need of steps j0 .. j0 + kPanSteps - 1, a step per thread: the force and torque
    // adjoints, from the adjoint of the state after the step through the integrator.
    const pg::FlightP<float> P = setup_flightp(a, f);
    auto load = [&](int j0, int buf) {
        if (j0 + 32 * warp >= n) return;
        const int j = min(j0 + tid, n - 1);
        FSt st, L1 = zero_state(), L0 = L1;
        F3 Fb, Tb, vb, LF, LT;
        load_ent(adj_ent(a, f, j), st, &Fb, &Tb, &vb);
        const float4* l4 = reinterpret_cast<const float4*>(adj_chunk(a, f, j >> 5) + 16 * (j & 31));
        const float4 l0 = l4[0], l1 = l4[1], l2 = l4[2], l3 = l4[3];
        L1.vel = pg::v3(l0.w, l1.x, l1.y);  // already with dt times the position's
        L1.w = pg::v3(l1.z, l1.w, l2.x);
        L1.q[0] = l2.y; L1.q[1] = l2.z; L1.q[2] = l2.w; L1.q[3] = l3.x;
        pg::M3<float> R, LR;
        pg::rot_rows(st.q, R);
#pragma unroll
        for (int r = 0; r < 3; r++)
#pragma unroll
            for (int q = 0; q < 3; q++) LR.a[r][q] = 0.f;
        pg::PostF<float> pf;
        (void)pg::step_post_f(P, st, R, Fb, Tb, pf);
        pg::LamP<float> LP = {};
        pg::step_post_adj_f(P, st, R, Fb, pf, L1, L0, &LF, &LT, LR, LP);
        if (j0 + tid >= n) LP = {};
        pan_params(LP, lane, lp[warp]);
        f2* k = sk[buf][tid];
        const float v[12] = {vb.x, vb.y, vb.z, st.w.x, st.w.y, st.w.z, -LF.x, -LF.y, -LF.z, LT.x, LT.y, LT.z};
#pragma unroll
        for (int q = 0; q < 6; q++) k[q] = bc(v[q]);
#pragma unroll
        for (int q = 0; q < 3; q++) {
            k[6 + q] = bc(-v[3 + q]);
            k[9 + q] = bc(v[6 + q]);
            k[12 + q] = bc(v[9 + q]);
            k[15 + q] = bc(-v[9 + q]);
        }
    };
    auto sweep = [&](auto two_pairs) {
        constexpr int NC = decltype(two_pairs)::value ? 2 : 1;
        load(first, 0);
        for (int j0 = first, buf = 0; j0 < n; j0 += kPanSteps, buf ^= 1) {
            __syncthreads();
            if (j0 + kPanSteps < n) load(j0 + kPanSteps, buf ^ 1);
            const int m = min(kPanSteps, n - j0);
#pragma unroll 1
            for (int st = 0; st < m; st++) {
                f2 k[kPanValues];
                const ulonglong2* src = reinterpret_cast<const ulonglong2*>(sk[buf][st]);
#pragma unroll
                for (int q = 0; q < kPanValues / 2; q++) {
                    const ulonglong2 x = src[q];
                    k[2 * q] = x.x;
                    k[2 * q + 1] = x.y;
                }
#pragma unroll
                for (int c = 0; c < NC; c++) pan_pair(pp[c], k, cf, acc[c]);
            }
        }
    };
    if (nt > 2 * kPanThreads) sweep(std::true_type{}); else sweep(std::false_type{});
    float* o = out + 8;
#pragma unroll
    for (int c = 0; c < 2; c++) {
        float v[2][7];
        upk(acc[c].rx, v[0][0], v[1][0]); upk(acc[c].ry, v[0][1], v[1][1]); upk(acc[c].rz, v[0][2], v[1][2]);
        upk(acc[c].nx, v[0][3], v[1][3]); upk(acc[c].ny, v[0][4], v[1][4]); upk(acc[c].nz, v[0][5], v[1][5]);
        upk(acc[c].ak, v[0][6], v[1][6]);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int i = 2 * (tid + c * kPanThreads) + h;
            if (i >= nt) continue;
            const float4 c4 = a.pc[off + i], n4 = a.pn[off + i];
            F3 Lc, Ln;
            float LA;
            pg::stage_adj(pg::v3(c4.x, c4.y, c4.z), pg::v3(n4.x, n4.y, n4.z), cg, rho, wp, wr,
                          pg::v3(v[h][0], v[h][1], v[h][2]), pg::v3(v[h][3], v[h][4], v[h][5]), v[h][6], &Lc, &LA, &Ln);
            o[0 * kNtMax + i] = Lc.x; o[1 * kNtMax + i] = Lc.y; o[2 * kNtMax + i] = Lc.z;
            o[3 * kNtMax + i] = LA;
            o[4 * kNtMax + i] = Ln.x; o[5 * kNtMax + i] = Ln.y; o[6 * kNtMax + i] = Ln.z;
        }
    }
    __syncthreads();
    if (tid == 0) {  // the part's share of mass and inertia; the first part has the release's
        float v[17];
#pragma unroll
        for (int q = 0; q < 17; q++) v[q] = lp[0][q] + lp[1][q] + lp[2][q];
        pg::LamP<float> LP;
        LP.mass = v[0]; LP.invmass = v[1];
#pragma unroll
        for (int q = 0; q < 6; q++) LP.I[q] = v[2 + q];
#pragma unroll
        for (int q = 0; q < 9; q++) LP.invI[q] = v[8 + q];
        FlightCtx c;
        flight_setup(a, f, c);
        if (part == 0) {
            FSt L = zero_state();
            const float* l = a.after + (size_t)f * 16;
            L.w = pg::v3(l[6], l[7], l[8]);
            F3 L1rel, wb1;
            (void)pg::release(c.sc, P, c.cg, &L1rel, &wb1);
            pg::release_adj(P, L1rel, wb1, L, LP);
        }
        float Lmass, LI[6];
        pg::printed_adj(P, c.sigma, c.beta, LP, &Lmass, LI);
        out[0] = Lmass;
#pragma unroll
        for (int q = 0; q < 6; q++) out[1 + q] = LI[q];
        out[7] = 0.f;
    }
    }
}

}  // namespace

namespace {
size_t jac_items(const GradArgs& a) { return (size_t)a.n_flights * ((a.rec_steps + kJacSteps - 1) / kJacSteps); }
}  // namespace

size_t grad_time_items(int n_flights, int rec_steps) {
    return (size_t)n_flights * ((rec_steps + kJacSteps - 1) / kJacSteps + (rec_steps + kAdjPart - 1) / kAdjPart);
}

cudaError_t launch_grad_time(const GradArgs& a, int nsm, cudaStream_t s) {
    if (!a.fsum || !a.rec || !a.after || !a.items || a.rec_steps % 32 != 0) return cudaErrorInvalidValue;
    constexpr int kChainSmem = 2 * kAdjChunk * (int)sizeof(float);
    const int nseg = (a.max_steps + a.K - 1) / a.K;
    const long long threads = (long long)a.n_flights * nseg, cap = (long long)jac_items(a);
    k_adj_states<<<(unsigned)((threads + 63) / 64), 64, 0, s>>>(a, nseg);
    k_adj_items<<<1, 1024, 0, s>>>(a, cap);
    k_adj_jacobian<<<kJacBlocks * nsm, kJacSteps, 0, s>>>(a);
    k_adj_chain<<<a.n_flights, 32, kChainSmem, s>>>(a);
    k_adj_panels<<<5 * nsm, kPanThreads, 0, s>>>(a, cap);
    return cudaGetLastError();
}

}  // namespace pe
