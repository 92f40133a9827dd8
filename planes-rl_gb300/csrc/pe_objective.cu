// pe_objective.cu -- the smoothed tail-aware objective from a forward pass only, in FP32 or FP64.
//
// The quantity pe_grad differentiates (pe_grad_model.h), evaluated without the adjoint: for
// finite differences, line searches, and as the FP64 yardstick of the FP32 gradient on the GPU.
// Unlike the evaluation path (pe_prepare.cu + pe_flight*.cu, the reference's float arithmetic),
// every stage here -- mesh, mass properties, panels, print variation, flight -- runs in the
// chosen precision, so central differences at a step of 1e-4 of a gene's range are not swamped by
// float rounding of the inputs.  Built without fast math.
//
//   k_obj_prepare   one block per plane: mesh, printability, mass properties (two passes over
//                   the triangles with block reductions) and panels, in T.
//   k_obj_forward   one block of kObjW warps per flight, persistent over a work queue: print
//                   variation, staging, release and the flight; writes the smoothed distance.
//   k_obj_forward4  the same with four flights per block, for FP64.
//   k_obj_flights   four flights per block with their integrators in one warp, for many flights in FP32.
//   k_obj_weights   one block per plane: the tail-aware objective of its distances.
#include <cuda_runtime.h>

#include "pe_grad_model.h"
#include "pe_internal.cuh"

namespace pe {

namespace {

constexpr int kObjThreads = 128;
constexpr int kObjW = 4;

template <class T>
__device__ __forceinline__ T warp_sum_t(T v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Reduction of N values over a block of kObjThreads: op 0 sum, 1 min, 2 max (every thread gets
// the results).
template <class T, int N>
__device__ __forceinline__ void block_reduce(T v[N], const int op[N], T (*scratch)[N]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < N; k++)
        for (int o = 16; o > 0; o >>= 1) {
            const T u = __shfl_xor_sync(0xffffffffu, v[k], o);
            v[k] = op[k] == 0 ? v[k] + u : (op[k] == 1 ? (u < v[k] ? u : v[k]) : (u > v[k] ? u : v[k]));
        }
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < N; k++) scratch[warp][k] = v[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; k++) {
        T t = scratch[0][k];
#pragma unroll
        for (int w = 1; w < kObjThreads / 32; w++) {
            const T u = scratch[w][k];
            t = op[k] == 0 ? t + u : (op[k] == 1 ? (u < t ? u : t) : (u > t ? u : t));
        }
        v[k] = t;
    }
    __syncthreads();
}

// ------------------------------------------------------------------ plane data in T
template <class T>
__global__ void __launch_bounds__(kObjThreads) k_obj_prepare(ObjArgs a) {
    using V3T = pg::V3<T>;
    __shared__ T g[kGenomeN];
    __shared__ V3T V[kNvMax];
    __shared__ T red[kObjThreads / 32][8];
    const int p = blockIdx.x, tid = threadIdx.x;
    T* out = reinterpret_cast<T*>(a.plane) + (size_t)p * kObjPlaneStride;
    if (tid < kGenomeN) g[tid] = (T)a.genomes[(size_t)p * kGenomeN + tid];
    __syncthreads();
    const pg::Topo tp = pg::topology(g);
    for (int i = tid; i < tp.nv; i += kObjThreads) V[i] = pg::mesh_vertex(g, tp, i);
    __syncthreads();
    // printability: the mesh extent against the print volume (src/common.h:294-307)
    {
        const T big = T(1e30f);
        T e[6] = {big, big, big, -big, -big, -big};
        for (int i = tid; i < tp.nv; i += kObjThreads) {
            e[0] = pg::p_min(e[0], V[i].x); e[1] = pg::p_min(e[1], V[i].y); e[2] = pg::p_min(e[2], V[i].z);
            e[3] = pg::p_max(e[3], V[i].x); e[4] = pg::p_max(e[4], V[i].y); e[5] = pg::p_max(e[5], V[i].z);
        }
        const int ops[6] = {1, 1, 1, 2, 2, 2};
        block_reduce<T, 6>(e, ops, reinterpret_cast<T(*)[6]>(red));
        const T lim = (T)(0.250f - 0.00045f);
        if (tid == 0)
            out[7] = (e[3] - e[0] <= lim && e[4] - e[1] <= lim && e[5] - e[2] <= lim) ? (T)tp.nt : T(0);
    }
    // mass properties
    T m4[4] = {T(0), T(0), T(0), T(0)};
    for (int i = tid; i < tp.nt; i += kObjThreads) {
        T mi;
        V3T mc;
        pg::tri_mass(V, tp, i, &mi, &mc);
        m4[0] += mi; m4[1] += mc.x; m4[2] += mc.y; m4[3] += mc.z;
    }
    const int sum4[4] = {0, 0, 0, 0};
    block_reduce<T, 4>(m4, sum4, reinterpret_cast<T(*)[4]>(red));
    T m = m4[0], mn;
    V3T c = pg::v3(m4[1], m4[2], m4[3]), np;
    pg::mass_com(g, &m, &c, &mn, &np);
    T I[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
    for (int i = tid; i < tp.nt; i += kObjThreads) pg::tri_inertia(V, tp, i, c, I);
    const int sum6[6] = {0, 0, 0, 0, 0, 0};
    block_reduce<T, 6>(I, sum6, reinterpret_cast<T(*)[6]>(red));
    pg::inertia_finish(mn, np, c, I);
    if (tid == 0) {
        out[0] = m;
#pragma unroll
        for (int q = 0; q < 6; q++) out[1 + q] = I[q];
    }
    T* pc = out + 8;
    for (int t = tid; t < tp.nt; t += kObjThreads) {
        V3T ct, n;
        T A;
        pg::panel(V, tp, c, t, &ct, &A, &n);
        pc[t] = ct.x; pc[kNtMax + t] = ct.y; pc[2 * kNtMax + t] = ct.z; pc[3 * kNtMax + t] = A;
        pc[4 * kNtMax + t] = n.x; pc[5 * kNtMax + t] = n.y; pc[6 * kNtMax + t] = n.z;
    }
}

// ------------------------------------------------------------------ flights in T
template <class T>
__global__ void __launch_bounds__(32 * kObjW) k_obj_forward(ObjArgs a) {
    using V3T = pg::V3<T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* part = reinterpret_cast<T*>(smem_raw);        // [2][kObjW][8]
    int* flight = reinterpret_cast<int*>(part + 2 * kObjW * 8);
    T* sp = part + 2 * kObjW * 8 + 2;                 // 7 x kNtMax staged panels (SoA)
    constexpr int nthr = 32 * kObjW;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_flights = a.pop * a.nseeds;
    for (;;) {
        if (tid == 0) *flight = atomicAdd(a.work, 1);
        __syncthreads();
        const int f = *flight;
        __syncthreads();
        if (f >= n_flights) break;
        const int p = f / a.nseeds, si = f - p * a.nseeds;
        const T* pl = reinterpret_cast<const T*>(a.plane) + (size_t)p * kObjPlaneStride;
        const int nt = (int)pl[7];
        if (nt <= 0) {  // does not fit the print volume
            if (tid == 0) a.dist[f] = -100.0;
            continue;
        }
        const int seed = a.seeds[si] + (a.vary ? p * 7919 : 0);
        Scenario S;
        scenario_desc(seed, &S);
        T sc[kScenN];
#pragma unroll
        for (int k = 0; k < kScenN; k++) sc[k] = (T)S.v[k];
        pg::FlightP<T> P;
        V3T cg;
        T sigma, beta[6], I[6];
#pragma unroll
        for (int q = 0; q < 6; q++) I[q] = pl[1 + q];
        pg::printed(sc, pl[0], I, P, &cg, &sigma, beta);
        P.phase = (T)seed_phase(seed);
        const T* pc = pl + 8;
        for (int i = tid; i < nt; i += nthr) {
            V3T rb, nb;
            T ak;
            pg::stage(pg::v3(pc[i], pc[kNtMax + i], pc[2 * kNtMax + i]), pc[3 * kNtMax + i],
                      pg::v3(pc[4 * kNtMax + i], pc[5 * kNtMax + i], pc[6 * kNtMax + i]), cg, sc[pg::SC_RHO],
                      sc[pg::SC_WP], sc[pg::SC_WR], &rb, &nb, &ak);
            sp[i] = rb.x; sp[kNtMax + i] = rb.y; sp[2 * kNtMax + i] = rb.z;
            sp[3 * kNtMax + i] = nb.x; sp[4 * kNtMax + i] = nb.y; sp[5 * kNtMax + i] = nb.z;
            sp[6 * kNtMax + i] = ak;
        }
        pg::St<T> s = pg::release(sc, P, cg, (V3T*)nullptr, (V3T*)nullptr);
        __syncthreads();
        pg::Pre<T> pr;
        pg::step_pre(P, s, pr);
        int par = 0, to_chunk = kChunk;
        for (int j = 0;; j++) {
            T acc[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
            for (int i = tid; i < nt; i += nthr) {
                V3T fo, tq;
                pg::panel_fwd(pr, pg::v3(sp[i], sp[kNtMax + i], sp[2 * kNtMax + i]),
                              pg::v3(sp[3 * kNtMax + i], sp[4 * kNtMax + i], sp[5 * kNtMax + i]), sp[6 * kNtMax + i],
                              P.cf, &fo, &tq);
                acc[0] += fo.x; acc[1] += fo.y; acc[2] += fo.z;
                acc[3] += tq.x; acc[4] += tq.y; acc[5] += tq.z;
            }
            T* mine = part + (par * kObjW + warp) * 8;
#pragma unroll
            for (int k = 0; k < 6; k++) acc[k] = warp_sum_t(acc[k]);
            if (lane == 0)
#pragma unroll
                for (int k = 0; k < 6; k++) mine[k] = acc[k];
            __syncthreads();
            T v[6];
#pragma unroll
            for (int k = 0; k < 6; k++) {
                T t = part[(par * kObjW) * 8 + k];
#pragma unroll
                for (int w = 1; w < kObjW; w++) t += part[(par * kObjW + w) * 8 + k];
                v[k] = t;
            }
            par ^= 1;
            const pg::St<T> nx = pg::step_post(P, s, pr, pg::v3(v[0], v[1], v[2]), pg::v3(v[3], v[4], v[5]));
            T d = T(0);
            int kind = 0;
            if (pg::terminate(s, nx, j, a.max_steps, &d, &kind)) {
                if (tid == 0) a.dist[f] = (double)d;
                break;
            }
            s = nx;
            if (--to_chunk == 0) { s.t = T((double)(j + 1)) * T(pg::kDt); to_chunk = kChunk; }  // src/sim.cu:113
            pg::step_pre(P, s, pr);
        }
    }
}

// One of a block's four flights, and the warp's of the same number.
template <class T>
struct ObjSlot {
    T part[kObjW][8];  // each warp's sums of the step's force and torque
    T pre[8];          // vb xyz, w xyz, skin friction
    T sp[7 * kNtMax];  // staged panels (SoA)
};

// The sums over a warp of 24 values per lane (six of each of four flights), transposed: a level halves
// the values a lane carries, 24 shuffles instead of 120, and each sum follows the xor tree that a
// butterfly over all lanes would.  Lane 8 m + 4 h + q (q < 3) returns component 3 h + q of flight m.
template <class T>
__device__ __forceinline__ T warp_sum24(T (&v)[24], int lane) {
    auto fold = [&](int m, int half) {
        const bool up = (lane & m) != 0;
#pragma unroll
        for (int i = 0; i < half; i++) {
            const T send = up ? v[i] : v[i + half];
            const T keep = up ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
        }
    };
    fold(16, 12);
    fold(8, 6);
    fold(4, 3);
    v[3] = T(0);
    fold(2, 2);
    fold(1, 1);
    return v[0];
}

// Four flights per block: all warps take the panels of every flight, each warp its own flight's integrator
// and gusts, so that a flight-step is a third of the warp instructions.  Two barriers per step and a longer
// chain, which FP64's panels outweigh at any number of flights.
template <class T>
__global__ void __launch_bounds__(32 * kObjW, 1) k_obj_forward4(ObjArgs a) {
    using V3T = pg::V3<T>;
    constexpr int nthr = 32 * kObjW;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ObjSlot<T>* slot = reinterpret_cast<ObjSlot<T>*>(smem_raw);
    __shared__ int s_nt[kObjW];  // panels of each slot's flight (0: none)
    static_assert(kObjW == 4, "warp_sum24 takes four flights");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_flights = a.pop * a.nseeds;
    ObjSlot<T>& mine = slot[warp];
    int f = 0, j = 0, to_chunk = 0;
    bool live = false;
    pg::FlightP<T> P;
    pg::St<T> s;
    pg::Pre<T> pr{};
    auto publish = [&]() {
        if (lane == 0) {
            mine.pre[0] = pr.vb.x; mine.pre[1] = pr.vb.y; mine.pre[2] = pr.vb.z;
            mine.pre[3] = pr.w.x; mine.pre[4] = pr.w.y; mine.pre[5] = pr.w.z;
        }
    };
    auto next_flight = [&]() {
        for (;;) {
            if (lane == 0) f = atomicAdd(a.work, 1);
            f = __shfl_sync(0xffffffffu, f, 0);
            live = f < n_flights;
            if (!live) {
                if (lane == 0) s_nt[warp] = 0;
                return;
            }
            const int p = f / a.nseeds, si = f - p * a.nseeds;
            const T* pl = reinterpret_cast<const T*>(a.plane) + (size_t)p * kObjPlaneStride;
            const int nt = (int)pl[7];
            if (nt <= 0) {  // does not fit the print volume
                if (lane == 0) a.dist[f] = -100.0;
                continue;
            }
            const int seed = a.seeds[si] + (a.vary ? p * 7919 : 0);
            Scenario S;
            scenario_desc(seed, &S);
            T sc[kScenN];
#pragma unroll
            for (int k = 0; k < kScenN; k++) sc[k] = (T)S.v[k];
            V3T cg;
            T sigma, beta[6], I[6];
#pragma unroll
            for (int q = 0; q < 6; q++) I[q] = pl[1 + q];
            pg::printed(sc, pl[0], I, P, &cg, &sigma, beta);
            P.phase = (T)seed_phase(seed);
            const T* pc = pl + 8;
            T* sp = mine.sp;
            for (int i = lane; i < nt; i += 32) {
                V3T rb, nb;
                T ak;
                pg::stage(pg::v3(pc[i], pc[kNtMax + i], pc[2 * kNtMax + i]), pc[3 * kNtMax + i],
                          pg::v3(pc[4 * kNtMax + i], pc[5 * kNtMax + i], pc[6 * kNtMax + i]), cg, sc[pg::SC_RHO],
                          sc[pg::SC_WP], sc[pg::SC_WR], &rb, &nb, &ak);
                sp[i] = rb.x; sp[kNtMax + i] = rb.y; sp[2 * kNtMax + i] = rb.z;
                sp[3 * kNtMax + i] = nb.x; sp[4 * kNtMax + i] = nb.y; sp[5 * kNtMax + i] = nb.z;
                sp[6 * kNtMax + i] = ak;
            }
            s = pg::release(sc, P, cg, (V3T*)nullptr, (V3T*)nullptr);
            pg::step_pre(P, s, pr);
            publish();
            if (lane == 0) {
                mine.pre[6] = P.cf;
                s_nt[warp] = nt;
            }
            j = 0;
            to_chunk = kChunk;
            return;
        }
    };
    next_flight();
    for (;;) {
        __syncthreads();
        if (!(s_nt[0] | s_nt[1] | s_nt[2] | s_nt[3])) break;
        T v[24];
#pragma unroll
        for (int m = 0; m < kObjW; m++) {
            T acc[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
            const T* pre = slot[m].pre;
            pg::Pre<T> q;
            q.vb = pg::v3(pre[0], pre[1], pre[2]);
            q.w = pg::v3(pre[3], pre[4], pre[5]);
            const int nt = s_nt[m];
            const T* sp = slot[m].sp;
            const T cf = pre[6];
            for (int i = tid; i < nt; i += nthr) {
                V3T fo, tq;
                pg::panel_fwd(q, pg::v3(sp[i], sp[kNtMax + i], sp[2 * kNtMax + i]),
                              pg::v3(sp[3 * kNtMax + i], sp[4 * kNtMax + i], sp[5 * kNtMax + i]), sp[6 * kNtMax + i],
                              cf, &fo, &tq);
                acc[0] += fo.x; acc[1] += fo.y; acc[2] += fo.z;
                acc[3] += tq.x; acc[4] += tq.y; acc[5] += tq.z;
            }
#pragma unroll
            for (int k = 0; k < 6; k++) v[6 * m + k] = acc[k];
        }
        const T total = warp_sum24(v, lane);
        if ((lane & 3) != 3) slot[lane >> 3].part[warp][3 * ((lane >> 2) & 1) + (lane & 3)] = total;
        __syncthreads();
        if (!live) continue;
        T w[6];
#pragma unroll
        for (int k = 0; k < 6; k++) {
            T t = mine.part[0][k];
#pragma unroll
            for (int q = 1; q < kObjW; q++) t += mine.part[q][k];
            w[k] = t;
        }
        const pg::St<T> nx = pg::step_post(P, s, pr, pg::v3(w[0], w[1], w[2]), pg::v3(w[3], w[4], w[5]));
        T d = T(0);
        int kind = 0;
        if (pg::terminate(s, nx, j, a.max_steps, &d, &kind)) {
            if (lane == 0) a.dist[f] = (double)d;
            next_flight();
        } else {
            s = nx;
            if (--to_chunk == 0) { s.t = T((double)(j + 1)) * T(pg::kDt); to_chunk = kChunk; }  // src/sim.cu:113
            j++;
            pg::step_pre(P, s, pr);
            publish();
        }
    }
}

// ------------------------------------------------------------------ many flights in FP32
// Four flights per block as in k_obj_forward4, and one warp turns all four while another moves them and
// takes their gusts (eight lanes a flight), other warps each step; state and constants stay in shared memory,
// which leaves 90 registers and five blocks per SM instead of four of 108.  Warp (k + flight) % 4 takes the
// panels i % 128 / 32 == k of a flight, so a short last round falls on another warp for each of the four.
// Bound by issue slots.  512 x 8: 2.52 -> 2.24 ms, 1500 x 8: 5.78 -> 4.83 (k_obj_forward4, then this); a
// lone flight's step takes a fifth longer than with a block of its own.
constexpr int kObjPad = (kNtMax + 31) / 32 * 32;  // staged panels, filled up with empty ones

struct ObjBlock {
    float4 pos_t[kObjW], vel[kObjW], q[kObjW], w[kObjW];
    float4 cst[6][kObjW];          // ObjConst
    float4 rows[2][kObjW][3];      // attitude of this step and the next: rows, skin friction in the last place
    float4 va[kObjW];              // air velocity
    float4 part[kObjW][2 * kObjW + 1];
    int nt[kObjW], flight[kObjW], step[kObjW];
    float4 rb[kObjW][kObjPad];     // centroid, half the density times the area
    float2 nxy[kObjW][kObjPad];    // normal
    float nz[kObjW][kObjPad];
};
struct alignas(16) ObjConst {
    float I[6], invI[9], cf;
    float mass, invmass, gust, phase, base_x, base_y, pad0, pad1;
};
static_assert(sizeof(ObjConst) == 6 * sizeof(float4), "ObjConst is six float4");

// Sums of products with their fused operations spelled out, so that results do not hang on how the compiler
// pairs them: a b + c d (+ e f).
__device__ __forceinline__ float sum2(float a, float b, float c, float d) { return __fmaf_rn(a, b, __fmul_rn(c, d)); }
__device__ __forceinline__ float sum3(float a, float b, float c, float d, float e, float f) {
    return __fmaf_rn(e, f, sum2(a, b, c, d));
}
using F3 = pg::V3<float>;
__device__ __forceinline__ F3 f3(float4 v) { return pg::v3(v.x, v.y, v.z); }

__device__ __forceinline__ F3 obj_wind(const ObjConst& c, F3 p, float t, F3 vel) {
    const float s = c.phase;
    auto arg = [&](float a, float x, float b, float cc) { return sum3(a, x, b, t, cc, s); };
    const float a1 = arg(0.9f, p.x, 1.3f, 1.0f), a2 = arg(2.3f, p.z, 2.1f, 1.7f), a3 = arg(4.1f, p.y, 3.3f, 0.4f);
    const float b1 = arg(1.1f, p.x, 1.7f, 2.2f), b2 = arg(3.1f, p.z, 2.9f, 0.9f);
    const float c1 = arg(1.4f, p.x, 2.3f, 3.1f), c2 = arg(2.7f, p.y, 1.9f, 1.2f);
    const float gx = sum3(0.55f, pg::p_sin(a1), 0.35f, pg::p_sin(a2), 0.25f, pg::p_sin(a3));
    const float gy = sum2(0.50f, pg::p_sin(b1), 0.30f, pg::p_sin(b2));
    const float gz = sum2(0.30f, pg::p_sin(c1), 0.20f, pg::p_sin(c2));
    const float G = c.gust;
    const float wx = __fmaf_rn(G, gx, c.base_x);
    const float wy = __fmaf_rn(G, gy, c.base_y);
    return pg::v3(__fadd_rn(vel.x, -wx), __fadd_rn(vel.y, -wy), __fmaf_rn(-G, gz, vel.z));
}

__device__ __forceinline__ void obj_publish_rotation(ObjBlock& b, int m, int par, bool write, const float (&q)[4], F3 w, float cf) {
    const float qw = q[0], x = q[1], y = q[2], z = q[3];
    const float yy = __fmul_rn(y, y), zz = __fmul_rn(z, z);
    const float r00 = __fmaf_rn(-2.f, __fadd_rn(yy, zz), 1.f), r11 = __fmaf_rn(-2.f, __fmaf_rn(x, x, zz), 1.f);
    const float r22 = __fmaf_rn(-2.f, __fmaf_rn(x, x, yy), 1.f);
    const float r01 = 2.f * sum2(x, y, -qw, z), r02 = 2.f * sum2(qw, y, x, z), r10 = 2.f * sum2(x, y, qw, z);
    const float r12 = 2.f * sum2(y, z, -qw, x), r20 = 2.f * sum2(-qw, y, x, z), r21 = 2.f * sum2(y, z, qw, x);
    if (!write) return;
    b.q[m] = make_float4(qw, x, y, z);
    b.w[m] = make_float4(w.x, w.y, w.z, 0.f);
    b.rows[par][m][0] = make_float4(r00, r01, r02, r10);
    b.rows[par][m][1] = make_float4(r11, r12, r20, r21);
    b.rows[par][m][2] = make_float4(r22, 0.f, 0.f, cf);
}
__device__ __forceinline__ void obj_publish_translation(ObjBlock& b, int m, bool write, const ObjConst& c, F3 pos, F3 vel, float t, int step) {
    const F3 va = obj_wind(c, pos, t, vel);
    if (!write) return;
    b.pos_t[m] = make_float4(pos.x, pos.y, pos.z, t);
    b.vel[m] = make_float4(vel.x, vel.y, vel.z, 0.f);
    b.step[m] = step;
    b.va[m] = make_float4(va.x, va.y, va.z, 0.f);
}

__device__ __forceinline__ F3 obj_sum(const ObjBlock& b, int m, int k) {
    F3 t = f3(b.part[m][k]);
#pragma unroll
    for (int w = 1; w < kObjW; w++) t = t + f3(b.part[m][2 * w + k]);
    return t;
}

__global__ void __launch_bounds__(32 * kObjW, 5) k_obj_flights(ObjArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ObjBlock& b = *reinterpret_cast<ObjBlock*>(smem_raw);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    int lane;
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));
    const int m = lane >> 3;
    const bool leads = (lane & 7) == 0;
    const int n_flights = a.pop * a.nseeds;
    if (lane == 0) b.nt[warp] = -1;
    __syncthreads();
    int par = 0;  // rows of the coming step
    for (int turn = 0;; turn = (turn + 1) & 3) {
        if ((b.nt[0] | b.nt[1] | b.nt[2] | b.nt[3]) < 0) {
            __syncthreads();  // every warp has seen it
            if (b.nt[warp] < 0) {
                for (;;) {
                    int f = 0;
                    if (lane == 0) f = atomicAdd(a.work, 1);
                    f = __shfl_sync(0xffffffffu, f, 0);
                    if (f >= n_flights) {
                        if (lane == 0) b.nt[warp] = 0;
                        break;
                    }
                    const int p = f / a.nseeds, si = f - p * a.nseeds;
                    const float* pl = reinterpret_cast<const float*>(a.plane) + (size_t)p * kObjPlaneStride;
                    const int nt = (int)pl[7];
                    if (nt <= 0) {  // does not fit the print volume
                        if (lane == 0) a.dist[f] = -100.0;
                        continue;
                    }
                    const int seed = a.seeds[si] + (a.vary ? p * 7919 : 0);
                    Scenario S;
                    scenario_desc(seed, &S);
                    float sc[kScenN];
#pragma unroll
                    for (int k = 0; k < kScenN; k++) sc[k] = S.v[k];
                    F3 cg;
                    float sigma, beta[6], I[6];
#pragma unroll
                    for (int q = 0; q < 6; q++) I[q] = pl[1 + q];
                    pg::FlightP<float> P;
                    pg::printed(sc, pl[0], I, P, &cg, &sigma, beta);
                    P.phase = seed_phase(seed);
                    const float* pc = pl + 8;
                    for (int i = lane; i - lane < nt; i += 32) {
                        F3 rb = pg::v3(0.f, 0.f, 0.f), nb = rb;
                        float ak = 0.f;
                        if (i < nt)
                            pg::stage(pg::v3(pc[i], pc[kNtMax + i], pc[2 * kNtMax + i]), pc[3 * kNtMax + i],
                                      pg::v3(pc[4 * kNtMax + i], pc[5 * kNtMax + i], pc[6 * kNtMax + i]), cg, sc[pg::SC_RHO],
                                      sc[pg::SC_WP], sc[pg::SC_WR], &rb, &nb, &ak);
                        b.rb[warp][i] = make_float4(rb.x, rb.y, rb.z, ak);
                        b.nxy[warp][i] = make_float2(nb.x, nb.y);
                        b.nz[warp][i] = nb.z;
                    }
                    const pg::St<float> s = pg::release(sc, P, cg, (F3*)nullptr, (F3*)nullptr);
                    ObjConst c;
#pragma unroll
                    for (int k = 0; k < 6; k++) c.I[k] = P.I[k];
#pragma unroll
                    for (int k = 0; k < 9; k++) c.invI[k] = P.invI[k];
                    c.cf = P.cf; c.mass = P.mass; c.invmass = P.invmass; c.gust = P.gust; c.phase = P.phase;
                    c.base_x = P.base_x; c.base_y = P.base_y; c.pad0 = c.pad1 = 0.f;
                    const float4* o = reinterpret_cast<const float4*>(&c);
                    if (lane == 0) {
#pragma unroll
                        for (int k = 0; k < 6; k++) b.cst[k][warp] = o[k];
                        b.nt[warp] = nt;
                        b.flight[warp] = f;
                    }
                    obj_publish_rotation(b, warp, par, lane == 0, s.q, s.w, c.cf);
                    obj_publish_translation(b, warp, lane == 0, c, s.pos, s.vel, s.t, 0);
                    break;
                }
            }
            __syncthreads();
        }
        if ((b.nt[0] | b.nt[1] | b.nt[2] | b.nt[3]) == 0) break;
        float v[24];
#pragma unroll
        for (int k = 0; k < kObjW; k++) {
            float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            const int nt = b.nt[k], i0 = 32 * ((warp - k) & 3);
            if (i0 < nt) {
                const float4 m0 = b.rows[par][k][0], m1 = b.rows[par][k][1], m2 = b.rows[par][k][2], va = b.va[k];
                pg::Pre<float> q;
                q.vb = pg::v3(sum3(m0.x, va.x, m0.w, va.y, m1.z, va.z), sum3(m0.y, va.x, m1.x, va.y, m1.w, va.z),
                              sum3(m0.z, va.x, m1.y, va.y, m2.x, va.z));
                q.w = f3(b.w[k]);
                const float4* rb = b.rb[k] + i0 + lane;
                const float2* nxy = b.nxy[k] + i0 + lane;
                const float* nz = b.nz[k] + i0 + lane;
                auto panel = [&](int o) {
                    const float4 r = rb[o];
                    const float2 n = nxy[o];
                    F3 fo, tq;
                    pg::panel_fwd(q, f3(r), pg::v3(n.x, n.y, nz[o]), r.w, m2.w, &fo, &tq);
                    acc[0] += fo.x; acc[1] += fo.y; acc[2] += fo.z;
                    acc[3] += tq.x; acc[4] += tq.y; acc[5] += tq.z;
                };
                panel(0);
                if (i0 + 128 < nt) {
                    panel(128);
                    if (i0 + 256 < nt) panel(256);
                }
            }
#pragma unroll
            for (int c = 0; c < 6; c++) v[6 * k + c] = acc[c];
        }
        const float total = warp_sum24(v, lane);
        if ((lane & 3) != 3) reinterpret_cast<float*>(&b.part[m][2 * ((warp - m) & 3)])[lane & 7] = total;
        __syncthreads();
        if (warp == turn) {
            ObjConst c;
            float4* o = reinterpret_cast<float4*>(&c);
#pragma unroll
            for (int k = 0; k < 4; k++) o[k] = b.cst[k][m];
            const F3 Tb = obj_sum(b, m, 1), w = f3(b.w[m]);
            const float4 q4 = b.q[m];
            const F3 Iw = pg::v3(sum3(c.I[0], w.x, c.I[3], w.y, c.I[4], w.z), sum3(c.I[3], w.x, c.I[1], w.y, c.I[5], w.z),
                                 sum3(c.I[5], w.y, c.I[4], w.x, c.I[2], w.z));
            const F3 gy = pg::v3(sum2(w.y, Iw.z, -w.z, Iw.y), sum2(w.z, Iw.x, -w.x, Iw.z), sum2(w.x, Iw.y, -w.y, Iw.x));
            const F3 tq = Tb - gy;
            const F3 dw = pg::v3(sum3(c.invI[0], tq.x, c.invI[1], tq.y, c.invI[2], tq.z), sum3(c.invI[3], tq.x, c.invI[4], tq.y, c.invI[5], tq.z),
                                 sum3(c.invI[6], tq.x, c.invI[7], tq.y, c.invI[8], tq.z));
            const float dt = pg::kDt;
            const F3 w1 = pg::v3(__fmaf_rn(dw.x, dt, w.x), __fmaf_rn(dw.y, dt, w.y), __fmaf_rn(dw.z, dt, w.z));
            const F3 wn = pg::clamp_len(w1, 150.f);
            const float q[4] = {q4.x, q4.y, q4.z, q4.w};
            const float dq[4] = {-sum3(q[1], wn.x, q[2], wn.y, q[3], wn.z), __fmaf_rn(-q[3], wn.y, sum2(q[0], wn.x, q[2], wn.z)),
                                 __fmaf_rn(q[3], wn.x, sum2(q[0], wn.y, -q[1], wn.z)), __fmaf_rn(-q[2], wn.x, sum2(q[0], wn.z, q[1], wn.y))};
            const float h = 0.5f * dt;
            float qn[4], l2 = 0.f;
#pragma unroll
            for (int k = 0; k < 4; k++) { qn[k] = __fmaf_rn(h, dq[k], q[k]); l2 = k ? __fmaf_rn(qn[k], qn[k], l2) : __fmul_rn(qn[k], qn[k]); }
            const float il = pg::p_rsqrt(l2);
            const float qo[4] = {qn[0] * il, qn[1] * il, qn[2] * il, qn[3] * il};
            __syncwarp();
            obj_publish_rotation(b, m, par ^ 1, leads, qo, wn, c.cf);
        } else if (warp == ((turn + 1) & 3)) {
            ObjConst c;
            float4* o = reinterpret_cast<float4*>(&c);
            o[4] = b.cst[4][m]; o[5] = b.cst[5][m];
            const float4 m0 = b.rows[par][m][0], m1 = b.rows[par][m][1], m2 = b.rows[par][m][2], p4 = b.pos_t[m];
            const F3 Fb = obj_sum(b, m, 0);
            F3 Fw = pg::v3(sum3(m0.x, Fb.x, m0.y, Fb.y, m0.z, Fb.z), sum3(m0.w, Fb.x, m1.x, Fb.y, m1.y, Fb.z),
                           sum3(m1.z, Fb.x, m1.w, Fb.y, m2.x, Fb.z));
            Fw.z = __fmaf_rn(-c.mass, pg::kGrav, Fw.z);
            const float dt = pg::kDt, kv = __fmul_rn(c.invmass, dt);
            const F3 vel = f3(b.vel[m]);
            const F3 vel1 = pg::v3(__fmaf_rn(Fw.x, kv, vel.x), __fmaf_rn(Fw.y, kv, vel.y), __fmaf_rn(Fw.z, kv, vel.z));
            pg::St<float> before{}, after{};
            before.pos = f3(p4);
            after.vel = pg::clamp_len(vel1, 60.f);
            after.pos = pg::v3(__fmaf_rn(after.vel.x, dt, before.pos.x), __fmaf_rn(after.vel.y, dt, before.pos.y), __fmaf_rn(after.vel.z, dt, before.pos.z));
            float t = __fadd_rn(p4.w, dt), d = 0.f;
            int kind = 0;
            const int step = b.step[m];
            const bool live = b.nt[m] > 0;
            const int flight = b.flight[m];
            const int ended = pg::terminate(before, after, step, a.max_steps, &d, &kind);
            __syncwarp();
            if (ended) {
                if (leads && live) { a.dist[flight] = (double)d; b.nt[m] = -1; }
            } else {
                if ((step + 1) % kChunk == 0) t = (float)(step + 1) * (float)pg::kDt;
                obj_publish_translation(b, m, leads, c, after.pos, after.vel, t, step + 1);
            }
        }
        par ^= 1;
        __syncthreads();
    }
}

template <class T>
__global__ void __launch_bounds__(32) k_obj_weights(ObjArgs a) {
    __shared__ T d[kGradMaxSeeds], w[kGradMaxSeeds];
    const int p = blockIdx.x, tid = threadIdx.x, S = a.nseeds;
    for (int s = tid; s < S; s += 32) d[s] = (T)a.dist[(size_t)p * S + s];
    __syncwarp();
    if (tid == 0) a.obj[p] = (double)pg::objective_weights(d, S, w);
}

template <class T>
size_t forward_smem() {
    return (size_t)(2 * kObjW * 8 + 2) * sizeof(T) + (size_t)7 * kNtMax * sizeof(T);
}

template <class T>
cudaError_t launch_t(const ObjArgs& a, int nsm, cudaStream_t s) {
    // FP32 by number of flights: milliseconds with a flight per block / four, 128 x 8 1.32 / 1.46, 256 x 8
    // 1.99 / 2.01, 384 x 8 2.36 / 2.18, 512 x 8 2.99 / 2.24.  FP64 with a flight per block / four: 17.1 / 17.1
    // at 16 x 2, 37.5 / 34.4 at 64 x 8, 162 / 93 at 512 x 8.
    constexpr bool FP32 = sizeof(T) == 4;
    const bool many = FP32 && (long long)a.pop * a.nseeds > 14LL * nsm;
    const void* fn;
    size_t smem;
    if constexpr (FP32) {
        fn = many ? (const void*)k_obj_flights : (const void*)k_obj_forward<T>;
        smem = many ? sizeof(ObjBlock) : forward_smem<T>();
    } else {
        fn = (const void*)k_obj_forward4<T>;
        smem = kObjW * sizeof(ObjSlot<T>);
    }
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int bpsm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bpsm, fn, 32 * kObjW, smem);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(a.work, 0, sizeof(int), s);
    if (e != cudaSuccess) return e;
    const int grid = (bpsm > 0 ? bpsm : 1) * nsm;
    k_obj_prepare<T><<<a.pop, kObjThreads, 0, s>>>(a);
    if constexpr (FP32) {
        if (many) k_obj_flights<<<grid, 32 * kObjW, smem, s>>>(a);
        else k_obj_forward<T><<<grid, 32 * kObjW, smem, s>>>(a);
    } else {
        k_obj_forward4<T><<<grid, 32 * kObjW, smem, s>>>(a);
    }
    if (a.obj) k_obj_weights<T><<<a.pop, 32, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_objective(const ObjArgs& a, int precision, int nsm, cudaStream_t s) {
    return precision == 64 ? launch_t<double>(a, nsm, s) : launch_t<float>(a, nsm, s);
}

}  // namespace pe
