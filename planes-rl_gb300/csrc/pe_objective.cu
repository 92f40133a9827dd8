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
//   k_obj_forward   few flights in FP32: one block of kObjW warps per flight, persistent over a work queue: print
//                   variation, staging, release and the flight; writes the smoothed distance.
//   k_obj_flights   four flights per block with their integrators in one warp, for many flights and FP64.
//   k_obj_weights   one block per plane: the tail-aware objective of its distances.
#include <cuda_runtime.h>

#include <algorithm>

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

// ------------------------------------------------------------------ few flights in FP32
__global__ void __launch_bounds__(32 * kObjW) k_obj_forward(ObjArgs a) {
    using T = float;
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

// ------------------------------------------------------------------ four flights per block
// All warps take the panels of every flight; then one warp turns all four flights and another moves them and
// takes their gusts (eight lanes a flight), other warps each step.  State and constants stay in shared memory,
// which leaves 90 registers and five blocks per SM in FP32.  Warp (k + flight) % 4 takes the panels
// i % 128 / 32 == k of a flight, so a short last round falls on another warp for each of the four.  Bound by
// issue slots (FP32) and the FP64 pipe.  With each warp running its own flight's integrator: FP32 512 x 8
// 2.52 ms, 1500 x 8 5.78, FP64 512 x 8 86; so 2.24, 4.83 and 72.  A lone FP32 flight's step takes a fifth
// longer than with a block of its own.
constexpr int kObjPad = (kNtMax + 31) / 32 * 32;  // staged panels, filled up with empty ones

template <class T>
struct alignas(16) Vec4 { T x, y, z, w; };
template <class T>
struct alignas(2 * sizeof(T)) Vec2 { T x, y; };

template <class T>
struct ObjBlock {
    using V4 = Vec4<T>;
    V4 pos_t[kObjW], vel[kObjW], q[kObjW], w[kObjW];
    V4 cst[6][kObjW];          // ObjConst
    V4 rows[2][kObjW][3];      // attitude of this step and the next: rows, skin friction in the last place
    V4 va[kObjW];              // air velocity
    V4 part[kObjW][2 * kObjW + 1];
    int nt[kObjW], flight[kObjW], step[kObjW];
    V4 rb[kObjW][kObjPad];     // centroid, half the density times the area
    Vec2<T> nxy[kObjW][kObjPad];    // normal
    T nz[kObjW][kObjPad];
};
template <class T>
struct alignas(16) ObjConst {
    T I[6], invI[9], cf;
    T mass, invmass, gust, phase, base_x, base_y, pad0, pad1;
};
static_assert(sizeof(ObjConst<float>) == 6 * sizeof(Vec4<float>), "ObjConst is six Vec4");

// Sums of products with their fused operations spelled out, so that results do not hang on how the compiler
// pairs them: a b + c d (+ e f).
__device__ __forceinline__ float fma_t(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mul_t(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_t(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_t(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_t(double a, double b) { return __dadd_rn(a, b); }
template <class T>
__device__ __forceinline__ T sum2(T a, T b, T c, T d) { return fma_t(a, b, mul_t(c, d)); }
template <class T>
__device__ __forceinline__ T sum3(T a, T b, T c, T d, T e, T f) { return fma_t(e, f, sum2(a, b, c, d)); }
template <class T>
__device__ __forceinline__ pg::V3<T> v3(const Vec4<T>& v) { return pg::v3(v.x, v.y, v.z); }

template <class T>
__device__ __forceinline__ pg::V3<T> obj_wind(const ObjConst<T>& c, pg::V3<T> p, T t, pg::V3<T> vel) {
    const T s = c.phase;
    auto arg = [&](T a, T x, T b, T cc) { return sum3(a, x, b, t, cc, s); };
    const T a1 = arg(T(0.9f), p.x, T(1.3f), T(1.0f)), a2 = arg(T(2.3f), p.z, T(2.1f), T(1.7f)), a3 = arg(T(4.1f), p.y, T(3.3f), T(0.4f));
    const T b1 = arg(T(1.1f), p.x, T(1.7f), T(2.2f)), b2 = arg(T(3.1f), p.z, T(2.9f), T(0.9f));
    const T c1 = arg(T(1.4f), p.x, T(2.3f), T(3.1f)), c2 = arg(T(2.7f), p.y, T(1.9f), T(1.2f));
    const T gx = sum3(T(0.55f), pg::p_sin(a1), T(0.35f), pg::p_sin(a2), T(0.25f), pg::p_sin(a3));
    const T gy = sum2(T(0.50f), pg::p_sin(b1), T(0.30f), pg::p_sin(b2));
    const T gz = sum2(T(0.30f), pg::p_sin(c1), T(0.20f), pg::p_sin(c2));
    const T G = c.gust;
    const T wx = fma_t(G, gx, c.base_x);
    const T wy = fma_t(G, gy, c.base_y);
    return pg::v3(add_t(vel.x, -wx), add_t(vel.y, -wy), fma_t(-G, gz, vel.z));
}

template <class T>
__device__ __forceinline__ void obj_publish_rotation(ObjBlock<T>& b, int m, int par, bool write, const T (&q)[4], pg::V3<T> w, T cf) {
    const T qw = q[0], x = q[1], y = q[2], z = q[3];
    const T yy = mul_t(y, y), zz = mul_t(z, z);
    const T r00 = fma_t(T(-2), add_t(yy, zz), T(1)), r11 = fma_t(T(-2), fma_t(x, x, zz), T(1));
    const T r22 = fma_t(T(-2), fma_t(x, x, yy), T(1));
    const T r01 = T(2) * sum2(x, y, -qw, z), r02 = T(2) * sum2(qw, y, x, z), r10 = T(2) * sum2(x, y, qw, z);
    const T r12 = T(2) * sum2(y, z, -qw, x), r20 = T(2) * sum2(-qw, y, x, z), r21 = T(2) * sum2(y, z, qw, x);
    if (!write) return;
    using V4 = Vec4<T>;
    b.q[m] = V4{qw, x, y, z};
    b.w[m] = V4{w.x, w.y, w.z, T(0)};
    b.rows[par][m][0] = V4{r00, r01, r02, r10};
    b.rows[par][m][1] = V4{r11, r12, r20, r21};
    b.rows[par][m][2] = V4{r22, T(0), T(0), cf};
}
template <class T>
__device__ __forceinline__ void obj_publish_translation(ObjBlock<T>& b, int m, bool write, const ObjConst<T>& c, pg::V3<T> pos, pg::V3<T> vel, T t, int step) {
    const pg::V3<T> va = obj_wind(c, pos, t, vel);
    if (!write) return;
    using V4 = Vec4<T>;
    b.pos_t[m] = V4{pos.x, pos.y, pos.z, t};
    b.vel[m] = V4{vel.x, vel.y, vel.z, T(0)};
    b.step[m] = step;
    b.va[m] = V4{va.x, va.y, va.z, T(0)};
}

template <class T>
__device__ __forceinline__ pg::V3<T> obj_sum(const ObjBlock<T>& b, int m, int k) {
    pg::V3<T> t = v3(b.part[m][k]);
#pragma unroll
    for (int w = 1; w < kObjW; w++) t = t + v3(b.part[m][2 * w + k]);
    return t;
}

template <class T>
__global__ void __launch_bounds__(32 * kObjW, sizeof(T) == 4 ? 5 : 2) k_obj_flights(ObjArgs a, int slots) {
    using Block = ObjBlock<T>;
    using V3T = pg::V3<T>;
    using V4 = Vec4<T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Block& b = *reinterpret_cast<Block*>(smem_raw);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    int lane;
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));
    const int m = lane >> 3;
    const bool leads = (lane & 7) == 0;
    const int n_flights = a.pop * a.nseeds;
    if (lane == 0) b.nt[warp] = warp < slots ? -1 : 0;
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
                    pg::FlightP<T> P;
                    pg::printed(sc, pl[0], I, P, &cg, &sigma, beta);
                    P.phase = (T)seed_phase(seed);
                    const T* pc = pl + 8;
                    for (int i = lane; i - lane < nt; i += 32) {
                        V3T rb = pg::v3(T(0), T(0), T(0)), nb = rb;
                        T ak = T(0);
                        if (i < nt)
                            pg::stage(pg::v3(pc[i], pc[kNtMax + i], pc[2 * kNtMax + i]), pc[3 * kNtMax + i],
                                      pg::v3(pc[4 * kNtMax + i], pc[5 * kNtMax + i], pc[6 * kNtMax + i]), cg, sc[pg::SC_RHO],
                                      sc[pg::SC_WP], sc[pg::SC_WR], &rb, &nb, &ak);
                        b.rb[warp][i] = V4{rb.x, rb.y, rb.z, ak};
                        b.nxy[warp][i] = Vec2<T>{nb.x, nb.y};
                        b.nz[warp][i] = nb.z;
                    }
                    const pg::St<T> s = pg::release(sc, P, cg, (V3T*)nullptr, (V3T*)nullptr);
                    ObjConst<T> c;
#pragma unroll
                    for (int k = 0; k < 6; k++) c.I[k] = P.I[k];
#pragma unroll
                    for (int k = 0; k < 9; k++) c.invI[k] = P.invI[k];
                    c.cf = P.cf; c.mass = P.mass; c.invmass = P.invmass; c.gust = P.gust; c.phase = P.phase;
                    c.base_x = P.base_x; c.base_y = P.base_y; c.pad0 = c.pad1 = T(0);
                    const V4* o = reinterpret_cast<const V4*>(&c);
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
        T v[24];
#pragma unroll
        for (int k = 0; k < kObjW; k++) {
            T acc[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
            const int nt = b.nt[k], i0 = 32 * ((warp - k) & 3);
            if (i0 < nt) {
                const V4 m0 = b.rows[par][k][0], m1 = b.rows[par][k][1], m2 = b.rows[par][k][2], va = b.va[k];
                pg::Pre<T> q;
                q.vb = pg::v3(sum3(m0.x, va.x, m0.w, va.y, m1.z, va.z), sum3(m0.y, va.x, m1.x, va.y, m1.w, va.z),
                              sum3(m0.z, va.x, m1.y, va.y, m2.x, va.z));
                q.w = v3(b.w[k]);
                const V4* rb = b.rb[k] + i0 + lane;
                const Vec2<T>* nxy = b.nxy[k] + i0 + lane;
                const T* nz = b.nz[k] + i0 + lane;
                auto panel = [&](int o) {
                    const V4 r = rb[o];
                    const Vec2<T> n = nxy[o];
                    V3T fo, tq;
                    pg::panel_fwd(q, v3(r), pg::v3(n.x, n.y, nz[o]), r.w, m2.w, &fo, &tq);
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
        const T total = warp_sum24(v, lane);
        if ((lane & 3) != 3) reinterpret_cast<T*>(&b.part[m][2 * ((warp - m) & 3)])[lane & 7] = total;
        __syncthreads();
        if (warp == turn) {
            ObjConst<T> c;
            V4* o = reinterpret_cast<V4*>(&c);
#pragma unroll
            for (int k = 0; k < 4; k++) o[k] = b.cst[k][m];
            const V3T Tb = obj_sum(b, m, 1), w = v3(b.w[m]);
            const V4 q4 = b.q[m];
            const V3T Iw = pg::v3(sum3(c.I[0], w.x, c.I[3], w.y, c.I[4], w.z), sum3(c.I[3], w.x, c.I[1], w.y, c.I[5], w.z),
                                 sum3(c.I[5], w.y, c.I[4], w.x, c.I[2], w.z));
            const V3T gy = pg::v3(sum2(w.y, Iw.z, -w.z, Iw.y), sum2(w.z, Iw.x, -w.x, Iw.z), sum2(w.x, Iw.y, -w.y, Iw.x));
            const V3T tq = Tb - gy;
            const V3T dw = pg::v3(sum3(c.invI[0], tq.x, c.invI[1], tq.y, c.invI[2], tq.z), sum3(c.invI[3], tq.x, c.invI[4], tq.y, c.invI[5], tq.z),
                                 sum3(c.invI[6], tq.x, c.invI[7], tq.y, c.invI[8], tq.z));
            const T dt = T(pg::kDt);
            const V3T w1 = pg::v3(fma_t(dw.x, dt, w.x), fma_t(dw.y, dt, w.y), fma_t(dw.z, dt, w.z));
            const V3T wn = pg::clamp_len(w1, T(150));
            const T q[4] = {q4.x, q4.y, q4.z, q4.w};
            const T dq[4] = {-sum3(q[1], wn.x, q[2], wn.y, q[3], wn.z), fma_t(-q[3], wn.y, sum2(q[0], wn.x, q[2], wn.z)),
                                 fma_t(q[3], wn.x, sum2(q[0], wn.y, -q[1], wn.z)), fma_t(-q[2], wn.x, sum2(q[0], wn.z, q[1], wn.y))};
            const T h = T(0.5) * dt;
            T qn[4], l2 = T(0);
#pragma unroll
            for (int k = 0; k < 4; k++) { qn[k] = fma_t(h, dq[k], q[k]); l2 = k ? fma_t(qn[k], qn[k], l2) : mul_t(qn[k], qn[k]); }
            const T il = pg::p_rsqrt(l2);
            const T qo[4] = {qn[0] * il, qn[1] * il, qn[2] * il, qn[3] * il};
            __syncwarp();
            obj_publish_rotation(b, m, par ^ 1, leads, qo, wn, c.cf);
        } else if (warp == ((turn + 1) & 3)) {
            ObjConst<T> c;
            V4* o = reinterpret_cast<V4*>(&c);
            o[4] = b.cst[4][m]; o[5] = b.cst[5][m];
            const V4 m0 = b.rows[par][m][0], m1 = b.rows[par][m][1], m2 = b.rows[par][m][2], p4 = b.pos_t[m];
            const V3T Fb = obj_sum(b, m, 0);
            V3T Fw = pg::v3(sum3(m0.x, Fb.x, m0.y, Fb.y, m0.z, Fb.z), sum3(m0.w, Fb.x, m1.x, Fb.y, m1.y, Fb.z),
                           sum3(m1.z, Fb.x, m1.w, Fb.y, m2.x, Fb.z));
            Fw.z = fma_t(-c.mass, T(pg::kGrav), Fw.z);
            const T dt = T(pg::kDt), kv = mul_t(c.invmass, dt);
            const V3T vel = v3(b.vel[m]);
            const V3T vel1 = pg::v3(fma_t(Fw.x, kv, vel.x), fma_t(Fw.y, kv, vel.y), fma_t(Fw.z, kv, vel.z));
            pg::St<T> before{}, after{};
            before.pos = v3(p4);
            after.vel = pg::clamp_len(vel1, T(60));
            after.pos = pg::v3(fma_t(after.vel.x, dt, before.pos.x), fma_t(after.vel.y, dt, before.pos.y), fma_t(after.vel.z, dt, before.pos.z));
            T t = add_t(p4.w, dt), d = T(0);
            int kind = 0;
            const int step = b.step[m];
            const bool live = b.nt[m] > 0;
            const int flight = b.flight[m];
            const int ended = pg::terminate(before, after, step, a.max_steps, &d, &kind);
            __syncwarp();
            if (ended) {
                if (leads && live) { a.dist[flight] = (double)d; b.nt[m] = -1; }
            } else {
                if ((step + 1) % kChunk == 0) t = T((double)(step + 1)) * T(pg::kDt);
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

constexpr size_t kForwardSmem = (size_t)(2 * kObjW * 8 + 2) * sizeof(float) + (size_t)7 * kNtMax * sizeof(float);

template <class T>
cudaError_t launch_t(const ObjArgs& a, int nsm, cudaStream_t s) {
    // Milliseconds with a flight per block / four.  FP32: 128 x 8 1.32 / 1.46, 256 x 8 1.99 / 2.01, 384 x 8
    // 2.36 / 2.18, 512 x 8 2.99 / 2.24.  FP64: 1 x 1 4.9 / 3.7, 20 x 8 26.6 / 23.9, 512 x 8 160 / 72.
    const void* fn = (const void*)k_obj_flights<T>;
    size_t smem = sizeof(ObjBlock<T>);
    bool single = false;
    if constexpr (sizeof(T) == 4) {
        single = (long long)a.pop * a.nseeds <= 14LL * nsm;
        if (single) {
            fn = (const void*)k_obj_forward;
            smem = kForwardSmem;
        }
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
    if (single) k_obj_forward<<<grid, 32 * kObjW, smem, s>>>(a);
    else {
        // few flights spread over the blocks: fewer of them in each, none idle (FP64, 100 steps: 1 x 8 2.29 -> 1.48 ms,
        // a block per flight 1.91; 64 x 8 5.77 -> 3.93, a block per flight 5.98)
        const int slots = (int)std::min<long long>(kObjW, ((long long)a.pop * a.nseeds + grid - 1) / grid);
        k_obj_flights<T><<<grid, 32 * kObjW, smem, s>>>(a, slots);
    }
    if (a.obj) k_obj_weights<T><<<a.pop, 32, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_objective(const ObjArgs& a, int precision, int nsm, cudaStream_t s) {
    return precision == 64 ? launch_t<double>(a, nsm, s) : launch_t<float>(a, nsm, s);
}

}  // namespace pe
