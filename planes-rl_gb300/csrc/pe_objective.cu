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
//   k_obj_forward4  the same with four flights per block, for many flights and for FP64.
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
// and gusts, so a flight-step is 1,100 warp instructions instead of 3,000 and twenty flights fill an SM
// instead of five (FP32).  Two barriers per step and a longer chain: for batches of many flights.
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
    // Measured with a flight / four flights per block, FP32: 1.81 / 1.99 ms at 256 x 8, 2.47 / 2.28 at
    // 384 x 8, 3.19 / 2.57 at 512 x 8, 7.76 / 5.55 at 1500 x 8; FP64: 17.1 / 17.1 at 16 x 2, 37.5 / 34.4 at
    // 64 x 8, 162 / 93 at 512 x 8.
    const bool four = sizeof(T) == 8 || (long long)a.pop * a.nseeds > 16LL * nsm;
    const void* fn = four ? (const void*)k_obj_forward4<T> : (const void*)k_obj_forward<T>;
    const size_t smem = four ? kObjW * sizeof(ObjSlot<T>) : forward_smem<T>();
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int bpsm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bpsm, fn, 32 * kObjW, smem);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(a.work, 0, sizeof(int), s);
    if (e != cudaSuccess) return e;
    const int grid = (bpsm > 0 ? bpsm : 1) * nsm;
    k_obj_prepare<T><<<a.pop, kObjThreads, 0, s>>>(a);
    if (four) k_obj_forward4<T><<<grid, 32 * kObjW, smem, s>>>(a);
    else k_obj_forward<T><<<grid, 32 * kObjW, smem, s>>>(a);
    if (a.obj) k_obj_weights<T><<<a.pop, 32, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_objective(const ObjArgs& a, int precision, int nsm, cudaStream_t s) {
    return precision == 64 ? launch_t<double>(a, nsm, s) : launch_t<float>(a, nsm, s);
}

}  // namespace pe
