// pe_flight_fast.cu -- the body-frame flight (pe_flight_fast.cuh) with a flight per 16 or 32 lanes of
// a warp: the engine's explicit shapes, pose recording, pe_grad's forward pass on large batches and
// the one-step probe.
#include "pe_flight_fast.cuh"

namespace pe {

// Record slot of step `step` in the reference's gpu_sim (src/sim.cu:115-121): every 600-step launch
// restarts its index at step0 / rec_every and advances it at each multiple of rec_every, so when
// rec_every does not divide 600 a launch's first record overwrites the previous launch's last.
__device__ __forceinline__ int rec_slot(int step, int every) {
    const int s0 = step - step % kChunk;
    const int before = s0 == 0 ? 0 : (s0 - 1) / every + 1;  // multiples of `every` in [0, s0)
    return s0 / every + (step / every + 1 - before) - 1;
}
__device__ __forceinline__ void rec_put(const FlightArgs& a, int flight, int step, const FlightState& st,
                                        float alive) {
    const int i = rec_slot(step, a.rec_every);
    if (i >= a.rec_cap) return;
    float4* r = reinterpret_cast<float4*>(a.rec + ((size_t)flight * a.rec_cap + i) * 8);
    r[0] = make_float4(st.pos.x, st.pos.y, st.pos.z, st.q.w);
    r[1] = make_float4(st.q.x, st.q.y, st.q.z, alive);
}
// The frozen pose of a finished flight at every record step after `from` (-1: from step 0; lanes
// share the steps).
__device__ __forceinline__ void rec_fill(const FlightArgs& a, int flight, int from, const FlightState& st, int j,
                                         int lanes) {
    const int first = from < 0 ? 0 : (from / a.rec_every + 1) * a.rec_every;
    for (int m = first + j * a.rec_every; m < kMaxSteps; m += lanes * a.rec_every) rec_put(a, flight, m, st, 0.f);
}

// CAP = 1 caps registers at 96 (launch bounds of 5 blocks x 128 threads), CAP = 2 at 128 (4 blocks
// x 128 threads): more flights reside per SM; spilled values go to L1-resident local memory.
// CAP = 3 launches one-warp blocks, 11 per SM (registers <= 184, no spills): at 16 lanes that is
// all the 2-flight slots shared memory holds (11 x (2 x 9,856 B + 1 KB reserved) of 228 KB), one
// warp more per SM than the uncapped kernel's 198 registers leave room for.
// HAND = true leaves the flights of the launch's last few to pe_flight_wide.cu (FlightArgs.landed), asked for
// every 16 steps outside the loop of the steps: inside it, even never taken, it cost 4 % of a 2,048 x 8 run.
// REC = true adds the reference's pose recording and launch grid (pe_sim only).
// GRAD = true is pe_grad's forward pass: every flight from its set-up record (FlightArgs.grad_setup),
// smoothed distances, and per flight its checkpoints, every step's body force and torque and how it
// ended (FlightArgs.grad_*); one launch over all flights.
template <int LPF, int CAP, bool REC = false, bool GRAD = false, bool HAND = false>
__global__ void __launch_bounds__(CAP == 3 ? 32 : (CAP ? 128 : 256), CAP == 1 ? 5 : (CAP == 2 ? 4 : (CAP == 3 ? 11 : 1)))
    k_flight_fast(FlightArgs a) {
    extern __shared__ float4 smem[];
    const int lane = threadIdx.x & 31;
    const int j = lane % LPF;
    const int slot = threadIdx.x / LPF;
    const PairedPanels pp = paired_view<LPF>((char*)smem + (size_t)slot * paired_bytes<LPF>());
    const unsigned mask = fast_mask<LPF>(lane);
    const int leader = lane - j;
    const int n_work = a.active_in ? *a.n_active_in : a.n_flights;
    while (true) {
        int f = 0;
        if (j == 0) f = atomicAdd(a.work, 1);
        f = __shfl_sync(mask, f, leader);
        if (f >= n_work) break;
        const int flight = a.active_in ? a.active_in[f] : f;
        const int p = flight / a.nseeds, s = flight - p * a.nseeds;
        const int nt = a.plane_nt[p];
        FastConst fc;
        vec3 cg;
        float air_rho, wp, wr;
        FlightState st;
        if (GRAD) {  // the gradient model's set-up of this flight
            grad_record(a, flight, &fc, &cg, &air_rho, &wp, &wr, &st);
            if (nt <= 0) {
                if (j == 0) {
                    a.dist[flight] = -100.0f;
                    a.steps[flight] = 0;
                    a.grad_kind[flight] = 0;
                    if (HAND) atomicAdd(a.landed, 1);
                }
                continue;
            }
        } else {
            MassProps pmp;
            Scenario sc;
            fast_setup(a, p, s, &fc, &cg, &air_rho, &wp, &wr, &pmp, &sc);
            if (a.step_begin == 0) {
                if (REC || nt > 0) release(sc, pmp, cg, &st);
                if (REC && a.spread > 0.f) {  // showcase launch grid, src/sim.cu:72-79
                    const int cols = 25;
                    st.pos.x = -(float)(p / cols) * a.spread * 1.4f;
                    st.pos.y = (float)((p % cols) - cols / 2) * a.spread;
                    st.pos.z = st.pos.z + 0.25f * sinf((float)p * 12.9898f);
                }
                if (nt <= 0) {
                    if (j == 0) {
                        a.dist[flight] = -100.0f;
                        a.steps[flight] = 0;
                        if (HAND) atomicAdd(a.landed, 1);
                    }
                    if (REC && a.rec) rec_fill(a, flight, -1, st, j, LPF);
                    continue;
                }
            } else {
                st = a.state[flight];
            }
        }
        float* ck = nullptr;
        float* fsum = nullptr;
        if (GRAD) {
            ck = a.grad_ck + (size_t)flight * a.grad_nck * 16;
            fsum = a.grad_fsum ? a.grad_fsum + (size_t)flight * a.max_steps * 8 : nullptr;
            if (j == 0) *reinterpret_cast<FlightState*>(ck) = st;  // the release state
        }
        __syncwarp(mask);
        fast_stage<LPF>(a, p, nt, j, cg, air_rho, wp, wr, pp);
        __syncwarp(mask);
        const int end = min(a.step_end, a.max_steps);
        int step = st.step, done = 0;
        float fit = 0.0f;
        StepOut so;
        so.kind = 0;
        int to_ck = GRAD ? a.grad_K : 0, ck_i = 0;  // steps to the next checkpoint, its index
        int seen = 0;                               // flights of the launch that had ended 16 steps ago
        while (step < end && !done) {
            int stop = end;
            if (HAND) {
                if (n_work - __shfl_sync(mask, seen, 0) <= a.hand_over) break;
                seen = *(volatile int*)a.landed;
                stop = min(end, (step | 15) + 1);
            }
            for (; step < stop; step++) {
                if (REC && a.rec && j == 0 && step % a.rec_every == 0) rec_put(a, flight, step, st, 1.f);
                done = fast_step<LPF>(fc, pp, nt, j, mask, st, step, a.max_steps, GRAD ? 1 : a.smooth, &fit, nullptr,
                                      GRAD ? &so : nullptr);
                if (GRAD && j == 0) {
                    if (fsum) {
                        float4* d4 = reinterpret_cast<float4*>(fsum + (size_t)step * 8);
                        d4[0] = make_float4(so.fb[0], so.fb[1], so.fb[2], so.fb[3]);
                        d4[1] = make_float4(so.fb[4], so.fb[5], 0.0f, 0.0f);
                    }
                }
                if (GRAD && --to_ck == 0) {  // after step + 1 = (ck_i + 1) * K steps
                    to_ck = a.grad_K;
                    ++ck_i;
                    if (!done && j == 0) {
                        FlightState c = st;  // as the next step starts: the clock restarts every 600 steps
                        if ((step + 1) % kChunk == 0) c.t = mul_((float)(step + 1), PE_DT);
                        *reinterpret_cast<FlightState*>(ck + (size_t)ck_i * 16) = c;
                    }
                }
                if (done) break;
            }
        }
        if (done) {
            if (GRAD && j == 0) a.grad_kind[flight] = so.kind;
            if (j == 0) {
                a.dist[flight] = fit;
                a.steps[flight] = step + 1;
                if (HAND) atomicAdd(a.landed, 1);
            }
            if (REC && a.rec) {
                __syncwarp(mask);  // lane 0's alive frames precede the frozen ones that may share a slot
                rec_fill(a, flight, step, st, j, LPF);
            }
        } else if (j == 0 && a.active_out) {
            st.step = step;
            a.state[flight] = st;
            int k = atomicAdd(a.n_active_out, 1);
            a.active_out[k] = flight;
        }
    }
}

template <int LPF>
__global__ void __launch_bounds__(256) k_debug_step_fast(FlightArgs a, const FlightState* state_in,
                                                         FlightState* state_out, float* FT, int* done_out,
                                                         float* fit_out, int step) {
    extern __shared__ float4 smem[];
    const int lane = threadIdx.x & 31;
    const int j = lane % LPF;
    const int slot = threadIdx.x / LPF;
    const PairedPanels pp = paired_view<LPF>((char*)smem + (size_t)slot * paired_bytes<LPF>());
    const unsigned mask = fast_mask<LPF>(lane);
    const int flight = blockIdx.x * (blockDim.x / LPF) + slot;
    if (flight >= a.n_flights) return;
    const int p = flight / a.nseeds, s = flight - p * a.nseeds;
    const int nt = a.plane_nt[p];
    FastConst fc;
    vec3 cg;
    float air_rho, wp, wr;
    fast_setup(a, p, s, &fc, &cg, &air_rho, &wp, &wr, nullptr, nullptr);
    fast_stage<LPF>(a, p, nt, j, cg, air_rho, wp, wr, pp);
    __syncwarp(mask);
    FlightState st = state_in[flight];
    float fit = 0.0f, sumw[6];
    int done = fast_step<LPF>(fc, pp, nt, j, mask, st, step, a.max_steps, 0, &fit, sumw);
    if (j == 0) {
        state_out[flight] = st;
        for (int c = 0; c < 6; c++) FT[flight * 6 + c] = sumw[c];
        done_out[flight] = done;
        fit_out[flight] = fit;
    }
}

template <int LPF>
static const void* fast_fn_lanes(int cap) {
    switch (cap) {
        case 1: return (const void*)&k_flight_fast<LPF, 1>;
        case 2: return (const void*)&k_flight_fast<LPF, 2>;
        case 3: return (const void*)&k_flight_fast<LPF, 3>;
        default: return (const void*)&k_flight_fast<LPF, 0>;
    }
}
static const void* fast_fn(const FlightShape& sh) {
    return sh.lanes == 16 ? fast_fn_lanes<16>(sh.cap) : fast_fn_lanes<32>(sh.cap);
}
template <int LPF>
static void launch_lanes(const FlightArgs& a, int cap, int grid, int threads, size_t smem, cudaStream_t s) {
    switch (cap) {
        case 1: k_flight_fast<LPF, 1><<<grid, threads, smem, s>>>(a); break;
        case 2: k_flight_fast<LPF, 2><<<grid, threads, smem, s>>>(a); break;
        case 3: k_flight_fast<LPF, 3><<<grid, threads, smem, s>>>(a); break;
        default: k_flight_fast<LPF, 0><<<grid, threads, smem, s>>>(a);
    }
}

size_t flight_fast_smem_bytes(const FlightShape& sh) {
    return (size_t)(sh.warps * 32 / sh.lanes) * (sh.lanes == 16 ? paired_bytes<16>() : paired_bytes<32>());
}

int flight_fast_blocks_per_sm(const FlightShape& sh) {
    const void* fn = fast_fn(sh);
    size_t smem = flight_fast_smem_bytes(sh);
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, sh.warps * 32, smem) != cudaSuccess) return 0;
    return nb;
}

cudaError_t flight_hand_configure(int* bps) {
    const size_t smem = 4 * paired_bytes<32>();
    const void* fn = (const void*)&k_flight_fast<32, 0, false, false, true>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int n = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, 128, smem);
    *bps = n > 0 ? n : 1;
    return e;
}

cudaError_t launch_flight_hand(const FlightArgs& a, int nsm, int bps, cudaStream_t s) {
    if (a.rec || a.spread > 0.f || !a.landed) return cudaErrorInvalidValue;
    k_flight_fast<32, 0, false, false, true><<<bps * nsm, 128, 4 * paired_bytes<32>(), s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_flight_fast(const FlightArgs& a, const FlightShape& sh, int grid, cudaStream_t s) {
    size_t smem = flight_fast_smem_bytes(sh);
    const void* fn = fast_fn(sh);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    if ((sh.cap && sh.warps > 4) || (sh.cap == 3 && sh.warps != 1) || sh.cap < 0 || sh.cap > 3)
        return cudaErrorInvalidValue;
    const int threads = sh.warps * 32;
    if (a.rec || a.spread > 0.f) {  // recording and the launch grid run in the default shape only
        if (sh.lanes != 16 || sh.cap) return cudaErrorInvalidValue;
        e = cudaFuncSetAttribute((const void*)&k_flight_fast<16, 0, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem);
        if (e != cudaSuccess) return e;
        k_flight_fast<16, 0, true><<<grid, threads, smem, s>>>(a);
    } else if (sh.lanes == 16) {
        launch_lanes<16>(a, sh.cap, grid, threads, smem, s);
    } else if (sh.lanes == 32) {
        launch_lanes<32>(a, sh.cap, grid, threads, smem, s);
    } else {
        return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t grad_forward_configure(int bps[2]) {
    const void* fn[2] = {(const void*)&k_flight_fast<32, 0, false, true, true>, (const void*)&k_flight_fast<16, 3, false, true>};
    const int threads[2] = {128, 32};
    const size_t smem[2] = {4 * paired_bytes<32>(), 2 * paired_bytes<16>()};
    for (int i = 0; i < 2; i++) {
        cudaError_t e = cudaFuncSetAttribute(fn[i], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem[i]);
        if (e != cudaSuccess) return e;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps[i], fn[i], threads[i], smem[i]);
        if (e != cudaSuccess) return e;
        if (bps[i] <= 0) bps[i] = 1;
    }
    return cudaSuccess;
}

cudaError_t launch_grad_forward(const FlightArgs& a, int nsm, const int bps[2], int wide_bps, int* wide_work,
                                cudaStream_t s) {
    if (!a.grad_setup || !a.grad_ck || !a.grad_kind || a.grad_K < 1 || a.step_begin != 0 ||
        a.step_end < a.max_steps || a.active_in)
        return cudaErrorInvalidValue;
    const long long per_sm = ((long long)a.n_flights + nsm - 1) / nsm;
    FlightArgs w = a;
    w.landed = nullptr;
    w.active_out = nullptr;
    w.n_active_out = nullptr;
    if (per_sm <= kWideFlights) return launch_flight_wide(w, nsm, wide_bps, s);
    if (per_sm > kGradLanesFlights) {
        k_flight_fast<16, 3, false, true><<<bps[1] * nsm, 32, 2 * paired_bytes<16>(), s>>>(w);
        return cudaGetLastError();
    }
    if (!a.landed || !a.active_out || !a.n_active_out || !wide_work) return cudaErrorInvalidValue;
    k_flight_fast<32, 0, false, true, true><<<bps[0] * nsm, 128, 4 * paired_bytes<32>(), s>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    w.active_in = a.active_out;
    w.n_active_in = a.n_active_out;
    w.work = wide_work;
    return launch_flight_wide(w, nsm, wide_bps, s);
}

cudaError_t launch_debug_step_fast(const FlightArgs& a, const FlightState* state_in, FlightState* state_out,
                                   float* FT, int* done, float* fit, int step, int lanes, cudaStream_t s) {
    const int threads = 128;
    const int per_block = threads / lanes;
    const int grid = (a.n_flights + per_block - 1) / per_block;
    const size_t smem = (size_t)per_block * (lanes == 16 ? paired_bytes<16>() : paired_bytes<32>());
    if (lanes == 16) {
        cudaFuncSetAttribute((const void*)&k_debug_step_fast<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        k_debug_step_fast<16><<<grid, threads, smem, s>>>(a, state_in, state_out, FT, done, fit, step);
    } else {
        cudaFuncSetAttribute((const void*)&k_debug_step_fast<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        k_debug_step_fast<32><<<grid, threads, smem, s>>>(a, state_in, state_out, FT, done, fit, step);
    }
    return cudaGetLastError();
}

}  // namespace pe
