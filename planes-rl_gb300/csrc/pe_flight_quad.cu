// pe_flight_quad.cu -- the body-frame flight (pe_flight_fast.cuh) with four flights per warp, for
// batches that fill the GPU.
//
// A step is a panel part, which 32 lanes share, and a scalar part (gusts, attitude, integrator) that
// every lane of a flight repeats.  With a flight per half warp the scalar part and the reduction took
// 209 of a flight-step's 461 warp instructions, and 2.7 warps per scheduler left 38 % of the cycles
// without a ready one.  Here a warp flies four flights: it evaluates their panels one flight after the
// other on all 32 lanes, reduces the four sets of sums in one transposed tree that leaves flight g's
// totals on lanes 8g..8g+7, and those eight lanes integrate it, so one instruction stream carries four
// scalar parts (358 instructions per flight-step, and planes of 88 and 172 pairs no longer share a
// warp's pass count).
//
// Room for 48 flights per SM (12 warps) instead of 22 comes from tensor memory: a lane always reads
// the same pairs, v, v + 32, v + 64, ..., so its first three pairs of each flight (14 words each; all of
// a monoplane) live in its own lane of TMEM, 12 x 42 of the 512 columns, written by tcgen05.st when the
// flight is staged and read back each step by tcgen05.ld.  The other pairs of a biplane (76 at most)
// stay in shared memory, 4.3 KB per flight, beside the flight's state and constants, which leave the
// registers to the panel part (142 of them, no spills).
//
// Bound: register reads.  A packed FMA of three register operands reads six registers through two
// banks, three cycles instead of the pipe's two; per flight-step 172 packed and 67 scalar FMA-pipe
// instructions take 592 cycles of a scheduler (411 by pipe rate, about 540 by reads).  16 warps of three
// flights (128 registers) took 203.9 ms where 12 of four took 189.3, so more warps do not help.
// Measured, 100,000 x 12 flights: 218.3 ms a flight per half warp, 195.2 four per warp with the state in
// registers, 189.3 in shared memory, 184.5 with warp-uniform control flow and the hand-over, 174.4 with
// the four flights' code unrolled (no copies between the folds), 173.0 with the packed constants in the
// constant bank, 172.1 with a gust sine per lane.
//
// The sums run in the fixed order of pe_flight_fast.cuh, so every distance and step count is
// bit-identical to the other kernels'.
#include "pe_flight_fast.cuh"

namespace pe {

namespace {

constexpr int kQuadWarps = 12;            // warps per block, one block per SM
constexpr int kQuadFlights = 4;           // flights per warp
constexpr int kTmPairs = 3;               // pairs per lane and flight in TMEM
constexpr int kTmWords = 14 * kTmPairs;   // 42 columns: 32 + 8 + 2
constexpr int kSmPairs = kNtMax / 2 - 32 * kTmPairs;  // 76 pairs of a flight in shared memory
constexpr int kSmSlots = kSmPairs + 1;    // and one of zeros for the lanes past the last pair
// Column regions of a warp quarter's three warps x four flights, each naturally aligned for its load.
constexpr int kTmCol32 = 0, kTmCol8 = 12 * 32, kTmCol2 = 12 * 40;
static_assert(kTmCol2 + 12 * 2 <= 512, "tensor memory has 512 columns");
static_assert(kQuadWarps == 12, "three warps per TMEM quarter");

struct QuadFlightSmem {
    float4 a[kSmSlots], b[kSmSlots], c[kSmSlots];
    float2 d[kSmSlots];
    float2 pad;
    float4 k[3];     // the step's constants: vb xyz, each twice, then wb xyz and the skin friction
    float4 rows[3];  // its attitude rows
    float4 st[4];    // the flight's state (FlightState)
    float4 fc[6];    // and constants (FastConst)
};
static_assert(sizeof(QuadFlightSmem) % 16 == 0, "float4 arrays of the next flight stay aligned");

__device__ __forceinline__ void tm_alloc_all(uint32_t* slot) {
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(slot);
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(at) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

union ConstWords {
    FastConst fc;
    float4 v[6];
    __device__ ConstWords() {}
};
union StateWords {
    FlightState st;
    float4 v[4];
    __device__ StateWords() {}
};
static_assert(sizeof(FastConst) <= sizeof(float4) * 6, "a flight's constants fit their record");

// One lane's 42 words of a flight.
struct TmWords { uint32_t w[kTmWords]; };

__device__ __forceinline__ void tm_store(uint32_t c32, uint32_t c8, uint32_t c2, const TmWords& x) {
    const uint32_t* w = x.w;
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(c32),
        "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "r"(w[8]), "r"(w[9]),
        "r"(w[10]), "r"(w[11]), "r"(w[12]), "r"(w[13]), "r"(w[14]), "r"(w[15]), "r"(w[16]), "r"(w[17]), "r"(w[18]),
        "r"(w[19]), "r"(w[20]), "r"(w[21]), "r"(w[22]), "r"(w[23]), "r"(w[24]), "r"(w[25]), "r"(w[26]), "r"(w[27]),
        "r"(w[28]), "r"(w[29]), "r"(w[30]), "r"(w[31])
        : "memory");
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(c8), "r"(w[32]),
                 "r"(w[33]), "r"(w[34]), "r"(w[35]), "r"(w[36]), "r"(w[37]), "r"(w[38]), "r"(w[39])
                 : "memory");
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(c2), "r"(w[40]), "r"(w[41]) : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// The loads and their wait are one statement, so no use of the words can move ahead of the wait; its outputs are
// written before its last input is read (&: none may share a register with an input).
__device__ __forceinline__ void tm_load(uint32_t c32, uint32_t c8, uint32_t c2, TmWords& x) {
    uint32_t* w = x.w;
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%42];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%32, %33, %34, %35, %36, %37, %38, %39}, [%43];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x2.b32 {%40, %41}, [%44];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=&r"(w[0]), "=&r"(w[1]), "=&r"(w[2]), "=&r"(w[3]), "=&r"(w[4]), "=&r"(w[5]), "=&r"(w[6]), "=&r"(w[7]), "=&r"(w[8]),
          "=&r"(w[9]), "=&r"(w[10]), "=&r"(w[11]), "=&r"(w[12]), "=&r"(w[13]), "=&r"(w[14]), "=&r"(w[15]), "=&r"(w[16]),
          "=&r"(w[17]), "=&r"(w[18]), "=&r"(w[19]), "=&r"(w[20]), "=&r"(w[21]), "=&r"(w[22]), "=&r"(w[23]), "=&r"(w[24]),
          "=&r"(w[25]), "=&r"(w[26]), "=&r"(w[27]), "=&r"(w[28]), "=&r"(w[29]), "=&r"(w[30]), "=&r"(w[31]), "=&r"(w[32]),
          "=&r"(w[33]), "=&r"(w[34]), "=&r"(w[35]), "=&r"(w[36]), "=&r"(w[37]), "=&r"(w[38]), "=&r"(w[39]), "=&r"(w[40]),
          "=&r"(w[41])
        : "r"(c32), "r"(c8), "r"(c2)
        : "memory");
}

__device__ __forceinline__ f2 word2(const TmWords& x, int i) {
    return pk(__uint_as_float(x.w[i]), __uint_as_float(x.w[i + 1]));
}

// A value that all lanes hold.  Every branch around the panel part hangs on such values, so that the
// compiler can prove the warp converged there and use the uniform datapath for its addresses
// and the step's rates (186.3 to 184.9 ms at 100,000 x 12; loaded as packed pairs instead: 176.3 to 174.4).
__device__ __forceinline__ unsigned uniform_(unsigned x) { return __reduce_or_sync(0xffffffffu, x); }
__device__ __forceinline__ int uniform_(int x) { return (int)uniform_((unsigned)x); }

__device__ __forceinline__ f2 bcu(unsigned x) {
    f2 r;
    asm volatile("mov.b64 %0, {%1, %1};" : "=l"(r) : "r"(x));
    return r;
}

// Staged pair q of a flight: 14 words in the order rbx, rby, rbz, ak, nbx, nby, nbz (even, odd panel).
__device__ __forceinline__ void quad_stage_pair(const FlightArgs& a, int off, int nt, int q, vec3 cg, float half_rho,
                                                float wp, float wr, float w[14]) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int i = 2 * q + h;
        float4 oa = make_float4(0, 0, 0, 0), ob = make_float4(0, 0, 0, 0);
        if (i < nt) fast_stage_one(a.pc[off + i], a.pn[off + i], cg, half_rho, wp, wr, &oa, &ob);
        w[h] = oa.x; w[2 + h] = oa.y; w[4 + h] = oa.z; w[6 + h] = oa.w;
        w[8 + h] = ob.x; w[10 + h] = ob.y; w[12 + h] = ob.z;
    }
}

// Level of the transposed reduction that halves two sets of six: lanes with bit `m` clear keep u,
// the others v.
__device__ __forceinline__ void fold6(float u[6], const float v[6], int m, bool up) {
#pragma unroll
    for (int c = 0; c < 6; c++) {
        const float send = up ? u[c] : v[c];
        const float keep = up ? v[c] : u[c];
        u[c] = add_(keep, __shfl_xor_sync(0xffffffffu, send, m));
    }
}

__global__ void __launch_bounds__(32 * kQuadWarps, 1) k_flight_quad(FlightArgs a) {
    extern __shared__ float4 smem[];
    __shared__ uint32_t s_tm;
    const int lane = threadIdx.x & 31, warp = uniform_((int)threadIdx.x >> 5);
    const int g = lane >> 3;  // the flight slot this lane integrates
    QuadFlightSmem* sf = reinterpret_cast<QuadFlightSmem*>(smem) + warp * kQuadFlights;
    if (warp == 0) tm_alloc_all(&s_tm);
    if (lane < kQuadFlights) {  // the zero pair of each flight
        sf[lane].a[kSmPairs] = sf[lane].b[kSmPairs] = sf[lane].c[kSmPairs] = make_float4(0, 0, 0, 0);
        sf[lane].d[kSmPairs] = make_float2(0, 0);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // a warp reaches the 32 TMEM lanes of its quarter; its four flights' columns follow its turn there
    const uint32_t tm = uniform_(s_tm) + ((uint32_t)(warp & 3) << 21);
    const int tm_first = (warp >> 2) * kQuadFlights;

    WindLane wl = wind_lane(lane, 0.0f);  // of this lane's slot, as
    int flight = -1, step = 0;
    unsigned deck2 = 0;         // slots whose plane has pairs in shared memory (warp-uniform)
    unsigned busy = 0;          // slots in flight (warp-uniform)
    bool more = true;
    while (true) {
        // refill the empty slots
        while (more && busy != 0xfu) {
            const int slot = __ffs(~busy) - 1;
            int f = 0;
            if (lane == 0) f = atomicAdd(a.work, 1);
            f = uniform_(f);
            if (f >= a.n_flights) { more = false; break; }
            const int p = f / a.nseeds, s = f - p * a.nseeds;
            const int nt = uniform_(a.plane_nt[p]);
            if (nt <= 0) {
                if (lane == 0) {
                    a.dist[f] = -100.0f;
                    a.steps[f] = 0;
                    atomicAdd(a.landed, 1);
                }
                continue;
            }
            ConstWords nfc;
            vec3 cg;
            float air_rho, wp, wr;
            MassProps pmp;
            Scenario sc;
            StateWords nst;
            fast_setup(a, p, s, &nfc.fc, &cg, &air_rho, &wp, &wr, &pmp, &sc);
            release(sc, pmp, cg, &nst.st);
            if (g == slot) { flight = f; step = 0; wl = wind_lane(lane, nfc.fc.phase); }
            if (lane == 0) {
#pragma unroll
                for (int i = 0; i < 6; i++) sf[slot].fc[i] = nfc.v[i];
#pragma unroll
                for (int i = 0; i < 4; i++) sf[slot].st[i] = nst.v[i];
            }
            const int off = a.plane_off[p];
            const float half_rho = mul_(0.5f, air_rho);
            TmWords tw;
#pragma unroll
            for (int k = 0; k < kTmPairs; k++) {
                float w[14];
                quad_stage_pair(a, off, nt, lane + 32 * k, cg, half_rho, wp, wr, w);
#pragma unroll
                for (int i = 0; i < 14; i++) tw.w[14 * k + i] = __float_as_uint(w[i]);
            }
            const int at = tm_first + slot;
            __syncwarp();
            tm_store(tm + kTmCol32 + 32 * at, tm + kTmCol8 + 8 * at, tm + kTmCol2 + 2 * at, tw);
            busy |= 1u << slot;
            deck2 &= ~(1u << slot);
            if (nt > 2 * 32 * kTmPairs) {
                deck2 |= 1u << slot;
                QuadFlightSmem& S = sf[slot];
                for (int q = lane; q < kSmPairs; q += 32) {
                    float w[14];
                    quad_stage_pair(a, off, nt, 32 * kTmPairs + q, cg, half_rho, wp, wr, w);
                    S.a[q] = make_float4(w[0], w[1], w[2], w[3]);
                    S.b[q] = make_float4(w[4], w[5], w[6], w[7]);
                    S.c[q] = make_float4(w[8], w[9], w[10], w[11]);
                    S.d[q] = make_float2(w[12], w[13]);
                }
            }
            __syncwarp();
        }
        if (busy == 0) break;

        // steps of the slots in flight until one of them ends
        const bool mine = (busy >> g) & 1u;
        bool leave, give = false;
        int tick = 0, seen = 0;
        do {
            // The flight's state, constants and attitude rows stay in shared memory over the panel
            // part, which needs the registers for independent pairs.
            {
                ConstWords cw;
                StateWords sw;
#pragma unroll
                for (int i = 0; i < 6; i++) cw.v[i] = sf[g].fc[i];
#pragma unroll
                for (int i = 0; i < 4; i++) sw.v[i] = sf[g].st[i];
                const StepPre pre = fast_pre<true>(cw.fc, sw.st, step, &wl);
                __syncwarp();  // the last step's reads of k are done
                if ((lane & 7) == 0) {
                    float4* k = sf[g].k;
                    const vec3 vb = pre.vb, wb = sw.st.wb;
                    k[0] = make_float4(vb.x, vb.x, vb.y, vb.y);
                    k[1] = make_float4(vb.z, vb.z, 0.0f, 0.0f);
                    k[2] = make_float4(wb.x, wb.y, wb.z, cw.fc.skin_cf);
                    sf[g].rows[0] = make_float4(pre.r0.x, pre.r0.y, pre.r0.z, pre.r1.x);
                    sf[g].rows[1] = make_float4(pre.r1.y, pre.r1.z, pre.r2.x, pre.r2.y);
                    sf[g].rows[2] = make_float4(pre.r2.z, sw.st.t, 0.0f, 0.0f);
                }
            }
            __syncwarp();
            float sum[6];
            // slots 0 and 2, folded over lane bit 4, then 1 and 3; the two results over lane bit 3
#pragma unroll
            for (int half = 0; half < 2; half++) {
                float u[6];
#pragma unroll
                for (int part = 0; part < 2; part++) {
                    const int slot = half + 2 * part;
                    float v[6] = {0, 0, 0, 0, 0, 0};
                    if ((busy >> slot) & 1u) {
                        const QuadFlightSmem& S = sf[slot];
                        const float4 k0 = S.k[0], k2 = S.k[2];
                        const float2 k1 = *reinterpret_cast<const float2*>(&S.k[1]);
                        PairConst k;
                        k.vbx = pk(k0.x, k0.y); k.vby = pk(k0.z, k0.w); k.vbz = pk(k1.x, k1.y);
                        const unsigned ux = uniform_(__float_as_uint(k2.x)), uy = uniform_(__float_as_uint(k2.y)),
                                       uz = uniform_(__float_as_uint(k2.z)), ucf = uniform_(__float_as_uint(k2.w));
                        const float cf = __uint_as_float(ucf);
                        k.wbx = bcu(ux); k.wby = bcu(uy); k.wbz = bcu(uz);
                        k.nwbx = bcu(ux ^ 0x80000000u); k.nwby = bcu(uy ^ 0x80000000u); k.nwbz = bcu(uz ^ 0x80000000u);
                        k.cf = bcu(ucf);
                        k.k19 = c_k19; k.tiny = c_tiny; k.mone = c_mone;
                        const int at = tm_first + slot;
                        TmWords x;
                        tm_load(tm + kTmCol32 + 32 * at, tm + kTmCol8 + 8 * at, tm + kTmCol2 + 2 * at, x);
                        PairAcc acc;
                        pair_eval<true>(word2(x, 0), word2(x, 2), word2(x, 4), word2(x, 6), word2(x, 8), word2(x, 10),
                                        word2(x, 12), k, cf, acc);
#pragma unroll
                        for (int n = 1; n < kTmPairs; n++) {
                            const int o = 14 * n;
                            pair_eval(word2(x, o), word2(x, o + 2), word2(x, o + 4), word2(x, o + 6), word2(x, o + 8),
                                      word2(x, o + 10), word2(x, o + 12), k, cf, acc);
                        }
                        if ((deck2 >> slot) & 1u) {
                            PairedPanels pp;
                            pp.a = const_cast<float4*>(S.a); pp.b = const_cast<float4*>(S.b);
                            pp.c = const_cast<float4*>(S.c); pp.d = const_cast<float2*>(S.d);
                            fast_pair(pp, lane, k, cf, acc);
                            fast_pair(pp, lane + 32, k, cf, acc);
                            fast_pair(pp, lane < kSmPairs - 64 ? lane + 64 : kSmPairs, k, cf, acc);
                        }
                        pair_acc_total(acc, v);
                    }
                    if (part == 0) {
#pragma unroll
                        for (int c = 0; c < 6; c++) u[c] = v[c];
                    } else {
                        fold6(u, v, 16, (lane & 16) != 0);
                    }
                }
                if (half == 0) {
#pragma unroll
                    for (int c = 0; c < 6; c++) sum[c] = u[c];
                } else {
                    fold6(sum, u, 8, (lane & 8) != 0);
                }
            }
            // eight lanes hold their flight's six values each: three, two, then one value per lane
            {
                const bool up4 = (lane & 4) != 0, up2 = (lane & 2) != 0, up1 = (lane & 1) != 0;
                float v[4];
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    const float send = up4 ? sum[i] : sum[i + 3];
                    const float keep = up4 ? sum[i + 3] : sum[i];
                    v[i] = add_(keep, __shfl_xor_sync(0xffffffffu, send, 4));
                }
                v[3] = 0.0f;
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const float send = up2 ? v[i] : v[i + 2];
                    const float keep = up2 ? v[i + 2] : v[i];
                    v[i] = add_(keep, __shfl_xor_sync(0xffffffffu, send, 2));
                }
                const float send = up1 ? v[0] : v[1];
                const float keep = up1 ? v[1] : v[0];
                const float t = add_(keep, __shfl_xor_sync(0xffffffffu, send, 1));
                // component c = 3 b4 + i, i = 2 b2 + b1
#pragma unroll
                for (int c = 0; c < 6; c++) {
                    const int i = c % 3;
                    sum[c] = __shfl_sync(0xffffffffu, t, (c / 3) * 4 + (i >> 1) * 2 + (i & 1), 8);
                }
            }
            float fit = 0.0f;
            int done = 0;
            ConstWords cw;
            StateWords sw;
            StepPre pre;
            {
#pragma unroll
                for (int i = 0; i < 6; i++) cw.v[i] = sf[g].fc[i];
#pragma unroll
                for (int i = 0; i < 4; i++) sw.v[i] = sf[g].st[i];
                const float4 w0 = sf[g].rows[0], w1 = sf[g].rows[1], w2 = sf[g].rows[2];
                pre.r0 = mk3(w0.x, w0.y, w0.z);
                pre.r1 = mk3(w0.w, w1.x, w1.y);
                pre.r2 = mk3(w1.z, w1.w, w2.x);
                sw.st.t = w2.y;
            }
            FastConst& fc = cw.fc;
            FlightState& st = sw.st;
            if (mine) done = fast_post(fc, pre, sum, st, step, a.max_steps, a.smooth, &fit, nullptr, nullptr);
            step++;
            __syncwarp();
            if ((lane & 7) == 0) {
#pragma unroll
                for (int i = 0; i < 4; i++) sf[g].st[i] = sw.v[i];
            }
            __syncwarp();
            leave = mine && done;
            if (leave && (lane & 7) == 0) {
                a.dist[flight] = fit;
                a.steps[flight] = step;
                atomicAdd(a.landed, 1);
            }
            // few flights left in the whole launch: hand this warp's over (judged on a count that was asked
            // for eight steps before, so that no step waits for it)
            if (!more && (++tick & 7) == 0) {
                give = a.n_flights - uniform_(seen) <= a.hand_over;
                seen = *(volatile int*)a.landed;
            }
        } while (!give && !__any_sync(0xffffffffu, leave));
        if (give) {
            if (mine && !leave && (lane & 7) == 0) {
                StateWords sw;
#pragma unroll
                for (int i = 0; i < 4; i++) sw.v[i] = sf[g].st[i];
                sw.st.step = step;
                a.state[flight] = sw.st;
                a.active_out[atomicAdd(a.n_active_out, 1)] = flight;
            }
            busy = 0;
        }
        const unsigned left = __ballot_sync(0xffffffffu, leave);
#pragma unroll
        for (int i = 0; i < kQuadFlights; i++)
            if ((left >> (8 * i)) & 1u) busy &= ~(1u << i);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(s_tm) : "memory");
}

constexpr size_t kQuadSmem = sizeof(QuadFlightSmem) * kQuadWarps * kQuadFlights;

}  // namespace

cudaError_t flight_quad_configure() {
    return cudaFuncSetAttribute(k_flight_quad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kQuadSmem);
}

cudaError_t launch_flight_quad(const FlightArgs& a, int nsm, cudaStream_t s) {
    // whole flights from their release, the last ones handed over
    if (a.rec || a.spread > 0.f || a.grad_setup || a.active_in || a.step_begin != 0 || a.step_end < a.max_steps ||
        !a.landed || !a.active_out || !a.n_active_out)
        return cudaErrorInvalidValue;
    k_flight_quad<<<nsm, 32 * kQuadWarps, kQuadSmem, s>>>(a);
    return cudaGetLastError();
}

}  // namespace pe
