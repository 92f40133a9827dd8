// pe_prepare.cu -- genome -> mesh -> mass properties -> packed panels (src/sim.cu:25-49).
//
// Three launches, k_mesh alone for at most kScanAlone genomes (each block counts the planes before its own):
//   k_topo_scan   triangle count of each genome from its topology genes alone, block-local
//                 exclusive scan, block totals out.
//   k_scan_tot    exclusive scan of the block totals (one block, 1024 at a time); also the
//                 grand total.
//   k_mesh        a block per plane: threads evaluate the mesh vertices in parallel into shared
//                 memory and every triangle's mass-property terms likewise; then each sum is one
//                 lane's, in emission order (the reference's order, so the sums round identically);
//                 the COM-relative panel SoA goes into the plane's exact prefix range.
// HBM traffic is small (140 B genome in, 32 B per panel out); the cost is the ordered sums.
#include "pe_internal.cuh"

namespace pe {

__global__ void __launch_bounds__(kScanBlock) k_topo_scan(PrepArgs a) {
    __shared__ int warp_tot[kScanBlock / 32];
    int p = blockIdx.x * kScanBlock + threadIdx.x;
    int n = 0;
    if (p < a.pop) {
        GenomeRef g{a.genomes + (size_t)p * kGenomeN};
        n = topology(g).nt;
        a.nt_topo[p] = n;
    }
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = n;
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[w] = x;
    __syncthreads();
    if (w == 0) {
        int t = warp_tot[lane];
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        warp_tot[lane] = t;  // inclusive
    }
    __syncthreads();
    int excl = x - n + (w > 0 ? warp_tot[w - 1] : 0);
    if (p < a.pop) a.pt.off[p] = excl;  // block-local for now
    if (threadIdx.x == kScanBlock - 1) a.block_sum[blockIdx.x] = excl + n;
}

// Exclusive scan of nblocks block totals in place, in tiles of 1024 with the running sum of the
// earlier tiles carried through shared memory (PE_MAX_POP planes are 4,096 tiles); grand total to
// *total.  One block: the tiles follow one another.
__global__ void __launch_bounds__(1024) k_scan_tot(int* block_sum, int nblocks, int* total) {
    __shared__ int warp_tot[32];
    __shared__ int carry;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < nblocks; base += 1024) {
        const int i = base + threadIdx.x;
        const int n = i < nblocks ? block_sum[i] : 0;
        int x = n;
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_tot[w] = x;
        __syncthreads();
        if (w == 0) {
            int t = warp_tot[lane];
            for (int o = 1; o < 32; o <<= 1) {
                int y = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= o) t += y;
            }
            warp_tot[lane] = t;
        }
        __syncthreads();
        const int c = carry;
        const int excl = c + x - n + (w > 0 ? warp_tot[w - 1] : 0);
        if (i < nblocks) block_sum[i] = excl;
        __syncthreads();  // every thread has read carry and warp_tot
        if (threadIdx.x == 1023) carry = excl + n;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

// A block per plane: all threads take the vertices and the sums' terms; then warp 0 adds in order while
// warp 1 finds the extent, and once more while the others write the panels.  Bound by the two chains of
// ordered sums and what leads up to them.  The preparation's launches together, with a warp per plane (two
// per block of 46 KB, eight per SM) and so: 21.5 -> 17.5 us for one plane, 31 -> 23 for 8 to 128 (14.3 and 19.3
// without the counting launch), 88 -> 69 for 3,001, 184 -> 141 for 8,192, 1,920 -> 1,430 for 100,000.
constexpr int kMeshThreads = 128;

// A small batch's preparation is its launches: 3.6 us of 18 at one genome, 5 of 24 at 128, for counting the
// planes' triangles; a block's own count of the planes before it takes a thread each.
constexpr int kScanAlone = kMeshThreads;

template <bool ALONE>
__global__ void __launch_bounds__(kMeshThreads, 8) k_mesh(PrepArgs a, int* total) {
    __shared__ float s_g[kGenomeN + 1];
    __shared__ vec3 s_v[kNvMax];
    __shared__ float s_com[5];
    __shared__ float s_terms[kMpTerms * kNtMax];
    __shared__ int s_nt, s_before[kMeshThreads / 32];
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int p = blockIdx.x;
    if (tid < kGenomeN) s_g[tid] = a.genomes[(size_t)p * kGenomeN + tid];
    if (ALONE) {  // triangles of the planes before this one, a thread each
        const int n = tid < p ? topology(GenomeRef{a.genomes + (size_t)tid * kGenomeN}).nt : 0;
        const int sum = __reduce_add_sync(0xffffffffu, n);
        if (lane == 0) s_before[w] = sum;
    }
    __syncthreads();
    GenomeRef g{s_g};
    const Topo tp = topology(g);
    for (int i = tid; i < tp.nv; i += kMeshThreads) s_v[i] = mesh_vertex(g, tp, i);
    const int off = ALONE ? s_before[0] + s_before[1] + s_before[2] + s_before[3]
                          : a.pt.off[p] + a.block_sum[p / kScanBlock];
    if (ALONE && tid == 0 && p == a.pop - 1) *total = off + tp.nt;
    __syncthreads();
    mass_first(s_v, tp, tid, kMeshThreads, s_terms);
    __syncthreads();
    if (w == 0) {
        mass_com(g, tp, lane, s_terms, s_com);
    } else if (w == 1) {
        // mesh extent (min/max are exact in any order), src/common.h:294-307
        vec3 lo = s_v[0], hi = lo;
        for (int i = lane; i < tp.nv; i += 32) {
            vec3 v = s_v[i];
            lo.x = fminf(lo.x, v.x); lo.y = fminf(lo.y, v.y); lo.z = fminf(lo.z, v.z);
            hi.x = fmaxf(hi.x, v.x); hi.y = fmaxf(hi.y, v.y); hi.z = fmaxf(hi.z, v.z);
        }
        for (int o = 16; o > 0; o >>= 1) {
            lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, o));
            lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, o));
            lo.z = fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, o));
            hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, o));
            hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, o));
            hi.z = fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, o));
        }
        vec3 ext = vsub(hi, lo);
        const float lim = PE_PRINT_LIMIT;
        const int printable = ext.x <= lim && ext.y <= lim && ext.z <= lim;
        if (lane == 0) {
            s_nt = printable ? tp.nt : 0;
            a.pt.nt[p] = s_nt;
            a.pt.off[p] = off;
            a.pt.ext[p] = make_float4(ext.x, ext.y, ext.z, (float)tp.nt);
        }
    }
    __syncthreads();
    const vec3 com = mk3(s_com[0], s_com[1], s_com[2]);
    mass_second(s_v, tp, tid, kMeshThreads, com, s_terms);
    __syncthreads();
    if (w == 0) {
        MassProps mp;
        mass_inertia(g, tp, lane, s_terms, s_com, &mp);
        if (lane == 0) {
            float* o = a.pt.mp + (size_t)p * kMpN;
            o[0] = mp.mass; o[1] = mp.invmass; o[2] = mp.com.x; o[3] = mp.com.y; o[4] = mp.com.z;
            for (int k = 0; k < 6; k++) o[5 + k] = mp.I[k];
            for (int k = 0; k < 9; k++) o[11 + k] = mp.invI[k];
        }
        return;
    }
    // COM-relative panels, src/sim.cu:40-48
    const int nt = s_nt;
    for (int t = tid - 32; t < nt; t += kMeshThreads - 32) {
        int ia, ib, ic; mesh_tri(tp, t, &ia, &ib, &ic);
        vec3 pa = vsub(s_v[ia], com), pb = vsub(s_v[ib], com), pcv = vsub(s_v[ic], com);
        vec3 nrm = vcross(vsub(pb, pa), vsub(pcv, pa));
        float A = 0.5f * vlen(nrm);
        vec3 ct = vscl(vadd(vadd(pa, pb), pcv), 1.0f / 3);
        a.pc[off + t] = make_float4(ct.x, ct.y, ct.z, A);
        vec3 n = A > 1e-12f ? vscl(nrm, 0.5f / A) : mk3(0, 0, 1);
        a.pn[off + t] = make_float4(n.x, n.y, n.z, 0.0f);
    }
}

cudaError_t set_station_mode(int ieee) {
    int v = ieee ? 1 : 0;
    return cudaMemcpyToSymbol(c_station_ieee, &v, sizeof(int));
}

int launch_prepare(const PrepArgs& a, int* d_total, cudaStream_t s) {
    int nb = (a.pop + kScanBlock - 1) / kScanBlock;
    if (a.pop <= kScanAlone) {
        k_mesh<true><<<a.pop, kMeshThreads, 0, s>>>(a, d_total);
        return 1;
    }
    k_topo_scan<<<nb, kScanBlock, 0, s>>>(a);
    k_scan_tot<<<1, 1024, 0, s>>>(a.block_sum, nb, d_total);
    k_mesh<false><<<a.pop, kMeshThreads, 0, s>>>(a, d_total);
    return 3;
}

}  // namespace pe
