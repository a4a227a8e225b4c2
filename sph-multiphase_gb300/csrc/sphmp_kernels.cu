// sphmp_kernels.cu — CUDA kernels of the multiphase SPH step for sm_103a.
//
// Reference parity notes (ZP-Z/sph-multiphase):
//  * the hash reproduces InitialSort (SPH_Solver/fluids/fluid_system_kern.cu:36-64)
//    with the same float operations, so cell ids are bit-identical;
//  * the sort reproduces thrust::sort_by_key's stable order (fluid_system_host.cu:164-166)
//    by ranking every cell's members by their pre-sort slot, and also builds the
//    internal order of the particle state (cells as sorted, members grouped by
//    h-subcell inside each cell);
//  * neighbour sums follow the reference formulas (fluid_system_kern.cu:183-424,
//    multiphase.cu:19-349) in FP32 over the pairs closer than h, found by the
//    bucket density kernel (one warp per h-subcell, the 27 h-subcells around it)
//    and kept as index lists for the force, drift and volume-fraction passes;
//  * the advance reproduces AdvanceParticles (fluid_system_kern.cu:426-534) with
//    un-contracted float operations, so it is bit-identical given the same accel.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <type_traits>

#include "sphmp_device.cuh"
#include "sphmp_features.cuh"
#include "sphmp_emit.h"
#include "sphmp_internal.h"

namespace sphmp {

namespace {

using namespace dev;

// ---------------------------------------------------------------------------
// Hash + histogram (GetParticleIndexCUDA)
// ---------------------------------------------------------------------------

// One block = one chunk of kHashBlock slots. In-grid slots take a rank inside
// their cell from a warp-aggregated atomic (the order is fixed later by the
// cell sort) and, with `sums` (the linear order only), are counted per kScanPer
// cells as well, so that the scan that follows at once in a step needs no pass of
// its own for its blocks' sums; out-of-grid slots
// get their exact rank inside the chunk, and the chunk totals, also summed per
// kHashBlock chunks, place them in slot order. The first block clears the
// control words of the sort and the passes after it.
__global__ void __launch_bounds__(kHashBlock) k_hash(const __grid_constant__ DevParams P,
                                                     const __grid_constant__ DevBuffers B,
                                                     const float4* __restrict__ pos4, int sums) {
    __shared__ uint32_t wcount[kHashBlock / 32];
    const int i = blockIdx.x * kHashBlock + threadIdx.x;
    if (i < kCtlWords) B.ctl[i] = 0u;
    if (i == 0) *B.counted = 1u;
    const bool valid = i < active_n(B);
    uint32_t key = kUndef;
    if (valid) {
        const float4 p = pos4[B.opos[i]];
        key = cell_key(P, p.x, p.y, p.z);
        B.key[i] = key;
        B.mgcell[i] = key;
        if (key != kUndef) B.octk[i] = (uint8_t)octant_of(P, p);  // for the per-cell octant order
    }
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    const bool in = valid && key != kUndef;
    const unsigned im = __ballot_sync(0xffffffffu, in);
    if (in) {
        const unsigned peers = __match_any_sync(im, key);
        const int leader = __ffs(peers) - 1;
        uint32_t base = 0;
        if ((int)lane == leader) base = atomicAdd(&B.ccount[key], (uint32_t)__popc(peers));
        base = __shfl_sync(peers, base, leader);
        B.arank[i] = base + __popc(peers & lanemask_lt());
    }
    // All go to the same few words, so a block adds up what it counts into one sum and adds that with
    // one atomic, for up to four sums, one after the other (slots are nearly in cell
    // order after a sort: one or two sums); the rest by warps. (One atomic a warp: 40
    // instead of 20 us at 1.3 M sorted slots; one sum a block and the rest one by one:
    // 127 us instead of 14.5 for 913 K slots as uploaded.)
    if (sums) {
        __shared__ volatile uint32_t shared_sum;
        const uint32_t sum = key / kScanPer;
        bool open = in;
        int left = __syncthreads_count((int)open);
        for (int round = 0; round < 4 && left > 0; round++) {
            if (open) shared_sum = sum;  // any of the open ones
            __syncthreads();
            const uint32_t f = shared_sum;
            const int same = __syncthreads_count((int)(open && sum == f));
            if (threadIdx.x == 0) atomicAdd(&B.bsum[f], (uint32_t)same);
            open = open && sum != f;
            left -= same;
        }
        if (left > 0) {
            const unsigned om = __ballot_sync(0xffffffffu, open);
            if (open) {
                const unsigned peers = __match_any_sync(om, sum);
                if ((int)lane == __ffs(peers) - 1) atomicAdd(&B.bsum[sum], (uint32_t)__popc(peers));
            }
        }
    }
    const bool und = valid && key == kUndef;
    const unsigned ub = __ballot_sync(0xffffffffu, und);
    if (!__syncthreads_or((int)und)) {  // the usual case
        if (threadIdx.x == 0) B.uchunk[blockIdx.x] = 0u;
        return;
    }
    if (lane == 0) wcount[warp] = __popc(ub);
    __syncthreads();
    if (warp == 0) {
        constexpr int nw = kHashBlock / 32;
        uint32_t v = lane < nw ? wcount[lane] : 0u;
        uint32_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if ((int)lane >= o) x += y;
        }
        if ((int)lane < nw) wcount[lane] = x - v;
        if ((int)lane == nw - 1) {
            B.uchunk[blockIdx.x] = x;
            atomicAdd(&B.usum[blockIdx.x / kHashBlock], x);
        }
    }
    __syncthreads();
    if (und) B.arank[i] = wcount[warp] + __popc(ub & lanemask_lt());
}

// The counts again from the keys of the last hash, for a GetGridList after they were
// cleared: by the sort of a captured step, or with counts that the caller uploaded.
// Whether they were is known on the device alone (a list may be replayed from a caller's
// graph), so this ends here if not.
__global__ void __launch_bounds__(kHashBlock) k_recount(const __grid_constant__ DevParams P,
                                                        const __grid_constant__ DevBuffers B) {
    if (*B.counted) return;
    const int n = active_n(B);
    const int chunks = (n + kHashBlock - 1) / kHashBlock;
    for (int g = blockIdx.x; g * kHashBlock < chunks; g += (int)gridDim.x) {
        const int k = g * kHashBlock + (int)threadIdx.x;
        __shared__ uint32_t part[kHashBlock / 32];
        const uint32_t v = __reduce_add_sync(0xffffffffu, k < chunks ? B.uchunk[k] : 0u);
        if (lane_id() == 0) part[threadIdx.x >> 5] = v;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t t = 0;
            for (int w = 0; w < kHashBlock / 32; w++) t += part[w];
            B.usum[g] = t;
        }
        __syncthreads();
    }
    for (int i = blockIdx.x * kHashBlock + (int)threadIdx.x; i < n; i += (int)gridDim.x * kHashBlock)
        if (B.key[i] != kUndef) atomicAdd(&B.ccount[B.key[i]], 1u);
}

// ---------------------------------------------------------------------------
// Prefix sums (GetGridListCUDA, part 1)
// ---------------------------------------------------------------------------

// Exclusive scan of one value per thread across a 1024-thread block.
template <class T>
__device__ __forceinline__ T block_excl_scan(T v, T* total) {
    __shared__ T ws[32];
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    T x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T y = __shfl_up_sync(0xffffffffu, x, o);
        if ((int)lane >= o) x += y;
    }
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    if (warp == 0) {
        T w = ws[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T y = __shfl_up_sync(0xffffffffu, w, o);
            if ((int)lane >= o) w += y;
        }
        ws[lane] = w;
    }
    __syncthreads();
    const T off = warp ? ws[warp - 1] : T(0);
    *total = ws[31];
    __syncthreads();
    return off + x - v;
}

__device__ __forceinline__ void load4(const uint32_t* in, int len, int idx, uint32_t v[4]) {
    if (idx + 3 < len && ((reinterpret_cast<uintptr_t>(in + idx) & 15u) == 0)) {
        const uint4 q = *reinterpret_cast<const uint4*>(in + idx);
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = (idx + k < len) ? in[idx + k] : 0u;
    }
}

// Counts of the cells at scan positions idx .. idx + 3: cell = position in the
// linear order, corder[position] in the Morton order.
__device__ __forceinline__ void load4_cells(const DevParams& P, const DevBuffers& B, int idx, uint32_t v[4]) {
    if (!P.morton) {
        load4(B.ccount, P.G, idx, v);
        return;
    }
#pragma unroll
    for (int k = 0; k < 4; k++) v[k] = idx + k < P.G ? B.ccount[B.corder[idx + k]] : 0u;
}

// Block sums of the cell counts in scan order, where the hash of the same step has not
// left them: the Morton order, and a cell list made by its own call, whose counts may
// be the caller's and whose order may have been changed since the hash. Such a list may
// be made twice from one hash, so the words that it counts with start from zero here
// (the queue of heavy particles is not among them: lists of neighbours may hold it).
__global__ void __launch_bounds__(kScanBlock) k_scan_reduce(const __grid_constant__ DevParams P,
                                                            const __grid_constant__ DevBuffers B) {
    const int idx = (blockIdx.x * kScanBlock + threadIdx.x) * kScanItems;
    if (idx < kListWords * kScanItems) B.ctl[idx / kScanItems] = 0u;
    uint32_t v[4];
    load4_cells(P, B, idx, v);
    uint32_t total;
    block_excl_scan(v[0] + v[1] + v[2] + v[3], &total);
    if (threadIdx.x == 0) B.bsum[blockIdx.x] = total;
}

// Cell starts, the reference's mgridoff / mgridcnt, the list of occupied cells and
// the list of cells too large for the warp sort, in one pass: every block adds up
// the sums of the blocks before it (a few dozen words) and scans its kScanPer
// counts together with their occupied flags (counts in the low 40 bits, flags
// above). `clear`: the counts are zeroed, for the next hash of captured steps. Bound by its chain: counts,
// two block scans, the stores, which take 16 bytes a thread and array (7 to 9 us at 11 K
// to 1.3 M particles; 10 to 13 with 4-byte stores and the counts read behind the first
// scan; three kernels, one of them a single block over the block sums and the chunks'
// out-of-grid counts, took 13 to 21).
__global__ void __launch_bounds__(kScanBlock) k_scan(const __grid_constant__ DevParams P,
                                                     const __grid_constant__ DevBuffers B, int clear) {
    __shared__ uint32_t act_base;
    const int idx = (blockIdx.x * kScanBlock + threadIdx.x) * kScanItems;
    uint32_t v[4];
    load4_cells(P, B, idx, v);  // beside the sums before, which the first block does not need
    uint32_t before = 0, run = 0;
    for (unsigned k = threadIdx.x; k < blockIdx.x; k += kScanBlock) before += B.bsum[k];
    if (blockIdx.x > 0) block_excl_scan(before, &run);
    uint64_t sum = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) sum += (uint64_t)v[k] + (v[k] ? 1ull << 40 : 0ull);
    uint64_t total;
    const uint64_t excl = block_excl_scan(sum, &total);
    if (threadIdx.x == 0) act_base = total >> 40 ? atomicAdd(B.act_n, (uint32_t)(total >> 40)) : 0u;
    __syncthreads();
    uint32_t at = act_base + (uint32_t)(excl >> 40);
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
        B.cstart[P.G] = run + (uint32_t)total;
        B.cstart[P.G + 1] = (uint32_t)active_n(B);
        *B.counted = clear ? 0u : 1u;
    }
    run += (uint32_t)excl;
    const bool four = !P.morton && idx + 3 < P.G;  // this thread's cells as 16-byte words
    if (four) {
        const uint32_t e0 = run + v[0], e1 = e0 + v[1], e2 = e1 + v[2], e3 = e2 + v[3];
        reinterpret_cast<uint4*>(B.cstart + idx)[0] = make_uint4(run, e0, e1, e2);
        reinterpret_cast<uint4*>(B.cend + idx)[0] = make_uint4(e0, e1, e2, e3);
        reinterpret_cast<uint4*>(B.mgridoff + idx)[0] = make_uint4(v[0] ? run : 0u, v[1] ? e0 : 0u, v[2] ? e1 : 0u, v[3] ? e2 : 0u);
        reinterpret_cast<uint4*>(B.mgridcnt + idx)[0] = make_uint4(v[0], v[1], v[2], v[3]);
        if (clear) reinterpret_cast<uint4*>(B.ccount + idx)[0] = make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (idx + k < P.G) {
            const int c = P.morton ? (int)B.corder[idx + k] : idx + k;
            if (!four) {
                B.cstart[c] = run;
                B.cend[c] = run + v[k];
                B.mgridoff[c] = v[k] ? (int32_t)run : 0;
                B.mgridcnt[c] = (int32_t)v[k];
                if (clear) B.ccount[c] = 0u;
            }
            if (v[k]) B.act[at++] = (uint32_t)c;
            if (v[k] > (uint32_t)kWarpSortMax) {
                if (v[k] > (uint32_t)kCtaSortMax) {
                    set_err(B, kErrCellOverflow);  // left unsorted; keep its octant ranges in bounds
                    for (int b = 0; b < 8; b++) B.oct_start[(size_t)c * 8 + b] = run;
                } else {
                    B.big[atomicAdd(B.big_n, 1u)] = (uint32_t)c;
                }
            }
        }
        run += v[k];
    }
}

// ---------------------------------------------------------------------------
// Scatter + per-cell stable order (GetGridListCUDA, part 2)
// ---------------------------------------------------------------------------

static_assert(kThreads == kHashBlock, "a scatter block holds one chunk of the hash");

__global__ void __launch_bounds__(kThreads) k_scatter(const __grid_constant__ DevParams P,
                                                      const __grid_constant__ DevBuffers B) {
    __shared__ uint32_t part[kThreads / 32];
    const int i = blockIdx.x * kThreads + threadIdx.x;
    const bool valid = i < active_n(B);
    const uint32_t key = valid ? B.key[i] : 0u;
    if (valid && key != kUndef) B.sidx[B.cstart[key] + B.arank[i]] = (uint32_t)i;
    const bool und = valid && key == kUndef;
    if (!__syncthreads_or((int)und)) return;
    // out-of-grid slots in the chunks before this one: whole groups of chunks, then this group's
    uint32_t v = 0;
    const unsigned grp = blockIdx.x / kHashBlock;
    for (unsigned k = threadIdx.x; k < grp; k += kThreads) v += B.usum[k];
    if (grp * kHashBlock + threadIdx.x < blockIdx.x) v += B.uchunk[grp * kHashBlock + threadIdx.x];
    v = __reduce_add_sync(0xffffffffu, v);
    if (lane_id() == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    if (!und) return;
    uint32_t d = B.cstart[P.G] + B.arank[i];
#pragma unroll
    for (int w = 0; w < kThreads / 32; w++) d += part[w];
    B.midsort[d] = (uint32_t)i;
    B.mgcell[d] = kUndef;
    B.mgndx[d] = kUndef;
    B.osrc[d] = B.opos[i];  // out-of-grid particles keep slot order at the end
    B.oidx[d] = d;
}

// Bitonic sort of 32*E keys held E per lane (element index = lane*E + r),
// ascending, entirely in registers.
template <int E>
__device__ __forceinline__ void warp_bitonic(uint32_t (&v)[E]) {
    const unsigned lane = lane_id();
    constexpr int M = 32 * E;
#pragma unroll
    for (int k = 2; k <= M; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= E) {
                const int lj = j / E;
#pragma unroll
                for (int r = 0; r < E; r++) {
                    const uint32_t o = __shfl_xor_sync(0xffffffffu, v[r], lj);
                    const unsigned idx = lane * E + r;
                    const bool asc = (idx & k) == 0;
                    const bool lower = (idx & j) == 0;
                    const uint32_t mn = min(v[r], o), mx = max(v[r], o);
                    v[r] = (lower == asc) ? mn : mx;
                }
            } else {
#pragma unroll
                for (int r = 0; r < E; r++) {
                    const int p = r ^ j;
                    if (p > r) {
                        const unsigned idx = lane * E + r;
                        const bool asc = (idx & k) == 0;
                        const uint32_t a = v[r], b = v[p];
                        const bool sw = asc ? (a > b) : (a < b);
                        v[r] = sw ? b : a;
                        v[p] = sw ? a : b;
                    }
                }
            }
        }
    }
}

// Write the internal order of cell c from the key (octant << shift | member index)
// held at sorted position q (cellstart + q is its internal index): the member's
// previous internal index src (osrc), its slot (oidx) and the bucket starts.
__device__ __forceinline__ void emit_octant(const DevBuffers& B, uint32_t c, uint32_t start, uint32_t cnt, uint32_t q,
                                            uint32_t key, uint32_t prev_oct, int shift, uint32_t src) {
    const uint32_t oct = key >> shift;
    const uint32_t idx = key & ((1u << shift) - 1u);
    if (q < cnt) {
        B.osrc[start + q] = src;
        B.oidx[start + q] = start + idx;
    }
    // bucket starts: every bucket in (prev_oct, oct] begins at q (8 marks past the end)
    const uint32_t hi = q < cnt ? oct : 8u;
    for (uint32_t b = prev_oct + 1; b <= hi && b < 8; b++) B.oct_start[(size_t)c * 8 + b] = start + q;
    if (q == cnt - 1)
        for (uint32_t b = oct + 1; b < 8; b++) B.oct_start[(size_t)c * 8 + b] = start + cnt;
}

// Queue the member windows after the first of bucket (c, b) = members [m0, m1)
// for the density pass (one warp per window of P.bwin members).
__device__ __forceinline__ void push_windows(const DevParams& P, const DevBuffers& B, uint32_t c, uint32_t b,
                                             uint32_t m0, uint32_t m1) {
    const uint32_t W = (uint32_t)P.bwin;
    if (m1 <= m0 + W) return;
    const uint32_t nw = (m1 - m0 - 1) / W;  // <= (m1 - m0) / kBucketWindowMin: wq never overflows
    const uint32_t base = atomicAdd(B.wq_n, nw);
    for (uint32_t i = 0; i < nw; i++) B.wq[base + i] = make_uint2(c * 8u + b, m0 + (i + 1) * W);
}

// Cell c, E members a lane: into the order of their slots (the reference's order), and
// from there by octant, which is a stable counting sort over the ballots of each
// octant: 5.5 us at 11 K slots, 20.5 at 913 K; with a second bitonic sort, and the
// bucket starts found between neighbouring keys, 7.2 and 32.
template <int E>
__device__ __forceinline__ void warp_sort_cell(const DevParams& P, const DevBuffers& B, uint32_t c, uint32_t start,
                                               uint32_t cnt) {
    uint32_t v[E];
    const unsigned lane = lane_id();
#pragma unroll
    for (int r = 0; r < E; r++) {
        const uint32_t idx = lane * E + r;
        v[r] = idx < cnt ? B.sidx[start + idx] : 0xFFFFFFFFu;
    }
    warp_bitonic<E>(v);
    uint32_t oct[E], src[E], q[E];
#pragma unroll
    for (int r = 0; r < E; r++) {
        const uint32_t idx = lane * E + r;
        oct[r] = 8u;
        src[r] = q[r] = 0u;
        if (idx < cnt) {
            oct[r] = B.octk[v[r]];
            src[r] = B.opos[v[r]];
            B.midsort[start + idx] = v[r];
            B.mgcell[start + idx] = c;
            B.mgndx[start + idx] = idx;
        }
    }
    uint32_t run = 0, first = 0;  // members before octant b; lane b: before its octant
#pragma unroll
    for (uint32_t b = 0; b < 8; b++) {
        uint32_t total = 0, below = 0;
#pragma unroll
        for (int r = 0; r < E; r++) {
            const uint32_t m = __ballot_sync(0xffffffffu, oct[r] == b);
            total += (uint32_t)__popc(m);
            below += (uint32_t)__popc(m & lanemask_lt());
        }
#pragma unroll
        for (int r = 0; r < E; r++)
            if (oct[r] == b) q[r] = run + below++;
        if (lane == b) first = run;
        run += total;
    }
#pragma unroll
    for (int r = 0; r < E; r++) {
        if (oct[r] < 8u) {
            B.osrc[start + q[r]] = src[r];
            B.oidx[start + q[r]] = start + lane * E + r;
        }
    }
    uint32_t next = __shfl_down_sync(0xffffffffu, first, 1);
    if (lane == 7) next = cnt;
    if (lane < 8) {
        B.oct_start[(size_t)c * 8 + lane] = start + first;
        if (cnt > (uint32_t)P.bwin) push_windows(P, B, c, lane, start + first, start + next);
    }
}

// One warp per cell (cells of up to kWarpSortMax members). Bound by the latency of its
// chain of loads (cell, its range, slots, octants) and of the sort. Six blocks per SM
// (at most 40 registers) let the warps' chains overlap.
__global__ void __launch_bounds__(kThreads, 6) k_cell_sort(const __grid_constant__ DevParams P,
                                                        const __grid_constant__ DevBuffers B) {
    const int nwarps = (gridDim.x * kThreads) >> 5;
    const uint32_t nact = *B.act_n;  // the occupied cells, listed by the scan
    for (uint32_t a = (blockIdx.x * kThreads + threadIdx.x) >> 5; a < nact; a += (uint32_t)nwarps) {
        const uint32_t c = B.act[a];
        const uint32_t start = B.cstart[c];
        const uint32_t cnt = B.cend[c] - start;
        if (cnt == 0 || cnt > (uint32_t)kWarpSortMax) continue;
        if (cnt <= 32) warp_sort_cell<1>(P, B, c, start, cnt);
        else if (cnt <= 64) warp_sort_cell<2>(P, B, c, start, cnt);
        else if (cnt <= 128) warp_sort_cell<4>(P, B, c, start, cnt);
        else warp_sort_cell<8>(P, B, c, start, cnt);
    }
}

__device__ __forceinline__ void cta_bitonic(uint32_t* sm, uint32_t M) {
    for (uint32_t k = 2; k <= M; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t t = threadIdx.x; t < M; t += blockDim.x) {
                const uint32_t p = t ^ j;
                if (p > t) {
                    const bool asc = (t & k) == 0;
                    const uint32_t a = sm[t], q = sm[p];
                    if (asc ? (a > q) : (a < q)) { sm[t] = q; sm[p] = a; }
                }
            }
            __syncthreads();
        }
    }
}

// One CTA per large cell (kWarpSortMax < members <= kCtaSortMax): bitonic sorts in shared memory.
__global__ void __launch_bounds__(1024) k_big_cell_sort(const __grid_constant__ DevParams P,
                                                        const __grid_constant__ DevBuffers B) {
    __shared__ uint32_t sm[kCtaSortMax];
    const uint32_t nbig = *B.big_n;
    for (uint32_t b = blockIdx.x; b < nbig; b += gridDim.x) {
        const uint32_t c = B.big[b];
        const uint32_t start = B.cstart[c];
        const uint32_t cnt = B.cend[c] - start;
        uint32_t M = 1;
        while (M < cnt) M <<= 1;
        for (uint32_t k = threadIdx.x; k < M; k += blockDim.x) sm[k] = k < cnt ? B.sidx[start + k] : 0xFFFFFFFFu;
        __syncthreads();
        cta_bitonic(sm, M);
        for (uint32_t k = threadIdx.x; k < cnt; k += blockDim.x) {
            B.midsort[start + k] = sm[k];
            B.mgcell[start + k] = c;
            B.mgndx[start + k] = k;
        }
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < M; k += blockDim.x)
            sm[k] = k < cnt ? (((uint32_t)B.octk[B.midsort[start + k]] << 13) | k) : 0xFFFFFFFFu;
        __syncthreads();
        cta_bitonic(sm, M);
        for (uint32_t q = threadIdx.x; q <= cnt && q < M + 1; q += blockDim.x) {
            const uint32_t k = q < cnt ? sm[q] : (8u << 13);
            const uint32_t pk = q == 0 ? 0xFFFFFFFFu : sm[q - 1];
            const uint32_t prev_oct = q == 0 ? 0xFFFFFFFFu : (pk >> 13);
            const uint32_t src = q < cnt ? B.opos[B.midsort[start + (k & 0x1FFFu)]] : 0u;
            emit_octant(B, c, start, cnt, q, k, prev_oct, 13, src);
        }
        __syncthreads();
        if (threadIdx.x < 8) {
            const uint32_t b0 = B.oct_start[(size_t)c * 8 + threadIdx.x];
            const uint32_t b1 = threadIdx.x == 7 ? start + cnt : B.oct_start[(size_t)c * 8 + threadIdx.x + 1];
            push_windows(P, B, c, threadIdx.x, b0, b1);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Reorder (RearrageDataCUDA)
// ---------------------------------------------------------------------------


// Every particle, out-of-grid ones included, moves to its new internal index
// (the reference gathers every slot: its `int cell != GRID_UNDEF` test at
// fluid_system_kern.cu:104-108 compares against a 64-bit literal on LP64 hosts
// and is always true there; out-of-grid particles are parked at (-1000)^3 by the
// advance), and the slot -> index map follows (no kernel reads opos between the
// cell order, which reads the old map, and this one).
__global__ void __launch_bounds__(kThreads) k_rearrange(const __grid_constant__ DevParams P,
                                                        const __grid_constant__ DevBuffers B,
                                                        const __grid_constant__ F4Set S, int clear) {
    const int o = blockIdx.x * kThreads + threadIdx.x;
    const int n = active_n(B);
    if (clear) {  // the sums the hash adds to, for the next one
        for (int k = o; k <= P.G / (int)kScanPer; k += (int)gridDim.x * kThreads) B.bsum[k] = 0u;
        for (int k = o; k <= (int)gridDim.x / kHashBlock; k += (int)gridDim.x * kThreads) B.usum[k] = 0u;
    }
    if (o >= n) return;
    uint32_t src = B.osrc[o];
    if (src >= (uint32_t)n) src = o;  // only after a cell-overflow error (flagged by the scan)
#pragma unroll
    for (int f = 0; f < kNumFloat4Fields; f++) S.out[f][o] = S.in[f][src];
    const uint32_t slot = B.oidx[o];
    if (slot < (uint32_t)n) B.opos[slot] = (uint32_t)o;
}

// New internal order = the sorted slot order (midsort given, no octant order).
__global__ void __launch_bounds__(kThreads) k_slot_order(const __grid_constant__ DevParams P,
                                                         const __grid_constant__ DevBuffers B) {
    const int s = blockIdx.x * kThreads + threadIdx.x;
    if (s >= active_n(B)) return;
    const uint32_t m = B.midsort[s];
    B.osrc[s] = m < (uint32_t)active_n(B) ? B.opos[m] : (uint32_t)s;
    B.oidx[s] = (uint32_t)s;
}

// ---------------------------------------------------------------------------
// Boundary volume (ComputeBoundaryDensity)
// ---------------------------------------------------------------------------

// kVolumeLanes lanes a particle share its candidate rows (one thread a particle is a
// serial chain of several hundred loads: 58 us at 11 K particles, 122 us at 1.3 M). A
// wall is a lattice, whose particles all round alike, and everything near it inherits
// their error, of one sign: with terms in plain FP32 the volumes were 7e-8 too small on
// average, which is what the mean residue of an IISPH solve then showed. So a term
// (h^2 - r^2)^3 carries its rounding errors (the differences of positions are exact but
// where a coordinate changes sign) and the volume is exact to a few 1e-9 before it is
// rounded once. In units in which the radius is 1 to 2 (vol_scale, a power of two). A
// sum costs 12, 133 and 162 us at 11 K, 1.3 M and 913 K particles; with plain terms 11,
// 103 and 125.
constexpr int kVolumeLanes = 8;

__global__ void __launch_bounds__(kThreads) k_boundary_volume(const __grid_constant__ DevParams P,
                                                              const __grid_constant__ DevBuffers B,
                                                              const float4* __restrict__ pos4) {
    const int t = blockIdx.x * kThreads + threadIdx.x;
    const int s = t / kVolumeLanes;
    const uint32_t g = (uint32_t)(t % kVolumeLanes);
    float4 pi = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t cell = kUndef;
    if (s < active_n(B)) {
        pi = pos4[s];
        if (pi.w < 0.f) cell = B.mgcell[s];
    }
    Kahan sum;
    float low = 0.f;  // the terms' rounding errors
    if (cell != kUndef)
        for_candidate_rows(P, B, cell, pi.x, pi.y, pi.z, [&](uint32_t j0, uint32_t j1) {
#pragma unroll 2
            for (uint32_t j = j0 + g; j < j1; j += kVolumeLanes) {
                const float4 pj = __ldg(&pos4[j]);
                const float x = (pi.x - pj.x) * P.vol_scale, y = (pi.y - pj.y) * P.vol_scale,
                            z = (pi.z - pj.z) * P.vol_scale;
                const float xx = __fmul_rn(x, x), yy = __fmul_rn(y, y), zz = __fmul_rn(z, z);
                if (pj.w < 0.f && xx + yy + zz < P.vol_r2[0]) {
                    // c = r2 - xx - yy - zz, each difference of two of which the first is the larger
                    const float c0 = __fsub_rn(P.vol_r2[0], xx), c1 = __fsub_rn(c0, yy), c = __fsub_rn(c1, zz);
                    float e = __fsub_rn(__fsub_rn(P.vol_r2[0], c0), xx);
                    e = __fadd_rn(e, __fsub_rn(__fsub_rn(c0, c1), yy));
                    e = __fadd_rn(e, __fsub_rn(__fsub_rn(c1, c), zz));
                    e = __fadd_rn(e, P.vol_r2[1]);
                    e = __fsub_rn(e, __fmaf_rn(x, x, -xx));
                    e = __fsub_rn(e, __fmaf_rn(y, y, -yy));
                    e = __fsub_rn(e, __fmaf_rn(z, z, -zz));
                    // (c + e)^3 = q c + what the two products and e leave
                    const float q = __fmul_rn(c, c), w = __fmul_rn(q, c);
                    low += __fmaf_rn(3.f * e, q, __fmaf_rn(__fmaf_rn(c, c, -q), c, __fmaf_rn(q, c, -w)));
                    sum.add(w);
                }
            }
        });
    __syncwarp();
#pragma unroll
    for (int o = kVolumeLanes / 2; o > 0; o >>= 1) {  // the pairwise sums, their rounding errors in low
        low = __fadd_rn(low, __shfl_xor_sync(0xffffffffu, low, o));
        sum.c = __fadd_rn(sum.c, __shfl_xor_sync(0xffffffffu, sum.c, o));
        add_exact(sum.s, low, __shfl_xor_sync(0xffffffffu, sum.s, o));
    }
    if (cell == kUndef || g != 0) return;
    // the volume 1 / (sum factor), the sum and the factor in two floats each
    const float v = sum.s * P.vol_factor[0];
    const float v0 = fmaf(low - sum.c, P.vol_factor[0], fmaf(sum.s, P.vol_factor[1], fmaf(sum.s, P.vol_factor[0], -v)));
    const float q = v == 0.f ? 1.f : 1.f / v;
    const float rest = fmaf(-q, v0, fmaf(-q, v, 1.f));  // 1 - q (v + v0)
    B.vtmp[s] = fabsf(rest) < 1e-6f ? fmaf(q, rest, q) : q;  // (else nothing was summed, or v is no ordinary float)
}

__global__ void __launch_bounds__(kThreads) k_boundary_volume_store(const __grid_constant__ DevParams P,
                                                                    const __grid_constant__ DevBuffers B,
                                                                    float4* __restrict__ pos4) {
    const int s = blockIdx.x * kThreads + threadIdx.x;
    if (s >= active_n(B) || B.mgcell[s] == kUndef) return;
    float4 p = pos4[s];
    if (!(p.w < 0.f)) return;
    p.w = -B.vtmp[s];
    pos4[s] = p;
    B.densp[s] = make_float2(-p.w, 0.f);
}

// ---------------------------------------------------------------------------
// Density + EOS pressure (MfComputePressureCUDA)
// ---------------------------------------------------------------------------

// Density + EOS and the neighbour lists, one warp per octant bucket (the members of
// one h-subcell). Every member of a bucket has its neighbours within the 27
// h-subcells around it: a pair closer than h is at most one subcell apart per
// axis, up to the rounding of the grid coordinate (a pair that rounding puts two
// subcells apart is within 1e-4 h of the cutoff, where the kernels and their
// gradients vanish to below 1e-7 of a typical term). The 27 subcells form 18
// contiguous index ranges (per (y, z) row: the x-neighbour bucket in the adjacent
// cell and the two buckets of the same cell); their concatenation is the bucket's
// candidate sequence. A warp takes one window of up to P.bwin (16, at most 32) members of a
// bucket and stages the bucket's candidates in shared memory, 256 at a time. The
// window's n fluid members share the lanes out: 32 / n lanes a member, each
// testing its share of the sequence two candidates at a time in packed FP32
// arithmetic, adding its density terms and appending the hits to a
// list of its own in shared memory. The lanes' lists of a member are then joined
// and written as rows of four indices. Bound by shared-memory accesses (78 % of
// the L1 data pipe) and the issue slots (63 %): about 14 instructions a candidate
// and lane, none of them across lanes. (The kernel this replaces had the lanes
// hold the candidates and walked the members, with ballots and selects per 32
// candidates and a shuffle reduction per member, and left mask words that a
// second kernel expanded: 174 M warp instructions at 442 K fluid particles
// against 126 M here; 404 against 373 us at 1.05 M, 33 against 13 us at 4 K. Shares
// that interleave take 12 us less, but put the lists out of sequence order, which
// cost the force and alpha passes 27 us of cache misses.) A lane adds at most 16
// pairs of terms before they go to its Kahan-compensated sum, and the lanes of a
// member are added pairwise (a scan) with their rounding errors. The difference
// h^2 - r^2 is formed with a squared radius that is exact as a float (dens_r2: both
// times a factor just above 1); h^2 itself rounds by up to 6e-8, for all terms
// alike (densities 8e-8 too large at h = 0.01 and 0.02, -5e-9 so). Warps take work
// items from a shared counter (their costs differ by orders of magnitude), each its first one without it (12.5
// instead of 14.3 us at 11 K particles): the first window of every bucket, then the
// further windows of large buckets, which the cell sort queued in wq, so that no
// bucket serialises on one warp. Members whose lists overflow their kMaxNbr
// entries get mask lists instead (overflow_masks) or, where the sequence is too
// long for those, are left to the cell search; they and members with more than
// P.heavy neighbours are queued in hq for the force and alpha passes.
// The candidate sequence of bucket (c, q): the 27 h-subcells around it as 18
// contiguous index ranges, two per (y, z) subcell row r = 0 .. 8 (the x-neighbour
// bucket in the adjacent cell, and both x buckets of the bucket's own cell
// column). Lane 2 r + part < 18 computes one range; the warp scans the lengths.
// rows[r] = {sequence offset of row r, offset of its second range, index minus
// offset in the first range, in the second}; rows[9].x = the sequence length T,
// returned. Cells are found relative to c (a neighbour subcell lies 0 or 1 cells
// away per axis), so nothing is divided.
__device__ __forceinline__ uint32_t bucket_rows(const DevParams& P, const DevBuffers& B, uint32_t c, uint32_t q,
                                                unsigned lane, uint4* rows) {
    const int ox = (int)(q & 1u), oz = (int)((q >> 1) & 1u), oy = (int)(q >> 2);
    uint32_t len = 0, st = 0;
    if (lane < 18) {
        const int r = (int)(lane >> 1), part = (int)(lane & 1u);
        const int sy = oy + r / 3 - 1, sz = oz + r % 3 - 1;  // subcell row relative to the cell's first
        const int oyz = ((sy & 1) * 2 + (sz & 1)) * 2;
        // the single x-neighbour bucket in the adjacent cell, or both of the bucket's own cell column
        const bool single = (ox == 0) == (part == 0);
        const int dx = single ? (ox == 0 ? -1 : 1) : 0;
        const int xlo = single && ox == 0 ? 1 : 0, xhi = single ? xlo : 1;
        const uint32_t cc = c + (uint32_t)(((sy >> 1) * P.rz + (sz >> 1)) * P.rx + dx);
        const uint32_t cs = __ldg(&B.cstart[cc]), ce = __ldg(&B.cend[cc]);
        if (cs < ce) {
            st = __ldg(&B.oct_start[(size_t)cc * 8 + oyz + xlo]);
            const uint32_t en = (oyz + xhi == 7) ? ce : __ldg(&B.oct_start[(size_t)cc * 8 + oyz + xhi + 1]);
            len = en - st;
        }
    }
    uint32_t inc = len;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, inc, d);
        if ((int)lane >= d) inc += v;
    }
    const uint32_t off = inc - len;
    if (lane <= 18) {
        uint32_t* d = &rows[lane >> 1].x + (lane & 1u);
        d[0] = off;
        d[2] = st - off;
    }
    __syncwarp();
    return __shfl_sync(0xffffffffu, inc, 31);
}


__device__ __forceinline__ uint32_t next_bucket(uint32_t* ctr, unsigned lane) {
    uint32_t v = 0;
    if (lane == 0) v = atomicAdd(ctr, 1u);
    return __shfl_sync(0xffffffffu, v, 0);
}

// The mask lists of the members `over` (a bit mask over the lanes, which hold the
// members' positions in pm) of window [w0, ...) of bucket bid: bit e of a
// member's mask stands for candidate e of the bucket's sequence (length T <= 32 *
// kMaskWords), whose index is e plus the offset of the sequence range holding e
// (btab). With the packed arithmetic of the density pass, so the same tests.
template <bool SS1>
__device__ __noinline__ void overflow_masks(const DevParams& P, const DevBuffers& B, const float4* __restrict__ pos4,
                                            uint32_t over, const float4 pm, uint32_t w0, uint32_t bid, uint32_t T,
                                            const uint4* rows) {
    const unsigned lane = lane_id();
    uint32_t* __restrict__ bt = B.btab + (size_t)bid * kTabStride;
    if (lane < 18) {
        const uint32_t* d = &rows[lane >> 1].x + (lane & 1u);
        bt[lane] = d[0];
        bt[20 + lane] = d[2];
    }
    if (lane == 18) bt[18] = T;
    int r = 0;  // the row holding e, which only grows
    for (uint32_t base = 0; base < T; base += 32u) {
        const uint32_t e = base + lane;
        float4 c = make_float4(__int_as_float(0x7f800000), 0.f, 0.f, 0.f);
        if (e < T) {
            while (rows[r + 1].x <= e) r++;
            const uint4 row = rows[r];
            c = __ldg(&pos4[e + (e < row.y ? row.z : row.w)]);
        }
        for (uint32_t om = over; om != 0u; om &= om - 1u) {
            const int i = __ffs(om) - 1;
            float dx = __fadd_rn(__shfl_sync(0xffffffffu, pm.x, i), -c.x);
            float dy = __fadd_rn(__shfl_sync(0xffffffffu, pm.y, i), -c.y);
            float dz = __fadd_rn(__shfl_sync(0xffffffffu, pm.z, i), -c.z);
            if (!SS1) {
                dx = __fmul_rn(dx, P.ss);
                dy = __fmul_rn(dy, P.ss);
                dz = __fmul_rn(dz, P.ss);
            }
            const float dsq = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
            const uint32_t t = w0 + (uint32_t)i;
            const uint32_t b = __ballot_sync(0xffffffffu, dsq < P.r2list && dsq > 0.f);
            if (lane == 0) B.nmask[(size_t)(base >> 5) * (size_t)P.cap + t] = b;
        }
    }
}

constexpr int kDensThreads = 128;
constexpr int kDensBlock = 256;  // candidates staged at a time
constexpr int kDensList = 64;    // hits a lane keeps per block of candidates
constexpr int kDensRow = kDensList + 4;  // bytes of its row (17 words: the lanes' rows start in different banks)

struct DensityWarp {  // one warp's shared memory
    float4 pxy[kDensBlock / 2];     // two candidates: {x0, x1, y0, y1}
    float4 pzw[kDensBlock / 2];     // {z0, z1, w0, w1}
    uint32_t cidx[kDensBlock];      // their indices
    uint8_t list[32 * kDensRow];    // the lanes' hits as positions in the block
    uint4 rows[10];                 // the candidate sequence (bucket_rows)
};

template <bool SS1>
__global__ void __launch_bounds__(kDensThreads, 7) k_density_bucket(const __grid_constant__ DevParams P,
                                                                    const __grid_constant__ DevBuffers B,
                                                                    const float4* __restrict__ pos4,
                                                                    const float4* __restrict__ alpha4) {
    __shared__ DensityWarp shared[kDensThreads / 32];
    const unsigned lane = lane_id();
    DensityWarp& W = shared[threadIdx.x >> 5];
    uint8_t* const row = W.list + lane * kDensRow;
    const uint32_t nb = *B.act_n * 8u;
    const uint32_t nitems = nb + *B.wq_n;  // the first window of every bucket, then the queued windows
    const size_t cap = (size_t)P.cap;
    const float r2list = P.r2list;
    const float kFar = __int_as_float(0x7f800000);  // +inf: never within range
    const uint32_t nwarps = gridDim.x * (kDensThreads / 32);
    for (uint32_t it = (blockIdx.x * kDensThreads + threadIdx.x) >> 5; it < nitems;
         it = nitems > nwarps ? nwarps + next_bucket(B.dctr, lane) : nitems) {
        uint32_t c, q, w0;
        if (it < nb) {
            c = __ldg(&B.act[it >> 3]);
            q = it & 7u;
            w0 = __ldg(&B.oct_start[(size_t)c * 8 + q]);
        } else {
            const uint2 e = B.wq[it - nb];
            c = e.x >> 3;
            q = e.x & 7u;
            w0 = e.y;
        }
        const uint32_t bid = c * 8u + q;
        const uint32_t m1 = q == 7 ? __ldg(&B.cend[c]) : __ldg(&B.oct_start[(size_t)bid + 1]);
        if (w0 >= m1) continue;
        const uint32_t w1 = min(m1, w0 + (uint32_t)P.bwin);
        // the window's members, one per lane; boundary members carry their volume and need no list
        float4 pm = make_float4(0.f, 0.f, 0.f, -1.f);
        float rho0 = 0.f;
        if (w0 + lane < w1) {
            pm = __ldg(&pos4[w0 + lane]);
            if (pm.w < 0.f) {
                B.densp[w0 + lane] = make_float2(-pm.w, 0.f);
                B.nbr_cnt[w0 + lane] = 0;
            } else {
                rho0 = __ldg(&alpha4[w0 + lane]).w;
            }
        }
        const uint32_t fluid = __ballot_sync(0xffffffffu, w0 + lane < w1 && pm.w >= 0.f);
        if (!fluid) continue;
        // L lanes a fluid member: lane l takes share l % L of member `src` (lane L ord + share)
        // (the quotients in float: half a unit away from the next whole number)
        const uint32_t nf = (uint32_t)__popc(fluid);
        const uint32_t L = (uint32_t)__fdividef(32.5f, (float)nf);
        const uint32_t ord = (uint32_t)__fdividef((float)lane + 0.5f, (float)L), share = lane - ord * L;
        uint32_t src = ord;
        if (fluid != (nf == 32u ? 0xffffffffu : (1u << nf) - 1u)) {  // boundary members among them
            if (fluid >> lane & 1u) W.list[__popc(fluid & lanemask_lt())] = (uint8_t)lane;
            __syncwarp();
            src = ord < nf ? W.list[ord] : 0u;
            __syncwarp();
        }
        const bool live = ord < nf;
        const uint32_t t = w0 + src;
        const float px = __shfl_sync(0xffffffffu, pm.x, (int)src), py = __shfl_sync(0xffffffffu, pm.y, (int)src),
                    pz = __shfl_sync(0xffffffffu, pm.z, (int)src);
        rho0 = __shfl_sync(0xffffffffu, rho0, (int)src);
        const float2 PX = make_float2(px, px), PY = make_float2(py, py), PZ = make_float2(pz, pz);
        const float2 SS = make_float2(P.ss, P.ss), R2 = make_float2(P.dens_r2, P.dens_r2), NEGA = make_float2(-P.dens_a, -P.dens_a), NEG1 = make_float2(-1.f, -1.f);
        const uint32_t T = bucket_rows(P, B, c, q, lane, W.rows);
        Kahan sum;
        uint32_t count = 0;  // the member's neighbours in the blocks so far
        for (uint32_t base = 0; base < T; base += kDensBlock) {
            const uint32_t n = min(T - base, (uint32_t)kDensBlock);
            // stage the candidates, a row of two ranges at a time
            float wmin = 0.f;
            uint4 rw = W.rows[0];
#pragma unroll 3
            for (int r = 0; r < 9; r++) {
                const uint4 next = W.rows[r + 1];
                uint32_t e = rw.x + lane, end = next.x;
                if (T > (uint32_t)kDensBlock) {  // the part of the row in this block
                    e = max(rw.x, base) + lane;
                    end = min(end, base + (uint32_t)kDensBlock);
                }
                for (; e < end; e += 32u) {
                    const uint32_t j = e + (e < rw.y ? rw.z : rw.w);
                    const float4 p = __ldg(&pos4[j]);
                    wmin = fminf(wmin, p.w);
                    const uint32_t l = e - base;
                    float* a = &W.pxy[l >> 1].x + (l & 1u);
                    float* b = &W.pzw[l >> 1].x + (l & 1u);
                    a[0] = p.x;
                    a[2] = p.y;
                    b[0] = p.z;
                    b[2] = p.w;
                    W.cidx[l] = j;
                }
                rw = next;
            }
            if (lane == 0 && (n & 1u)) {  // the odd last one's partner: out of range, no weight
                float4& a = W.pxy[n >> 1];
                float4& b = W.pzw[n >> 1];
                a.y = a.w = b.y = kFar;
                b.w = 0.f;
            }
            const bool any_bnd = __any_sync(0xffffffffu, wmin < 0.f);
            __syncwarp();
            // this lane's pairs, an odd number (lanes in step then read different banks)
            const uint32_t npairs = (n + 1u) >> 1;
            const uint32_t each = (uint32_t)__fdividef((float)(npairs + L) - 0.5f, (float)L) | 1u;
            const uint32_t p0 = min(npairs, share * each), p1 = min(npairs, p0 + each);
            auto dist2 = [&](const float4 a, const float4 b) {
                float2 dx = __ffma2_rn(make_float2(a.x, a.y), NEG1, PX), dy = __ffma2_rn(make_float2(a.z, a.w), NEG1, PY),
                       dz = __ffma2_rn(make_float2(b.x, b.y), NEG1, PZ);
                if (!SS1) {
                    dx = __fmul2_rn(dx, SS);
                    dy = __fmul2_rn(dy, SS);
                    dz = __fmul2_rn(dz, SS);
                }
                return __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
            };
            // a neighbour: within the list radius and not at the same place (every consumer of
            // the lists skips r = 0), so not the member itself
            auto near = [&](float d2) { return d2 < r2list && d2 > 0.f; };
            // the walk over them. With boundary candidates in the block or without (the usual
            // case): the weight of a candidate is its mass, or rho0 V for a boundary particle.
            uint32_t hits = 0;
            auto walk = [&](auto with_boundary, auto bounded) {
                constexpr bool BND = decltype(with_boundary)::value;
                uint32_t p = p0;
                while (p < p1) {
                    float2 acc = make_float2(0.f, 0.f);
                    const uint32_t end = min(p1, p + 16u);
#pragma unroll 2
                    for (; p < end; p++) {
                        const float4 a = W.pxy[p], b = W.pzw[p];
                        const float2 d2 = dist2(a, b);
                        float2 cc = __ffma2_rn(d2, NEGA, R2);  // a (r2 - d2), rounded once
                        cc.x = fmaxf(cc.x, 0.f);               // 0 outside h (and for the padding)
                        cc.y = fmaxf(cc.y, 0.f);
                        const float2 c3 = __fmul2_rn(__fmul2_rn(cc, cc), cc);
                        float2 wt = make_float2(b.z, b.w);
                        if (BND) {
                            wt.x = wt.x < 0.f ? rho0 * -wt.x : wt.x;
                            wt.y = wt.y < 0.f ? rho0 * -wt.y : wt.y;
                        }
                        acc = __ffma2_rn(c3, wt, acc);
                        // every candidate is stored after the hits so far and stays if it is one
                        // (no branch; a full row keeps its last byte for this)
                        row[decltype(bounded)::value ? min(hits, (uint32_t)kDensList) : hits] = (uint8_t)(2u * p);
                        hits += near(d2.x) ? 1u : 0u;
                        row[decltype(bounded)::value ? min(hits, (uint32_t)kDensList) : hits] = (uint8_t)(2u * p + 1u);
                        hits += near(d2.y) ? 1u : 0u;
                    }
                    sum.add(acc.x + acc.y);
                }
            };
            if (live) {
                // four lanes or more a member: at most 33 pairs each, the row holds them all
                if (L >= 4u) {
                    if (any_bnd) walk(std::true_type{}, std::false_type{});
                    else walk(std::false_type{}, std::false_type{});
                } else {
                    if (any_bnd) walk(std::true_type{}, std::true_type{});
                    else walk(std::false_type{}, std::true_type{});
                }
            }
            __syncwarp();
            // the member's hits before this lane's, and all of them
            uint32_t before = hits;
            for (uint32_t o = 1; o < L; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, before, o);
                if (share >= o) before += v;
            }
            const int last = (int)min(lane - share + L - 1u, 31u);
            const uint32_t total = __shfl_sync(0xffffffffu, before, last);
            before -= hits;
            if (!__any_sync(0xffffffffu, total > (uint32_t)kDensList)) {
                // join the lanes' rows in the member's first one, then write rows of four
                uint8_t* const joined = W.list + (lane - share) * kDensRow;
                if (share != 0u)
                    for (uint32_t i = 0; i < hits; i++) joined[before + i] = row[i];
                __syncwarp();
                if ((count & 3u) == 0u && count + total <= (uint32_t)kMaxNbr) {
                    uint4* const out = reinterpret_cast<uint4*>(B.nbr) + t;
                    for (uint32_t k = share; 4u * k < total; k += L) {
                        const uchar4 e = *reinterpret_cast<const uchar4*>(joined + 4u * k);  // past the end: any bytes
                        out[((size_t)(count >> 2) + k) * cap] = make_uint4(W.cidx[e.x], W.cidx[e.y], W.cidx[e.z], W.cidx[e.w]);
                    }
                } else {
                    for (uint32_t k = share; k < total; k += L)
                        if (count + k < (uint32_t)kMaxNbr) B.nbr[nbr_at(cap, t, count + k)] = W.cidx[joined[k]];
                }
            } else if (live) {  // too many for the rows: found again, stored one by one
                uint32_t k = count + before;
                for (uint32_t p = p0; p < p1; p++) {
                    const float2 d2 = dist2(W.pxy[p], W.pzw[p]);
                    if (near(d2.x)) {
                        if (k < (uint32_t)kMaxNbr) B.nbr[nbr_at(cap, t, k)] = W.cidx[2u * p];
                        k++;
                    }
                    if (near(d2.y)) {
                        if (k < (uint32_t)kMaxNbr) B.nbr[nbr_at(cap, t, k)] = W.cidx[2u * p + 1u];
                        k++;
                    }
                }
            }
            count += total;
            __syncwarp();  // before the candidates and rows are rewritten
        }
        float dens = sum.s, low = -sum.c;  // of this lane and the member's lanes before it
        for (uint32_t o = 1; o < L; o <<= 1) {
            const float v = __shfl_up_sync(0xffffffffu, dens, o), v0 = __shfl_up_sync(0xffffffffu, low, o);
            if (share >= o) {
                low += v0;
                add_exact(dens, low, v);
            }
        }
        dens += low;
        const bool own = live && share == L - 1u;  // holds the whole sum
        // lists that overflowed: mask lists, or the cell search where the sequence is too long for them
        const bool over = own && count > (uint32_t)kMaxNbr;
        const bool masked = T <= 32u * kMaskWords;
        if (__any_sync(0xffffffffu, over) && masked)
            overflow_masks<SS1>(P, B, pos4, __reduce_or_sync(0xffffffffu, over ? 1u << src : 0u), pm, w0, bid, T,
                                W.rows);
        const bool heavy = own && count > P.heavy;  // P.heavy <= kMaxNbr
        if (own) {
            B.nbr_cnt[t] = over ? (masked ? kMaskList | bid : kRescan) : heavy ? count | kHeavyFlag : count;
            B.densp[t] = density_result(P, dens, rho0);
        }
        const uint32_t hb = __ballot_sync(0xffffffffu, heavy);
        if (hb) {  // queued for the force and alpha passes
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(B.hq_n, (uint32_t)__popc(hb));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (heavy) B.hq[at + __popc(hb & lanemask_lt())] = t;
        }
    }
}

__global__ void __launch_bounds__(kThreads) k_density(const __grid_constant__ DevParams P,
                                                      const __grid_constant__ DevBuffers B,
                                                      const float4* __restrict__ pos4,
                                                      const float4* __restrict__ alpha4) {
    const int s = blockIdx.x * kThreads + threadIdx.x;
    if (s >= active_n(B) || B.mgcell[s] == kUndef) return;
    const float4 pi = pos4[s];
    if (pi.w < 0.f) {  // boundary: carries its volume, no pressure, needs no list
        B.densp[s] = make_float2(-pi.w, 0.f);
        B.nbr_cnt[s] = 0;
        return;
    }
    const float rho0 = alpha4[s].w;
    Kahan sum;
    uint32_t cnt = 0;
    for_candidates(P, B, B.mgcell[s], pi.x, pi.y, pi.z, [&](uint32_t j) {
        const float4 pj = __ldg(&pos4[j]);
        const float dx = (pi.x - pj.x) * P.ss, dy = (pi.y - pj.y) * P.ss, dz = (pi.z - pj.z) * P.ss;
        const float dsq = dx * dx + dy * dy + dz * dz;
        if (dsq < P.r2) {
            const float c = fmaxf(fmaf(-P.dens_a, dsq, P.dens_r2), 0.f);
            const float m = pj.w > 0.f ? pj.w : rho0 * (-pj.w);
            sum.add(c * c * c * m);
        }
        if (dsq > 0.f && dsq < P.r2list) {
            if (cnt < (uint32_t)kMaxNbr) B.nbr[nbr_at((size_t)P.cap, (uint32_t)s, cnt)] = j;
            cnt++;
        }
    });
    B.nbr_cnt[s] = cnt;
    B.densp[s] = density_result(P, sum.s, rho0);
}

// ---------------------------------------------------------------------------
// Force + drift velocity (MfComputeForceCUDA, MfComputeDriftVelCUDA)
// ---------------------------------------------------------------------------

// Force + drift of one in-grid fluid particle, neighbours gathered from global
// memory through its list (or the cell search).
template <bool FORCE, bool DRIFT, int NP>
__device__ __forceinline__ void force_drift_one(const DevParams& P, const DevBuffers& B,
                                                const float4* __restrict__ pos4, const float4* __restrict__ vel4,
                                                const float4* __restrict__ alpha4, const float4* __restrict__ aprev4,
                                                const float4* __restrict__ vev4, int s, const float4 pi) {
    ForceDrift<FORCE, DRIFT, NP> acc;
    acc.init(P, pi, vel4[s], B.densp[s], alpha4[s]);
    for_slot_list<false>(P, B, s, pi.x, pi.y, pi.z, [&](uint32_t j) {
        // every load first (list entries are almost always neighbours), so that
        // consecutive neighbours' gathers overlap
        const float4 pj = __ldg(&pos4[j]);
        const float2 dpj = __ldg(&B.densp[j]);
        const float4 vj = FORCE ? __ldg(&vel4[j]) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 aj = DRIFT ? __ldg(&alpha4[j]) : make_float4(0.f, 0.f, 0.f, 0.f);
        acc.pair(P, pj, dpj, vj, aj);
    });
    acc.finish(P, B, s, DRIFT ? aprev4[s] : make_float4(0.f, 0.f, 0.f, 0.f),
               DRIFT ? vev4[s] : make_float4(0.f, 0.f, 0.f, 0.f));
}

// Force + drift of heavy particle s by the whole warp (every lane calls with
// the same s): the lanes share its neighbours out, their partial sums are
// added, lane 0 stores.
template <bool FORCE, bool DRIFT, int NP>
__device__ __forceinline__ void force_drift_warp(const DevParams& P, const DevBuffers& B,
                                                 const float4* __restrict__ pos4, const float4* __restrict__ vel4,
                                                 const float4* __restrict__ alpha4, const float4* __restrict__ aprev4,
                                                 const float4* __restrict__ vev4, int s) {
    const float4 pi = pos4[s];
    ForceDrift<FORCE, DRIFT, NP> acc;
    acc.init(P, pi, vel4[s], B.densp[s], alpha4[s]);
    warp_for_slot_list(P, B, s, pi.x, pi.y, pi.z, [&](uint32_t j) {
        const float4 pj = __ldg(&pos4[j]);
        const float2 dpj = __ldg(&B.densp[j]);
        const float4 vj = FORCE ? __ldg(&vel4[j]) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 aj = DRIFT ? __ldg(&alpha4[j]) : make_float4(0.f, 0.f, 0.f, 0.f);
        acc.pair(P, pj, dpj, vj, aj);
    });
    acc.template reduce<32>();
    if (lane_id() == 0)
        acc.finish(P, B, s, DRIFT ? aprev4[s] : make_float4(0.f, 0.f, 0.f, 0.f),
                   DRIFT ? vev4[s] : make_float4(0.f, 0.f, 0.f, 0.f));
}

// The work counter (hctr) of each pass over the queue of heavy particles.
template <bool FORCE, bool DRIFT>
constexpr int kHeavyCounter = FORCE && !DRIFT ? 1 : 0;
constexpr int kHeavyCounterAlpha = 2;

// Force + drift, L lanes per particle (walk_lanes); every warp first takes heavy
// particles from the queue (whole warp per particle) while any are left. With the
// drift it also writes every in-grid particle's neighbour record for the alpha and
// project-U passes of the step.
template <bool FORCE, bool DRIFT, int NP, int L>
__global__ void __launch_bounds__(kThreads, 4) k_force_drift(const __grid_constant__ DevParams P,
                                                             const __grid_constant__ DevBuffers B,
                                                             const float4* __restrict__ pos4,
                                                             const float4* __restrict__ vel4,
                                                             const float4* __restrict__ alpha4,
                                                             const float4* __restrict__ aprev4,
                                                             const float4* __restrict__ vev4) {
    if (P.list_mode != 0) {
        const unsigned lane = lane_id();
        const uint32_t nh = *B.hq_n;
        uint32_t* ctr = &B.hctr[kHeavyCounter<FORCE, DRIFT>];
        for (uint32_t h = next_item(ctr, nh, lane); h < nh; h = next_item(ctr, nh, lane))
            force_drift_warp<FORCE, DRIFT, NP>(P, B, pos4, vel4, alpha4, aprev4, vev4, (int)B.hq[h]);
    }
    const int s = (int)((blockIdx.x * (unsigned)kThreads + threadIdx.x) / L);
    const unsigned g = threadIdx.x % L;
    const bool in = s < active_n(B) && B.mgcell[s] != kUndef;
    if (L == 1 && !in) return;
    const float4 pi = in ? pos4[s] : make_float4(0.f, 0.f, 0.f, -1.f);
    if (in && g == 0 && pi.w < 0.f) {
        if (FORCE) B.accel4[s] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (DRIFT) {
            const float a0[3] = {0.f, 0.f, 0.f};
            const float u0[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            write_nrec(B, s, pi, -1.f, vev4[s], a0, u0);
        }
    }
    const bool walk = !(pi.w < 0.f) && !is_heavy(P, B.nbr_cnt[s]);  // heavy: taken from the queue
    if (L == 1) {
        if (walk) force_drift_one<FORCE, DRIFT, NP>(P, B, pos4, vel4, alpha4, aprev4, vev4, s, pi);
        return;
    }
    if (!__any_sync(0xffffffffu, walk)) return;
    ForceDrift<FORCE, DRIFT, NP> acc;
    const int si = walk ? s : 0;
    acc.init(P, pi, vel4[si], B.densp[si], alpha4[si]);
    if (walk)
        group_for_slot_list<L>(P, B, s, g, pi.x, pi.y, pi.z, [&](uint32_t j) {
            const float4 pj = __ldg(&pos4[j]);
            const float2 dpj = __ldg(&B.densp[j]);
            const float4 vj = FORCE ? __ldg(&vel4[j]) : make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 aj = DRIFT ? __ldg(&alpha4[j]) : make_float4(0.f, 0.f, 0.f, 0.f);
            acc.pair(P, pj, dpj, vj, aj);
        });
    __syncwarp();
    acc.template reduce<L>();
    if (walk && g == 0)
        acc.finish(P, B, s, DRIFT ? aprev4[s] : make_float4(0.f, 0.f, 0.f, 0.f),
                   DRIFT ? vev4[s] : make_float4(0.f, 0.f, 0.f, 0.f));
}

// Force + drift of a corrected large step: the same pass, also filling the
// corrector's features from the neighbours it gathers (alpha4 is gathered
// even without drift). Features and ids cover every particle. Bound by the latency of
// its gathers with 16 warps an SM: 52 sums and the neighbours in flight take 126
// registers (96 spill: 320 us). What the walk does not need stays out of them:
// the own features are stored before it, the sums scaled after it. 895 K slots, two
// phases: 264 us (306 with the own features and scales held and applied to every pair).
constexpr int kFeatThreads = 128;
template <bool DRIFT, int NP>
__global__ void __launch_bounds__(kFeatThreads, 4) k_force_drift_feat(const __grid_constant__ DevParams P,
                                                                  const __grid_constant__ DevBuffers B,
                                                                  const float4* __restrict__ pos4,
                                                                  const float4* __restrict__ vel4,
                                                                  const float4* __restrict__ alpha4,
                                                                  const float4* __restrict__ aprev4,
                                                                  const float4* __restrict__ vev4, float* feat,
                                                                  int32_t* ids, float vs, float dt_large) {
    const int s = blockIdx.x * kFeatThreads + threadIdx.x;
    if (s >= active_n(B)) return;
    float* row = feat + (size_t)s * kLearnedFeatures;
    if (B.mgcell[s] == kUndef) {
        store_no_features(row, &ids[s]);
        return;
    }
    const float4 pi = pos4[s];
    if (pi.w < 0.f) {
        B.accel4[s] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (DRIFT) {
            const float a0[3] = {0.f, 0.f, 0.f};
            const float u0[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            write_nrec(B, s, pi, -1.f, vev4[s], a0, u0);
        }
        store_no_features(row, &ids[s]);
        return;
    }
    const float4 vi = vel4[s], ai = alpha4[s];
    const float2 di = B.densp[s];
    ForceDrift<true, DRIFT, NP> acc;
    acc.init(P, pi, vi, di, ai);
    LearnedFeatures lf;
    lf.init(P, pi, vi, ai, di, vs, row);
    for_slot_list(P, B, s, pi.x, pi.y, pi.z, [&](uint32_t j) {
        const float4 pj = __ldg(&pos4[j]);
        const float2 dpj = __ldg(&B.densp[j]);
        const float4 vj = __ldg(&vel4[j]);
        const float4 aj = __ldg(&alpha4[j]);
        acc.pair(P, pj, dpj, vj, aj);
        lf.pair(P, pj, dpj, vj, aj);
    });
    const float4 gi = aprev4[s];
    lf.store(P, gi, vs, dt_large, row);
    acc.finish(P, B, s, DRIFT ? gi : make_float4(0.f, 0.f, 0.f, 0.f), DRIFT ? vev4[s] : make_float4(0.f, 0.f, 0.f, 0.f));
    ids[s] = B.bornid[__float_as_uint(gi.w)];
}

// Surface tension (reference SurfaceTension, fluid_system_kern.cu:569-625): all
// 27 cells, squared distance compared with the radius K*h, added to accel.
__global__ void __launch_bounds__(kThreads) k_surface_tension(const __grid_constant__ DevParams P,
                                                              const __grid_constant__ DevBuffers B,
                                                              const float4* __restrict__ pos4) {
    const int s = blockIdx.x * kThreads + threadIdx.x;
    if (s >= active_n(B)) return;
    const uint32_t gc = B.mgcell[s];
    if (gc == kUndef) return;
    const float4 pi = pos4[s];
    const float tR = sqrtf(P.st_K * P.st_K * (P.h * P.h));
    float rx = 0.f, ry = 0.f, rz = 0.f;
    for (int c = 0; c < 27; c++) {
        const uint32_t cell = gc + (uint32_t)P.neighborid[c];
        const uint32_t j0 = B.cstart[cell], j1 = B.cend[cell];
        for (uint32_t j = j0; j < j1; j++) {
            const float4 pj = __ldg(&pos4[j]);
            const float dx = (pi.x - pj.x) * P.ss, dy = (pi.y - pj.y) * P.ss, dz = (pi.z - pj.z) * P.ss;
            float dsq = dx * dx + dy * dy + dz * dz;
            if (dsq != 0.f && dsq <= tR) {
                dsq = sqrtf(dsq);
                const float fm = P.st_C * cosf(1.5f * 3.14159f * dsq / tR) / dsq;
                rx += dx * fm; ry += dy * fm; rz += dz * fm;
            }
        }
    }
    float4 a = B.accel4[s];
    a.x += rx; a.y += ry; a.z += rz;
    B.accel4[s] = a;
}

// Project-U force (ComputeForce_projectu, multiphase.cu:578-616), one thread
// per particle: writes accel (the reference's mforce) and the XSPH correction of
// every in-grid fluid particle. In-grid boundary particles get accel 0, as in the
// force pass; boundary and out-of-grid particles get a zero correction (the
// reference leaves both untouched for them).
template <int NP>
__global__ void __launch_bounds__(kThreads) k_force_projectu(const __grid_constant__ DevParams P,
                                                             const __grid_constant__ DevBuffers B,
                                                             const float4* __restrict__ pos4,
                                                             const float4* __restrict__ vel4,
                                                             const float4* __restrict__ vev4,
                                                             const float4* __restrict__ alpha_cur,
                                                             const float4* __restrict__ alpha_pre,
                                                             const float4* __restrict__ aprev4) {
    const int s = blockIdx.x * kThreads + threadIdx.x;
    if (s >= active_n(B)) return;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 pi = pos4[s];
    if (B.mgcell[s] == kUndef || pi.w < 0.f) {
        if (B.mgcell[s] != kUndef) B.accel4[s] = zero;
        B.velxcor[s] = zero;
        return;
    }
    float3 um[NP];
#pragma unroll
    for (int k = 0; k < NP; k++) {
        const float4 u = B.drift4[(size_t)k * P.cap + s];
        um[k] = make_float3(u.x, u.y, u.z);
    }
    ProjectU<NP> acc;
    acc.init(pi, vev4[s], B.densp[s], vel4[s].w, alpha_cur[s].w, alpha_pre[s], um);
    for_slot_list(P, B, s, pi.x, pi.y, pi.z, [&](uint32_t j) {
        const float4 pj = __ldg(&pos4[j]);
        const float2 dpj = __ldg(&B.densp[j]);
        const float4 vej = __ldg(&vev4[j]);
        const float viscj = __ldg(&vel4[j].w);
        const float4 aj = __ldg(&alpha_pre[j]);
        float4 uj[NP];
#pragma unroll
        for (int k = 0; k < NP; k++) uj[k] = __ldg(&B.drift4[(size_t)k * P.cap + j]);
        float mj = pj.w, rho0j = 1.f;
        if (pj.w < 0.f) {  // boundary: raw mass (per origin) and rest density
            mj = __ldg(&B.mass_raw[__float_as_uint(__ldg(&aprev4[j].w))]);
            rho0j = __ldg(&alpha_cur[j].w);
        }
        acc.pair(P, pj, dpj, vej, viscj, rho0j, mj, aj, uj);
    });
    B.accel4[s] = make_float4(acc.fx, acc.fy, acc.fz, 0.f);
    B.velxcor[s] = make_float4(acc.xx, acc.xy, acc.xz, 0.f);
}

// The same force in a step, the neighbours' positions, velocities, start-of-step
// fractions and drift velocities from the records that the drift pass of this step
// wrote; L lanes a particle (walk_lanes), the heavy ones from the queue. Bound by its
// loads as well (seven a neighbour, eight with the gathers): 14, 31, 82, 141 and 413 us
// at 12 K, 63 K, 244 K, 421 K and 1.3 M slots against 39, 45, 92, 145 and 438.
template <int NP, int L>
__global__ void __launch_bounds__(kThreads, 3) k_force_projectu_rec(const __grid_constant__ DevParams P,
                                                                    const __grid_constant__ DevBuffers B,
                                                                    const float4* __restrict__ pos4,
                                                                    const float4* __restrict__ vel4,
                                                                    const float4* __restrict__ vev4,
                                                                    const float4* __restrict__ alpha_cur,
                                                                    const float4* __restrict__ alpha_pre,
                                                                    const float4* __restrict__ aprev4) {
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    ProjectU<NP> acc;
    auto init = [&](int i, const float4 pi) {
        float3 um[NP];
#pragma unroll
        for (int k = 0; k < NP; k++) {
            const float4 u = B.drift4[(size_t)k * P.cap + i];
            um[k] = make_float3(u.x, u.y, u.z);
        }
        acc.init(pi, vev4[i], B.densp[i], vel4[i].w, alpha_cur[i].w, alpha_pre[i], um);
    };
    auto pair = [&](uint32_t j) {
        const float4* __restrict__ r = B.nrec + (size_t)j * kNrecFloat4;
        const float4 r0 = __ldg(r), r1 = __ldg(r + 1), r2 = __ldg(r + 2), r3 = __ldg(r + 3), r4 = __ldg(r + 4);
        const float2 dpj = __ldg(&B.densp[j]);
        const float viscj = __ldg(&vel4[j].w);
        float4 uj[NP];
        uj[0] = make_float4(r2.z, r2.w, r3.x, 0.f);
        if (NP > 1) uj[NP > 1 ? 1 : 0] = make_float4(r3.y, r3.z, r3.w, 0.f);
        if (NP > 2) uj[NP > 2 ? 2 : 0] = make_float4(r4.x, r4.y, r4.z, 0.f);
        float mj = r4.w, rho0j = 1.f;
        if (r4.w < 0.f) {  // boundary: raw mass (per origin) and rest density
            mj = __ldg(&B.mass_raw[__float_as_uint(__ldg(&aprev4[j].w))]);
            rho0j = __ldg(&alpha_cur[j].w);
        }
        acc.pair(P, make_float4(r0.x, r0.y, r0.z, r4.w), dpj, make_float4(r1.x, r1.y, r1.z, 0.f), viscj, rho0j, mj,
                 make_float4(r1.w, r2.x, r2.y, 0.f), uj);
    };
    auto store = [&](int i) {
        B.accel4[i] = make_float4(acc.fx, acc.fy, acc.fz, 0.f);
        B.velxcor[i] = make_float4(acc.xx, acc.xy, acc.xz, 0.f);
    };
    if (P.list_mode != 0) {
        const unsigned lane = lane_id();
        const uint32_t nh = *B.hq_n;
        uint32_t* ctr = &B.hctr[kHeavyCounter<true, false>];
        for (uint32_t h = next_item(ctr, nh, lane); h < nh; h = next_item(ctr, nh, lane)) {
            const int sh = (int)B.hq[h];
            const float4 pi = pos4[sh];
            init(sh, pi);
            warp_for_slot_list(P, B, sh, pi.x, pi.y, pi.z, pair);
            acc.template reduce<32>();
            if (lane == 0) store(sh);
        }
    }
    const int s = (int)((blockIdx.x * (unsigned)kThreads + threadIdx.x) / L);
    const unsigned g = threadIdx.x % L;
    const bool in = s < active_n(B);
    const int si = in ? s : 0;
    const float4 pi = pos4[si];
    const bool grid = B.mgcell[si] != kUndef, fluid = grid && !(pi.w < 0.f);
    if (in && g == 0 && !fluid) {
        if (grid) B.accel4[s] = zero;
        B.velxcor[s] = zero;
    }
    const bool walk = in && fluid && !is_heavy(P, B.nbr_cnt[si]);
    if (!__any_sync(0xffffffffu, walk)) return;
    init(si, pi);
    if (walk) {
        if (L == 1) for_slot_list(P, B, s, pi.x, pi.y, pi.z, pair);
        else group_for_slot_list<L>(P, B, s, g, pi.x, pi.y, pi.z, pair);
    }
    __syncwarp();
    if (L > 1) acc.template reduce<L>();
    if (walk && g == 0) store(s);
}

// ---------------------------------------------------------------------------
// Volume-fraction advance, correction, advection
// ---------------------------------------------------------------------------

// Alpha change of particle s with neighbours gathered from global memory (the
// separate alpha-advance pass of the reference call order).
template <int NP>
__device__ __forceinline__ void alpha_change_slot(const DevParams& P, const DevBuffers& B,
                                                  const float4* __restrict__ pos4, const float4* __restrict__ vev4,
                                                  const float4* __restrict__ alpha4, int s, const float4 pi,
                                                  const float4 vei, const float4 ai, float (&out)[3]) {
    AlphaChange<NP> acc;
    acc.init(pi, vei, ai, B.drift4 + s, (size_t)P.cap);
    for_slot_list(P, B, s, pi.x, pi.y, pi.z, [&](uint32_t j) {
        // every load first, so that consecutive neighbours' gathers overlap
        const float4 pj = __ldg(&pos4[j]);
        const float2 dpj = __ldg(&B.densp[j]);
        const float4 vej = __ldg(&vev4[j]);
        const float4 aj = __ldg(&alpha4[j]);
        float4 uj[NP];
#pragma unroll
        for (int k = 0; k < NP; k++) uj[k] = __ldg(&B.drift4[(size_t)k * P.cap + j]);
        acc.pair(P, pj, pj.w * dpj.x, vej, aj, uj);
    });
    acc.result(P, out);
}

// Separate alpha advance: new fractions into alpha4 out (restdens copied).
template <int NP>
__global__ void __launch_bounds__(kThreads) k_alpha_advance(const __grid_constant__ DevParams P,
                                                            const __grid_constant__ DevBuffers B,
                                                            const float4* __restrict__ pos4,
                                                            const float4* __restrict__ vev4,
                                                            const float4* __restrict__ alpha_in,
                                                            float4* __restrict__ alpha_out) {
    const int s = blockIdx.x * kThreads + threadIdx.x;
    if (s >= active_n(B)) return;
    const float4 ai = alpha_in[s];
    const float4 pi = pos4[s];
    if (B.mgcell[s] == kUndef || pi.w < 0.f) {
        alpha_out[s] = ai;
        return;
    }
    float na[3] = {ai.x, ai.y, ai.z};
    alpha_change_slot<NP>(P, B, pos4, vev4, alpha_in, s, pi, vev4[s], ai, na);
    alpha_out[s] = make_float4(na[0], na[1], na[2], ai.w);
}

// The pair of a particle and its neighbour j in the alpha change, j's data from
// the neighbour record that the drift (or force + drift) pass of this step wrote
// (five 16-byte loads per neighbour instead of seven separate gathers).
template <int NP>
__device__ __forceinline__ void nrec_pair(const DevParams& P, const DevBuffers& B, uint32_t j, AlphaChange<NP>& acc) {
    float4 q[5];
    read_nrec<NP>(B, j, q);
    const float4 r0 = q[0], r1 = q[1], r2 = q[2], r3 = q[3], r4 = q[4];
    float4 uj[NP];
    uj[0] = make_float4(r2.z, r2.w, r3.x, 0.f);
    if (NP > 1) uj[NP > 1 ? 1 : 0] = make_float4(r3.y, r3.z, r3.w, 0.f);
    if (NP > 2) uj[NP > 2 ? 2 : 0] = make_float4(r4.x, r4.y, r4.z, 0.f);
    acc.pair(P, r0, r0.w, make_float4(r1.x, r1.y, r1.z, 0.f), make_float4(r1.w, r2.x, r2.y, 0.f), uj);
}

// Alpha change of in-grid particle s, by one thread.
template <int NP>
__device__ __forceinline__ void alpha_change_nrec(const DevParams& P, const DevBuffers& B, int s, const float4 pi,
                                                  const float4 vei, const float4 ai, float (&out)[3]) {
    AlphaChange<NP> acc;
    acc.init(pi, vei, ai, B.drift4 + s, (size_t)P.cap);
    for_slot_list(P, B, s, pi.x, pi.y, pi.z, [&](uint32_t j) { nrec_pair<NP>(P, B, j, acc); });
    acc.result(P, out);
}

// Alpha change of heavy particle s by the whole warp (every lane calls with the
// same s and gets the result).
template <int NP>
__device__ __forceinline__ void alpha_change_nrec_warp(const DevParams& P, const DevBuffers& B, int s, const float4 pi,
                                                       const float4 vei, const float4 ai, float (&out)[3]) {
    AlphaChange<NP> acc;
    acc.init(pi, vei, ai, B.drift4 + s, (size_t)P.cap);
    warp_for_slot_list(P, B, s, pi.x, pi.y, pi.z, [&](uint32_t j) { nrec_pair<NP>(P, B, j, acc); });
    acc.template reduce<32>();
    acc.result(P, out);
}

// Alpha change of in-grid particle s shared out over the L lanes of its group (g this
// lane; every lane of the warp calls, `walk` where there is something to do).
template <int NP, int L>
__device__ __forceinline__ void alpha_change_nrec_group(const DevParams& P, const DevBuffers& B, int s, unsigned g,
                                                        bool walk, const float4 pi, const float4 vei, const float4 ai,
                                                        float (&out)[3]) {
    AlphaChange<NP> acc;
    acc.init(pi, vei, ai, B.drift4 + s, (size_t)P.cap);
    if (walk) group_for_slot_list<L>(P, B, s, g, pi.x, pi.y, pi.z, [&](uint32_t j) { nrec_pair<NP>(P, B, j, acc); });
    __syncwarp();
    acc.template reduce<L>();
    if (walk) acc.result(P, out);
}

// The same alpha advance in a step, where the drift pass has just written the neighbour
// records: those instead of seven gathers a neighbour (that pass's load units were
// 91 % busy with them), L lanes a particle (walk_lanes), the heavy ones from the
// queue. Bound by the records' loads (L1). 12, 53, 94 and 264 us at 12 K, 244 K,
// 421 K and 1.3 M slots against 27, 86, 129 and 356 with the gathers; the drift pass
// pays up to 9 us for writing the records.
template <int NP, int L>
__global__ void __launch_bounds__(kThreads, 4) k_alpha_advance_rec(const __grid_constant__ DevParams P,
                                                                   const __grid_constant__ DevBuffers B,
                                                                   const float4* __restrict__ pos4,
                                                                   const float4* __restrict__ vev4,
                                                                   const float4* __restrict__ alpha_in,
                                                                   float4* __restrict__ alpha_out) {
    if (P.list_mode != 0) {
        const unsigned lane = lane_id();
        const uint32_t nh = *B.hq_n;
        uint32_t* ctr = &B.hctr[kHeavyCounterAlpha];
        for (uint32_t h = next_item(ctr, nh, lane); h < nh; h = next_item(ctr, nh, lane)) {
            const int sh = (int)B.hq[h];
            const float4 ai = alpha_in[sh];
            float na[3] = {ai.x, ai.y, ai.z};
            alpha_change_nrec_warp<NP>(P, B, sh, pos4[sh], vev4[sh], ai, na);
            if (lane == 0) alpha_out[sh] = make_float4(na[0], na[1], na[2], ai.w);
        }
    }
    const int s = (int)((blockIdx.x * (unsigned)kThreads + threadIdx.x) / L);
    const unsigned g = threadIdx.x % L;
    const bool in = s < active_n(B);
    const int si = in ? s : 0;
    const float4 pi = pos4[si], ai = alpha_in[si];
    const bool sum = in && B.mgcell[si] != kUndef && !(pi.w < 0.f);
    const bool heavy = sum && is_heavy(P, B.nbr_cnt[si]);  // taken from the queue
    const bool walk = sum && !heavy;
    float na[3] = {ai.x, ai.y, ai.z};
    if (L == 1) {
        if (walk) alpha_change_nrec<NP>(P, B, s, pi, vev4[s], ai, na);
    } else if (__any_sync(0xffffffffu, walk)) {
        alpha_change_nrec_group<NP, L>(P, B, si, g, walk, pi, vev4[si], ai, na);
    }
    if (in && g == 0 && !heavy) alpha_out[s] = make_float4(na[0], na[1], na[2], ai.w);
}

// Separate correction, in place: fractions in alpha_cur, start-of-step in alpha_pre.
template <int NP>
__global__ void __launch_bounds__(kThreads) k_correction(const __grid_constant__ DevParams P,
                                                         const __grid_constant__ DevBuffers B,
                                                         float4* alpha_cur, const float4* alpha_pre,
                                                         float4* __restrict__ vel4,
                                                         const float4* __restrict__ pos4) {
    const int s = blockIdx.x * kThreads + threadIdx.x;
    if (s >= active_n(B)) return;
    if (B.mgcell[s] == kUndef || pos4[s].w < 0.f) return;
    const float4 ac = alpha_cur[s];
    const float4 ap = alpha_pre[s];
    float a[3] = {ac.x, ac.y, ac.z};
    const float apre[3] = {ap.x, ap.y, ap.z};
    float pmod, nr, nv;
    correct<NP>(P, a, apre, B.densp[s].x, ac.w, pmod, nr, nv);
    alpha_cur[s] = make_float4(a[0], a[1], a[2], nr);
    float4 v = vel4[s];
    v.w = nv;
    vel4[s] = v;
    B.pmod[s] = pmod;
}

// Separate advance, in place.
__global__ void __launch_bounds__(kThreads) k_advance(const __grid_constant__ DevParams P,
                                                      const __grid_constant__ DevBuffers B, float4* pos4,
                                                      float4* vel4, float4* vev4, float4* aprev4) {
    const int s = blockIdx.x * kThreads + threadIdx.x;
    if (s >= active_n(B)) return;
    float4 p = pos4[s];
    if (p.w < 0.f) return;
    float4 v = vel4[s];
    if (B.mgcell[s] == kUndef) {
        p.x = -1000.f; p.y = -1000.f; p.z = -1000.f;
        v.x = 0.f; v.y = 0.f; v.z = 0.f;
        pos4[s] = p;
        vel4[s] = v;
        return;
    }
    float4 ve = vev4[s], ap = aprev4[s];
    advance_one(P, p, v, ve, ap, B.accel4[s]);
    pos4[s] = p;
    vel4[s] = v;
    vev4[s] = ve;
    aprev4[s] = ap;
}

// Alpha + correction + advance of one slot whose alpha sum (in-grid fluid
// particles) is `anew`; writes the five float4 fields to the other buffer.
template <int NP, bool MP>
__device__ __forceinline__ void pass_c_finish(const DevParams& P, const DevBuffers& B, const F4Set& S, int s,
                                              bool undef, float4 p, float4 ve, float4 al, const float (&anew)[3]) {
    float4 v = S.in[VEL][s], ap = S.in[APREV][s];
    pass_c_slot<NP, MP>(P, B, s, undef, p, v, ve, al, ap, [&](float (&a)[3]) {
        a[0] = anew[0];
        a[1] = anew[1];
        a[2] = anew[2];
    });
    S.out[POS][s] = p;
    S.out[VEL][s] = v;
    S.out[VEV][s] = ve;
    S.out[ALPHA][s] = al;
    S.out[APREV][s] = ap;
}

// Fused alpha advance + correction + advance, one thread per particle: reads the
// cur buffers, writes every float4 field of every particle into the other
// buffer. Every warp first takes heavy particles from the queue (whole warp per
// alpha sum, lane 0 finishes the particle) while any are left.
template <int NP, bool MP, int L>
__global__ void __launch_bounds__(kThreads, 4) k_pass_c(const __grid_constant__ DevParams P,
                                                        const __grid_constant__ DevBuffers B,
                                                        const __grid_constant__ F4Set S) {
    if (MP && P.list_mode != 0) {
        const unsigned lane = lane_id();
        const uint32_t nh = *B.hq_n;
        uint32_t* ctr = &B.hctr[kHeavyCounterAlpha];
        for (uint32_t h = next_item(ctr, nh, lane); h < nh; h = next_item(ctr, nh, lane)) {
            const int sh = (int)B.hq[h];
            float a[3];
            const float4 p = S.in[POS][sh], ve = S.in[VEV][sh], al = S.in[ALPHA][sh];
            alpha_change_nrec_warp<NP>(P, B, sh, p, ve, al, a);
            if (lane == 0) pass_c_finish<NP, MP>(P, B, S, sh, false, p, ve, al, a);
        }
    }
    const int s = (int)((blockIdx.x * (unsigned)kThreads + threadIdx.x) / L);
    const unsigned g = threadIdx.x % L;
    const bool in = s < active_n(B);
    if (L == 1 && !in) return;
    const int si = in ? s : 0;
    const float4 p = S.in[POS][si], ve = S.in[VEV][si], al = S.in[ALPHA][si];
    const bool undef = B.mgcell[si] == kUndef;
    // the alpha sum is needed for in-grid fluid particles (pass_c_slot)
    const bool sum = MP && in && !undef && !(p.w < 0.f);
    const bool heavy = sum && is_heavy(P, B.nbr_cnt[si]);  // taken from the queue
    const bool walk = sum && !heavy;
    float anew[3] = {al.x, al.y, al.z};
    if (L == 1) {
        if (heavy) return;
        if (walk) alpha_change_nrec<NP>(P, B, s, p, ve, al, anew);
    } else if (__any_sync(0xffffffffu, walk)) {
        alpha_change_nrec_group<NP, L>(P, B, si, g, walk, p, ve, al, anew);
    }
    if (L == 1 || (in && g == 0 && !heavy)) pass_c_finish<NP, MP>(P, B, S, s, undef, p, ve, al, anew);
}

// ---------------------------------------------------------------------------
// FP64 conservation sums
// ---------------------------------------------------------------------------

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__global__ void __launch_bounds__(kThreads) k_conservation(const __grid_constant__ DevParams P,
                                                           const __grid_constant__ DevBuffers B,
                                                           const float4* __restrict__ pos4,
                                                           const float4* __restrict__ alpha4) {
    __shared__ double sh[6][kThreads / 32];
    double acc[6] = {0, 0, 0, 0, 0, 0};  // mass, volume, vol_k (3), max |sum alpha - 1|
    const int n = active_n(B);
    for (int s = blockIdx.x * kThreads + threadIdx.x; s < n; s += gridDim.x * kThreads) {
        if (B.mgcell[s] == kUndef) continue;
        const float4 p = pos4[s];
        if (p.w < 0.f) continue;
        const double m = p.w;
        const double vol = m * (double)B.densp[s].x;
        const float4 a = alpha4[s];
        const float al[3] = {a.x, a.y, a.z};
        acc[0] += m;
        acc[1] += vol;
        double sa = 0.0;
        for (int k = 0; k < P.nphase; k++) {
            acc[2 + k] += (double)al[k] * vol;
            sa += (double)al[k];
        }
        acc[5] = fmax(acc[5], fabs(sa - 1.0));
    }
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 5; q++) {
        const double v = warp_sum_d(acc[q]);
        if (lane == 0) sh[q][warp] = v;
    }
    double mx = acc[5];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) sh[5][warp] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 0; q < 5; q++) {
            double t = 0.0;
            for (int w = 0; w < kThreads / 32; w++) t += sh[q][w];
            atomicAdd(&B.red[q], t);
        }
        double m = 0.0;
        for (int w = 0; w < kThreads / 32; w++) m = fmax(m, sh[5][w]);
        atomicMax(reinterpret_cast<unsigned long long*>(&B.red[5]), (unsigned long long)__double_as_longlong(m));
    }
}

// ---------------------------------------------------------------------------
// Active count and device-side emission
// ---------------------------------------------------------------------------

__global__ void k_set_count(const __grid_constant__ DevBuffers B, int n) { *B.nact = n; }

// FluidSystem::EmitParticles (SPH_Solver/fluids/fluid_system.cpp:619-641) on the
// device, one block: at every frame that is a multiple of E.interval, the sites
// of `layers` disks (EmitImmediate, :644-673; InsertParticles, :676-700) are
// appended after the active slots and the device count grows; at capacity the
// remaining sites are dropped (AddParticle returns -1 there) and the capacity
// error bit is set. The sites, their jitter (stream E.seed + frame, two draws
// per site in (layer, i, j) order) and every record field are computed with the
// operations of the host generator sphmp_emit_disk in the same order, without
// contraction, so the records are the ones sphmp_emit_disk + sphmp_emit_aos
// would upload; a block-wide scan keeps the slot order of the accepted sites.
__global__ void __launch_bounds__(kScanBlock) k_emit(const __grid_constant__ DevParams P,
                                                     const __grid_constant__ DevBuffers B,
                                                     const __grid_constant__ F4Set S,
                                                     const __grid_constant__ DevEmitter E) {
    __shared__ int sh_frame, sh_base;
    if (threadIdx.x == 0) {
        sh_frame = *B.frame;
        sh_base = *B.nact;
    }
    __syncthreads();
    const int f = sh_frame;
    if (E.interval <= 0 || f % E.interval != 0) {
        if (threadIdx.x == 0) *B.frame = f + 1;
        return;
    }
    const uint32_t base = (uint32_t)sh_base;
    const uint32_t room = (uint32_t)P.cap - base;
    const int side = 2 * E.res + 1;
    const uint32_t per_layer = (uint32_t)(side * side);
    const uint32_t m = per_layer * (uint32_t)E.layers;
    const uint64_t seed = E.seed + (uint64_t)f;
    const float js = __fmul_rn(E.jitter, E.spacing);
    const float jh = __fmul_rn(js, 0.5f);
    const float r2 = __fmul_rn(E.radius, E.radius);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t written = 0;
    for (uint32_t c0 = 0; c0 < m; c0 += kScanBlock) {
        const uint32_t k = c0 + threadIdx.x;
        bool ok = false;
        float t0 = 0.f, t2 = 0.f;
        int layer = 0;
        if (k < m) {
            layer = (int)(k / per_layer);
            const uint32_t rem = k - (uint32_t)layer * per_layer;
            const int i = (int)(rem / (uint32_t)side) - E.res;
            const int j = (int)(rem % (uint32_t)side) - E.res;
            const float jx = __fsub_rn(__fmul_rn(__fmul_rn(uniform01(seed, 2ull * k), E.jitter), E.spacing), jh);
            const float jz = __fsub_rn(__fmul_rn(__fmul_rn(uniform01(seed, 2ull * k + 1ull), E.jitter), E.spacing), jh);
            t0 = __fadd_rn(__fmul_rn((float)i, E.spacing), jx);
            t2 = __fadd_rn(__fmul_rn((float)j, E.spacing), jz);
            const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(t0, t0), __fmul_rn(0.f, 0.f)), __fmul_rn(t2, t2));
            ok = !(d2 > r2);
        }
        uint32_t total;
        const uint32_t off = block_excl_scan(ok ? 1u : 0u, &total);
        const uint32_t q = written + off;
        if (ok && q < room) {
            const uint32_t idx = base + q;
            const float centre[3] = {E.pos[0], __fadd_rn(E.pos[1], __fmul_rn((float)layer, E.spacing)), E.pos[2]};
            float x[3], v[3];
#pragma unroll
            for (int a = 0; a < 3; a++) {
                x[a] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(E.rot[a][0], t0), __fmul_rn(E.rot[a][1], 0.f)),
                                           __fmul_rn(E.rot[a][2], t2)),
                                 centre[a]);
                v[a] = __fmul_rn(E.dir[a], E.vel);
            }
            S.out[POS][idx] = make_float4(x[0], x[1], x[2], E.mass);
            S.out[VEL][idx] = make_float4(v[0], v[1], v[2], E.visc);
            S.out[VEV][idx] = make_float4(v[0], v[1], v[2], 0.f);
            S.out[ALPHA][idx] = make_float4(E.onehot == 0 ? 1.f : 0.f, E.onehot == 1 ? 1.f : 0.f,
                                            E.onehot == 2 ? 1.f : 0.f, E.restdens);
            S.out[APREV][idx] = make_float4(0.f, 0.f, 0.f, __uint_as_float(idx));
            B.opos[idx] = idx;
            B.oidx[idx] = idx;
            B.densp[idx] = make_float2(0.f, 0.f);
            B.accel4[idx] = zero;
            B.color[idx] = make_float4(__fdiv_rn((float)f, 200.0f), 0.5f, 0.8f, 0.5f);
            B.bornid[idx] = (int32_t)idx;
            B.mass_raw[idx] = E.mass;
        }
        written += total;
    }
    if (threadIdx.x == 0) {
        if (written > room) set_err(B, kErrCapacity);
        *B.nact = (int)(base + min(written, room));
        *B.frame = f + 1;
    }
}

// ---------------------------------------------------------------------------
// Transfers
// ---------------------------------------------------------------------------

__device__ __forceinline__ bool finite3(float x, float y, float z) { return isfinite(x) && isfinite(y) && isfinite(z); }

__global__ void __launch_bounds__(kThreads) k_unpack_aos(const __grid_constant__ DevParams P,
                                                         const __grid_constant__ DevBuffers B,
                                                         const __grid_constant__ F4Set S,
                                                         const sphmp_display_pack* __restrict__ disp,
                                                         const float4* __restrict__ calc, int calc_words, int start,
                                                         int end) {
    const int i = start + blockIdx.x * kThreads + threadIdx.x;
    if (i >= end) return;
    // the records as 16-byte words: two of the display record, the first four of the
    // calculation record's 14 (the others are the solid fields: not used, and not always
    // uploaded, so that the records are 4 or 14 words apart)
    const float4* __restrict__ dq = reinterpret_cast<const float4*>(disp + (i - start));
    const float4* __restrict__ cq = calc + (size_t)(i - start) * calc_words;
    const float4 d0 = __ldcs(dq), d1 = __ldcs(dq + 1);
    const float4 c0 = __ldcs(cq), c1 = __ldcs(cq + 1), c2 = __ldcs(cq + 2), c3 = __ldcs(cq + 3);
    const sphmp_display_pack d = {{d0.x, d0.y, d0.z}, {d0.w, d1.x, d1.y, d1.z}, __float_as_int(d1.w)};
    struct {
        float vel[3], veleval[3], pressure, dens, restdens, mass, visc;
        int32_t bornid;
        float accel[3];
    } c = {{c0.x, c0.y, c0.z}, {c0.w, c1.x, c1.y}, c1.z, c1.w, c2.x, c2.y, c2.z, __float_as_int(c2.w), {c3.x, c3.y, c3.z}};
    int type = d.type;
    if (type != SPHMP_TYPE_FLUID && type != SPHMP_TYPE_BOUNDARY) {
        set_err(B, kErrType);
        type = SPHMP_TYPE_FLUID;
    }
    if (!finite3(d.pos[0], d.pos[1], d.pos[2])) set_err(B, kErrNotFinite);
    float w;
    if (type == SPHMP_TYPE_BOUNDARY) {
        w = -fabsf(c.dens);
        if (!(w < 0.f)) w = -1.f;  // a boundary needs a negative tag; the volume pass sets the value
    } else {
        w = c.mass;
        if (!(w > 0.f) || !isfinite(w)) {
            set_err(B, kErrBadMass);
            w = 1.f;
        }
    }
    S.out[POS][i] = make_float4(d.pos[0], d.pos[1], d.pos[2], w);
    S.out[VEL][i] = make_float4(c.vel[0], c.vel[1], c.vel[2], c.visc);
    S.out[VEV][i] = make_float4(c.veleval[0], c.veleval[1], c.veleval[2], 0.f);
    // one-hot volume fraction at the first phase whose rest density matches
    int ph = 0;
    for (int k = 0; k < P.nphase; k++)
        if (P.dens_k[k] == c.restdens) { ph = k; break; }
    S.out[ALPHA][i] = make_float4(ph == 0 ? 1.f : 0.f, ph == 1 ? 1.f : 0.f, ph == 2 ? 1.f : 0.f, c.restdens);
    S.out[APREV][i] = make_float4(0.f, 0.f, 0.f, __uint_as_float((uint32_t)i));
    B.opos[i] = (uint32_t)i;  // freshly written slots sit at their own internal index
    B.oidx[i] = (uint32_t)i;
    B.densp[i] = make_float2(c.dens, c.pressure);
    B.accel4[i] = make_float4(c.accel[0], c.accel[1], c.accel[2], 0.f);
    B.color[i] = make_float4(d.color[0], d.color[1], d.color[2], d.color[3]);
    B.bornid[i] = c.bornid;
    B.mass_raw[i] = c.mass;
}

// Writes the reference records of slots [0, n), a warp 32 of them: each lane
// gathers its particle, the warp writes the 224-byte calculation records as one
// contiguous run of 16-byte words (14 a record, the first four through shared
// memory, the solid fields zero). One thread a record with 4-byte stores at a
// stride of 224 bytes took 458 us for 1.3 M records (337 MB), this 73 us.
constexpr int kPackThreads = 128;
static_assert(sizeof(sphmp_display_pack) == 32 && sizeof(sphmp_calc_pack) == 14 * 16, "the record layouts");

__global__ void __launch_bounds__(kPackThreads) k_pack_aos(const __grid_constant__ DevParams P,
                                                           const __grid_constant__ DevBuffers B,
                                                           const __grid_constant__ F4Set S, sphmp_display_pack* disp,
                                                           sphmp_calc_pack* calc, int n) {
    __shared__ float4 sm[kPackThreads / 32][32][5];  // four words a record, one of padding
    const int slot = blockIdx.x * kPackThreads + threadIdx.x;
    const unsigned lane = lane_id();
    float4(&rec)[32][5] = sm[threadIdx.x >> 5];
    if (slot < n) {
        const int i = (int)B.opos[slot];
        const float4 p = S.in[POS][i];
        const uint32_t o = __float_as_uint(S.in[APREV][i].w);
        const bool bnd = p.w < 0.f;
        const float4 col = B.color[o];
        float4* dq = reinterpret_cast<float4*>(disp + slot);
        dq[0] = make_float4(p.x, p.y, p.z, col.x);
        dq[1] = make_float4(col.y, col.z, col.w, __int_as_float(bnd ? SPHMP_TYPE_BOUNDARY : SPHMP_TYPE_FLUID));
        if (calc != nullptr) {
            const float4 v = S.in[VEL][i], ve = S.in[VEV][i], ac = B.accel4[i];
            const float2 dp = B.densp[i];
            rec[lane][0] = make_float4(v.x, v.y, v.z, ve.x);
            rec[lane][1] = make_float4(ve.y, ve.z, bnd ? 0.f : dp.y, bnd ? -p.w : dp.x);
            rec[lane][2] = make_float4(S.in[ALPHA][i].w, B.mass_raw[o], v.w, __int_as_float(B.bornid[o]));
            rec[lane][3] = make_float4(ac.x, ac.y, ac.z, 0.f);
        }
    }
    if (calc == nullptr) return;
    __syncwarp();
    const int first = slot - (int)lane;
    const int words = 14 * max(0, min(32, n - first));
    float4* __restrict__ cq = reinterpret_cast<float4*>(calc + first);
    for (int k = (int)lane; k < words; k += 32) {
        const int r = k / 14, q = k % 14;
        __stcs(&cq[k], q < 4 ? rec[r][q] : make_float4(0.f, 0.f, 0.f, 0.f));
    }
}

__global__ void __launch_bounds__(kThreads) k_pack_field(const __grid_constant__ DevParams P,
                                                         const __grid_constant__ DevBuffers B,
                                                         const __grid_constant__ F4Set S, int field,
                                                         const float4* __restrict__ alpha_c,
                                                         const float4* __restrict__ alpha_p, void* stage, int n) {
    const int t = blockIdx.x * kThreads + threadIdx.x;  // slot (stage index)
    if (t >= n) return;
    const int i = (int)B.opos[t];                         // internal index
    float* f = reinterpret_cast<float*>(stage);
    int32_t* q = reinterpret_cast<int32_t*>(stage);
    const float4 p = S.in[POS][i];
    const uint32_t o = __float_as_uint(S.in[APREV][i].w);
    switch (field) {
        case SPHMP_F_POS: f[3 * t] = p.x; f[3 * t + 1] = p.y; f[3 * t + 2] = p.z; break;
        case SPHMP_F_VEL: { const float4 v = S.in[VEL][i]; f[3 * t] = v.x; f[3 * t + 1] = v.y; f[3 * t + 2] = v.z; } break;
        case SPHMP_F_VELEVAL: { const float4 v = S.in[VEV][i]; f[3 * t] = v.x; f[3 * t + 1] = v.y; f[3 * t + 2] = v.z; } break;
        case SPHMP_F_PRESSURE: f[t] = p.w < 0.f ? 0.f : B.densp[i].y; break;
        case SPHMP_F_DENS: f[t] = p.w < 0.f ? -p.w : B.densp[i].x; break;
        case SPHMP_F_RESTDENS: f[t] = alpha_c[i].w; break;
        case SPHMP_F_VISC: f[t] = S.in[VEL][i].w; break;
        case SPHMP_F_ACCEL: { const float4 a = B.accel4[i]; f[3 * t] = a.x; f[3 * t + 1] = a.y; f[3 * t + 2] = a.z; } break;
        case SPHMP_F_ALPHA: { const float4 a = alpha_c[i]; f[3 * t] = a.x; f[3 * t + 1] = a.y; f[3 * t + 2] = a.z; } break;
        case SPHMP_F_ALPHA_PRE: { const float4 a = alpha_p[i]; f[3 * t] = a.x; f[3 * t + 1] = a.y; f[3 * t + 2] = a.z; } break;
        case SPHMP_F_DRIFT:
            for (int k = 0; k < 3; k++) {
                const float4 u = B.drift4[(size_t)k * P.cap + i];
                f[9 * t + 3 * k] = u.x; f[9 * t + 3 * k + 1] = u.y; f[9 * t + 3 * k + 2] = u.z;
            }
            break;
        case SPHMP_F_APREV: { const float4 a = S.in[APREV][i]; f[3 * t] = a.x; f[3 * t + 1] = a.y; f[3 * t + 2] = a.z; } break;
        case SPHMP_F_PMOD: f[t] = B.pmod[i]; break;
        case SPHMP_F_VELXCOR: { const float4 x = B.velxcor[i]; f[3 * t] = x.x; f[3 * t + 1] = x.y; f[3 * t + 2] = x.z; } break;
        case SPHMP_F_TYPE: q[t] = p.w < 0.f ? SPHMP_TYPE_BOUNDARY : SPHMP_TYPE_FLUID; break;
        case SPHMP_F_MASS: f[t] = B.mass_raw[o]; break;
        case SPHMP_F_BORNID: q[t] = B.bornid[o]; break;
        default: break;
    }
}

__global__ void __launch_bounds__(kThreads) k_unpack_field(const __grid_constant__ DevParams P,
                                                           const __grid_constant__ DevBuffers B,
                                                           const __grid_constant__ F4Set S, int field,
                                                           float4* alpha_c, float4* alpha_p, const void* stage,
                                                           int n) {
    const int t = blockIdx.x * kThreads + threadIdx.x;  // slot (stage index)
    if (t >= n) return;
    const int i = (int)B.opos[t];                         // internal index
    const float* f = reinterpret_cast<const float*>(stage);
    float4* const __restrict__* out = S.out;
    switch (field) {
        case SPHMP_F_POS: { float4 p = out[POS][i]; p.x = f[3 * t]; p.y = f[3 * t + 1]; p.z = f[3 * t + 2]; out[POS][i] = p; } break;
        case SPHMP_F_VEL: { float4 v = out[VEL][i]; v.x = f[3 * t]; v.y = f[3 * t + 1]; v.z = f[3 * t + 2]; out[VEL][i] = v; } break;
        case SPHMP_F_VELEVAL: { float4 v = out[VEV][i]; v.x = f[3 * t]; v.y = f[3 * t + 1]; v.z = f[3 * t + 2]; out[VEV][i] = v; } break;
        case SPHMP_F_PRESSURE: { float2 d = B.densp[i]; d.y = f[t]; B.densp[i] = d; } break;
        case SPHMP_F_RESTDENS: { float4 a = alpha_c[i]; a.w = f[t]; alpha_c[i] = a; } break;
        case SPHMP_F_VISC: { float4 v = out[VEL][i]; v.w = f[t]; out[VEL][i] = v; } break;
        case SPHMP_F_ACCEL: B.accel4[i] = make_float4(f[3 * t], f[3 * t + 1], f[3 * t + 2], 0.f); break;
        case SPHMP_F_ALPHA: { float4 a = alpha_c[i]; a.x = f[3 * t]; a.y = f[3 * t + 1]; a.z = f[3 * t + 2]; alpha_c[i] = a; } break;
        case SPHMP_F_ALPHA_PRE: { float4 a = alpha_p[i]; a.x = f[3 * t]; a.y = f[3 * t + 1]; a.z = f[3 * t + 2]; alpha_p[i] = a; } break;
        case SPHMP_F_DRIFT:
            for (int k = 0; k < 3; k++)
                B.drift4[(size_t)k * P.cap + i] = make_float4(f[9 * t + 3 * k], f[9 * t + 3 * k + 1], f[9 * t + 3 * k + 2], 0.f);
            break;
        case SPHMP_F_APREV: { float4 a = out[APREV][i]; a.x = f[3 * t]; a.y = f[3 * t + 1]; a.z = f[3 * t + 2]; out[APREV][i] = a; } break;
        case SPHMP_F_PMOD: B.pmod[i] = f[t]; break;
        default: break;
    }
}

inline int blocks_for(int n, int t = kThreads) { return (n + t - 1) / t; }

// Blocks of kThreads for `lanes` threads per particle.
inline int walk_blocks(int n, int lanes) { return (int)(((long long)n * lanes + kThreads - 1) / kThreads); }

// Blocks of `threads` that are resident at once on the whole device (for
// kernels that loop over a device-side work count).
template <class K>
int resident_grid(K kernel, int threads) {
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, 0);
    if (sms <= 0) sms = 1;
    if (per <= 0) per = 1;
    return sms * per;
}

F4Set make_set(const DevBuffers& B, const int* cur, bool to_alt) {
    F4Set S;
    for (int f = 0; f < kNumFloat4Fields; f++) {
        S.in[f] = B.f4[f][cur[f]];
        S.out[f] = B.f4[f][to_alt ? cur[f] ^ 1 : cur[f]];
    }
    return S;
}

}  // namespace

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------

void launch_clear_counts(const DevBuffers& B, cudaStream_t s) { cudaMemsetAsync(B.ccount, 0, B.count_bytes, s); }

void launch_hash(const DevParams& P, const DevBuffers& B, const int* cur, bool sums, cudaStream_t s) {
    if (P.n <= 0) {
        cudaMemsetAsync(B.ctl, 0, sizeof(uint32_t) * kCtlWords, s);
        return;
    }
    k_hash<<<blocks_for(P.n, kHashBlock), kHashBlock, 0, s>>>(P, B, B.f4[POS][cur[POS]], sums && !P.morton ? 1 : 0);
}

void launch_recount(const DevParams& P, const DevBuffers& B, cudaStream_t s) {
    if (P.n > 0) k_recount<<<min(blocks_for(P.n, kHashBlock), 152 * 4), kHashBlock, 0, s>>>(P, B);
}

void launch_cell_starts(const DevParams& P, const DevBuffers& B, bool sums, bool clear, cudaStream_t s) {
    const int nb = (P.G + (int)kScanPer - 1) / (int)kScanPer;
    if (P.morton || !sums) k_scan_reduce<<<nb, kScanBlock, 0, s>>>(P, B);
    k_scan<<<nb, kScanBlock, 0, s>>>(P, B, clear ? 1 : 0);
}

void launch_cell_order(const DevParams& P, const DevBuffers& B, cudaStream_t s) {
    if (P.n <= 0) return;
    k_scatter<<<blocks_for(P.n), kThreads, 0, s>>>(P, B);
    // one warp a cell, at most one cell a particle
    const int grid = min(blocks_for(min(P.G, P.n), kThreads / 32), 152 * 16);
    k_cell_sort<<<grid, kThreads, 0, s>>>(P, B);
    k_big_cell_sort<<<64, 1024, 0, s>>>(P, B);
}

void launch_rearrange(const DevParams& P, const DevBuffers& B, const int* cur, bool slot_order, bool clear,
                      cudaStream_t s) {
    if (P.n <= 0) return;
    if (slot_order) k_slot_order<<<blocks_for(P.n), kThreads, 0, s>>>(P, B);
    k_rearrange<<<blocks_for(P.n), kThreads, 0, s>>>(P, B, make_set(B, cur, true), clear ? 1 : 0);
}

void launch_boundary_volume(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s) {
    if (P.n <= 0) return;
    const int g = (int)(((long long)P.n * kVolumeLanes + kThreads - 1) / kThreads);
    k_boundary_volume<<<g, kThreads, 0, s>>>(P, B, B.f4[POS][cur[POS]]);
    k_boundary_volume_store<<<blocks_for(P.n), kThreads, 0, s>>>(P, B, B.f4[POS][cur[POS]]);
}

void launch_density(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s) {
    if (P.n <= 0) return;
    cudaMemsetAsync(B.hq_n, 0, sizeof(uint32_t), s);  // its lists queue nobody: what the queue holds is of other lists
    k_density<<<blocks_for(P.n), kThreads, 0, s>>>(P, B, B.f4[POS][cur[POS]], B.f4[ALPHA][cur[ALPHA]]);
}

// `fresh`: the hash of this step has cleared the control words and no pass has used them since.
void launch_density_oct(const DevParams& P, const DevBuffers& B, const int* cur, bool fresh, cudaStream_t s) {
    if (P.n <= 0) return;
    const float4* pos = B.f4[POS][cur[POS]];
    const float4* alpha = B.f4[ALPHA][cur[ALPHA]];
    if (!fresh) {
        cudaMemsetAsync(B.dctr, 0, sizeof(uint32_t), s);
        cudaMemsetAsync(B.hq_n, 0, sizeof(uint32_t), s);
    }
    if (P.ss == 1.0f)
        k_density_bucket<true><<<resident_grid(k_density_bucket<true>, kDensThreads), kDensThreads, 0, s>>>(P, B, pos, alpha);
    else
        k_density_bucket<false><<<resident_grid(k_density_bucket<false>, kDensThreads), kDensThreads, 0, s>>>(P, B, pos, alpha);
}

// Lanes that share a particle in the list walks of the force and alpha passes. One
// thread a particle walks its neighbours as a chain of dependent gathers, which
// only many warps hide: a chip of 152 SMs holds 155,648 threads of these kernels
// (four blocks of 256 an SM). With fewer particles more lanes each are faster
// until they fill it; with more, the lanes' shuffles and repeated loads of the
// particle's own data only cost. Force + drift and alpha passes together, us, at
// one, two, four and eight lanes: 51, 33, 25, 21 at 22 K slots; 54, 38, 30, 38 at
// 49 K; 60, 57, 59, 69 at 106 K; 127, 107, 123, 165 at 244 K; 199, 186, 222, 299
// at 421 K; 322, 338, 420, 585 at 778 K; 518, 580, 720, 1012 at 1.3 M.
// (The project-U force keeps three blocks an SM: 43, 29, 29, 31 us at 63 K; 86, 84,
// 88, 107 at 244 K; 141, 150, 166, 201 at 421 K.)
static int walk_lanes(int n, int blocks = 4) {
    const int resident = 152 * blocks * kThreads;
    return n <= resident / 6 ? 8 : n <= resident / 2 ? 4 : n <= 3 * resident ? 2 : 1;
}

template <bool F, bool D, int NP>
static void fd_lanes(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s) {
    const float4* pos = B.f4[POS][cur[POS]];
    const float4* vel = B.f4[VEL][cur[VEL]];
    const float4* al = B.f4[ALPHA][cur[ALPHA]];
    const float4* ap = B.f4[APREV][cur[APREV]];
    const float4* ve = B.f4[VEV][cur[VEV]];
    switch (walk_lanes(P.n)) {
        case 8: k_force_drift<F, D, NP, 8><<<walk_blocks(P.n, 8), kThreads, 0, s>>>(P, B, pos, vel, al, ap, ve); break;
        case 4: k_force_drift<F, D, NP, 4><<<walk_blocks(P.n, 4), kThreads, 0, s>>>(P, B, pos, vel, al, ap, ve); break;
        case 2: k_force_drift<F, D, NP, 2><<<walk_blocks(P.n, 2), kThreads, 0, s>>>(P, B, pos, vel, al, ap, ve); break;
        default: k_force_drift<F, D, NP, 1><<<walk_blocks(P.n, 1), kThreads, 0, s>>>(P, B, pos, vel, al, ap, ve); break;
    }
}

template <bool F, bool D>
static void fd_dispatch(const DevParams& P, const DevBuffers& B, const int* cur, bool fresh, cudaStream_t s) {
    // the heavy-particle queue's work counter
    if (!fresh) cudaMemsetAsync(&B.hctr[kHeavyCounter<F, D>], 0, sizeof(uint32_t), s);
    if (!D) fd_lanes<F, false, 0>(P, B, cur, s);
    else if (P.nphase == 1) fd_lanes<F, true, 1>(P, B, cur, s);
    else if (P.nphase == 2) fd_lanes<F, true, 2>(P, B, cur, s);
    else fd_lanes<F, true, 3>(P, B, cur, s);
}

void launch_force_drift(const DevParams& P, const DevBuffers& B, const int* cur, bool force, bool drift, bool fresh,
                        cudaStream_t s) {
    if (P.n <= 0 || (!force && !drift)) return;
    if (force && drift) fd_dispatch<true, true>(P, B, cur, fresh, s);
    else if (force) fd_dispatch<true, false>(P, B, cur, fresh, s);
    else fd_dispatch<false, true>(P, B, cur, fresh, s);
}

void launch_force_drift_features(const DevParams& P, const DevBuffers& B, const int* cur, float* feat, int32_t* ids,
                                 float vs, float dt_large, cudaStream_t s) {
    if (P.n <= 0) return;
    const float4* pos = B.f4[POS][cur[POS]];
    const float4* vel = B.f4[VEL][cur[VEL]];
    const float4* al = B.f4[ALPHA][cur[ALPHA]];
    const float4* ap = B.f4[APREV][cur[APREV]];
    const float4* ve = B.f4[VEV][cur[VEV]];
    const int g = blocks_for(P.n, kFeatThreads);
    if (!P.multiphase) {
        k_force_drift_feat<false, 0><<<g, kFeatThreads, 0, s>>>(P, B, pos, vel, al, ap, ve, feat, ids, vs, dt_large);
        return;
    }
    switch (P.nphase) {
        case 1: k_force_drift_feat<true, 1><<<g, kFeatThreads, 0, s>>>(P, B, pos, vel, al, ap, ve, feat, ids, vs, dt_large); break;
        case 2: k_force_drift_feat<true, 2><<<g, kFeatThreads, 0, s>>>(P, B, pos, vel, al, ap, ve, feat, ids, vs, dt_large); break;
        default: k_force_drift_feat<true, 3><<<g, kFeatThreads, 0, s>>>(P, B, pos, vel, al, ap, ve, feat, ids, vs, dt_large); break;
    }
}

void launch_surface_tension(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s) {
    if (P.n <= 0) return;
    k_surface_tension<<<blocks_for(P.n), kThreads, 0, s>>>(P, B, B.f4[POS][cur[POS]]);
}

template <int NP>
static void projectu_lanes(const DevParams& P, const DevBuffers& B, const int* cur, int pre, cudaStream_t s) {
    const float4 *pos = B.f4[POS][cur[POS]], *vel = B.f4[VEL][cur[VEL]], *vev = B.f4[VEV][cur[VEV]],
                 *ac = B.f4[ALPHA][cur[ALPHA]], *ap = B.f4[ALPHA][pre], *apv = B.f4[APREV][cur[APREV]];
    switch (walk_lanes(P.n, 3)) {
        case 8: k_force_projectu_rec<NP, 8><<<walk_blocks(P.n, 8), kThreads, 0, s>>>(P, B, pos, vel, vev, ac, ap, apv); break;
        case 4: k_force_projectu_rec<NP, 4><<<walk_blocks(P.n, 4), kThreads, 0, s>>>(P, B, pos, vel, vev, ac, ap, apv); break;
        case 2: k_force_projectu_rec<NP, 2><<<walk_blocks(P.n, 2), kThreads, 0, s>>>(P, B, pos, vel, vev, ac, ap, apv); break;
        default: k_force_projectu_rec<NP, 1><<<walk_blocks(P.n, 1), kThreads, 0, s>>>(P, B, pos, vel, vev, ac, ap, apv); break;
    }
}

void launch_force_projectu(const DevParams& P, const DevBuffers& B, const int* cur, int pre, bool in_step, bool fresh,
                           cudaStream_t s) {
    if (P.n <= 0) return;
    if (in_step) {
        if (!fresh) cudaMemsetAsync(&B.hctr[kHeavyCounter<true, false>], 0, sizeof(uint32_t), s);
        if (P.nphase == 1) projectu_lanes<1>(P, B, cur, pre, s);
        else if (P.nphase == 2) projectu_lanes<2>(P, B, cur, pre, s);
        else projectu_lanes<3>(P, B, cur, pre, s);
        return;
    }
    const float4* pos = B.f4[POS][cur[POS]];
    const float4* vel = B.f4[VEL][cur[VEL]];
    const float4* vev = B.f4[VEV][cur[VEV]];
    const float4* ac = B.f4[ALPHA][cur[ALPHA]];
    const float4* ap = B.f4[ALPHA][pre];
    const float4* apv = B.f4[APREV][cur[APREV]];
    const int g = blocks_for(P.n);
    switch (P.nphase) {
        case 1: k_force_projectu<1><<<g, kThreads, 0, s>>>(P, B, pos, vel, vev, ac, ap, apv); break;
        case 2: k_force_projectu<2><<<g, kThreads, 0, s>>>(P, B, pos, vel, vev, ac, ap, apv); break;
        default: k_force_projectu<3><<<g, kThreads, 0, s>>>(P, B, pos, vel, vev, ac, ap, apv); break;
    }
}

template <int NP>
static void alpha_lanes(const DevParams& P, const DevBuffers& B, const float4* pos, const float4* vev, const float4* ain,
                        float4* aout, cudaStream_t s) {
    switch (walk_lanes(P.n)) {
        case 8: k_alpha_advance_rec<NP, 8><<<walk_blocks(P.n, 8), kThreads, 0, s>>>(P, B, pos, vev, ain, aout); break;
        case 4: k_alpha_advance_rec<NP, 4><<<walk_blocks(P.n, 4), kThreads, 0, s>>>(P, B, pos, vev, ain, aout); break;
        case 2: k_alpha_advance_rec<NP, 2><<<walk_blocks(P.n, 2), kThreads, 0, s>>>(P, B, pos, vev, ain, aout); break;
        default: k_alpha_advance_rec<NP, 1><<<walk_blocks(P.n, 1), kThreads, 0, s>>>(P, B, pos, vev, ain, aout); break;
    }
}

void launch_alpha_advance(const DevParams& P, const DevBuffers& B, const int* cur, bool in_step, bool fresh,
                          cudaStream_t s) {
    if (P.n <= 0) return;
    const float4* pos = B.f4[POS][cur[POS]];
    const float4* vev = B.f4[VEV][cur[VEV]];
    const float4* ain = B.f4[ALPHA][cur[ALPHA]];
    float4* aout = B.f4[ALPHA][cur[ALPHA] ^ 1];
    if (in_step) {
        if (!fresh) cudaMemsetAsync(&B.hctr[kHeavyCounterAlpha], 0, sizeof(uint32_t), s);
        if (P.nphase == 1) alpha_lanes<1>(P, B, pos, vev, ain, aout, s);
        else if (P.nphase == 2) alpha_lanes<2>(P, B, pos, vev, ain, aout, s);
        else alpha_lanes<3>(P, B, pos, vev, ain, aout, s);
        return;
    }
    const int g = blocks_for(P.n);
    switch (P.nphase) {
        case 1: k_alpha_advance<1><<<g, kThreads, 0, s>>>(P, B, pos, vev, ain, aout); break;
        case 2: k_alpha_advance<2><<<g, kThreads, 0, s>>>(P, B, pos, vev, ain, aout); break;
        default: k_alpha_advance<3><<<g, kThreads, 0, s>>>(P, B, pos, vev, ain, aout); break;
    }
}

void launch_correction(const DevParams& P, const DevBuffers& B, const int* cur, int pre, cudaStream_t s) {
    if (P.n <= 0) return;
    float4* ac = B.f4[ALPHA][cur[ALPHA]];
    const float4* ap = B.f4[ALPHA][pre];
    float4* vel = B.f4[VEL][cur[VEL]];
    const float4* pos = B.f4[POS][cur[POS]];
    const int g = blocks_for(P.n);
    switch (P.nphase) {
        case 1: k_correction<1><<<g, kThreads, 0, s>>>(P, B, ac, ap, vel, pos); break;
        case 2: k_correction<2><<<g, kThreads, 0, s>>>(P, B, ac, ap, vel, pos); break;
        default: k_correction<3><<<g, kThreads, 0, s>>>(P, B, ac, ap, vel, pos); break;
    }
}

void launch_advance(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s) {
    if (P.n <= 0) return;
    k_advance<<<blocks_for(P.n), kThreads, 0, s>>>(P, B, B.f4[POS][cur[POS]], B.f4[VEL][cur[VEL]],
                                                    B.f4[VEV][cur[VEV]], B.f4[APREV][cur[APREV]]);
}

template <int NP>
static void pass_c_lanes(const DevParams& P, const DevBuffers& B, const F4Set& S, cudaStream_t s) {
    switch (walk_lanes(P.n)) {
        case 8: k_pass_c<NP, true, 8><<<walk_blocks(P.n, 8), kThreads, 0, s>>>(P, B, S); break;
        case 4: k_pass_c<NP, true, 4><<<walk_blocks(P.n, 4), kThreads, 0, s>>>(P, B, S); break;
        case 2: k_pass_c<NP, true, 2><<<walk_blocks(P.n, 2), kThreads, 0, s>>>(P, B, S); break;
        default: k_pass_c<NP, true, 1><<<walk_blocks(P.n, 1), kThreads, 0, s>>>(P, B, S); break;
    }
}

void launch_pass_c(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s) {
    if (P.n <= 0) return;
    const F4Set S = make_set(B, cur, true);
    if (!P.multiphase) k_pass_c<1, false, 1><<<blocks_for(P.n), kThreads, 0, s>>>(P, B, S);
    else if (P.nphase == 1) pass_c_lanes<1>(P, B, S, s);
    else if (P.nphase == 2) pass_c_lanes<2>(P, B, S, s);
    else pass_c_lanes<3>(P, B, S, s);
}

void launch_conservation(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s) {
    cudaMemsetAsync(B.red, 0, sizeof(double) * 16, s);
    if (P.n <= 0) return;
    k_conservation<<<min(blocks_for(P.n), 152 * 8), kThreads, 0, s>>>(P, B, B.f4[POS][cur[POS]],
                                                                      B.f4[ALPHA][cur[ALPHA]]);
}

void launch_set_count(const DevBuffers& B, int n, cudaStream_t s) { k_set_count<<<1, 1, 0, s>>>(B, n); }

void launch_emit(const DevParams& P, const DevBuffers& B, const int* cur, const DevEmitter& E, cudaStream_t s) {
    k_emit<<<1, kScanBlock, 0, s>>>(P, B, make_set(B, cur, false), E);
}

void launch_unpack_aos(const DevParams& P, const DevBuffers& B, const int* cur, const sphmp_display_pack* d,
                       const void* c, int calc_bytes, int start, int end, cudaStream_t s) {
    if (end <= start) return;
    k_unpack_aos<<<blocks_for(end - start), kThreads, 0, s>>>(P, B, make_set(B, cur, false), d,
                                                             static_cast<const float4*>(c), calc_bytes / 16, start, end);
}

void launch_pack_aos(const DevParams& P, const DevBuffers& B, const int* cur, sphmp_display_pack* d,
                     sphmp_calc_pack* c, int n, cudaStream_t s) {
    if (n <= 0) return;
    k_pack_aos<<<blocks_for(n, kPackThreads), kPackThreads, 0, s>>>(P, B, make_set(B, cur, false), d, c, n);
}

void launch_pack_field(const DevParams& P, const DevBuffers& B, const int* cur, int field, int alpha_cur,
                       int alpha_pre, void* stage, int n, cudaStream_t s) {
    if (n <= 0) return;
    k_pack_field<<<blocks_for(n), kThreads, 0, s>>>(P, B, make_set(B, cur, false), field,
                                                     B.f4[ALPHA][alpha_cur], B.f4[ALPHA][alpha_pre], stage, n);
}

void launch_unpack_field(const DevParams& P, const DevBuffers& B, const int* cur, int field, int alpha_cur,
                         int alpha_pre, const void* stage, int n, cudaStream_t s) {
    if (n <= 0) return;
    k_unpack_field<<<blocks_for(n), kThreads, 0, s>>>(P, B, make_set(B, cur, false), field,
                                                       B.f4[ALPHA][alpha_cur], B.f4[ALPHA][alpha_pre], stage, n);
}

}  // namespace sphmp
