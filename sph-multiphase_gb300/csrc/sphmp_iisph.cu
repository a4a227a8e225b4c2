// sphmp_iisph.cu — the reference's IISPH step (implicit incompressible SPH) for
// sm_103a: ComputeDensityIISPH, ComputeDii / ComputeAii (PredictAdvection), the
// relaxed-Jacobi pressure iteration (Pressure_DP, Pressure_Iter) and
// IntegrateIISPH, SPH_Solver/fluids/fluid_system_kern.cu:637-1115, driven as
// fluid_system_host.cu:504-557 drives them.
//
// The reference scans 27 cells of edge 2h for every particle in every kernel and
// every iteration: 1,728 candidates for about 33 neighbours within h. Here the
// 27 cells (gc + neighborid[c]; each cell the index range [cstart, cend) of the
// sort) are scanned once a step, by warps that share their candidates among 8
// particles, for the density (cubic spline of support 2h); the scan also writes
// every particle's fluid neighbours within h and boundary neighbours within 2h as
// index lists, which every other sum walks, several lanes per particle. The
// kernels, cut-offs and formulas are the reference's (the advection viscosity
// within 2h, every other gradient sum within h). As in the reference, `dens` (densp.x) holds the density itself
// after the IISPH density pass, not its inverse. The per-particle IISPH arrays
// (d_ii, a_ii, predicted density, the pressure iterate and the terms its
// neighbours gather) live in DevBuffers.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "sphmp_device.cuh"
#include "sphmp_internal.h"

namespace sphmp {

namespace {

using namespace dev;

// kern (fluid_system_kern.cu:637-645) without its factor kspline: the cubic
// spline of support 2h at q = r / h <= 2.
__device__ __forceinline__ float ii_kern(float q) {
    const float t = 2.f - q;
    return q > 1.f ? __fmul_rn(0.25f, t * t * t)
                   : 1.f - __fmul_rn(__fmul_rn(1.5f, q), q) + __fmul_rn(0.75f, q * q * q);
}

// nablakern (:647-671): its gradient at x_ij is x_ij times this factor.
__device__ __forceinline__ float ii_nabla(const DevParams& P, float r) {
    const float q = r / P.h;
    if (q > 2.f) return 0.f;
    if (q > 1.f) return 0.75f * (2.f - q) * (2.f - q) * (-1.f) / P.h / r * P.kspline;
    return (-3.f * q + 2.25f * q * q) / P.h / r * P.kspline;
}

// The same within h, where (-3 q + 2.25 q^2) / q = 2.25 q - 3: no division. The
// factors that all pairs share (2.25 / h, and kspline / h^2 for whole sums) are
// rounded once from double or split, since their error would not average out.
struct NablaH {
    float c1, c0;  // 2.25 / h in two parts
    double k;      // kspline / h^2
    __device__ __forceinline__ explicit NablaH(const DevParams& P) {
        const double c = P.ii_c1;
        c1 = (float)c;
        c0 = (float)(c - (double)c1);
        k = P.ii_k;
    }
    // (the small part last: added to 3 it would vanish, which put 6e-8 of one sign into a_ii)
    __device__ __forceinline__ float operator()(float r) const { return fmaf(c0, r, fmaf(c1, r, -3.f)); }
    __device__ __forceinline__ float sum(float v) const { return (float)((double)v * k); }
};

__device__ __forceinline__ bool ii_fluid(const DevParams& P, const DevBuffers& B, int s, const float4* pos4) {
    return s < active_n(B) && B.mgcell[s] != kUndef && !(pos4[s].w < 0.f);
}

// ---------------------------------------------------------------------------
// Scans of the 27 cells, one warp for 8 consecutive particles
// ---------------------------------------------------------------------------

constexpr int kScanMembers = 8;
constexpr uint32_t kIiSearch = 0xffffffffu;  // nbr_cnt: the lists overflowed
constexpr int kScanThreads = 64;  // small blocks: warps with members (fluid) and without spread evenly over the SMs
constexpr int kScanWarps = kScanThreads / 32;

// Up to 27 cells (`cell` of the lanes below 27, kUndef for none) as index ranges:
// their starts and their offsets in the concatenated sequence go to the warp's
// shared table (roff[27] = its length, returned).
__device__ __forceinline__ uint32_t scan_ranges(const DevBuffers& B, uint32_t cell, unsigned lane, uint32_t* rstart,
                                                uint32_t* roff) {
    uint32_t st = 0, len = 0;
    if (lane < 27 && cell != kUndef) {
        st = __ldg(&B.cstart[cell]);
        len = __ldg(&B.cend[cell]) - st;
    }
    uint32_t inc = len;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, inc, d);
        if ((int)lane >= d) inc += v;
    }
    __syncwarp();  // the previous cell's table is read no more
    if (lane < 27) {
        rstart[lane] = st;
        roff[lane] = inc - len;
    }
    const uint32_t T = __shfl_sync(0xffffffffu, inc, 31);
    if (lane == 27) roff[27] = T;
    __syncwarp();
    return T;
}

// Visits, with a whole warp, the candidates of the particles its first lanes
// hold (`mine`; cell: the one each was sorted into): for each of their cells, the
// cells around it (`around` gets that cell and the lanes whose particle lies in
// it as a bit mask, and gives every lane below 27 a cell to search or kUndef),
// `chunk` with that mask and 32 candidates at a time, one a lane (index j, position pj; far
// away with w = 0 past the end), loaded one chunk ahead.
template <class A, class F>
__device__ __forceinline__ void scan_cells(const DevBuffers& B, const float4* __restrict__ pos4, bool mine,
                                           uint32_t cell, uint32_t* rstart, uint32_t* roff, A&& around, F&& chunk) {
    const unsigned lane = lane_id();
    const float kFar = __int_as_float(0x7f800000);
    unsigned todo = __ballot_sync(0xffffffffu, mine);
    while (todo) {
        const uint32_t gc = __shfl_sync(0xffffffffu, cell, __ffs(todo) - 1);
        const unsigned members = __ballot_sync(0xffffffffu, mine && cell == gc);
        todo &= ~members;
        const uint32_t T = scan_ranges(B, around(gc, members), lane, rstart, roff);
        int r = 0;
        uint32_t jn = 0;
        float4 pn;
        auto load = [&](uint32_t e) {
            pn = make_float4(kFar, kFar, kFar, 0.f);
            if (e < T) {
                while (roff[r + 1] <= e) r++;
                jn = rstart[r] + (e - roff[r]);
                pn = __ldg(&pos4[jn]);
            }
        };
        load(lane);
        for (uint32_t base = 0; base < T; base += 32) {
            const uint32_t j = jn;
            const float4 pj = pn;
            load(base + 32 + lane);
            chunk(members, j, pj);
        }
    }
}

// The sums over all lanes of each member's v, with their rounding errors: lane i gets
// member i's as sum + rest. Halves of the members go to halves of the lanes three times,
// then the four lanes of a member are added.
__device__ __forceinline__ void sum_members(float (&v)[kScanMembers], float& sum, float& rest) {
    static_assert(kScanMembers == 8, "three halvings");
    const unsigned lane = lane_id();
    float low[kScanMembers] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int o = 16, k = kScanMembers / 2; o > 0; o >>= 1, k >>= 1) {
        const bool up = (lane & (unsigned)o) != 0;
#pragma unroll
        for (int i = 0; i < (k > 0 ? k : 1); i++) {
            const float keep = k > 0 && up ? v[i + k] : v[i], keep0 = k > 0 && up ? low[i + k] : low[i];
            const float give = k > 0 && !up ? v[i + k] : v[i], give0 = k > 0 && !up ? low[i + k] : low[i];
            v[i] = keep;
            low[i] = keep0 + __shfl_xor_sync(0xffffffffu, give0, o);
            add_exact(v[i], low[i], __shfl_xor_sync(0xffffffffu, give, o));
        }
    }
    const int at = (int)((lane & 4u) << 2 | (lane & 2u) << 2 | (lane & 1u) << 2);  // where member `lane` ended up
    sum = __shfl_sync(0xffffffffu, v[0], at);
    rest = __shfl_sync(0xffffffffu, low[0], at);
}

// ComputeDensityIISPH (:1067-1115): rho_i = sum over every candidate of kern(x_ij) m_j,
// m_j = mass_j (fluid) or restdens_i V_j (boundary); also the lists of the fluid
// neighbours with 0 < r < h (entries 0, 1, ...) and of the boundary neighbours
// with 0 < r < 2h (entries kMaxNbr - 1, kMaxNbr - 2, ...), their counts in the low
// and high halves of nbr_cnt (kIiSearch when both do not fit: the walks then
// search the cells), and the particles that have them in iis_list (any order).
// The density is held in two parts (iis_rho_lo: what rounding to densp.x left) and its
// sums over masses and volumes apart (rest density times volume rounds alike for all of
// a wall's lattice): the residue of a solve is a mean of differences from the rest
// density, in which 1e-9 of the density of one sign shows as 1e-7 (33 K particles,
// ten iterations: 6e-7 off without these, 1e-8 with them).
// DENSITY false: the lists only. Issue-bound: a candidate costs its distance to
// every member (two at a time in packed FP32) and, within 2h, about 20
// instructions; the cut-offs compare squared distances with the smallest ones
// whose root is not below h and 2h (P.ii_cut), so no lane takes an exact root.
// At 33 K fluid and 43 K boundary particles: 517 us with one thread a particle
// over its own 1,728 candidates (a serial chain in a fifth of the warps the chip
// holds), 147 us shared by eight with exact roots and divisions, 109 us so.
template <bool DENSITY>
__global__ void __launch_bounds__(kScanThreads) k_ii_density(const __grid_constant__ DevParams P,
                                                             const __grid_constant__ DevBuffers B,
                                                             const float4* __restrict__ pos4,
                                                             const float4* __restrict__ alpha4) {
    __shared__ uint32_t tab[kScanWarps][2][28];
    __shared__ float2 mem[kScanWarps][kScanMembers / 2][3];  // x, y, z of two members each
    const unsigned lane = lane_id();
    const int w = threadIdx.x >> 5;
    const int s0 = (int)(blockIdx.x * kScanWarps + w) * kScanMembers;
    const int s = s0 + (int)lane;
    const bool mine = lane < kScanMembers && ii_fluid(P, B, s, pos4);
    const unsigned all = __ballot_sync(0xffffffffu, mine);
    if (!all) return;
    uint32_t cell = kUndef;
    if (mine) cell = B.mgcell[s];
    if (lane < kScanMembers) {
        float* m = &mem[w][lane >> 1][0].x + (lane & 1u);
        const float4 pm = mine ? pos4[s] : make_float4(0.f, 0.f, 0.f, 0.f);
        m[0] = pm.x;
        m[2] = pm.y;
        m[4] = pm.z;
    }
    __syncwarp();
    const float2 SS = make_float2(P.ss, P.ss);
    const float cut_h = P.ii_cut[0], cut_2h = P.ii_cut[1];
    const float ir2 = P.ii_ir2[0], ir20 = P.ii_ir2[1];
    float2 acc[kScanMembers];  // sums over masses, over boundary volumes
    uint32_t cf[kScanMembers], cb[kScanMembers];
#pragma unroll
    for (int i = 0; i < kScanMembers; i++) {
        acc[i] = make_float2(0.f, 0.f);
        cf[i] = cb[i] = 0;
    }
    scan_cells(B, pos4, mine, cell, tab[w][0], tab[w][1], [&](uint32_t gc, unsigned) { return gc + (uint32_t)P.neighborid[min(lane, 26u)]; },
               [&](unsigned members, uint32_t j, const float4 pj) {
        const float2 NX = make_float2(-pj.x, -pj.x), NY = make_float2(-pj.y, -pj.y), NZ = make_float2(-pj.z, -pj.z);
        const float cm = fmaxf(pj.w, 0.f), cv = fmaxf(-pj.w, 0.f);  // mass, or boundary volume
        const bool any_b = __any_sync(0xffffffffu, cv > 0.f);
        // the fluid neighbours' cut-off, the boundary neighbours' (0 for candidates of the other kind)
        const float cutf = cm > 0.f ? cut_h : 0.f, cutb = cv > 0.f ? cut_2h : 0.f;
#pragma unroll
        for (int p = 0; p < kScanMembers / 2; p++) {
            if (!(members >> (2 * p) & 3u)) continue;
            float2 dx = __fadd2_rn(mem[w][p][0], NX), dy = __fadd2_rn(mem[w][p][1], NY),
                   dz = __fadd2_rn(mem[w][p][2], NZ);
            dx = __fmul2_rn(dx, SS);
            dy = __fmul2_rn(dy, SS);
            dz = __fmul2_rn(dz, SS);
            const float2 d2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
            // r^2 / h^2, not 0 for the member itself
            const float2 qq2 = __ffma2_rn(d2, make_float2(ir2, ir2),
                                          __ffma2_rn(d2, make_float2(ir20, ir20), make_float2(1e-30f, 1e-30f)));
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int i = 2 * p + h;
                if (!(members >> i & 1u)) continue;
                const float dsq = h ? d2.y : d2.x;
                if (!__any_sync(0xffffffffu, dsq < cut_2h)) continue;
                if (DENSITY) {
                    // q = r / h to its last bit (a Newton step of the root): the density's mean is a
                    // small part of the residue's terms, so a bias of 1e-9 shows there. (The root
                    // after the division by h^2: a root times 1 / h = 80 takes few values between
                    // two floats, and rounds by -4e-9 on average.)
                    const float qq = h ? qq2.y : qq2.x;
                    const float rs = rsqrtf(qq), q0 = qq * rs;
                    const float q = fminf(fmaf(0.5f * rs, fmaf(-q0, q0, qq), q0), 2.f);
                    const float k = ii_kern(q);
                    acc[i] = __ffma2_rn(make_float2(k, k), make_float2(cm, cv), acc[i]);
                }
                const bool hit = dsq < cutf && dsq > 0.f;
                const unsigned b = __ballot_sync(0xffffffffu, hit);
                if (b) {
                    const uint32_t k = cf[i] + __popc(b & lanemask_lt());
                    if (hit && k < (uint32_t)kMaxNbr) B.nbr[nbr_at((size_t)P.cap, (uint32_t)(s0 + i), k)] = j;
                    cf[i] += __popc(b);
                }
                if (any_b) {
                    const bool hb = dsq < cutb && dsq > 0.f;
                    const unsigned bb = __ballot_sync(0xffffffffu, hb);
                    const uint32_t k = cb[i] + __popc(bb & lanemask_lt());
                    if (hb && k < (uint32_t)kMaxNbr)
                        B.nbr[nbr_at((size_t)P.cap, (uint32_t)(s0 + i), (uint32_t)kMaxNbr - 1u - k)] = j;
                    cb[i] += __popc(bb);
                }
            }
        }
    });
    float rho = 0.f, lo = 0.f;
    if (DENSITY) {
        float sum, rest, sumb, restb, part[kScanMembers];
#pragma unroll
        for (int i = 0; i < kScanMembers; i++) part[i] = acc[i].x;
        sum_members(part, sum, rest);
#pragma unroll
        for (int i = 0; i < kScanMembers; i++) part[i] = acc[i].y;
        sum_members(part, sumb, restb);
        // (mass sum + rest density times volume sum) kspline
        const float r0 = mine ? alpha4[s].w : 0.f, b = r0 * sumb;
        rest += fmaf(r0, sumb, -b) + r0 * restb;
        add_exact(sum, rest, b);
        const float p = sum * P.kspline, e = fmaf(sum, P.kspline, -p) + rest * P.kspline;
        rho = p + e;
        lo = (p - rho) + e;
    }
#pragma unroll
    for (int i = 0; i < kScanMembers; i++)
        if (lane == (unsigned)i && mine)
            B.nbr_cnt[s] = cf[i] + cb[i] <= (uint32_t)kMaxNbr ? cf[i] | (cb[i] << 16) : kIiSearch;
    if (mine) {
        if (DENSITY) B.densp[s].x = rho;
        B.iis_rho_lo[s] = lo;
    }
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(&B.iis_ctl[3], (uint32_t)__popc(all));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (mine) B.iis_list[at + __popc(all & lanemask_lt())] = (uint32_t)s;
}

// a / (b + c) rounded once more than exactly: the reference takes the sum and
// the quotient in double (c a double literal's product) and rounds to float;
// the sum's rounding error and the quotient's remainder are carried in float.
__device__ __forceinline__ float ii_quot(float a, float b, float c_hi, float c_lo) {
    const float s = __fadd_rn(b, c_hi);
    const float bb = __fsub_rn(s, b);
    const float e = __fadd_rn(__fadd_rn(__fsub_rn(b, __fsub_rn(s, bb)), __fsub_rn(c_hi, bb)), c_lo);
    const float q = a / s;
    const float rem = fmaf(-q, e, fmaf(-q, s, a));
    return q + rem / s;
}

// ---------------------------------------------------------------------------
// Sums over the lists, L lanes per particle
// ---------------------------------------------------------------------------

// The particle of a group of L consecutive lanes (-1: none).
template <int L>
__device__ __forceinline__ int ii_particle(const DevBuffers& B) {
    const uint32_t q = (blockIdx.x * kThreads + threadIdx.x) / L;
    return q < B.iis_ctl[3] ? (int)__ldg(&B.iis_list[q]) : -1;
}

// Visits the fluid neighbours of particle s within h (BOUNDARY: its boundary
// neighbours within 2h), the L lanes of its group taking every L-th group of
// four list entries: `get` loads what a neighbour gives beside its position, `f`
// gets that, the position, x_ij, and |x_ij| in (0, h) or (0, 2h). The four
// neighbours' loads are issued together.
template <int L, bool BOUNDARY, class G, class F>
__device__ __forceinline__ void ii_walk(const DevParams& P, const DevBuffers& B, const float4* __restrict__ pos4,
                                        int s, const float4 pi, G&& get, F&& f) {
    const uint32_t g = threadIdx.x % L;
    using R = decltype(get(0u));
    auto visit = [&](const float4 pj, const R& rec) {
        const float dx = (pi.x - pj.x) * P.ss, dy = (pi.y - pj.y) * P.ss, dz = (pi.z - pj.z) * P.ss;
        f(rec, pj, dx, dy, dz, sqrtf(dx * dx + dy * dy + dz * dz));
    };
    const uint32_t raw = B.nbr_cnt[s];
    if (raw != kIiSearch) {
        const uint32_t cnt = BOUNDARY ? raw >> 16 : raw & 0xffffu;
        const uint4* __restrict__ grp = reinterpret_cast<const uint4*>(B.nbr) + s;
        for (uint32_t k = 4u * g; k < cnt; k += 4u * L) {
            const uint32_t row = BOUNDARY ? (uint32_t)kMaxNbr / 4u - 1u - (k >> 2) : k >> 2;
            uint4 q = __ldg(grp + (size_t)row * (size_t)P.cap);
            if (BOUNDARY) q = make_uint4(q.w, q.z, q.y, q.x);
            // entries past the end of the list repeat its last group's first one, which is not visited again
            const uint32_t j[4] = {q.x, k + 1u < cnt ? q.y : q.x, k + 2u < cnt ? q.z : q.x, k + 3u < cnt ? q.w : q.x};
            float4 pj[4];
            R rec[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                pj[i] = __ldg(&pos4[j[i]]);
                rec[i] = get(j[i]);
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (k + (uint32_t)i < cnt) visit(pj[i], rec[i]);
        }
        return;
    }
    const uint32_t gc = B.mgcell[s];
    for (int c = 0; c < 27; c++) {
        const uint32_t cell = gc + (uint32_t)P.neighborid[c];
        const uint32_t j1 = __ldg(&B.cend[cell]);
        for (uint32_t j = __ldg(&B.cstart[cell]) + g; j < j1; j += L) {
            const float4 pj = __ldg(&pos4[j]);
            const float dx = (pi.x - pj.x) * P.ss, dy = (pi.y - pj.y) * P.ss, dz = (pi.z - pj.z) * P.ss;
            const float dsq = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));  // as the lists' test
            if ((BOUNDARY ? pj.w < 0.f : pj.w > 0.f) && dsq < P.ii_cut[BOUNDARY ? 1 : 0] && dsq > 0.f) visit(pj, get(j));
        }
    }
}

// ComputeDii, first half (:673-760): the advection acceleration (the boundary's
// artificial viscosity within 2h plus gravity; the fluid terms are commented
// out in the reference) and veleval = vel + a dt.
template <int L>
__global__ void __launch_bounds__(kThreads) k_ii_advect(const __grid_constant__ DevParams P,
                                                        const __grid_constant__ DevBuffers B,
                                                        const float4* __restrict__ pos4,
                                                        const float4* __restrict__ vel4, float4* __restrict__ vev4,
                                                        const float4* __restrict__ alpha4) {
    const int s = ii_particle<L>(B);
    float ax = 0.f, ay = 0.f, az = 0.f;
    float4 vi = make_float4(0.f, 0.f, 0.f, 0.f);
    if (s >= 0) {
        vi = vel4[s];
        const float rho0 = alpha4[s].w;
        const double c0 = (double)(P.h * P.h) * 0.01;
        const float c_hi = (float)c0, c_lo = (float)(c0 - (double)c_hi);
        ii_walk<L, true>(P, B, pos4, s, pos4[s], [&](uint32_t j) { return __ldg(&vel4[j]); },
                         [&](const float4 vj, const float4 pj, float dx, float dy, float dz, float r) {
            float pij = dx * (vi.x - vj.x) + dy * (vi.y - vj.y) + dz * (vi.z - vj.z);
            if (pij < 0.f) {
                pij = ii_quot(pij, r * r, c_hi, c_lo);
                pij = pij * P.bvisc * P.h / 2.f / rho0;
                pij = rho0 * (-pj.w) * pij;
                const float f = ii_nabla(P, r);
                ax += dx * f * pij;
                ay += dy * f * pij;
                az += dz * f * pij;
            }
        });
    }
    ax = group_sum<L>(ax); ay = group_sum<L>(ay); az = group_sum<L>(az);
    if (s < 0 || threadIdx.x % L != 0) return;
    ax += P.grav[0]; ay += P.grav[1]; az += P.grav[2];
    vev4[s] = make_float4(vi.x + ax * P.dt, vi.y + ay * P.dt, vi.z + az * P.dt, 0.f);
}

// ComputeDii, second half, and ComputeAii (:762-908) in one walk: d_ii = -sum
// nabla W_ij m_j / rho_i^2 dt^2; rho_adv = rho_i + sum (veleval_i - veleval_j).nabla
// W_ij m_j dt; p_l = 0.5 p_i; a_ii = sum (d_ii - d_ji).nabla W_ij m_j with d_ji =
// nabla W_ij m_i / rho_i^2 dt^2, which is d_ii.(sum nabla W_ij m_j) - (m_i / rho_i^2
// dt^2) sum |nabla W_ij|^2 m_j (both terms negative: nothing cancels).
template <int L>
__global__ void __launch_bounds__(kThreads) k_ii_aii(const __grid_constant__ DevParams P,
                                                     const __grid_constant__ DevBuffers B,
                                                     const float4* __restrict__ pos4,
                                                     const float4* __restrict__ vev4) {
    const int s = ii_particle<L>(B);
    const NablaH N(P);
    float sx = 0.f, sy = 0.f, sz = 0.f, s2 = 0.f, change = 0.f;
    if (s >= 0) {
        const float4 vei = vev4[s];
        ii_walk<L, false>(P, B, pos4, s, pos4[s], [&](uint32_t j) { return __ldg(&vev4[j]); },
                          [&](const float4 vej, const float4 pj, float dx, float dy, float dz, float r) {
            const float f = N(r);
            const float nx = dx * f, ny = dy * f, nz = dz * f;
            sx += nx * pj.w; sy += ny * pj.w; sz += nz * pj.w;
            s2 += (nx * nx + ny * ny + nz * nz) * pj.w;
            change += ((vei.x - vej.x) * nx + (vei.y - vej.y) * ny + (vei.z - vej.z) * nz) * pj.w;
        });
    }
    sx = group_sum<L>(sx); sy = group_sum<L>(sy); sz = group_sum<L>(sz);
    s2 = group_sum<L>(s2);
    change = group_sum<L>(change);
    if (s < 0 || threadIdx.x % L != 0) return;
    sx = N.sum(sx); sy = N.sum(sy); sz = N.sum(sz);
    s2 = N.sum(N.sum(s2));
    const float2 dpi = B.densp[s];
    const float rho = dpi.x, mi = pos4[s].w;
    const float dx = -sx / rho / rho * P.dt * P.dt, dy = -sy / rho / rho * P.dt * P.dt,
                dz = -sz / rho / rho * P.dt * P.dt;
    B.iis_aii[s] = (dx * sx + dy * sy + dz * sz) - mi / rho / rho * P.dt * P.dt * s2;
    float radv = rho, rest = 0.f;
    add_exact(radv, rest, fmaf(N.sum(change), P.dt, B.iis_rho_lo[s]));
    B.iis_rho_adv[s] = radv;
    B.iis_dii[s] = make_float4(dx, dy, dz, rest);
    B.iis_pl[s] = 0.5f * dpi.y;
}

// What the neighbours gather of p_l in Pressure_DP is p_l (m / rho / rho).
__global__ void __launch_bounds__(kThreads) k_ii_pm(const __grid_constant__ DevParams P,
                                                    const __grid_constant__ DevBuffers B,
                                                    const float4* __restrict__ pos4) {
    const int s = ii_particle<1>(B);
    if (s >= 0) B.iis_pm[s] = B.iis_pl[s] * (pos4[s].w / B.densp[s].x / B.densp[s].x);
}

// Pressure_DP (:910-958): sum_j d_ij p_j = -dt dt sum nabla W_ij p_l,j m_j / rho_j
// / rho_j, and d_ii p_l + that, which is what Pressure_Iter gathers of a
// neighbour (16 bytes instead of two float4 and p_l).
template <int L>
__global__ void __launch_bounds__(kThreads) k_ii_dp(const __grid_constant__ DevParams P,
                                                    const __grid_constant__ DevBuffers B,
                                                    const float4* __restrict__ pos4) {
    if (B.iis_ctl[1]) return;  // the solve has ended
    const int s = ii_particle<L>(B);
    const NablaH N(P);
    float dx_ = 0.f, dy_ = 0.f, dz_ = 0.f;
    if (s >= 0)
        ii_walk<L, false>(P, B, pos4, s, pos4[s], [&](uint32_t j) { return __ldg(&B.iis_pm[j]); },
                          [&](float pm, const float4, float dx, float dy, float dz, float r) {
            const float f = N(r) * pm;
            dx_ -= dx * f; dy_ -= dy * f; dz_ -= dz * f;
        });
    dx_ = group_sum<L>(dx_); dy_ = group_sum<L>(dy_); dz_ = group_sum<L>(dz_);
    if (s < 0 || threadIdx.x % L != 0) return;
    const float4 dii = B.iis_dii[s];
    const float pl = B.iis_pl[s];
    const float4 d = make_float4(N.sum(dx_) * P.dt * P.dt, N.sum(dy_) * P.dt * P.dt, N.sum(dz_) * P.dt * P.dt, 0.f);
    B.iis_dijpj[s] = d;
    B.iis_dsum[s] = make_float4(dii.x * pl + d.x, dii.y * pl + d.y, dii.z * pl + d.z, 0.f);
}

// Pressure_Iter (:960-1050) with omega 0.1: p_l1 = (1 - omega) p_l + omega / a_ii
// (rho0 - rho_adv - t), t = sum over fluid j within h of m_j (dijpj_i - d_jj p_l,j -
// (dijpj_j - d_ji p_l,i)).nabla W_ij (p_l1 = p_l where |a_ii| < 1e-5); the density
// residue rho_adv + t + a_ii p_l - rho0; accel = (d_ii p_l + dijpj) / dt / dt and
// pressure = p_l1, which is also the next iteration's p_l (:535; no other particle
// reads it here, so in place). Boundary particles have residue 0; the FP64 sums of
// the residue over all slots and of |residue| over in-grid fluid particles are
// published by the last block, which also counts the iteration and ends the solve
// (iis_ctl[1]) once `min_iter` iterations are done and the mean |residue| is at
// most `tol` (tol < 0: never).
template <int L>
__global__ void __launch_bounds__(kThreads) k_ii_iter(const __grid_constant__ DevParams P,
                                                      const __grid_constant__ DevBuffers B,
                                                      const float4* __restrict__ pos4,
                                                      const float4* __restrict__ alpha4, double tol, int min_iter) {
    if (B.iis_ctl[1]) return;  // the solve has ended
    // the blocks that hold particles (one when there is none) take part in the sums
    const unsigned nblk = max(1u, (B.iis_ctl[3] * L + kThreads - 1u) / kThreads);
    if (blockIdx.x >= nblk) return;
    const int s = ii_particle<L>(B);
    const bool own = s >= 0 && threadIdx.x % L == 0;
    const NablaH N(P);
    float ut = 0.f, mr = 0.f, pli = 0.f;
    float4 pi = make_float4(0.f, 0.f, 0.f, 0.f), dpi = pi;
    if (s >= 0) {
        pi = pos4[s];
        dpi = B.iis_dijpj[s];
        const float rho = B.densp[s].x;
        pli = B.iis_pl[s];
        mr = pi.w / rho / rho;
        const float ci = N.sum(mr * P.dt * P.dt * pli);  // d_ji p_l,i = (nabla W_ij / k) ci
        ii_walk<L, false>(P, B, pos4, s, pi, [&](uint32_t j) { return __ldg(&B.iis_dsum[j]); },
                          [&](const float4 ej, const float4 pj, float dx, float dy, float dz, float r) {
            const float f = N(r);
            const float nx = dx * f, ny = dy * f, nz = dz * f;
            const float tx = dpi.x - ej.x + nx * ci, ty = dpi.y - ej.y + ny * ci, tz = dpi.z - ej.z + nz * ci;
            ut += pj.w * (tx * nx + ty * ny + tz * nz);
        });
    }
    ut = group_sum<L>(ut);
    __shared__ float res[kThreads / L];
    if (threadIdx.x % L == 0) {
        float rv = 0.f;
        if (own) {
            const float4 dii = B.iis_dii[s];
            const float omega = 0.1f, aii = B.iis_aii[s], rho0 = alpha4[s].w, radv = B.iis_rho_adv[s];
            ut = N.sum(ut);
            const float off = ((radv - rho0) + dii.w) + ut;  // rho_adv - rho0 before it is rounded to rho's size
            const float pl1 = fabsf(aii) < 0.00001f ? pli : fmaf(omega, -off / aii - pli, pli);
            rv = fmaf(aii, pli, off);
            B.iis_pl[s] = pl1;
            B.iis_pm[s] = pl1 * mr;
            auto over_dt2 = [&](float v) { return fmaf(v, P.ii_idt2[0], v * P.ii_idt2[1]); };
            B.accel4[s] = make_float4(over_dt2(dii.x * pli + dpi.x), over_dt2(dii.y * pli + dpi.y),
                                      over_dt2(dii.z * pli + dpi.z), 0.f);
            B.densp[s].y = pl1;
        }
        res[threadIdx.x / L] = rv;
    }
    // every block leaves its sums in vtmp (three doubles a block), the last one adds
    // them up in a fixed order
    __shared__ double sh[3][kThreads / 32];
    __shared__ bool last;
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    const int nown = __syncthreads_count(own);
    double* part = reinterpret_cast<double*>(B.vtmp);
    if (warp == 0) {
        double r_all = 0.0, r_abs = 0.0;
        for (int k = (int)lane; k < kThreads / L; k += 32) {
            r_all += (double)res[k];
            r_abs += (double)fabsf(res[k]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            r_all += __shfl_xor_sync(0xffffffffu, r_all, o);
            r_abs += __shfl_xor_sync(0xffffffffu, r_abs, o);
        }
        if (lane < 3) {
            __stcg(&part[lane * nblk + blockIdx.x], lane == 0 ? r_all : lane == 1 ? r_abs : (double)nown);
            __threadfence();  // before the block's ticket
        }
    }
    __syncthreads();
    if (threadIdx.x == 0)  // wraps to 0 for the next iteration
        last = atomicInc(&B.iis_ctl[0], nblk - 1u) == nblk - 1u;
    __syncthreads();
    if (!last) return;
    __threadfence();
    double a[3] = {0.0, 0.0, 0.0};
    for (unsigned k = threadIdx.x; k < nblk; k += kThreads)
        for (int q = 0; q < 3; q++) a[q] += __ldcg(&part[q * nblk + k]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        for (int q = 0; q < 3; q++) a[q] += __shfl_xor_sync(0xffffffffu, a[q], o);
    if (lane == 0)
        for (int q = 0; q < 3; q++) sh[q][warp] = a[q];
    __syncthreads();
    if (threadIdx.x != 0) return;
    double tot[3] = {0.0, 0.0, 0.0};
    for (int q = 0; q < 3; q++) {
        for (int w = 0; w < kThreads / 32; w++) tot[q] += sh[q][w];
        B.red[11 + q] = tot[q];
    }
    const uint32_t it = ++B.iis_ctl[2];
    if ((int)it >= min_iter && (tot[2] > 0.0 ? tot[1] / tot[2] : 0.0) <= tol) B.iis_ctl[1] = 1u;
}

// The start of a solve or of a single iteration.
__global__ void k_ii_begin(const __grid_constant__ DevBuffers B) {
    if (threadIdx.x < 3) {
        B.iis_ctl[threadIdx.x] = 0u;
        B.red[11 + threadIdx.x] = 0.0;
    }
}

// IntegrateIISPH (:1052-1065): vel = veleval + accel dt; pos += vel dt / simscale.
__global__ void __launch_bounds__(kThreads) k_ii_integrate(const __grid_constant__ DevParams P,
                                                           const __grid_constant__ DevBuffers B,
                                                           float4* __restrict__ pos4, float4* __restrict__ vel4,
                                                           const float4* __restrict__ vev4) {
    const int s = blockIdx.x * kThreads + threadIdx.x;
    if (!ii_fluid(P, B, s, pos4)) return;
    const float4 ve = vev4[s], a = B.accel4[s];
    float4 v = vel4[s], p = pos4[s];
    v.x = ve.x + a.x * P.dt;
    v.y = ve.y + a.y * P.dt;
    v.z = ve.z + a.z * P.dt;
    p.x += v.x * P.dt / P.ss;
    p.y += v.y * P.dt / P.ss;
    p.z += v.z * P.dt / P.ss;
    vel4[s] = v;
    pos4[s] = p;
}

inline int blocks_for(int n) { return (n + kThreads - 1) / kThreads; }

}  // namespace

// Blocks of the list walks: L lanes per particle.
template <int L>
int walk_blocks(int n) {
    return (int)(((long long)n * L + kThreads - 1) / kThreads);
}

int scan_blocks(int n) {
    return (n + kScanMembers * kScanWarps - 1) / (kScanMembers * kScanWarps);
}

// Lanes per particle of the list walks: at 33 K fluid particles of about 33
// neighbours an iteration takes 27 us with four, 28 us with two and 38 us with
// eight lanes (Pressure_DP and Pressure_Iter; 903 us with one thread a particle
// searching the 27 cells): four have two rounds of four gathers in flight each.
constexpr int kWalkLanes = 4;

static void scan(bool density, const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s) {
    cudaMemsetAsync(&B.iis_ctl[3], 0, sizeof(uint32_t), s);
    if (P.n <= 0) return;
    const float4 *pos = B.f4[POS][cur[POS]], *al = B.f4[ALPHA][cur[ALPHA]];
    if (density) k_ii_density<true><<<scan_blocks(P.n), kScanThreads, 0, s>>>(P, B, pos, al);
    else k_ii_density<false><<<scan_blocks(P.n), kScanThreads, 0, s>>>(P, B, pos, al);
}

void launch_iisph_density(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s) {
    scan(true, P, B, cur, s);
}

void launch_iisph_lists(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s) {
    scan(false, P, B, cur, s);
}

void launch_iisph_predict(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s) {
    if (P.n <= 0) return;
    const int g = walk_blocks<kWalkLanes>(P.n);
    float4* vev = B.f4[VEV][cur[VEV]];
    k_ii_advect<kWalkLanes><<<g, kThreads, 0, s>>>(P, B, B.f4[POS][cur[POS]], B.f4[VEL][cur[VEL]], vev,
                                                   B.f4[ALPHA][cur[ALPHA]]);
    k_ii_aii<kWalkLanes><<<g, kThreads, 0, s>>>(P, B, B.f4[POS][cur[POS]], vev);
}

void launch_iisph_begin(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s) {
    k_ii_begin<<<1, 32, 0, s>>>(B);
    if (P.n <= 0) return;
    k_ii_pm<<<blocks_for(P.n), kThreads, 0, s>>>(P, B, B.f4[POS][cur[POS]]);
}

void launch_iisph_iteration(const DevParams& P, const DevBuffers& B, const int* cur, double tol, int min_iter,
                            cudaStream_t s) {
    if (P.n <= 0) return;
    const int g = walk_blocks<kWalkLanes>(P.n);
    k_ii_dp<kWalkLanes><<<g, kThreads, 0, s>>>(P, B, B.f4[POS][cur[POS]]);
    k_ii_iter<kWalkLanes><<<g, kThreads, 0, s>>>(P, B, B.f4[POS][cur[POS]], B.f4[ALPHA][cur[ALPHA]], tol, min_iter);
}

void launch_iisph_integrate(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s) {
    if (P.n <= 0) return;
    k_ii_integrate<<<blocks_for(P.n), kThreads, 0, s>>>(P, B, B.f4[POS][cur[POS]], B.f4[VEL][cur[VEL]],
                                                        B.f4[VEV][cur[VEV]]);
}

}  // namespace sphmp
