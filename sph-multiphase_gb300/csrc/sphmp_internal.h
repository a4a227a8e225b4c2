// sphmp_internal.h — device-side data layout and kernel launchers of the
// GB300 multiphase SPH step (shared by sphmp_kernels.cu and sphmp_api.cu).
//
// Particle state lives in HBM as structure-of-arrays in an internal order: the
// in-grid particles grouped by the reference's 2h cell (cell c occupies the same
// index range [cstart[c], cstart[c+1]) as its slots in the reference's sorted
// order) and, inside a cell, by h-subcell (octant); out-of-grid particles follow
// in slot order. opos[slot] and oidx[index] map between the reference's slots
// and internal indices; every reference-facing array (mgcell, midsort, mgndx,
// mgridoff, mgridcnt) and every transfer is in slot order. Every per-particle
// array that survives a step is a float4 so neighbour gathers are single
// 16-byte loads, and each is double-buffered: a pass that moves or advances
// particles reads buffer `cur` and writes buffer `cur ^ 1`.
//
//   pos4   : x, y, z (sim units), w = mass (fluid) or -V_b (boundary volume)
//   vel4   : vx, vy, vz, visc
//   vev4   : veleval x, y, z, (unused)
//   alpha4 : alpha_0, alpha_1, alpha_2, restdens
//   aprev4 : gravity - total accel of the last advance (x, y, z), w = origin slot
//            (bits of a uint32: the slot the particle was uploaded to)
//
// Per-step arrays (single buffer): densp (1/rho or V_b, pressure), accel4,
// drift4 (phase-major: drift of phase k for slot i at [k * cap + i]), pmod,
// velxcor (XSPH correction of the project-U force).
// Per-origin arrays (never moved): color, bornid, raw calc mass.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "sphmp.h"
#include "sphmp_learned.h"

namespace sphmp {

constexpr uint32_t kUndef = 0xFFFFFFFFu;
constexpr int kHashBlock = 256;       // threads per hash block (= one chunk for out-of-grid ranks)
constexpr int kScanBlock = 1024;      // threads per scan block
constexpr int kScanItems = 4;         // items per thread in the scan
constexpr uint32_t kScanPer = kScanBlock * kScanItems;  // cells per scan block
constexpr int kCtlWords = 16;         // control words of the sort and the passes (DevBuffers::ctl)
constexpr int kListWords = 3;         // the first of them: those a cell list counts with (act_n, wq_n, big_n)
constexpr int kWarpSortMax = 256;     // cells up to this size are sorted by one warp
constexpr int kCtaSortMax = 8192;     // larger cells up to this size are sorted by one CTA
constexpr int kNumFloat4Fields = 5;   // pos4, vel4, vev4, alpha4, aprev4
constexpr int kMaxNbr = 256;          // index-list capacity per particle (more: the passes rescan)
constexpr int kNrecFloat4 = 5;        // float4 per neighbour record of the alpha and project-U passes
// Bucket neighbour lists: a bitmask over the bucket's candidate sequence (the 27
// h-subcells around it as 18 index ranges), one word per 32 candidates.
constexpr int kMaskWords = 64;        // mask words per particle (more candidates: the passes rescan)
constexpr int kTabStride = 40;        // per bucket: [0..18] range ends in the sequence, [20..37] index - sequence
constexpr uint32_t kBucketWindow = 32;  // largest member window of one density work item (one member per lane)
constexpr uint32_t kBucketWindowMin = 8;
// Members that take one work item unless the caller says otherwise: n of them get
// 32 / n lanes each, so that 17 to 31 leave lanes idle, while small windows stage the same
// candidates more often. A state of 93 neighbours a particle, 1.05 M particles: the density
// pass 570, 582, 543, 580 and 576 us a step with 32, 24, 16, 12 and 10; as laid out (about
// eight members a bucket) the step is the same down to 16 and 1 to 3 % slower at 10.
constexpr uint32_t kBucketWindowDefault = 16;
constexpr uint32_t kMaskList = 0x80000000u;  // nbr_cnt flag: bucket mask list, low bits = bucket (cell * 8 + octant)
constexpr uint32_t kRescan = 0x7fffffffu;    // nbr_cnt value: no list, search the cells
// Heavy particles (long lists, overflowed lists, cell searches) are queued in hq by
// the density pass and taken by whole warps in the force and alpha passes; an
// index list of a heavy particle carries this flag over its length.
constexpr uint32_t kHeavyFlag = 0x40000000u;
constexpr uint32_t kHeavyList = 128;         // default: index lists longer than this are heavy

// Error bits accumulated in the device error word (1 << sphmp_status).
constexpr uint32_t kErrCellOverflow = 1u << SPHMP_ERR_CELL_OVERFLOW;
constexpr uint32_t kErrType = 1u << SPHMP_ERR_UNSUPPORTED_TYPE;
constexpr uint32_t kErrNotFinite = 1u << SPHMP_ERR_NOT_FINITE;
constexpr uint32_t kErrBadMass = 1u << SPHMP_ERR_BAD_MASS;
constexpr uint32_t kErrCapacity = 1u << SPHMP_ERR_CAPACITY;

// Scalars every kernel needs, passed by value.
struct DevParams {
    int n;           // launch size: the active slots, or the capacity while a device emitter runs
                     // (kernels bound themselves by the device counter, active_n)
    int cap;         // capacity (stride of phase-major arrays)
    int G;           // grid cells
    int rx, ry, rz;  // grid resolution
    float gmin[3];
    float fac[3];    // gridIdfac
    float srad[3];   // search radius h/simscale in cell units per axis, plus a rounding margin
    float ss;        // simscale
    float h, r2;     // smoothing radius and its square
    float ih, ir2;   // their reciprocals
    float dens_r2, dens_a;  // density terms (a (h^2 - r^2))^3 m: a h^2, and the a just above 1 that makes it a float
    float dens_k6[2];       // kpoly6 / a^3 in two parts
    float vol_scale;      // boundary volumes (k_boundary_volume): scale of a difference of positions,
    float vol_r2[2];      // the squared radius at that scale and the sums' factor, in two parts each
    float vol_factor[2];
    float r2list;    // squared radius of the neighbour list (r2 plus a rounding margin)
    int list_mode;   // 0: no list, 1: index lists in nbr (written by the last density pass)
    int narrow;      // 1: positions are the ones the cell lists were built from (the cell
                     // search may skip the cells beyond h of the current position)
    float dt;
    float kpoly6, kspikydiff;
    float kspline;   // 1 / (pi h^3), the cubic spline of the IISPH step
    float bvisc;
    float grav[3];
    int nphase;
    int multiphase;
    float dens_k[3], visc_k[3];
    float relax, sigma, cont, cont1, cont2, pintstiff;
    float omega, visc_factor;  // boundary factors of the project-U force
    int eos;
    float eos_k;
    int st_on;
    float st_K, st_C;
    int neighborid[27];
    int morton;      // 1: cells in Z-order in the sorted arrays (corder), 0: the reference's linear order
    int bwin;        // members per work item of the bucket density pass (8..32)
    uint32_t heavy;  // index lists longer than this are heavy (queued in hq)
    // IISPH: 2.25 / h, kspline / h^2, 1 / h^2 and 1 / dt^2 in two parts each, and the smallest
    // floats whose square root is not below h and 2h (the cut-offs on squared distances)
    double ii_c1, ii_k;
    float ii_ir2[2], ii_idt2[2];
    float ii_cut[2];
};

struct DevBuffers {
    float4* f4[kNumFloat4Fields][2];  // pos4, vel4, vev4, alpha4, aprev4 double buffers
    float2* densp;
    float4* accel4;
    float4* drift4;   // [3 * cap]
    float4* velxcor;  // [cap] XSPH velocity correction of the project-U force
    float* pmod;
    uint32_t* mgcell;   // sorted cell id per slot (unsorted key after the hash)
    uint32_t* midsort;  // pre-sort slot of each sorted slot
    uint32_t* mgndx;    // rank in cell
    int32_t* mgridoff;  // [G]
    int32_t* mgridcnt;  // [G]
    uint32_t* key;      // [cap] unsorted cell key per slot
    uint8_t* octk;      // [cap] octant (h-subcell inside the cell) per slot, in-grid slots only
    uint32_t* arank;    // [cap] rank inside the bin (atomic order; exact for out-of-grid)
    uint32_t* sidx;     // [cap] scatter target (pre-sort slots grouped by cell)
    // One allocation of count_bytes, all zero before a hash: a memset queued with it, but in the
    // library's captured steps, whose sorts clear what they have read
    uint32_t* ccount;   // [G + 4] particles per cell
    uint32_t* bsum;     // [G / kScanPer + 2] particles per kScanPer cells (linear order)
    uint32_t* usum;     // [cap / kHashBlock^2 + 2] out-of-grid slots per kHashBlock hash chunks
    uint32_t* counted;  // [1] 1: ccount and usum hold what the last hash's keys count to, 0: cleared since
    size_t count_bytes;
    uint32_t* cstart;   // [G + 2] exclusive scan of ccount in the cell order; cstart[G] = in-grid count,
                        // cstart[G+1] = n
    uint32_t* cend;     // [G] end of each cell's range (cstart[c + 1] in the linear order only)
    uint32_t* corder;   // [G] cells in Z-order (the scan order of the Morton mode)
    uint32_t* uchunk;   // [cap / kHashBlock + 2] out-of-grid count per hash chunk
    uint32_t* big;      // [cap / (kWarpSortMax+1) + 2] cells above the warp sort's size
    // Control words, one allocation of kCtlWords cleared by the hash (the first kListWords
    // also by a cell list of its own call): the pointers to single words below (act_n,
    // wq_n, big_n, hq_n, dctr, hctr) point into it
    uint32_t* ctl;
    uint32_t* big_n;    // [1] entries in big
    float4* color;      // [cap] per origin
    int32_t* bornid;    // [cap] per origin
    float* mass_raw;    // [cap] per origin
    uint32_t* err;      // device error word
    double* red;        // [16] FP64 reduction results
    float* vtmp;        // [cap + 64] scratch (boundary volumes; block sums of the IISPH residue)
    uint32_t* nbr;      // [kMaxNbr * cap] neighbour indices, groups of 4 column-major: entry k of s at ((k / 4) * cap + s) * 4 + k % 4
    uint32_t* nbr_cnt;  // [cap] list of particle s: index count (<= kMaxNbr), with kHeavyFlag if heavy; overflowed: kMaskList | bucket or kRescan
    uint32_t* nmask;    // [kMaskWords * cap] bucket mask lists (of overflowed index lists), column-major: word k of particle s at k * cap + s
    uint32_t* btab;     // [8 * G * kTabStride] candidate ranges of each bucket with a mask list
    uint32_t* dctr;     // [1] work counter of the bucket density kernel
    uint2* wq;          // [cap / kBucketWindowMin + 16] member windows after the first of large buckets:
                        // x = bucket (cell * 8 + octant), y = first member (internal index)
    uint32_t* wq_n;     // [1] entries in wq (filled by the cell sort)
    uint32_t* hq;       // [cap] heavy particles (internal index), filled by the density pass
    uint32_t* hq_n;     // [1] entries in hq
    uint32_t* hctr;     // [3] work counters over hq of the drift (or force + drift), force (or project-U) and alpha passes
    // IISPH step (sphmp_iisph.cu; one allocation, at iis_dii): d_ii, sum_j d_ij p_j, d_ii p_l + sum_j d_ij p_j (float4,
    // w unused but for d_ii's: what rho_adv's rounding left), a_ii, the predicted density, the pressure iterate p_l,
    // p_l m / rho^2, what rounding left of the density
    float4* iis_dii;
    float4* iis_dijpj;
    float4* iis_dsum;
    float* iis_aii;
    float* iis_rho_adv;
    float* iis_pl;
    float* iis_pm;
    float* iis_rho_lo;
    uint32_t* iis_ctl;  // [4] finished blocks of the running iteration, 1 when the solve has ended, iterations,
                        // particles in iis_list
    uint32_t* iis_list; // [cap] in-grid fluid particles with IISPH lists (any order)
    float4* nrec;       // [kNrecFloat4 * cap] neighbour records of the alpha and project-U passes (written by the drift pass)
    // Internal order: inside every 2h cell, members grouped by the h-subcell
    // (octant) they occupy, octant index (oy * 2 + oz) * 2 + ox.
    uint32_t* opos;     // [cap] internal index of each reference slot
    uint32_t* oidx;     // [cap] reference slot of each internal index (after the last sort)
    uint32_t* osrc;     // [cap] previous internal index of each new internal index (sort -> rearrange)
    uint32_t* oct_start;// [8 * G] first internal index of bucket (cell, octant)
    uint32_t* act;      // [G] cells with members (any order)
    uint32_t* act_n;    // [1] number of entries in act
    int32_t* nact;      // [1] active slots (device-side emission grows it inside a step)
    int32_t* frame;     // [1] steps since the device emitter was set
    uint32_t* esum;     // [1] scratch of the emission kernel
};

// Device-side disk emitter (the reference's EmitParticles, run before the sort
// of every step whose frame is a multiple of `interval`).
struct DevEmitter {
    float rot[3][3];   // columns (newx, dir, newz) of EmitImmediate's rotation
    float pos[3];
    float dir[3];
    float vel, radius, spacing, jitter;
    float mass, restdens, visc;  // of the emitted phase (massArr, densArr, viscArr)
    unsigned long long seed;
    int res;           // sites per half axis: int(radius / spacing)
    int layers, interval;
    int onehot;        // volume-fraction phase: the first whose rest density is `restdens`
};

#ifdef __CUDACC__
// The active slot count every kernel bounds itself by.
__device__ __forceinline__ int active_n(const DevBuffers& B) { return *B.nact; }
#endif

enum Field4 { POS = 0, VEL = 1, VEV = 2, ALPHA = 3, APREV = 4 };

// Input and output buffers of the five float4 fields for one kernel launch.
struct F4Set {
    const float4* __restrict__ in[kNumFloat4Fields];
    float4* __restrict__ out[kNumFloat4Fields];
};

// Record the text returned by sphmp_last_error on the calling thread (sphmp_api.cu).
sphmp_status record_error(sphmp_status st, const char* msg);

// ---- launchers (sphmp_kernels.cu) ----
// All take the current double-buffer selectors in `cur` (one per Field4).
// zero the counts the hash adds to (DevBuffers::ccount)
void launch_clear_counts(const DevBuffers& B, cudaStream_t s);
// cell keys, ranks and counts (the counts zero before), control words cleared; with
// `sums` also the sums of the counts in the linear order
void launch_hash(const DevParams& P, const DevBuffers& B, const int* cur, bool sums, cudaStream_t s);
// the counts again from the last hash's keys, if they have been cleared since (decided on the device)
void launch_recount(const DevParams& P, const DevBuffers& B, cudaStream_t s);
// GetGridList in two halves: cell starts (a scan of the counts, whose sums the hash
// of the same step left with `sums`; with `clear` the counts are zeroed), then the
// scatter, the per-cell stable ordering and the per-cell octant order
void launch_cell_starts(const DevParams& P, const DevBuffers& B, bool sums, bool clear, cudaStream_t s);
void launch_cell_order(const DevParams& P, const DevBuffers& B, cudaStream_t s);
// move every particle to its new internal index (osrc) and update opos; with
// `slot_order`, the new internal order is the reference's sorted slot order
// (for a rearrange that did not follow this library's grid list); with `clear`
// the rest of the counts is zeroed
void launch_rearrange(const DevParams& P, const DevBuffers& B, const int* cur, bool slot_order, bool clear,
                      cudaStream_t s);
void launch_boundary_volume(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s);
void launch_density(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s);
// octant-order density (needs the octant order of this sort); writes slot lists.
// `fresh` here and below: the control words the pass counts with are still as the
// hash of this step cleared them (otherwise they are cleared first)
void launch_density_oct(const DevParams& P, const DevBuffers& B, const int* cur, bool fresh, cudaStream_t s);
void launch_force_drift(const DevParams& P, const DevBuffers& B, const int* cur, bool force, bool drift, bool fresh,
                        cudaStream_t s);
void launch_surface_tension(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s);
// project-U force: start-of-step fractions in alpha4[pre], rest densities in alpha4[cur[ALPHA]]
// in_step: the drift pass of this step has just written the neighbour records, which are read instead of the fields
void launch_force_projectu(const DevParams& P, const DevBuffers& B, const int* cur, int pre, bool in_step, bool fresh,
                           cudaStream_t s);
// alpha advance: reads alpha4[cur], writes alpha4[cur^1] (new fractions, same restdens)
void launch_alpha_advance(const DevParams& P, const DevBuffers& B, const int* cur, bool in_step, bool fresh, cudaStream_t s);
// correction: fractions in alpha4[cur[ALPHA]], start-of-step fractions in alpha4[pre]; in place
void launch_correction(const DevParams& P, const DevBuffers& B, const int* cur, int pre, cudaStream_t s);
// advance in place on the cur buffers
void launch_advance(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s);
// fused alpha + correction + advance of a step: reads cur, writes cur^1 for all five float4 fields
void launch_pass_c(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s);
void launch_conservation(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s);
// IISPH step (sphmp_iisph.cu): density (densp.x = rho, and the index lists in nbr /
// nbr_cnt of the fluid neighbours within h, which the next two need; `lists` writes
// only those), PredictAdvection (veleval, d_ii, rho_adv, p_l = p / 2, a_ii), the start
// of a solve, one pressure iteration (accel, pressure = the next p_l; FP64 residue
// sums in red[11..13], iis_ctl[1] set when the solve has ended), integration
void launch_iisph_density(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s);
void launch_iisph_lists(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s);
void launch_iisph_predict(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s);
void launch_iisph_begin(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s);
void launch_iisph_iteration(const DevParams& P, const DevBuffers& B, const int* cur, double tol, int min_iter,
                            cudaStream_t s);
void launch_iisph_integrate(const DevParams& P, const DevBuffers& B, const int* cur, cudaStream_t s);
// set the device counter of active slots
void launch_set_count(const DevBuffers& B, int n, cudaStream_t s);
// device-side emission into the current buffers (one block)
void launch_emit(const DevParams& P, const DevBuffers& B, const int* cur, const DevEmitter& E, cudaStream_t s);

// learned large step: the force (+ drift) pass that also fills the corrector's
// features of every particle (feat [n][48], ids = bornid, -1 without features;
// sphmp_kernels.cu), and the correction of the step's result by the network
// outputs y [n][4] (sphmp_learned.cu)
void launch_force_drift_features(const DevParams& P, const DevBuffers& B, const int* cur, float* feat, int32_t* ids,
                                 float vs, float dt_large, cudaStream_t s);
void launch_apply_correction(const DevParams& P, const DevBuffers& B, const int* cur, const float* y,
                             const float* out_scale, const int32_t* ids, float dt_large, float* corr, cudaStream_t s);

// differences of state b against state a (see sphmp_compare_states); map: scratch of map_size
// entries (bornid -> index of a), out: 7 doubles (6 sums, then the maximum)
void launch_compare(const DevParams& Pa, const DevBuffers& Ba, const int* cur_a, const DevParams& Pb,
                    const DevBuffers& Bb, const int* cur_b, int32_t* map, int map_size, double* out, cudaStream_t s);

// transfers (staging buffers hold reference records; the calculation records of an
// upload calc_bytes apart, at least their first kCalcUsed bytes: all that the upload reads)
constexpr int kCalcUsed = 64;
void launch_unpack_aos(const DevParams& P, const DevBuffers& B, const int* cur, const sphmp_display_pack* d,
                       const void* c, int calc_bytes, int start, int end, cudaStream_t s);
void launch_pack_aos(const DevParams& P, const DevBuffers& B, const int* cur, sphmp_display_pack* d,
                     sphmp_calc_pack* c, int n, cudaStream_t s);
// field pack/unpack through a float/uint32 staging array; `aux` = alpha_pre buffer selector
void launch_pack_field(const DevParams& P, const DevBuffers& B, const int* cur, int field, int alpha_cur,
                       int alpha_pre, void* stage, int n, cudaStream_t s);
void launch_unpack_field(const DevParams& P, const DevBuffers& B, const int* cur, int field, int alpha_cur,
                         int alpha_pre, const void* stage, int n, cudaStream_t s);

// the corrector network as the large step uses it (sphmp_learned.cu)
cudaError_t corrector_forward_on(sphmp_corrector* c, const float* x, int n, float* y, uint32_t* err, cudaStream_t s);
const float* corrector_out_scale(const sphmp_corrector* c);  // device [4]
int corrector_device(const sphmp_corrector* c);

}  // namespace sphmp
