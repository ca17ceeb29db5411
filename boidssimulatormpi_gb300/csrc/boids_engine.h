// boids_engine.h -- constants and kernel launchers shared by the C-ABI host
// code (boids_capi.cpp, compiled by g++) and the kernels (boids_kernels.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>

#include "boids_softfp.h"

namespace boidsgpu {

// Every comparison of the reference that mixes a float with a double is
// replaced by an exactly equivalent float comparison against a constant the
// host derives once:
//   (double)f <  d   <=>  f <  up(d)      (up: smallest float >= d)
//   (double)f >  d   <=>  f >  dn(d)      (dn: largest float  <= d)
// The radius test of Boid::isInsideArea (src/boid.cpp:28),
// (double)sqrtf(d2) < r, becomes d2 < d2_lim with d2_lim the smallest float
// whose correctly rounded square root reaches r; the view-cone test
// acos(c) <= pi*a (src/boid.cpp:34-35) becomes cstar <= c <= 1, with cstar
// found on the host with the same acosf the reference calls.
inline float f_dn(double d)  // largest float <= d
{
    float f = (float)d;
    if ((double)f > d) f = std::nextafter(f, -INFINITY);
    return f;
}

inline float f_up(double d)  // smallest float >= d
{
    float f = (float)d;
    if ((double)f < d) f = std::nextafter(f, INFINITY);
    return f;
}

// Conservative filter radius: the exact distance test can only accept a
// pair whose approximate distance is below this (rounding of the image
// shift and of the filter's own arithmetic is far below the margin).
inline double filter_ulp(float F) { return std::nextafter(std::fmax(F, 1.0f), INFINITY) - std::fmax(F, 1.0f); }
inline double filter_radius(float rmax, float F) { return (double)rmax * (1.0 + 1e-4) + 8.0 * filter_ulp(F); }

// The all-pairs product filter's angle scale and least sum.  It sums
// cos(2 pi dx / F) over the axes, for a pair within rf at least
// 3 - (2 pi rf / F)^2 / 2 (cos a >= 1 - a^2 / 2).  Rounding cosines and sines
// (at most 1) to half precision moves each by at most 2^-12, an axis's sum by
// 2 sqrt(2) 2^-12 + 2^-23: 2.08e-3 over the axes; the angles of coordinates up
// to 4 F (2^-23 relative), sincospif, the FP32 sum of eight products and min's
// own split into two half-precision terms add less than 1e-4.
// Three cosines never sum to less than -3: -4 passes every pair, whatever the
// radius, and its terms stay within half precision.  A field so small that the
// scale overflows gets angles of zero, which pass every pair, too.
// The terms of a boid are w = -min (at most 4) and u, what w's rounding left
// of it; a boid too far outside the field for its angles adds kApPass to both.
// Rows and columns past the last boid have kApPad in their place: no angles
// and -16, which rejects them with every boid (w + kApPass + u < 16).
constexpr float kApPass = 8.f;
constexpr uint32_t kApPad = 0xcc00u;  // -16 in half precision
struct ApFilter {
    float turn, min;
};
inline ApFilter ap_filter(double rf, double F)
{
    const double r = 2.0 * 3.141592653589793 * (rf * (1.0 + 1e-4) + 8.0 * filter_ulp((float)F)) / F;
    const float turn = (float)(2.0 / F);
    return ApFilter{std::isfinite(turn) ? turn : 0.f, f_dn(std::fmax(-4.0, 3.0 - r * r / 2.0 - 2.3e-3))};
}

struct RuleConst {
    float d2_lim;     // radius test: d2 < d2_lim
    float cstar;      // smallest c with (double)acosf(c) <= M_PI*sight_angle
    int32_t all_round;  // sight_angle >= 1.0: the cone test is skipped
    int32_t pad;
};

enum { RULE_COH = 0, RULE_SEP = 1, RULE_ALI = 2 };

struct StepConst {
    uint32_t n;          // boids
    int32_t G;           // device cells per axis along y and z (>= 3), 0 for all-pairs
    int32_t Gx;          // device cells along x: 4 * G (each a quarter of a y/z cell)
    double F;            // field size (host side only)
    SoftDouble Fsd;      // the field size in integer form, for exact float +- double
    float Ff;            // (float)F, for approximate filters
    float F_dn;          // dn(F): wrap test x > F
    float halfF_dn;      // dn(F/2): minimum-image tests
    float inv_side;      // y/z cells per unit length of the device grid
    float inv_subx;      // x cells per unit length (4 * inv_side)
    float side;          // y/z cell side (approximate, for row trimming)
    float trim_r2;       // squared radius, with margin, used to trim a boid's rows
    float filt_r2;       // squared radius of the conservative fast filter
    float box_lim;       // all-pairs box filter: ||dx| - F/2| > box_lim
    float halfFf;        // (float)(F/2) for the box filter
    float ap_turn, ap_min;  // all-pairs product filter: 2 / F, least sum of the axes' cosines of a pair in reach
    float cc, cs, ca;    // (float) force coefficients: cohesion, separation, alignment
    float vmax_dn, vmin_up;  // speed clamp tests
    float vmax_f, vmin_f;    // speed clamp scale factors (float)vmax, (float)vmin
    float d2_any;        // largest d2_lim of the three rules
    float cone_band;     // approximate cone tests closer than this to a threshold are redone exactly
    // View-cone pre-test of the candidate filters, on when every rule has a
    // cone that rejects c <= 0 (cstar > 0): a candidate whose approximate
    // v . r is below -|v| * dot_eps has an exact v . r < 0 and fails all
    // three rules.  dot_eps bounds the approximation's error per unit |v|.
    float dot_eps;
    int32_t cone_pre;
    // The dense kernel's half-precision filter (two candidates per
    // instruction) works on coordinates relative to the cell's centre times
    // hsc (a power of two putting them within +-0.5) and velocities times
    // hvsc (a power of two putting |v| <= vmax within 0.5).  hfilt bounds the
    // half-precision squared distance of any pair within the filter radius;
    // a pair is dropped behind the boid when its half-precision v . r is
    // below -(hdot0 + hdot1 |v| hvsc), which bounds that dot product's error.
    float hsc, hvsc, hfilt, hdot0, hdot1;
    int32_t id_bits;     // bits needed for the largest boid id, rounded up to a multiple of 4
    RuleConst rule[3];   // cohesion, separation, alignment
    // the reference's overlapping grid, for Boid::grid_index parity
    int32_t refG;
    float refGS, refR;
    // Place of this flock in a batched ensemble (all zero for one flock):
    // its cells are global cells [cell_base, cell_base + Gx*G*G), its boids
    // occupy state slots [slot_base, slot_base + n), and slot = cell start
    // (a prefix over all flocks' counts) + slot_off, the padding that aligns
    // every flock to kSlotAlign slots.  Boid ids are local to the flock.
    uint32_t cell_base;
    uint32_t slot_base;
    uint32_t slot_off;
    uint32_t flock;
    // Which full-size cells the CTA-per-cell kernel takes (the results do not
    // depend on it): those holding dense_min boids or more, those holding
    // defer_min or more whose 27-cell neighbourhood holds over cand_defer
    // boids, and any non-empty cell whose neighbourhood holds over lone_cand.
    uint32_t dense_min, defer_min, cand_defer, lone_cand;
    uint32_t tuned;  // the split applies whatever the size: those were set by boids_set_tuning, or an autotuner
                     // found the split with them faster than the choice between it and a warp per boid
};

// A batched ensemble's flock table, in device memory.  Every block of
// kSlotAlign state slots belongs to one flock, so a CTA of that many threads
// serves one flock and can hold its StepConst in shared memory.
constexpr int kSlotAlign = 128;
struct FlockTable {
    const StepConst *ks;        // per flock
    const uint16_t *blk_flock;  // per block of kSlotAlign slots
    const uint32_t *cell4;      // per flock: cell_base / 4 (ascending)
    uint32_t count;             // flocks
    uint32_t nslots;            // padded slots of all flocks
};

// Device scratch of one engine handle.  Sizes in elements.
struct DevBuffers {
    float4 *pos[2], *vel[2];   // ping-pong state, float4 (w of pos = id bits)
    uint32_t *key, *rank;      // per slot: device cell and rank inside it
    uint32_t *count;           // per cell (padded): boids binned so far
    uint32_t *lstart;          // per cell (padded): exclusive scan inside a tile
    uint32_t *bsum;            // per scan tile: offset of the tile
    uint32_t *ticket;          // scan completion counter, and its sum of pairs (2 words, zero between scans)
    uint32_t *ap_cnt, *ap_list;  // all-pairs: per boid neighbour count and list
    uint4 *ap_emb;             // all-pairs: per boid filter vector
    float *forces;             // 9 per boid (id order), optional
    float *stage;              // 6 per boid, host<->device staging
    int32_t *cells8;           // 8 per boid (id order)
    int32_t *dcnt;             // 3 per boid (id order)
    uint64_t *dhash;           // 3 per boid (id order)
    uint32_t *dense_list;      // dense kernel work items (cell, first boid), this step (dense_list_capacity words)
    uint32_t *dense_n;         // dense items, the step's work queue, deferred sparse boids, pairs of boids that
                               // share an x cell (4 words)
    uint32_t *defer;           // sparse boids deferred to further passes: (slot, lo_id), 2 words per slot (null: none);
                               // a flock's entries start at its slot_base
    uint32_t *defer_cnt;       // deferred boids per flock (a single flock: dense_n + 2)
    uint64_t *ovf;             // per slot, kOvfCap entries: the accepted neighbours a deferred boid's
                               // first pass could not keep (null: none)
    uint32_t *ovf_n;           // per slot: how many there were (over kOvfCap: the row is incomplete)
    uint64_t *wscratch;        // dense kernel: wcap entries per CTA, a huge cell's candidates filed by window
    uint32_t wcap;             // (null / 0: every window scans the neighbourhood)
    // Side stream on which the deferred boids run beside the dense kernel,
    // forked from and joined back to the engine's stream (null: in order).
    cudaStream_t aux;
    cudaEvent_t fork, join, cjoin;  // cjoin: the classification's end (it runs beside the scatter)
    uint32_t *slot_of;         // slot of each id after the scatter (from its flock's slot_base), for steps that
                               // go a warp per boid (null: none does)
    uint8_t *dflag;            // per full-size cell: 1 when the dense kernel takes it
    void *carry;               // per slot, kCarryBytes: partial sums between id windows (null: no windows)
    double crowd_min, crowd_max;  // an ensemble: the pairs from which, and up to which, its boids go a warp each
    uint32_t *flag;            // set_state range check (1 word)
    uint32_t ncell, ncell_pad, nscan_blocks;
    uint32_t sms;              // SMs of the device (a handle's)
    uint32_t dense_grid;       // CTAs of the dense-cell kernel
    uint32_t ap_cap;
};

constexpr int kScanTile = 2048;       // cells per scan block (256 threads x 8)
constexpr int kListCap = 12;          // grid engine, thread-per-boid kernel: sorted neighbours kept per pass
constexpr int kOvfCap = 24;           // accepted neighbours beyond those a deferred boid's first pass keeps
// Defaults, measured on the bench workload (N = 2^20 from a uniform start,
// steps 5-25), the same flock after 1000 steps, and gathered flocks of 16 384
// and 65 536 boids: dense_min 16 beats 12 on all four (3-6 %); lone_cand 64
// costs 5x on the uniform start, as many small cells become CTA work items,
// and lone_cand above 96 costs the small gathered flocks 5-20 %.  Clustered
// flocks run another 15-40 % faster with lower thresholds still, which the
// autotuners pick.
constexpr int kDenseMin = 16;         // default dense_min
constexpr int kDeferMin = 4;          // default defer_min
constexpr int kCandDefer = 192;       // default cand_defer
constexpr int kLoneCand = 96;         // default lone_cand
constexpr int kCarryBytes = 72;       // partial sums of one boid between id windows
constexpr uint32_t kWinScratch = 32768;  // most candidates a CTA files by window (twice what 32 windows hold)

// Dense-cell threshold sets the autotuners try, {dense_min, defer_min,
// cand_defer, lone_cand}; the first is the default.  Crowded (clustered)
// states favour low thresholds, uniform states high ones.
constexpr uint32_t kNever = 1u << 30;
constexpr uint32_t kTuneCand[][4] = {
    {16, 4, 192, 96}, {12, 4, 192, 96}, {12, 4, 192, 384}, {12, 4, 192, 64}, {12, 4, 192, 48},
    {8, 2, 96, 128}, {4, 2, 64, 128}, {8, 4, 128, 64}, {kNever, kNever, kNever, 1024},
};
constexpr int kTuneCount = sizeof(kTuneCand) / sizeof(kTuneCand[0]);

// The dense kernel's work items are (full-size cell, first boid) pairs, one
// per kDenseItem boids of a dense cell, so that the boids of one crowded
// cell spread over several CTAs.  Every item gathers and sorts its cell's
// neighbourhood.  Where that takes id windows (over kDenseCap candidates), a
// remainder of up to half an item is shared among the cell's other items
// (dense_per_item), and while a CTA has many items to come it takes up to
// kDenseTake at once and does a cell's in a row together: without either,
// uniform flocks of 16 to 48 times the reference's density took 5 to 13 % longer
// than with items of 128 boids (2^20 boids at 32 times, us a step: 7110, now
// 6405, 6265 with those; at 16 times 3670, 3245, 3465), which in turn cost
// gathered flocks 10 to 30 % up to 2^19 boids (262 143 400 updates after a
// uniform start 777, now 655; 2^20 2350 and 2030).  Sharing remainders in all
// cells, or taking several items at once until fewer are left (kDenseLeft 1, 2),
// cost those 2 to 10 %; in flocks of 41 000 to 65 537 boids, whose items are few,
// sharing any cost 2 to 4 % (at 56 times the density 837 and 860).
constexpr int kDenseItem = 32;
constexpr uint32_t kDenseShare = 100000;  // boids from which remainders are shared
constexpr uint32_t kDenseTake = 4;  // most items taken at once ...
constexpr uint32_t kDenseLeft = 3;  // ... which is those left over, for every CTA so many times
constexpr int kDenseRound = 64;     // boids whose results a CTA holds in shared memory, over an item's most
// Words the work list can need in one step: at most one item per non-empty
// cell plus one per kDenseItem boids, and never more than one per boid, two
// words per item.
inline size_t dense_list_capacity(size_t ncell, size_t n)
{
    const size_t by_cells = ncell / 4;
    const size_t items = (by_cells < n ? by_cells : n) + n / kDenseItem + 1;
    return 2 * (items < n ? items : n);
}
// Flocks of up to this many boids (all flocks of an ensemble together) are
// always updated a warp per boid (k_grid_warp).  A
// step with either, us: 32 768 boids uniform 58 / 74, gathered 90 / 215;
// 49 152 uniform 75 / 71, gathered 124 / 251; 65 537 uniform 95 / 73.  The
// line lies where a uniform flock takes the same time with both.
constexpr uint32_t kWarpBoids = 40960;
// Larger ones, up to kCrowdBoids boids (an ensemble's kCrowdSlots), are sent
// there or by the split step for step, on the device, by the pairs of boids
// that share an x cell (counted by the scan): a warp per boid from
// crowd_line pairs a boid up to crowd_top, above which boids
// accept more neighbours than k_grid_warp's list holds.  Without id windows in
// the split (the allocation-free step) there is no upper line.  A uniform flock
// at the reference's density has 0.29 n pairs, a gathered one 1 to 3.2 n.  A
// step, us, by the split / a warp per boid: 65 537 boids at 0.53 n 106 / 111,
// at 0.72 n 194 / 117, at 1.3 n 290 / 134, at 3.0 n 264 / 177; 131 072 at
// 0.55 n 145 / 190, at 0.75 n 252 / 210, at 1.3 n 370 / 238; 262 143 at 0.75 n
// 331 / 430, at 0.94 n 419 / 412, at 1.3 n 511 / 447, at 3.1 n 632 / 614;
// 370 000 at 1.3 n 626 / 620, at 3.1 n 870 / 860.  Without id windows in the
// split (the allocation-free step), 65 537 at 2.3 n 2990 / 163.  Ensembles of
// flocks that gather together, whose split has no side stream and no
// deferral: 65 536 slots at 0.38 n 116 / 133, at 0.46 n 141 / 135; 131 072 at
// 0.68 n 225 / 239, at 0.79 n 269 / 243; 262 144 at 0.68 n 359 / 431, at 0.79 n
// 429 / 440, at 1.0 n 533 / 462; 491 520 at 0.79 n 725 / 792, at 1.0 n 891 / 826.
// Flocks collapsed into clusters, at 4, 8 and 16 n pairs: 50 000
// boids 353 / 156, 233 / 250, 339 / 693; 262 143 599 / 653, 689 / 1170,
// 1053 / 9348; an ensemble of 16 flocks of 8192 at 4 and 8 n 550 / 392 and
// 465 / 517.  Flocks of up to kWarpBoids, which know no such line, take longer
// than by the split only where they have collapsed, from 24 576 boids on (at most
// 2.1 times, 40 960 in clusters of 4000: 2242 / 1180).
constexpr uint32_t kCrowdBoids = 1u << 18, kCrowdSlots = 1u << 19;
constexpr double kCrowdTop = 8.5, kCrowdTopSlope = 1.6e-5, kCrowdTopEnsemble = 6.0;
enum CrowdKind { CROWD_HANDLE, CROWD_BARE, CROWD_ENSEMBLE };  // the split's form: a handle's, the allocation-free step's, ...
// The pairs a boid from which a flock goes a warp per boid: even is what the
// flock would have spread evenly over its cells, n the boids (slots) of the step.
inline double crowd_line(double even, double n, CrowdKind kind)
{
    const bool many = kind == CROWD_ENSEMBLE;
    // (Thin flocks of a small ensemble have gathered further by then: 100 flocks of
    // 1000 at a quarter of the density at 0.41 n 211 / 173 us.)
    const double thin = 0.75 * std::fmin(0., even - 0.29);
    const double line = many ? std::fmin(0.2 + 3.8e-6 * n + thin, 0.78 + 2.5e-7 * n)
                             : (kind == CROWD_HANDLE ? 0.47 : 0.35) + 1.75e-6 * n;
    // From 3.3 times the reference's density on a flock that is still even
    // makes full items of all its cells, the split's best state, until so many
    // cells have more candidates than the shared list (or, in small flocks, too few
    // items): at 6 times the density 262 143 boids 445 / 554 us a step, 65 537
    // 144 / 164, the allocation-free step of 262 143 520 / 553, 48 flocks of 8192
    // 733 / 988; at 8 times 65 537 216 / 201; at 12 times 131 072 429 / 416.
    if (even >= 0.95) {
        const double most = many ? 1.2 + 2.3e-11 * n * n : (kind == CROWD_HANDLE ? 1.6 + 1e-5 * n : (n < 150000 ? 0. : 2.));
        return std::fmax(line, std::fmin(1.5 * even, most));
    }
    // From 1.45 times on its cells of a few boids have too many candidates for a
    // thread each: an ensemble's split is at its worst (16 flocks of 16 384 at twice
    // the density 658 / 457).
    return many && even >= 0.42 ? even - 0.45 : line;
}
// And up to which: beyond what an even flock has, as long as k_grid_warp's lists
// hold the neighbours that its boids accept on average (at 24 times the density, 103
// of them, 65 537 boids 487 / 351 us, 262 143 1331 / 1207; at 48 times, 206, 632 /
// 883 and 2310 / 2763; at 56 times, 240, 1413 / 929 and 11 900 / 2865).  The line
// falls with the ids that a boid's search has to pass over, which are an ensemble's
// flock's own, however many flocks there are.
constexpr double kCrowdSeen = 207.;  // 3.5 deviations below the lists' 256
inline double crowd_top(double even, double seen, double n, CrowdKind kind)
{
    return (kind == CROWD_ENSEMBLE ? kCrowdTopEnsemble : kCrowdTop - kCrowdTopSlope * n) +
           (seen <= kCrowdSeen ? even : 0.);
}
// The neighbours that a boid of an even flock accepts: the most of its rules' view cones hold.
inline double crowd_seen(const StepConst &k)
{
    double most = 0.;
    for (const RuleConst &q : k.rule) {
        const double r = std::sqrt((double)q.d2_lim) / k.F;
        most = std::fmax(most, k.n * 4.18879 * r * r * r * (q.all_round ? 1. : (1. - (double)q.cstar) / 2.));
    }
    return most;
}
// The autotuners time the default set with the choice above (or the split, if
// the flock has no other: routed == false), the others with the split.  What a
// flock gains now it can lose many times over once its state has changed: on a
// uniform flock the set without dense cells is the fastest by 1 to 5 % (65 537
// boids 67 us a step for 69, 262 143 143 for 148), and with it the same flock
// took 1222 and 2270 us once it had gathered, where the choice takes 146 and
// 522.  So a routed flock leaves the default for a set faster by kTuneMargin
// only, and the choice only where the split with that set beats the choice with
// it by as much (262 143 boids in small clusters 446 us for 680).
constexpr float kTuneMargin = 1.1f;
// The set to keep, from every set's time.
inline int tune_choice(const float *ms, bool routed)
{
    int best = 0;
    for (int c = 1; c < kTuneCount; ++c)
        if (ms[c] < ms[best]) best = c;
    return routed && !(ms[best] * kTuneMargin < ms[0]) ? 0 : best;
}
// Whether that set comes with the split alone, from its times with it and with the choice.
inline bool tune_splits(float split_ms, float choice_ms) { return split_ms * kTuneMargin < choice_ms; }
// Up to this many boids and cells (padded) a flock's counting sort is one
// CTA's work (k_grid_sort, k_grid_bin_one).
constexpr uint32_t kSortBoids = 1024, kSortCells = 4096;
// Up to this many boids and cells (padded) the allocation-free step's counting
// sort is one kernel (k_grid_bin): on the eight SMs of its cluster the scatter
// of more takes longer than the launches it saves.
constexpr uint32_t kBinBoids = 16384, kBinCells = 65536;
constexpr int kDenseCap = 512;        // candidates of a dense cell held in shared memory
// Boids per item of a dense cell of b boids with ncand candidates (share: the
// step has kDenseShare boids or more).
__host__ __device__ inline uint32_t dense_per_item(uint32_t b, uint32_t ncand, bool share)
{
    if (!share || ncand <= (uint32_t)kDenseCap || b <= kDenseItem) return kDenseItem;
    const uint32_t items = (b + kDenseItem / 2) / kDenseItem;
    return (b + items - 1) / items;
}
static_assert(kDenseItem + kDenseItem / 2 <= kDenseRound, "an item is one round");
constexpr int kDenseCtasPerSm = 8;   // resident CTAs of the dense-cell kernel per SM (its launch bounds)
constexpr int kApCap = 256;           // all-pairs engine: neighbours kept per boid (more: an O(N) scan)
constexpr uint32_t kMaxBoids = 1u << 29;  // slot index packs into 29 bits
constexpr int kMaxGridAxis = 812;          // device cells per axis: 4 G^3 < 2^31

// Launchers.  Each returns the launch's cudaError_t and adds the number of
// kernels it launched to *launches.
// Packs ids [i0, i1) of an id-ordered state (slot = id); bad: the range
// check's flag (nullable); bin (nullable): also the grid keys of those slots,
// as launch_grid_keys (a single flock; count cleared beforehand).
cudaError_t launch_pack(const float *pos3, const float *vel3, float4 *pos4, float4 *vel4, uint32_t i0, uint32_t i1,
                        uint32_t *bad, float hi, const StepConst *bin, uint32_t *key, uint32_t *rank,
                        uint32_t *count, cudaStream_t s, uint64_t *launches);
// Slot order -> id order: the slot of every id into slot_of (n words of
// scratch), then ids [i0, i1) gathered into pos3/vel3 (either nullable).
cudaError_t launch_unpack_index(const float4 *pos4, uint32_t *slot_of, uint32_t n, cudaStream_t s,
                                uint64_t *launches);
cudaError_t launch_unpack_gather(const float4 *pos4, const float4 *vel4, const uint32_t *slot_of, float *pos3,
                                 float *vel3, uint32_t i0, uint32_t i1, uint32_t n, cudaStream_t s,
                                 uint64_t *launches);
// One .ptcl frame in id order: pframe gets 3 floats per boid, or 12 with
// forces (xyz + the nine get_force floats; zeros when force9 is null);
// vframe (nullable) gets vx,vy,vz.
cudaError_t launch_frame(const float4 *pos4, const float4 *vel4, const float *force9, float *pframe,
                         float *vframe, int with_forces, uint32_t n, cudaStream_t s, uint64_t *launches);
// ft == nullptr: one flock described by k; else a batched ensemble (k unused).
cudaError_t launch_grid_keys(const StepConst &k, const float4 *pos, uint32_t *key, uint32_t *rank,
                             uint32_t *count, cudaStream_t s, uint64_t *launches,
                             const FlockTable *ft = nullptr);
// Scan of the cell counts; clears the step's work counters.
cudaError_t launch_grid_scan(const StepConst &k, const DevBuffers &b, cudaStream_t s, uint64_t *launches,
                             const FlockTable *ft = nullptr);
// After the scan: the dense-cell classification (flags and work list) of
// every full-size cell.
cudaError_t launch_grid_classify(const StepConst &k, const DevBuffers &b, cudaStream_t s, uint64_t *launches,
                                 const FlockTable *ft = nullptr);
cudaError_t launch_grid_scatter(const StepConst &k, const DevBuffers &b, int from, bool zero_counts,
                                cudaStream_t s, uint64_t *launches, const FlockTable *ft = nullptr);
// Rules + integration over the sorted state b.pos[from]; writes the new state
// to b.pos[1-from], or with pos3/vel3 in id order to those (diag == false), or
// neighbour-set fingerprints (diag == true).
cudaError_t launch_grid_force(const StepConst &k, const DevBuffers &b, int from, bool diag,
                              bool record_forces, cudaStream_t s, uint64_t *launches,
                              const FlockTable *ft = nullptr, float *pos3 = nullptr, float *vel3 = nullptr);
// Whether a flock's counting sort from an id-ordered state is one kernel, and
// that kernel: pos3/vel3 sorted into b.pos[1], b.vel[1].
bool grid_bin_small(const StepConst &k, const DevBuffers &b);
cudaError_t launch_grid_bin(const StepConst &k, const DevBuffers &b, const float *pos3, const float *vel3,
                            cudaStream_t s, uint64_t *launches);
cudaError_t launch_allpairs(const StepConst &k, const DevBuffers &b, int from, bool diag,
                            bool record_forces, cudaStream_t s, uint64_t *launches);
cudaError_t launch_ref_cells(const StepConst &k, const float4 *pos, int32_t *cells8, cudaStream_t s,
                             uint64_t *launches);

// Opt the dense-cell kernels in to their shared memory on the current device
// (done before a stream capture, where it could not be).
cudaError_t grid_prepare();

// Ensemble statistics of the binned state b.pos[from] (see boids_kernels.cu):
// acc gets kStatAcc doubles per flock, com 3 per flock, largest the largest
// linked group per flock; link is the per-flock link distance; *err != 0
// after the launch means a union-find walk hit its bound.  Uses b.key and
// b.rank as scratch.
constexpr int kStatAcc = 16;
cudaError_t launch_ensemble_stats(const DevBuffers &b, int from, const FlockTable &ft, const float *link,
                                  double *acc, double *com, uint32_t *largest, uint32_t *err, cudaStream_t s,
                                  uint64_t *launches);

}  // namespace boidsgpu
