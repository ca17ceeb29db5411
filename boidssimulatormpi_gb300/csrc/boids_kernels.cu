// boids_kernels.cu -- sm_103a kernels for the per-timestep boid update.
//
// Arithmetic contract: every value the reference computes in float is
// computed here with the same IEEE operations in the same order (explicit
// __f*_rn intrinsics, and the file is built with --fmad=false).  Every
// float-vs-double comparison of the reference is replaced by the equivalent
// float comparison prepared on the host (boids_engine.h), and its two
// float-plus-double roundings by integer emulation (boids_softfp.h): the
// kernels issue no FP64 instruction.  Neighbours are accumulated in
// ascending boid id, the order of the reference's loops
// (src/boid_simulation.cpp:161, src/boid_simulation_grid.cpp:191), so the
// results are bit-identical to the reference's, not merely close.
//
// Grid step = scan of cell counts -> the scatter into cell order -> the rules.
// A flock of up to kWarpBoids boids, and a larger one while it is gathered
// (kCrowdBoids), is updated by k_grid_warp or k_grid_warp_queue, a warp per
// boid.  Else every full-size cell is classified (beside the scatter) and the
// boids are split by the occupancy of their cell:
//   k_grid_sparse  one thread per boid; candidates of the 27 cells around it
//                  are filtered, exactly tested (the warp's hits dealt to all
//                  its lanes), and kept sorted by id; boids that need more
//                  than one pass are queued, with the neighbours their list
//                  could not keep, for
//   k_grid_sparse_more, which runs their further passes in full warps beside
//   k_grid_dense   one CTA per about 32 boids of a crowded cell; the 27-cell
//                  candidates are sorted by id once in shared memory, and a
//                  warp per boid filters, tests and adds them up in id order.
// All integrate, write the new state in place of the sorted slot and bin it
// for the next step (cell key + rank from an atomic count).
#include "boids_engine.h"

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace boidsgpu {


// ------------------------------------------------------------------ exact reference arithmetic

// Vector3D::norm (src/vector3D.cpp:64-67): sqrt((x*x + y*y) + z*z).
__device__ __forceinline__ float nrm3(float x, float y, float z)
{
    return __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z)));
}

// Minimum-image coordinate of boid j seen from boid i
// (src/boid_simulation_grid.cpp:200-214): float difference compared with
// F/2 in double; the shift is (float)((double)x -+ F), reproduced exactly by
// add_f32_f64_rn without any FP64 instruction.
__device__ __forceinline__ float image1(float xj, float xi, const StepConst &k)
{
    if (__fsub_rn(xj, xi) > k.halfF_dn) return add_f32_f64_rn(xj, k.Fsd, 1);
    if (__fsub_rn(xi, xj) > k.halfF_dn) return add_f32_f64_rn(xj, k.Fsd, 0);
    return xj;
}

__device__ __forceinline__ float3 image3(float3 pj, float3 pi, const StepConst &k)
{
    return make_float3(image1(pj.x, pi.x, k), image1(pj.y, pi.y, k), image1(pj.z, pi.z, k));
}

__device__ __forceinline__ float3 xyz(float4 a) { return make_float3(a.x, a.y, a.z); }

// Per-boid constants of the sight vector: |v| exactly, and an approximate
// reciprocal for the cheap cone pre-test.
struct Sight {
    float3 v;
    float nv, inv_nv;
};

__device__ __forceinline__ Sight make_sight(float3 v)
{
    Sight s;
    s.v = v;
    s.nv = nrm3(v.x, v.y, v.z);
    s.inv_nv = __fdividef(1.0f, s.nv);
    return s;
}

// The cone tests redone with the exact cosine c = dot / (|v| * |r|)
// (correctly rounded division and square root, as the reference's floats).
// Kept out of line: it is rarely needed, and inlined the compiler would
// predicate it into every candidate test.
__device__ __noinline__ int cone_flags_exact(float dot, float nv, float d2, float lim0, float lim1, float lim2,
                                             float cs0, float cs1, float cs2, int round_mask)
{
    const float c = __fdiv_rn(dot, __fmul_rn(nv, __fsqrt_rn(d2)));
    const float lim[3] = {lim0, lim1, lim2}, cs[3] = {cs0, cs1, cs2};
    int f = 0;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const bool in_cone = ((round_mask >> r) & 1) || (c >= cs[r] && c <= 1.0f);  // NaN: false
        if (d2 < lim[r] && in_cone) f |= 1 << r;
    }
    return f;
}

// The three Boid::isInsideArea tests (src/boid.cpp:27-42) for an imaged
// target t; bit 0 cohesion, bit 1 separation, bit 2 alignment.
//
// The cone test compares c = dot / (|v| * |r|) (float, correctly rounded
// division and square root) with cstar.  An approximate cosine (hardware
// reciprocal square root, error < 1e-6) settles every case farther than
// cone_band from cstar and from 1; only the rest pay for the exact c.
__device__ __forceinline__ int pair_flags(float3 pi, const Sight &s, float3 t, const StepConst &k)
{
    const float dx = __fsub_rn(pi.x, t.x), dy = __fsub_rn(pi.y, t.y), dz = __fsub_rn(pi.z, t.z);
    // squared norm, (x*x + y*y) + z*z; relativePos = -d has the same one
    const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
    if (!(d2 < k.d2_any)) return 0;
    // v . relativePos with relativePos = t - pi = -d: round-to-nearest is
    // symmetric under negation, so the reference's ((v.x r.x + v.y r.y) +
    // v.z r.z) is exactly the negated sum over d
    const float dot =
        -__fadd_rn(__fadd_rn(__fmul_rn(s.v.x, dx), __fmul_rn(s.v.y, dy)), __fmul_rn(s.v.z, dz));
    const float ca = dot * rsqrtf(d2) * s.inv_nv;  // approximate cosine
    bool exact = !(d2 > 1e-30f) || !(fabsf(ca) < 2.0f);  // tiny distance, 0/0, overflow
    int f = 0;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const RuleConst &q = k.rule[r];
        if (!(d2 < q.d2_lim)) continue;
        if (q.all_round) { f |= 1 << r; continue; }
        if (fabsf(ca - q.cstar) < k.cone_band || fabsf(ca - 1.0f) < k.cone_band) exact = true;
        else if (ca > q.cstar && ca < 1.0f) f |= 1 << r;
    }
    if (exact) {
        f = cone_flags_exact(dot, s.nv, d2, k.rule[0].d2_lim, k.rule[1].d2_lim, k.rule[2].d2_lim,
                             k.rule[0].cstar, k.rule[1].cstar, k.rule[2].cstar,
                             k.rule[0].all_round | (k.rule[1].all_round << 1) | (k.rule[2].all_round << 2));
    }
    return f;
}

struct Acc {
    float3 coh, sep, ali;
    int ncoh, nsep, nali;
    uint64_t h[3];
};
static_assert(sizeof(Acc) == kCarryBytes, "the carry buffer holds one Acc per slot");

__device__ __forceinline__ void acc_zero(Acc &a)
{
    a.coh = a.sep = a.ali = make_float3(0.f, 0.f, 0.f);
    a.ncoh = a.nsep = a.nali = 0;
    a.h[0] = a.h[1] = a.h[2] = 0;
}

// splitmix64 finaliser: the id fingerprint of the neighbour-set diagnostics.
__device__ __forceinline__ uint64_t id_hash(uint32_t id)
{
    uint64_t z = (uint64_t)id + 0x9e3779b97f4a7c15ULL;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
}

// One accepted neighbour, in the reference's order of rules
// (src/boid_simulation_grid.cpp:219-238).
template <bool DIAG>
__device__ __forceinline__ void acc_add(Acc &a, float3 pi, float3 t, float3 vj, int f, uint32_t idj)
{
    if (f & 1) {
        a.ncoh++;
        a.coh.x = __fadd_rn(a.coh.x, t.x);
        a.coh.y = __fadd_rn(a.coh.y, t.y);
        a.coh.z = __fadd_rn(a.coh.z, t.z);
    }
    if (f & 2) {
        a.nsep++;
        const float dx = __fsub_rn(pi.x, t.x), dy = __fsub_rn(pi.y, t.y), dz = __fsub_rn(pi.z, t.z);
        const float n = nrm3(dx, dy, dz);  // Vector3D::normalized
        a.sep.x = __fadd_rn(a.sep.x, __fdiv_rn(dx, n));
        a.sep.y = __fadd_rn(a.sep.y, __fdiv_rn(dy, n));
        a.sep.z = __fadd_rn(a.sep.z, __fdiv_rn(dz, n));
    }
    if (f & 4) {
        a.nali++;
        a.ali.x = __fadd_rn(a.ali.x, vj.x);
        a.ali.y = __fadd_rn(a.ali.y, vj.y);
        a.ali.z = __fadd_rn(a.ali.z, vj.z);
    }
    if (DIAG) {
        const uint64_t h = id_hash(idj);
        if (f & 1) a.h[0] += h;
        if (f & 2) a.h[1] += h;
        if (f & 4) a.h[2] += h;
    }
}

// Rule finalisation (src/boid_simulation_grid.cpp:243-252): returns the three
// scaled rule forces, which are also get_force's values (:319-334).
__device__ __forceinline__ void acc_finish(const Acc &a, float3 pi, float3 vi, const StepConst &k,
                                           float3 &fc, float3 &fs, float3 &fa)
{
    float3 coh = a.coh, ali = a.ali;
    if (a.ncoh != 0) {
        const float q = __int2float_rn(a.ncoh);
        coh.x = __fsub_rn(__fdiv_rn(coh.x, q), pi.x);
        coh.y = __fsub_rn(__fdiv_rn(coh.y, q), pi.y);
        coh.z = __fsub_rn(__fdiv_rn(coh.z, q), pi.z);
    }
    if (a.nali != 0) {
        const float q = __int2float_rn(a.nali);
        ali.x = __fsub_rn(__fdiv_rn(ali.x, q), vi.x);
        ali.y = __fsub_rn(__fdiv_rn(ali.y, q), vi.y);
        ali.z = __fsub_rn(__fdiv_rn(ali.z, q), vi.z);
    }
    fc = make_float3(__fmul_rn(coh.x, k.cc), __fmul_rn(coh.y, k.cc), __fmul_rn(coh.z, k.cc));
    fs = make_float3(__fmul_rn(a.sep.x, k.cs), __fmul_rn(a.sep.y, k.cs), __fmul_rn(a.sep.z, k.cs));
    fa = make_float3(__fmul_rn(ali.x, k.ca), __fmul_rn(ali.y, k.ca), __fmul_rn(ali.z, k.ca));
}

// Periodic wrap (src/boid_simulation_grid.cpp:274-289): (float)(F + x) or
// (float)(x - F), both computed in double by the reference.
__device__ __forceinline__ float wrap1(float x, const StepConst &k)
{
    if (x < 0.0f) return add_f32_f64_rn(x, k.Fsd, 0);
    if (x > k.F_dn) return add_f32_f64_rn(x, k.Fsd, 1);
    return x;
}

// Integration of one boid (src/boid_simulation_grid.cpp:262-289).
__device__ __forceinline__ void integrate(float3 &x, float3 &v, float3 fc, float3 fs, float3 fa,
                                          const StepConst &k)
{
    // dv = c_coh*coh + c_sep*sep + c_ali*ali, left to right
    v.x = __fadd_rn(v.x, __fadd_rn(__fadd_rn(fc.x, fs.x), fa.x));
    v.y = __fadd_rn(v.y, __fadd_rn(__fadd_rn(fc.y, fs.y), fa.y));
    v.z = __fadd_rn(v.z, __fadd_rn(__fadd_rn(fc.z, fs.z), fa.z));
    const float n = nrm3(v.x, v.y, v.z);
    if (n > 0.0f && n > k.vmax_dn) {
        v.x = __fmul_rn(__fdiv_rn(v.x, n), k.vmax_f);
        v.y = __fmul_rn(__fdiv_rn(v.y, n), k.vmax_f);
        v.z = __fmul_rn(__fdiv_rn(v.z, n), k.vmax_f);
    } else if (n > 0.0f && n < k.vmin_up) {
        v.x = __fmul_rn(__fdiv_rn(v.x, n), k.vmin_f);
        v.y = __fmul_rn(__fdiv_rn(v.y, n), k.vmin_f);
        v.z = __fmul_rn(__fdiv_rn(v.z, n), k.vmin_f);
    }
    x.x = wrap1(__fadd_rn(x.x, v.x), k);
    x.y = wrap1(__fadd_rn(x.y, v.y), k);
    x.z = wrap1(__fadd_rn(x.z, v.z), k);
}

// ------------------------------------------------------------------ device grid

// Device cells: side R' (>= the largest radius with margin) along y and z,
// R'/4 along x.  A y/z "row" of cells is contiguous in the sorted state, and
// the quarter-width x cells let a boid scan only the x-interval a sphere of
// radius R' reaches in each neighbouring row.
__device__ __forceinline__ int cell1(float x, const StepConst &k)
{
    const int c = __float2int_rz(__fmul_rn(x, k.inv_side));
    return min(max(c, 0), k.G - 1);
}

__device__ __forceinline__ int subcell_x(float x, const StepConst &k)
{
    const int c = __float2int_rz(__fmul_rn(x, k.inv_subx));
    return min(max(c, 0), k.Gx - 1);
}

__device__ __forceinline__ uint32_t cell_key(float3 p, const StepConst &k)
{
    return (uint32_t)((cell1(p.z, k) * k.G + cell1(p.y, k)) * k.Gx + subcell_x(p.x, k));
}

__device__ __forceinline__ uint32_t cell_start(const uint32_t *__restrict__ lstart,
                                               const uint32_t *__restrict__ bsum, uint32_t c)
{
    return __ldg(lstart + c) + __ldg(bsum + c / kScanTile);
}

// First state slot of global cell c of the flock described by k.
__device__ __forceinline__ uint32_t slot_start(const uint32_t *__restrict__ lstart,
                                               const uint32_t *__restrict__ bsum, uint32_t c, const StepConst &k)
{
    return cell_start(lstart, bsum, c) + k.slot_off;
}

// The constants of the flock that owns block blk of kSlotAlign slots, copied
// into shared memory by the whole CTA (ends with a barrier).
__device__ __forceinline__ void load_flock(StepConst &dst, const FlockTable &ft, uint32_t f)
{
    static_assert(sizeof(StepConst) % 4 == 0, "StepConst is copied as words");
    const uint32_t *src = reinterpret_cast<const uint32_t *>(ft.ks + f);
    uint32_t *d = reinterpret_cast<uint32_t *>(&dst);
    for (int i = threadIdx.x; i < (int)(sizeof(StepConst) / 4); i += blockDim.x) d[i] = __ldg(src + i);
    __syncthreads();
}

// Where a rule kernel writes one boid's result.
struct GridOut {
    float4 *pos_out, *vel_out;
    float *pos3_out, *vel3_out;  // the caller's id-ordered arrays instead (null: the records above)
    uint32_t *key_out, *rank_out, *count;  // null for the all-pairs engine
    float *forces;
    int32_t *dcnt;
    uint64_t *dhash;
    Acc *carry;  // per slot: partial sums of huge cells between id windows (null: no windows)
    uint32_t *defer, *defer_cnt;  // k_grid_sparse's deferred boids: (slot, lo_id) pairs from the flock's slot_base,
                                  // and their count per flock (null: none)
    uint64_t *ovf;                // per slot, kOvfCap: a deferred boid's accepted neighbours beyond its list
    uint32_t *ovf_n;              // per slot: their number (null: not recorded)
    uint64_t *wscratch;           // k_grid_dense: wcap entries per CTA for bucketing huge cells' windows (null: none)
    uint32_t wcap;
};

template <bool DIAG>
__device__ __forceinline__ void finish_boid(const Acc &a, float4 p4, float3 vi, uint32_t s, const GridOut &o,
                                            const StepConst &k)
{
    // output row of the boid: its id, after the boids of earlier flocks
    const uint32_t id = __float_as_uint(p4.w) + (k.slot_base - k.slot_off);
    if (DIAG) {
        o.dcnt[3 * id + 0] = a.ncoh; o.dcnt[3 * id + 1] = a.nsep; o.dcnt[3 * id + 2] = a.nali;
        o.dhash[3 * id + 0] = a.h[0]; o.dhash[3 * id + 1] = a.h[1]; o.dhash[3 * id + 2] = a.h[2];
        return;
    }
    const float3 pi = xyz(p4);
    float3 fc, fs, fa;
    acc_finish(a, pi, vi, k, fc, fs, fa);
    float3 x = pi, v = vi;
    integrate(x, v, fc, fs, fa, k);
    if (o.pos3_out) {
        float *po = o.pos3_out + (size_t)3 * id, *vo = o.vel3_out + (size_t)3 * id;
        po[0] = x.x; po[1] = x.y; po[2] = x.z;
        vo[0] = v.x; vo[1] = v.y; vo[2] = v.z;
    } else {
        o.pos_out[s] = make_float4(x.x, x.y, x.z, p4.w);
        o.vel_out[s] = make_float4(v.x, v.y, v.z, 0.f);
    }
    if (o.key_out) {  // binning for the next step
        const uint32_t c = k.cell_base + cell_key(x, k);
        o.key_out[s] = c;
        o.rank_out[s] = atomicAdd(o.count + c, 1u);
    }
    if (o.forces) {
        float *f = o.forces + (size_t)9 * id;
        f[0] = fc.x; f[1] = fc.y; f[2] = fc.z;
        f[3] = fs.x; f[4] = fs.y; f[5] = fs.z;
        f[6] = fa.x; f[7] = fa.y; f[8] = fa.z;
    }
}

// ------------------------------------------------------------------ state packing

// Packs ids [i0, i1) of an id-ordered state into float4 records, slot = id
// (w of pos = id bits).  With bad != null, a coordinate outside [0, hi] (or
// NaN) sets *bad.  With key != null the boid is also binned for the grid
// (k_grid_keys' work, fused): cell_key clamps every coordinate into the
// grid, so a state that fails the range check still bins in bounds.
__global__ void k_pack(const float *__restrict__ pos3, const float *__restrict__ vel3,
                       float4 *__restrict__ pos4, float4 *__restrict__ vel4, uint32_t i0, uint32_t i1,
                       uint32_t *__restrict__ bad, float hi, uint32_t *__restrict__ key,
                       uint32_t *__restrict__ rank, uint32_t *__restrict__ count, StepConst k)
{
    const uint32_t i = i0 + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= i1) return;
    const float x = pos3[3 * (size_t)i], y = pos3[3 * (size_t)i + 1], z = pos3[3 * (size_t)i + 2];
    pos4[i] = make_float4(x, y, z, __uint_as_float(i));
    vel4[i] = make_float4(vel3[3 * (size_t)i], vel3[3 * (size_t)i + 1], vel3[3 * (size_t)i + 2], 0.f);
    if (bad && !(x >= 0.f && x <= hi && y >= 0.f && y <= hi && z >= 0.f && z <= hi)) *bad = 1u;
    if (key) {
        const uint32_t c = k.cell_base + cell_key(make_float3(x, y, z), k);
        key[i] = c;
        rank[i] = atomicAdd(count + c, 1u);
    }
}

// Slot order -> id order (the reference's getters index by id), first pass:
// the slot of every id.  A valid state holds each id in [0, n) once; other
// ids are skipped.
__global__ void k_unpack_index(const float4 *__restrict__ pos4, uint32_t *__restrict__ slot_of, uint32_t n)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const uint32_t id = __float_as_uint(__ldg(reinterpret_cast<const float *>(pos4) + 4 * (size_t)s + 3));
    if (id < n) slot_of[id] = s;
}

// Second pass, ids [i0, i1): a thread per id gathers its records, so that a
// warp's stores are contiguous (a thread per slot would scatter six 4-byte
// stores to random ids).
__global__ void k_unpack_gather(const float4 *__restrict__ pos4, const float4 *__restrict__ vel4,
                                const uint32_t *__restrict__ slot_of, float *__restrict__ pos3,
                                float *__restrict__ vel3, uint32_t i0, uint32_t i1, uint32_t n)
{
    const uint32_t i = i0 + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= i1) return;
    const uint32_t s = min(__ldg(slot_of + i), n - 1);
    if (pos3) {
        const float4 p = __ldg(pos4 + s);
        pos3[3 * (size_t)i] = p.x; pos3[3 * (size_t)i + 1] = p.y; pos3[3 * (size_t)i + 2] = p.z;
    }
    if (vel3) {
        const float4 v = __ldg(vel4 + s);
        vel3[3 * (size_t)i] = v.x; vel3[3 * (size_t)i + 1] = v.y; vel3[3 * (size_t)i + 2] = v.z;
    }
}

// One output frame in the .ptcl layout of src/main.cpp:246-277: position
// (+ get_force's nine floats) per boid, and optionally the velocity, both in
// id order.  A thread per state slot; the scattered stores land in L2.
__global__ void k_frame(const float4 *__restrict__ pos4, const float4 *__restrict__ vel4,
                        const float *__restrict__ force9, float *__restrict__ pframe,
                        float *__restrict__ vframe, int with_forces, uint32_t n)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const float4 p = pos4[s];
    const uint32_t id = __float_as_uint(p.w);
    const size_t stride = with_forces ? 12 : 3;
    float *o = pframe + stride * id;
    o[0] = p.x; o[1] = p.y; o[2] = p.z;
    if (with_forces) {
        const float *f = force9 ? force9 + (size_t)9 * id : nullptr;
#pragma unroll
        for (int c = 0; c < 9; ++c) o[3 + c] = f ? f[c] : 0.0f;
    }
    if (vframe) {
        const float4 v = vel4[s];
        vframe[(size_t)3 * id] = v.x; vframe[(size_t)3 * id + 1] = v.y; vframe[(size_t)3 * id + 2] = v.z;
    }
}

// ------------------------------------------------------------------ counting-sort binning

// Programmatic dependent launch, in the chains of a small flock's steps: the
// next kernel's CTAs are set up while this one's last ones run, and wait here
// for its end (and its writes) before they touch anything.  A kernel launched
// without the attribute passes straight through.  (The next kernel is let in
// after this one's own wait: letting it in before took 1 to 5 % longer from
// 1000 to 5000 boids.)
__device__ __forceinline__ void chain_wait()
{
    asm volatile("griddepcontrol.wait;\ngriddepcontrol.launch_dependents;" ::: "memory");
}

// The measure that sends a step's boids to a warp each or to the cells' split:
// the pairs of boids that share an x cell, counted by k_grid_scan.  It lives on
// the device, so a captured step follows the flock as it gathers.
struct Crowd {
    uint32_t *pairs;  // null: the route was chosen on the host
    uint32_t min;     // a warp per boid: from this many pairs
    uint32_t span;    // to min + span - 1
};
__device__ __forceinline__ bool crowded(const Crowd &c) { return c.pairs && __ldcg(c.pairs) - c.min < c.span; }
// The most boids of a cell that count: their pairs cannot overflow a word in
// flocks of up to 2^19 boids.
constexpr uint32_t kCrowdCap = 4096;

template <bool MULTI>
__global__ void k_grid_keys(const float4 *__restrict__ pos, uint32_t *__restrict__ key,
                            uint32_t *__restrict__ rank, uint32_t *__restrict__ count, StepConst kp, FlockTable ft)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= (MULTI ? ft.nslots : kp.n)) return;
    const StepConst &k = MULTI ? ft.ks[ft.blk_flock[s / kSlotAlign]] : kp;
    if (s - k.slot_base >= k.n) return;  // padding between flocks
    const uint32_t c = k.cell_base + cell_key(xyz(pos[s]), k);
    key[s] = c;
    rank[s] = atomicAdd(count + c, 1u);
}

// Exclusive scan of the per-cell counts.  Each block scans one tile of
// kScanTile cells into lstart and publishes its total; the last block to
// finish (completion ticket, no waiting) turns the totals into tile offsets
// in bsum.  start(c) = lstart[c] + bsum[c / kScanTile].
constexpr int kScanThreads = 256;
constexpr int kScanItems = kScanTile / kScanThreads;  // 8

template <int NT>
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t *warp_tot, uint32_t &total)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[w] = x;
    __syncthreads();
    if (w == 0) {
        uint32_t t = lane < NT / 32 ? warp_tot[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        if (lane < NT / 32) warp_tot[lane] = t;  // inclusive warp totals
    }
    __syncthreads();
    total = warp_tot[NT / 32 - 1];
    const uint32_t before = (w > 0 ? warp_tot[w - 1] : 0) + x - v;
    __syncthreads();  // warp_tot is reused by the next call
    return before;
}

__global__ void __launch_bounds__(kScanThreads)
k_grid_scan(const uint32_t *__restrict__ count, uint32_t *__restrict__ lstart, uint32_t *bsum,
            uint32_t *ticket, uint32_t nblocks, uint32_t *__restrict__ work, int measure)
{
    __shared__ uint32_t warp_tot[kScanThreads / 32], block_pairs;
    __shared__ bool is_last;
    if (threadIdx.x == 0) block_pairs = 0;
    chain_wait();
    const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    const uint4 a = *reinterpret_cast<const uint4 *>(count + base);
    const uint4 b = *reinterpret_cast<const uint4 *>(count + base + 4);
    const uint32_t v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t sum = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) sum += v[i];
    uint32_t total;
    uint32_t run = block_excl_scan<kScanThreads>(sum, warp_tot, total);
    uint32_t o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) { o[i] = run; run += v[i]; }
    *reinterpret_cast<uint4 *>(lstart + base) = make_uint4(o[0], o[1], o[2], o[3]);
    *reinterpret_cast<uint4 *>(lstart + base + 4) = make_uint4(o[4], o[5], o[6], o[7]);
    if (measure) {
        uint32_t pairs = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t c = min(v[i], kCrowdCap);
            if (c > 1) pairs += c * (c - 1) / 2;
        }
        pairs = __reduce_add_sync(0xffffffffu, pairs);
        if ((threadIdx.x & 31) == 0 && pairs) atomicAdd(&block_pairs, pairs);
        __syncthreads();  // every warp's pairs before the block's ticket
    }
    if (threadIdx.x == 0) {
        if (measure && block_pairs) atomicAdd(ticket + 1, block_pairs);
        bsum[blockIdx.x] = total;
        __threadfence();
        is_last = atomicAdd(ticket, 1u) == nblocks - 1;
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    uint32_t carry = 0;
    for (uint32_t c0 = 0; c0 < nblocks; c0 += kScanThreads) {
        const uint32_t i = c0 + threadIdx.x;
        const uint32_t t = i < nblocks ? __ldcg(bsum + i) : 0u;
        uint32_t chunk;
        const uint32_t ex = block_excl_scan<kScanThreads>(t, warp_tot, chunk);
        if (i < nblocks) bsum[i] = carry + ex;
        carry += chunk;
    }
    if (threadIdx.x == 0) {
        *ticket = 0;  // ready for the next launch
        if (work) {   // this step's work counters
            work[0] = work[1] = work[2] = 0;
            if (measure) work[3] = atomicExch(ticket + 1, 0u);
        }
    }
}

template <bool MULTI>
__global__ void k_grid_scatter(const float4 *__restrict__ pin, const float4 *__restrict__ vin,
                               const uint32_t *__restrict__ key, const uint32_t *rank,
                               const uint32_t *__restrict__ lstart, const uint32_t *__restrict__ bsum,
                               float4 *__restrict__ pout, float4 *__restrict__ vout,
                               uint32_t *__restrict__ count_to_zero, uint32_t *slot_of, Crowd crowd,
                               uint32_t n, FlockTable ft)
{
    chain_wait();
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t off = 0, first = 0;  // the flock's padding and first slot
    if (MULTI) {
        if (s >= ft.nslots) return;
        const StepConst &k = ft.ks[ft.blk_flock[s / kSlotAlign]];
        if (s - k.slot_base >= k.n) return;
        off = k.slot_off;
        first = k.slot_base;
    } else if (s >= n) {
        return;
    }
    const uint32_t c = key[s];
    const bool table = slot_of && (!crowd.pairs || crowded(crowd));
    const uint32_t d = cell_start(lstart, bsum, c) + rank[s] + off;
    const float4 p = pin[s];
    pout[d] = p;
    vout[d] = vin[s];
    if (table) slot_of[first + __float_as_uint(p.w)] = d;
    if (count_to_zero) count_to_zero[c] = 0;  // every binned cell, for the next step's keys
}

// Scan and scatter of a flock of at most kSortBoids boids and kSortCells cells
// in one CTA: the boids' records are loaded beside the counts, and the scanned
// starts are read back from shared memory.  The starts in lstart are final
// (bsum is zero).  Bound by one load, one block scan and one store, where
// k_grid_scan and k_grid_scatter are six dependent trips to L2 and a launch: a
// step of 1000 boids of test.ini 20.9 us, 22.7 with those, of 100 boids 13.2
// (15.9), of 1024 of marun2019.ini 15.9 (17.4).  With two boids a thread and
// twice the cells 2048 boids gained nothing, with four 4096 lost 20 %.
constexpr int kSortThreads = kSortBoids;
static_assert(kSortCells == 4 * kSortThreads, "a thread takes one boid and one vector of counts");

__global__ void __launch_bounds__(kSortThreads)
k_grid_sort(const float4 *__restrict__ pin, const float4 *__restrict__ vin, const uint32_t *__restrict__ key,
            const uint32_t *__restrict__ rank, uint32_t *count, uint32_t *__restrict__ lstart,
            uint32_t *__restrict__ bsum, uint32_t ncell_pad, uint32_t tiles, float4 *__restrict__ pout,
            float4 *__restrict__ vout, int zero_counts, uint32_t *__restrict__ slot_of, uint32_t n)
{
    __shared__ uint32_t warp_tot[kSortThreads / 32];
    __shared__ __align__(16) uint32_t start[kSortCells];
    const uint32_t t = threadIdx.x, c0 = 4 * t;
    chain_wait();
    uint4 a = make_uint4(0, 0, 0, 0);
    if (c0 < ncell_pad) a = *reinterpret_cast<const uint4 *>(count + c0);
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f), v = p;
    uint32_t c = 0, r = 0, total;
    if (t < n) {
        c = key[t];
        r = rank[t];
        p = pin[t];
        v = vin[t];
    }
    const uint32_t run = block_excl_scan<kSortThreads>(a.x + a.y + a.z + a.w, warp_tot, total);
    if (c0 < ncell_pad) {
        const uint4 x = make_uint4(run, run + a.x, run + a.x + a.y, run + a.x + a.y + a.z);
        *reinterpret_cast<uint4 *>(start + c0) = x;
        *reinterpret_cast<uint4 *>(lstart + c0) = x;
        if (zero_counts) *reinterpret_cast<uint4 *>(count + c0) = make_uint4(0, 0, 0, 0);  // for the next step's keys
    }
    if (t < tiles) bsum[t] = 0;
    __syncthreads();
    if (t >= n) return;
    const uint32_t d = start[c] + r;
    pout[d] = p;
    vout[d] = v;
    slot_of[__float_as_uint(p.w)] = d;
}

// The allocation-free step's counting sort of as small a flock, from the
// caller's id-ordered arrays: the counts and ranks never leave shared memory
// (a step of 1000 boids of test.ini 24 us, 31.5 with k_grid_bin).
__global__ void __launch_bounds__(kSortThreads)
k_grid_bin_one(const float *__restrict__ pos3, const float *__restrict__ vel3, uint32_t *__restrict__ lstart,
               uint32_t *__restrict__ bsum, uint32_t ncell_pad, uint32_t tiles, float4 *__restrict__ pout,
               float4 *__restrict__ vout, uint32_t *__restrict__ slot_of, StepConst k)
{
    __shared__ uint32_t warp_tot[kSortThreads / 32];
    __shared__ __align__(16) uint32_t start[kSortCells];  // the counts, then the starts
    const uint32_t t = threadIdx.x, c0 = 4 * t;
    chain_wait();
    uint4 &mine = *reinterpret_cast<uint4 *>(start + c0);
    mine = make_uint4(0, 0, 0, 0);
    float3 p = make_float3(0.f, 0.f, 0.f), v = p;
    uint32_t c = 0, r = 0, total;
    if (t < k.n) {
        p = make_float3(pos3[3 * t], pos3[3 * t + 1], pos3[3 * t + 2]);
        v = make_float3(vel3[3 * t], vel3[3 * t + 1], vel3[3 * t + 2]);
        c = cell_key(p, k);
    }
    __syncthreads();
    if (t < k.n) r = atomicAdd(start + c, 1u);
    __syncthreads();
    const uint4 a = mine;
    const uint32_t run = block_excl_scan<kSortThreads>(a.x + a.y + a.z + a.w, warp_tot, total);
    const uint4 x = make_uint4(run, run + a.x, run + a.x + a.y, run + a.x + a.y + a.z);
    mine = x;
    if (c0 < ncell_pad) *reinterpret_cast<uint4 *>(lstart + c0) = x;
    if (t < tiles) bsum[t] = 0;
    __syncthreads();
    if (t >= k.n) return;
    const uint32_t d = start[c] + r;
    pout[d] = make_float4(p.x, p.y, p.z, __uint_as_float(t));
    vout[d] = make_float4(v.x, v.y, v.z, 0.f);
    slot_of[t] = d;
}

// The allocation-free step's counting sort of a small flock in one kernel,
// from the caller's id-ordered arrays: a cluster of kBinCtas CTAs clears the
// counts, keys and counts the boids, scans the counts (a contiguous part each,
// the parts' totals exchanged through distributed shared memory) and scatters
// the boids.  The cell starts in lstart are final (bsum is zero).
//
// Bound by the chain of its phases (about 10 us), which replaces a clear and
// three kernels: the step of 16 384 gathered boids takes 59 us where it took
// 75 with those and an unpacking after the rules.  It pays only from unsorted input: without the first phases it takes
// as long as k_grid_scan and k_grid_scatter (a handle's step of 1000 boids
// 29.3 against 28.0 us, of 16 384 57 against 55).
constexpr int kBinCtas = 8, kBinThreads = 1024;

__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__global__ void __cluster_dims__(kBinCtas, 1, 1) __launch_bounds__(kBinThreads)
k_grid_bin(const float *__restrict__ pos3, const float *__restrict__ vel3, uint32_t *key, uint32_t *rank,
           uint32_t *count, uint32_t *lstart, uint32_t *__restrict__ bsum, uint32_t ncell_pad, uint32_t tiles,
           float4 *__restrict__ pout, float4 *__restrict__ vout, uint32_t *slot_of, StepConst k)
{
    __shared__ uint32_t warp_tot[kBinThreads / 32], totals[kBinCtas];
    const uint32_t cta = blockIdx.x, t = threadIdx.x, at = cta * kBinThreads + t;
    chain_wait();
    constexpr uint32_t kAll = kBinCtas * kBinThreads;
    for (uint32_t c = 4 * at; c < ncell_pad; c += 4 * kAll)
        *reinterpret_cast<uint4 *>(count + c) = make_uint4(0, 0, 0, 0);
    cluster_sync();
    for (uint32_t i = at; i < k.n; i += kAll) {
        const uint32_t c = cell_key(make_float3(pos3[3 * i], pos3[3 * i + 1], pos3[3 * i + 2]), k);
        key[i] = c;
        rank[i] = atomicAdd(count + c, 1u);
    }
    cluster_sync();
    // this thread's cells, in groups of four: a contiguous part of the CTA's
    const uint32_t groups = ncell_pad / 4, per = (groups + kAll - 1) / kAll;
    const uint32_t g0 = min(groups, at * per), g1 = min(groups, g0 + per);
    uint32_t sum = 0;
    for (uint32_t g = g0; g < g1; ++g) {
        const uint4 v = __ldcg(reinterpret_cast<const uint4 *>(count) + g);
        sum += v.x + v.y + v.z + v.w;
    }
    uint32_t total;
    uint32_t run = block_excl_scan<kBinThreads>(sum, warp_tot, total);
    if (t < kBinCtas) {  // the CTA's total to every CTA of the cluster
        const uint32_t mine = (uint32_t)__cvta_generic_to_shared(totals + cta);
        uint32_t there;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(mine), "r"(t));
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(there), "r"(total) : "memory");
    }
    for (uint32_t b = at; b < tiles; b += kAll) bsum[b] = 0;
    cluster_sync();
    for (uint32_t c = 0; c < cta; ++c) run += totals[c];
    for (uint32_t g = g0; g < g1; ++g) {
        const uint4 v = __ldcg(reinterpret_cast<const uint4 *>(count) + g);
        reinterpret_cast<uint4 *>(lstart)[g] = make_uint4(run, run + v.x, run + v.x + v.y, run + v.x + v.y + v.z);
        run += v.x + v.y + v.z + v.w;
    }
    cluster_sync();
    for (uint32_t i = at; i < k.n; i += kAll) {
        const uint32_t d = __ldcg(lstart + __ldcg(key + i)) + __ldcg(rank + i);
        pout[d] = make_float4(pos3[3 * i], pos3[3 * i + 1], pos3[3 * i + 2], __uint_as_float(i));
        vout[d] = make_float4(vel3[3 * i], vel3[3 * i + 1], vel3[3 * i + 2], 0.f);
        slot_of[i] = d;  // (may be rank[i])
    }
}

// ------------------------------------------------------------------ neighbourhood segments

// The 27 cells around (cx, cy, cz) form 9 rows of 3 cells along x; a row is
// one run of consecutive cell indices, or two where x wraps.  Segment q of
// a boid (0 <= q < 9 * runs) is run q % runs of row q / runs.  (sx, sy, sz)
// moves a boid of the segment next to the centre cell across the periodic
// faces (approximately, for the filters only).
struct Seg {
    uint32_t c0, c1;  // cells [c0, c1)
    float sx, sy, sz;
};

__device__ __forceinline__ int seg_runs(int cx, const StepConst &k) { return (cx == 0 || cx == k.G - 1) ? 2 : 1; }

// Segment q of the 27 full-size cells around full-size cell (cx, cy, cz),
// in x-cell indices (4 per full-size cell).
__device__ __forceinline__ Seg segment(int cx, int cy, int cz, int q, int runs, const StepConst &k)
{
    const int G = k.G, Gx = k.Gx;
    const int row = q / runs, run = q - row * runs;
    int z = cz + row / 3 - 1, y = cy + row % 3 - 1;
    float sz = 0.f, sy = 0.f;
    if (z < 0) { z += G; sz = -k.Ff; } else if (z >= G) { z -= G; sz = k.Ff; }
    if (y < 0) { y += G; sy = -k.Ff; } else if (y >= G) { y -= G; sy = k.Ff; }
    const uint32_t r0 = (uint32_t)(z * G + y) * (uint32_t)Gx;
    const int x0 = 4 * cx;
    if (runs == 1) return Seg{r0 + x0 - 4, r0 + x0 + 8, 0.f, sy, sz};
    if (cx == 0) return run == 0 ? Seg{r0 + Gx - 4, r0 + Gx, -k.Ff, sy, sz} : Seg{r0, r0 + 8, 0.f, sy, sz};
    return run == 0 ? Seg{r0 + Gx - 8, r0 + Gx, 0.f, sy, sz} : Seg{r0, r0 + 4, k.Ff, sy, sz};
}

// Which kernel takes the boids of a full-size cell: k_grid_dense when the
// cell is crowded (dense_min boids or more), or holds defer_min or more with
// over cand_defer candidates in its 27 cells, or holds any boid with over
// lone_cand candidates (sorting a crowded neighbourhood once per cell beats
// sorting it per boid); else k_grid_sparse.  Cells with more than kDenseCap
// candidates need the dense kernel's id windows (windows != 0).
__device__ __forceinline__ bool dense_rule(uint32_t b, uint32_t ncand, const StepConst &k, int windows)
{
    const bool want = b >= k.dense_min || (b >= k.defer_min && ncand > k.cand_defer) || ncand > k.lone_cand;
    return b > 0 && want && (ncand <= (uint32_t)kDenseCap || windows);
}

// Per full-size cell, after the scan (from the cell starts alone, so that it
// can run beside the scatter): the dense flag the thread-per-boid kernel
// reads, and the dense kernel's work list.
template <bool MULTI>
__global__ void k_grid_classify(const uint32_t *__restrict__ lstart,
                                const uint32_t *__restrict__ bsum, uint8_t *__restrict__ dflag,
                                uint32_t *__restrict__ dense_list, uint32_t *__restrict__ dense_n, uint32_t nfull,
                                int windows, bool share, Crowd crowd, StepConst kp, FlockTable ft)
{
    chain_wait();
    const uint32_t cg = blockIdx.x * blockDim.x + threadIdx.x;
    if (cg >= nfull) return;
    if (crowded(crowd)) {  // no items, and no boids for k_grid_sparse
        dflag[cg] = 1;
        return;
    }
    // boids of the cell from the scan (the counts may be zeroed meanwhile by
    // the scatter, which runs beside this kernel)
    const uint32_t b = cell_start(lstart, bsum, 4 * cg + 4) - cell_start(lstart, bsum, 4 * cg);
    uint8_t flag = 0;
    if (b > 0) {
        uint32_t f = 0;
        if (MULTI) {  // the flock: last with cell4 <= cg
            uint32_t hi = ft.count;
            while (hi - f > 1) {
                const uint32_t mid = (f + hi) / 2;
                if (__ldg(ft.cell4 + mid) <= cg) f = mid; else hi = mid;
            }
        }
        const StepConst &k = MULTI ? ft.ks[f] : kp;
        const uint32_t c = cg - k.cell_base / 4;
        const int G = k.G;
        const int cx = (int)(c % G), cy = (int)((c / G) % G), cz = (int)(c / ((uint32_t)G * G));
        const int runs = seg_runs(cx, k);
        uint32_t ncand = 0;
        for (int q = 0; q < 9 * runs; ++q) {
            const Seg sg = segment(cx, cy, cz, q, runs, k);
            ncand += cell_start(lstart, bsum, k.cell_base + sg.c1) - cell_start(lstart, bsum, k.cell_base + sg.c0);
        }
        if (dense_rule(b, ncand, k, windows)) {
            flag = 1;
            const uint32_t per = dense_per_item(b, ncand, share), items = (b + per - 1) / per;
            const uint32_t at = atomicAdd(dense_n, items);
            for (uint32_t r = 0; r < items; ++r) {
                dense_list[2 * (at + r)] = cg;
                dense_list[2 * (at + r) + 1] = r * per;
            }
        }
    }
    dflag[cg] = flag;
}

// ------------------------------------------------------------------ sparse cells: thread per boid

// One thread per boid (slot).  In each of the 9 neighbouring y/z rows the
// boid scans only the x cells a sphere of radius sqrt(trim_r2) around it
// reaches, and drops rows it cannot reach.
//
// All lanes of a warp walk their own candidates in lock-step (a flat loop of
// max-over-warp length).  Candidates passing the squared-distance filter are
// buffered, and whenever one buffer is nearly full the warp runs the exact
// tests of all its lanes' hits, dealt to its lanes 32 at a time whichever
// lane found them, so the expensive test runs with nearly every lane busy.  The
// filter drops candidates behind the boid (the view-cone pre-test,
// StepConst::dot_eps).  Accepted neighbours are kept sorted by id,
// at most kListA per pass; a boid with more takes further passes, each
// keeping the next kListA ids, so accumulation is always in ascending id --
// for a single flock in k_grid_sparse_more, so that those passes run in full
// warps.  The per-boid tables (segments, hit buffer, sorted list) live in
// shared memory, one column per thread: as local memory they overflow L1 and
// every access goes to L2.
constexpr int kBufA = 16;     // (13: 172 us a step of 262 143 boids for 167; 18 and more: 23 warps on an SM)
constexpr int kListA = kListCap;
constexpr int kRT = 128;      // threads of k_grid_sparse_more
constexpr int kSegA = 18;     // at most 9 rows x 2 runs (a run split where x wraps)
// Candidates loaded together in the filter loop: 3 keeps the kernel within
// 80 registers; with 2 a step was 1-2 % slower, with 4 (96 registers) 4 %.
constexpr int kCandStep = 3;
static_assert(kBufA > kCandStep, "the hit buffer holds an iteration's hits");

struct GridIn {
    const float4 *__restrict__ pos;
    const float4 *__restrict__ vel;
    const uint32_t *__restrict__ lstart;
    const uint32_t *__restrict__ bsum;
    const uint8_t *__restrict__ dflag;  // per full-size cell: taken by k_grid_dense
    const uint32_t *__restrict__ slot_of;  // k_grid_warp: slot of each id, from its flock's slot_base
    Crowd crowd;
    int chain;  // k_grid_sparse and k_grid_dense were launched in a chain
    bool share;  // dense_per_item
};

struct SparseSmem {              // of one warp, a column per lane
    uint32_t seg0[kSegA][32];    // first slot | x shift << 29 | (z shift < 0) << 31
    uint32_t seg1[kSegA][32];    // end slot   | y shift << 29 | (z shift > 0) << 31
    uint16_t buf[kBufA][32];     // filter hits: offset in the segment | segment << 8 | rules << 13
    uint64_t lst[kListA][32];    // accepted neighbours, sorted: id << 32 | slot | flags << 29
};

// The segments of the boid at pi, whose full-size cell is (cy, cz) along y
// and z, into the lane's columns of sm.seg0/seg1: in each neighbour row,
// the x cells that a sphere of radius sqrt(trim_r2) around it reaches.
// Empty runs are not stored.  Returns the number of candidates.
__device__ __forceinline__ uint32_t sparse_segments(SparseSmem &sm, int t, float3 pi, int cy, int cz,
                                                    const GridIn &g, const StepConst &k)
{
    const int G = k.G, Gx = k.Gx;
    const float eps = k.side * 1e-5f;
    int nseg = 0;
    uint32_t ncand = 0;
#pragma unroll
    for (int r = 0; r < 9; ++r) {
        const int dz = r / 3 - 1, dy = r % 3 - 1;
        const float ddy = dy == 0 ? 0.f : fmaxf(0.f, dy < 0 ? pi.y - (float)cy * k.side - eps
                                                          : (float)(cy + 1) * k.side - pi.y - eps);
        const float ddz = dz == 0 ? 0.f : fmaxf(0.f, dz < 0 ? pi.z - (float)cz * k.side - eps
                                                          : (float)(cz + 1) * k.side - pi.z - eps);
        const float rem = k.trim_r2 - ddy * ddy - ddz * ddz;
        if (!(rem > 0.f)) continue;
        const float rx = sqrtf(rem);
        // a boid in the field reaches at most one row length beyond either
        // end; the clamp only keeps a state outside the field (never made
        // by the update, refused by boids_set_state) within the cell tables
        const int lo = max(__float2int_rd((pi.x - rx) * k.inv_subx), 1 - Gx);
        const int hi = min(__float2int_rd((pi.x + rx) * k.inv_subx), 2 * Gx - 2);
        int a0 = lo, a1 = hi + 1, c0 = 0, c1 = 0;  // x-cell runs [a0, a1) and [c0, c1)
        uint32_t ca = 0, cb = 0;  // x shifts of the runs, 2-bit two's complement: 3 = -F, 1 = +F
        if (lo < 0) { a0 = lo + Gx; a1 = Gx; ca = 3; c1 = min(hi + 1, Gx); }
        else if (hi >= Gx) { a1 = Gx; c1 = hi + 1 - Gx; cb = 1; }
        int zz = cz + dz, yy = cy + dy;
        zz = zz < 0 ? zz + G : (zz >= G ? zz - G : zz);
        yy = yy < 0 ? yy + G : (yy >= G ? yy - G : yy);
        const uint32_t rb = k.cell_base + (uint32_t)(zz * G + yy) * (uint32_t)Gx;
        // y and z shifts of the row, as the x shifts
        const uint32_t ysh = cy + dy < 0 ? 3u : (cy + dy >= G ? 1u : 0u);
        const uint32_t w0 = cz + dz < 0 ? 0x80000000u : 0u, w1 = (ysh << 29) | (cz + dz >= G ? 0x80000000u : 0u);
        if (a1 > a0) {
            const uint32_t j0 = slot_start(g.lstart, g.bsum, rb + a0, k), j1 = slot_start(g.lstart, g.bsum, rb + a1, k);
            if (j1 > j0) {
                sm.seg0[nseg][t] = j0 | (ca << 29) | w0;
                sm.seg1[nseg][t] = j1 | w1;
                ncand += j1 - j0;
                ++nseg;
            }
        }
        if (c1 > c0) {
            const uint32_t j0 = slot_start(g.lstart, g.bsum, rb + c0, k), j1 = slot_start(g.lstart, g.bsum, rb + c1, k);
            if (j1 > j0) {
                sm.seg0[nseg][t] = j0 | (cb << 29) | w0;
                sm.seg1[nseg][t] = j1 | w1;
                ncand += j1 - j0;
                ++nseg;
            }
        }
    }
    return ncand;
}

// The same segments with the loads of all rows in flight together, for
// k_grid_sparse_more, whose boids reach nearly every row and whose warps are
// few: a step of 2^20 boids 25 updates after a uniform start 766 -> 737 us, 100
// after 1790 -> 1703, 400 after 2224 -> 2180.  (In k_grid_sparse it was 3 %
// slower on a uniform flock, which skips a fifth of the corner rows.)
__device__ __forceinline__ uint32_t sparse_segments_ahead(SparseSmem &sm, int t, float3 pi, int cy, int cz,
                                                    const GridIn &g, const StepConst &k)
{
    const int G = k.G, Gx = k.Gx;
    const float eps = k.side * 1e-5f;
    auto row_base = [&](int r) {  // first cell of the row
        int zz = cz + r / 3 - 1, yy = cy + r % 3 - 1;
        zz = zz < 0 ? zz + G : (zz >= G ? zz - G : zz);
        yy = yy < 0 ? yy + G : (yy >= G ? yy - G : yy);
        return k.cell_base + (uint32_t)(zz * G + yy) * (uint32_t)Gx;
    };
    auto reach = [&](int r, int &lo, int &hi) {  // the x cells [lo, hi] of the row (false: none)
        const int dz = r / 3 - 1, dy = r % 3 - 1;
        const float ddy = dy == 0 ? 0.f : fmaxf(0.f, dy < 0 ? pi.y - (float)cy * k.side - eps
                                                          : (float)(cy + 1) * k.side - pi.y - eps);
        const float ddz = dz == 0 ? 0.f : fmaxf(0.f, dz < 0 ? pi.z - (float)cz * k.side - eps
                                                          : (float)(cz + 1) * k.side - pi.z - eps);
        const float rem = k.trim_r2 - ddy * ddy - ddz * ddz;
        const float rx = rem > 0.f ? sqrtf(rem) : 0.f;
        // a boid in the field reaches at most one row length beyond either
        // end; the clamp only keeps a state outside the field (never made
        // by the update, refused by boids_set_state) within the cell tables
        lo = max(__float2int_rd((pi.x - rx) * k.inv_subx), 1 - Gx);
        hi = min(__float2int_rd((pi.x + rx) * k.inv_subx), 2 * Gx - 2);
        return rem > 0.f;
    };
    // the slots of every row's first run (up to the end of the row): all loads
    // are issued before the first is used
    uint32_t j0[9], j1[9], wrapped = 0;  // bit 2 r: the run begins before the row, 2 r + 1: it ends behind it
#pragma unroll
    for (int r = 0; r < 9; ++r) {
        int lo, hi;
        const bool in = reach(r, lo, hi);
        const int a0 = min(lo < 0 ? lo + Gx : lo, Gx);
        const int a1 = !in ? a0 : (lo < 0 ? Gx : max(a0, min(hi + 1, Gx)));
        const uint32_t rb = row_base(r);
        j0[r] = slot_start(g.lstart, g.bsum, rb + a0, k);
        j1[r] = slot_start(g.lstart, g.bsum, rb + a1, k);
        if (in && lo < 0) wrapped |= 1u << (2 * r);
        else if (in && hi >= Gx) wrapped |= 2u << (2 * r);
    }
    int nseg = 0;
    uint32_t ncand = 0;
#pragma unroll
    for (int r = 0; r < 9; ++r) {
        // shifts, 2-bit two's complement (3 = -F, 1 = +F): x of the first run, y; z
        const int dz = r / 3 - 1, dy = r % 3 - 1;
        const uint32_t ysh = cy + dy < 0 ? 3u : (cy + dy >= G ? 1u : 0u);
        const uint32_t w0 = cz + dz < 0 ? 0x80000000u : 0u, w1 = (ysh << 29) | (cz + dz >= G ? 0x80000000u : 0u);
        if (j1[r] > j0[r]) {
            sm.seg0[nseg][t] = j0[r] | ((wrapped >> (2 * r)) & 1u ? 3u << 29 : 0u) | w0;
            sm.seg1[nseg][t] = j1[r] | w1;
            ncand += j1[r] - j0[r];
            ++nseg;
        }
        if ((wrapped >> (2 * r)) & 3u) {  // the run's other part, across the periodic face
            int lo, hi;
            reach(r, lo, hi);
            const int c1 = lo < 0 ? min(hi + 1, Gx) : hi + 1 - Gx;
            if (c1 > 0) {
                const uint32_t rb = row_base(r);
                const uint32_t k0 = slot_start(g.lstart, g.bsum, rb, k), k1 = slot_start(g.lstart, g.bsum, rb + c1, k);
                if (k1 > k0) {
                    sm.seg0[nseg][t] = k0 | (lo < 0 ? 0u : 1u << 29) | w0;
                    sm.seg1[nseg][t] = k1 | w1;
                    ncand += k1 - k0;
                    ++nseg;
                }
            }
        }
    }
    return ncand;
}

// The m neighbours of the lane's column of sm.lst (sorted by id) added to
// a in that order, each entry's loads issued one entry ahead.
template <bool DIAG>
__device__ __forceinline__ void list_accumulate(const SparseSmem &sm, int t, int m, float3 pi, Acc &a,
                                                const GridIn &g, const StepConst &k)
{
    uint64_t e_next = m > 0 ? sm.lst[0][t] : 0;
    float4 p_next = make_float4(0.f, 0.f, 0.f, 0.f), v_next = p_next;
    if (m > 0) {
        p_next = __ldg(g.pos + ((uint32_t)e_next & 0x1fffffffu));
        v_next = __ldg(g.vel + ((uint32_t)e_next & 0x1fffffffu));
    }
    for (int q = 0; q < m; ++q) {
        const uint64_t e = e_next;
        const float4 pj = p_next, vv = v_next;
        if (q + 1 < m) {
            e_next = sm.lst[q + 1][t];
            p_next = __ldg(g.pos + ((uint32_t)e_next & 0x1fffffffu));
            v_next = __ldg(g.vel + ((uint32_t)e_next & 0x1fffffffu));
        }
        const int f = (int)(((uint32_t)e) >> 29);
        const float3 tt = image3(xyz(pj), pi, k);
        const float3 vj = (f & 4) ? xyz(vv) : make_float3(0.f, 0.f, 0.f);
        acc_add<DIAG>(a, pi, tt, vj, f, (uint32_t)(e >> 32));
    }
}

// One pass of a warp (all lanes call it together) over the candidates of its
// lanes that still need one: the filter, the exact tests of the buffered
// hits, and the accepted neighbours with ids above lo_id kept sorted in the
// lane's column of sm.lst, at most kListA.  Those lanes then accumulate
// their list; a lane that accepted more than the list held keeps need and
// moves lo_id up to the last id it accumulated.  With ovf (this lane's row),
// every accepted neighbour that leaves the list or never enters it is
// appended there, up to kOvfCap of them, and counted in ovf_n.
template <bool DIAG>
__device__ __forceinline__ void sparse_pass(SparseSmem &sm, int t, uint32_t s, float3 pi, const Sight &sight,
                                            float dot_lim, uint32_t nc, bool &need, int64_t &lo_id, Acc &a,
                                            const GridIn &g, const StepConst &k, uint64_t *ovf, uint32_t &ovf_n,
                                            bool &moved)
{
    const float3 vi = sight.v;
    const uint32_t mine = need ? nc : 0;
    const uint32_t max_nc = __reduce_max_sync(0xffffffffu, mine);
    int m = 0, nb = 0;
    uint32_t more = 0;  // accepted neighbours with id > lo_id in this pass
    int qs = -1;
    uint32_t j = 0, jend = 0;  // global slots [j, jend) of the current segment
    moved = false;
    uint32_t tag = 0;          // the segment << 8, plus the offset of slot j in it
    float qx = 0.f, qy = 0.f, qz = 0.f;
    // the next segment (none is empty): its slots and the query point
    auto advance = [&]() {
        ++qs;
        const uint32_t w0 = sm.seg0[qs][t], w1 = sm.seg1[qs][t];
        j = w0 & 0x1fffffffu;
        jend = w1 & 0x1fffffffu;
        // the candidate's image is pj + shift: test pj against pi - shift
        const int vx = (int)(w0 << 1) >> 30, vy = (int)(w1 << 1) >> 30;
        const int vz = (int)(w1 >> 31) - (int)(w0 >> 31);
        qx = __fmaf_rn(-__int2float_rn(vx), k.Ff, pi.x);
        qy = __fmaf_rn(-__int2float_rn(vy), k.Ff, pi.y);
        qz = __fmaf_rn(-__int2float_rn(vz), k.Ff, pi.z);
        tag = (uint32_t)qs << 8;
    };
    auto filter = [&](float4 pj, float3 q, uint32_t jc, uint32_t entry) {
        const float dx = pj.x - q.x, dy = pj.y - q.y, dz = pj.z - q.z;
        const float d2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
        const float dv = __fmaf_rn(vi.z, dz, __fmaf_rn(vi.y, dy, __fmul_rn(vi.x, dx)));
        if (d2 < k.filt_r2 && dv >= dot_lim && jc != s) sm.buf[nb++][t] = (uint16_t)entry;
    };
    // kCandStep candidates per iteration, so that their loads are in flight
    // together; the buffers are flushed with room for the next kCandStep hits
    for (uint32_t it = 0; it < max_nc; it += kCandStep) {
        bool vc[kCandStep];
        uint32_t cc[kCandStep], sc[kCandStep];  // candidate slots and their buffer entries
        float3 qc[kCandStep];
        float4 pc[kCandStep];
#pragma unroll
        for (int u = 0; u < kCandStep; ++u) {
            vc[u] = it + u < mine;
            cc[u] = 0;
            sc[u] = 0;
            qc[u] = make_float3(0.f, 0.f, 0.f);
            if (vc[u]) {
                if (j == jend) advance();
                cc[u] = j++;
                qc[u] = make_float3(qx, qy, qz);
                sc[u] = tag++;
            }
        }
#pragma unroll
        for (int u = 0; u < kCandStep; ++u) pc[u] = vc[u] ? __ldg(g.pos + cc[u]) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int u = 0; u < kCandStep; ++u)
            if (vc[u]) filter(pc[u], qc[u], cc[u], sc[u]);
        // exact tests of the buffered hits, the whole warp together
        const bool far = (tag & 255u) >= 256u - kCandStep;  // the offsets are about to run out
        if (__any_sync(0xffffffffu, nb > kBufA - kCandStep || far) || it + kCandStep >= max_nc) {
            // The warp's hits are tested 32 at a time whatever lane found
            // them (hit i of the lanes' buffers laid end to end goes to lane
            // i % 32), so that a lane with many hits does not hold the warp
            // for as many rounds; each verdict goes back into the finder's
            // buffer (slot | rules << 29, rules 0: not accepted), and each
            // lane then files its own accepted hits in its sorted list.
            const int lane = t;
            int incl = nb;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const int total = __shfl_sync(0xffffffffu, incl, 31);
            const int excl = incl - nb;
            const int lo32 = (int)lo_id;  // ids are below 2^29
            __syncwarp();  // the buffers are written
            for (int base = 0; base < total; base += 32) {
                const int i = base + lane;
                int L = 0;  // the last lane whose hits start at or before i
#pragma unroll
                for (int st = 16; st > 0; st >>= 1) {
                    const int e = __shfl_sync(0xffffffffu, excl, L + st);
                    if (e <= i) L += st;
                }
                const int q = i - __shfl_sync(0xffffffffu, excl, L);
                const float3 po = make_float3(__shfl_sync(0xffffffffu, pi.x, L), __shfl_sync(0xffffffffu, pi.y, L),
                                              __shfl_sync(0xffffffffu, pi.z, L));
                Sight so;
                so.v = make_float3(__shfl_sync(0xffffffffu, sight.v.x, L), __shfl_sync(0xffffffffu, sight.v.y, L),
                                   __shfl_sync(0xffffffffu, sight.v.z, L));
                so.nv = __shfl_sync(0xffffffffu, sight.nv, L);
                so.inv_nv = __shfl_sync(0xffffffffu, sight.inv_nv, L);
                const int olo = __shfl_sync(0xffffffffu, lo32, L);
                if (i < total) {
                    const uint32_t wb = sm.buf[q][L];
                    const uint32_t w0 = sm.seg0[wb >> 8][L], w1 = sm.seg1[wb >> 8][L];
                    const float4 pj = __ldg(g.pos + ((w0 & 0x1fffffffu) + (wb & 255u)));
                    int f = 0;
                    if ((int)__float_as_uint(pj.w) > olo) {
                        // a filter hit from a segment without periodic shift is
                        // nearer than F/2 on every axis: its own minimum image
                        const float3 tt = ((w0 | w1) & 0xe0000000u) ? image3(xyz(pj), po, k) : xyz(pj);
                        f = pair_flags(po, so, tt, k);
                    }
                    sm.buf[q][L] = (uint16_t)(wb | ((uint32_t)f << 13));
                }
            }
            __syncwarp();  // the verdicts are written
            for (int q = 0; q < nb; ++q) {
                const uint32_t hit = sm.buf[q][t];
                if (!(hit >> 13)) continue;
                const uint32_t jb = (sm.seg0[(hit >> 8) & 31u][t] & 0x1fffffffu) + (hit & 255u);
                const uint32_t en = jb | ((hit >> 13) << 29);
                const uint32_t idj = __float_as_uint(__ldg(&g.pos[jb].w));
                ++more;
                const uint64_t e = ((uint64_t)idj << 32) | (uint64_t)en;
                int w;
                if (m < kListA) {
                    w = m++;
                } else {
                    // the list is full: e or its last entry leaves it
                    const uint64_t last = sm.lst[kListA - 1][t];
                    w = e < last ? kListA - 1 : -1;
                    if (ovf) {
                        if (ovf_n < (uint32_t)kOvfCap) ovf[ovf_n] = w < 0 ? e : last;
                        ++ovf_n;
                    }
                    if (w < 0) continue;
                }
                while (w > 0 && sm.lst[w - 1][t] > e) { sm.lst[w][t] = sm.lst[w - 1][t]; --w; }
                sm.lst[w][t] = e;
            }
            __syncwarp();  // the buffers are free for the next hits
            nb = 0;
            if (far) {  // the segment goes on from here
                sm.seg0[qs][t] += tag & 255u;
                tag &= ~255u;
                moved = true;
            }
        }
    }
    if (need) {
        list_accumulate<DIAG>(sm, t, m, pi, a, g, k);
        if (more <= (uint32_t)m) need = false;
        else lo_id = (int64_t)(sm.lst[m - 1][t] >> 32);
    }
}

// A deferred boid's further passes from its overflow row (on <= kOvfCap
// entries, every accepted neighbour with an id above lo_id): the next
// kListA ids sorted in the lane's column of sm.lst and accumulated, until
// none is left.  Per lane; no candidate is walked again.
template <bool DIAG>
__device__ __forceinline__ void ovf_passes(SparseSmem &sm, int t, const uint64_t *__restrict__ row, uint32_t on,
                                           int64_t lo_id, float3 pi, Acc &a, const GridIn &g, const StepConst &k)
{
    for (;;) {
        int m = 0;
        uint32_t more = 0;
        for (uint32_t q = 0; q < on; ++q) {
            const uint64_t e = row[q];
            if ((int64_t)(e >> 32) <= lo_id) continue;
            ++more;
            int w;
            if (m < kListA) w = m++;
            else if (e < sm.lst[kListA - 1][t]) w = kListA - 1;
            else continue;
            while (w > 0 && sm.lst[w - 1][t] > e) { sm.lst[w][t] = sm.lst[w - 1][t]; --w; }
            sm.lst[w][t] = e;
        }
        list_accumulate<DIAG>(sm, t, m, pi, a, g, k);
        if (more <= (uint32_t)m) return;
        lo_id = (int64_t)(sm.lst[m - 1][t] >> 32);
    }
}

// One warp a CTA, so that a warp's tables are free for the next as soon as it
// is done (and those whose boids all lie in dense cells are gone at once), and
// tables small enough for 24 of them on an SM (with the system's 1 KB each):
// a hit is an offset of 8 bits in a segment, and a segment that goes on beyond
// 255 slots is moved on behind a flush.  Against CTAs of four warps with whole
// slots in their buffers a step takes, us: 262 143 boids 167 (172), 2^20 one
// update after a uniform start 377 (374), 6 after 406 (414), 20 after 803
// (847), 100 after 1600 (1701), 400 after 2075 (2178), 2^22 4 after 1390 (1425).
// (With whole slots in one warp's buffer, 21 on an SM: 420 after 6.)  An
// ensemble's CTAs have four warps, for one copy of the flock's constants: with
// one a step of 16 uniform flocks of 16 384 took 188 us for 165, 15 updates
// after 290 for 260; gathered 812 for 825.
__host__ __device__ constexpr int sparse_warps(bool ensemble) { return ensemble ? 4 : 1; }
template <bool DIAG, bool MULTI>
__global__ void __launch_bounds__(32 * sparse_warps(MULTI), 24 / sparse_warps(MULTI))
k_grid_sparse(GridIn g, GridOut o, StepConst kp, FlockTable ft)
{
    constexpr int kW = sparse_warps(MULTI);
    static_assert(kSlotAlign % (32 * kW) == 0, "a CTA serves one flock");
    // the tables, and an ensemble's flock's constants
    __shared__ __align__(16) unsigned char smem[kW * sizeof(SparseSmem) + (MULTI ? sizeof(StepConst) : 0)];
    SparseSmem &sm = reinterpret_cast<SparseSmem *>(smem)[kW > 1 ? threadIdx.x >> 5 : 0];
    StepConst &kf = *reinterpret_cast<StepConst *>(smem + (MULTI ? kW * sizeof(SparseSmem) : 0));
    if (g.chain) chain_wait();
    if (MULTI) load_flock(kf, ft, ft.blk_flock[blockIdx.x * 32 * kW / kSlotAlign]);
    const StepConst &k = MULTI ? kf : kp;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    // this warp's boids outside dense cells (the others are k_grid_dense's)
    const uint32_t s = blockIdx.x * 32 * kW + threadIdx.x;
    bool act = s - k.slot_base < k.n;
    const float4 p4 = act ? g.pos[s] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 v4 = act ? g.vel[s] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float3 pi = xyz(p4);
    const int cy = cell1(pi.y, k), cz = cell1(pi.z, k);
    if (act) act = !__ldg(g.dflag + (k.cell_base / 4 + (uint32_t)((cz * k.G + cy) * k.G + cell1(pi.x, k))));
    if (!__any_sync(0xffffffffu, act)) return;
    uint32_t nc = act ? sparse_segments(sm, lane, pi, cy, cz, g, k) : 0;
    const Sight sight = make_sight(xyz(v4));
    const float dot_lim = k.cone_pre ? -(sight.nv * k.dot_eps) : -INFINITY;  // cone pre-test
    Acc a;
    acc_zero(a);
    int64_t lo_id = -1;  // ids <= lo_id were accumulated by earlier passes
    bool need = act;
    uint32_t ovf_n = 0;
    bool moved;
    sparse_pass<DIAG>(sm, lane, s, pi, sight, dot_lim, nc, need, lo_id, a, g, k,
                      o.ovf && act ? o.ovf + (size_t)s * kOvfCap : nullptr, ovf_n, moved);
    if (o.defer) {
        // Boids with more accepted neighbours than one list holds go to
        // k_grid_sparse_more with their partial sums: every further pass
        // walks all of a lane's candidates, however few lanes of the warp
        // still need one, and there they run in full warps.
        const unsigned nbal = __ballot_sync(0xffffffffu, need);
        uint32_t q0 = 0;
        if (lane == 0 && nbal) q0 = atomicAdd(o.defer_cnt + k.flock, (uint32_t)__popc(nbal));
        q0 = __shfl_sync(0xffffffffu, q0, 0);
        if (need) {
            const uint32_t q = k.slot_base + q0 + __popc(nbal & below);
            o.defer[2 * q] = s;
            o.defer[2 * q + 1] = (uint32_t)lo_id;
            o.carry[s] = a;
            if (o.ovf) o.ovf_n[s] = ovf_n;
        } else if (act) {
            finish_boid<DIAG>(a, p4, sight.v, s, o, k);
        }
        return;
    }
    while (__any_sync(0xffffffffu, need)) {
        if (moved) nc = sparse_segments(sm, lane, pi, cy, cz, g, k);
        sparse_pass<DIAG>(sm, lane, s, pi, sight, dot_lim, nc, need, lo_id, a, g, k, nullptr, ovf_n, moved);
    }
    if (act) finish_boid<DIAG>(a, p4, sight.v, s, o, k);
}

// The boids k_grid_sparse deferred: thread per queued boid, its segments
// recomputed, further passes from its partial sums.  A single flock's queue
// is walked grid-stride; in an ensemble CTA b takes the b-th block of 128
// entries of its flock's queue (the flock of slot block b), so that a CTA
// serves one flock.
template <bool DIAG, bool MULTI>
__global__ void __launch_bounds__(kRT)
k_grid_sparse_more(GridIn g, GridOut o, StepConst kp, FlockTable ft)
{
    __shared__ SparseSmem wsm[kRT / 32];
    __shared__ __align__(8) uint32_t kf_words[MULTI ? sizeof(StepConst) / 4 : 1];
    StepConst &kf = *reinterpret_cast<StepConst *>(kf_words);
    const int t = threadIdx.x, lane = t & 31;
    SparseSmem &sm = wsm[t >> 5];
    uint32_t first = 0, count, stride;  // entries [first + base, first + count), base += stride
    uint32_t base = blockIdx.x * kRT;
    if (MULTI) {
        const uint32_t f = ft.blk_flock[blockIdx.x];
        const uint32_t sb = __ldg(&ft.ks[f].slot_base);
        count = o.defer_cnt[f];
        base = blockIdx.x * kRT - sb;  // this CTA's block of the flock's queue
        if (base >= count) return;     // uniform over the CTA
        first = sb;
        stride = count;                // one block per CTA
        load_flock(kf, ft, f);
    } else {
        count = o.defer_cnt[0];
        stride = gridDim.x * kRT;
    }
    const StepConst &k = MULTI ? kf : kp;
    for (; base < count; base += stride) {
        if (base + (uint32_t)(t & ~31) >= count) break;  // the whole warp is idle
        const uint32_t i = base + t;
        const bool act = i < count;
        const uint32_t s = act ? o.defer[2 * (first + i)] : 0u;
        int64_t lo_id = act ? (int64_t)o.defer[2 * (first + i) + 1] : -1;
        Acc a;
        if (act) a = o.carry[s];
        else acc_zero(a);
        const float4 p4 = act ? g.pos[s] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 v4 = act ? g.vel[s] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float3 pi = xyz(p4);
        // a boid whose first pass recorded all the neighbours it could not
        // keep takes them from its overflow row; the others walk their
        // candidates again
        const uint32_t on = act && o.ovf ? o.ovf_n[s] : (uint32_t)kOvfCap + 1;
        const bool from_row = on <= (uint32_t)kOvfCap;
        if (from_row) ovf_passes<DIAG>(sm, lane, o.ovf + (size_t)s * kOvfCap, on, lo_id, pi, a, g, k);
        bool need = act && !from_row;
        uint32_t nc = need ? sparse_segments_ahead(sm, lane, pi, cell1(pi.y, k), cell1(pi.z, k), g, k) : 0;
        const Sight sight = make_sight(xyz(v4));
        const float dot_lim = k.cone_pre ? -(sight.nv * k.dot_eps) : -INFINITY;
        uint32_t ovf_n = 0;
        bool moved = false;
        while (__any_sync(0xffffffffu, need)) {
            if (moved) nc = sparse_segments_ahead(sm, lane, pi, cell1(pi.y, k), cell1(pi.z, k), g, k);
            sparse_pass<DIAG>(sm, lane, s, pi, sight, dot_lim, nc, need, lo_id, a, g, k, nullptr, ovf_n, moved);
        }
        if (act) finish_boid<DIAG>(a, p4, sight.v, s, o, k);
    }
}

// ------------------------------------------------------------------ a warp per boid

// k_grid_warp: the 32 lanes of a warp update one boid together, straight from
// the cell table: the flocks too small to fill the GPU with a thread per boid
// or a CTA per cell.
//
//   1. lane r takes row r of the boid's nine neighbour rows: the x cells its
//      sphere reaches, as runs of slots (sparse_segments' rule, a row a lane);
//   2. the runs are walked with 8, 16 or 32 lanes each, four, two or one at a
//      time, by the longest run, so that short rows share an iteration and no
//      lane searches for its run; candidates passing the float filter are
//      compacted into a queue, and every 32 of them take the exact tests;
//   3. accepted neighbours (at most kWarpList at a time) are put in id order:
//      by counting smaller ids up to 32 of them, by one bucket pass over their
//      id range beyond;
//   4. 32 at a time in id order, each lane prepares one neighbour's summands
//      (image, velocity, normalised offset), and nine lanes add them up, one
//      component each.  A neighbour a rule does not accept contributes +0,
//      which leaves a float sum that started at +0 unchanged (such a sum is
//      never -0), so every sum is the reference's sequence of additions;
//   5. the boid is finished by nine lanes, a component each.
//
// A boid that accepts more than kWarpList neighbours starts over in warp_many,
// which needs no sort: the filter's hits are marked in a bit map over ids.
//
// Bound by instruction issue once every SM has its 32 warps, by the length of
// one boid's chain of loads, tests and sums below that (about 14 us).  A step
// of 1000 boids of test.ini takes 21 us (28 before its counting sort was one
// kernel) where the split of cells over k_grid_sparse and k_grid_dense took 109
// (their few CTAs leave most SMs idle), gathered flocks of 16 384 boids 54 us
// (188), of 32 768 boids 90 us (215), uniform ones 35 us (63) and 56 us (74), all
// with the counting sort.  Per-boid work is about five times k_grid_sparse's on a
// uniform flock (1240 warp instructions against 206 a boid), hence kWarpBoids.
constexpr int kWarpWarps = 4;    // warps of a CTA
constexpr int kWarpCtas = 8;     // CTAs per SM
constexpr int kWarpList = 256;   // accepted neighbours kept
constexpr int kWarpBuckets = 128;
constexpr int kWarpIds = 8192;   // ids of a window of warp_many

struct WarpSmem {  // of one warp
    uint32_t lid[kWarpList], lsl[kWarpList];  // accepted: id; slot | rules << 29
    uint8_t ord[kWarpList];                   // the list's entries in id order
    union {
        float st[9][32 + 4];                  // summands of 32 neighbours, by component
        struct {
            uint32_t cnt[kWarpBuckets + 4];   // the ordering's bucket counters
            uint8_t at[kWarpList];            // an entry's arrival in its bucket
            uint8_t ent[kWarpList];           // entries by bucket
        } b;
    } u;
    float4 shift[18];                         // run: image shift
    uint2 run[18];                            // run: first slot | wrapped << 31, length
    uint32_t queue[64];                       // filter hits, a ring: slot | wrapped << 31
};
static_assert(kWarpList <= 256, "entries are named in a byte");

// The warp's n list entries in id order into sm.ord.
__device__ __forceinline__ void warp_order(WarpSmem &sm, int lane, int n)
{
    uint32_t *lid = sm.lid;
    if (n <= 32) {
        const uint32_t id = lane < n ? lid[lane] : 0xffffffffu;
        if (lane >= n) lid[lane] = 0xffffffffu;
        else sm.ord[lane] = (uint8_t)lane;  // equal ids (a state no update makes) leave no stale entry
        __syncwarp();
        int rank = 0;
        for (int j = 0; j < n; j += 4) {
            const uint4 w = *reinterpret_cast<const uint4 *>(lid + j);
            rank += (w.x < id) + (w.y < id) + (w.z < id) + (w.w < id);
        }
        if (lane < n) sm.ord[rank] = (uint8_t)lane;
        __syncwarp();
        return;
    }
    // one bucket pass over the ids' range, then each entry's place inside its
    // bucket by counting the smaller ids there
    uint32_t *cnt = sm.u.b.cnt;
    *reinterpret_cast<uint4 *>(cnt + 4 * lane) = make_uint4(0, 0, 0, 0);
    uint32_t mn = 0xffffffffu, mx = 0;
    for (int i = lane; i < n; i += 32) {
        const uint32_t id = lid[i];
        mn = min(mn, id);
        mx = max(mx, id);
        sm.ord[i] = (uint8_t)i;
    }
    mn = __reduce_min_sync(0xffffffffu, mn);
    mx = __reduce_max_sync(0xffffffffu, mx);
    static_assert(kWarpBuckets == 128, "four buckets a lane, 2^7 of them");
    const uint32_t range = mx - mn;
    const int shift = range >> 7 ? 32 - __clz(range) - 7 : 0;
    __syncwarp();
    for (int i = lane; i < n; i += 32) sm.u.b.at[i] = (uint8_t)atomicAdd(cnt + ((lid[i] - mn) >> shift), 1u);
    __syncwarp();
    const uint4 c = *reinterpret_cast<const uint4 *>(cnt + 4 * lane);
    const uint32_t sum = c.x + c.y + c.z + c.w;
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    const uint32_t ex = incl - sum;
    *reinterpret_cast<uint4 *>(cnt + 4 * lane) = make_uint4(ex, ex + c.x, ex + c.x + c.y, ex + c.x + c.y + c.z);
    if (lane == 31) cnt[kWarpBuckets] = incl;
    __syncwarp();
    for (int i = lane; i < n; i += 32) sm.u.b.ent[cnt[(lid[i] - mn) >> shift] + sm.u.b.at[i]] = (uint8_t)i;
    __syncwarp();
    for (int i = lane; i < n; i += 32) {
        const uint32_t id = lid[i], b = (id - mn) >> shift, b0 = cnt[b], b1 = cnt[b + 1];
        uint32_t rank = b0;
        if (b1 - b0 > 1)
            for (uint32_t j = b0; j < b1; ++j) rank += lid[sm.u.b.ent[j]] < id;
        sm.ord[rank] = (uint8_t)i;
    }
    __syncwarp();
}

// One boid's sums: lane c < 9 holds component c of (cohesion, separation,
// alignment) in acc; the counts (and the diagnostics' id hashes, each lane's
// own part) are beside it.
struct WarpSums {
    float acc;
    int ncoh, nsep, nali;
    uint64_t h[3];
};

// Adds up to 32 neighbours, a lane each in ascending id, accepted by rules f
// (0: none): image t, velocity vj.  The accepted are compacted into the
// columns of sm.u.st, and lanes 0-8 add those up.
template <bool DIAG>
__device__ __forceinline__ void warp_add(WarpSmem &sm, int lane, int f, float3 t, float4 vj, uint32_t id, float3 pi,
                                         WarpSums &a)
{
    constexpr unsigned kAll = 0xffffffffu;
    const unsigned am = __ballot_sync(kAll, f != 0);
    if (!am) return;
    const int m = __popc(am);
    const bool co = f & 1, se = f & 2, al = f & 4;
    const unsigned em = __ballot_sync(kAll, se);
    a.ncoh += __popc(__ballot_sync(kAll, co));
    a.nsep += __popc(em);
    a.nali += __popc(__ballot_sync(kAll, al));
    float(&st)[9][36] = sm.u.st;
    if (f) {
        const int c = __popc(am & ((1u << lane) - 1u));
        st[0][c] = co ? t.x : 0.f;
        st[1][c] = co ? t.y : 0.f;
        st[2][c] = co ? t.z : 0.f;
        st[6][c] = al ? vj.x : 0.f;
        st[7][c] = al ? vj.y : 0.f;
        st[8][c] = al ? vj.z : 0.f;
        if (em) {
            float3 u = make_float3(0.f, 0.f, 0.f);
            if (se) {  // Vector3D::normalized of pi - t
                const float dx = __fsub_rn(pi.x, t.x), dy = __fsub_rn(pi.y, t.y), dz = __fsub_rn(pi.z, t.z);
                const float n = nrm3(dx, dy, dz);
                u = make_float3(__fdiv_rn(dx, n), __fdiv_rn(dy, n), __fdiv_rn(dz, n));
            }
            st[3][c] = u.x;
            st[4][c] = u.y;
            st[5][c] = u.z;
        }
        if (DIAG) {
            const uint64_t h = id_hash(id);
            if (co) a.h[0] += h;
            if (se) a.h[1] += h;
            if (al) a.h[2] += h;
        }
    }
    // columns m .. up to a multiple of four: +0
    const int pad = (4 - m) & 3;
    if ((lane & 3) < pad) st[lane >> 2][m + (lane & 3)] = 0.f;
    if (lane < pad) st[8][m + lane] = 0.f;
    __syncwarp();
    if (lane < 9 && (em || lane < 3 || lane >= 6)) {
        const float *row = st[lane];
        for (int c = 0; c < m; c += 4) {
            const float4 x = *reinterpret_cast<const float4 *>(row + c);
            a.acc = __fadd_rn(a.acc, x.x);
            a.acc = __fadd_rn(a.acc, x.y);
            a.acc = __fadd_rn(a.acc, x.z);
            a.acc = __fadd_rn(a.acc, x.w);
        }
    }
    __syncwarp();
}

// The search of a boid that accepts more than kWarpList neighbours: for
// windows of kWarpIds ids in ascending order, the filter's hits are marked in
// a bit map of the window, its bits are expanded in id order, and the hits
// found through the id -> slot table take the exact tests and are added up,
// 32 at a time.  Out of line: it is rare.
template <bool DIAG>
__device__ __noinline__ WarpSums warp_many(WarpSmem *smp, const float4 *__restrict__ gpos,
                                           const float4 *__restrict__ gvel, const uint32_t *__restrict__ slot_of,
                                           const StepConst &k, uint32_t s, float3 pi, Sight si, float dot_lim, int nr,
                                           bool shifted)
{
    constexpr unsigned kAll = 0xffffffffu;
    WarpSmem &sm = *smp;
    const int lane = threadIdx.x & 31;
    uint32_t *map = sm.lid;                                   // kWarpIds bits
    uint16_t *hits = reinterpret_cast<uint16_t *>(sm.lsl);    // lsl and ord: a group's hits and the rest before it
    constexpr int kGroup = 16;                                // map words expanded at a time
    static_assert(kWarpIds == 32 * kWarpList, "the map takes the list's ids");
    static_assert(2 * (32 * kGroup + 32) <= sizeof(sm.lsl) + sizeof(sm.ord), "a group's hits fit");
    WarpSums a{};
    for (uint32_t w0 = 0; w0 < k.n; w0 += kWarpIds) {
        for (int i = lane; i < kWarpList; i += 32) map[i] = 0;
        __syncwarp();
        for (int r = 0; r < nr; ++r) {
            const uint2 rn = sm.run[r];
            const float4 sh = sm.shift[r];
            const float3 q = make_float3(pi.x - sh.x, pi.y - sh.y, pi.z - sh.z);
            for (uint32_t off = lane; off < rn.y; off += 32) {
                const uint32_t slot = (rn.x & 0x7fffffffu) + off;
                const float4 pj = __ldg(gpos + slot);
                const float dx = pj.x - q.x, dy = pj.y - q.y, dz = pj.z - q.z;
                const float d2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
                const float dv = __fmaf_rn(si.v.z, dz, __fmaf_rn(si.v.y, dy, __fmul_rn(si.v.x, dx)));
                const uint32_t id = __float_as_uint(pj.w) - w0;
                if (d2 < k.filt_r2 && dv >= dot_lim && slot != s && id < (uint32_t)kWarpIds)
                    atomicOr(map + (id >> 5), 1u << (id & 31));
            }
        }
        __syncwarp();
        int nh = 0;  // hits waiting
        for (int g0 = 0; g0 < kWarpList; g0 += kGroup) {
            uint32_t bits = lane < kGroup ? map[g0 + lane] : 0u;
            int incl = __popc(bits);
#pragma unroll
            for (int o = 1; o < kGroup; o <<= 1) {
                const int y = __shfl_up_sync(kAll, incl, o);
                if (lane >= o) incl += y;
            }
            int at = nh + incl - __popc(bits);
            nh += __shfl_sync(kAll, incl, kGroup - 1);
            while (bits) {
                hits[at++] = (uint16_t)(((g0 + lane) << 5) + __ffs(bits) - 1);
                bits &= bits - 1;
            }
            __syncwarp();
            int h0 = 0;
            const int enough = g0 + kGroup < kWarpList ? 32 : 1;
            while (nh >= enough) {
                int f = 0;
                uint32_t id = 0;
                float3 t = make_float3(0.f, 0.f, 0.f);
                float4 vj = make_float4(0.f, 0.f, 0.f, 0.f);
                if (lane < nh) {
                    id = w0 + hits[h0 + lane];
                    const uint32_t slot = __ldg(slot_of + k.slot_base + id);
                    const float4 pj = __ldg(gpos + slot);
                    t = shifted ? image3(xyz(pj), pi, k) : xyz(pj);
                    f = pair_flags(pi, si, t, k);
                    if (f) vj = __ldg(gvel + slot);
                }
                warp_add<DIAG>(sm, lane, f, t, vj, id, pi, a);
                const int done = min(nh, 32);
                h0 += done;
                nh -= done;
            }
            // the rest to the front
            const uint16_t rest = lane < nh ? hits[h0 + lane] : 0;
            __syncwarp();
            if (lane < nh) hits[lane] = rest;
            __syncwarp();
        }
    }
    return a;
}

// finish_boid by the lanes of a warp.
template <bool DIAG>
__device__ __forceinline__ void warp_finish(WarpSums &a, float4 p4, float3 vi, uint32_t s, int lane, const GridOut &o,
                                            const StepConst &k)
{
    constexpr unsigned kAll = 0xffffffffu;
    const uint32_t out = __float_as_uint(p4.w) + (k.slot_base - k.slot_off);  // the boid's output row
    if (DIAG) {
#pragma unroll
        for (int r = 0; r < 3; ++r) {
#pragma unroll
            for (int q = 16; q > 0; q >>= 1) a.h[r] += __shfl_xor_sync(kAll, a.h[r], q);
        }
        if (lane == 0) {
            o.dcnt[3 * out + 0] = a.ncoh; o.dcnt[3 * out + 1] = a.nsep; o.dcnt[3 * out + 2] = a.nali;
            o.dhash[3 * out + 0] = a.h[0]; o.dhash[3 * out + 1] = a.h[1]; o.dhash[3 * out + 2] = a.h[2];
        }
        return;
    }
    const int r = lane / 3, c = lane - 3 * r;
    const float pc = c == 0 ? p4.x : (c == 1 ? p4.y : p4.z), vc = c == 0 ? vi.x : (c == 1 ? vi.y : vi.z);
    float f = a.acc;
    const int q = r == 0 ? a.ncoh : a.nali;
    if (r != 1 && q != 0) f = __fsub_rn(__fdiv_rn(a.acc, __int2float_rn(q)), r == 0 ? pc : vc);
    f = __fmul_rn(f, r == 0 ? k.cc : (r == 1 ? k.cs : k.ca));
    const float fs = __shfl_sync(kAll, f, c + 3), fa = __shfl_sync(kAll, f, c + 6);
    // lanes 0-2: a component each (the others' values are not used)
    float v = __fadd_rn(vc, __fadd_rn(__fadd_rn(f, fs), fa));
    const float n = nrm3(__shfl_sync(kAll, v, 0), __shfl_sync(kAll, v, 1), __shfl_sync(kAll, v, 2));
    if (n > 0.0f && n > k.vmax_dn) v = __fmul_rn(__fdiv_rn(v, n), k.vmax_f);
    else if (n > 0.0f && n < k.vmin_up) v = __fmul_rn(__fdiv_rn(v, n), k.vmin_f);
    const float x = lane < 3 ? wrap1(__fadd_rn(pc, v), k) : p4.w;
    const float x0 = __shfl_sync(kAll, x, 0), x1 = __shfl_sync(kAll, x, 1), x2 = __shfl_sync(kAll, x, 2);
    if (o.pos3_out) {
        if (lane < 3) {
            o.pos3_out[(size_t)3 * out + lane] = x;
            o.vel3_out[(size_t)3 * out + lane] = v;
        }
    } else if (lane < 4) {
        reinterpret_cast<float *>(o.pos_out + s)[lane] = x;
        reinterpret_cast<float *>(o.vel_out + s)[lane] = lane < 3 ? v : 0.f;
    }
    if (o.key_out && lane == 0) {  // binning for the next step
        const uint32_t cell = k.cell_base + cell_key(make_float3(x0, x1, x2), k);
        o.key_out[s] = cell;
        o.rank_out[s] = atomicAdd(o.count + cell, 1u);
    }
    if (o.forces && lane < 9)
        o.forces[(size_t)9 * out + lane] = f;
}

// The update of the boid in slot s, by the 32 lanes of a warp.
template <bool DIAG>
__device__ __forceinline__ void warp_boid(WarpSmem &sm, const GridIn &g, const GridOut &o, const StepConst &k, uint32_t s,
                                          int lane)
{
    constexpr unsigned kAll = 0xffffffffu;
    const unsigned below = (1u << lane) - 1u;
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 p4 = __ldg(g.pos + s);
    const float3 pi = xyz(p4);
    const Sight si = make_sight(xyz(__ldg(g.vel + s)));
    const float dot_lim = k.cone_pre ? -(si.nv * k.dot_eps) : -INFINITY;

    // ---- the boid's runs of candidates, a row per lane
    const int G = k.G, Gx = k.Gx;
    uint32_t ja = 0, la = 0, jb = 0, lb = 0;
    float sx0 = 0.f, sx1 = 0.f, sy = 0.f, sz = 0.f;
    if (lane < 9) {
        const int cy = cell1(pi.y, k), cz = cell1(pi.z, k);
        const int dz = lane / 3 - 1, dy = lane - 3 * (lane / 3) - 1;
        const float eps = k.side * 1e-5f;
        const float ddy = dy == 0 ? 0.f : fmaxf(0.f, dy < 0 ? pi.y - (float)cy * k.side - eps
                                                          : (float)(cy + 1) * k.side - pi.y - eps);
        const float ddz = dz == 0 ? 0.f : fmaxf(0.f, dz < 0 ? pi.z - (float)cz * k.side - eps
                                                          : (float)(cz + 1) * k.side - pi.z - eps);
        const float rem = k.trim_r2 - ddy * ddy - ddz * ddz;
        if (rem > 0.f) {
            const float rx = rem * rsqrtf(rem);  // trim_r2's margin covers its rounding
            // clamped as in sparse_segments: a state outside the field stays within the cell tables
            const int lo = max(__float2int_rd((pi.x - rx) * k.inv_subx), 1 - Gx);
            const int hi = min(__float2int_rd((pi.x + rx) * k.inv_subx), 2 * Gx - 2);
            int a0 = lo, a1 = hi + 1, c0 = 0, c1 = 0;
            if (lo < 0) { a0 = lo + Gx; a1 = Gx; sx0 = -k.Ff; c1 = min(hi + 1, Gx); }
            else if (hi >= Gx) { a1 = Gx; c1 = hi + 1 - Gx; sx1 = k.Ff; }
            int zz = cz + dz, yy = cy + dy;
            if (zz < 0) { zz += G; sz = -k.Ff; } else if (zz >= G) { zz -= G; sz = k.Ff; }
            if (yy < 0) { yy += G; sy = -k.Ff; } else if (yy >= G) { yy -= G; sy = k.Ff; }
            const uint32_t rb = k.cell_base + (uint32_t)(zz * G + yy) * (uint32_t)Gx;
            if (a1 > a0) {
                ja = slot_start(g.lstart, g.bsum, rb + a0, k);
                la = slot_start(g.lstart, g.bsum, rb + a1, k) - ja;
            }
            if (c1 > c0) {
                jb = slot_start(g.lstart, g.bsum, rb + c0, k);
                lb = slot_start(g.lstart, g.bsum, rb + c1, k) - jb;
            }
        }
    }
    const bool wa = sx0 != 0.f || sy != 0.f || sz != 0.f, wb = sx1 != 0.f || sy != 0.f || sz != 0.f;
    const unsigned ba = __ballot_sync(kAll, la != 0), bb = __ballot_sync(kAll, lb != 0);
    const bool shifted = __any_sync(kAll, (la && wa) || (lb && wb));
    const int na = __popc(ba), nr = na + __popc(bb);  // non-empty runs
    if (la) {
        const int q = __popc(ba & below);
        sm.run[q] = make_uint2(ja | (wa ? 0x80000000u : 0u), la);
        sm.shift[q] = make_float4(sx0, sy, sz, 0.f);
    }
    if (lb) {
        const int q = na + __popc(bb & below);
        sm.run[q] = make_uint2(jb | (wb ? 0x80000000u : 0u), lb);
        sm.shift[q] = make_float4(sx1, sy, sz, 0.f);
    }
    // lanes per run: 8 or 16 where every run fits, else 32
    const uint32_t longest = __reduce_max_sync(kAll, max(la, lb));
    const int wsh = longest <= 8 ? 3 : (longest <= 16 ? 4 : 5);
    const int rstep = 32 >> wsh, rsub = lane >> wsh;
    const uint32_t off0 = lane & ((1 << wsh) - 1);
    __syncwarp();

    WarpSums a{};
    int nl = 0, nq = 0;  // accepted; filter hits waiting in the ring
    uint32_t qh = 0;     // the ring's head
    for (int r = 0; r < nr; r += rstep) {
        const int ri = r + rsub;
        const uint2 rn = ri < nr ? sm.run[ri] : make_uint2(0u, 0u);
        float3 q = pi;  // the query point: the candidate's image is pj + shift
        if (shifted && ri < nr) {
            const float4 sh = sm.shift[ri];
            q = make_float3(pi.x - sh.x, pi.y - sh.y, pi.z - sh.z);
        }
        // (a run longer than its lanes is walked by the whole warp: its length
        // is the same in every lane)
        uint32_t base = 0;
        do {
            const uint32_t off = base + off0;
            bool hit = false;
            const uint32_t w = rn.x + off, slot = w & 0x7fffffffu;
            if (off < rn.y) {
                const float4 pj = __ldg(g.pos + slot);
                const float dx = pj.x - q.x, dy = pj.y - q.y, dz = pj.z - q.z;
                const float d2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
                const float dv = __fmaf_rn(si.v.z, dz, __fmaf_rn(si.v.y, dy, __fmul_rn(si.v.x, dx)));
                hit = d2 < k.filt_r2 && dv >= dot_lim && slot != s;
            }
            const unsigned hm = __ballot_sync(kAll, hit);
            if (hit) sm.queue[(qh + nq + __popc(hm & below)) & 63] = w;
            nq += __popc(hm);
            // exact tests of the hits, 32 at a time; the last candidates' hits
            // whatever their number
            base += 32;
            const int enough = r + rstep < nr || base < rn.y ? 32 : 1;
            while (nq >= enough) {
                __syncwarp();
                int f = 0;
                uint32_t id = 0, js = 0;
                if (lane < nq) {
                    const uint32_t e = sm.queue[(qh + lane) & 63];
                    js = e & 0x7fffffffu;
                    const float4 pj = __ldg(g.pos + js);
                    id = __float_as_uint(pj.w);
                    // a hit from a run without periodic shift is its own minimum image
                    const float3 t = (e >> 31) ? image3(xyz(pj), pi, k) : xyz(pj);
                    f = pair_flags(pi, si, t, k);
                }
                const int done = min(nq, 32);
                qh += done;
                nq -= done;
                const unsigned am = __ballot_sync(kAll, f != 0);
                const int at = nl + __popc(am & below);
                if (f && at < kWarpList) {
                    sm.lid[at] = id;
                    sm.lsl[at] = js | ((uint32_t)f << 29);
                }
                nl += __popc(am);
            }
        } while (base < rn.y);
        if (nl > kWarpList) break;
    }
    __syncwarp();
    if (nl > kWarpList) {
        a = warp_many<DIAG>(&sm, g.pos, g.vel, g.slot_of, k, s, pi, si, dot_lim, nr, shifted);
    } else if (nl > 0) {
        // the accepted neighbours in id order, the next 32 neighbours' loads in
        // flight under each 32's sums
        warp_order(sm, lane, nl);
        uint32_t e = 0;
        float4 pj = zero4, vj = zero4;
        auto load = [&](int i) {
            e = 0;
            if (i < nl) {
                e = sm.lsl[sm.ord[i]];
                pj = __ldg(g.pos + (e & 0x1fffffffu));
                vj = __ldg(g.vel + (e & 0x1fffffffu));
            }
        };
        load(lane);
        for (int c0 = 0; c0 < nl; c0 += 32) {
            const int f = (int)(e >> 29);
            const float3 t = shifted ? image3(xyz(pj), pi, k) : xyz(pj);
            const float4 v = vj;
            const uint32_t id = __float_as_uint(pj.w);
            load(c0 + 32 + lane);
            warp_add<DIAG>(sm, lane, f, t, v, id, pi, a);
        }
    }
    warp_finish<DIAG>(a, p4, si.v, s, lane, o, k);
}

template <bool DIAG, bool MULTI>
__global__ void __launch_bounds__(kWarpWarps * 32, kWarpCtas)
k_grid_warp(GridIn g, GridOut o, StepConst kp, FlockTable ft)
{
    __shared__ WarpSmem sms[kWarpWarps];
    __shared__ __align__(8) uint32_t kf_words[MULTI ? sizeof(StepConst) / 4 : 1];
    StepConst &kf = *reinterpret_cast<StepConst *>(kf_words);
    chain_wait();
    if (MULTI) load_flock(kf, ft, ft.blk_flock[blockIdx.x * kWarpWarps / kSlotAlign]);
    const StepConst &k = MULTI ? kf : kp;
    const uint32_t s = blockIdx.x * kWarpWarps + (threadIdx.x >> 5);
    if (s - k.slot_base >= k.n) return;
    warp_boid<DIAG>(sms[threadIdx.x >> 5], g, o, k, s, threadIdx.x & 31);
}

// The same where the scan's measure decides whether the boids come here: a
// grid that fills the GPU once, whose CTAs take kWarpWarps consecutive boids at
// a time from a queue, so that a step that does not come here costs one short
// launch (2 us; a CTA per four boids, most of them to end at once, took 24 us
// at 65 537 boids and 100 at 262 143).  Bound as k_grid_warp.  Consecutive
// boids share their candidates in L1: a queue of single boids per warp took
// 149 us a step for 134 (65 537 boids, 1.3 n pairs), four boids in turn per
// warp 173.
template <bool DIAG, bool MULTI>
__global__ void __launch_bounds__(kWarpWarps * 32, kWarpCtas)
k_grid_warp_queue(GridIn g, GridOut o, uint32_t *__restrict__ taken, StepConst kp, FlockTable ft)
{
    chain_wait();
    if (!crowded(g.crowd)) return;
    static_assert(kSlotAlign % kWarpWarps == 0, "the boids taken together are of one flock");
    __shared__ WarpSmem sms[kWarpWarps];
    __shared__ __align__(8) uint32_t kf_words[MULTI ? sizeof(StepConst) / 4 : 1];
    __shared__ uint32_t at;
    StepConst &kf = *reinterpret_cast<StepConst *>(kf_words);
    if (MULTI && threadIdx.x == 0) kf.flock = ~0u;
    for (;;) {
        if (threadIdx.x == 0) at = kWarpWarps * atomicAdd(taken, 1u);
        __syncthreads();
        const uint32_t s = at + (threadIdx.x >> 5);
        if (at >= (MULTI ? ft.nslots : kp.n)) return;
        if (MULTI) {
            const uint32_t f = ft.blk_flock[at / kSlotAlign];
            if (f != kf.flock) {
                __syncthreads();
                load_flock(kf, ft, f);
            }
        }
        const StepConst &k = MULTI ? kf : kp;
        if (s - k.slot_base < k.n) warp_boid<DIAG>(sms[threadIdx.x >> 5], g, o, k, s, threadIdx.x & 31);
        __syncthreads();
    }
}

// ------------------------------------------------------------------ dense cells: CTA per cell

// Stable LSD radix sort of n 64-bit keys held in shared memory, on bits
// [lo, lo + nbits), kRadixBits bits per pass; NT threads each own a
// contiguous run.  hist holds kRadixWords(NT) words: counter i lives at
// i + i / 16, which keeps the (digit, thread) column walks free of bank
// conflicts.  Returns the buffer that holds the sorted keys.  It is the
// CTA-per-cell kernel's fallback sort (block_bucket_sort), so it favours a
// small counter table over few passes.
__device__ __forceinline__ int hpad(int i) { return i + (i >> 4); }
constexpr int kRadixBits = 2, kRadixDigits = 1 << kRadixBits;
__host__ __device__ constexpr int kRadixWords(int nt) { return kRadixDigits * nt + kRadixDigits * nt / 16; }

template <int NT>
__device__ uint64_t *block_radix_sort(uint64_t *a, uint64_t *b, uint32_t *hist, int n, int lo, int nbits)
{
    __shared__ uint32_t wsum[NT / 32];
    constexpr int D = kRadixDigits;
    const int t = threadIdx.x;
    // an odd run length keeps the threads' 64-bit reads a[t * K + i] at most
    // 2-way bank conflicted
    const int K = ((n + NT - 1) / NT) | 1;
    const int i0 = min(n, t * K), i1 = min(n, i0 + K);
    for (int bit = lo; bit < lo + nbits; bit += kRadixBits) {
#pragma unroll
        for (int d = 0; d < D; ++d) hist[hpad(d * NT + t)] = 0;
        for (int i = i0; i < i1; ++i) hist[hpad((int)((uint32_t)(a[i] >> bit) & (D - 1)) * NT + t)]++;
        __syncthreads();
        // exclusive scan of hist in (digit, thread) order; thread t owns D entries
        uint32_t loc[D], sum = 0;
#pragma unroll
        for (int q = 0; q < D; ++q) { loc[q] = hist[hpad(D * t + q)]; sum += loc[q]; }
        uint32_t total;
        uint32_t pre = block_excl_scan<NT>(sum, wsum, total);
#pragma unroll
        for (int q = 0; q < D; ++q) { hist[hpad(D * t + q)] = pre; pre += loc[q]; }
        __syncthreads();
        for (int i = i0; i < i1; ++i) {
            const uint64_t v = a[i];
            b[hist[hpad((int)((uint32_t)(v >> bit) & (D - 1)) * NT + t)]++] = v;
        }
        __syncthreads();
        uint64_t *tmp = a; a = b; b = tmp;
    }
    return a;
}

// Sort of n (<= kDenseCap) 64-bit keys (id << 16 | payload) by id, ids
// distinct: one bucket pass over the ids' actual range, then each key's place
// inside its bucket by counting the smaller ids there.  Keys whose ids bunch
// into a few buckets (more than kBucketMax in one) go to the radix sort
// instead, so the result never depends on the id distribution and the cost
// never grows quadratically.  NT threads; `cnt` holds kRadixWords(NT) >=
// kBuckets + 1 words.
// Returns the buffer that holds the sorted keys.
constexpr int kBuckets = 512;
constexpr int kBucketMax = 24;
static_assert(kRadixWords(128) >= kBuckets + 1, "the bucket counters fit the radix table");

template <int NT>
__device__ uint64_t *block_bucket_sort(uint64_t *a, uint64_t *b, uint32_t *cnt, int n, int id_bits)
{
    static_assert(kBuckets % NT == 0, "buckets per thread");
    constexpr int kPer = kBuckets / NT;
    __shared__ uint32_t red[2][NT / 32];
    __shared__ uint32_t info[2];  // id shift, largest bucket
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    // the ids' range
    uint32_t mn = 0xffffffffu, mx = 0;
    for (int i = t; i < n; i += NT) {
        const uint32_t id = (uint32_t)(a[i] >> 16);
        mn = min(mn, id);
        mx = max(mx, id);
    }
    mn = __reduce_min_sync(0xffffffffu, mn);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) { red[0][wid] = mn; red[1][wid] = mx; }
    for (int i = t; i <= kBuckets; i += NT) cnt[i] = 0;
    __syncthreads();
    mn = red[0][0];
    mx = red[1][0];
#pragma unroll
    for (int w = 1; w < NT / 32; ++w) { mn = min(mn, red[0][w]); mx = max(mx, red[1][w]); }
    // bucket = (id - mn) >> shift, shift the least with range >> shift < kBuckets
    const uint32_t range = n > 0 ? mx - mn : 0;
    const int shift = range < (uint32_t)kBuckets ? 0 : 32 - __clz(range) - 9;  // kBuckets = 2^9
    // each key's rank among its bucket's arrivals, and the bucket counts
    uint32_t rk[kDenseCap / NT], bk[kDenseCap / NT];
#pragma unroll
    for (int r = 0; r < kDenseCap / NT; ++r) {
        const int i = t + r * NT;
        if (i < n) {
            bk[r] = ((uint32_t)(a[i] >> 16) - mn) >> shift;
            rk[r] = atomicAdd(&cnt[bk[r]], 1u);
        }
    }
    __syncthreads();
    // exclusive scan of the counts; the largest bucket
    uint32_t loc[kPer], sum = 0, big = 0;
#pragma unroll
    for (int q = 0; q < kPer; ++q) { loc[q] = cnt[t * kPer + q]; sum += loc[q]; big = max(big, loc[q]); }
    big = __reduce_max_sync(0xffffffffu, big);
    if (lane == 0) red[1][wid] = big;
    uint32_t total;
    uint32_t pre = block_excl_scan<NT>(sum, red[0], total);
#pragma unroll
    for (int q = 0; q < kPer; ++q) { cnt[t * kPer + q] = pre; pre += loc[q]; }
    if (t == 0) {
        uint32_t m = 0;
#pragma unroll
        for (int w = 0; w < NT / 32; ++w) m = max(m, red[1][w]);
        info[1] = m;
    }
    if (t == NT - 1) cnt[kBuckets] = pre;
    __syncthreads();
    if (info[1] > (uint32_t)kBucketMax) return block_radix_sort<NT>(a, b, cnt, n, 16, id_bits);
    // file the keys by bucket, then place each inside its bucket
#pragma unroll
    for (int r = 0; r < kDenseCap / NT; ++r) {
        const int i = t + r * NT;
        if (i < n) b[cnt[bk[r]] + rk[r]] = a[i];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kDenseCap / NT; ++r) {
        const int i = t + r * NT;
        if (i < n) {
            const uint32_t b0 = cnt[bk[r]], b1 = cnt[bk[r] + 1];
            const uint64_t key = b[b0 + rk[r]];
            const uint32_t id = (uint32_t)(key >> 16);
            uint32_t below = 0;
            for (uint32_t j = b0; j < b1; ++j) below += (uint32_t)(b[j] >> 16) < id;
            a[b0 + below] = key;
        }
    }
    __syncthreads();
    return a;
}

constexpr int kDT = 128;                       // threads of k_grid_dense
constexpr int kDenseKT = kDenseCap / kDT;      // candidates per thread when the list is full

constexpr int kMaxCuts = 32;                   // id windows of a huge cell planned at once

// A warp's ring of filter hits: an iteration adds at most 64 to fewer than 32.
constexpr int kHitRing = 128;
// Columns of a warp's staged summands, padded so that the nine rows' 16-byte
// reads fall into different banks.
constexpr int kSumCols = 36;

// Shared memory of k_grid_dense.  Regions whose lifetimes do not overlap
// share storage: the sort keys become the id-ordered candidate array, and the
// gather slots and sort counters become the warps' staged summands.
struct DenseSmem {
    union {
        uint64_t keys[2][kDenseCap];  // (id << 16) | (segment << 11) | gather index
        float4 spos[kDenseCap];       // candidates in id order, periodic images; w = slot
    } u;
    union {
        struct {
            uint32_t gslot[kDenseCap];      // state slot, by gather index
            uint32_t hist[kRadixWords(kDT)];  // sort counters (block_bucket_sort, block_radix_sort)
        } s;
        __align__(16) float st[kDT / 32][9][kSumCols];  // per warp: a round's summands, by component
    } v;
    uint16_t hits[kDT / 32][kHitRing];     // per warp: filter hits (candidates), a ring
    uint32_t res[12][kDenseRound + 1];     // a round's sums and counts, by boid
    uint32_t seg_j0[18], seg_k0[19];
    float seg_s[18][3];
    // the next item, the end of those taken from the queue, all items, how many to take next
    uint32_t work, wend, wall, wtake;
    uint32_t flock;
    uint32_t nw, cut;              // huge cells: window size, histogram cut
    uint32_t wcut[kMaxCuts], nwcut, wlast;  // huge cells: planned window ends (ids), and the bins they take
    uint32_t woff[kMaxCuts + 1];           // and, when bucketed, each planned window's first scratch entry
    uint32_t wbucketed;
    uint32_t wtot[kDT / 32];       // block scan scratch
    float svx[kDenseCap], svy[kDenseCap], svz[kDenseCap];  // candidates' velocities, id order
    // candidates' coordinates relative to the cell centre, scaled by hsc, in
    // half precision, two candidates per word (one pad entry for odd counts)
    __half2 hx[kDenseCap / 2 + 1], hy[kDenseCap / 2 + 1], hz[kDenseCap / 2 + 1];
    StepConst kf;  // the current cell's flock (batched ensembles)
};
static_assert(kDenseCap <= 2048, "gather index must fit 11 bits");

// The candidates of the id-ordered list hold their periodic images as seen
// from the cell, exactly as the reference computes them: a candidate of a
// segment across a periodic face is shifted by the field size on that axis
// ((float)((double)x -+ F)), the others are unshifted.  That is the
// reference's own minimum image for every pair it can accept: such a pair is
// nearer than the largest sight radius R, which is at most F/3 (at least 3
// device cells per axis), so across a face the reference's test
// |xj - xi| > F/2 holds (|xj - xi| > F - R) and inside the field it fails
// (|xj - xi| < R).  Where the reference images a candidate otherwise, it is
// farther than R from the boid in both placements and no rule accepts it.

// Id window of a huge cell (more than kDenseCap candidates): the largest hi
// such that the candidates with ids in [lo, hi) fit the shared list.  A
// histogram of the candidates' ids over kWinBins bins is cut where the
// running count passes kDenseCap; if the first bin alone is over, the span
// narrows to that bin.  A boid is a candidate at most once (G >= 3), so a
// bin one id wide always fits and the search ends.
constexpr int kWinBins = 1024;

__device__ uint32_t dense_window(DenseSmem &sm, const GridIn &g, int ns, uint32_t lo, uint32_t nid)
{
    static_assert(kWinBins * 4 <= sizeof(sm.u.keys[0]), "window histogram lives in the first sort buffer");
    static_assert(kWinBins % kDT == 0, "bins per thread");
    constexpr int kPer = kWinBins / kDT;
    uint32_t *hist = reinterpret_cast<uint32_t *>(sm.u.keys[0]);
    const int t = threadIdx.x;
    uint32_t span_hi = nid;
    for (;;) {
        const uint32_t w = (span_hi - lo + kWinBins - 1) / kWinBins;
        for (int i = t; i < kWinBins; i += kDT) hist[i] = 0;
        if (t == 0) sm.cut = kWinBins;
        __syncthreads();
        for (int sgi = 0; sgi < ns; ++sgi) {
            const uint32_t j0 = sm.seg_j0[sgi], len = sm.seg_k0[sgi + 1] - sm.seg_k0[sgi];
            for (uint32_t q = t; q < len; q += kDT) {
                const uint32_t id = __float_as_uint(__ldg(&g.pos[j0 + q].w));
                if (id >= lo && id < span_hi) atomicAdd(&hist[(id - lo) / w], 1u);
            }
        }
        __syncthreads();
        uint32_t loc = 0;
#pragma unroll 8
        for (int i = 0; i < kPer; ++i) loc += hist[t * kPer + i];
        uint32_t total;
        uint32_t run = block_excl_scan<kDT>(loc, sm.wtot, total);
        if (run + loc > (uint32_t)kDenseCap) {
            for (int i = 0; i < kPer; ++i) {
                run += hist[t * kPer + i];
                if (run > (uint32_t)kDenseCap) {
                    atomicMin(&sm.cut, (uint32_t)(t * kPer + i));
                    break;
                }
            }
        }
        __syncthreads();
        const uint32_t cut = sm.cut;
        __syncthreads();  // hist and cut are rewritten next
        if (cut >= (uint32_t)kWinBins) return span_hi;
        if (cut > 0) return lo + cut * w;
        span_hi = lo + w;  // w > 1 here: a one-id bin holds at most one candidate
    }
}

// The next id windows of a huge cell, from id lo, planned from one histogram of
// its candidates' ids (kWinBins bins, so narrow that one holds a quarter of the
// list where ids are spread evenly): window ends are cut greedily where the
// running count would pass kDenseCap, at most kMaxCuts of them; when they are
// done, the next are planned.  A window that begins with a bin that alone
// overflows the list is cut by dense_window instead.  One histogram pass
// for all windows, where dense_window needs one per window.  With a scratch
// of cap entries (this CTA's) that holds the planned windows, a second pass
// files the candidates by bin, and each planned window is then read from
// the scratch instead of scanning the whole neighbourhood again; an entry is
// id << 34 | segment << 29 | slot.
__device__ void dense_window_plan(DenseSmem &sm, const GridIn &g, int ns, uint32_t lo, uint32_t nid,
                                  uint64_t *scratch, uint32_t cap)
{
    static_assert((kWinBins + 1) * 4 <= sizeof(sm.u), "the prefix counts live in the sort buffers");
    static_assert(kWinBins % kDT == 0, "bins per thread");
    constexpr int kPer = kWinBins / kDT;
    uint32_t *hist = reinterpret_cast<uint32_t *>(&sm.u);
    const int t = threadIdx.x;
    const uint32_t even = (uint32_t)((uint64_t)nid * (kDenseCap / 4) / sm.seg_k0[ns]);
    const uint32_t w = max(1u, min((nid - lo + kWinBins - 1) / kWinBins, even));  // ids of a bin
    for (int i = t; i <= kWinBins; i += kDT) hist[i] = 0;
    __syncthreads();
    for (int sgi = 0; sgi < ns; ++sgi) {
        const uint32_t j0 = sm.seg_j0[sgi], len = sm.seg_k0[sgi + 1] - sm.seg_k0[sgi];
        for (uint32_t q = t; q < len; q += kDT) {
            const uint32_t id = __float_as_uint(__ldg(&g.pos[j0 + q].w)), bin = (id - lo) / w;
            if (id >= lo && bin < (uint32_t)kWinBins) atomicAdd(&hist[bin], 1u);
        }
    }
    __syncthreads();
    // exclusive prefix: hist[b] = candidates in bins below b, hist[kWinBins] in all bins
    uint32_t loc[kPer], sum = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i) { loc[i] = hist[t * kPer + i]; sum += loc[i]; }
    uint32_t total;
    uint32_t pre = block_excl_scan<kDT>(sum, sm.wtot, total);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kPer; ++i) { hist[t * kPer + i] = pre; pre += loc[i]; }
    if (t == kDT - 1) hist[kWinBins] = pre;
    __syncthreads();
    if (t == 0) {
        uint32_t start = 0, nc = 0;
        while (start < (uint32_t)kWinBins && nc < (uint32_t)kMaxCuts) {
            const uint32_t target = hist[start] + (uint32_t)kDenseCap;
            uint32_t lo_b = start, hi_b = kWinBins + 1;  // hist[lo_b] <= target < hist[hi_b]
            while (hi_b - lo_b > 1) {
                const uint32_t mid = (lo_b + hi_b) / 2;
                if (hist[mid] <= target) lo_b = mid; else hi_b = mid;
            }
            if (lo_b == start) break;  // bin `start` alone holds more than the list
            sm.wcut[nc++] = min(nid, lo + lo_b * w);
            sm.woff[nc] = hist[lo_b];
            start = lo_b;
        }
        sm.nwcut = nc;
        sm.wlast = start;
        sm.woff[0] = 0;
        // bucket the planned windows' candidates when the scratch holds them
        sm.wbucketed = nc > 0 && scratch != nullptr && sm.woff[nc] <= cap;
    }
    __syncthreads();
    if (!sm.wbucketed) return;
    // File every candidate of the planned windows at its bin's next entry
    // (the prefix counts become running ends): a window is then the
    // contiguous run woff[c] .. woff[c + 1] of the scratch, in bin order.
    const uint32_t last_bin = sm.wlast;
    for (int sgi = 0; sgi < ns; ++sgi) {
        const uint32_t j0 = sm.seg_j0[sgi], len = sm.seg_k0[sgi + 1] - sm.seg_k0[sgi];
        for (uint32_t q = t; q < len; q += kDT) {
            const uint32_t slot = j0 + q;
            const uint32_t id = __float_as_uint(__ldg(&g.pos[slot].w));
            const uint32_t bin = (id - lo) / w;
            if (id >= lo && bin < last_bin)
                scratch[atomicAdd(&hist[bin], 1u)] = ((uint64_t)id << 34) | ((uint64_t)sgi << 29) | slot;
        }
    }
    __syncthreads();
}

// One CTA takes a work item or a few at a time (dynamic queue): a crowded cell
// and about kDenseItem of its boids (a cell with more boids is several items,
// taken by several CTAs, or done together by one).  The cell's 27-cell
// candidates are sorted by id, once for the items done together.  Then each
// warp takes a boid at a time: its lanes filter the list in half precision, 64 candidates an iteration, the hits are compacted into
// the warp's queue, 32 of them at a time take the exact tests, and the
// accepted, compacted again, are added up by nine lanes, one component of the
// three rules' sums each.  The list is in id order and every compaction keeps
// it, so the sums are in ascending id, as the reference accumulates.  A cell
// with more than kDenseCap candidates is done in ascending id windows that
// each fit the list; the sums are carried from window to window through
// o.carry.
//
// Bound by instruction issue (76 % of the slots at 8 CTAs per SM, N = 2^20
// after 1000 updates: 2.20 ms).  A warp per boid replaced a lane per (boid, chunk of
// candidates) with rule masks and a lane per sum: that form needed a round of
// up to 72 boids to fill its lanes, so items held up to 128 boids and a small
// flock's few items left most SMs idle.  Items of 32 boids and no barrier
// between a boid's filter and its sums took a step of 1000 boids of test.ini
// from 209 to 108 us, of gathered flocks of 16 384 boids from 250 to 188 us,
// of 65 537 from 376 to 264, of 262 143 from 697 to 603 and of 2^20 from 2350
// to 2228 (alternating runs of both builds on one GB300).
template <bool DIAG, bool MULTI>
__global__ void __launch_bounds__(kDT, kDenseCtasPerSm)
k_grid_dense(GridIn g, GridOut o, const uint32_t *__restrict__ dense_list, uint32_t *__restrict__ dense_n,
             StepConst kp, FlockTable ft)
{
    extern __shared__ __align__(16) unsigned char dense_smem_raw[];
    DenseSmem &sm = *reinterpret_cast<DenseSmem *>(dense_smem_raw);
    const int t = threadIdx.x;
    if (g.chain) chain_wait();
    // how many items to take next, from those that are left: several while the
    // CTAs have many to come, one by one towards the end
    auto take_of = [&](uint32_t left) { return min(max(left / (kDenseLeft * gridDim.x), 1u), kDenseTake); };
    if (t == 0) {
        sm.work = sm.wend = 0;
        sm.wall = dense_n[0];
        sm.wtake = take_of(sm.wall);
    }
    for (;;) {
        if (t == 0 && sm.work >= sm.wend) {  // the next items from the queue
            const uint32_t take = sm.wtake, first = atomicAdd(dense_n + 1, take), all = sm.wall;
            sm.work = first;
            sm.wend = min(all, first + take);
            sm.wtake = take_of(all - min(all, first + take * gridDim.x));  // when the other CTAs have taken as many
        }
        __syncthreads();
        const uint32_t w = sm.work, wend = sm.wend;
        if (w >= wend) break;
        const uint32_t cg = dense_list[2 * w];        // global full-size cell
        const uint32_t rbeg = dense_list[2 * w + 1];  // the items' first boid of the cell
        uint32_t run = 1;                             // items of that cell, done together
#pragma unroll
        for (uint32_t q = 1; q < kDenseTake; ++q)
            if (w + q < wend && dense_list[2 * (w + q)] == cg) run = q + 1;
        if (MULTI) {
            if (t == 0) {  // the flock: last with cell4 <= cg
                uint32_t lo = 0, hi = ft.count;
                while (hi - lo > 1) {
                    const uint32_t mid = (lo + hi) / 2;
                    if (__ldg(ft.cell4 + mid) <= cg) lo = mid; else hi = mid;
                }
                sm.flock = lo;
            }
            __syncthreads();
            load_flock(sm.kf, ft, sm.flock);
        }
        const StepConst &k = MULTI ? sm.kf : kp;
        const uint32_t c = cg - k.cell_base / 4;  // full-size cell inside the flock
        const int G = k.G;
        const int cx = (int)(c % G), cy = (int)((c / G) % G), cz = (int)(c / ((uint32_t)G * G));
        const int runs = seg_runs(cx, k), ns = 9 * runs;
        if (t < 32) {  // the segments, and their starts in the gather order (a warp scan of their lengths)
            uint32_t len = 0;
            if (t < ns) {
                const Seg sg = segment(cx, cy, cz, t, runs, k);
                const uint32_t j0 = slot_start(g.lstart, g.bsum, k.cell_base + sg.c0, k);
                len = slot_start(g.lstart, g.bsum, k.cell_base + sg.c1, k) - j0;
                sm.seg_j0[t] = j0;
                sm.seg_s[t][0] = sg.sx; sm.seg_s[t][1] = sg.sy; sm.seg_s[t][2] = sg.sz;
            }
            uint32_t incl = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (t >= o) incl += y;
            }
            if (t < ns) sm.seg_k0[t + 1] = incl;
            if (t == 0) sm.seg_k0[0] = 0;
        }
        __syncthreads();
        const uint32_t ncand = sm.seg_k0[ns];
        const uint32_t own0 = slot_start(g.lstart, g.bsum, 4 * cg, k);
        const uint32_t b = slot_start(g.lstart, g.bsum, 4 * cg + 4, k) - own0;
        const bool huge = ncand > (uint32_t)kDenseCap;
        if (huge && !o.carry) {  // not listed so by k_grid_classify; kept for safety
            __syncthreads();
            if (t == 0) sm.work = w + run;
            continue;
        }

        uint32_t lo = 0;  // this window's ids: [lo, hi)
        uint32_t wi = 0;  // windows of the present plan that are done (0: one is due)
        for (;;) {
            uint32_t hi = k.n, nw = ncand;
            if (huge) {
                if (wi == 0)
                    dense_window_plan(sm, g, ns, lo, k.n,
                                      o.wscratch ? o.wscratch + (size_t)blockIdx.x * o.wcap : nullptr, o.wcap);
                const bool planned = wi < sm.nwcut;
                hi = planned ? sm.wcut[wi] : dense_window(sm, g, ns, lo, k.n);
                // gather the window's (id, segment, gather index) keys
                if (planned && sm.wbucketed) {  // its run of the scratch
                    const uint64_t *run = o.wscratch + (size_t)blockIdx.x * o.wcap + sm.woff[wi];
                    const uint32_t len = sm.woff[wi + 1] - sm.woff[wi];
                    for (uint32_t q = t; q < len; q += kDT) {
                        const uint64_t e = __ldcg(run + q);
                        sm.v.s.gslot[q] = (uint32_t)e & 0x1fffffffu;
                        sm.u.keys[0][q] = ((e >> 34) << 16) | (((uint32_t)(e >> 29) & 0x1fu) << 11) | q;
                    }
                    if (t == 0) sm.nw = len;
                } else {  // a scan of the whole neighbourhood for the window's ids
                    if (t == 0) sm.nw = 0;
                    __syncthreads();
                    for (int sgi = 0; sgi < ns; ++sgi) {
                        const uint32_t j0 = sm.seg_j0[sgi], len = sm.seg_k0[sgi + 1] - sm.seg_k0[sgi];
                        for (uint32_t q = t; q < len; q += kDT) {
                            const uint32_t slot = j0 + q;
                            const uint32_t id = __float_as_uint(__ldg(&g.pos[slot].w));
                            if (id >= lo && id < hi) {
                                const uint32_t qq = atomicAdd(&sm.nw, 1u);
                                sm.v.s.gslot[qq] = slot;
                                sm.u.keys[0][qq] = ((uint64_t)id << 16) | ((uint32_t)sgi << 11) | qq;
                            }
                        }
                    }
                }
                wi = wi + 1 < sm.nwcut ? wi + 1 : 0;
                __syncthreads();
                nw = sm.nw;
            } else {
                // gather every candidate's (id, segment, gather index) key; a
                // thread's q only grows, so its segment search goes on from
                // where the last one stopped
                uint32_t sgi = 0;
                for (uint32_t q = t; q < ncand; q += kDT) {
                    while (q >= sm.seg_k0[sgi + 1]) ++sgi;
                    const uint32_t slot = sm.seg_j0[sgi] + (q - sm.seg_k0[sgi]);
                    sm.v.s.gslot[q] = slot;
                    sm.u.keys[0][q] = ((uint64_t)__float_as_uint(__ldg(&g.pos[slot].w)) << 16) | (sgi << 11) | q;
                }
                __syncthreads();
            }
            const uint64_t *sorted =
                block_bucket_sort<kDT>(sm.u.keys[0], sm.u.keys[1], sm.v.s.hist, (int)nw, k.id_bits);
            // lay the candidates out in id order over the dead sort buffers
            // (thread t takes positions t, t + kDT, ...: no bank conflicts)
            const float3 cen = make_float3(((float)cx + 0.5f) * k.side, ((float)cy + 0.5f) * k.side,
                                           ((float)cz + 0.5f) * k.side);
            uint32_t slot_r[kDenseKT], seg_r[kDenseKT];
#pragma unroll
            for (int i = 0; i < kDenseKT; ++i) {
                const int q = t + i * kDT;
                if (q < (int)nw) {
                    const uint64_t key = sorted[q];
                    slot_r[i] = sm.v.s.gslot[(uint32_t)key & 0x7ffu];
                    seg_r[i] = ((uint32_t)key >> 11) & 0x1fu;
                }
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < kDenseKT; ++i) {
                const int q = t + i * kDT;
                if (q < (int)nw) {
                    const float4 p = __ldg(g.pos + slot_r[i]);
                    const float *sh = sm.seg_s[seg_r[i]];
                    // the candidate's periodic image as the reference computes
                    // it, (float)((double)x -+ F) on each shifted axis
                    float4 im = make_float4(p.x, p.y, p.z, __uint_as_float(slot_r[i]));
                    if (sh[0] != 0.f) im.x = add_f32_f64_rn(p.x, k.Fsd, sh[0] < 0.f);
                    if (sh[1] != 0.f) im.y = add_f32_f64_rn(p.y, k.Fsd, sh[1] < 0.f);
                    if (sh[2] != 0.f) im.z = add_f32_f64_rn(p.z, k.Fsd, sh[2] < 0.f);
                    sm.u.spos[q] = im;
                    const float4 v = __ldg(g.vel + slot_r[i]);
                    sm.svx[q] = v.x;
                    sm.svy[q] = v.y;
                    sm.svz[q] = v.z;
                    const float4 cq = sm.u.spos[q];
                    reinterpret_cast<__half *>(sm.hx)[q] = __float2half_rn((cq.x - cen.x) * k.hsc);
                    reinterpret_cast<__half *>(sm.hy)[q] = __float2half_rn((cq.y - cen.y) * k.hsc);
                    reinterpret_cast<__half *>(sm.hz)[q] = __float2half_rn((cq.z - cen.z) * k.hsc);
                }
            }
            if (t == 0 && (nw & 1)) {  // pad the last pair with a candidate far out of reach
                reinterpret_cast<__half *>(sm.hx)[nw] = __float2half_rn(30000.f);
                reinterpret_cast<__half *>(sm.hy)[nw] = __float2half_rn(30000.f);
                reinterpret_cast<__half *>(sm.hz)[nw] = __float2half_rn(30000.f);
            }
            __syncthreads();
            const bool first = lo == 0, last = hi >= k.n;

            // A warp per boid of the item.  The candidates are in id order, so the
            // filter's hits, the accepted among them and their summands are too.
            const uint32_t npairs = (nw + 1) / 2;
            const int lane = t & 31, wid = t >> 5;
            const unsigned below = (1u << lane) - 1u;
            uint16_t *hits = sm.hits[wid];
            float(&st)[9][kSumCols] = sm.v.st[wid];
            const uint32_t iend = min(b, rbeg + run * dense_per_item(b, ncand, g.share));
            for (uint32_t r0 = rbeg; r0 < iend; r0 += kDenseRound) {  // a round's results at a time
                const uint32_t rend = min(iend, r0 + (uint32_t)kDenseRound);
                for (uint32_t i = r0 + wid; i < rend; i += kDT / 32) {
                    const uint32_t s = own0 + i;
                    const float3 pi = xyz(__ldg(g.pos + s));
                    const Sight si = make_sight(xyz(__ldg(g.vel + s)));
                    // lane c < 9: component c of (cohesion, separation, alignment)
                    float acc = 0.f;
                    int ncoh = 0, nsep = 0, nali = 0;
                    uint64_t h0 = 0, h1 = 0, h2 = 0;
                    if (!first) {  // the earlier id windows' sums
                        const Acc *cin = o.carry + s;
                        if (lane < 9) acc = reinterpret_cast<const float *>(cin)[lane];
                        ncoh = cin->ncoh;
                        nsep = cin->nsep;
                        nali = cin->nali;
                    }
                    // The filter in half precision, two candidates per instruction:
                    // it keeps every pair within the filter radius and drops only
                    // pairs whose exact v . r is negative (the bounds are in hfilt,
                    // hdot0 and hdot1); the exact tests decide the rest.
                    const __half2 bx = __float2half2_rn((pi.x - cen.x) * k.hsc);
                    const __half2 by = __float2half2_rn((pi.y - cen.y) * k.hsc);
                    const __half2 bz = __float2half2_rn((pi.z - cen.z) * k.hsc);
                    const float vt = si.nv * k.hvsc;
                    const bool pre = k.cone_pre && vt <= 1.0f;
                    const __half2 hvx = __float2half2_rn(pre ? si.v.x * k.hvsc : 0.f);
                    const __half2 hvy = __float2half2_rn(pre ? si.v.y * k.hvsc : 0.f);
                    const __half2 hvz = __float2half2_rn(pre ? si.v.z * k.hvsc : 0.f);
                    const __half2 hf2 = __half2half2(__float2half_ru(k.hfilt));
                    const __half2 hd2 = __half2half2(pre ? __float2half_rd(-(k.hdot0 + k.hdot1 * vt))
                                                         : __ushort_as_half((unsigned short)0xfc00u));  // -inf
                    uint32_t qh = 0, nq = 0;  // the ring's head and length, the same in every lane
                    for (uint32_t p0 = 0; p0 < npairs; p0 += 32) {
                        const uint32_t pp = p0 + lane;
                        unsigned keep = 0;
                        if (pp < npairs) {
                            const __half2 dx = __hsub2(sm.hx[pp], bx), dy = __hsub2(sm.hy[pp], by),
                                          dz = __hsub2(sm.hz[pp], bz);
                            const __half2 d2 = __hfma2(dz, dz, __hfma2(dy, dy, __hmul2(dx, dx)));
                            const __half2 dv = __hfma2(hvz, dz, __hfma2(hvy, dy, __hmul2(hvx, dx)));
                            keep = __hlt2_mask(d2, hf2) & __hge2_mask(dv, hd2);
                        }
                        const bool e0 = keep & 1u, e1 = keep >> 16;
                        const unsigned m0 = __ballot_sync(0xffffffffu, e0), m1 = __ballot_sync(0xffffffffu, e1);
                        uint32_t at = qh + nq + __popc(m0 & below) + __popc(m1 & below);
                        if (e0) hits[at++ & (kHitRing - 1)] = (uint16_t)(2 * pp);
                        if (e1) hits[at & (kHitRing - 1)] = (uint16_t)(2 * pp + 1);
                        nq += __popc(m0) + __popc(m1);
                        // exact tests of 32 hits at a time, and the sums of those accepted;
                        // the last pairs' hits whatever their number
                        const uint32_t enough = p0 + 32 < npairs ? 32u : 1u;
                        while (nq >= enough) {
                            __syncwarp();
                            int f = 0;
                            float4 cq = make_float4(0.f, 0.f, 0.f, 0.f);
                            uint32_t q = 0;
                            if ((uint32_t)lane < nq) {
                                q = hits[(qh + lane) & (kHitRing - 1)];
                                cq = sm.u.spos[q];
                                if (__float_as_uint(cq.w) != s) f = pair_flags(pi, si, xyz(cq), k);
                            }
                            const uint32_t done = min(nq, 32u);
                            qh += done;
                            nq -= done;
                            const unsigned am = __ballot_sync(0xffffffffu, f != 0);
                            if (!am) continue;
                            const int m = __popc(am);
                            const bool co = f & 1, se = f & 2, al = f & 4;
                            const unsigned cm = __ballot_sync(0xffffffffu, co), em = __ballot_sync(0xffffffffu, se),
                                           lm = __ballot_sync(0xffffffffu, al);
                            ncoh += __popc(cm);
                            nsep += __popc(em);
                            nali += __popc(lm);
                            // Column by column, lanes 0-8 add the accepted up, a component
                            // each.  A rule that did not accept a neighbour adds +0, which
                            // leaves a float sum that started at +0 unchanged (it is never
                            // -0): every sum is the reference's sequence of additions.
                            if (f) {
                                const int c = __popc(am & below);
                                st[0][c] = co ? cq.x : 0.f;
                                st[1][c] = co ? cq.y : 0.f;
                                st[2][c] = co ? cq.z : 0.f;
                                st[6][c] = al ? sm.svx[q] : 0.f;
                                st[7][c] = al ? sm.svy[q] : 0.f;
                                st[8][c] = al ? sm.svz[q] : 0.f;
                                if (em) {
                                    float3 u = make_float3(0.f, 0.f, 0.f);
                                    if (se) {  // Vector3D::normalized of pi - t
                                        const float dx = __fsub_rn(pi.x, cq.x), dy = __fsub_rn(pi.y, cq.y),
                                                    dz = __fsub_rn(pi.z, cq.z);
                                        const float n = nrm3(dx, dy, dz);
                                        u = make_float3(__fdiv_rn(dx, n), __fdiv_rn(dy, n), __fdiv_rn(dz, n));
                                    }
                                    st[3][c] = u.x;
                                    st[4][c] = u.y;
                                    st[5][c] = u.z;
                                }
                                if (DIAG) {
                                    const uint64_t h = id_hash(__float_as_uint(__ldg(&g.pos[__float_as_uint(cq.w)].w)));
                                    if (co) h0 += h;
                                    if (se) h1 += h;
                                    if (al) h2 += h;
                                }
                            }
                            // columns m .. up to a multiple of four: +0
                            const int pad = (4 - m) & 3;
                            if (lane < 9 * 4 && (lane & 3) < pad) st[lane >> 2][m + (lane & 3)] = 0.f;
                            if (lane < pad) st[8][m + lane] = 0.f;
                            __syncwarp();
                            if (lane < 9 && (em || lane < 3 || lane >= 6)) {
                                const float *row = st[lane];
                                for (int c = 0; c < m; c += 4) {
                                    const float4 x = *reinterpret_cast<const float4 *>(row + c);
                                    acc = __fadd_rn(acc, x.x);
                                    acc = __fadd_rn(acc, x.y);
                                    acc = __fadd_rn(acc, x.z);
                                    acc = __fadd_rn(acc, x.w);
                                }
                            }
                            __syncwarp();
                        }
                    }
                    const uint32_t word = lane < 9 ? __float_as_uint(acc)
                                                   : (uint32_t)(lane == 9 ? ncoh : (lane == 10 ? nsep : nali));
                    if (DIAG) {
#pragma unroll
                        for (int q = 16; q > 0; q >>= 1) {
                            h0 += __shfl_xor_sync(0xffffffffu, h0, q);
                            h1 += __shfl_xor_sync(0xffffffffu, h1, q);
                            h2 += __shfl_xor_sync(0xffffffffu, h2, q);
                        }
                        if (lane == 0) {
                            uint64_t *hs =
                                last ? o.dhash + 3 * (size_t)(__float_as_uint(g.pos[s].w) + (k.slot_base - k.slot_off))
                                     : o.carry[s].h;
                            const uint64_t *hc = first ? nullptr : o.carry[s].h;
                            hs[0] = h0 + (hc ? hc[0] : 0);
                            hs[1] = h1 + (hc ? hc[1] : 0);
                            hs[2] = h2 + (hc ? hc[2] : 0);
                        }
                        if (last && lane >= 9 && lane < 12)
                            o.dcnt[3 * (size_t)(__float_as_uint(g.pos[s].w) + (k.slot_base - k.slot_off)) + lane - 9] =
                                (int)word;
                    }
                    if (lane < 12) {
                        if (!last) reinterpret_cast<uint32_t *>(o.carry + s)[lane] = word;
                        else if (!DIAG) sm.res[lane][i - r0] = word;
                    }
                }
                __syncthreads();  // the list is free, the results are written
                if (!DIAG && last && (uint32_t)t < rend - r0) {
                    const uint32_t s = own0 + r0 + t;
                    Acc a;
                    uint32_t *aw = reinterpret_cast<uint32_t *>(&a);
#pragma unroll
                    for (int c = 0; c < 12; ++c) aw[c] = sm.res[c][t];
                    finish_boid<DIAG>(a, g.pos[s], xyz(g.vel[s]), s, o, k);
                }
                if (last && rend < iend) __syncthreads();  // the results are read
            }
            if (last) break;
            lo = hi;
        }
        if (t == 0) sm.work = w + run;
    }
}

// ------------------------------------------------------------------ all-pairs engine

// Every ordered pair is tested by a filter that is a matrix product.  A boid's
// coordinates become the cosines and sines of 2 pi x / F, 2 pi y / F and
// 2 pi z / F: six half-precision values whose inner product with another
// boid's is the sum over the axes of cos(2 pi (xi - xj) / F), which is periodic
// by itself, with no minimum image to take.  A pair within the radius r has a
// sum of at least 3 - (2 pi r / F)^2 / 2; StepConst::ap_min is that less the
// rounding's bound, so the filter drops no pair the exact tests accept (it
// keeps a ball of about 1.05 r at r = F / 32).  Two further terms, w_i * 1 and
// 1 * u_j, subtract ap_min (w + u = -ap_min, u the rounding of w), and pass
// every pair of a boid so far outside the field (over 4 F) that its angles are
// not exact enough.
//
// 64 boids a warp against 8 at a time: four mma.m16n8k8, and an AND over their
// 16 results a lane, whose sign says whether any pair passed.  Survivors are
// queued per warp and take the exact tests 32 at a time; accepted neighbours are
// appended to the boid's list (unordered).
//
// Bound by the tensor pipe and the work on its results (68 % and, on the ALU,
// 65 % busy, 62 % of the issue slots): 1024 pairs take 58 warp instructions,
// where a box filter on the FP32 offsets took 15.7 per pair and thread.
// N = 65 536, F = 1.6: an update takes 0.411 ms from a uniform start (1.82 with
// that filter), 1.0e13 pairs/s, and 0.452 over the next 60; 65 537 boids 0.412 (0.674 with a last tile's missing rows not
// rejected by the product).  Only the j tile of a step in which some pair passed
// is looked through: 0.427 ms with both before the last change, 0.415 with it.  One code path tests the queue: inlined at each of the 32
// results it cost 0.1 ms in instruction fetches.  mma.sync serves better than
// tcgen05 here: the product is eight deep and every one of its N^2 results has
// to come back through registers to be compared, so the tensor rate is not
// what counts.
constexpr int kApThreads = 128;
constexpr int kApTilesM = 4;                                  // 16-boid tiles of a warp
constexpr int kApWarpI = 16 * kApTilesM;                      // its boids i
constexpr int kApTileI = kApWarpI * (kApThreads / 32);        // 256
constexpr int kApTileJ = 1024;                                // most boids j of a CTA
static_assert(kApCap <= kWarpList, "k_ap_accumulate orders a boid's list in shared memory");

// A boid's filter vector: per axis (cos, sin), then (w, u).
__global__ void k_ap_embed(const float4 *__restrict__ pos, uint4 *__restrict__ emb, uint32_t n, StepConst k)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = pos[i];
    const float far = fmaxf(fmaxf(fabsf(p.x), fabsf(p.y)), fabsf(p.z));
    const float c[3] = {p.x, p.y, p.z};
    __half2 h[4];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        float sn = 0.f, cs = 0.f;
        if (fabsf(c[d]) <= 4.f * k.Ff) sincospif(c[d] * k.ap_turn, &sn, &cs);
        h[d] = __floats2half2_rn(cs, sn);
    }
    // (a NaN coordinate, which no rule accepts, leaves its cosine and sine zero)
    const __half w = __float2half_rn(-k.ap_min);
    const float pass = far > 4.f * k.Ff ? kApPass : 0.f, u = -k.ap_min - __half2float(w);
    h[3] = __floats2half2_rn(__half2float(w) + pass, u + pass);
    emb[i] = *reinterpret_cast<const uint4 *>(h);
}

__global__ void __launch_bounds__(kApThreads)
k_ap_pairs(const float4 *__restrict__ pos, const float4 *__restrict__ vel, const uint4 *__restrict__ emb,
           uint32_t *__restrict__ cnt, uint32_t *__restrict__ list, uint32_t cap, uint32_t tile_j, StepConst k)
{
    __shared__ uint4 sj[kApTileJ];                     // the j's vectors, (1, u) last
    __shared__ uint32_t queue[kApThreads / 32][64];    // per warp: surviving pairs, i << 10 | j in their tiles
    constexpr unsigned kAll = 0xffffffffu;
    const uint32_t n = k.n;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const unsigned below = (1u << lane) - 1u;
    const uint32_t j0 = blockIdx.y * tile_j, jn = min(tile_j, n - j0), jpad = (jn + 15) & ~15u;
    const uint32_t i0 = blockIdx.x * kApTileI + wid * kApWarpI;
    for (uint32_t q = threadIdx.x; q < jpad; q += kApThreads) {
        uint4 e = make_uint4(0, 0, 0, kApPad << 16);  // past the end: no angles, and a u that rejects every pair
        if (q < jn) e = emb[j0 + q];
        e.w = (e.w & 0xffff0000u) | 0x3c00u;
        sj[q] = e;
    }
    uint32_t a[kApTilesM][2];  // rows g and g + 8 of each tile, terms 2t and 2t + 1
    const uint32_t *ew = reinterpret_cast<const uint32_t *>(emb);
#pragma unroll
    for (int m = 0; m < kApTilesM; ++m)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint32_t i = i0 + 16 * m + 8 * r + g;
            a[m][r] = i < n ? ew[4 * (size_t)i + t] : (t == 3 ? kApPad : 0u);  // past the end: the same by its w
            if (t == 3) a[m][r] = (a[m][r] & 0xffffu) | 0x3c000000u;  // (w, 1)
        }
    __syncthreads();
    if (i0 >= n) return;
    uint32_t *q = queue[wid];
    int nq = 0;
    auto test = [&](int from, int count) {  // the exact tests of queue entries [from, from + count)
        __syncwarp();
        if (lane < count) {
            const uint32_t e = q[from + lane];
            const uint32_t i = i0 + (e >> 10), tj = e & 1023u, j = j0 + tj;
            if (i != j && i < n && tj < jn) {
                const float3 p = xyz(pos[i]);
                const Sight s = make_sight(xyz(vel[i]));
                const int f = pair_flags(p, s, image3(xyz(pos[j]), p, k), k);
                if (f) {
                    const uint32_t at = atomicAdd(cnt + i, 1u);
                    if (at < cap) list[(size_t)i * cap + at] = j | ((uint32_t)f << 29);
                }
            }
        }
        __syncwarp();
    };
    const uint32_t *bw = reinterpret_cast<const uint32_t *>(sj) + 4 * g + t;
    for (uint32_t jt = 0; jt < jpad; jt += 16) {  // two tiles of 8 j
        float d[2][kApTilesM][4];
        int all[2] = {-1, -1};  // sign set: no pair of the j tile passed
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t b = bw[4 * (jt + 8 * h)];
#pragma unroll
            for (int m = 0; m < kApTilesM; ++m) {
                float(&x)[4] = d[h][m];
                asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, "
                    "{%7, %7, %7, %7};"
                    : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3])
                    : "r"(a[m][0]), "r"(a[m][1]), "r"(b), "f"(0.f));
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int m = 0; m < kApTilesM; ++m)
#pragma unroll
                for (int r = 0; r < 4; ++r) all[h] &= __float_as_int(d[h][m][r]);
        if (!__any_sync(kAll, (all[0] & all[1]) >= 0)) continue;
        // a bit per result, the first one highest: 0 for a pair that passed
        uint32_t miss = 0xffffffffu;
        static_assert(2 * kApTilesM * 4 == 32, "a lane's results fill a word");
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (!__any_sync(kAll, all[h] >= 0)) {
                miss = (miss << 16) | 0xffffu;
                continue;
            }
#pragma unroll
            for (int m = 0; m < kApTilesM; ++m)
#pragma unroll
                for (int r = 0; r < 4; ++r) miss = __funnelshift_l(__float_as_uint(d[h][m][r]), miss, 1);
        }
        for (;;) {  // each lane's next passing pair
            const unsigned hm = __ballot_sync(kAll, ~miss != 0);
            if (!hm) break;
            if (~miss != 0) {
                const int x = __clz(~miss), r = x & 3, m = (x >> 2) & 3, h = x >> 4;
                miss |= 0x80000000u >> x;
                q[nq + __popc(hm & below)] =
                    ((uint32_t)(16 * m + (r >> 1) * 8 + g) << 10) | (jt + 8 * h + 2 * t + (r & 1));
            }
            nq += __popc(hm);
            if (nq >= 32) {
                nq -= 32;
                test(nq, 32);
            }
        }
    }
    test(0, nq);
}

// Then a warp per boid: its neighbours in id order, added up and the boid
// finished as in k_grid_warp.  A boid with more than `cap` neighbours takes
// all boids in order instead, 32 at a time.  The lists are scattered 4-byte
// stores of the pass before, whose sectors the first read fills from DRAM: a
// warp loads its next boid's record, count and first 32 entries before it
// works on the present one's (67 us at N = 65 536; 189 us with a CTA per four
// boids that waits for them).
template <bool DIAG>
__global__ void __launch_bounds__(kWarpWarps * 32, kWarpCtas)
k_ap_accumulate(const float4 *__restrict__ pos, const float4 *__restrict__ vel, uint32_t *__restrict__ cnt,
                const uint32_t *__restrict__ list, uint32_t cap, GridOut o, StepConst k)
{
    __shared__ WarpSmem sms[kWarpWarps];
    WarpSmem &sm = sms[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    const uint32_t step = gridDim.x * kWarpWarps;
    uint32_t i = blockIdx.x * kWarpWarps + (threadIdx.x >> 5);
    if (i >= k.n) return;
    float4 p4 = __ldg(pos + i), v4 = __ldg(vel + i);
    uint32_t m = cnt[i], e0 = list[(size_t)i * cap + lane];  // (entries past the count are not used)
    __syncwarp();  // every lane has its count before lane 0 clears it
    for (;;) {
        const uint32_t nx = i + step;
        float4 p_next = zero4, v_next = zero4;
        uint32_t m_next = 0, e_next = 0;
        if (nx < k.n) {
            p_next = __ldg(pos + nx);
            v_next = __ldg(vel + nx);
            m_next = cnt[nx];
            e_next = list[(size_t)nx * cap + lane];
        }
        const uint32_t *mine = list + (size_t)i * cap;
        const float3 pi = xyz(p4);
        const Sight si = make_sight(xyz(v4));
        if (lane == 0) cnt[i] = 0;  // ready for the next step
        WarpSums a{};
        if (m <= cap) {
            for (uint32_t q = lane; q < m; q += 32) {
                const uint32_t e = q < 32 ? e0 : mine[q];
                sm.lid[q] = e & 0x1fffffffu;
                sm.lsl[q] = e;
            }
            __syncwarp();
            if (m > 0) warp_order(sm, lane, (int)m);
            uint32_t e = 0;
            float4 pj = zero4, vj = zero4;
            auto load = [&](uint32_t q) {
                e = 0;
                if (q < m) {
                    e = sm.lsl[sm.ord[q]];
                    pj = __ldg(pos + (e & 0x1fffffffu));
                    vj = __ldg(vel + (e & 0x1fffffffu));
                }
            };
            load(lane);
            for (uint32_t q0 = 0; q0 < m; q0 += 32) {
                const int f = (int)(e >> 29);
                const uint32_t j = e & 0x1fffffffu;
                const float3 t = image3(xyz(pj), pi, k);
                const float4 v = vj;
                load(q0 + 32 + lane);
                warp_add<DIAG>(sm, lane, f, t, v, j, pi, a);
            }
        } else {
            for (uint32_t j0 = 0; j0 < k.n; j0 += 32) {
                const uint32_t j = j0 + lane;
                int f = 0;
                float3 t = make_float3(0.f, 0.f, 0.f);
                float4 vj = zero4;
                if (j < k.n && j != i) {
                    const float4 pj = pos[j];
                    const bool nx = fabsf(fabsf(pj.x - pi.x) - k.halfFf) > k.box_lim;
                    const bool ny = fabsf(fabsf(pj.y - pi.y) - k.halfFf) > k.box_lim;
                    const bool nz = fabsf(fabsf(pj.z - pi.z) - k.halfFf) > k.box_lim;
                    if (nx && ny && nz) {
                        t = image3(xyz(pj), pi, k);
                        f = pair_flags(pi, si, t, k);
                        if (f) vj = vel[j];
                    }
                }
                warp_add<DIAG>(sm, lane, f, t, vj, j, pi, a);
            }
        }
        warp_finish<DIAG>(a, p4, si.v, i, lane, o, k);
        if (nx >= k.n) break;
        i = nx;
        p4 = p_next;
        v4 = v_next;
        m = m_next;
        e0 = e_next;
        __syncwarp();  // the list is rewritten
    }
}

// ------------------------------------------------------------------ reference cell indices

// Boid::grid_index as update_list_grid computes it
// (src/boid_simulation_grid.cpp:400-443), written in id order.
__global__ void k_ref_cells(const float4 *__restrict__ pos, int32_t *__restrict__ cells8, StepConst k)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= k.n) return;
    const float4 p = pos[s];
    const uint32_t id = __float_as_uint(p.w);
    const unsigned G = (unsigned)k.refG;
    const float GS = k.refGS, R = k.refR;
    const float c[3] = {p.x, p.y, p.z};
    int g[3][2];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        int g0 = __float2int_rz(__fdiv_rn(c[d], GS));
        if ((unsigned)g0 == G) g0 = (int)G - 1;
        const float pig = __fsub_rn(c[d], __fmul_rn(__int2float_rn(g0), GS));
        g[d][0] = g0;
        if (pig <= R) g[d][1] = (int)(((unsigned)(g0 - 1) + G) % G);
        else if (pig >= __fsub_rn(GS, R)) g[d][1] = (int)(((unsigned)g0 + 1) % G);
        else g[d][1] = -1;
    }
    int32_t out[8];
    int n = 0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        if (g[0][i] == -1) continue;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            if (g[1][j] == -1) continue;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if (g[2][q] == -1) continue;
                out[n++] = (int32_t)((unsigned)g[0][i] + (unsigned)g[1][j] * G + (unsigned)g[2][q] * G * G);
            }
        }
    }
    for (int q = 0; q < 8; ++q) cells8[(size_t)8 * id + q] = q < n ? out[q] : -1;
}

// ------------------------------------------------------------------ launchers

static inline unsigned blocks_for(uint32_t n, unsigned t) { return (n + t - 1) / t; }

// Launches a kernel that begins with chain_wait, with programmatic dependence
// on the kernel before it when chain is set.
template <class... P, class... A>
static cudaError_t launch_chain(bool chain, void (*kernel)(P...), unsigned grid, unsigned block, size_t smem,
                                cudaStream_t st, A... args)
{
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    cudaLaunchAttribute a{};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &a;
    c.numAttrs = chain ? 1 : 0;
    return cudaLaunchKernelEx(&c, kernel, P(args)...);
}

// Whether every boid goes to k_grid_warp: flocks (or ensembles) of at most
// kWarpBoids slots, unless the cells' split was set by hand.
static inline bool grid_by_warp(const StepConst &k, const DevBuffers &b, const FlockTable *ft)
{
    return b.slot_of && !k.tuned && (ft ? ft->nslots : k.n) <= kWarpBoids;
}

// Larger flocks that have the table of slots are sent there or by the cells'
// split in each step, on the device.
static inline Crowd crowd_route(const StepConst &k, const DevBuffers &b, const FlockTable *ft)
{
    if (!b.slot_of || k.tuned || grid_by_warp(k, b, ft)) return Crowd{nullptr, 0, 0};
    const double n = ft ? ft->nslots : k.n;
    const double even = n / (2. * b.ncell);
    const double from = ft ? b.crowd_min : n * crowd_line(even, n, b.carry ? CROWD_HANDLE : CROWD_BARE);
    const double to = !b.carry ? 4e9 : (ft ? b.crowd_max : n * crowd_top(even, crowd_seen(k), n, CROWD_HANDLE));
    const uint32_t min = (uint32_t)fmin(4e9, from);
    return Crowd{b.dense_n + 3, min, (uint32_t)fmax(0., fmin(4e9, to) - min)};
}

cudaError_t launch_pack(const float *pos3, const float *vel3, float4 *pos4, float4 *vel4, uint32_t i0, uint32_t i1,
                        uint32_t *bad, float hi, const StepConst *bin, uint32_t *key, uint32_t *rank,
                        uint32_t *count, cudaStream_t st, uint64_t *launches)
{
    if (i1 <= i0) return cudaSuccess;
    const StepConst none{};
    k_pack<<<blocks_for(i1 - i0, 256), 256, 0, st>>>(pos3, vel3, pos4, vel4, i0, i1, bad, hi, bin ? key : nullptr,
                                                      rank, count, bin ? *bin : none);
    ++*launches;
    return cudaGetLastError();
}

cudaError_t launch_unpack_index(const float4 *pos4, uint32_t *slot_of, uint32_t n, cudaStream_t st,
                                uint64_t *launches)
{
    if (n == 0) return cudaSuccess;
    k_unpack_index<<<blocks_for(n, 256), 256, 0, st>>>(pos4, slot_of, n);
    ++*launches;
    return cudaGetLastError();
}

cudaError_t launch_unpack_gather(const float4 *pos4, const float4 *vel4, const uint32_t *slot_of, float *pos3,
                                 float *vel3, uint32_t i0, uint32_t i1, uint32_t n, cudaStream_t st,
                                 uint64_t *launches)
{
    if (i1 <= i0) return cudaSuccess;
    k_unpack_gather<<<blocks_for(i1 - i0, 256), 256, 0, st>>>(pos4, vel4, slot_of, pos3, vel3, i0, i1, n);
    ++*launches;
    return cudaGetLastError();
}

cudaError_t launch_frame(const float4 *pos4, const float4 *vel4, const float *force9, float *pframe,
                         float *vframe, int with_forces, uint32_t n, cudaStream_t st, uint64_t *launches)
{
    if (n == 0) return cudaSuccess;
    k_frame<<<blocks_for(n, 256), 256, 0, st>>>(pos4, vel4, force9, pframe, vframe, with_forces, n);
    ++*launches;
    return cudaGetLastError();
}

cudaError_t launch_grid_keys(const StepConst &k, const float4 *pos, uint32_t *key, uint32_t *rank,
                             uint32_t *count, cudaStream_t st, uint64_t *launches, const FlockTable *ft)
{
    const uint32_t n = ft ? ft->nslots : k.n;
    if (n == 0) return cudaSuccess;
    if (ft) k_grid_keys<true><<<blocks_for(n, 256), 256, 0, st>>>(pos, key, rank, count, k, *ft);
    else k_grid_keys<false><<<blocks_for(n, 256), 256, 0, st>>>(pos, key, rank, count, k, FlockTable{});
    ++*launches;
    return cudaGetLastError();
}

// Whether launch_grid_scatter does the scan's work, too.
static inline bool grid_sort_small(const StepConst &k, const DevBuffers &b, const FlockTable *ft)
{
    return !ft && grid_by_warp(k, b, ft) && k.n <= kSortBoids && b.ncell_pad <= kSortCells;
}

cudaError_t launch_grid_scan(const StepConst &k, const DevBuffers &b, cudaStream_t st, uint64_t *launches,
                             const FlockTable *ft)
{
    if (grid_sort_small(k, b, ft) && k.n) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    const bool by_cells = !grid_by_warp(k, b, ft);
    if (by_cells && ft && b.defer_cnt && (e = cudaMemsetAsync(b.defer_cnt, 0, sizeof(uint32_t) * ft->count, st)) != cudaSuccess)
        return e;  // an ensemble's per-flock deferred counts
    *launches += 1;
    return launch_chain(!by_cells, k_grid_scan, b.nscan_blocks, kScanThreads, 0, st, b.count, b.lstart, b.bsum, b.ticket,
                        b.nscan_blocks, by_cells ? b.dense_n : nullptr, crowd_route(k, b, ft).pairs != nullptr);
}

bool grid_bin_small(const StepConst &k, const DevBuffers &b)
{
    return grid_by_warp(k, b, nullptr) && k.n > 0 && k.n <= kBinBoids && b.ncell_pad <= kBinCells;
}

cudaError_t launch_grid_bin(const StepConst &k, const DevBuffers &b, const float *pos3, const float *vel3,
                            cudaStream_t st, uint64_t *launches)
{
    if (grid_sort_small(k, b, nullptr))
        k_grid_bin_one<<<1, kSortThreads, 0, st>>>(pos3, vel3, b.lstart, b.bsum, b.ncell_pad, b.nscan_blocks, b.pos[1],
                                                   b.vel[1], b.slot_of, k);
    else k_grid_bin<<<kBinCtas, kBinThreads, 0, st>>>(pos3, vel3, b.key, b.rank, b.count, b.lstart, b.bsum, b.ncell_pad,
                                                 b.nscan_blocks, b.pos[1], b.vel[1], b.slot_of, k);
    *launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_grid_classify(const StepConst &k, const DevBuffers &b, cudaStream_t st, uint64_t *launches,
                                 const FlockTable *ft)
{
    if (grid_by_warp(k, b, ft)) return cudaSuccess;
    cudaError_t e;
    const uint32_t nfull = b.ncell / 4;
    const int windows = b.carry != nullptr;
    const Crowd crowd = crowd_route(k, b, ft);
    // with a side stream the classification runs beside what the caller
    // queues next (the scatter); launch_grid_force waits for it
    cudaStream_t cs = st;
    const bool side = b.aux != nullptr, chain = !side && !ft;
    if (side) {
        if ((e = cudaEventRecord(b.fork, st)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(b.aux, b.fork, 0)) != cudaSuccess) return e;
        cs = b.aux;
    }
    e = launch_chain(chain, ft ? k_grid_classify<true> : k_grid_classify<false>, blocks_for(nfull, 256), 256, 0, cs,
                     b.lstart, b.bsum, b.dflag, b.dense_list, b.dense_n, nfull, windows, (ft ? ft->nslots : k.n) >= kDenseShare, crowd, k,
                     ft ? *ft : FlockTable{});
    if (e != cudaSuccess) return e;
    if (side && (e = cudaEventRecord(b.cjoin, b.aux)) != cudaSuccess) return e;
    *launches += 1;
    return cudaSuccess;
}

cudaError_t launch_grid_scatter(const StepConst &k, const DevBuffers &b, int from, bool zero_counts,
                                cudaStream_t st, uint64_t *launches, const FlockTable *ft)
{
    const uint32_t n = ft ? ft->nslots : k.n;
    if (n == 0) return cudaSuccess;
    if (grid_sort_small(k, b, ft)) {
        ++*launches;
        return launch_chain(true, k_grid_sort, 1, kSortThreads, 0, st, b.pos[from], b.vel[from], b.key, b.rank, b.count,
                            b.lstart, b.bsum, b.ncell_pad, b.nscan_blocks, b.pos[1 - from], b.vel[1 - from],
                            (int)zero_counts, b.slot_of, k.n);
    }
    uint32_t *cz = zero_counts ? b.count : nullptr;
    const Crowd crowd = crowd_route(k, b, ft);
    uint32_t *so = grid_by_warp(k, b, ft) || crowd.pairs ? b.slot_of : nullptr;
    ++*launches;
    return launch_chain(grid_by_warp(k, b, ft) || (!ft && !b.aux), ft ? k_grid_scatter<true> : k_grid_scatter<false>, blocks_for(n, 256),
                        256, 0, st, b.pos[from], b.vel[from], b.key, b.rank, b.lstart, b.bsum, b.pos[1 - from],
                        b.vel[1 - from], cz, so, crowd, n, ft ? *ft : FlockTable{});
}

namespace {

// The dense kernel's shared memory exceeds the 48 KB default: opt in once
// per device and instantiation.
template <bool DIAG, bool MULTI>
cudaError_t dense_smem_opt_in()
{
    static uint64_t done = 0;  // bit per device ordinal
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev < 64 ? 1ull << dev : 0;
    if (bit && (__atomic_load_n(&done, __ATOMIC_ACQUIRE) & bit)) return cudaSuccess;
    e = cudaFuncSetAttribute(k_grid_dense<DIAG, MULTI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(DenseSmem));
    if (e == cudaSuccess && bit) __atomic_fetch_or(&done, bit, __ATOMIC_RELEASE);
    return e;
}

template <bool DIAG, bool MULTI>
cudaError_t grid_force(const StepConst &k, const GridIn &g, const GridOut &o, const DevBuffers &b, unsigned nsp,
                       const FlockTable &ft, cudaStream_t st)
{
    if (grid_by_warp(k, b, MULTI ? &ft : nullptr)) {
        return launch_chain(true, k_grid_warp<DIAG, MULTI>, blocks_for(MULTI ? ft.nslots : k.n, kWarpWarps),
                            kWarpWarps * 32, 0, st, g, o, k, ft);
    }
    cudaError_t e = dense_smem_opt_in<DIAG, MULTI>();
    if (e != cudaSuccess) return e;
    if (g.crowd.pairs) {
        e = launch_chain(true, k_grid_warp_queue<DIAG, MULTI>, b.dense_grid, kWarpWarps * 32, 0, st, g, o,
                         b.dense_n + 1, k, ft);
        if (e != cudaSuccess) return e;
    }
    if (b.aux && (e = cudaStreamWaitEvent(st, b.cjoin, 0)) != cudaSuccess) return e;  // the classification
    e = launch_chain(g.chain, k_grid_sparse<DIAG, MULTI>, nsp * (kRT / 32 / sparse_warps(MULTI)),
                     32 * sparse_warps(MULTI), 0, st, g, o, k, ft);
    if (e != cudaSuccess) return e;
    const unsigned nmore = MULTI ? nsp : min(nsp, 2 * b.dense_grid);
    if (o.defer && b.aux) {
        // the deferred boids and the dense cells are disjoint: run them side by side
        if ((e = cudaEventRecord(b.fork, st)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(b.aux, b.fork, 0)) != cudaSuccess) return e;
        k_grid_sparse_more<DIAG, MULTI><<<nmore, kRT, 0, b.aux>>>(g, o, k, ft);
        if ((e = cudaEventRecord(b.join, b.aux)) != cudaSuccess) return e;
        k_grid_dense<DIAG, MULTI><<<b.dense_grid, kDT, sizeof(DenseSmem), st>>>(g, o, b.dense_list, b.dense_n, k, ft);
        if ((e = cudaStreamWaitEvent(st, b.join, 0)) != cudaSuccess) return e;
        return cudaGetLastError();
    }
    if (o.defer) k_grid_sparse_more<DIAG, MULTI><<<nmore, kRT, 0, st>>>(g, o, k, ft);
    return launch_chain(g.chain && !o.defer, k_grid_dense<DIAG, MULTI>, b.dense_grid, kDT, sizeof(DenseSmem), st, g, o,
                        b.dense_list, b.dense_n, k, ft);
}

}  // namespace

cudaError_t launch_grid_force(const StepConst &k, const DevBuffers &b, int from, bool diag, bool record_forces,
                              cudaStream_t st, uint64_t *launches, const FlockTable *ft, float *pos3, float *vel3)
{
    const uint32_t n = ft ? ft->nslots : k.n;
    if (n == 0) return cudaSuccess;
    GridIn g{b.pos[from], b.vel[from], b.lstart, b.bsum, b.dflag, b.slot_of, crowd_route(k, b, ft), !b.aux && !ft, n >= kDenseShare};
    GridOut o{};
    o.carry = static_cast<Acc *>(b.carry);
    o.wscratch = b.carry ? b.wscratch : nullptr;
    o.wcap = o.wscratch ? b.wcap : 0;
    if (b.defer && b.defer_cnt && b.carry) {
        o.defer = b.defer;
        o.defer_cnt = b.defer_cnt;
        if (b.ovf && b.ovf_n) {
            o.ovf = b.ovf;
            o.ovf_n = b.ovf_n;
        }
    }
    if (diag) {
        o.dcnt = b.dcnt;
        o.dhash = b.dhash;
    } else {
        o.pos_out = b.pos[1 - from];
        o.vel_out = b.vel[1 - from];
        o.pos3_out = pos3;
        o.vel3_out = vel3;
        o.key_out = b.key;
        o.rank_out = b.rank;
        o.count = b.count;
        o.forces = record_forces ? b.forces : nullptr;
    }
    const unsigned nsp = blocks_for(n, kRT);
    const FlockTable none{};
    cudaError_t e;
    if (ft) e = diag ? grid_force<true, true>(k, g, o, b, nsp, *ft, st) : grid_force<false, true>(k, g, o, b, nsp, *ft, st);
    else e = diag ? grid_force<true, false>(k, g, o, b, nsp, none, st) : grid_force<false, false>(k, g, o, b, nsp, none, st);
    if (e == cudaSuccess) *launches += grid_by_warp(k, b, ft) ? 1 : 2 + (o.defer ? 1 : 0) + (g.crowd.pairs ? 1 : 0);
    return e;
}

cudaError_t launch_allpairs(const StepConst &k, const DevBuffers &b, int from, bool diag, bool record_forces,
                            cudaStream_t st, uint64_t *launches)
{
    if (k.n == 0) return cudaSuccess;
    k_ap_embed<<<blocks_for(k.n, 128), 128, 0, st>>>(b.pos[from], b.ap_emb, k.n, k);
    // the j tiles shrink until the GPU has a few CTAs per SM: where every pair
    // passes the filter (a small field), the exact tests are the work
    uint32_t tile_j = kApTileJ;
    while (tile_j > 16 && (uint64_t)blocks_for(k.n, kApTileI) * blocks_for(k.n, tile_j) < 4 * b.sms) tile_j /= 2;
    dim3 grid(blocks_for(k.n, kApTileI), blocks_for(k.n, tile_j));
    k_ap_pairs<<<grid, kApThreads, 0, st>>>(b.pos[from], b.vel[from], b.ap_emb, b.ap_cnt, b.ap_list, b.ap_cap, tile_j,
                                            k);
    *launches += 1;
    cudaError_t e = cudaGetLastError();
    ++*launches;
    if (e != cudaSuccess) return e;
    GridOut o{};
    if (diag) {
        o.dcnt = b.dcnt;
        o.dhash = b.dhash;
    } else {
        o.pos_out = b.pos[1 - from];
        o.vel_out = b.vel[1 - from];
        o.forces = record_forces ? b.forces : nullptr;
    }
    const unsigned nb = min(blocks_for(k.n, kWarpWarps), b.sms * kWarpCtas), nt = kWarpWarps * 32;
    if (diag) {
        k_ap_accumulate<true><<<nb, nt, 0, st>>>(b.pos[from], b.vel[from], b.ap_cnt, b.ap_list, b.ap_cap, o, k);
    } else {
        k_ap_accumulate<false><<<nb, nt, 0, st>>>(b.pos[from], b.vel[from], b.ap_cnt, b.ap_list, b.ap_cap, o, k);
    }
    ++*launches;
    return cudaGetLastError();
}

cudaError_t launch_ref_cells(const StepConst &k, const float4 *pos, int32_t *cells8, cudaStream_t st,
                             uint64_t *launches)
{
    if (k.n == 0) return cudaSuccess;
    k_ref_cells<<<blocks_for(k.n, 256), 256, 0, st>>>(pos, cells8, k);
    ++*launches;
    return cudaGetLastError();
}


// ------------------------------------------------------------------ ensemble statistics
//
// Order statistics of every flock of a batched ensemble, on a freshly binned
// state (sorted slots, valid cell tables).  Sums are FP64.  Per flock the
// accumulator holds kStatAcc doubles:
//   0-2  sum of unit velocities        3-5  sum of velocities
//   6-8  sum of sin(2 pi x / F)        9-11 sum of cos(2 pi x / F)
//   12-14 sum of r_hat x v_hat (about the centre of mass)
//   15   sum of capped nearest-neighbour distances
namespace {

constexpr int kStatThreads = kSlotAlign;
constexpr uint32_t kFindCap = 1u << 24;  // bound on union-find walks (far above any tree height)

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Block-reduce NV doubles per thread into acc[0..NV) with one atomic each.
template <int NV>
__device__ __forceinline__ void block_sum_to(const double (&v)[NV], double *acc)
{
    __shared__ double part[NV][kStatThreads / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const double s = warp_sum(v[i]);
        if (lane == 0) part[i][w] = s;
    }
    __syncthreads();
    if (threadIdx.x < NV) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < kStatThreads / 32; ++q) s += part[threadIdx.x][q];
        atomicAdd(acc + threadIdx.x, s);
    }
}

__device__ __forceinline__ uint32_t uf_find(const uint32_t *parent, uint32_t x, uint32_t *err)
{
    for (uint32_t it = 0; it < kFindCap; ++it) {
        const uint32_t p = __ldcg(parent + x);
        if (p == x) return x;
        x = p;
    }
    atomicOr(err, 1u);
    return x;
}

// Lock-free union: hook the larger root under the smaller one; a failed CAS
// means that root was hooked meanwhile, so retry from the new roots.
__device__ __forceinline__ void uf_union(uint32_t *parent, uint32_t a, uint32_t b, uint32_t *err)
{
    for (uint32_t it = 0; it < kFindCap; ++it) {
        a = uf_find(parent, a, err);
        b = uf_find(parent, b, err);
        if (a == b) return;
        const uint32_t hi = a > b ? a : b, lo = a > b ? b : a;
        const uint32_t old = atomicCAS(parent + hi, hi, lo);
        if (old == hi) return;
        a = lo;
        b = old;
    }
    atomicOr(err, 2u);
}

}  // namespace

__global__ void __launch_bounds__(kStatThreads)
k_stat_moments(const float4 *__restrict__ pos, const float4 *__restrict__ vel, FlockTable ft, double *acc,
               uint32_t *__restrict__ parent)
{
    __shared__ StepConst kf;
    load_flock(kf, ft, ft.blk_flock[blockIdx.x]);
    const uint32_t s = blockIdx.x * kStatThreads + threadIdx.x;
    parent[s] = s;
    double v[12] = {};
    if (s - kf.slot_base < kf.n) {
        const float4 p = pos[s], u = vel[s];
        const double vx = u.x, vy = u.y, vz = u.z;
        const double sp = sqrt(vx * vx + vy * vy + vz * vz);
        if (sp > 0.0) { v[0] = vx / sp; v[1] = vy / sp; v[2] = vz / sp; }
        v[3] = vx; v[4] = vy; v[5] = vz;
        const double inv = 2.0 / kf.F;
        sincospi(p.x * inv, &v[6], &v[9]);
        sincospi(p.y * inv, &v[7], &v[10]);
        sincospi(p.z * inv, &v[8], &v[11]);
    }
    block_sum_to<12>(v, acc + (size_t)kf.flock * kStatAcc);
}

// Centre of mass per flock: the periodic (circular) mean on each axis.
__global__ void k_stat_com(const double *__restrict__ acc, const StepConst *__restrict__ ks, uint32_t count,
                           double *__restrict__ com)
{
    const uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= count) return;
    const double *a = acc + (size_t)f * kStatAcc;
    const double F = ks[f].F;
    for (int d = 0; d < 3; ++d) {
        double c = atan2(a[6 + d], a[9 + d]) / (2.0 * 3.141592653589793) * F;
        if (c < 0.0) c += F;
        com[3 * f + d] = c;
    }
}

// Milling sum, capped nearest-neighbour distances and the union of every
// pair nearer than the link distance (the flock's cohesion sight distance),
// over the 27 full-size cells around each boid.
__global__ void __launch_bounds__(kStatThreads)
k_stat_pairs(GridIn g, FlockTable ft, const double *__restrict__ com, const float *__restrict__ link,
             double *acc, uint32_t *parent, uint32_t *err)
{
    __shared__ StepConst kf;
    load_flock(kf, ft, ft.blk_flock[blockIdx.x]);
    const StepConst &k = kf;
    const uint32_t s = blockIdx.x * kStatThreads + threadIdx.x;
    double v[4] = {};
    if (s - k.slot_base < k.n) {
        const float4 p4 = g.pos[s], u = g.vel[s];
        const float3 pi = xyz(p4);
        // r_hat x v_hat about the periodic centre of mass
        double r[3] = {pi.x - com[3 * k.flock], pi.y - com[3 * k.flock + 1], pi.z - com[3 * k.flock + 2]};
        for (int d = 0; d < 3; ++d) {
            if (r[d] > 0.5 * k.F) r[d] -= k.F;
            else if (r[d] < -0.5 * k.F) r[d] += k.F;
        }
        const double rn = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
        const double vx = u.x, vy = u.y, vz = u.z;
        const double sp = sqrt(vx * vx + vy * vy + vz * vz);
        if (rn > 0.0 && sp > 0.0) {
            const double a0 = r[0] / rn, a1 = r[1] / rn, a2 = r[2] / rn;
            const double b0 = vx / sp, b1 = vy / sp, b2 = vz / sp;
            v[0] = a1 * b2 - a2 * b1;
            v[1] = a2 * b0 - a0 * b2;
            v[2] = a0 * b1 - a1 * b0;
        }
        const int cx = cell1(pi.x, k), cy = cell1(pi.y, k), cz = cell1(pi.z, k);
        const int runs = seg_runs(cx, k);
        const float lk = link[k.flock];
        float nn2 = k.side * k.side;
        for (int q = 0; q < 9 * runs; ++q) {
            const Seg sg = segment(cx, cy, cz, q, runs, k);
            const uint32_t j0 = slot_start(g.lstart, g.bsum, k.cell_base + sg.c0, k);
            const uint32_t j1 = slot_start(g.lstart, g.bsum, k.cell_base + sg.c1, k);
            for (uint32_t j = j0; j < j1; ++j) {
                if (j == s) continue;
                const float4 pj = __ldg(g.pos + j);
                const float dx = pj.x + sg.sx - pi.x, dy = pj.y + sg.sy - pi.y, dz = pj.z + sg.sz - pi.z;
                const float d2 = dx * dx + dy * dy + dz * dz;
                nn2 = fminf(nn2, d2);
                if (j > s && d2 < lk * lk) uf_union(parent, s, j, err);
            }
        }
        v[3] = sqrt((double)nn2);
    }
    block_sum_to<4>(v, acc + (size_t)k.flock * kStatAcc + 12);
}

// Component sizes: every boid adds one to its root's count.
__global__ void k_stat_roots(FlockTable ft, const uint32_t *parent, uint32_t *__restrict__ size, uint32_t *err)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= ft.nslots) return;
    const StepConst &k = ft.ks[ft.blk_flock[s / kSlotAlign]];
    if (s - k.slot_base >= k.n) return;
    atomicAdd(size + uf_find(parent, s, err), 1u);
}

__global__ void k_stat_largest(FlockTable ft, const uint32_t *__restrict__ parent, const uint32_t *__restrict__ size,
                               uint32_t *__restrict__ largest)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= ft.nslots) return;
    const StepConst &k = ft.ks[ft.blk_flock[s / kSlotAlign]];
    if (s - k.slot_base >= k.n || parent[s] != s) return;
    atomicMax(largest + k.flock, size[s]);
}

cudaError_t launch_ensemble_stats(const DevBuffers &b, int from, const FlockTable &ft, const float *link,
                                  double *acc, double *com, uint32_t *largest, uint32_t *err, cudaStream_t st,
                                  uint64_t *launches)
{
    const unsigned nb = ft.nslots / kStatThreads;
    uint32_t *parent = b.key, *size = b.rank;  // free between a step's binning and its rule pass
    cudaError_t e;
    if ((e = cudaMemsetAsync(acc, 0, sizeof(double) * kStatAcc * ft.count, st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(largest, 0, sizeof(uint32_t) * ft.count, st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(size, 0, sizeof(uint32_t) * ft.nslots, st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(err, 0, sizeof(uint32_t), st)) != cudaSuccess) return e;
    k_stat_moments<<<nb, kStatThreads, 0, st>>>(b.pos[from], b.vel[from], ft, acc, parent);
    k_stat_com<<<blocks_for(ft.count, 128), 128, 0, st>>>(acc, ft.ks, ft.count, com);
    GridIn g{b.pos[from], b.vel[from], b.lstart, b.bsum};  // k_stat_pairs reads only cells
    k_stat_pairs<<<nb, kStatThreads, 0, st>>>(g, ft, com, link, acc, parent, err);
    k_stat_roots<<<blocks_for(ft.nslots, 256), 256, 0, st>>>(ft, parent, size, err);
    k_stat_largest<<<blocks_for(ft.nslots, 256), 256, 0, st>>>(ft, parent, size, largest);
    *launches += 5;
    return cudaGetLastError();
}

cudaError_t grid_prepare()
{
    cudaError_t e;
    if ((e = dense_smem_opt_in<false, false>()) != cudaSuccess) return e;
    if ((e = dense_smem_opt_in<true, false>()) != cudaSuccess) return e;
    if ((e = dense_smem_opt_in<false, true>()) != cudaSuccess) return e;
    return dense_smem_opt_in<true, true>();
}

}  // namespace boidsgpu
