// nw_srd.cu — the SRD collision (ParticleSystem::_solventUpdate,
// simulation/particleSystem.cpp:341-413): cell hashes and counts, the members
// of every cell in stable order, the collision and the solvent's streaming.
//
// The solvent is stored in the cell order of the last collision.  Between two
// collisions a particle moves by its streaming step and the grid by the
// difference of the two shifts, so a cell's solvent lies in a few old cells
// around it, one contiguous run of the stored solvent per row of old cells:
// two or three cells a row and two or three rows, about 19 candidates for 4.4
// members at density 4.  Every lane of the collision reads the hashes of its
// cell's runs, in ascending storage order, and keeps its own: the members
// come out in the stable order, without slots, buckets or a sort of them.
// How far particles can have stepped follows from the largest displacement,
// taken while they streamed.  Where that does not hold (positions set from
// outside since, a displacement of more than a cell or two, grids that do not
// tile the box) the solvent is bucketed by counting and each cell's bucket
// sorted; both give the same order, so the results are the same to the bit.
//
// On 400,000 beads, 4,000,000 solvent particles and 1,000,000 cells (device
// times under a profiler) the hashes take 20 + 9 us (46 us with the slots that
// buckets need), the bucketing none (21-37 us) and the collision 94 us
// (119 us from buckets, with their order, a search for each slot's cell and
// the results staged once more); the whole call of ten updates went from 373
// to 324 us.
//
#include <algorithm>

#include "nw_engine.h"

namespace nw {

namespace {

uint32_t cdiv(uint64_t a, uint32_t b) { return (uint32_t)((a + b - 1) / b); }

__device__ __forceinline__ float geo_float(const StepBuffers& S, uint32_t buf, uint32_t k)
{
    return __uint_as_float(S.srd_state[kSrdGeo + 8u * buf + k]);
}

struct SrdSteps {
    int ordered;
    int lo[3], n[3];
};

// Steps between the cell of a particle at the last collision and at this
// one.  On an axis with cells of edge a, q = (x + shift) / a lay in [X, X + 1)
// and has changed by d = (new shift - old shift) / a and by at most `most`
// (plus rounding, a few ulp of the largest coordinate and of the shifts, which
// may be far larger than the box): floor(q) - X is between floor(d - s) and
// floor(1 + d + s).  Walls clamp both cells, so there a step
// may also be shorter, down to none.
__device__ __forceinline__ SrdSteps srd_steps(const DevParams& P, const uint32_t (&g)[5], float3 shift)
{
    SrdSteps w;
    const float most = __uint_as_float(g[kSrdStep]);
    w.ordered = g[kSrdHeld] != 0u && P.srd_tiles_box != 0 && most <= (float)kSrdSteps;
    const float now[3] = {shift.x, shift.y, shift.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        w.lo[a] = 0;
        w.n[a] = 1;
        if (P.srd_grid[a] == 1u) continue;
        const float was = __uint_as_float(g[a]);
        const float d = (now[a] - was) * P.srd_per_len[a];
        const float s = most + P.srd_slack[a] + kSrdRound * (fabsf(now[a]) + fabsf(was)) * P.srd_per_len[a];
        if (!(fabsf(d) + s <= 8.0f)) {
            w.ordered = 0;
            continue;
        }
        int lo = (int)floorf(d - s), hi = (int)floorf(1.0f + d + s);
        if (P.bnd[a] != NW_PERIODIC) {
            lo = min(lo, 0);
            hi = max(hi, 0);
        }
        w.lo[a] = lo;
        w.n[a] = hi - lo + 1;
        // one wrap reaches every old cell, and none of them twice
        const int G = (int)P.srd_grid[a];
        if (w.n[a] > kSrdSteps || w.n[a] > G || hi > G || lo < -G) w.ordered = 0;
    }
    return w;
}

// The old cells start .. start + n - 1 of an axis in ascending order of their
// index: element s of them, wrapped on a periodic axis; false beyond a wall.
__device__ __forceinline__ bool old_cell(int start, int n, int s, int G, bool per, int& out)
{
    int t = s;
    if (per) {
        // the elements from index 0 of the axis on come first
        const int first = start < 0 ? -start : G - start;
        if (first > 0 && first < n) {
            t = s + first;
            if (t >= n) t -= n;
        }
    }
    int v = start + t;
    if (per) {
        if (v < 0) v += G;
        else if (v >= G) v -= G;
    }
    out = v;
    return v >= 0 && v < G;
}

// The runs of stored solvent that hold the members of the cells
// x .. x + len - 1 of row (y, z): piece p of them, in ascending order of the
// storage; one row of old cells in one piece, or in two where the row wraps.
__device__ __forceinline__ void old_run(const DevParams& P, const uint32_t* __restrict__ old, const int* lo,
                                        const int* n, int x, int len, int y, int z, int p, uint32_t& begin,
                                        uint32_t& end)
{
    const int G0 = (int)P.srd_grid[0], G1 = (int)P.srd_grid[1], G2 = (int)P.srd_grid[2];
    begin = end = 0;
    const int r = p >> 1, tz = n[1] == 1 ? r : n[1] == 2 ? r >> 1 : n[1] == 3 ? (r * 11) >> 5 : r >> 2;  // r / n[1]
    const int ty = r - tz * n[1];
    int oz, oy;
    if (tz >= n[2]) return;
    if (!old_cell(z - (lo[2] + n[2] - 1), n[2], tz, G2, P.bnd[2] == NW_PERIODIC, oz)) return;
    if (!old_cell(y - (lo[1] + n[1] - 1), n[1], ty, G1, P.bnd[1] == NW_PERIODIC, oy)) return;
    int a = x - (lo[0] + n[0] - 1), b = x + len - 1 - lo[0];
    const bool second = (p & 1) != 0;
    if (P.bnd[0] != NW_PERIODIC) {
        if (second) return;
        a = max(a, 0);
        b = min(b, G0 - 1);
    } else if (b - a + 1 >= G0) {
        if (second) return;
        a = 0;
        b = G0 - 1;
    } else if (a < 0 && b >= 0) {
        if (second) b = G0 - 1, a += G0;
        else a = 0;
    } else if (a < G0 && b >= G0) {
        if (second) b = G0 - 1;
        else a = 0, b -= G0;
    } else {
        if (second) return;
        if (b < 0) a += G0, b += G0;
        else if (a >= G0) a -= G0, b -= G0;
    }
    if (a > b) return;
    const uint32_t row = ((uint32_t)oz * (uint32_t)G1 + (uint32_t)oy) * (uint32_t)G0;
    begin = old[row + (uint32_t)a];
    end = old[row + (uint32_t)b + 1u];
}

// take(q, k) by the lanes of the warp for each stored solvent particle k that
// belongs to cell c0 + q, q in [first, last], in ascending order: along the lanes,
// call by call.
constexpr int kRunLoads = 5;  // a row of 34 old cells at density 4 in one batch of loads, mostly
// ahead(k, m) by the lane that found them, for runs of m particles from k on
// that will be read.
template <class Ahead, class Take>
__device__ __forceinline__ void for_warp_solvent(const DevParams& P, const uint32_t* __restrict__ hash,
                                                 const uint32_t* __restrict__ old, const int* lo, const int* n,
                                                 uint32_t c0, uint32_t first, uint32_t last, Ahead ahead, Take take)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t G0 = P.srd_grid[0], G1 = P.srd_grid[1];
    const uint32_t ncell = min(last + 1u, P.srd_ncells - c0);
    for (uint32_t l = first; l < ncell;) {  // the cells, one grid row at a time
        const uint32_t c = c0 + l;
        uint32_t z = 0, rest = c;
        if (P.srd_grid[2] > 1u) {
            z = fast_div(c, P.sdiv_xy_m, P.sdiv_xy_k);
            rest = c - z * (G0 * G1);
        }
        const uint32_t y = fast_div(rest, P.sdiv_x_m, P.sdiv_x_k), x = rest - y * G0;
        const uint32_t len = min(ncell - l, G0 - x);
        uint32_t begin, end;
        old_run(P, old, lo, n, (int)x, (int)len, (int)y, (int)z, (int)lane, begin, end);
        if (begin < end) ahead(begin, end - begin);
        uint32_t pieces = __ballot_sync(0xffffffffu, begin < end);
        while (pieces) {
            const int p = __ffs(pieces) - 1;
            pieces &= pieces - 1u;
            const uint32_t e0 = __shfl_sync(0xffffffffu, begin, p) + lane;
            int left = (int)(__shfl_sync(0xffffffffu, end, p) - e0);  // of this lane's, every 32nd
            const int most = (int)__shfl_sync(0xffffffffu, left, 0);
            const uint32_t* __restrict__ run = hash + e0;
            for (int o = 0; o < most; o += 32 * kRunLoads) {
                uint32_t h[kRunLoads];
#pragma unroll
                for (int q = 0; q < kRunLoads; ++q) h[q] = 32 * q < left ? run[32 * q] : kEmpty;
#pragma unroll
                for (int q = 0; q < kRunLoads; ++q) {
                    const uint32_t d = h[q] - c;
                    if (d < len) take(l + d, e0 + (uint32_t)(o + 32 * q));
                }
                run += 32 * kRunLoads;
                left -= 32 * kRunLoads;
            }
        }
        l += len;
    }
}

__device__ __forceinline__ void copy16_async(float4* to, const float4* from)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from)
                 : "memory");
}
// Brings a run of global memory (16-byte aligned, a multiple of 16 bytes) into L2.
__device__ __forceinline__ void fetch_l2(const float4* from, uint32_t bytes)
{
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(from), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The largest streaming step of a warp's particles, in cells (non-negative
// floats order as their bits), into the geometry of the buffer written.
__device__ __forceinline__ void keep_largest_step(const StepBuffers& S, uint32_t buf, uint32_t bits)
{
    uint32_t* word = S.srd_state + kSrdGeo + 8u * buf + kSrdStep;
    const uint32_t m = __reduce_max_sync(0xffffffffu, bits);
    if ((threadIdx.x & 31u) == 0u && m > *(volatile uint32_t*)word) atomicMax(word, m);
}

// Streaming step of one particle in cells, as float bits (those of a NaN
// exceed every number's).
__device__ __forceinline__ uint32_t step_bits(const DevParams& P, float3 dr)
{
    return max(__float_as_uint(fabsf(dr.x) * P.srd_per_len[0]),
               max(__float_as_uint(fabsf(dr.y) * P.srd_per_len[1]), __float_as_uint(fabsf(dr.z) * P.srd_per_len[2])));
}

// A particle's way from `was`: its streaming step on periodic axes; on the
// others also what a wall put it back by where it was outside.
__device__ __forceinline__ float3 way_of(const DevParams& P, float3 dr, float4 was, float3 now)
{
    return make_float3(P.bnd[0] == NW_PERIODIC ? dr.x : now.x - was.x, P.bnd[1] == NW_PERIODIC ? dr.y : now.y - was.y,
                       P.bnd[2] == NW_PERIODIC ? dr.z : now.z - was.z);
}

// A particle far outside the box has no bounded step.  Only a bucketed
// collision looks: from there on particles move by a few cells at a time and
// are wrapped, or stopped at walls.
__device__ __forceinline__ bool near_box(const DevParams& P, float3 p)
{
    return fabsf(p.x - P.srd_mid[0]) <= P.srd_reach[0] && fabsf(p.y - P.srd_mid[1]) <= P.srd_reach[1] &&
           fabsf(p.z - P.srd_mid[2]) <= P.srd_reach[2];
}

// The beads of a cell: the first kBeadSlots to arrive in a table, one load for
// the collision, any more in a linked list.  take(k, bead) for each, unordered.
constexpr uint32_t kBeadSlots = 4;
template <class Take>
__device__ __forceinline__ void for_cell_beads(const StepBuffers& S, uint32_t c, uint32_t nbc, Take take)
{
    const uint4 t = *reinterpret_cast<const uint4*>(S.srd_btab + (size_t)c * kBeadSlots);
    if (nbc > 0u) take(0u, t.x);
    if (nbc > 1u) take(1u, t.y);
    if (nbc > 2u) take(2u, t.z);
    if (nbc > 3u) take(3u, t.w);
    if (nbc > kBeadSlots) {
        uint32_t e = S.srd_bhead[c];
        S.srd_bhead[c] = kEmpty;
        for (uint32_t k = kBeadSlots; k < nbc && e != kEmpty; ++k, e = S.srd_bnext[e]) take(k, e);
    }
}

// SRD cell hash and count of every bead, and the beads of each cell.  The grid shift of a scheduled collision is drawn once per block; the
// first block writes it, and what follows from it for the collision that
// begins, for the kernels after this one.
__global__ void __launch_bounds__(256) srd_bead_hash_kernel(const DevParams P, const StepBuffers S, uint32_t step_off,
                                                            int shift_from_step, float3 shift, uint32_t buf_sel)
{
    pdl_enter();
    __shared__ float s_shift[3];
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    const unsigned long long step = *S.step_base + step_off;
    const uint32_t cur = buf_sel < 2u ? buf_sel : (uint32_t)(step & 1ull);
    float4 p4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < P.nb) p4 = (cur ? S.pos2[1] : S.pos2[0])[i];
    if (threadIdx.x == 0) {
        uint32_t sc = 0, geo[2][5];
        if (blockIdx.x == 0) {  // on their way beside the step counter
            sc = *S.scur;
#pragma unroll
            for (uint32_t k = 0; k < 5u; ++k) {
                geo[0][k] = S.srd_state[kSrdGeo + k];
                geo[1][k] = S.srd_state[kSrdGeo + 8u + k];
            }
        }
        const float3 d = shift_from_step ? srd_shift_of(P, step) : shift;
        s_shift[0] = d.x;
        s_shift[1] = d.y;
        s_shift[2] = d.z;
        if (blockIdx.x == 0) {
#pragma unroll
            for (uint32_t k = 0; k < 5u; ++k) geo[0][k] = sc ? geo[1][k] : geo[0][k];
            const SrdSteps w = srd_steps(P, geo[0], d);
            uint32_t* st = S.srd_state;
            st[kSrdSrc] = sc;
            st[kSrdOrdered] = (uint32_t)w.ordered;
            for (int a = 0; a < 3; ++a) {
                st[kSrdLo + a] = (uint32_t)w.lo[a];
                st[kSrdN + a] = (uint32_t)w.n[a];
            }
            // the buffer that this collision fills
            uint32_t* g = st + kSrdGeo + 8u * (sc ^ 1u);
            g[0] = __float_as_uint(d.x);
            g[1] = __float_as_uint(d.y);
            g[2] = __float_as_uint(d.z);
            g[kSrdStep] = 0u;
            g[kSrdHeld] = 1u;
            *S.srd_nbig = 0;  // the list is filled by the collision that follows
        }
    }
    __syncthreads();
    if (i >= P.nb) return;
    const uint32_t h = srd_hash(P, f3(p4), make_float3(s_shift[0], s_shift[1], s_shift[2]));
    S.srd_hash[i] = h;
    const uint32_t k = atomicAdd(&S.srd_bcount[h], 1u);
    if (k < kBeadSlots) S.srd_btab[(size_t)h * kBeadSlots + k] = i;
    else S.srd_bnext[i] = atomicExch(&S.srd_bhead[h], i);
}

// One axis of srd_hash where it is periodic, step by step the same arithmetic.
__device__ __forceinline__ uint32_t srd_axis(const DevParams& P, int a, float x, float shift)
{
    const uint32_t G = P.srd_grid[a];
    float rel = (x + shift) - P.origin[a];
    if (rel >= P.box[a]) rel -= P.box[a];
    else if (rel < 0.0f) rel += P.box[a];
    const float q = rel * P.srd_inv_cell[a];
    int g = (int)floorf(q);
    if (fabsf(q - rintf(q)) <= fabsf(q) * 5.0e-7f) g = (int)floorf(rel / P.srd_cell[a]);  // floor_div
    return (uint32_t)g < G ? (uint32_t)g : wrap_mod(g, G);  // of a power of two also the mask
}

// srd_hash on one layer with both axes periodic (P.srd_flat)
__device__ __forceinline__ uint32_t srd_hash_flat(const DevParams& P, float4 p, float3 shift)
{
    return srd_axis(P, 1, p.y, shift.y) * P.srd_grid[0] + srd_axis(P, 0, p.x, shift.x);
}

constexpr uint32_t kHashPer = 4;  // solvent particles per thread of srd_hash_kernel

// SRD cell hash and count of every solvent particle.  Where the solvent will
// be bucketed (srd_steps: not ordered) its slots are taken too, one atomic
// per run of equal keys along the warp.
__global__ void __launch_bounds__(256) srd_hash_kernel(const DevParams P, const StepBuffers S)
{
    pdl_enter();
    const uint32_t t = threadIdx.x;
    const uint32_t sc = S.srd_state[kSrdSrc];
    const bool ordered = S.srd_state[kSrdOrdered] != 0u;
    const float3 sh = make_float3(geo_float(S, sc ^ 1u, 0), geo_float(S, sc ^ 1u, 1), geo_float(S, sc ^ 1u, 2));
    const uint32_t first = blockIdx.x * (256u * kHashPer) + t;
    const float4* __restrict__ sp = sc ? S.spos2[1] : S.spos2[0];
    float4 p4[kHashPer];
#pragma unroll
    for (uint32_t q = 0; q < kHashPer; ++q)
        if (first + 256u * q < P.ns) p4[q] = sp[first + 256u * q];
    uint32_t* __restrict__ hash = S.srd_hash + P.nb;
    if (ordered) {
#pragma unroll
        for (uint32_t q = 0; q < kHashPer; ++q) {
            const uint32_t i = first + 256u * q;
            if (i >= P.ns) continue;
            const uint32_t h = P.srd_flat ? srd_hash_flat(P, p4[q], sh) : srd_hash(P, f3(p4[q]), sh);
            hash[i] = h;
            atomicAdd(&S.srd_scount[h], 1u);
        }
        return;
    }
    // every lane of the warp takes part (blockDim is a multiple of 32)
    const uint32_t lane = t & 31u;
    const uint32_t upto = (2u << lane) - 1u;  // lanes 0..lane (all 32 bits for lane 31)
#pragma unroll
    for (uint32_t q = 0; q < kHashPer; ++q) {
        const uint32_t i = first + 256u * q;
        const bool valid = i < P.ns;
        uint32_t h = kEmpty;  // no cell hash
        if (valid) {
            h = srd_hash(P, f3(p4[q]), sh);
            hash[i] = h;
        }
        const uint32_t prev = __shfl_up_sync(0xffffffffu, h, 1);
        const uint32_t heads = __ballot_sync(0xffffffffu, lane == 0u || prev != h);
        const uint32_t start = 31u - (uint32_t)__clz(heads & upto);
        const uint32_t after = heads & ~upto;
        const uint32_t end = after ? (uint32_t)(__ffs(after) - 1) : 32u;
        uint32_t base = 0;
        if (valid && lane == start) base = atomicAdd(&S.srd_scount[h], end - start);
        base = __shfl_sync(0xffffffffu, base, (int)start);
        if (valid) S.srd_slot[i] = base + (lane - start);
    }
}

// Bucket the solvent by cell, where the collision will not find it through
// the old cell order.
__global__ void __launch_bounds__(256) srd_scatter_kernel(const DevParams P, const StepBuffers S)
{
    pdl_enter();
    if (S.srd_state[kSrdOrdered]) return;
    const uint32_t* __restrict__ soff = S.srd_state[kSrdSrc] ? S.srd_soff2[0] : S.srd_soff2[1];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < P.ns; i += gridDim.x * blockDim.x)
        S.srd_stmp[soff[S.srd_hash[P.nb + i]] + S.srd_slot[i]] = i;
}

// SRD collision.  A warp owns 32 consecutive cells; their members are one
// contiguous range of the stable (cell, index) order and their solvent one
// contiguous range of the new solvent storage.  The warp reads the hashes of
// the old cells around its own and enters each member, with its cell's lane,
// at the next place of its cell in the staging (beads come from the cell's
// table; without the old cell order each lane sorts its cell's bucket).  The members' velocities are
// gathered with asynchronous copies, each lane takes its cell's sums from
// shared memory, then every lane updates the members of its slots with the
// cell's factors from shared memory, loading a slot's position ahead, and
// writes the stable order and the streamed solvent straight to their places,
// which are consecutive along the warp.
//
// Per cell, in the member order (the cell's beads, then its solvent, each by
// index): the reference's isokinetic scaling (particles_kernel_impl.cuh:605-637)
// or none, the mass-weighted cell mean (:560-594), the +/- alpha rotation of
// (v - u) (:640-691), the relative-velocity thermostat when selected, and the
// solvent's ballistic streaming by dt_srd (solvent_integrator, :145-205).
// Beads are written in place, the solvent to the other solvent buffer.
// A warp holding more than kWarpCap members takes its cells in rounds that
// fit.  A cell of more than kLaneCap members goes to srd_collide_big_kernel
// (a warp per cell), so that no lane's serial loops run far longer than its
// neighbours'; its members go to its buckets.
//
// What bounds it: 61M warp instructions (of 1,900 a warp some 400 find the
// members, 500 are the two serial sums over a cell, whose longest of 32 has 10
// members for 4.4 on average, 500 the update) at 58 % of the issue rate, and
// the shared-memory pipe at 56 %; DRAM moves 306 MB in 92 us.  With blocks of
// four warps, 8 of them resident, more warps spilled (9 blocks 105 us, 10
// blocks 103 us) and fewer (7 blocks) took 102 us; batches of 3 or 8 loads along
// a run 99 and 100 us.  Fetching the runs' velocities and positions into L2 while
// their hashes are looked through took 97 to 94.5 us, blocks of two warps (16
// resident) instead of four 94.2 to 92.4 (eight: 97.9), copies past L1 another 0.8.
constexpr int kCollideWarps = 2;

// Rounded products, whatever is added to them (the compiled modes round alike).
__device__ __forceinline__ float3 scaled_rn(float f, float4 V)
{
    return make_float3(__fmul_rn(f, V.x), __fmul_rn(f, V.y), __fmul_rn(f, V.z));
}

// apply_boundaries on a box periodic in every axis
__device__ __forceinline__ void wrap_periodic(const DevParams& P, float3& p)
{
    float* x = &p.x;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float L0 = P.origin[a], L = P.box[a];
        if (x[a] < L0) x[a] += L;
        else if (x[a] > L + L0) x[a] -= L;
    }
}

// 192 members per warp: 32 cells at up to 6 members on average
constexpr uint32_t kWarpCap = 192;
static_assert(kLaneCap <= kWarpCap, "a cell of the warp path fits the staging alone");
constexpr uint32_t kToBucket = 0x80000000u;  // a place in the bucket array rather than in the staging

struct __align__(16) CellFactors {
    float ux, uy, uz, sa;
    float lam1, lam2;
    uint32_t sorted;  // stable-order position of staged slot j of this cell: sorted + j
    uint32_t beads;   // beads up to and with this cell's (bit 31: scale by lam2)
};

// Compiled for the two usual collisions on periodic boxes, where the flags are
// constants: kRelative, the relative-velocity thermostat with beads rotated,
// and kLab, the reference's own; kAny reads them.
enum SrdMode { kAny = 0, kRelative = 1, kLab = 2 };

template <int kMode>
__global__ void __launch_bounds__(kCollideWarps * 32, 16) srd_collide_kernel(const DevParams P, const StepBuffers S,
                                                                         uint32_t step_off, float dt_srd,
                                                                         uint32_t buf_sel)
{
    pdl_enter();
    __shared__ uint2 s_m[kCollideWarps][kWarpCap];  // members: index, cell's lane
    __shared__ float4 s_v[kCollideWarps][kWarpCap];
    __shared__ CellFactors s_f[kCollideWarps][32];
    __shared__ uint32_t s_at[kCollideWarps][32];  // next free place of each cell's solvent
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = c < P.srd_ncells;
    const unsigned long long step = *S.step_base + step_off;
    const uint32_t cur = buf_sel < 2u ? buf_sel : (uint32_t)(step & 1ull);
    const uint32_t a = S.srd_state[kSrdSrc];
    const bool ordered = S.srd_state[kSrdOrdered] != 0u;
    if (c == 0) *S.scur = a ^ 1u;  // read again by the next collision only
    const float4* __restrict__ sv_old = a ? S.svel2[1] : S.svel2[0];
    const float4* __restrict__ sp_old = a ? S.spos2[1] : S.spos2[0];
    float4* __restrict__ sv_new = a ? S.svel2[0] : S.svel2[1];
    float4* __restrict__ sp_new = a ? S.spos2[0] : S.spos2[1];
    const uint32_t* __restrict__ soff = a ? S.srd_soff2[0] : S.srd_soff2[1];
    float4* __restrict__ bvel = cur ? S.vel2[1] : S.vel2[0];
    uint32_t b0 = 0, nbc = 0, s0 = 0, nsc = 0;
    if (valid) {
        b0 = S.srd_boff[c];
        nbc = S.srd_boff[c + 1] - b0;
        s0 = soff[c];
        nsc = soff[c + 1] - s0;
    }
    const uint32_t nall = nbc + nsc;
    const uint32_t start = b0 + s0;  // particles before this cell in the stable order
    if (valid) {
        S.srd_start[c] = nall ? start : kEmpty;
        S.srd_end[c] = nall ? start + nall : kEmpty;
    }
    // a cell of more than kLaneCap members is collided by a whole warp in
    // srd_collide_big_kernel, from its buckets; here it counts as empty
    const bool big = nall > kLaneCap;
    if (big) {
        S.srd_big[atomicAdd(S.srd_nbig, 1u)] = c;
        if (nbc) for_cell_beads(S, c, nbc, [&](uint32_t k, uint32_t e) { S.srd_btmp[b0 + k] = e; });
    }
    const uint32_t n = big ? 0u : nall;
    const uint32_t incl = warp_incl_scan(n);
    const uint32_t loc = incl - n;  // this cell's members in the warp's staging
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    const bool any_big = __any_sync(0xffffffffu, big) != 0;
    if (total == 0u && !any_big) {  // uniform over the warp
        if (valid) S.srd_mean[c] = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    const bool lab = kMode == kLab || (kMode == kAny && P.srd_thermo == NW_SRD_THERMO_REF_LAB);
    const bool rel = kMode == kRelative || (kMode == kAny && P.srd_thermo == NW_SRD_THERMO_CELL_REL);
    const bool rotate_beads = kMode == kRelative || (kMode == kAny && P.srd_rotate_beads);
    const float ca = P.srd_cos_a;
    uint32_t moved = 0u;  // largest streaming step (float bits)
    // Rounds of consecutive cells whose members fit the staging buffers
    // (one round unless the warp holds more than kWarpCap members).
    uint32_t first = 0;
    while (first < 32u) {
        const uint32_t base = __shfl_sync(0xffffffffu, loc, (int)first);
        const uint32_t fm = __ballot_sync(0xffffffffu, lane >= first && loc + n - base <= kWarpCap);
        const uint32_t last = 31u - (uint32_t)__clz(fm);
        const uint32_t rtotal = __shfl_sync(0xffffffffu, loc + n, (int)last) - base;
        const bool mine = lane >= first && lane <= last;
        const uint32_t at0 = loc - base;  // this cell's first place in the staging
        // members of the round's cells in stable order: ids < nb are beads, nb + k
        // is solvent k
        if (mine && n > 0) {
            uint2* ids = &s_m[w][at0];
            if (nbc) {
                for_cell_beads(S, c, nbc, [&](uint32_t k, uint32_t e) {
                    uint32_t m = k;  // insertion by index
                    while (m > 0 && ids[m - 1].x > e) {
                        ids[m] = ids[m - 1];
                        --m;
                    }
                    ids[m] = make_uint2(e, lane);
                });
            }
            s_f[w][lane].sorted = start - at0;
        }
        if (ordered) {
            const uint32_t at = big ? kToBucket | s0 : at0 + nbc;
            s_at[w][lane] = at;
            __syncwarp();
            const int lo[3] = {(int)S.srd_state[kSrdLo], (int)S.srd_state[kSrdLo + 1], (int)S.srd_state[kSrdLo + 2]};
            const int ns[3] = {(int)S.srd_state[kSrdN], (int)S.srd_state[kSrdN + 1], (int)S.srd_state[kSrdN + 2]};
            for_warp_solvent(P, S.srd_hash + P.nb, a ? S.srd_soff2[1] : S.srd_soff2[0], lo, ns, c - lane, first,
                             last, [&](uint32_t k, uint32_t m) {
                                 fetch_l2(sv_old + k, m * 16u);
                                 fetch_l2(sp_old + k, m * 16u);
                             },
                             [&](uint32_t q, uint32_t i) {
                                 const uint32_t to = atomicAdd(&s_at[w][q], 1u);
                                 if (to < kWarpCap) s_m[w][to] = make_uint2(P.nb + i, q);
                                 else if (any_big && to >= kToBucket && (to ^ kToBucket) < P.ns)
                                     S.srd_stmp[to ^ kToBucket] = i;
                             });
            __syncwarp();
            // the counts and the runs come from the same hashes; a difference is
            // reported, and the slots left point at solvent 0
            if (mine) {
                const uint32_t got = s_at[w][lane] - at;
                if (got != nsc) {
                    atomicOr(S.err, (uint32_t)NW_EFLAG_BAD_INDEX);
                    for (uint32_t k = got < nsc ? got : 0u; k < nsc; ++k) {
                        if (big) S.srd_stmp[s0 + k] = 0u;
                        else s_m[w][at0 + nbc + k] = make_uint2(P.nb, lane);
                    }
                }
            }
            __syncwarp();
            // lanes of one call may have entered a cell's members in any order
            bool swapped = false;
            for (uint32_t j = lane + 1u; j < rtotal; j += 32u) {
                const uint2 x = s_m[w][j], y = s_m[w][j - 1u];
                swapped |= x.y == y.y && x.x < y.x;
            }
            if (__any_sync(0xffffffffu, swapped) && mine && n > 0) {
                uint2* ids = &s_m[w][at0 + nbc];
                for (uint32_t k = 1; k < nsc; ++k) {
                    const uint2 x = ids[k];
                    uint32_t m = k;
                    while (m > 0 && ids[m - 1].x > x.x) {
                        ids[m] = ids[m - 1];
                        --m;
                    }
                    ids[m] = x;
                }
            }
        } else if (mine && n > 0) {
            uint2* ids = &s_m[w][at0];
            for (uint32_t k = nbc; k < n; ++k) {
                const uint32_t x = P.nb + S.srd_stmp[s0 + (k - nbc)];
                uint32_t m = k;
                while (m > nbc && ids[m - 1].x > x) {
                    ids[m] = ids[m - 1];
                    --m;
                }
                ids[m] = make_uint2(x, lane);
            }
        }
        __syncwarp();
        // stable-order position of slot 0 (with big cells among them, the cells'
        // members are not consecutive there)
        const uint32_t sorted0 = __shfl_sync(0xffffffffu, start, (int)first);
        for (uint32_t j = lane; j < rtotal; j += 32u) {
            const uint2 m = s_m[w][j];
            copy16_async(&s_v[w][j], m.x < P.nb ? bvel + m.x : sv_old + (m.x - P.nb));
            S.srd_sorted_index[(any_big ? s_f[w][m.y].sorted : sorted0) + j] = m.x;
        }
        copy_commit();
        // the position of this lane's first slot, on its way during the sums
        uint2 m = make_uint2(0u, 0u);
        if (lane < rtotal) m = s_m[w][lane];
        float4 P4 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (m.x >= P.nb && lane < rtotal) P4 = sp_old[m.x - P.nb];
        copy_wait<0>();
        __syncwarp();
        // per cell, by its lane: [lab isokinetic factor], mean velocity, rotation
        // sign, [relative-velocity thermostat factor]
        if (mine) {
            float3 u = zero3();
            if (n > 0) {
                float lam1 = 1.0f, lam2 = 1.0f;
                bool scale2 = false;
                const float4* V_ = &s_v[w][at0];
                float E = 0.f;
                if (lab)
                    for (uint32_t k = 0; k < n; ++k) {
                        const float4 V = V_[k];
                        const float3 v = f3(V);
                        E += (0.5f * V.w) * dot3(v, v);
                    }
                // reference isokinetic rule: lambda scales every member before the mean
                lam1 = lab ? sqrtf(P.srd_kT / E) : 1.0f;
                float M = 0.f;
#pragma unroll 2
                for (uint32_t k = 0; k < n; ++k) {
                    const float4 V = V_[k];
                    u += V.w * (lab ? scaled_rn(lam1, V) : f3(V));
                    M += V.w;
                }
                if (M > 0.f) {
                    const float inv = 1.0f / M;
                    u = u * inv;
                }
                // rotation by +alpha or -alpha with equal probability
                const bool plus = u01(rng_draw(P, c, step, kRngSrdRot).x) > 0.5f;
                const float sa = plus ? P.srd_sin_a : -P.srd_sin_a;
                if (rel) {
                    uint32_t nrot = 0;
                    float ke = 0.f;
#pragma unroll 2
                    for (uint32_t k = 0; k < n; ++k) {
                        if (k < nbc && !rotate_beads) continue;
                        const float4 V = V_[k];
                        const float3 d = (lab ? scaled_rn(lam1, V) : f3(V)) - u;
                        const float rx = d.x * ca - d.y * sa;
                        const float ry = d.x * sa + d.y * ca;
                        ke += (0.5f * V.w) * (rx * rx + ry * ry);
                        ++nrot;
                    }
                    if (nrot >= 2u && ke > 0.f) {
                        lam2 = sqrtf(((float)(nrot - 1u) * P.srd_kT) / ke);
                        scale2 = true;
                    }
                }
                CellFactors& f = s_f[w][lane];
                f.ux = u.x;
                f.uy = u.y;
                f.uz = u.z;
                f.sa = sa;
                f.lam1 = lam1;
                f.lam2 = lam2;
                f.beads = (b0 + nbc) | (scale2 ? 0x80000000u : 0u);
            }
            if (valid && !big) S.srd_mean[c] = make_float4(u.x, u.y, u.z, 0.f);
        }
        __syncwarp();
        // every member updated by the lane of its slot: rotation, thermostat,
        // solvent streaming; the solvent goes to its place in the new storage
        for (uint32_t j = lane; j < rtotal; j += 32u) {
            uint2 next = make_uint2(0u, 0u);
            float4 next_p = make_float4(0.f, 0.f, 0.f, 0.f);
            if (j + 32u < rtotal) {
                next = s_m[w][j + 32u];
                if (next.x >= P.nb) next_p = sp_old[next.x - P.nb];
            }
            const CellFactors f = s_f[w][m.y];
            const float3 uq = make_float3(f.ux, f.uy, f.uz);
            const bool is_bead = m.x < P.nb;
            const float4 V = s_v[w][j];
            float3 v = lab ? scaled_rn(f.lam1, V) : f3(V);
            if (!is_bead || rotate_beads) {
                const float3 d = v - uq;
                const float rx = fmaf(d.x, ca, -__fmul_rn(d.y, f.sa));
                const float ry = fmaf(d.x, f.sa, __fmul_rn(d.y, ca));
                v = make_float3(uq.x + rx, uq.y + ry, uq.z + d.z);
                if (f.beads >> 31) v = make_float3(uq.x + f.lam2 * (v.x - uq.x), uq.y + f.lam2 * (v.y - uq.y), v.z);
            }
            if (is_bead) {
                if (lab || rotate_beads) bvel[m.x] = make_float4(v.x, v.y, v.z, V.w);
            } else {
                float3 p = f3(P4);
                const float3 dr = dt_srd * v;
                p = make_float3(fmaf(dt_srd, v.x, p.x), fmaf(dt_srd, v.y, p.y), fmaf(dt_srd, v.z, p.z));
                if constexpr (kMode == kAny) apply_boundaries(P, p, v, dr, 0.0f);
                else wrap_periodic(P, p);
                const float3 way = kMode == kAny ? way_of(P, dr, P4, p) : dr;
                moved = max(moved, ordered || near_box(P, p) ? step_bits(P, way) : kEmpty);
                const uint32_t d = (any_big ? f.sorted : sorted0) + j - (f.beads & 0x7fffffffu);
                sp_new[d] = make_float4(p.x, p.y, p.z, P4.w);
                sv_new[d] = make_float4(v.x, v.y, v.z, V.w);
            }
            m = next;
            P4 = next_p;
        }
        __syncwarp();
        first = last + 1u;
    }
    keep_largest_step(S, a ^ 1u, moved);
}

__device__ __forceinline__ float warp_allsum(float x)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// The collision of srd_collide_kernel for one cell of more than kLaneCap
// members, by one warp: members ranked by index in shared memory (the stable
// order; beyond kBigCap members the bucket order, and the overflow is
// reported), velocities gathered once into shared memory, sums as
// lane-strided partials combined by a fixed butterfly (the same result on
// every run), then the per-member update by all lanes.
__global__ void __launch_bounds__(kBigWarps * 32) srd_collide_big_kernel(const DevParams P, const StepBuffers S,
                                                                         uint32_t step_off, float dt_srd,
                                                                         uint32_t buf_sel)
{
    pdl_enter();
    __shared__ uint32_t s_in[kBigWarps][kBigCap];
    __shared__ uint32_t s_id[kBigWarps][kBigCap];
    __shared__ float4 s_v[kBigWarps][kBigCap];
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint32_t nbig = *S.srd_nbig;
    const unsigned long long step = *S.step_base + step_off;
    const uint32_t cur = buf_sel < 2u ? buf_sel : (uint32_t)(step & 1ull);
    const uint32_t a = S.srd_state[kSrdSrc];
    const float4* __restrict__ sv_old = S.svel2[a];
    const float4* __restrict__ sp_old = S.spos2[a];
    float4* __restrict__ sv_new = S.svel2[a ^ 1u];
    float4* __restrict__ sp_new = S.spos2[a ^ 1u];
    const uint32_t* __restrict__ soff = S.srd_soff2[a ^ 1u];
    float4* __restrict__ bvel = S.vel2[cur];
    const bool lab = P.srd_thermo == NW_SRD_THERMO_REF_LAB;
    const bool rel = P.srd_thermo == NW_SRD_THERMO_CELL_REL;
    uint32_t moved = 0u;
    for (uint32_t q = blockIdx.x * kBigWarps + w; q < nbig; q += gridDim.x * kBigWarps) {
        const uint32_t c = S.srd_big[q];
        const uint32_t b0 = S.srd_boff[c], b1 = S.srd_boff[c + 1];
        const uint32_t s0 = soff[c], s1 = soff[c + 1];
        const uint32_t nbc = b1 - b0, n = nbc + (s1 - s0);
        const uint32_t start = b0 + s0;
        // beyond kBigCap members: bucket order, reported, bounded work
        const bool fits = n <= kBigCap;
        if (!fits && lane == 0) atomicOr(S.err, (uint32_t)NW_EFLAG_CELL_OVERFLOW);
        auto raw = [&](uint32_t k) -> uint32_t {
            return k < nbc ? S.srd_btmp[b0 + k] : P.nb + S.srd_stmp[s0 + (k - nbc)];
        };
        if (fits) {
            for (uint32_t k = lane; k < n; k += 32) s_in[w][k] = raw(k);
            __syncwarp();
            uint32_t ranks = 0;
            for (uint32_t k = lane; k < n; k += 32) {
                const uint32_t x = s_in[w][k];
                uint32_t r = 0;
                for (const uint32_t* y = s_in[w]; y < s_in[w] + n; ++y) r += *y < x;
                s_id[w][r] = x;
                ranks += r;
            }
            // ranks of indices that repeat fall short: they would leave places unwritten
            if (__reduce_add_sync(0xffffffffu, ranks) != n * (n - 1u) / 2u)
                for (uint32_t k = lane; k < n; k += 32) s_id[w][rank_of(s_in[w], n, k)] = s_in[w][k];
            __syncwarp();
        }
        auto member = [&](uint32_t k) -> uint32_t { return fits ? s_id[w][k] : raw(k); };
        auto vel_of = [&](uint32_t k, uint32_t id) -> float4 {
            return fits ? s_v[w][k] : (id < P.nb ? bvel[id] : sv_old[id - P.nb]);
        };
        float E = 0.f;
        for (uint32_t k = lane; k < n; k += 32) {
            const uint32_t id = member(k);
            S.srd_sorted_index[start + k] = id;
            const float4 V = id < P.nb ? bvel[id] : sv_old[id - P.nb];
            if (fits) s_v[w][k] = V;
            E += (0.5f * V.w) * (V.x * V.x + V.y * V.y + V.z * V.z);
        }
        __syncwarp();
        E = warp_allsum(E);
        const float lam1 = lab ? sqrtf(P.srd_kT / E) : 1.0f;
        float ux = 0.f, uy = 0.f, uz = 0.f, M = 0.f;
        for (uint32_t k = lane; k < n; k += 32) {
            const float4 V = vel_of(k, member(k));
            const float sx = lab ? lam1 * V.x : V.x, sy = lab ? lam1 * V.y : V.y, sz = lab ? lam1 * V.z : V.z;
            ux += V.w * sx;
            uy += V.w * sy;
            uz += V.w * sz;
            M += V.w;
        }
        ux = warp_allsum(ux);
        uy = warp_allsum(uy);
        uz = warp_allsum(uz);
        M = warp_allsum(M);
        if (M > 0.f) {
            const float inv = 1.0f / M;
            ux *= inv;
            uy *= inv;
            uz *= inv;
        }
        const bool plus = u01(rng_draw(P, c, step, kRngSrdRot).x) > 0.5f;
        const float sa = plus ? P.srd_sin_a : -P.srd_sin_a, ca = P.srd_cos_a;
        float lam2 = 1.0f;
        bool scale2 = false;
        if (rel) {
            float ke = 0.f, nrot = 0.f;
            for (uint32_t k = lane; k < n; k += 32) {
                if (member(k) < P.nb && !P.srd_rotate_beads) continue;
                const float4 V = vel_of(k, member(k));
                const float dx = (lab ? lam1 * V.x : V.x) - ux, dy = (lab ? lam1 * V.y : V.y) - uy;
                const float rx = dx * ca - dy * sa, ry = dx * sa + dy * ca;
                ke += (0.5f * V.w) * (rx * rx + ry * ry);
                nrot += 1.f;
            }
            ke = warp_allsum(ke);
            nrot = warp_allsum(nrot);
            if (nrot >= 2.f && ke > 0.f) {
                lam2 = sqrtf(((nrot - 1.f) * P.srd_kT) / ke);
                scale2 = true;
            }
        }
        for (uint32_t k = lane; k < n; k += 32) {
            const uint32_t id = member(k);
            const bool is_bead = id < P.nb;
            const float4 V = vel_of(k, id);
            float3 v = lab ? make_float3(lam1 * V.x, lam1 * V.y, lam1 * V.z) : f3(V);
            if (!is_bead || P.srd_rotate_beads) {
                const float dx = v.x - ux, dy = v.y - uy, dz = v.z - uz;
                const float rx = dx * ca - dy * sa, ry = dx * sa + dy * ca;
                v = make_float3(ux + rx, uy + ry, uz + dz);
                if (scale2) v = make_float3(ux + lam2 * (v.x - ux), uy + lam2 * (v.y - uy), v.z);
            }
            if (is_bead) {
                if (lab || P.srd_rotate_beads) bvel[id] = make_float4(v.x, v.y, v.z, V.w);
            } else {
                const float4 P4 = sp_old[id - P.nb];
                float3 p = f3(P4);
                const float3 dr = dt_srd * v;
                p = make_float3(fmaf(dt_srd, v.x, p.x), fmaf(dt_srd, v.y, p.y), fmaf(dt_srd, v.z, p.z));
                apply_boundaries(P, p, v, dr, 0.0f);
                moved = max(moved, near_box(P, p) ? step_bits(P, way_of(P, dr, P4, p)) : kEmpty);
                const uint32_t dst = s0 + (k - nbc);
                sp_new[dst] = make_float4(p.x, p.y, p.z, P4.w);
                sv_new[dst] = make_float4(v.x, v.y, v.z, V.w);
            }
        }
        if (lane == 0) S.srd_mean[c] = make_float4(ux, uy, uz, 0.f);
        __syncwarp();
    }
    keep_largest_step(S, a ^ 1u, moved);
}

}  // namespace

#define NW_MARK(name) \
    if (prof) prof->mark(name)

uint64_t enqueue_srd(const DevParams& P, const StepBuffers& B, uint32_t srd_nchunks, uint32_t step_off, float dt_srd,
                     int shift_from_step, float3 shift, cudaStream_t s, Prof* prof, uint32_t buf_sel)
{
    if (P.ntotal == 0) return 0;
    const uint32_t some = 1u;  // every kernel is launched also for no beads or no solvent
    NW_MARK("srd_bead_hash");
    launch_pdl(srd_bead_hash_kernel, std::max(some, cdiv(P.nb, 256)), 256, 0, s, P, B, step_off, shift_from_step, shift,
               buf_sel);
    NW_MARK("srd_hash");
    launch_pdl(srd_hash_kernel, std::max(some, cdiv(P.ns, 256 * kHashPer)), 256, 0, s, P, B);
    NW_MARK("srd_chunk_sum");
    // bead and solvent counts side by side (grid rows 0 and 1)
    launch_pdl(chunk_sum_kernel, dim3(srd_nchunks, 2), 512, 0, s, B.srd_bcount, P.srd_ncells, B.srd_bchunk,
               B.srd_scount, B.srd_schunk);
    NW_MARK("srd_scan_cells");
    // the offsets of the buffer that this collision fills: [1] when it reads buffer 0
    launch_pdl(scan_cells_kernel<false>, dim3(srd_nchunks, 2), 512, 0, s, B.srd_bcount, B.srd_bchunk, P.srd_ncells,
               B.srd_boff, nullptr, nullptr, B.srd_scount, B.srd_schunk, B.srd_soff2[1], B.srd_soff2[0],
               B.srd_state + kSrdSrc);
    NW_MARK("srd_scatter");
    launch_pdl(srd_scatter_kernel, std::max(some, std::min(cdiv(P.ns, 256), 8u * 152u)), 256, 0, s, P, B);
    NW_MARK("srd_collide");
    const bool periodic = P.bnd[0] == NW_PERIODIC && P.bnd[1] == NW_PERIODIC && P.bnd[2] == NW_PERIODIC;
    auto* collide = periodic && P.srd_thermo == NW_SRD_THERMO_CELL_REL && P.srd_rotate_beads
                        ? srd_collide_kernel<kRelative>
                    : periodic && P.srd_thermo == NW_SRD_THERMO_REF_LAB && !P.srd_rotate_beads
                        ? srd_collide_kernel<kLab>
                        : srd_collide_kernel<kAny>;
    const bool dense = (uint64_t)P.ntotal > 8ull * P.srd_ncells;
    launch_pdl(collide, cdiv(P.srd_ncells, kCollideWarps * 32), kCollideWarps * 32, 0, s, P, B, step_off, dt_srd,
               buf_sel);
    NW_MARK("srd_collide_big");
    // Few cells of a fresh dilute solvent are big, but many of a late state,
    // crowded at walls or by the beads: a block for 1,024 cells and at least one
    // an SM, two between walls; in a dense solvent for 256 cells and at least two
    // an SM.  Calls of ten updates, after 200 of them / 60,000, us, with a block for
    // 1,024 cells alone, with 152 blocks at least, 304, and 912 always: 22,056 beads
    // 58.0 / 84.2, 58.6 / 76.4, 59.2 / 75.2, 63.1 / 80.5; 5,460 between walls
    // 61.4 / 99, 61.8 / 79.0, 62.3 / 77.5, 64.9 / 83; 11,925 between walls 83.4 / 140,
    // 84.0 / 121, 84.4 / 114.5, late 118 with 912; 30,000 between walls 68.0 / 130,
    // 68.7 / 123, 69.3 / 108.6, late 109.  Dense, five updates after 100 / 12,500,
    // with a block for four cells (up to 912) and with 304: 4,800 REF_DEM beads on
    // 64 x 64 solvent cells 86.5 / 97, 78.3 / 89.5; 72,000 on 256 x 256 153 / 163,
    // 142 / 153; 180,000 on 512 x 512 331 / 342, 326 / 346.
    const uint32_t big_blocks =
        std::max(dense || !periodic ? 304u : 152u, cdiv(P.srd_ncells, dense ? 256u : 1024u));
    launch_pdl(srd_collide_big_kernel, std::min(kSrdBigBlocks, big_blocks), kBigWarps * 32, 0, s, P, B, step_off,
               dt_srd, buf_sel);
    return 7;
}

}  // namespace nw
