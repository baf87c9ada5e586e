// nw_fused.cuh — launchers of the cell-list step path (nw_fused.cu, nw_fused_planar.cu;
// device code in nw_fused_impl.cuh).
#pragma once

#include "nw_kernels.cuh"

namespace nw {

// Options of the pro part of the single-system kernels:
//   kProLazyTangent  tangents are not stored by the step (WCA worms of more
//                    than three beads, whose step never reads them); the
//                    handle API computes them when they are read
//   kProInsert       every update's pro part fills its cell list, and no
//                    bead_list launch follows (inserts())
constexpr uint32_t kProLazyTangent = 1u, kProInsert = 2u;
__host__ __device__ __forceinline__ uint32_t pro_flags(const DevParams& P)
{
    return P.model == NW_MODEL_WCA_WORMS && P.L > 3u ? kProLazyTangent : 0u;
}
// Small Verlet systems fill every update's cell list in the pro part, although
// only list builds read it: the atomics and the clearing cost less than a
// launch that mostly leaves at once (about 1.2 us).  That holds while the
// threads of two successive updates fit the chip together, six blocks of 256 on
// each of 152 SMs, so that the next update's blocks wait on the chip and not
// for it.  40 updates of planar beads, filled in the pro part / by the launch
// (us): 60,000 264 / 274, 80,000 281 / 299, 110,000 285 / 310, 120,000 403 / 320,
// 130,000 405 / 351; 20 in 3D: 80,000 216 / 219, 100,000 232 / 227, 130,000
// 286 / 256; ten with SRD: 40,000 101 / 103, 100,000 134 / 131, 130,000
// 164 / 149.  Calls of one update keep the launch.
constexpr uint64_t kInsertThreads = 152ull * 6ull * 256ull / 2ull;
bool inserts(const DevParams& P, int nsteps);

// Within one call, the bead state of planar Verlet systems between updates is
// packed: two float4 a bead (x, y, velocity; partial and previous force)
// instead of four, since z, the radius and the mass stay as they are and the
// forces have z = 0.  The first update reads and the last writes the API's
// arrays, and so does an update with a collision, which reads and changes bead
// velocities in them.  A kernel that leaves the packed form takes z, radius
// and mass from the buffer of the last update that wrote the API's arrays.
// 40 updates of 2,000,000 beads: 3.76 -> 3.15 ms (128 of 306 MB a launch less),
// ten of 400,000 with SRD 327 -> 301 us, 20 of 64 replicas 1.23 -> 1.12 ms.
constexpr uint32_t kPackedIn = 1u, kPackedOut = 2u;
__host__ __device__ __forceinline__ bool packs(const DevParams& P)
{
    return planar_system(P) && P.vl_on && !P.reverse_on && P.lgrid[2] == 1u && P.L <= 256u &&
           (pro_flags(P) & kProLazyTangent) != 0u;
}
// Tangents of the current positions as the pro part computes them.
uint64_t launch_bead_tangents(const DevParams& P, const float4* pos, float4* tan, cudaStream_t s);

// Threads per block of the bead kernels: 256 where that gives every SM two
// blocks, else 128, so that a small system's warps spread over the SMs (their
// latency is what counts there).  128 / 256, us: 40 updates of planar beads
// 4,000 210 / 220, 40,000 238 / 245, 77,000 260 / 269, 160,000 350 / 358, 300,000
// 527 / 517; 20 in 3D: 26,000 176 / 181, 50,000 186 / 192, 77,000 203 / 198,
// 120,000 283 / 283; ten with SRD: 10,000 83.5 / 84.4, 25,000 90.3 / 89.6, 50,000
// 95.2 / 96.1, 77,000 112 / 111 (several systems of 10,000 in turn 45.8 / 44.9).
uint32_t bead_threads(uint64_t nb);
// Filaments per block of the filament-aligned kernels (about bead_threads).
uint32_t list_filaments_per_block(uint32_t L, uint32_t nf);

// pro(n) with n = *step_base + off: integrate .. hash, insert into list n.
// packed: kPackedOut or 0.
// insert: kProInsert or 0.
uint64_t launch_bead_pro(const DevParams& P, const StepBuffers& B, uint32_t off, float dt, uint32_t packed,
                         uint32_t insert, cudaStream_t s);
// Verlet systems: the cell list of update n, built only when the pair pass
// of update n rebuilds the neighbour lists (launch after the pro part of n).
// packed: whether update n left its state packed.
uint64_t launch_bead_list(const DevParams& P, const StepBuffers& B, uint32_t off, bool packed, cudaStream_t s);
// epi(n): pair forces from list n; force = complete F_n.
uint64_t launch_bead_epi(const DevParams& P, const StepBuffers& B, uint32_t off, cudaStream_t s);
// epi(n) followed by pro(n+1) in one kernel; packed: kPackedIn | kPackedOut;
// from: parity of the offset of the last update in the API's arrays (-1, the
// state before the call, is odd).
uint64_t launch_bead_fused(const DevParams& P, const StepBuffers& B, uint32_t off, float dt, uint32_t packed,
                           uint32_t from, uint32_t insert, cudaStream_t s);

// ---- batched replicas (nw_batch.cu) ------------------------------------------

// One replica of a batch as its blocks see it: its parameter block and where
// its beads, list cells, neighbour lists and blocks start in the batch's
// concatenated buffers.
struct ReplicaSlot {
    DevParams P;
    float dt;
    uint32_t bead_off;  // first bead
    uint32_t cell_off;  // first list cell
    uint32_t blk0;      // first block of the launch
    uint32_t nblk;      // blocks of this replica
    uint32_t fpb;       // filaments per block
    uint32_t lblk0, lnblk;  // the same of the list launch (list_blocks of the replica's beads)
    unsigned long long nbr_off;  // first neighbour-list word
};

// kBatchList: a replica's cell list of update n when its pair pass will
// rebuild the Verlet lists (Verlet replicas; launched after each pro part), by
// list_blocks blocks of a replica, which mostly leave at once
enum BatchMode { kBatchPro = 0, kBatchEpi = 1, kBatchFused = 2, kBatchList = 3 };

// Blocks that build one replica's cell list: up to eight, and eight beads a
// thread, four of them in flight, from 16,384 beads (of 256 threads) on.  The
// launch costs with its blocks where no replica rebuilds, a rebuild with the
// beads of a thread.  20 updates of replicas x beads, eight blocks each whatever
// the size / this rule / a thread a bead, us: 1 x 400,000 549 / 350 / 390,
// 16 x 100,000 1,803 / 1,301 / 1,540, 8 x 60,000 630 / 483 / 513, 64 x 60,000
// 3,555 / 3,049 / 3,541, 64 x 20,000 1,261 / 1,187 / 1,386, 64 x 4,000
// 471 / 473 / 489; 16 beads a thread 8 x 60,000 517, four 466, but 64 uneven
// replicas of 250 to 60,000 beads 1,057 instead of 1,038 (1,031 with eight blocks).
inline uint32_t list_blocks(uint32_t beads, uint32_t threads)
{
    const uint32_t one = (beads + threads - 1u) / threads, eight = (one + 7u) / 8u;  // blocks for one and eight beads a thread
    return eight > 8u ? eight : one < 8u ? one : 8u;
}
// One launch over all replicas: block b serves replica block_rep[b].  S holds
// the batch's base pointers; `threads` >= every replica's fpb * L; planar =
// every replica is a planar system.
void launch_batch(int mode, const ReplicaSlot* table, const uint32_t* block_rep, uint32_t blocks, uint32_t threads,
                  size_t smem, uint32_t cap, const StepBuffers& S, uint32_t off, bool planar, uint32_t packed,
                  cudaStream_t s);

// The two-component launches (nw_fused_planar.cu) behind the launchers above.
uint64_t launch_bead_pro_planar(const DevParams& P, const StepBuffers& B, uint32_t off, float dt, uint32_t packed,
                                uint32_t insert, cudaStream_t s);
uint64_t launch_bead_tangents_planar(const DevParams& P, const float4* pos, float4* tan, cudaStream_t s);
uint64_t launch_bead_epi_planar(const DevParams& P, const StepBuffers& B, uint32_t off, cudaStream_t s);
uint64_t launch_bead_fused_planar(const DevParams& P, const StepBuffers& B, uint32_t off, float dt, uint32_t packed,
                                  uint32_t from, uint32_t insert, cudaStream_t s);
void launch_batch_planar(int mode, const ReplicaSlot* table, const uint32_t* block_rep, uint32_t blocks,
                         uint32_t threads, size_t smem, uint32_t cap, const StepBuffers& S, uint32_t off,
                         uint32_t packed, cudaStream_t s);

}  // namespace nw
