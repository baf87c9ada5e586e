// nw_kernels.cu — definitions of the non-template step kernels declared in
// nw_kernels.cuh (one translation unit owns each kernel).
#include "nw_kernels.cuh"

namespace nw {

namespace {

// The filament pass with D vector components (D = 2: planar systems).
template <int D>
__device__ __forceinline__ void filament_pass(const DevParams& P, const StepBuffers& S, uint32_t step_off, float dt,
                                              uint32_t fpb)
{
    extern __shared__ float4 sm[];
    const uint32_t L = P.L;
    const uint32_t beads = fpb * L;
    const uint32_t t = threadIdx.x;
    const uint32_t w0 = blockIdx.x * fpb;
    const uint32_t i = w0 * L + t;
    const bool active = t < beads && i < P.nb;
    const unsigned long long step = *S.step_base + step_off;

    float4 nP = make_float4(0.f, 0.f, 0.f, 0.f), nV = nP, nFo = nP;
    if (active) {
        const float4 P4 = S.pos[i], V4 = S.vel[i], F4 = S.force[i], Fo4 = S.force_old[i];
        float3 p = f3(P4), v = f3(V4);
        const float3 f = f3(F4), fo = f3(Fo4);
        // velocity Verlet (particles_kernel_impl.cuh:93-97), per axis
        auto verlet = [dt](float fa, float foa, float& va, float& pa) {
            va += (0.5f * (fa + foa)) * dt;
            const float d = va * dt + ((0.5f * fa) * dt) * dt;
            pa += d;
            return d;
        };
        float3 dr;
        dr.x = verlet(f.x, fo.x, v.x, p.x);
        dr.y = verlet(f.y, fo.y, v.y, p.y);
        dr.z = D == 3 ? verlet(f.z, fo.z, v.z, p.z) : 0.f;
        apply_boundaries<D>(P, p, v, dr, P.radius);
        nP = make_float4(p.x, p.y, p.z, P4.w);
        nV = make_float4(v.x, v.y, v.z, V4.w);
        nFo = make_float4(f.x, f.y, D == 3 ? f.z : 0.f, Fo4.w);
    }
    if (P.reverse_on) {
        // reverseFilamentsKernel (particles_kernel_impl.cuh:820-857)
        if (active) {
            sm[t] = nP;
            sm[beads + t] = nV;
            sm[2 * beads + t] = nFo;
        }
        __syncthreads();
        if (active) {
            const uint32_t wl = t / L, c = t - wl * L;
            const float u = u01(rng_draw(P, w0 + wl, step, kRngReverse).x);
            if (u <= P.reverse_p) {
                const uint32_t src = wl * L + (L - 1u - c);
                nP = sm[src];
                nV = sm[beads + src];
                nFo = sm[2 * beads + src];
            }
        }
        __syncthreads();
    }
    if (active) sm[t] = nP;
    __syncthreads();
    if (!active) return;

    const uint32_t wl = t / L, c = t - wl * L;
    const float4* R = sm + wl * L;
    float3 fs = zero3();
    if (P.langevin_on) {
        // langevinKernel (particles_kernel_impl.cuh:859-874), Philox noise in registers
        const float3 g = noise3(P, rng_draw(P, i, step, kRngLangevin));
        float3 fl = zero3() - P.gamma * f3(nV);
        fl += g;
        fs = D == 3 ? fl : make_float3(fl.x, fl.y, 0.f);
    }
    // bending contributions in the reference's triple order p = c-2, c-1, c
    if (L >= 3) {
        if (c >= 2) fs = addv<D>(fs, bend_triple<D>(P, f3(R[c - 2]), f3(R[c - 1]), f3(R[c])).fk);
        if (c >= 1 && c + 1 < L) fs = addv<D>(fs, bend_triple<D>(P, f3(R[c - 1]), f3(R[c]), f3(R[c + 1])).fj);
        if (c + 2 < L) fs = addv<D>(fs, bend_triple<D>(P, f3(R[c]), f3(R[c + 1]), f3(R[c + 2])).fi);
    }
    bool wt = false;
    float3 tg = zero3();
    if (L >= 3) {
        if (c == 0) {
            tg = tangent_of<D>(P, f3(R[0]), f3(R[1]));
            wt = true;
        } else if (c == L - 1) {
            if (L > 3) {
                tg = tangent_of<D>(P, f3(R[L - 2]), f3(R[L - 1]));
                wt = true;
            }
        } else {
            tg = tangent_of<D>(P, f3(R[c - 1]), f3(R[c + 1]));
            wt = true;
        }
    }
    if (P.model == NW_MODEL_WCA_WORMS) {
        const float3 me = f3(R[c]);
        if (c > 0) wca_bond<D>(P, me, f3(R[c - 1]), fs);
        if (c + 1 < L) wca_bond_drive<D>(P, me, f3(R[c + 1]), fs);
    }
    S.pos[i] = nP;
    S.vel[i] = nV;
    S.force_old[i] = nFo;
    S.force[i] = make_float4(fs.x, fs.y, fs.z, 0.f);
    if (wt) S.tangent[i] = make_float4(tg.x, tg.y, tg.z, 0.f);
    if (!finitev<D>(f3(nP)) || !finitev<D>(fs)) atomicOr(S.err, (uint32_t)NW_EFLAG_NONFINITE);

    const uint32_t h = bead_hash(P, f3(nP));
    S.hash[i] = h;
    S.slot[i] = count_into_cell(S.cell_count, h);
}

}  // namespace

__global__ void __launch_bounds__(1024) filament_pass_kernel(const DevParams P, const StepBuffers S, uint32_t step_off,
                                                             float dt, uint32_t fpb)
{
    pdl_enter();
    if (planar_system(P)) filament_pass<2>(P, S, step_off, dt, fpb);
    else filament_pass<3>(P, S, step_off, dt, fpb);
}

__global__ void __launch_bounds__(512) chunk_sum_kernel(const uint32_t* __restrict__ a, uint32_t m,
                                                        uint32_t* __restrict__ chunk, const uint32_t* __restrict__ a2,
                                                        uint32_t* __restrict__ chunk2)
{
    pdl_enter();
    if (blockIdx.y) {
        a = a2;
        chunk = chunk2;
    }
    __shared__ uint32_t s_w[16];
    const uint32_t c0 = blockIdx.x * kChunk;
    uint32_t x = 0;
    if (c0 + kChunk <= m) {
        const uint4* v = reinterpret_cast<const uint4*>(a + c0);
        for (uint32_t k = threadIdx.x; k < kChunk / 4u; k += 512u) {
            const uint4 q = v[k];
            x += q.x + q.y + q.z + q.w;
        }
    } else {
        for (uint32_t k = threadIdx.x; k < kChunk; k += 512u)
            if (c0 + k < m) x += a[c0 + k];
    }
    x = warp_sum(x);
    if ((threadIdx.x & 31u) == 0) s_w[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x < 32) {
        uint32_t y = threadIdx.x < 16 ? s_w[threadIdx.x] : 0u;
        y = warp_sum(y);
        if (threadIdx.x == 0) chunk[blockIdx.x] = y;
    }
}

__global__ void __launch_bounds__(256) scatter_kernel(const uint32_t* __restrict__ hash,
                                                      const uint32_t* __restrict__ slot,
                                                      const uint32_t* __restrict__ offset, uint32_t* __restrict__ tmp,
                                                      uint32_t n)
{
    pdl_enter();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) tmp[offset[hash[i]] + slot[i]] = i;
}

// collideFilamentsKernel's force on the bead at sorted position p, from the
// sorted arrays in global memory (added to force[original index]).
__device__ __forceinline__ void ref_pair_bead(const DevParams& P, const StepBuffers& S, uint32_t p)
{
    const float3 r = f3(S.sorted_pos[p]);
    const float3 v = f3(S.sorted_vel[p]);
    const float3 t = f3(S.sorted_tan[p]);
    const int3 g = grid_pos(P, r);
    const uint32_t me = S.sorted_index[p];
    if (me >= P.nb) {
        atomicOr(S.err, (uint32_t)NW_EFLAG_BAD_INDEX);
        return;
    }
    const uint32_t fI = me / P.L, cI = me - fI * P.L;
    float3 total = zero3();
    if (P.grid[2] == 1u) {
        float3 cs[9];
#pragma unroll
        for (int y = -1; y <= 1; ++y)
#pragma unroll
            for (int x = -1; x <= 1; ++x) {
                const uint32_t h = cell_hash(P, cell_coord(P, 0, g.x + x), cell_coord(P, 1, g.y + y), cell_coord(P, 2, g.z));
                cs[(y + 1) * 3 + (x + 1)] = ref_cell_sum(P, S, h, p, r, v, t, fI, cI);
            }
#pragma unroll
        for (int z = 0; z < 3; ++z)
#pragma unroll
            for (int k = 0; k < 9; ++k) total += cs[k];
    } else {
        for (int z = -1; z <= 1; ++z)
            for (int y = -1; y <= 1; ++y)
                for (int x = -1; x <= 1; ++x) {
                    const uint32_t h =
                        cell_hash(P, cell_coord(P, 0, g.x + x), cell_coord(P, 1, g.y + y), cell_coord(P, 2, g.z + z));
                    total += ref_cell_sum(P, S, h, p, r, v, t, fI, cI);
                }
    }
    float4 F = S.force[me];
    F.x += total.x;
    F.y += total.y;
    F.z += total.z;
    S.force[me] = F;
    if (!finite3(f3(F))) atomicOr(S.err, (uint32_t)NW_EFLAG_NONFINITE);
}

__global__ void __launch_bounds__(256) pair_ref_kernel(const DevParams P, const StepBuffers S)
{
    pdl_enter();
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < P.nb) ref_pair_bead(P, S, p);
}

// ---- REF_DEM pair pass of a single z layer -------------------------------------
//
// The thread-per-bead form above (the reference's own layout) spends most of
// its issue slots on divergence: each lane walks 27 cells of 0-2 members and
// branches per member (8 of 32 lanes active in the reference's kernel on the
// 400k-bead lattice).  Here a group of kRefG lanes serves a bead and strides
// over its candidates: the members of the 3 x 3 cells around its own, three
// contiguous runs of the sorted arrays (one per row, cells x-1 .. x+1), whose
// ends are two cell offsets each.  Neighbouring beads share their runs, so the
// gathers hit L1.  A bead's candidates enter four partial sums in turn, two a
// lane, combined in a fixed order, so results do not depend on scheduling.  With one z layer
// every (x, y) neighbour cell is reached by the reference's three z offsets,
// so the bead's sum is added three times; a cell reached by two x or y offsets
// (grids narrower than 3 cells, walls) is visited twice, as in the reference.
// Same pair laws as collideCell (particles_kernel_impl.cuh:427-556), with the
// divisions by the separation taken from a Newton-refined reciprocal.
//
// 400,000 beads on 1,024 x 1,024 cells (3.4 candidates a bead): 116 us with
// tiles of 32 x 4 cells and their halo staged in shared memory (59 KB and six
// barriers a block for 49 beads); 53 us with four lanes a bead, 41 us with two
// (24M warp instructions; the pair law of the longest of 16 beads' lists).

__device__ __forceinline__ float3 ref_pair_law(const DevParams& P, float3 r, float3 v, float3 t, float3 r2, float3 v2,
                                               float3 t2, bool same, bool bonded)
{
    float3 rel = r2 - r;
    min_image(P, rel);
    const float q = dot3(rel, rel);
    const float d = sqrt_nr(q, rsqrtf(q));
    const float id = rcp_nr(d);
    const float3 n = rel * id;
    float3 F = zero3();
    const float cd = P.radius + P.radius;
    if (bonded) {
        // bondHookean (:466-473)
        F = (-P.bond_k * (P.bond_r0 - d)) * n;
    } else if (d < cd) {
        // collideParticles (:427-462)
        const float3 rv = v2 - v;
        const float3 tv = rv - dot3(rv, n) * n;
        F = (-P.spring * (cd - d)) * n;
        F += P.damping * rv;
        F += P.shear * tv;
    }
    // extensileForce (:477-487): other filaments, anti-aligned tangents
    if (!same && dot3(t, t2) < -0.5f) F += ((-P.activity) * (t - t2)) * (0.5f * id);
    return F;
}


__global__ void __launch_bounds__(256) pair_ref_runs_kernel(const DevParams P, const StepBuffers S)
{
    pdl_enter();
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t p = t / kRefG, g = t % kRefG;
    const bool live = p < P.nb;
    float3 s0 = zero3(), s1 = zero3();  // candidates g, g + 4, .. and g + 2, g + 6, ..
    uint32_t me = 0;
    if (live) {
        me = S.sorted_index[p];
        const uint32_t h = S.sorted_hash[p];
        const float3 r = f3(S.sorted_pos[p]), v = f3(S.sorted_vel[p]), tn = f3(S.sorted_tan[p]);
        const uint32_t fbase = me - me % P.L;
        struct Candidate {
            uint32_t o;
            float4 r, v, t;
        };
        auto fetch = [&](uint32_t j) -> Candidate {
            return Candidate{__ldg(&S.sorted_index[j]), __ldg(&S.sorted_pos[j]), __ldg(&S.sorted_vel[j]),
                             __ldg(&S.sorted_tan[j])};
        };
        auto visit = [&](const Candidate& c, float3& sum) {
            if (c.o == me) return;
            const bool same = c.o - fbase < P.L;
            sum += ref_pair_law(P, r, v, tn, f3(c.r), f3(c.v), f3(c.t), same,
                                same && (c.o == me + 1u || c.o + 1u == me));
        };
        const uint32_t y = fast_div(h, P.div_gx_m, P.div_gx_k), x = h - y * P.grid[0];
        const bool inside = x >= 1u && x + 1u < P.grid[0];
        uint32_t a[3], n[3];
#pragma unroll
        for (int dy = 0; dy < 3; ++dy) {
            const uint32_t c = cell_hash(P, x, cell_coord(P, 1, (int)y + dy - 1), 0u);
            a[dy] = n[dy] = 0u;
            if (inside) {
                a[dy] = S.cell_offset[c - 1u];
                n[dy] = min(S.cell_offset[c + 2u] - a[dy], 3u * kPairCap);  // longer runs were reported by the sort
            }
        }
        if (inside) {
            const uint32_t m = n[0] + n[1] + n[2];
            auto at = [&](uint32_t k) {
                return k < n[0] ? a[0] + k : (k < n[0] + n[1] ? a[1] + (k - n[0]) : a[2] + (k - n[0] - n[1]));
            };
            for (uint32_t k = g; k < m; k += 4u) {
                const bool two = k + 2u < m;
                const Candidate c0 = fetch(at(k)), c1 = fetch(two ? at(k + 2u) : p);  // p: itself, passed over
                visit(c0, s0);
                visit(c1, s1);
            }
        } else {
            uint32_t k = 0;  // candidates before the cell
            for (int dy = -1; dy <= 1; ++dy)
                for (int dx = -1; dx <= 1; ++dx) {
                    const uint32_t c = cell_hash(P, cell_coord(P, 0, (int)x + dx), cell_coord(P, 1, (int)y + dy), 0u);
                    const uint32_t b = S.cell_offset[c], m = min(S.cell_offset[c + 1u] - b, kPairCap);
                    for (uint32_t q = (g - k) % kRefG; q < m; q += kRefG)
                        visit(fetch(b + q), ((k + q) & 2u) ? s1 : s0);
                    k += m;
                }
        }
    }
    // ((0 + 1) + (2 + 3)) of the four partial sums, whatever the group's size
    static_assert(kRefG == 2, "two lanes, two partial sums each");
    float3 sum;
    sum.x = (s0.x + __shfl_xor_sync(0xffffffffu, s0.x, 1)) + (s1.x + __shfl_xor_sync(0xffffffffu, s1.x, 1));
    sum.y = (s0.y + __shfl_xor_sync(0xffffffffu, s0.y, 1)) + (s1.y + __shfl_xor_sync(0xffffffffu, s1.y, 1));
    sum.z = (s0.z + __shfl_xor_sync(0xffffffffu, s0.z, 1)) + (s1.z + __shfl_xor_sync(0xffffffffu, s1.z, 1));
    if (live && g == 0) {
        if (me >= P.nb) {
            atomicOr(S.err, (uint32_t)NW_EFLAG_BAD_INDEX);
            return;
        }
        const float3 tot = (sum + sum) + sum;  // the three z offsets of one layer
        float4 F = S.force[me];
        F.x += tot.x;
        F.y += tot.y;
        F.z += tot.z;
        S.force[me] = F;
        if (!finite3(f3(F))) atomicOr(S.err, (uint32_t)NW_EFLAG_NONFINITE);
    }
}

namespace {

// WCA pair forces from the sorted arrays with D vector components.
template <int D>
__device__ __forceinline__ void pair_wca(const DevParams& P, const StepBuffers& S)
{
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= P.nb) return;
    const float3 r = f3(S.sorted_pos[p]);
    const uint32_t me = S.sorted_index[p];
    if (me >= P.nb) {
        atomicOr(S.err, (uint32_t)NW_EFLAG_BAD_INDEX);
        return;
    }
    const uint32_t fbase = (me / P.L) * P.L;
    float3 f = zero3();
    for_neighbour_cells<false>(P, r, S.sorted_hash[p], [&](uint32_t h) {
        uint32_t s0, s1;
        if (!cell_range(P, S, h, s0, s1)) return;
        for (uint32_t j = s0; j < s1; ++j) {
            if (j == p) continue;
            const uint32_t o = __ldg(&S.sorted_index[j]);
            if (lj_excluded(P, me, o, fbase)) continue;
            float3 dr = subv<D>(f3(__ldg(&S.sorted_pos[j])), r);
            min_image_near<D>(P, dr);
            const float rr = dotv<D>(dr, dr);
            if (rr > P.lj_rc2) continue;
            sub_scaled<D>(f, wca_lj(P, rr), dr);
        }
    });
    float4 F = S.force[me];
    F.x += f.x;
    F.y += f.y;
    if constexpr (D == 3) F.z += f.z;
    S.force[me] = F;
    if (!finitev<D>(f3(F))) atomicOr(S.err, (uint32_t)NW_EFLAG_NONFINITE);
}

}  // namespace

__global__ void __launch_bounds__(256) pair_wca_kernel(const DevParams P, const StepBuffers S)
{
    pdl_enter();
    if (planar_system(P)) pair_wca<2>(P, S);
    else pair_wca<3>(P, S);
}

__global__ void advance_step_kernel(unsigned long long* step_base, unsigned long long k)
{
    pdl_enter();
    *step_base += k;
}

}  // namespace nw

namespace {

__global__ void math_probe_kernel(const float* a, const float* b, uint32_t n, float4* out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float x = a[i], y = b[i];
    const float r = rsqrtf(x);
    out[i] = make_float4(nw::rcp_nr(x), nw::sqrt_nr(x, r), nw::div_nr(x, y), r);
}

}  // namespace

extern "C" nw_status nw_math_probe(const float* a, const float* b, uint32_t n, float* out)
{
    if (!a || !b || !out) return NW_ERR_INVALID;
    if (n == 0) return NW_OK;
    float *da = nullptr, *db = nullptr, *dout = nullptr;
    cudaError_t e = cudaMalloc(&da, (size_t)n * 4);
    if (e == cudaSuccess) e = cudaMalloc(&db, (size_t)n * 4);
    if (e == cudaSuccess) e = cudaMalloc(&dout, (size_t)n * 16);
    if (e == cudaSuccess) e = cudaMemcpy(da, a, (size_t)n * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(db, b, (size_t)n * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        math_probe_kernel<<<(n + 255) / 256, 256>>>(da, db, n, reinterpret_cast<float4*>(dout));
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, dout, (size_t)n * 16, cudaMemcpyDeviceToHost);
    cudaFree(da);
    cudaFree(db);
    cudaFree(dout);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return NW_ERR_CUDA;
    }
    return NW_OK;
}
