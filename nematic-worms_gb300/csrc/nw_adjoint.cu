// nw_adjoint.cu — differentiable rollout of the WCA worm step
// (include/nwgb_adjoint.h): a forward pass on frozen neighbour lists with a
// fixed noise realisation, checkpoints every `segment` steps, and a
// hand-written adjoint of the force and integrate steps.
//
// Step of update m (mass 1, the engine's ordering):
//   v_m = v_{m-1} + dt/2 (F_{m-1} + F_{m-2})
//   r_m = wrap(r_{m-1} + dt v_m + dt^2/2 F_{m-1})
//   F_m = -gamma v_m + sigma xi_m + Fc(r_m; theta)
// with Fc = eps F_lj + k_bend F_bend + k_bond F_bond + F_act F_drive (each
// term linear in its parameter).  Adjoint of update m, from the adjoints
// (lr, lv, lF, lFo) of (r_m, v_m, F_m, F_{m-1}):
//   lr~ = lr + Jc^T lF          lv~ = lv - gamma lF + dt lr~
//   lF(m-1) = lFo + dt^2/2 lr~ + dt/2 lv~,   lFo(m-1) = dt/2 lv~
//   lr(m-1) = lr~,  lv(m-1) = lv~,  dL/dtheta_k += lF . F_k(r_m)
// Jc^T lF: the LJ, bond and bending terms are conservative (symmetric
// Jacobian), so Jc^T lF = Jc lF is taken as a directional derivative (dual
// numbers for the bending triple, closed forms for the central pair laws);
// the drive F_i = F_act (r_{i+1} - r_i)/|.| is not, and is transposed
// explicitly.  Every bead's output has one writer; per-block parameter
// gradients are summed in a fixed order, so runs are bit-reproducible.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "../../include/nwgb_adjoint.h"
#include "nw_engine.h"

using namespace nw;

namespace {

// Vectors of N components: three, or two where the whole state lies in the
// plane (planar below).
template <class T, int N>
struct Vec {
    T c[N];
};
#define NW_EACH _Pragma("unroll") for (int q = 0; q < N; ++q)
template <class T, int N>
__device__ __forceinline__ Vec<T, N> zero()
{
    Vec<T, N> r;
    NW_EACH r.c[q] = T(0);
    return r;
}
template <class T, int N>
__device__ __forceinline__ Vec<T, N> operator+(Vec<T, N> a, Vec<T, N> b)
{
    Vec<T, N> r;
    NW_EACH r.c[q] = a.c[q] + b.c[q];
    return r;
}
template <class T, int N>
__device__ __forceinline__ Vec<T, N> operator-(Vec<T, N> a, Vec<T, N> b)
{
    Vec<T, N> r;
    NW_EACH r.c[q] = a.c[q] - b.c[q];
    return r;
}
template <class T, int N>
__device__ __forceinline__ Vec<T, N> operator-(Vec<T, N> a)
{
    Vec<T, N> r;
    NW_EACH r.c[q] = -a.c[q];
    return r;
}
template <class T, int N, class S>
__device__ __forceinline__ Vec<T, N> operator*(S s, Vec<T, N> a)
{
    Vec<T, N> r;
    NW_EACH r.c[q] = T(s) * a.c[q];
    return r;
}
template <class T, int N>
__device__ __forceinline__ T dot(Vec<T, N> a, Vec<T, N> b)
{
    if constexpr (N == 2) return a.c[0] * b.c[0] + a.c[1] * b.c[1];
    else return a.c[0] * b.c[0] + a.c[1] * b.c[1] + a.c[2] * b.c[2];
}

// Dual number a + b e (e^2 = 0): value and directional derivative.
template <class T>
struct D {
    T v, d;
};
template <class T>
__device__ __forceinline__ D<T> operator+(D<T> a, D<T> b)
{
    return D<T>{a.v + b.v, a.d + b.d};
}
template <class T>
__device__ __forceinline__ D<T> operator-(D<T> a, D<T> b)
{
    return D<T>{a.v - b.v, a.d - b.d};
}
template <class T>
__device__ __forceinline__ D<T> operator-(D<T> a)
{
    return D<T>{-a.v, -a.d};
}
template <class T>
__device__ __forceinline__ D<T> operator*(D<T> a, D<T> b)
{
    return D<T>{a.v * b.v, a.v * b.d + a.d * b.v};
}
template <class T>
__device__ __forceinline__ D<T> operator/(D<T> a, D<T> b)
{
    const T q = a.v / b.v;
    return D<T>{q, (a.d - q * b.d) / b.v};
}
template <class T>
__device__ __forceinline__ D<T> dsqrt(D<T> a)
{
    const T s = sqrt(a.v);
    return D<T>{s, a.d / (T(2) * s)};
}
template <class T>
__device__ __forceinline__ T dsqrt(T a)
{
    return sqrt(a);
}
template <class T>
__device__ __forceinline__ T inverse(T a)
{
    return T(1) / a;
}
template <class T>
__device__ __forceinline__ D<T> inverse(D<T> a)
{
    const T q = T(1) / a.v;
    return D<T>{q, (T(0) - q * a.d) / a.v};
}
// a x + a y, rounded as written in every kernel that evaluates it
__device__ __forceinline__ float sum_of_products(float a, float x, float y) { return fmaf(a, x, __fmul_rn(a, y)); }
__device__ __forceinline__ double sum_of_products(double a, double x, double y) { return fma(a, x, __dmul_rn(a, y)); }
template <class T>
__device__ __forceinline__ D<T> sum_of_products(D<T> a, D<T> x, D<T> y)
{
    return a * x + a * y;
}
template <class T>
__device__ __forceinline__ T val(T a)
{
    return a;
}
template <class T>
__device__ __forceinline__ T val(D<T> a)
{
    return a.v;
}
template <class T>
__device__ __forceinline__ void shift(T& a, T s)
{
    a -= s;
}
template <class T>
__device__ __forceinline__ void shift(D<T>& a, T s)
{
    a.v -= s;
}

template <class T>
struct Vec4;
template <>
struct Vec4<float> {
    using type = float4;
    using half = float2;
};
template <>
struct Vec4<double> {
    using type = double4;
    using half = double2;
};

template <class T>
struct AdjParams {
    uint32_t nb, L, R, N;
    int32_t dim;
    T box[3], half[3], origin[3];
    T two_s6, lj_unit, rc2, rl2;
    int32_t exclude;
    T r0, gamma, sigma, dt;
    int32_t langevin_on;
    T eps, kbend, kbond, fact;
    unsigned long long seed;
    uint32_t lg[3], lcells, cap, ncap;
    T linv[3];
    uint32_t fpb, L_m, L_k;  // filaments per block, multiply-shift divisor by L
};

template <class T, int N>
__device__ __forceinline__ Vec<T, N> ld(const typename Vec4<T>::type* a, uint32_t i)
{
    Vec<T, N> r;
    if constexpr (N == 2) {  // half the bytes of the entry
        const auto q = *reinterpret_cast<const typename Vec4<T>::half*>(a + i);
        r.c[0] = q.x;
        r.c[1] = q.y;
    } else {
        const typename Vec4<T>::type q = a[i];
        r.c[0] = q.x;
        r.c[1] = q.y;
        r.c[2] = q.z;
    }
    return r;
}
template <class T, int N>
__device__ __forceinline__ void st(typename Vec4<T>::type* a, uint32_t i, Vec<T, N> x)
{
    typename Vec4<T>::type q;
    q.x = x.c[0];
    q.y = x.c[1];
    if constexpr (N == 3) q.z = x.c[2];
    else q.z = T(0);
    q.w = T(0);
    a[i] = q;
}

// Minimum image on the value (the shift is piecewise constant: no tangent).
template <class T, int N, class S>
__device__ __forceinline__ void min_img(const AdjParams<T>& P, Vec<S, N>& d)
{
    NW_EACH
    {
        const T v = val(d.c[q]);
        if (v > P.half[q]) shift(d.c[q], P.box[q]);
        else if (v < -P.half[q]) shift(d.c[q], -P.box[q]);
    }
}

// Bending triple with unit stiffness in scalar type S (T or D<T>):
// A = 1/(d_ij d_jk), F_i = -A (b - a (a.b)/|a|^2), F_k = -A (b (a.b)/|b|^2 - a),
// F_j = -F_i - F_k with a = r_j - r_i, b = r_k - r_j.
template <class S, int N>
struct Tri {
    Vec<S, N> fi, fj, fk;
};
template <class T, class S, int N>
__device__ __forceinline__ Tri<S, N> bend_unit(const AdjParams<T>& P, Vec<S, N> ri, Vec<S, N> rj, Vec<S, N> rk)
{
    Vec<S, N> a = rj - ri, b = rk - rj;
    min_img(P, a);
    min_img(P, b);
    const S qa = dot(a, a), qb = dot(b, b), dd = dot(a, b);
    const S A = inverse(dsqrt(qa * qb));
    const S sa = dd / qa, sb = dd / qb;
    Tri<S, N> t;
    NW_EACH
    {
        const S x = b.c[q] - a.c[q] * sa, y = b.c[q] * sb - a.c[q];
        t.fi.c[q] = -(A * x);
        t.fk.c[q] = -(A * y);
        t.fj.c[q] = sum_of_products(A, x, y);
    }
    return t;
}

template <class T, int N>
__device__ __forceinline__ Vec<T, N> noise(const AdjParams<T>& P, uint32_t rep, uint32_t li, unsigned long long step)
{
    const unsigned long long key = P.seed + rep;
    const uint4 x = philox4x32_10(make_uint4(li, (uint32_t)step, (uint32_t)(step >> 32), kRngLangevin), (uint32_t)key,
                                  (uint32_t)(key >> 32));
    T s, c;
    const T r0 = sqrt(T(-2) * log(T(u01(x.x))));
    sincospi(T(2) * T(u01(x.y)), &s, &c);
    const T z0 = r0 * c, z1 = r0 * s;
    Vec<T, N> g;
    g.c[0] = P.sigma * z0;
    g.c[1] = P.sigma * z1;
    if constexpr (N == 3) {
        T z2 = T(0);
        if (P.dim >= 3) {
            const T r1 = sqrt(T(-2) * log(T(u01(x.z))));
            T s1, c1;
            sincospi(T(2) * T(u01(x.w)), &s1, &c1);
            z2 = r1 * c1;
        }
        g.c[2] = P.sigma * z2;
    }
    return g;
}

// ---- list build -------------------------------------------------------------------

template <class T>
__device__ __forceinline__ uint32_t lcell(const AdjParams<T>& P, Vec<T, 3> r, uint32_t rep)
{
    const T* x = r.c;
    uint32_t c[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int G = (int)P.lg[a];
        int g = G == 1 ? 0 : (int)floor((x[a] - P.origin[a]) * P.linv[a]);
        g %= G;
        if (g < 0) g += G;
        c[a] = (uint32_t)g;
    }
    return rep * P.lcells + (c[2] * P.lg[1] + c[1]) * P.lg[0] + c[0];
}

template <class T>
__global__ void __launch_bounds__(256) adj_bin_kernel(const AdjParams<T> P, const typename Vec4<T>::type* __restrict__ r,
                                                      uint32_t* __restrict__ cnt, uint32_t* __restrict__ slot,
                                                      uint32_t* __restrict__ err)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    const uint32_t h = lcell(P, ld<T, 3>(r, i), i / P.nb);
    const uint32_t k = atomicAdd(cnt + h, 1u);
    if (k < P.cap) slot[(size_t)h * P.cap + k] = i;
    else atomicOr(err, (uint32_t)NW_EFLAG_CELL_OVERFLOW);
}

// Neighbours of bead i within lj_rcut + skin (not itself, not same-filament
// pairs within lj_exclude), ascending: the order does not depend on the
// order the cells were filled in.  A row of three cells at a time: their
// counts and first members in flight together, then the members' positions.
// The list grows by insertion in a column of shared memory (capacities up to
// kListCols; in its global column beyond that) and is written out once.
// 256,000 beads at three neighbours take 37 us; it was 43 us with one cell and
// one member at a time, remainders for every neighbour cell and the insertion
// in global memory.
constexpr uint32_t kListThreads = 128, kListCols = 32;
template <class T, bool kShared>
__global__ void __launch_bounds__(kListThreads) adj_list_kernel(const AdjParams<T> P, const typename Vec4<T>::type* __restrict__ r,
                                                       const uint32_t* __restrict__ cnt,
                                                       const uint32_t* __restrict__ slot, uint32_t* __restrict__ nbr,
                                                       uint32_t* __restrict__ nnb, uint32_t* __restrict__ err)
{
    __shared__ uint32_t s_col[kShared ? kListCols * kListThreads : 1];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    uint32_t* col = kShared ? s_col + threadIdx.x : nbr + i;
    const size_t row = kShared ? kListThreads : P.N;
    const uint32_t rep = i / P.nb, li = i - rep * P.nb;
    const uint32_t fbase = i - li % P.L;
    const Vec<T, 3> ri = ld<T, 3>(r, i);
    const uint32_t own = lcell(P, ri, rep) - rep * P.lcells;
    const int G[3] = {(int)P.lg[0], (int)P.lg[1], (int)P.lg[2]};
    int c[3];
    const uint32_t cyz = own / P.lg[0];
    c[0] = (int)(own - cyz * P.lg[0]);
    c[2] = (int)(cyz / P.lg[1]);
    c[1] = (int)cyz - c[2] * G[1];
    uint32_t k = 0;
    auto visit = [&](uint32_t j, Vec<T, 3> rj) {
        if (j == i) return;
        const int d = (int)j - (int)i;
        if (d <= P.exclude && d >= -P.exclude && j - fbase < P.L) return;
        Vec<T, 3> dr = rj - ri;
        min_img(P, dr);
        if (dot(dr, dr) > P.rl2) return;
        if (k < P.ncap) {  // insertion into the ascending list
            uint32_t p = k;
            while (p > 0 && col[(p - 1) * row] > j) {
                col[p * row] = col[(p - 1) * row];
                --p;
            }
            col[p * row] = j;
        }
        ++k;
    };
    // cell c + o of an axis, wrapped; with fewer than three cells the repeats are skipped
    auto cell = [&](int a, int o, int& x) -> bool {
        if (G[a] < 3 && o != 0 && (G[a] == 1 || o == 1)) return false;
        x = c[a] + o;
        if (x < 0) x += G[a];
        else if (x >= G[a]) x -= G[a];
        return true;
    };
    for (int dz = -1; dz <= 1; ++dz) {
        int z;
        if (!cell(2, dz, z)) continue;
        for (int dy = -1; dy <= 1; ++dy) {
            int y;
            if (!cell(1, dy, y)) continue;
            const uint32_t base = rep * P.lcells + (uint32_t)((z * G[1] + y) * G[0]);
            uint32_t m[3], h[3];
            uint4 first[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                int x = 0;
                const bool ok = cell(0, q - 1, x);
                h[q] = base + (uint32_t)x;
                m[q] = ok ? cnt[h[q]] : 0u;
                first[q] = *reinterpret_cast<const uint4*>(slot + (size_t)h[q] * P.cap);
            }
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                if (m[q] > P.cap) m[q] = P.cap;
                const uint32_t j[4] = {first[q].x, first[q].y, first[q].z, first[q].w};
                Vec<T, 3> x[4];
#pragma unroll
                for (uint32_t p = 0; p < 4u; ++p)
                    if (p < m[q]) x[p] = ld<T, 3>(r, j[p]);
#pragma unroll
                for (uint32_t p = 0; p < 4u; ++p)
                    if (p < m[q]) visit(j[p], x[p]);
                for (uint32_t p = 4; p < m[q]; ++p) {
                    const uint32_t jj = slot[(size_t)h[q] * P.cap + p];
                    visit(jj, ld<T, 3>(r, jj));
                }
            }
        }
    }
    if (kShared)
        for (uint32_t p = 0; p < k && p < P.ncap; ++p) nbr[(size_t)p * P.N + i] = col[p * row];
    nnb[i] = k < P.ncap ? k : P.ncap;
    if (k > P.ncap) atomicOr(err, (uint32_t)NW_EFLAG_NEIGHBOR_OVERFLOW);
}

// ---- forward ---------------------------------------------------------------------

// A block owns P.fpb whole filaments, one thread per bead, so what a bead
// shares with its chain neighbours goes through shared memory: each bending
// triple is evaluated once, by the thread of its first bead, and each bond
// once, by the thread before it (the other end takes the same numbers, the
// separation negated).  Threads without a bead still reach every barrier.
struct Place {
    uint32_t t, i, c;  // thread, bead, place along the filament
    bool on;
};
template <class T>
__device__ __forceinline__ Place place_of(const AdjParams<T>& P)
{
    Place p;
    p.t = threadIdx.x;
    p.c = p.t - fast_div(p.t, P.L_m, P.L_k) * P.L;
    p.i = blockIdx.x * P.fpb * P.L + p.t;
    p.on = p.t < P.fpb * P.L && p.i < P.N;
    return p;
}

// Columns of shared memory, one entry per thread.
template <class T>
struct Columns {
    T* base;
    uint32_t n;
    template <int N>
    __device__ __forceinline__ Vec<T, N> get(uint32_t k, uint32_t t) const
    {
        Vec<T, N> x;
        NW_EACH x.c[q] = base[(k * N + q) * n + t];
        return x;
    }
    template <int N>
    __device__ __forceinline__ void put(uint32_t k, uint32_t t, Vec<T, N> x) const
    {
        NW_EACH base[(k * N + q) * n + t] = x.c[q];
    }
    __device__ __forceinline__ T& at(uint32_t k, uint32_t t) const { return base[k * n + t]; }
};
template <class T>
__device__ __forceinline__ Columns<T> columns()
{
    extern __shared__ double s_raw[];
    return Columns<T>{reinterpret_cast<T*>(s_raw), blockDim.x};
}
constexpr uint32_t kForceCols = 13, kStepCols = 19;  // columns the two kernels below use, at most

template <class T>
__device__ __forceinline__ T lj_fm_unit(const AdjParams<T>& P, T q)
{
    const T iq = T(1) / q;
    const T iq4 = iq * iq * iq * iq;
    return P.lj_unit * (P.two_s6 * iq4 * iq * iq * iq - iq4);
}

// Force of the state (r, v) on every bead of the block.
template <class T, int N>
__device__ __forceinline__ Vec<T, N> adj_force(const AdjParams<T>& P, const Place& b, Vec<T, N> ri, Vec<T, N> vi,
                                           const typename Vec4<T>::type* __restrict__ r,
                                           const uint32_t* __restrict__ nbr, const uint32_t* __restrict__ nnb,
                                           unsigned long long step)
{
    // vector columns: positions, bonds, second and third force of the triples; the bonds' factor
    const Columns<T> S = columns<T>();
    constexpr uint32_t kFactor = 4 * N;
    using V = Vec<T, N>;
    if (b.on) S.put(0, b.t, ri);
    __syncthreads();
    V fi = zero<T, N>(), dn = fi;  // own triple's first force, bond to the next bead
    T cb = T(0), cd = T(0);
    if (b.on && b.c + 1 < P.L) {
        const V r1 = S.template get<N>(0, b.t + 1);
        dn = r1 - ri;
        min_img(P, dn);
        const T d = sqrt(dot(dn, dn));
        cb = P.kbond * (T(1) - P.r0 / d);
        cd = P.fact / d;
        S.put(1, b.t, dn);
        S.at(kFactor, b.t) = cb;
        if (b.c + 2 < P.L) {
            const Tri<T, N> t = bend_unit(P, ri, r1, S.template get<N>(0, b.t + 2));
            fi = t.fi;
            S.put(2, b.t, t.fj);
            S.put(3, b.t, t.fk);
        }
    }
    __syncthreads();
    V f = zero<T, N>();
    if (!b.on) return f;
    if (P.langevin_on) {
        const uint32_t rep = b.i / P.nb, li = b.i - rep * P.nb;
        f = noise<T, N>(P, rep, li, step) - P.gamma * vi;
    }
    // bending, in the engine's triple order (first bead c-2, c-1, c)
    if (b.c >= 2) f = f + P.kbend * S.template get<N>(3, b.t - 2);
    if (b.c >= 1 && b.c + 1 < P.L) f = f + P.kbend * S.template get<N>(2, b.t - 1);
    if (b.c + 2 < P.L) f = f + P.kbend * fi;
    // bonds and drive
    if (b.c >= 1) f = f + S.at(kFactor, b.t - 1) * (-S.template get<N>(1, b.t - 1));
    if (b.c + 1 < P.L) {
        f = f + cb * dn;
        f = f + cd * dn;
    }
    // LJ over the frozen list, four neighbours fetched together
    const uint32_t k = nnb[b.i];
    const uint32_t* __restrict__ col = nbr + b.i;
    for (uint32_t m = 0; m < k; m += 4u) {
        uint32_t j[4];
#pragma unroll
        for (uint32_t q = 0; q < 4u; ++q) j[q] = m + q < k ? col[(size_t)(m + q) * P.N] : b.i;
        V x[4];
#pragma unroll
        for (uint32_t q = 0; q < 4u; ++q) x[q] = ld<T, N>(r, j[q]);
#pragma unroll
        for (uint32_t q = 0; q < 4u; ++q) {
            if (m + q >= k) break;
            V dr = x[q] - ri;
            min_img(P, dr);
            const T d2 = dot(dr, dr);
            if (d2 > P.rc2) continue;
            f = f - (P.eps * lj_fm_unit(P, d2)) * dr;
        }
    }
    return f;
}

// The state of a rollout between updates: positions, velocities, the force of
// the last update and of the one before.
template <class T>
struct AdjState {
    typename Vec4<T>::type *r, *v, *F, *Fo;
};

template <class T, int N>
__device__ __forceinline__ void adj_integrate(const AdjParams<T>& P, uint32_t i, Vec<T, N> ri, Vec<T, N> vi,
                                              Vec<T, N> f, Vec<T, N> fo, const AdjState<T>& out)
{
    const Vec<T, N> vn = vi + (T(0.5) * P.dt) * (f + fo);
    Vec<T, N> rn = ri + P.dt * vn + (T(0.5) * P.dt * P.dt) * f;
    NW_EACH
    {
        if (rn.c[q] < P.origin[q]) rn.c[q] += P.box[q];
        else if (rn.c[q] > P.origin[q] + P.box[q]) rn.c[q] -= P.box[q];
    }
    st(out.v, i, vn);
    st(out.r, i, rn);
    st(out.F, i, f);
}

// The first update of a segment, as far as its force: from the checkpoint.
template <class T, int N>
__global__ void __launch_bounds__(256) adj_first_kernel(const AdjParams<T> P, const AdjState<T> in,
                                                        const AdjState<T> out)
{
    pdl_enter();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    adj_integrate(P, i, ld<T, N>(in.r, i), ld<T, N>(in.v, i), ld<T, N>(in.F, i), ld<T, N>(in.Fo, i), out);
}

// kLast false: the force of the update whose positions are in.r and the
// integration of the next one (in.v and in.F, the force of the update before,
// are replaced; positions go to another buffer, since other blocks still read
// these).  kLast: only the force, and the whole state to the checkpoint `out`.
// One launch per update: for 64 x 4,000 beads it reads and writes 100 bytes a
// bead of L2-resident state; the separate integration (6.2 us) and the force
// kernel that evaluated every triple three times and every bond twice
// (15.7 us) took 22 us an update, this one 14.4 us with two components.
template <class T, int N, bool kLast, int MAXT>
__global__ void __launch_bounds__(MAXT) adj_update_kernel(const AdjParams<T> P, const AdjState<T> in,
                                                          const AdjState<T> out, const uint32_t* __restrict__ nbr,
                                                          const uint32_t* __restrict__ nnb, unsigned long long step)
{
    pdl_enter();
    const Place b = place_of(P);
    Vec<T, N> ri = zero<T, N>(), vi = ri;
    if (b.on) {
        ri = ld<T, N>(in.r, b.i);
        vi = ld<T, N>(in.v, b.i);
    }
    const Vec<T, N> f = adj_force(P, b, ri, vi, in.r, nbr, nnb, step);
    if (!b.on) return;
    const Vec<T, N> fo = ld<T, N>(in.F, b.i);
    if (kLast) {
        st(out.r, b.i, ri);
        st(out.v, b.i, vi);
        st(out.F, b.i, f);
        st(out.Fo, b.i, fo);
    } else {
        adj_integrate(P, b.i, ri, vi, f, fo, out);
    }
}

// ---- adjoint ---------------------------------------------------------------------

// Sum of a thread's gradient terms: a double, or for single-precision terms
// the unevaluated sum hi + lo of two floats with every rounding error of hi
// kept in lo (Knuth's two-sum, TAOCP vol. 2, 4.2.2).  The double-precision
// unit does two operations a clock and SM: converting and adding the terms in
// double, and reducing them along the warps, was 10 us of the step kernel's
// 29 us for 64 x 4,000 beads (now 18.8).
template <class T>
struct Sum {
    double v = 0.0;
    __device__ __forceinline__ void add(double x) { v += x; }
    __device__ __forceinline__ void add(const Sum& o) { v += o.v; }
    __device__ __forceinline__ double get() const { return v; }
};
template <>
struct Sum<float> {
    float hi = 0.f, lo = 0.f;
    __device__ __forceinline__ void add(float x)
    {
        const float s = __fadd_rn(hi, x), t = __fsub_rn(s, hi);
        lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, t)), __fsub_rn(x, t)));
        hi = s;
    }
    __device__ __forceinline__ void add(const Sum& o)
    {
        add(o.hi);
        lo = __fadd_rn(lo, o.lo);
    }
    __device__ __forceinline__ double get() const { return (double)hi + (double)lo; }
};

// One adjoint update.  G: the type whose Sum gathers the gradient terms, double
// where single-precision terms overflow its pair (backward_t).  Triples and bonds are evaluated once each, like the
// forces above; the thread of a triple or bond also takes its share of the
// parameter gradients for all its beads.  For 64 x 4,000 beads the kernel that
// took every triple's dual numbers three times and every bond's terms twice
// ran 35.6 us an update, this one 18.8 us.
template <class T, int N, int MAXT, class G = T>
__global__ void __launch_bounds__(MAXT) adj_step_kernel(const AdjParams<T> P, const typename Vec4<T>::type* __restrict__ r,
                                                        const uint32_t* __restrict__ nbr,
                                                        const uint32_t* __restrict__ nnb,
                                                        typename Vec4<T>::type* __restrict__ lr,
                                                        typename Vec4<T>::type* __restrict__ lv,
                                                        const typename Vec4<T>::type* __restrict__ lF_in,
                                                        typename Vec4<T>::type* __restrict__ lF_out,
                                                        typename Vec4<T>::type* __restrict__ lFo,
                                                        double* __restrict__ gacc)
{
    pdl_enter();
    __shared__ Sum<G> s_g[4][MAXT + MAXT / 32];
    // vector columns: positions, lF, bond and drive terms, second and third
    // derivative of the triples; the drives' factor
    const Columns<T> S = columns<T>();
    constexpr uint32_t kFactor = 6 * N;
    using V = Vec<T, N>;
    const Place b = place_of(P);
    Sum<G> g[4];  // eps, k_bend, k_bond, F_act
    V ri = zero<T, N>(), lfi = ri;
    if (b.on) {
        ri = ld<T, N>(r, b.i);
        lfi = ld<T, N>(lF_in, b.i);
        S.put(0, b.t, ri);
        S.put(1, b.t, lfi);
    }
    __syncthreads();
    V ti = zero<T, N>(), xb = ti, yd = ti;  // triple's first derivative, bond term, drive term
    T cd = T(0);
    if (b.on && b.c + 1 < P.L) {
        const V r1 = S.template get<N>(0, b.t + 1), l1 = S.template get<N>(1, b.t + 1);
        // bond (central: phi(q) dr with phi = k (1 - r0 / sqrt q))
        V dr = r1 - ri;
        min_img(P, dr);
        const T q2 = dot(dr, dr), d = sqrt(q2);
        const V del = l1 - lfi;
        const T phi = T(1) - P.r0 / d, dphi = T(0.5) * P.r0 / (q2 * d);
        g[2].add(phi * dot(lfi, dr));
        g[2].add(phi * dot(l1, -dr));
        xb = phi * del + (dphi * T(2) * dot(dr, del)) * dr;
        // own drive F_i = F_act dr / d: d/dr_i = -A, A l = (l - dr (dr . l) / d^2) / d;
        // the next bead takes +A l
        g[3].add(dot(lfi, dr) / d);
        cd = P.fact / d;
        yd = lfi - (dot(dr, lfi) / q2) * dr;
        S.put(2, b.t, xb);
        S.put(3, b.t, yd);
        S.at(kFactor, b.t) = cd;
        if (b.c + 2 < P.L) {
            // bending: directional derivative of the unit triple forces along lF
            const V r2 = S.template get<N>(0, b.t + 2), l2 = S.template get<N>(1, b.t + 2);
            Vec<D<T>, N> a0, a1, a2;
            NW_EACH
            {
                a0.c[q] = D<T>{ri.c[q], lfi.c[q]};
                a1.c[q] = D<T>{r1.c[q], l1.c[q]};
                a2.c[q] = D<T>{r2.c[q], l2.c[q]};
            }
            const Tri<D<T>, N> t = bend_unit(P, a0, a1, a2);
            V fi, fj, fk, tj, tk;
            NW_EACH
            {
                fi.c[q] = t.fi.c[q].v;
                fj.c[q] = t.fj.c[q].v;
                fk.c[q] = t.fk.c[q].v;
                ti.c[q] = t.fi.c[q].d;
                tj.c[q] = t.fj.c[q].d;
                tk.c[q] = t.fk.c[q].d;
            }
            g[1].add(dot(lfi, fi));
            g[1].add(dot(l1, fj));
            g[1].add(dot(l2, fk));
            S.put(4, b.t, tj);
            S.put(5, b.t, tk);
        }
    }
    __syncthreads();
    if (b.on) {
        V jt = zero<T, N>();
        if (b.c >= 2) jt = jt + P.kbend * S.template get<N>(5, b.t - 2);
        if (b.c >= 1 && b.c + 1 < P.L) jt = jt + P.kbend * S.template get<N>(4, b.t - 1);
        if (b.c + 2 < P.L) jt = jt + P.kbend * ti;
        if (b.c >= 1) jt = jt + P.kbond * (-S.template get<N>(2, b.t - 1));
        if (b.c + 1 < P.L) {
            jt = jt + P.kbond * xb;
            jt = jt - cd * yd;
        }
        if (b.c >= 1) jt = jt + S.at(kFactor, b.t - 1) * S.template get<N>(3, b.t - 1);
        // LJ over the frozen list: F_i = -eps fm(q) dr, fm' from q
        const uint32_t k = nnb[b.i];
        const uint32_t* __restrict__ col = nbr + b.i;
        for (uint32_t m = 0; m < k; m += 4u) {
            uint32_t j[4];
#pragma unroll
            for (uint32_t q = 0; q < 4u; ++q) j[q] = m + q < k ? col[(size_t)(m + q) * P.N] : b.i;
            V x[4];
#pragma unroll
            for (uint32_t q = 0; q < 4u; ++q) x[q] = ld<T, N>(r, j[q]);
#pragma unroll
            for (uint32_t q = 0; q < 4u; ++q) {
                if (m + q >= k) break;
                V dr = x[q] - ri;
                min_img(P, dr);
                const T d2 = dot(dr, dr);
                if (d2 > P.rc2) continue;
                const T iq = T(1) / d2;
                const T iq4 = iq * iq * iq * iq;
                const T fm = P.lj_unit * (P.two_s6 * iq4 * iq * iq * iq - iq4);
                const T dfm = P.lj_unit * (T(-7) * P.two_s6 * iq4 * iq4 + T(4) * iq4 * iq);
                const V del = ld<T, N>(lF_in, j[q]) - lfi;
                g[0].add(-fm * dot(lfi, dr));
                jt = jt - P.eps * ((dfm * T(2) * dot(dr, del)) * dr + fm * del);
            }
        }
        const V lrt = ld<T, N>(lr, b.i) + jt;
        V lvt = ld<T, N>(lv, b.i);
        if (P.langevin_on) lvt = lvt - P.gamma * lfi;
        lvt = lvt + P.dt * lrt;
        const V lfn = ld<T, N>(lFo, b.i) + (T(0.5) * P.dt * P.dt) * lrt + (T(0.5) * P.dt) * lvt;
        st(lF_out, b.i, lfn);
        st(lFo, b.i, (T(0.5) * P.dt) * lvt);
        st(lr, b.i, lrt);
        st(lv, b.i, lvt);
    }
    // per-block parameter gradient, one writer per block: a fixed summation
    // order (each lane of the first warp one eighth of the threads' sums of a
    // parameter, then the eighths)
    const uint32_t pad = b.t + (b.t >> 5);  // the lanes' runs start in different banks
#pragma unroll
    for (int q = 0; q < 4; ++q) s_g[q][pad] = g[q];
    __syncthreads();
    if (threadIdx.x < 32) {
        const uint32_t q = threadIdx.x & 3u, part = (blockDim.x + 7u) / 8u, t0 = (threadIdx.x >> 2) * part;
        Sum<G> x;
        for (uint32_t t = t0; t < t0 + part && t < blockDim.x; ++t) x.add(s_g[q][t + (t >> 5)]);
        double v = x.get();
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (threadIdx.x < 4) gacc[blockIdx.x * 4u + q] += v;
    }
}

// ---- conversions -------------------------------------------------------------------

// xyz of a float4 array; *off_plane is set where a z component exceeds most, or is NaN
template <class T>
__global__ void from_f4_kernel(const float4* __restrict__ a, typename Vec4<T>::type* __restrict__ b, uint32_t n,
                               uint32_t* __restrict__ off_plane, float most)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const float4 q = i < n ? a[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < n) {
        Vec<T, 3> x;
        x.c[0] = q.x;
        x.c[1] = q.y;
        x.c[2] = q.z;
        st(b, i, x);
    }
    if (__any_sync(0xffffffffu, !(fabsf(q.z) <= most)) && (threadIdx.x & 31u) == 0u) *off_plane = 1u;
}

template <class T>
__global__ void to_f4_kernel(const typename Vec4<T>::type* __restrict__ a, float4* __restrict__ b,
                             const float4* __restrict__ wsrc, uint32_t n)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const Vec<T, 3> x = ld<T, 3>(a, i);
        b[i] = make_float4((float)x.c[0], (float)x.c[1], (float)x.c[2], wsrc ? wsrc[i].w : 0.f);
    }
}

// xyz of the state in double (x, y, z, 0) quadruples, at either precision
template <class T>
__global__ void to_d4_kernel(const typename Vec4<T>::type* __restrict__ a, double* __restrict__ b, uint32_t n)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const Vec<T, 3> x = ld<T, 3>(a, i);
        b[4 * (size_t)i] = (double)x.c[0];
        b[4 * (size_t)i + 1] = (double)x.c[1];
        b[4 * (size_t)i + 2] = (double)x.c[2];
        b[4 * (size_t)i + 3] = 0.0;
    }
}

uint32_t nblocks(uint32_t n) { return (n + 255u) / 256u; }

}  // namespace

struct nw_adjoint {
    NwConfig cfg;
    int R = 0, horizon = 0, seg = 0, prec = 32;
    uint32_t nb = 0, N = 0, nseg = 0;
    cudaStream_t own = nullptr, stream = nullptr;
    size_t elem = 16;  // bytes of one stored vector
    void *r[2] = {nullptr, nullptr}, *v = nullptr, *F = nullptr;  // state between updates
    void *r_end = nullptr, *v_end = nullptr;                      // final state of the last forward
    uint32_t fpb = 1, threads = 256, blocks = 1;                  // filaments, threads per block and blocks of the update
    void *r0 = nullptr, *v0 = nullptr;
    float4* w_pos = nullptr;  // w components of the initial positions (radius) and velocities (mass)
    float4* w_vel = nullptr;
    void* ck = nullptr;    // checkpoints: [nseg][4][N]
    void* traj = nullptr;  // positions of one segment: [seg][N]
    void *lr = nullptr, *lv = nullptr, *lF[2] = {nullptr, nullptr}, *lFo = nullptr;
    uint32_t *cnt = nullptr, *slot = nullptr, *nbr = nullptr, *nnb = nullptr, *err = nullptr;
    double* gacc = nullptr;
    std::vector<void*> allocs;
    double theta[4] = {0, 0, 0, 0};
    bool have_forward = false;
    bool planar = false;  // two-dimensional, every z of the initial state is zero and stays so
    float fwd_ms = 0.f, bwd_ms = 0.f;
    uint32_t lg[3] = {1, 1, 1}, lcells = 1, cap = 16, ncap = 32;
};

namespace {

template <class T>
AdjParams<T> adj_params(const nw_adjoint* a, const double th[4])
{
    const NwConfig& c = a->cfg;
    AdjParams<T> P;
    std::memset(&P, 0, sizeof(P));
    P.nb = a->nb;
    P.L = c.filament_size;
    P.R = (uint32_t)a->R;
    P.N = a->N;
    P.dim = c.dim;
    for (int k = 0; k < 3; ++k) {
        P.box[k] = (T)c.box[k];
        P.half[k] = (T)c.box[k] / T(2);
        P.origin[k] = (T)c.origin[k];
        P.lg[k] = a->lg[k];
        P.linv[k] = (T)a->lg[k] / (T)c.box[k];
    }
    const double s6 = std::pow((double)c.lj_sigma, 6.0);
    P.two_s6 = (T)(2.0 * s6);
    P.lj_unit = (T)(24.0 * s6);
    P.rc2 = (T)((double)c.lj_rcut * (double)c.lj_rcut);
    const double skin = c.neighbor_skin > 0.0f ? c.neighbor_skin : 0.3 * c.lj_sigma;
    P.rl2 = (T)(((double)c.lj_rcut + skin) * ((double)c.lj_rcut + skin));
    P.exclude = c.lj_exclude;
    P.r0 = (T)c.bond_r0;
    P.gamma = (T)c.gamma;
    double s2 = 2.0 * (double)c.gamma * (double)c.kT;
    if (c.noise_dt_scaling) s2 /= (double)c.dt;
    P.sigma = (T)std::sqrt(s2);
    P.dt = (T)c.dt;
    P.langevin_on = 1;
    P.eps = (T)th[0];
    P.kbend = (T)th[1];
    P.kbond = (T)th[2];
    P.fact = (T)th[3];
    P.seed = c.seed;
    P.lcells = a->lcells;
    P.cap = a->cap;
    P.ncap = a->ncap;
    P.fpb = a->fpb;
    fast_div_params(P.L, P.L_m, P.L_k);
    return P;
}

// Blocks of whole filaments, up to 256 beads (a longer filament takes one of
// up to 1,024): 256 threads where that fills the chip four times over, else
// fewer, down to 64, so that a small rollout spreads over the SMs.  Double
// precision runs at two operations a clock and SM there: 6,765 beads take
// 27 blocks of 256 threads, on as many of the 152 SMs, or 123 of 64.
void update_shape(nw_adjoint* a)
{
    const uint32_t L = a->cfg.filament_size;
    uint32_t want = 256;
    while (want > 64u && (uint64_t)a->N < (uint64_t)want * 4u * 152u) want >>= 1;
    a->fpb = L >= want ? 1u : want / L;
    a->threads = (a->fpb * L + 31u) & ~31u;
    const uint64_t nf = (uint64_t)a->N / L;
    a->blocks = (uint32_t)((nf + a->fpb - 1) / a->fpb);
}

void* at(void* base, size_t index, const nw_adjoint* a)
{
    return static_cast<char*>(base) + index * (size_t)a->N * a->elem;
}

template <class T>
cudaError_t build_lists(nw_adjoint* a, const AdjParams<T>& P, const void* r)
{
    using V = typename Vec4<T>::type;
    cudaError_t e = cudaMemsetAsync(a->cnt, 0, (size_t)a->R * a->lcells * 4, a->stream);
    if (e != cudaSuccess) return e;
    adj_bin_kernel<T><<<nblocks(a->N), 256, 0, a->stream>>>(P, static_cast<const V*>(r), a->cnt, a->slot, a->err);
    const uint32_t nblk = (a->N + kListThreads - 1) / kListThreads;
    auto* list = a->ncap <= kListCols ? adj_list_kernel<T, true> : adj_list_kernel<T, false>;
    list<<<nblk, kListThreads, 0, a->stream>>>(P, static_cast<const V*>(r), a->cnt, a->slot, a->nbr, a->nnb, a->err);
    return cudaGetLastError();
}

template <class T>
AdjState<T> ck_state(nw_adjoint* a, uint32_t s)
{
    using V = typename Vec4<T>::type;
    return AdjState<T>{static_cast<V*>(at(a->ck, (size_t)s * 4, a)), static_cast<V*>(at(a->ck, (size_t)s * 4 + 1, a)),
                       static_cast<V*>(at(a->ck, (size_t)s * 4 + 2, a)),
                       static_cast<V*>(at(a->ck, (size_t)s * 4 + 3, a))};
}

// Updates of segment s (1-based update m uses noise counter m - 1) from its
// checkpoint, on lists built from the checkpoint's positions.  With keep the
// positions after update m are left in traj[m - m0] and the last update stops
// at its positions; without, the state after the segment goes to the next
// checkpoint, or after the last segment to the final state.
template <class T, int N>
cudaError_t run_segment(nw_adjoint* a, const AdjParams<T>& P, uint32_t s, bool keep)
{
    using V = typename Vec4<T>::type;
    const int m0 = (int)s * a->seg + 1, m1 = std::min(a->horizon, (int)(s + 1) * a->seg) + 1;
    const AdjState<T> ck = ck_state<T>(a, s);
    cudaError_t e = build_lists<T>(a, P, ck.r);
    if (e != cudaSuccess) return e;
    const bool end = s + 1 == a->nseg;
    auto pos = [&](int m) -> V* {  // positions after update m
        return static_cast<V*>(keep ? at(a->traj, (size_t)(m - m0), a) : a->r[m & 1]);
    };
    auto work = [&](int m) {
        AdjState<T> w{pos(m), static_cast<V*>(a->v), static_cast<V*>(a->F), nullptr};
        if (!keep && end && m == m1 - 1) w.r = static_cast<V*>(a->r_end), w.v = static_cast<V*>(a->v_end);
        return w;
    };
    launch_pdl(adj_first_kernel<T, N>, nblocks(a->N), 256, 0, a->stream, P, ck, work(m0));
    const size_t smem = (size_t)a->threads * kForceCols * sizeof(T);
    for (int m = m0; m < m1 - 1; ++m) {
        auto* up = a->threads > 256 ? adj_update_kernel<T, N, false, 1024> : adj_update_kernel<T, N, false, 256>;
        launch_pdl(up, a->blocks, a->threads, smem, a->stream, P, work(m), work(m + 1), a->nbr, a->nnb,
                   (unsigned long long)(m - 1));
    }
    if (!keep && !end) {
        auto* up = a->threads > 256 ? adj_update_kernel<T, N, true, 1024> : adj_update_kernel<T, N, true, 256>;
        launch_pdl(up, a->blocks, a->threads, smem, a->stream, P, work(m1 - 1), ck_state<T>(a, s + 1), a->nbr, a->nnb,
                   (unsigned long long)(m1 - 2));
    }
    return cudaGetLastError();
}

// Shared memory beyond the default 48 KB, for filaments of more than 256 beads.
template <class T, int N>
cudaError_t allow_long_filaments()
{
    const int force = 1024 * kForceCols * (int)sizeof(T), step = 1024 * kStepCols * (int)sizeof(T);
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(adj_update_kernel<T, N, false, 1024>, attr, force);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(adj_update_kernel<T, N, true, 1024>, attr, force);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(adj_step_kernel<T, N, 1024>, attr, step);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(adj_step_kernel<T, N, 1024, double>, attr, step);
    return e;
}

nw_status st_of(cudaError_t e)
{
    if (e == cudaSuccess) return NW_OK;
    cudaGetLastError();
    return e == cudaErrorMemoryAllocation ? NW_ERR_NOMEM : NW_ERR_CUDA;
}

nw_status check_err(nw_adjoint* a)
{
    uint32_t f = 0;
    cudaError_t e = cudaMemcpyAsync(&f, a->err, 4, cudaMemcpyDeviceToHost, a->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(a->stream);
    if (e != cudaSuccess) return st_of(e);
    if (f) {
        cudaMemsetAsync(a->err, 0, 4, a->stream);
        cudaStreamSynchronize(a->stream);
        return NW_ERR_CELL_OVERFLOW;
    }
    return NW_OK;
}

template <class T>
nw_status forward_t(nw_adjoint* a, const double th[4], float* pos_out, float* vel_out)
{
    using V = typename Vec4<T>::type;
    const AdjParams<T> P = adj_params<T>(a, th);
    const size_t bytes = (size_t)a->N * a->elem;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, a->stream);
    const AdjState<T> ck = ck_state<T>(a, 0);
    cudaError_t e = cudaMemcpyAsync(ck.r, a->r0, bytes, cudaMemcpyDeviceToDevice, a->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(ck.v, a->v0, bytes, cudaMemcpyDeviceToDevice, a->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(ck.F, 0, bytes, a->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(ck.Fo, 0, bytes, a->stream);
    for (uint32_t s = 0; s < a->nseg && e == cudaSuccess; ++s) e = a->planar ? run_segment<T, 2>(a, P, s, false) : run_segment<T, 3>(a, P, s, false);
    cudaEventRecord(e1, a->stream);
    if (e == cudaSuccess && pos_out)
        to_f4_kernel<T><<<nblocks(a->N), 256, 0, a->stream>>>(static_cast<const V*>(a->r_end), (float4*)pos_out, a->w_pos,
                                                              a->N);
    if (e == cudaSuccess && vel_out)
        to_f4_kernel<T><<<nblocks(a->N), 256, 0, a->stream>>>(static_cast<const V*>(a->v_end), (float4*)vel_out, a->w_vel,
                                                              a->N);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(a->stream);
    if (e == cudaSuccess) cudaEventElapsedTime(&a->fwd_ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (e != cudaSuccess) return st_of(e);
    const nw_status st = check_err(a);
    if (st != NW_OK) return st;
    std::memcpy(a->theta, th, sizeof(a->theta));
    a->have_forward = true;
    return NW_OK;
}

template <class T, int N, class G>
auto step_kernel(const nw_adjoint* a)
{
    return a->threads > 256 ? adj_step_kernel<T, N, 1024, G> : adj_step_kernel<T, N, 256, G>;
}

template <class T, class G = T>
nw_status backward_t(nw_adjoint* a, const float* gpos, const float* gvel, double out[4], bool planar)
{
    using V = typename Vec4<T>::type;
    const AdjParams<T> P = adj_params<T>(a, a->theta);
    const size_t bytes = (size_t)a->N * a->elem;
    const uint32_t nbk = a->blocks;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, a->stream);
    uint32_t* off = a->err + 1;
    cudaError_t e = cudaMemsetAsync(off, 0, 4, a->stream);
    for (int k = 0; k < 2; ++k)
        from_f4_kernel<T><<<nblocks(a->N), 256, 0, a->stream>>>((const float4*)(k ? gvel : gpos),
                                                                static_cast<V*>(k ? a->lv : a->lr), a->N, off, FLT_MAX);
    if (e == cudaSuccess) e = cudaMemsetAsync(a->lF[0], 0, bytes, a->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(a->lFo, 0, bytes, a->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(a->gacc, 0, (size_t)nbk * 4 * sizeof(double), a->stream);
    uint32_t cur = 0;
    for (int s = (int)a->nseg - 1; s >= 0 && e == cudaSuccess; --s) {
        e = planar ? run_segment<T, 2>(a, P, (uint32_t)s, true) : run_segment<T, 3>(a, P, (uint32_t)s, true);
        const int m0 = s * a->seg + 1, m1 = std::min(a->horizon, (s + 1) * a->seg) + 1;
        for (int m = m1 - 1; m >= m0 && e == cudaSuccess; --m) {
            auto* step = planar ? step_kernel<T, 2, G>(a) : step_kernel<T, 3, G>(a);
            launch_pdl(step, nbk, a->threads, (size_t)a->threads * kStepCols * sizeof(T), a->stream, P,
                       static_cast<const V*>(at(a->traj, (size_t)(m - m0), a)), a->nbr, a->nnb, static_cast<V*>(a->lr),
                       static_cast<V*>(a->lv), static_cast<const V*>(a->lF[cur]), static_cast<V*>(a->lF[cur ^ 1u]),
                       static_cast<V*>(a->lFo), a->gacc);
            cur ^= 1u;
            e = cudaGetLastError();
        }
    }
    cudaEventRecord(e1, a->stream);
    std::vector<double> g((size_t)nbk * 4);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(g.data(), a->gacc, g.size() * sizeof(double), cudaMemcpyDeviceToHost, a->stream);
    uint32_t undefined = 0;  // z gradients that are infinite or NaN reach the parameters: times 0, as NaN
    if (e == cudaSuccess && planar) e = cudaMemcpyAsync(&undefined, off, 4, cudaMemcpyDeviceToHost, a->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(a->stream);
    if (e == cudaSuccess) cudaEventElapsedTime(&a->bwd_ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (e != cudaSuccess) return st_of(e);
    const nw_status st = check_err(a);
    if (st != NW_OK) return st;
    if (undefined) return backward_t<T, G>(a, gpos, gvel, out, false);
    for (int q = 0; q < 4; ++q) {
        double x = 0.0;
        for (uint32_t b = 0; b < nbk; ++b) x += g[(size_t)b * 4 + q];
        out[q] = x;
    }
    // a pair of floats makes NaN of an infinite term or sum: again in doubles
    if constexpr (std::is_same_v<G, float>)
        for (int q = 0; q < 4; ++q)
            if (!std::isfinite(out[q])) return backward_t<T, double>(a, gpos, gvel, out, planar);
    return NW_OK;
}

}  // namespace

extern "C" {

nw_status nw_adj_create(const NwConfig* cfg, int n_replicas, int horizon, int segment, int precision,
                        nw_adjoint** out)
{
    if (!out) return NW_ERR_INVALID;
    *out = nullptr;
    if (!cfg || n_replicas <= 0 || horizon <= 0 || segment <= 0 || (precision != 32 && precision != 64))
        return NW_ERR_INVALID;
    nw_status st = nw_config_validate(cfg);
    if (st != NW_OK) return st;
    if (cfg->model != NW_MODEL_WCA_WORMS || cfg->srd_enabled || cfg->reverse_probability > 0.0f)
        return NW_ERR_UNSUPPORTED;
    for (int k = 0; k < 3; ++k)
        if (cfg->boundary[k] != NW_PERIODIC) return NW_ERR_UNSUPPORTED;
    const uint64_t nb = (uint64_t)cfg->num_filaments * cfg->filament_size;
    if (nb == 0 || nb * (uint64_t)n_replicas >= (1ull << 31)) return NW_ERR_INVALID;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return NW_ERR_NO_DEVICE;
    }
    nw_adjoint* a = new nw_adjoint();
    a->cfg = *cfg;
    a->R = n_replicas;
    a->horizon = horizon;
    a->seg = segment;
    a->prec = precision;
    a->nb = (uint32_t)nb;
    a->N = (uint32_t)(nb * (uint64_t)n_replicas);
    a->nseg = (uint32_t)((horizon + segment - 1) / segment);
    a->elem = precision == 64 ? 32 : 16;
    const double skin = cfg->neighbor_skin > 0.0f ? cfg->neighbor_skin : 0.3 * cfg->lj_sigma;
    const double rl = (double)cfg->lj_rcut + skin;
    a->lcells = 1;
    for (int k = 0; k < 3; ++k) {
        uint32_t G = 1;
        if (cfg->grid[k] > 1) {
            const double g = std::floor((double)cfg->box[k] / (rl * 1.0001));
            G = g >= 1.0 ? (uint32_t)g : 1u;
        }
        a->lg[k] = G;
        a->lcells *= G;
    }
    a->ncap = cfg->neighbor_capacity ? cfg->neighbor_capacity : 32u;
    a->cap = 16;
    // a blocking stream: the rollout's own work is ordered with the legacy
    // default stream, on which callers such as torch produce the upstream
    // gradients it reads (a non-blocking stream could read them unfinished)
    if (cudaStreamCreateWithFlags(&a->own, cudaStreamDefault) != cudaSuccess) {
        delete a;
        return NW_ERR_CUDA;
    }
    a->stream = a->own;
    auto A = [&](void** p, size_t bytes) {
        if (st != NW_OK) return;
        if (cudaMalloc(p, bytes ? bytes : 16) != cudaSuccess) {
            cudaGetLastError();
            st = NW_ERR_NOMEM;
            return;
        }
        a->allocs.push_back(*p);
    };
    const size_t vb = (size_t)a->N * a->elem;
    update_shape(a);
    for (int k = 0; k < 2; ++k) A(&a->r[k], vb);
    A(&a->v, vb);
    A(&a->F, vb);
    A(&a->r_end, vb);
    A(&a->v_end, vb);
    A(&a->r0, vb);
    A(&a->v0, vb);
    A((void**)&a->w_pos, (size_t)a->N * 16);
    A((void**)&a->w_vel, (size_t)a->N * 16);
    A(&a->ck, vb * 4 * a->nseg);
    A(&a->traj, vb * (size_t)segment);
    A(&a->lr, vb);
    A(&a->lv, vb);
    A(&a->lF[0], vb);
    A(&a->lF[1], vb);
    A(&a->lFo, vb);
    A((void**)&a->cnt, (size_t)a->R * a->lcells * 4);
    A((void**)&a->slot, (size_t)a->R * a->lcells * a->cap * 4);
    A((void**)&a->nbr, (size_t)a->N * a->ncap * 4);
    A((void**)&a->nnb, (size_t)a->N * 4);
    A((void**)&a->err, 16);
    A((void**)&a->gacc, (size_t)a->blocks * 4 * sizeof(double));
    if (st == NW_OK) st = st_of(cudaMemset(a->err, 0, 16));
    if (st == NW_OK && a->threads > 256)
        st = st_of(precision == 64 ? allow_long_filaments<double, 3>() : allow_long_filaments<float, 3>());
    if (st == NW_OK && a->threads > 256)
        st = st_of(precision == 64 ? allow_long_filaments<double, 2>() : allow_long_filaments<float, 2>());
    if (st != NW_OK) {
        nw_adj_destroy(a);
        return st;
    }
    *out = a;
    return NW_OK;
}

nw_status nw_adj_destroy(nw_adjoint* a)
{
    if (!a) return NW_ERR_INVALID;
    cudaStreamSynchronize(a->stream);
    for (void* p : a->allocs) cudaFree(p);
    if (a->own) cudaStreamDestroy(a->own);
    delete a;
    return NW_OK;
}

nw_status nw_adj_set_stream(nw_adjoint* a, void* stream)
{
    if (!a) return NW_ERR_INVALID;
    cudaStreamSynchronize(a->stream);
    a->stream = stream ? (cudaStream_t)stream : a->own;
    return NW_OK;
}

nw_status nw_adj_set_state(nw_adjoint* a, const float* d_pos, const float* d_vel)
{
    if (!a || !d_pos || !d_vel) return NW_ERR_INVALID;
    const uint32_t nbk = nblocks(a->N);
    uint32_t* off = a->err + 1;
    if (cudaMemsetAsync(off, 0, 4, a->stream) != cudaSuccess) return st_of(cudaGetLastError());
    if (a->prec == 64) {
        from_f4_kernel<double><<<nbk, 256, 0, a->stream>>>((const float4*)d_pos, (double4*)a->r0, a->N, off, 0.f);
        from_f4_kernel<double><<<nbk, 256, 0, a->stream>>>((const float4*)d_vel, (double4*)a->v0, a->N, off, 0.f);
    } else {
        from_f4_kernel<float><<<nbk, 256, 0, a->stream>>>((const float4*)d_pos, (float4*)a->r0, a->N, off, 0.f);
        from_f4_kernel<float><<<nbk, 256, 0, a->stream>>>((const float4*)d_vel, (float4*)a->v0, a->N, off, 0.f);
    }
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(a->w_pos, d_pos, (size_t)a->N * 16, cudaMemcpyDeviceToDevice, a->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(a->w_vel, d_vel, (size_t)a->N * 16, cudaMemcpyDeviceToDevice, a->stream);
    uint32_t out = 1;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&out, off, 4, cudaMemcpyDeviceToHost, a->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(a->stream);
    // z stays zero where the box holds it (else each update wraps it towards the box)
    const float lo = a->cfg.origin[2], hi = lo + a->cfg.box[2];
    a->planar = a->cfg.dim == 2 && out == 0u && lo <= 0.f && hi >= 0.f;
    a->have_forward = false;
    return st_of(e);
}

nw_status nw_adj_forward(nw_adjoint* a, const double theta[4], float* d_pos_out, float* d_vel_out)
{
    if (!a || !theta) return NW_ERR_INVALID;
    for (int q = 0; q < 4; ++q)
        if (!std::isfinite(theta[q])) return NW_ERR_INVALID;
    return a->prec == 64 ? forward_t<double>(a, theta, d_pos_out, d_vel_out)
                         : forward_t<float>(a, theta, d_pos_out, d_vel_out);
}

nw_status nw_adj_final_state_f64(nw_adjoint* a, double* d_pos_out, double* d_vel_out)
{
    if (!a || !a->have_forward) return NW_ERR_INVALID;
    cudaError_t e = cudaSuccess;
    if (a->prec == 64) {
        using V = typename Vec4<double>::type;
        if (d_pos_out) to_d4_kernel<double><<<nblocks(a->N), 256, 0, a->stream>>>(static_cast<const V*>(a->r_end), d_pos_out, a->N);
        if (d_vel_out) to_d4_kernel<double><<<nblocks(a->N), 256, 0, a->stream>>>(static_cast<const V*>(a->v_end), d_vel_out, a->N);
    } else {
        using V = typename Vec4<float>::type;
        if (d_pos_out) to_d4_kernel<float><<<nblocks(a->N), 256, 0, a->stream>>>(static_cast<const V*>(a->r_end), d_pos_out, a->N);
        if (d_vel_out) to_d4_kernel<float><<<nblocks(a->N), 256, 0, a->stream>>>(static_cast<const V*>(a->v_end), d_vel_out, a->N);
    }
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(a->stream);
    return e == cudaSuccess ? NW_OK : st_of(e);
}

nw_status nw_adj_backward(nw_adjoint* a, const float* d_grad_pos, const float* d_grad_vel, double grad_theta[4])
{
    if (!a || !d_grad_pos || !d_grad_vel || !grad_theta) return NW_ERR_INVALID;
    if (!a->have_forward) return NW_ERR_INVALID;
    return a->prec == 64 ? backward_t<double>(a, d_grad_pos, d_grad_vel, grad_theta, a->planar)
                         : backward_t<float>(a, d_grad_pos, d_grad_vel, grad_theta, a->planar);
}

nw_status nw_adj_timings(const nw_adjoint* a, float* forward_ms, float* backward_ms)
{
    if (!a) return NW_ERR_INVALID;
    if (forward_ms) *forward_ms = a->fwd_ms;
    if (backward_ms) *backward_ms = a->bwd_ms;
    return NW_OK;
}

}  // extern "C"
