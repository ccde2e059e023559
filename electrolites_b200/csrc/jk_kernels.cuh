// Kernel templates of the B200 J/K engine: one instantiation per
// angular-momentum class (li lj | lk ll), generated by
// electrolites_b200/codegen/gen_classes.py.
//
// Work decomposition (persistent grid over a sorted task list):
//   * one launch per class covers a list of plan views (one molecule for an
//     ordinary build, every molecule of a batch in a batched build);
//   * the pairs of a class are sorted by Schwarz decade (largest first),
//     then by primitive-pair count, so the kets that can pass the Schwarz
//     test q_ij + q_kl + max(dm_cond) > log(tol) form a prefix (binary
//     search, task_rows_kernel) and the lanes of a warp evaluate kets of
//     equal or similar primitive loops; each (view, bra pair) prefix is cut
//     into chunks of at most `chunk` kets, and a prefix sum over the chunk
//     counts numbers the tasks of the class;
//   * register form (jk_reg_kernel): every warp claims its own tasks, screens
//     the task's kets against the density blocks the build reads (K: D_ik,
//     D_il, D_jk, D_jl; J: D_ij, D_kl -- the reference's fill_vk_tasks /
//     fill_vjk_tasks tests, electrolites/kernels/fastk_prologue.cu:137-165,
//     electrolites/kernels/fastjk_prologue.cu:26-57), compacts the survivors
//     into a warp queue with ballots and evaluates one quartet per lane with
//     the 2D integrals and (e0|f0) accumulators in registers; warps never
//     wait on each other;
//   * team form (jk_team_kernel, large classes): a block claims a task, a team
//     of threads evaluates one quartet; the roots and 2D integrals of each
//     primitive quartet are staged in shared memory and every lane
//     accumulates the (e0|f0) row of one e-component;
//   * after the primitive sums the transfers (e0|f0) -> (ij|kl) run once per
//     quartet, and the quartet is digested into half-J / half-K accumulators
//     (J_h[k,l] += (ij|kl) (D+D^T)[i,j], J_h[i,j] += (ij|kl) (D+D^T)[k,l];
//     K_h[i,k], K_h[i,l], K_h[j,k], K_h[j,l] with D[j,l], D[j,k], D[i,l],
//     D[i,k]); the full matrices are J_h + J_h^T and K_h(D) + K_h(D^T)^T.
//     J terms and K terms are digested only when their own screening test
//     passed (quartet_bounds);
//   * mixed precision: a warp's batch of 32 quartets whose screened bounds
//     q_ij + q_kl + log max|D| are all below log(threshold) is evaluated in
//     FP32 (FP32 primitive records and Rys table, VRR, accumulation and
//     transfers), then digested and accumulated in FP64;
//   * range separation: the long-range operator erf(omega r)/r replaces
//     a_ij + a_kl by a_ij + a_kl + a_ij a_kl / omega^2 in the primitive
//     quartet (one fma);
//   * sharding: with shard_size > 1 this GPU takes the tasks
//     t = shard_rank + shard_size * n of every launch.
#pragma once
#include <cstdint>
#include <cstdio>
#include <type_traits>
#include <cuda_runtime.h>
#include "jk_device.cuh"
#include "jk_launch.h"

#define JK_NEG_INF (-3.0e38f)

// The views of a launch live in its kernel parameters (LaunchParams): one
// for an ordinary build, up to JK_VTAB for a batched one.  Their fields are
// read through the constant cache where they are used, so they hold no
// registers across the quartet loop.

// ---------------------------------------------------------------------------
// Rys roots and weights: table in shared memory (small orders) or global
// ---------------------------------------------------------------------------
template <bool SMEM>
__device__ __forceinline__ double2 ld2(const double2 *p)
{
    if constexpr (SMEM) return *p; else return __ldg(p);
}

template <bool SMEM>
__device__ __forceinline__ double rys_poly8_t(const double2 *__restrict__ cr, double s,
                                              double s2, double s4)
{
    const double2 c01 = ld2<SMEM>(cr), c23 = ld2<SMEM>(cr + 1), c45 = ld2<SMEM>(cr + 2);
    const double2 c67 = ld2<SMEM>(cr + 3);
    const double p0 = fma(c01.y, s, c01.x), p1 = fma(c23.y, s, c23.x);
    const double p2 = fma(c45.y, s, c45.x), p3 = fma(c67.y, s, c67.x);
    return fma(fma(p3, s2, p2), s4, fma(p1, s2, p0));
}

// cheb: the order-N block of the table (shared or global); tab: the whole
// global table (for the large-x limit)
template <int N, bool SMEM>
__device__ __forceinline__ void rys_eval(double x, const double *__restrict__ cheb,
                                         const double *__restrict__ tab, double *r, double *w)
{
    static_assert(RYS_DEGREE == 7, "rys_poly8_t evaluates degree 7");
    if (x >= rys_xmax<N>()) {
        const double ix = rsqrt(x);
        const double inv = ix * ix;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            r[i] = __ldg(tab + RYS_LARGEX_OFF + (N - 1) * RYS_NMAX + i) * inv;
            w[i] = __ldg(tab + RYS_LARGEX_OFF + RYS_NMAX * RYS_NMAX + (N - 1) * RYS_NMAX + i) * ix;
        }
        return;
    }
    int it;
    double s;
    rys_locate(x, it, s);
    const double s2 = s * s, s4 = s2 * s2;
    // the shared copy pads every interval by one 16-byte slot (rys_smem_stride)
    constexpr int STRIDE = 2 * N * (RYS_DEGREE + 1) + (SMEM ? 2 : 0);
    const double2 *c = reinterpret_cast<const double2 *>(cheb + it * STRIDE);
#pragma unroll
    for (int row = 0; row < 2 * N; ++row) {
        const double v = rys_poly8_t<SMEM>(c + row * (RYS_DEGREE + 1) / 2, s, s2, s4);
        if (row < N) r[row] = v; else w[row - N] = v;
    }
}

// Boys functions F_0 .. F_L, F_j = (-1)^j d^j F_0/dx^j, of the order-N (1 or 2)
// J/K classes from the shared Boys table (BOYS_STRIDE doubles per entry, an
// odd number of 16-byte slots, so that lanes at different entries spread over
// the banks): value and derivatives of one polynomial, four (N = 1) or five
// 16-byte loads where the rows of the Rys table take eight or sixteen.  (The
// shared-memory path and the FP64 pipe bound these classes: on (H2O)_96
// 6-31G* UHF they were at 52-63% and 30%.)  tab: the whole global table.
template <int N>
constexpr int boys_degree()
{
    return N == 1 ? BOYS1_DEGREE : BOYS2_DEGREE;
}
template <int N>
constexpr int boys_entries()
{
    return N == 1 ? BOYS1_ENTRIES : BOYS2_ENTRIES;
}
#define BOYS_STRIDE 10
static_assert(BOYS1_DEGREE + 3 == BOYS_STRIDE && BOYS2_DEGREE + 1 == BOYS_STRIDE, "Boys table stride");

template <int N, int L>
__device__ __forceinline__ void boys_eval(double x, const double *boys, const double *__restrict__ tab,
                                          double *f)
{
    constexpr int DEG = boys_degree<N>();
    if (x >= rys_xmax<N>()) {   // F_0 = sqrt(pi / x) / 2, F_(j+1) = (2 j + 1) / (2 x) F_j
        double ix, rx;
        // (an overflowed distance: x <= 1.1e300 by its high word, F ~ 0)
        rsqrt_rcp(__hiloint2double(min(__double2hiint(x), 0x7e3a0000), __double2loint(x)), ix, rx);
        const double hx = __ldg(tab + RYS_LARGEX_OFF) * rx;            // 1 / (2 x)
        f[0] = __ldg(tab + RYS_LARGEX_OFF + RYS_NMAX * RYS_NMAX) * ix;
#pragma unroll
        for (int j = 0; j < L; ++j) f[j + 1] = f[j] * ((2 * j + 1) * hx);
        return;
    }
    const bool g1 = x >= BOYS_SEG1;
    const double h = g1 ? BOYS_H1 : BOYS_H0, ih = g1 ? 1.0 / BOYS_H1 : 1.0 / BOYS_H0;
    // nearest integer to x / h in the low mantissa bits (1.5 * 2^52 added)
    const double m = fma(x, ih, 6755399441055744.0);
    const double y = fma(-(m - 6755399441055744.0), h, x);
    const int it = __double2loint(m) + (g1 ? BOYS_OFF1 : 0);
    const double2 *cp = reinterpret_cast<const double2 *>(boys + it * BOYS_STRIDE);
    double c[DEG + 1], p[L + 1];
#pragma unroll
    for (int k = 0; k <= DEG; k += 2) {
        const double2 v = cp[k / 2];
        c[k] = v.x;
        c[k + 1] = v.y;
    }
    // Horner, with p[j] = P^(j) / j!
    p[0] = c[DEG];
#pragma unroll
    for (int s = 1; s <= DEG; ++s) {
#pragma unroll
        for (int j = L; j > 0; --j) {
            if (s == j) p[j] = p[j - 1];
            if (s > j) p[j] = fma(p[j], y, p[j - 1]);
        }
        p[0] = fma(p[0], y, c[DEG - s]);
    }
    double sf = 1.0;   // (-1)^j j!
#pragma unroll
    for (int j = 0; j <= L; ++j) {
        f[j] = sf * p[j];
        sf *= -(j + 1);
    }
}

// one row of the table (team form: a lane per row)
template <int N>
__device__ __forceinline__ double rys_row(double x, const double *__restrict__ tab, int row)
{
    if (x >= rys_xmax<N>()) {
        const double ix = rsqrt(x);
        return row < N ? __ldg(tab + RYS_LARGEX_OFF + (N - 1) * RYS_NMAX + row) * ix * ix
                       : __ldg(tab + RYS_LARGEX_OFF + RYS_NMAX * RYS_NMAX + (N - 1) * RYS_NMAX + row - N) * ix;
    }
    int it;
    double s;
    rys_locate(x, it, s);
    const double s2 = s * s, s4 = s2 * s2;
    const double2 *cr = reinterpret_cast<const double2 *>(
        tab + rys_offset<N>() + it * (2 * N * (RYS_DEGREE + 1)) + row * (RYS_DEGREE + 1));
    return rys_poly8_t<false>(cr, s, s2, s4);
}

template <bool SMEM>
__device__ __forceinline__ float4 ld4(const float4 *p)
{
    if constexpr (SMEM) return *p; else return __ldg(p);
}

// Single-precision roots and weights (mixed form): the degree-7 table of
// order N, cheb32 its order-N block (shared copy with one 16-byte pad slot
// per interval, or global), tab the whole double table (large-x limit).
// Large x (Hermite limit) in FP64 from the double table's nodes, as the
// plain form evaluates it: only the polynomial fit below the switch point
// runs in FP32.
template <int N, bool SMEM>
__device__ __forceinline__ void rys_eval_f32(float x, const float *__restrict__ cheb32,
                                             const double *__restrict__ tab, float *r, float *w)
{
    if (x >= (float)rys_xmax<N>()) {
        const double ix = rsqrt((double)x);
        const double inv = ix * ix;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            r[i] = (float)(__ldg(tab + RYS_LARGEX_OFF + (N - 1) * RYS_NMAX + i) * inv);
            w[i] = (float)(__ldg(tab + RYS_LARGEX_OFF + RYS_NMAX * RYS_NMAX + (N - 1) * RYS_NMAX + i) * ix);
        }
        return;
    }
    int it;
    float s;
    rys_locate_f32(x, it, s);
    const float s2 = s * s, s4 = s2 * s2;
    constexpr int STRIDE = 2 * N * (RYS_DEGREE_F32 + 1) + (SMEM ? 4 : 0);
    const float4 *c = reinterpret_cast<const float4 *>(cheb32 + it * STRIDE);
#pragma unroll
    for (int row = 0; row < 2 * N; ++row) {
        const float4 lo = ld4<SMEM>(c + 2 * row), hi = ld4<SMEM>(c + 2 * row + 1);
        const float p0 = fmaf(lo.y, s, lo.x), p1 = fmaf(lo.w, s, lo.z);
        const float p2 = fmaf(hi.y, s, hi.x), p3 = fmaf(hi.w, s, hi.z);
        const float v = fmaf(fmaf(p3, s2, p2), s4, fmaf(p1, s2, p0));
        if (row < N) r[row] = v; else w[row - N] = v;
    }
}

// ---------------------------------------------------------------------------
// screening: logs of the quartet's density-weighted Schwarz bounds, for its
// K terms (blocks D_ik, D_il, D_jk, D_jl: the reference's K-only test,
// electrolites/kernels/fastk_prologue.cu:146-159) and for its J terms
// (blocks D_ij, D_kl: its J test, electrolites/kernels/fastjk_prologue.cu:
// 26-57).  A quartet is evaluated when either passes, and each kind of term
// is digested only when its own test passes -- the screening of separate
// J-only and K-only builds.  In a cluster most quartets of distant pairs
// pass for J alone (their own pair densities are large, the cross blocks
// are not), and their K loads and atomics are skipped.
// ---------------------------------------------------------------------------
// A ket's shells, bound and density come from compact copies in ket order:
// the candidates (about two per surviving quartet) read whole lines, where the
// pair records gave each lane a line of its own.
// br: the bra pair, kk: the ket; returns the ket's primitive count
__device__ __forceinline__ int quartet_bounds(const PlanView &V, const PairRec &br, int kk, float &bK,
                                               float &bJ)
{
    const int4 s = __ldg(V.scr + kk);
    const float q = br.q + __int_as_float(s.z);
    const float *dc = V.dm_cond;
    const int nb = V.nbas;
    bK = bJ = JK_NEG_INF;
    if (V.n_k) {
        const float *di = dc + br.ish * nb, *dj = dc + br.jsh * nb;
        bK = q + fmaxf(fmaxf(__ldg(di + s.x), __ldg(di + s.y)), fmaxf(__ldg(dj + s.x), __ldg(dj + s.y)));
    }
    if (V.n_j) {
        const float dkl = V.dkl ? __ldg(V.dkl + kk) : __ldg(dc + s.x * nb + s.y);
        bJ = q + fmaxf(__ldg(dc + br.ish * nb + br.jsh), dkl);
    }
    return s.w;
}

// A queued quartet: its ket index with two flags on top.
#define JK_Q_NOJ 0x40000000   // J test failed: no J terms
#define JK_Q_NOK 0x20000000   // K test failed: no K terms
#define JK_Q_LOW 0x10000000   // bound below the mixed-precision threshold
#define JK_Q_KET 0x0fffffff

__device__ __forceinline__ int queue_entry(int kk, float bK, float bJ, float log_tol)
{
    return kk | (bJ > log_tol ? 0 : JK_Q_NOJ) | (bK > log_tol ? 0 : JK_Q_NOK);
}

// Element of a matrix in the plan's AO order: component a of the shell whose
// first AO is r0 (row) with component b of the one at c0 (column); the
// components of a shell are ao_step apart (in, jn, kn: times a row).
template <int L, class VIEW>
__device__ __forceinline__ int ao_step(const VIEW &V)
{
    if constexpr (L > 0) return V.ns[L - 1]; else return 0;
}

template <class C>
struct AoIndex {
    size_t nao, in, jn, kn;
    int j, k, l;
    template <class VIEW>
    __device__ __forceinline__ explicit AoIndex(const VIEW &V)
        : nao(V.nao), in(ao_step<C::LI>(V) * (size_t)V.nao), jn(ao_step<C::LJ>(V) * (size_t)V.nao),
          kn(ao_step<C::LK>(V) * (size_t)V.nao), j(ao_step<C::LJ>(V)), k(ao_step<C::LK>(V)),
          l(ao_step<C::LL>(V))
    {
    }
    __device__ __forceinline__ size_t operator()(int r0, int a, size_t rn, int c0, int b, int cs) const
    {
        return r0 * nao + a * rn + (c0 + b * cs);
    }
};

__device__ __forceinline__ const double *kdens(const PlanView &V, int d, size_t nao2)
{
    return d < V.n_ka ? V.dmK + d * nao2 : V.dmKT + (d - V.n_ka) * nao2;
}

// densities whose bra-pair J elements J_h[i,j] a warp sums in registers over
// a task (one atomic per element per task instead of per quartet)
template <class C>
constexpr int jb_dens()
{
    return C::NI * C::NJ <= 6 ? 2 : 0;
}

// the same for the J engine's bra-side x-space elements J~_P[e]
template <class C>
constexpr int jxb_dens()
{
    return C::NE <= 6 ? 2 : 0;
}

// ---------------------------------------------------------------------------
// digestion of a whole quartet held in registers (register form)
// g[((i*NJ + j)*NK + k)*NL + l]
// ---------------------------------------------------------------------------
// JDIG = false: K only (the J engine takes J)
template <class C, bool JDIG = true>
__device__ __forceinline__ void digest_quartet(const PlanView &V, const double *g,
                                               int i0, int j0, int k0, int l0, double *jb,
                                               bool doJ, bool doK, bool full)
{
    constexpr int NI = C::NI, NJ = C::NJ, NK = C::NK, NL = C::NL, NIJ = NI * NJ;
    constexpr int JBD = JDIG ? jb_dens<C>() : 0;
    const AoIndex<C> ax(V);
    const size_t nao2 = ax.nao * ax.nao;
    const int n_j = JDIG && doJ ? V.n_j : 0, n_k = doK ? V.n_k : 0;
    const int n_jall = JDIG ? V.n_j : 0;
    for (int d = 0; d < n_j; ++d) {
        const double *ds = V.dsJ + d * nao2;
        double *jh = V.Jh + d * nao2;
        {   // J_h[k,l] += sum_ij g (D+D^T)[i,j]
            double dij[NIJ];
#pragma unroll
            for (int i = 0; i < NI; ++i)
#pragma unroll
                for (int j = 0; j < NJ; ++j) dij[i * NJ + j] = __ldg(ds + ax(i0, i, ax.in, j0, j, ax.j));
#pragma unroll
            for (int k = 0; k < NK; ++k)
#pragma unroll
                for (int l = 0; l < NL; ++l) {
                    double s = 0.;
#pragma unroll
                    for (int ij = 0; ij < NIJ; ++ij) s = fma(g[(ij * NK + k) * NL + l], dij[ij], s);
                    atomicAdd(jh + ax(k0, k, ax.kn, l0, l, ax.l), s);
                }
        }
    }
    // J_h[i,j] += sum_kl g (D+D^T)[k,l] for densities past the register
    // accumulators: every lane adds to the same bra elements, so a full warp
    // sums them with shuffles first (this loop runs alike on every lane: a
    // lane whose J test failed adds zero)
    for (int d = JBD; d < n_jall; ++d) {
        const double *ds = V.dsJ + d * nao2;
        double *jh = V.Jh + d * nao2;
        double dkl[NK * NL];
#pragma unroll
        for (int k = 0; k < NK; ++k)
#pragma unroll
            for (int l = 0; l < NL; ++l) dkl[k * NL + l] = doJ ? __ldg(ds + ax(k0, k, ax.kn, l0, l, ax.l)) : 0.;
#pragma unroll
        for (int ij = 0; ij < NIJ; ++ij) {
            double s = 0.;
#pragma unroll
            for (int kl = 0; kl < NK * NL; ++kl) s = fma(g[ij * NK * NL + kl], dkl[kl], s);
            if (full) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if ((threadIdx.x & 31) == 0) atomicAdd(jh + ax(i0, ij / NJ, ax.in, j0, ij % NJ, ax.j), s);
            } else if (doJ) {
                atomicAdd(jh + ax(i0, ij / NJ, ax.in, j0, ij % NJ, ax.j), s);
            }
        }
    }
#pragma unroll
    for (int d = 0; d < JBD; ++d) {
        if (d < n_j) {
            const double *ds = V.dsJ + d * nao2;
            double dkl[NK * NL];
#pragma unroll
            for (int k = 0; k < NK; ++k)
#pragma unroll
                for (int l = 0; l < NL; ++l) dkl[k * NL + l] = __ldg(ds + ax(k0, k, ax.kn, l0, l, ax.l));
#pragma unroll
            for (int ij = 0; ij < NIJ; ++ij) {
                double s = jb[d * NIJ + ij];
#pragma unroll
                for (int kl = 0; kl < NK * NL; ++kl) s = fma(g[ij * NK * NL + kl], dkl[kl], s);
                jb[d * NIJ + ij] = s;
            }
        }
    }
    // densities in pairs (2p, 2p+1): one 16-byte load per element of both;
    // classes whose largest density block (NI x NK) exceeds 18 elements, and
    // the large one-block classes ((e0|f0) > 27), read one density at a time
    // (the pair arrays would add to their spills)
    int d0 = 0;
    if (NI * NK <= 18 && C::NE * C::NF <= 27 && V.dmK2) {
        for (; d0 + 1 < n_k; d0 += 2) {
            const double2 *D2 = V.dmK2 + (size_t)(d0 >> 1) * nao2;
            double *kh0 = V.Kh + d0 * nao2, *kh1 = kh0 + nao2;
            {   // K_h[i,k] += sum_jl g D[j,l]
                double2 dd[NJ * NL];
#pragma unroll
                for (int j = 0; j < NJ; ++j)
#pragma unroll
                    for (int l = 0; l < NL; ++l)
                        dd[j * NL + l] = __ldg(D2 + ax(j0, j, ax.jn, l0, l, ax.l));
#pragma unroll
                for (int i = 0; i < NI; ++i)
#pragma unroll
                    for (int k = 0; k < NK; ++k) {
                        double s0 = 0., s1 = 0.;
#pragma unroll
                        for (int j = 0; j < NJ; ++j)
#pragma unroll
                            for (int l = 0; l < NL; ++l) {
                                const double gv = g[((i * NJ + j) * NK + k) * NL + l];
                                s0 = fma(gv, dd[j * NL + l].x, s0);
                                s1 = fma(gv, dd[j * NL + l].y, s1);
                            }
                        atomicAdd(kh0 + ax(i0, i, ax.in, k0, k, ax.k), s0);
                        atomicAdd(kh1 + ax(i0, i, ax.in, k0, k, ax.k), s1);
                    }
            }
            {   // K_h[i,l] += sum_jk g D[j,k]
                double2 dd[NJ * NK];
#pragma unroll
                for (int j = 0; j < NJ; ++j)
#pragma unroll
                    for (int k = 0; k < NK; ++k)
                        dd[j * NK + k] = __ldg(D2 + ax(j0, j, ax.jn, k0, k, ax.k));
#pragma unroll
                for (int i = 0; i < NI; ++i)
#pragma unroll
                    for (int l = 0; l < NL; ++l) {
                        double s0 = 0., s1 = 0.;
#pragma unroll
                        for (int j = 0; j < NJ; ++j)
#pragma unroll
                            for (int k = 0; k < NK; ++k) {
                                const double gv = g[((i * NJ + j) * NK + k) * NL + l];
                                s0 = fma(gv, dd[j * NK + k].x, s0);
                                s1 = fma(gv, dd[j * NK + k].y, s1);
                            }
                        atomicAdd(kh0 + ax(i0, i, ax.in, l0, l, ax.l), s0);
                        atomicAdd(kh1 + ax(i0, i, ax.in, l0, l, ax.l), s1);
                    }
            }
            {   // K_h[j,k] += sum_il g D[i,l]
                double2 dd[NI * NL];
#pragma unroll
                for (int i = 0; i < NI; ++i)
#pragma unroll
                    for (int l = 0; l < NL; ++l)
                        dd[i * NL + l] = __ldg(D2 + ax(i0, i, ax.in, l0, l, ax.l));
#pragma unroll
                for (int j = 0; j < NJ; ++j)
#pragma unroll
                    for (int k = 0; k < NK; ++k) {
                        double s0 = 0., s1 = 0.;
#pragma unroll
                        for (int i = 0; i < NI; ++i)
#pragma unroll
                            for (int l = 0; l < NL; ++l) {
                                const double gv = g[((i * NJ + j) * NK + k) * NL + l];
                                s0 = fma(gv, dd[i * NL + l].x, s0);
                                s1 = fma(gv, dd[i * NL + l].y, s1);
                            }
                        atomicAdd(kh0 + ax(j0, j, ax.jn, k0, k, ax.k), s0);
                        atomicAdd(kh1 + ax(j0, j, ax.jn, k0, k, ax.k), s1);
                    }
            }
            {   // K_h[j,l] += sum_ik g D[i,k]
                double2 dd[NI * NK];
#pragma unroll
                for (int i = 0; i < NI; ++i)
#pragma unroll
                    for (int k = 0; k < NK; ++k)
                        dd[i * NK + k] = __ldg(D2 + ax(i0, i, ax.in, k0, k, ax.k));
#pragma unroll
                for (int j = 0; j < NJ; ++j)
#pragma unroll
                    for (int l = 0; l < NL; ++l) {
                        double s0 = 0., s1 = 0.;
#pragma unroll
                        for (int i = 0; i < NI; ++i)
#pragma unroll
                            for (int k = 0; k < NK; ++k) {
                                const double gv = g[((i * NJ + j) * NK + k) * NL + l];
                                s0 = fma(gv, dd[i * NK + k].x, s0);
                                s1 = fma(gv, dd[i * NK + k].y, s1);
                            }
                        atomicAdd(kh0 + ax(j0, j, ax.jn, l0, l, ax.l), s0);
                        atomicAdd(kh1 + ax(j0, j, ax.jn, l0, l, ax.l), s1);
                    }
            }
        }
    }
    for (int d = d0; d < n_k; ++d) {
        const double *D = kdens(V, d, nao2);
        double *kh = V.Kh + d * nao2;
        {   // K_h[i,k] += sum_jl g D[j,l]
            double dd[NJ * NL];
#pragma unroll
            for (int j = 0; j < NJ; ++j)
#pragma unroll
                for (int l = 0; l < NL; ++l) dd[j * NL + l] = __ldg(D + ax(j0, j, ax.jn, l0, l, ax.l));
#pragma unroll
            for (int i = 0; i < NI; ++i)
#pragma unroll
                for (int k = 0; k < NK; ++k) {
                    double s = 0.;
#pragma unroll
                    for (int j = 0; j < NJ; ++j)
#pragma unroll
                        for (int l = 0; l < NL; ++l)
                            s = fma(g[((i * NJ + j) * NK + k) * NL + l], dd[j * NL + l], s);
                    atomicAdd(kh + ax(i0, i, ax.in, k0, k, ax.k), s);
                }
        }
        {   // K_h[i,l] += sum_jk g D[j,k]
            double dd[NJ * NK];
#pragma unroll
            for (int j = 0; j < NJ; ++j)
#pragma unroll
                for (int k = 0; k < NK; ++k) dd[j * NK + k] = __ldg(D + ax(j0, j, ax.jn, k0, k, ax.k));
#pragma unroll
            for (int i = 0; i < NI; ++i)
#pragma unroll
                for (int l = 0; l < NL; ++l) {
                    double s = 0.;
#pragma unroll
                    for (int j = 0; j < NJ; ++j)
#pragma unroll
                        for (int k = 0; k < NK; ++k)
                            s = fma(g[((i * NJ + j) * NK + k) * NL + l], dd[j * NK + k], s);
                    atomicAdd(kh + ax(i0, i, ax.in, l0, l, ax.l), s);
                }
        }
        {   // K_h[j,k] += sum_il g D[i,l]
            double dd[NI * NL];
#pragma unroll
            for (int i = 0; i < NI; ++i)
#pragma unroll
                for (int l = 0; l < NL; ++l) dd[i * NL + l] = __ldg(D + ax(i0, i, ax.in, l0, l, ax.l));
#pragma unroll
            for (int j = 0; j < NJ; ++j)
#pragma unroll
                for (int k = 0; k < NK; ++k) {
                    double s = 0.;
#pragma unroll
                    for (int i = 0; i < NI; ++i)
#pragma unroll
                        for (int l = 0; l < NL; ++l)
                            s = fma(g[((i * NJ + j) * NK + k) * NL + l], dd[i * NL + l], s);
                    atomicAdd(kh + ax(j0, j, ax.jn, k0, k, ax.k), s);
                }
        }
        {   // K_h[j,l] += sum_ik g D[i,k]
            double dd[NI * NK];
#pragma unroll
            for (int i = 0; i < NI; ++i)
#pragma unroll
                for (int k = 0; k < NK; ++k) dd[i * NK + k] = __ldg(D + ax(i0, i, ax.in, k0, k, ax.k));
#pragma unroll
            for (int j = 0; j < NJ; ++j)
#pragma unroll
                for (int l = 0; l < NL; ++l) {
                    double s = 0.;
#pragma unroll
                    for (int i = 0; i < NI; ++i)
#pragma unroll
                        for (int k = 0; k < NK; ++k)
                            s = fma(g[((i * NJ + j) * NK + k) * NL + l], dd[i * NK + k], s);
                    atomicAdd(kh + ax(j0, j, ax.jn, l0, l, ax.l), s);
                }
        }
    }
}

// The sums over the warp of sixteen values per lane, lane l getting that of
// v[l % 16]: halves exchanged step by step, 16 double shuffles for sixteen
// sums where a shuffle reduction of each takes 80.
__device__ __forceinline__ double warp_sum16(double *v)
{
#pragma unroll
    for (int h = 8; h > 0; h >>= 1) {
        const bool up = threadIdx.x & h;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const double keep = up ? v[k + h] : v[k], send = up ? v[k] : v[k + h];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, send, h);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 16);
}

// ---------------------------------------------------------------------------
// register form: one quartet per thread, arithmetic type T
// ---------------------------------------------------------------------------
// J engine digest of one quartet held in registers: its (e0|f0) block acc,
// scaled by fac, contracted with the x-space densities of the two pairs
// instead of being transferred to (ij|kl).  With H^P, H^Q the pairs'
// transfers, (ij|kl) = sum_ef H^P[ij,e] H^Q[kl,f] (e0|f0), so the J digest
//   J_h(Q)[kl] += sum_ij (ij|kl) (D+D^T)[ij],  J_h(P)[ij] += sum_kl (ij|kl) (D+D^T)[kl]
// becomes J~_Q[f] += sum_e (e0|f0) D~_P[e] and J~_P[e] += sum_f (e0|f0) D~_Q[f]
// with D~ = H^T (D+D^T); the pair kernels apply the transfers once per pair.
// Every lane of a full batch shares P: its terms are summed over the warp.
// Here for the f components [F0, F1) (one pass's), acc[e * (F1 - F0) + f - F0].
template <class C, class T, int F0, int F1>
__device__ __forceinline__ void jx_quartet(const ClassArgs &A, const PlanView &V, const T *acc,
                                           double fac, const PairRec &br, const PairRec &kt,
                                           double *jxb, bool doJ, bool full)
{
    constexpr int NE = C::NE, NF = C::NF, NFP = F1 - F0, JXD = jxb_dens<C>();
    const int n_j = V.n_j;
    const size_t xb = (size_t)br.xoff * n_j, xk = (size_t)kt.xoff * n_j + F0;
    for (int d = 0; d < n_j; ++d) {
        if (doJ) {   // ket side
            double s[NFP];
#pragma unroll
            for (int f = 0; f < NFP; ++f) s[f] = 0.;
#pragma unroll
            for (int e = 0; e < NE; ++e) {
                const double db = __ldg(A.jx_dens + xb + d * NE + e);
#pragma unroll
                for (int f = 0; f < NFP; ++f) s[f] = fma(double(acc[e * NFP + f]), db, s[f]);
            }
#pragma unroll
            for (int f = 0; f < NFP; ++f) atomicAdd(A.jx_acc + xk + d * NF + f, fac * s[f]);
        }
        double dk[NFP];   // bra side (a lane whose J test failed adds zero)
#pragma unroll
        for (int f = 0; f < NFP; ++f) dk[f] = doJ ? fac * __ldg(A.jx_dens + xk + d * NF + f) : 0.;
        auto term = [&](int e) {
            double s = 0.;
#pragma unroll
            for (int f = 0; f < NFP; ++f) s = fma(double(acc[e * NFP + f]), dk[f], s);
            return s;
        };
        if (d < JXD) {               // summed over the task in registers
#pragma unroll
            for (int e = 0; e < NE; ++e) {
                const double s = term(e);
#pragma unroll
                for (int dd = 0; dd < JXD; ++dd)
                    if (dd == d) jxb[dd * NE + e] += s;
            }
        } else if (full) {           // summed over the warp, 16 elements at a time
#pragma unroll
            for (int e0 = 0; e0 < NE; e0 += 16) {
                double v[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) v[e] = e0 + e < NE ? term(e0 + e) : 0.;
                const double s = warp_sum16(v);
                const int e = e0 + (threadIdx.x & 15);
                if ((threadIdx.x & 16) == 0 && e < NE) atomicAdd(A.jx_acc + xb + d * NE + e, s);
            }
        } else if (doJ) {
#pragma unroll
            for (int e = 0; e < NE; ++e) atomicAdd(A.jx_acc + xb + d * NE + e, term(e));
        }
    }
}

// Part `part` of `parts` of a quartet's primitive quartets: every kstep-th ket
// primitive from kp0 and every bstep-th bra primitive from bp0, the ket
// primitives divided first.  False when nothing is left for this part.
__device__ __forceinline__ bool split_part(int part, int parts, int nket, int nbra, int &kp0,
                                           int &kstep, int &bp0, int &bstep)
{
    kstep = min(parts, nket);
    bstep = parts / kstep;
    bp0 = part / kstep;
    kp0 = part - bp0 * kstep;
    return bp0 < bstep && bp0 < nbra;
}

// The primitive loops of one quartet, pass P: acc[e * NFP + f] += its (e0|f0)
// integrals for the NFP f components of the pass, over every kstep-th ket
// primitive from kp0 and every bstep-th bra primitive from bp0
template <class C, class T, bool SMEM, int OP, int P>
__device__ __forceinline__ void reg_accum(const ClassArgs &A, const PlanView &V, const PairRec &br,
                                          const PairRec &kt, const double *__restrict__ sbra,
                                          const float *__restrict__ sbra32,
                                          const double *__restrict__ cheb,
                                          const float *__restrict__ cheb32, int kp0, int kstep,
                                          int bp0, int bstep, T *acc)
{
    constexpr int N = C::NROOTS;
    constexpr int NACC = C::NE * (C::pass_f(P + 1) - C::pass_f(P));
#pragma unroll
    for (int n = 0; n < NACC; ++n) acc[n] = T(0);
    if constexpr (sizeof(T) == 8) {
        // the ket's primitive records from the field-major copy: field f of
        // primitive k at ks[(k * JK_SOA_FIELDS + f) * JK_SOA_TILE], so the
        // lanes of a warp (neighbouring kets) read neighbouring doubles
        constexpr int sn = JK_SOA_TILE;
        const double *ks = V.prim_soa + kt.soa + kp0 * (JK_SOA_FIELDS * sn);
        const int kn = kstep * (JK_SOA_FIELDS * sn);
        // one pass over the primitive quartets per operator term: the
        // integrals are linear in the operator, so the terms share the
        // accumulators (a second term re-reads the ket primitives).  The
        // one-term pass reads its omega from the kernel parameters and
        // leaves the coefficient to the symmetry factor below.
        auto pass = [&](const double io2, const double ct) {
            double n[JK_SOA_FIELDS];
            const double *kr = ks;
#pragma unroll
            for (int f = 0; f < JK_SOA_FIELDS; ++f) n[f] = __ldg(kr + f * sn);
            for (int kp = kp0; kp < kt.nprim; kp += kstep) {
                // the next ket primitive's record is loaded while this one is used
                double v[JK_SOA_FIELDS];
#pragma unroll
                for (int f = 0; f < JK_SOA_FIELDS; ++f) v[f] = n[f];
                if (kp + kstep < kt.nprim) {
                    kr += kn;
#pragma unroll
                    for (int f = 0; f < JK_SOA_FIELDS; ++f) n[f] = __ldg(kr + f * sn);
                }
                const double akl = v[PR_A], hiq = v[PR_HIA], kq = v[PR_KP] * ct;
                const double Qx = v[PR_PX], Qy = v[PR_PX + 1], Qz = v[PR_PX + 2];
                const double QCx = v[PR_PAX], QCy = v[PR_PAX + 1], QCz = v[PR_PAX + 2];
                for (int bp = bp0; bp < br.nprim; bp += bstep) {
                    // the record in 16-byte loads (the same for every lane)
                    const double2 *s = reinterpret_cast<const double2 *>(sbra + bp * JK_PRIM_STRIDE);
                    const double2 s01 = s[0], s23 = s[1], s45 = s[2], s67 = s[3], s89 = s[4];
                    const double aij = s01.x, hip = s01.y;
                    const double PQx = s23.y - Qx, PQy = s45.x - Qy, PQz = s45.y - Qz;
                    const double PAx = s67.x, PAy = s67.y, PAz = s89.x;
                    // inv_om2 = 1/omega^2 > 0: the long-range erf(omega r)/r
                    // operator, whose Rys quadrature is the Coulomb one with
                    // a_ij + a_kl replaced by a_ij + a_kl + a_ij a_kl / omega^2
                    double rs, is;
                    rsqrt_rcp(fma(aij * akl, io2, aij + akl), rs, is);
                    const double rr = fma(PQx, PQx, fma(PQy, PQy, PQz * PQz));
                    const double x = aij * akl * is * rr;
                    const double pref = s23.x * kq * rs;
                    if constexpr (N <= 2) {
                        double F[C::LIJ + C::LKL + 1];
                        boys_eval<N, C::LIJ + C::LKL>(x, cheb, A.rys, F);
#pragma unroll
                        for (int m = 0; m <= C::LIJ + C::LKL; ++m) F[m] *= pref;
                        const double sp = is * akl, sq = is * aij;   // W - P = -sp PQ, W - Q = sq PQ
                        C::boys_acc(F, PAx, PAy, PAz, -sp * PQx, -sp * PQy, -sp * PQz, QCx, QCy, QCz,
                                    sq * PQx, sq * PQy, sq * PQz, hip, sp, 0.5 * is, acc);
                        continue;
                    }
                    double r[N], w[N];
                    rys_eval<N, SMEM>(x, cheb, A.rys, r, w);
#pragma unroll
                    for (int n = 0; n < N; ++n) {
                        const double uis = r[n] * is;
                        const double up = uis * akl, uq = uis * aij;
                        C::template root_acc<P, double>(fma(-up, PQx, PAx), fma(-up, PQy, PAy),
                                                     fma(-up, PQz, PAz), fma(uq, PQx, QCx),
                                                     fma(uq, PQy, QCy), fma(uq, PQz, QCz),
                                                     0.5 * uis, fma(-hip, up, hip),
                                                     fma(-hiq, uq, hiq), w[n] * pref, acc);
                    }
                }
            }
        };
        if constexpr (OP == 1) {
            pass(A.op_inv_om2[0], 1.0);
        } else {
            for (int t = 0; t < 2; ++t) pass(A.op_inv_om2[t], A.op_coef[t]);
        }
    } else {
        // single precision throughout: FP32 copies of the primitive records
        // (ket from global, bra staged in shared memory), no conversions
        const float4 *r4 = reinterpret_cast<const float4 *>(V.prim32 + (size_t)kt.prim0 * JK_PRIM32_STRIDE);
        auto pass = [&](const float io2, const float ct) {   // operator terms, as above
            const float4 *r0 = r4 + kp0 * (JK_PRIM32_STRIDE / 4);
            float4 n0 = __ldg(r0), n1 = __ldg(r0 + 1), n2 = __ldg(r0 + 2);
            for (int kp = kp0; kp < kt.nprim; kp += kstep) {
                const float4 v0 = n0, v1 = n1, v2 = n2;
                if (kp + kstep < kt.nprim) {
                    const float4 *rn = r4 + (kp + kstep) * (JK_PRIM32_STRIDE / 4);
                    n0 = __ldg(rn);
                    n1 = __ldg(rn + 1);
                    n2 = __ldg(rn + 2);
                }
                const float akl = v0.x, hiq = v0.y, kq = v0.z * ct;
                const float Qx = v0.w, Qy = v1.x, Qz = v1.y;
                const float QCx = v1.z, QCy = v1.w, QCz = v2.x;
                for (int bp = bp0; bp < br.nprim; bp += bstep) {
                    const float *s = sbra32 + bp * JK_PRIM32_STRIDE;
                    const float aij = s[PR_A], hip = s[PR_HIA];
                    const float PQx = s[PR_PX] - Qx, PQy = s[PR_PX + 1] - Qy;
                    const float PQz = s[PR_PX + 2] - Qz;
                    float r[N], w[N];
                    const float rs = rsqrtf(fmaf(aij * akl, io2, aij + akl));
                    const float is = rs * rs;
                    const float rr = fmaf(PQx, PQx, fmaf(PQy, PQy, PQz * PQz));
                    const float x = aij * akl * is * rr;
                    const float pref = s[PR_KP] * kq * rs;
                    if (SMEM && A.mixed_tab)
                        rys_eval_f32<N, true>(x, cheb32, A.rys, r, w);
                    else
                        rys_eval_f32<N, false>(x, cheb32, A.rys, r, w);
                    const float PAx = s[PR_PAX], PAy = s[PR_PAX + 1], PAz = s[PR_PAX + 2];
#pragma unroll
                    for (int n = 0; n < N; ++n) {
                        const float uis = r[n] * is;
                        const float up = uis * akl, uq = uis * aij;
                        C::template root_acc<P, float>(fmaf(-up, PQx, PAx), fmaf(-up, PQy, PAy),
                                                    fmaf(-up, PQz, PAz), fmaf(uq, PQx, QCx),
                                                    fmaf(uq, PQy, QCy), fmaf(uq, PQz, QCz),
                                                    0.5f * uis, fmaf(-hip, up, hip),
                                                    fmaf(-hiq, uq, hiq), w[n] * pref, acc);
                    }
                }
            }
        };
        if constexpr (OP == 1) {
            pass((float)A.op_inv_om2[0], 1.0f);
        } else {
            for (int t = 0; t < 2; ++t) pass((float)A.op_inv_om2[t], (float)A.op_coef[t]);
        }
    }
}

// f columns [F0, F1) of the block, scaled by fac, through the bra transfer:
// tb[(f - F0) * NIJ + ij]
template <class C, class T, int F0, int F1>
__device__ __forceinline__ void reg_bra(const PairRec &br, const T *acc, T fac, T *tb)
{
    constexpr int NE = C::NE, NIJ = C::NI * C::NJ, NFP = F1 - F0;
#pragma unroll
    for (int f = 0; f < NFP; ++f) {
        T col[NE];
#pragma unroll
        for (int e = 0; e < NE; ++e) col[e] = acc[e * NFP + f] * fac;
        C::template hrr_bra<T>(col, tb + f * NIJ, T(br.ABx), T(br.ABy), T(br.ABz));
    }
}

// one pass: accumulation, J engine, bra transfer; then the passes after it
template <class C, class T, bool SMEM, int OP, int JX, int P>
__device__ __forceinline__ void reg_passes(const ClassArgs &A, const PlanView &V, const PairRec &br,
                                           const PairRec &kt, const double *__restrict__ sbra,
                                           const float *__restrict__ sbra32,
                                           const double *__restrict__ cheb,
                                           const float *__restrict__ cheb32, int kp0, int kstep,
                                           int bp0, int bstep, T fac, double *jb, bool doJ,
                                           bool doK, bool full, T *tb)
{
    constexpr int F0 = C::pass_f(P), F1 = C::pass_f(P + 1);
    {
        T acc[C::NE * (F1 - F0)];
        reg_accum<C, T, SMEM, OP, P>(A, V, br, kt, sbra, sbra32, cheb, cheb32, kp0, kstep, bp0, bstep,
                                     acc);
        if constexpr (JX != 0)   // J engine: J without transfers
            jx_quartet<C, T, F0, F1>(A, V, acc, double(fac), br, kt, jb, doJ, full);
        if (JX != 2 && doK) reg_bra<C, T, F0, F1>(br, acc, fac, tb + F0 * C::NI * C::NJ);
    }
    if constexpr (P + 1 < C::NPASS)
        reg_passes<C, T, SMEM, OP, JX, P + 1>(A, V, br, kt, sbra, sbra32, cheb, cheb32, kp0, kstep,
                                              bp0, bstep, fac, jb, doJ, doK, full, tb);
}

// OP: operator terms (1: op_inv_om2[0], op_coef[0] read from the kernel
// parameters; 2: both terms of ClassArgs); JX: 0 the (ij|kl) digest, 1 the
// J engine for J and the digest for K, 2 the J engine alone (J-only builds)
// SPLIT: the quartet's primitive quartets are shared by `parts` lanes, this
// one the part-th of them (a partial batch, reg_task); each digests its own
// partial integrals, which enter J and K linearly
template <class C, class T, bool SMEM, int OP, int JX, bool SPLIT>
__device__ __forceinline__ void reg_quartet(const ClassArgs &A, const PlanView &V,
                                            const PairRec &br, const double *__restrict__ sbra,
                                            const float *__restrict__ sbra32,
                                            int entry, double sym, const double *__restrict__ cheb,
                                            const float *__restrict__ cheb32, double *jb,
                                            bool full, int part, int parts)
{
    const int kk = entry & JK_Q_KET;
    constexpr int NF = C::NF, NIJ = C::NI * C::NJ, NKL = C::NK * C::NL;
    const PairRec kt = V.ket[kk];
    int kp0 = 0, kstep = 1, bp0 = 0, bstep = 1;
    if constexpr (SPLIT) {
        if (!split_part(part, parts, kt.nprim, br.nprim, kp0, kstep, bp0, bstep)) return;
    }
    const T fac = T((kt.ish == kt.jsh ? 0.5 * sym : sym) * (OP == 1 ? A.op_coef[0] : 1.0));
    // the digest of (ij|kl): J and K, or the K of a quartet kept for it (J engine)
    const bool doJ = !(entry & JK_Q_NOJ), doK = V.n_k != 0 && !(entry & JK_Q_NOK);
    T tb[NF * NIJ];
    reg_passes<C, T, SMEM, OP, JX, 0>(A, V, br, kt, sbra, sbra32, cheb, cheb32, kp0, kstep, bp0, bstep,
                                      fac, jb, doJ, JX == 0 || doK, full, tb);
    if constexpr (JX == 2) return;
    if (JX == 1 && !doK) return;   // nothing for K: no transfers
    double g[NIJ * NKL];
#pragma unroll
    for (int ij = 0; ij < NIJ; ++ij) {
        T row[NF], o[NKL];
#pragma unroll
        for (int f = 0; f < NF; ++f) row[f] = tb[f * NIJ + ij];
        C::template hrr_ket<T>(row, o, T(kt.ABx), T(kt.ABy), T(kt.ABz));
#pragma unroll
        for (int kl = 0; kl < NKL; ++kl) g[ij * NKL + kl] = double(o[kl]);
    }
    digest_quartet<C, JX == 0>(V, g, br.i0, br.j0, kt.i0, kt.j0, jb, doJ, doK, full);
}

// ---------------------------------------------------------------------------
// task claiming (one lane claims, the warp gets the result)
// ---------------------------------------------------------------------------
struct Task {
    int view, bra, k0, k1;
};

// First index in [lo, hi] whose value exceeds t, or hi (v non-decreasing): the
// 32 lanes probe at a time, three dependent loads for 32 000 rows where a
// binary search takes fifteen -- as long as a small task's own work.
__device__ __forceinline__ int warp_upper_bound(const int *v, int lo, int hi, int t, int lane)
{
    while (lo < hi) {
        const int step = (hi - lo + 31) >> 5, p = lo + lane * step;
        const int n = __popc(__ballot_sync(0xffffffffu, p < hi && v[p] <= t));   // probes at most t
        if (n == 0) break;
        hi = min(hi, lo + n * step);
        lo += (n - 1) * step + 1;
    }
    return lo;
}

// Task t of this launch -> row (search of the chunk prefix over the launch's
// rows) -> view (search of the views' first rows) -> bra pair and ket range.
// Lane 0 claims; every lane gets the task.
template <int NV>
__device__ __forceinline__ bool claim_task(const LaunchParams<NV> &P, int t_begin, int t_end,
                                           int chunk, Task &T)
{
    const ClassArgs &A = P.a;
    const int lane = threadIdx.x & 31;
    int t = 0;
    if (lane == 0) t = t_begin + A.shard_rank + A.shard_size * atomicAdd(A.counter, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= t_end) return false;
    const int row = warp_upper_bound(A.row_prefix, A.row_begin, A.row_end - 1, t, lane);
    const int c = t - (row > A.row_first ? A.row_prefix[row - 1] : 0);
    T.view = 0;
    if constexpr (NV > 1)        // last view with row0 <= row
        T.view = warp_upper_bound(A.view_row0 + A.view_begin, 0, A.nvl, row, lane) - 1;
    T.bra = row - P.v[T.view].row0;
    T.k0 = c * chunk;
    T.k1 = min(A.row_ncand[row], T.k0 + chunk);
    return true;
}

// first and one-past-last task of a launch
__device__ __forceinline__ void launch_tasks(const ClassArgs &A, int &t_begin, int &t_end)
{
    t_begin = A.row_begin > A.row_first ? A.row_prefix[A.row_begin - 1] : 0;
    t_end = A.row_end > A.row_first ? A.row_prefix[A.row_end - 1] : 0;
}

// ---------------------------------------------------------------------------
// register-form kernel: warp-level tasks
// ---------------------------------------------------------------------------
template <class C>
constexpr bool rys_smem()
{
    return C::NROOTS <= 4;
}

// doubles per interval of the shared copy: one 16-byte pad slot each, so
// that lanes reading different intervals spread over all bank groups
template <class C>
constexpr int rys_smem_stride()
{
    return 2 * C::NROOTS * (RYS_DEGREE + 1) + 2;
}

// the one- and two-root classes read the Boys table instead (JX = 3, the
// McMurchie-Davidson J, keeps the Rys table)
template <class C, int JX>
constexpr bool boys_class()
{
    return C::NROOTS <= 2 && JX != 3;
}

template <class C, int JX>
constexpr int rys_smem_doubles()
{
    if (boys_class<C, JX>()) return boys_entries<C::NROOTS>() * BOYS_STRIDE;
    return rys_smem<C>() ? rys_nint<C::NROOTS>() * rys_smem_stride<C>() : 0;
}

// the single-precision table of the mixed form, same padding (in floats)
template <class C>
constexpr int rys32_smem_stride()
{
    return 2 * C::NROOTS * (RYS_DEGREE_F32 + 1) + 4;
}

// doubles of shared memory the single-precision table takes (0 when the
// build has no FP32 quartets or the class reads the tables from global)
template <class C>
__host__ __device__ constexpr int rys32_smem_doubles(int mixed)
{
    return rys_smem<C>() && mixed ? (rys_nint<C::NROOTS>() * rys32_smem_stride<C>() + 1) / 2 : 0;
}

// blocks per SM of the register form: small classes ((e0|f0) <= 12) two
// 256-thread blocks (<= 128 registers), mid-size ones (<= 27) three
// 128-thread blocks (<= 170 registers: their accumulators spill at 128),
// larger ones keep their accumulators in registers at one 256-thread block
template <class C>
constexpr int reg_min_blocks()
{
    // (ss|ss), (e0|f0) = 1: three 256-thread blocks (80 registers, 96 bytes
    // of spills) measured 36.5 -> 34.4 ms on (H2O)_96 6-31G* UHF; (ps|ss)
    // lost at that cap (47.7 -> 50.5 ms) and keeps two
    return C::NE * C::NF == 1 ? 3 : (C::NE * C::NF <= 12 ? 2 : (C::NE * C::NF <= 27 ? 3 : 1));
}

// threads per block: 128 for the mid-size classes (3 blocks of 4 warps at
// <= 170 registers), 256 otherwise
template <class C>
constexpr int reg_threads()
{
    return reg_min_blocks<C>() == 3 && C::NE * C::NF > 1 ? 128 : 256;
}

#include "jk_mdj.cuh"

// Per-warp state of the register form across its tasks.
struct RegWarp {
    double *sbra;       // staged bra primitive records
    double *sdh;        // McMurchie-Davidson J: the bra's Hermite densities
    float *sbra32;      // their FP32 copies (mixed form)
    int *q;             // queue of surviving quartets
    const double *cheb; // Rys table (shared copy or global)
    const float *cheb32; // single-precision Rys table (shared copy or global)
    int staged_v, staged_b;
    unsigned long long nq, npq, nq32;
};

// The surviving quartets of a task, kets [k0, k1), handed on in batches of 32
// (batch(queue entries, how many, split)), the last of them partial (split:
// std::true_type; ONE_COPY: always, so that the batch's code is there once).
template <bool ONE_COPY, class BATCH>
__device__ __forceinline__ void ket_batches(const PlanView &V, const PairRec &br, int k0, int k1,
                                            int *q, int lane, float log_tol, float log_mixed,
                                            BATCH batch)
{
    int nq = 0;
    for (int base = k0;; base += 32) {
        const bool more = base < k1;
        if (more) {
            const int kk = base + lane;
            float bK = JK_NEG_INF, bJ = JK_NEG_INF;
            if (kk < k1) quartet_bounds(V, br, kk, bK, bJ);
            const float bound = fmaxf(bK, bJ);
            const unsigned m = __ballot_sync(0xffffffffu, bound > log_tol);
            if (bound > log_tol)
                q[nq + __popc(m & ((1u << lane) - 1u))] =
                    queue_entry(kk, bK, bJ, log_tol) | (bound < log_mixed ? JK_Q_LOW : 0);
            nq += __popc(m);
            __syncwarp();
        }
        if (nq >= 32 || (ONE_COPY && !more && nq > 0)) {
            const int n = ONE_COPY ? min(nq, 32) : 32;
            batch(q, n, std::integral_constant<bool, ONE_COPY>());
            if (lane < nq - 32) q[lane] = q[32 + lane];
            __syncwarp();
            nq -= n;
        }
        if (!more) break;
    }
    if (!ONE_COPY && nq > 0) batch(q, nq, std::true_type());
}

// The same with the quartets queued by their ket's primitive count, five
// buckets a factor of two apart, because the lanes of a batch run as long as
// its largest count: in the order of the list a (H2O)_6 6-31G* build fills
// 0.52 of the lanes of its (ss|ss) primitive loops, (H2O)_24 0.77, (H2O)_96
// 0.96.  What is left of every bucket at the task's end makes the last
// batches.  Sorting costs the screening five ballots per 32 candidates, the
// batches neighbours in the list and the kernel registers: gradients, whose
// primitive quartets cost more, always sort ((H2O)_17 UHF 34.9 -> 27.7 ms);
// batched J/K builds sort where the ket class is small (PlanView::buckets;
// 24 molecules of up to 10 waters 15.3 -> 14.2 ms), single builds never
// ((H2O)_96 251 -> 268 ms, (H2O)_21 def2-SVP 9.7 -> 10.3).
#define JK_BUCKETS 5
#define JK_QUEUE (JK_BUCKETS * 64)

template <bool ONE_COPY, class BATCH>
__device__ __forceinline__ void ket_batches_sorted(const PlanView &V, const PairRec &br, int k0,
                                                   int k1, int *q, int lane, bool sort, float log_tol,
                                                   float log_mixed, BATCH batch)
{
    unsigned cnt = 0;                // queued per bucket, six bits each
    for (int base = k0;; base += 32) {
        const bool more = base < k1;
        int left = 0, at = 0;
        if (more) {
            const int kk = base + lane;
            float bK = JK_NEG_INF, bJ = JK_NEG_INF;
            int np = 0;
            if (kk < k1) np = quartet_bounds(V, br, kk, bK, bJ);
            if (!sort) np = 64;
            const float bound = fmaxf(bK, bJ);
            const int entry = queue_entry(kk, bK, bJ, log_tol) | (bound < log_mixed ? JK_Q_LOW : 0);
            const int bucket = bound > log_tol ? (np < 24) + (np < 12) + (np < 6) + (np < 3) : -1;
#pragma unroll
            for (int b = 0; b < JK_BUCKETS; ++b) {
                if (b && !sort) break;
                const unsigned m = __ballot_sync(0xffffffffu, bucket == b);
                if (bucket == b)
                    q[b * 64 + (cnt >> 6 * b & 63) + __popc(m & ((1u << lane) - 1u))] = entry;
                cnt += (unsigned)__popc(m) << 6 * b;
            }
        } else {
#pragma unroll
            for (int b = 0; b < JK_BUCKETS; ++b) {   // at most 31 of each
                const int c = cnt >> 6 * b & 63;
                const int e = lane < c ? q[b * 64 + lane] : 0;
                __syncwarp();
                if (lane < c) q[left + lane] = e;
                left += c;
            }
        }
        __syncwarp();
        for (;;) {
            const unsigned full = cnt & 0x20820820u;   // bit 5 of every bucket's count
            const int b = (__ffs(full) - 1) / 6;
            if (more ? full == 0 : at >= left) break;
            const int *src = q + (more ? b * 64 : at);
            const int n = more ? 32 : min(32, left - at);
            if (!ONE_COPY && n == 32)
                batch(src, n, std::false_type());
            else
                batch(src, n, std::true_type());
            at += 32;
            if (more) {
                if (lane < (int)(cnt >> 6 * b & 63) - 32) q[b * 64 + lane] = q[b * 64 + 32 + lane];
                cnt -= 32u << 6 * b;
                __syncwarp();
            }
        }
        if (!more) break;
    }
}

// one task of the register form: bra pair task.bra of view V against kets
// [task.k0, task.k1); SORT: the batched kernels' queue by primitive count
template <class C, bool SMEM, int OP, int JX, bool SORT>
__device__ __forceinline__ void reg_task(const ClassArgs &A, const PlanView &V, const Task &task,
                                         RegWarp &w, int lane)
{
    constexpr int NIJ = C::NI * C::NJ;
    constexpr int JBD = jb_dens<C>();
    const int b = task.bra;
    const PairRec br = V.bra[b];
    if (b != w.staged_b || task.view != w.staged_v) {
        __syncwarp();
        const double *src = V.prim + (size_t)br.prim0 * JK_PRIM_STRIDE;
        for (int t = lane; t < br.nprim * JK_PRIM_STRIDE; t += 32) w.sbra[t] = src[t];
        if (A.mixed) {
            const float *src32 = V.prim32 + (size_t)br.prim0 * JK_PRIM32_STRIDE;
            for (int t = lane; t < br.nprim * JK_PRIM32_STRIDE; t += 32) w.sbra32[t] = src32[t];
        }
        __syncwarp();
        if constexpr (JX == 3) {   // the bra's Hermite densities, per primitive and density
            constexpr int NTP = md_nt(C::LI + C::LJ);
            for (int t = lane; t < br.nprim * JK_MD_DENS; t += 32) {
                const int bp = t / JK_MD_DENS, d = t - bp * JK_MD_DENS;
                double *dh = w.sdh + t * NTP;
                if (d < V.n_j) {
                    md_bra_dens<C>(V, br, w.sbra + bp * JK_PRIM_STRIDE, d, dh);
                } else {
                    for (int h = 0; h < NTP; ++h) dh[h] = 0.;
                }
            }
            __syncwarp();
        }
        w.staged_b = b;
        w.staged_v = task.view;
    }
    const double sym_b = br.ish == br.jsh ? 0.5 : 1.0;
    const bool diag = V.bra == V.ket;
    const float log_tol = V.log_tol, log_mixed = A.mixed ? A.mixed_log_thr : JK_NEG_INF;
    // task-level register sums: J_h[i,j] of the digest, or the J engine's
    // bra-side J~_P[e]
    constexpr int NJB = JX == 3 ? JK_MD_DENS * NIJ : (JX != 0 ? jxb_dens<C>() * C::NE : JBD * NIJ);
    double jb[NJB > 0 ? NJB : 1];
#pragma unroll
    for (int n = 0; n < NJB; ++n) jb[n] = 0.;
    // A batch of up to 32 quartets (ket_batches) runs in FP32 when every one of
    // them is below the mixed-precision threshold, in FP64 otherwise (the kets
    // are sorted by Schwarz bound, so batches are mostly of one kind).  The
    // lanes of a partial batch without a quartet take a share of another's
    // primitive quartets.
    auto batch = [&](const int *src, int n, auto split) {
        constexpr bool SPLIT = decltype(split)::value;
        const int parts = SPLIT && JX != 3 ? 32 / n : 1, part = SPLIT && JX != 3 ? lane / n : 0;
        const bool on = lane < n * parts;
        const int e2 = src[on ? lane - part * n : 0], k2 = e2 & JK_Q_KET;
        const bool low = JX != 3 && __all_sync(0xffffffffu, e2 & JK_Q_LOW);
        if (on) {
            const double sym = diag && k2 == b ? 0.5 * sym_b : sym_b;
            if constexpr (JX == 3) {
                md_quartet<C, SMEM>(A, V, br, w.sbra, w.sdh, e2, sym, w.cheb, jb);
            } else if (low) {
                reg_quartet<C, float, SMEM, OP, JX, SPLIT>(A, V, br, w.sbra, w.sbra32, e2, sym, w.cheb,
                                                           w.cheb32, jb, n == 32, part, parts);
            } else {
                reg_quartet<C, double, SMEM, OP, JX, SPLIT>(A, V, br, w.sbra, w.sbra32, e2, sym, w.cheb,
                                                            w.cheb32, jb, n == 32, part, parts);
            }
            if (part == 0) w.npq += (unsigned long long)br.nprim * V.ket[k2].nprim;
        }
        w.nq += n;
        if (low) w.nq32 += n;
        __syncwarp();
    };
    // the larger classes' quartet code once, for full and partial batches alike
    constexpr bool ONE_COPY = C::NE * C::NF > 27;
    if constexpr (SORT)
        ket_batches_sorted<ONE_COPY>(V, br, task.k0, task.k1, w.q, lane, V.buckets, log_tol, log_mixed,
                                     batch);
    else
        ket_batches<ONE_COPY>(V, br, task.k0, task.k1, w.q, lane, log_tol, log_mixed, batch);
    // bra-pair J elements of this task: one atomic per element
    if constexpr (JX == 3) {
        const AoIndex<C> ax(V);
#pragma unroll
        for (int d = 0; d < JK_MD_DENS; ++d) {
            if (d < V.n_j) {
#pragma unroll
                for (int ij = 0; ij < NIJ; ++ij) {
                    double v = jb[d * NIJ + ij];
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                    if (lane == 0)
                        atomicAdd(V.Jh + d * ax.nao * ax.nao + ax(br.i0, ij / C::NJ, ax.in, br.j0, ij % C::NJ, ax.j), v);
                }
            }
        }
    } else if constexpr (JX != 0) {
        constexpr int JXD = jxb_dens<C>();
        const size_t xb = (size_t)br.xoff * V.n_j;
#pragma unroll
        for (int d = 0; d < JXD; ++d) {
            if (d < V.n_j) {
#pragma unroll
                for (int e = 0; e < C::NE; ++e) {
                    double v = jb[d * C::NE + e];
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                    if (lane == 0) atomicAdd(A.jx_acc + xb + d * C::NE + e, v);
                }
            }
        }
    } else if constexpr (JBD > 0) {
        const AoIndex<C> ax(V);
#pragma unroll
        for (int d = 0; d < JBD; ++d) {
            if (d < V.n_j) {
#pragma unroll
                for (int ij = 0; ij < NIJ; ++ij) {
                    double v = jb[d * NIJ + ij];
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                    if (lane == 0)
                        atomicAdd(V.Jh + d * ax.nao * ax.nao + ax(br.i0, ij / C::NJ, ax.in, br.j0, ij % C::NJ, ax.j), v);
                }
            }
        }
    }
}

__device__ __forceinline__ void copy16_async(void *smem, const void *global)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(smem)),
                 "l"(global)
                 : "memory");
}

// (the McMurchie-Davidson J instantiation, JX = 3, holds its Hermite
// tensors beside the accumulators: one block per SM, all 255 registers)
template <class C, int NT, int NV, int OP, int JX>
__global__ void __launch_bounds__(NT, JX == 3 ? 1 : reg_min_blocks<C>())
    jk_reg_kernel(const __grid_constant__ LaunchParams<NV> P)
{
    const ClassArgs &A = P.a;
    constexpr int NW = NT / 32;
    constexpr bool SMEM = rys_smem<C>();
    constexpr int TAB = rys_smem_doubles<C, JX>();
    extern __shared__ double smem[];
    __shared__ int s_q[NW][NV > 1 ? JK_QUEUE : 64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int TAB32 = rys32_smem_doubles<C>(A.mixed_tab);
    float *smem32 = reinterpret_cast<float *>(smem + TAB);
    int t_begin, t_end;
    launch_tasks(A, t_begin, t_end);
    // the grid is sized for a large molecule: with fewer tasks than warps the
    // blocks past four tasks each leave before they stage the table
    if ((long long)blockIdx.x * 4 >= t_end - t_begin) return;
    if constexpr (SMEM) {
        // table rows of an interval are contiguous, the shared copy pads each
        // interval by one 16-byte slot: asynchronous 16-byte copies, all in
        // flight at once (the loop of 8-byte loads and stores took longer than
        // a small molecule's whole class)
        constexpr bool BOYS = boys_class<C, JX>();
        constexpr int U = BOYS ? (boys_degree<C::NROOTS>() + 1) / 2   // 16-byte units of an interval
                               : C::NROOTS * (RYS_DEGREE + 1);
        constexpr int SU = BOYS ? BOYS_STRIDE / 2 : U + 1;            // and in the shared copy
        constexpr int NINT = BOYS ? boys_entries<C::NROOTS>() : rys_nint<C::NROOTS>();
        const double2 *src = reinterpret_cast<const double2 *>(
            A.rys + (!BOYS ? rys_offset<C::NROOTS>() : C::NROOTS == 1 ? BOYS1_TABLE_OFF : BOYS2_TABLE_OFF));
        double2 *dst = reinterpret_cast<double2 *>(smem);
        for (int t = threadIdx.x; t < NINT * U; t += NT)
            copy16_async(dst + t / U * SU + t % U, src + t);
        if (TAB32) {
            constexpr int U32 = 2 * C::NROOTS * (RYS_DEGREE_F32 + 1) / 4;
            const float4 *src32 = reinterpret_cast<const float4 *>(A.rys32 + rys32_offset<C::NROOTS>());
            float4 *dst32 = reinterpret_cast<float4 *>(smem32);
            for (int t = threadIdx.x; t < rys_nint<C::NROOTS>() * U32; t += NT)
                copy16_async(dst32 + t + t / U32, src32 + t);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
    }
    RegWarp w;
    w.cheb = SMEM ? smem : A.rys + rys_offset<C::NROOTS>();
    w.cheb32 = SMEM && A.mixed_tab ? smem32 : A.rys32 + rys32_offset<C::NROOTS>();
    w.sbra = smem + TAB + TAB32 + warp * A.max_bra_prim * JK_PRIM_STRIDE;
    w.sbra32 = reinterpret_cast<float *>(smem + TAB + TAB32 + NW * A.max_bra_prim * JK_PRIM_STRIDE) +
               warp * A.max_bra_prim * JK_PRIM32_STRIDE;
    // McMurchie-Davidson J builds are FP64 only: their Hermite densities take
    // the place of the FP32 records
    w.sdh = JX == 3 ? smem + TAB + TAB32 + NW * A.max_bra_prim * JK_PRIM_STRIDE +
                          (size_t)warp * A.max_bra_prim * JK_MD_DENS * md_nt(C::LI + C::LJ)
                    : nullptr;
    w.q = s_q[warp];
    w.staged_v = w.staged_b = -1;
    w.nq = w.npq = w.nq32 = 0;
    const int chunk = *A.chunk;
    Task task;
    while (claim_task(P, t_begin, t_end, chunk, task))
        reg_task<C, SMEM, OP, JX, (NV > 1)>(A, P.v[task.view], task, w, lane);
    if (lane == 0) {
        if (A.nquartets) atomicAdd(A.nquartets, w.nq);
        if (A.nquartets32 && w.nq32) atomicAdd(A.nquartets32, w.nq32);
    }
    unsigned long long npq = w.npq;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) npq += __shfl_down_sync(0xffffffffu, npq, o);
    if (lane == 0 && A.nprimq && npq) atomicAdd(A.nprimq, npq);
}

// ---------------------------------------------------------------------------
// team form
// ---------------------------------------------------------------------------
template <class C>
__device__ __forceinline__ void team_sync(int team)
{
    if constexpr (C::TEAM == 16) {
        __syncwarp(0xFFFFu << (16 * (team & 1)));
    } else if constexpr (C::TEAM == 32) {
        __syncwarp();
    } else {
        asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "r"(C::TEAM) : "memory");
    }
}

// Shared-memory layout of one team (doubles): Rys roots/weights, the 2D
// integrals of one primitive quartet, the bra-transferred block H[ij][f],
// and one region that holds first (e0|f0) and then (ij|kl).  The rows of those
// blocks have an odd length: lanes that take a row each (the accumulators'
// store, the J contraction over e, the ket transfer) are otherwise a multiple
// of NF or NKL doubles apart, all on a few banks ((fp|dp): 165 of 310 million
// shared wavefronts were conflicts, the data path at 86%).  Builds:
// (H2O)_13 def2-TZVP UHF 44.2 -> 42.8 ms, (H2O)_96 6-31G* UHF 233.5 -> 228.6.
template <class C>
struct TeamLayout {
    static constexpr int GW = C::LKL + 1;
    static constexpr int GSZ = ((C::LIJ + 1) * GW) | 1;   // odd: the lanes that write a table each
    static constexpr int NIJ = C::NI * C::NJ;
    static constexpr int NKL = C::NK * C::NL;
    static constexpr int SF = C::NF | 1;     // row of the (e0|f0) and H[ij][f] blocks
    static constexpr int SQ = NKL | 1;       // row of the (ij|kl) block
    static constexpr int RW = 0;
    static constexpr int G = 2 * C::NROOTS;
    static constexpr int H = G + C::NROOTS * 3 * GSZ;
    static constexpr int E = H + NIJ * SF;
    static constexpr int ESZ = C::NE * SF > NIJ * SQ ? C::NE * SF : NIJ * SQ;
    static constexpr int SIZE = ((E + ESZ) + 1) & ~1;
};

// sum over (a, b), a < NA, b < NB, of g[a GA + b GB] D[a da + b db], D in global
// memory: the loop over a stays a loop.  The steps are run-time values (the
// plan's AO order), so the unrolled loops formed a 64-bit address per element
// and held them all: up to 3 KB of spills per thread in teams of up to 32 lanes,
// 4 to 18 KB in larger ones and 40 in (ff|ff), where none, up to 1.3 KB and 6.5
// are left ((ff|fd) of batches 2.4).  (H2O)_8 def2-TZVP with three
// non-symmetric densities 50.6 -> 36.2 ms, eight symmetric ones of (H2O)_6
// 21.4 -> 15.7, a mixed batch of 16 clusters of up to six 73.7 -> 62.9.
template <int NA, int NB, int GA, int GB>
__device__ __forceinline__ double block_dot(const double *g, const double *__restrict__ D, size_t da, int db)
{
    double s = 0.;
#pragma unroll 1
    for (int a = 0; a < NA; ++a) {
#pragma unroll
        for (int b = 0; b < NB; ++b) s = fma(g[a * GA + b * GB], __ldg(D + b * db), s);
        D += da;
    }
    return s;
}

// digestion of a quartet held in shared memory, g[(i*NJ + j)*SQ + k*NL + l],
// spread over the lanes of a team: one atomic per J/K element per quartet
template <class C>
__device__ __forceinline__ void digest_shared(const PlanView &V, const double *g,
                                              int i0, int j0, int k0, int l0, int tl, bool doJ,
                                              bool doK)
{
    constexpr int NI = C::NI, NJ = C::NJ, NK = C::NK, NL = C::NL, NKL = NK * NL;
    constexpr int SQ = TeamLayout<C>::SQ, SI = NJ * SQ;
    const AoIndex<C> ax(V);
    const size_t nao2 = ax.nao * ax.nao;
    for (int d = 0; d < (doJ ? V.n_j : 0); ++d) {
        const double *ds = V.dsJ + d * nao2;
        double *jh = V.Jh + d * nao2;
        for (int o = tl; o < NKL + NI * NJ; o += C::TEAM) {
            if (o < NKL) {
                const int k = o / NL, l = o - (o / NL) * NL;
                atomicAdd(jh + ax(k0, k, ax.kn, l0, l, ax.l),
                          block_dot<NI, NJ, SI, SQ>(g + o, ds + ax(i0, 0, 0, j0, 0, 0), ax.in, ax.j));
            } else {
                const int ij = o - NKL, i = ij / NJ, j = ij - (ij / NJ) * NJ;
                atomicAdd(jh + ax(i0, i, ax.in, j0, j, ax.j),
                          block_dot<NK, NL, NL, 1>(g + ij * SQ, ds + ax(k0, 0, 0, l0, 0, 0), ax.kn, ax.l));
            }
        }
    }
    constexpr int N1 = NI * NK, N2 = NI * NL, N3 = NJ * NK, N4 = NJ * NL;
    for (int d = 0; d < (doK ? V.n_k : 0); ++d) {
        const double *D = kdens(V, d, nao2);
        double *kh = V.Kh + d * nao2;
        for (int o = tl; o < N1 + N2 + N3 + N4; o += C::TEAM) {
            if (o < N1) {              // K_h[i,k] += sum_jl g D[j,l]
                const int i = o / NK, k = o - (o / NK) * NK;
                atomicAdd(kh + ax(i0, i, ax.in, k0, k, ax.k),
                          block_dot<NJ, NL, SQ, 1>(g + i * SI + k * NL, D + ax(j0, 0, 0, l0, 0, 0), ax.jn, ax.l));
            } else if (o < N1 + N2) {  // K_h[i,l] += sum_jk g D[j,k]
                const int t = o - N1, i = t / NL, l = t - (t / NL) * NL;
                atomicAdd(kh + ax(i0, i, ax.in, l0, l, ax.l),
                          block_dot<NJ, NK, SQ, NL>(g + i * SI + l, D + ax(j0, 0, 0, k0, 0, 0), ax.jn, ax.k));
            } else if (o < N1 + N2 + N3) {  // K_h[j,k] += sum_il g D[i,l]
                const int t = o - N1 - N2, j = t / NK, k = t - (t / NK) * NK;
                atomicAdd(kh + ax(j0, j, ax.jn, k0, k, ax.k),
                          block_dot<NI, NL, SI, 1>(g + j * SQ + k * NL, D + ax(i0, 0, 0, l0, 0, 0), ax.in, ax.l));
            } else {                   // K_h[j,l] += sum_ik g D[i,k]
                const int t = o - N1 - N2 - N3, j = t / NL, l = t - (t / NL) * NL;
                atomicAdd(kh + ax(j0, j, ax.jn, l0, l, ax.l),
                          block_dot<NI, NK, SI, NL>(g + j * SQ + l, D + ax(i0, 0, 0, k0, 0, 0), ax.in, ax.k));
            }
        }
    }
}

// The team form's K digest from density blocks the team stages in shared
// memory once per quartet (the digest reads each element NJ NL to NI NK
// times): per density d at st + d * k_stage_doubles, D[i,k] (NI x NK),
// D[i,l] (NI x NL), D[j,k] (NJ x NK), D[j,l] (NJ x NL)
template <class C>
constexpr int k_stage_doubles()
{
    return (C::NI + C::NJ) * (C::NK + C::NL);
}

template <class C>
__device__ __forceinline__ void k_stage(const PlanView &V, double *st, int i0, int j0, int k0,
                                        int l0, int tl)
{
    constexpr int NI = C::NI, NJ = C::NJ, NK = C::NK, NL = C::NL, KST = k_stage_doubles<C>();
    const AoIndex<C> ax(V);
    const size_t nao2 = ax.nao * ax.nao;
    for (int t = tl; t < V.n_k * KST; t += C::TEAM) {
        const int d = t / KST;
        int r = t - d * KST, row, col;
        if (r < NI * NK) {
            row = i0 + r / NK * ao_step<C::LI>(V);
            col = k0 + r % NK * ax.k;
        } else if ((r -= NI * NK) < NI * NL) {
            row = i0 + r / NL * ao_step<C::LI>(V);
            col = l0 + r % NL * ax.l;
        } else if ((r -= NI * NL) < NJ * NK) {
            row = j0 + r / NK * ax.j;
            col = k0 + r % NK * ax.k;
        } else {
            r -= NJ * NK;
            row = j0 + r / NL * ax.j;
            col = l0 + r % NL * ax.l;
        }
        st[t] = __ldg(kdens(V, d, nao2) + (size_t)row * ax.nao + col);
    }
}

template <class C>
__device__ __forceinline__ void digest_k_staged(const PlanView &V, const double *g,
                                                const double *st, int i0, int j0, int k0, int l0,
                                                int tl)
{
    constexpr int NI = C::NI, NJ = C::NJ, NK = C::NK, NL = C::NL, NKL = NK * NL;
    constexpr int SQ = TeamLayout<C>::SQ;
    constexpr int KST = k_stage_doubles<C>();
    constexpr int N1 = NI * NK, N2 = NI * NL, N3 = NJ * NK, N4 = NJ * NL;
    const AoIndex<C> ax(V);
    const size_t nao2 = ax.nao * ax.nao;
    for (int d = 0; d < V.n_k; ++d) {
        const double *Dik = st + d * KST, *Dil = Dik + N1, *Djk = Dil + N2, *Djl = Djk + N3;
        double *kh = V.Kh + d * nao2;
        for (int o = tl; o < N1 + N2 + N3 + N4; o += C::TEAM) {
            double s = 0.;
            if (o < N1) {              // K_h[i,k] += sum_jl g D[j,l]
                const int i = o / NK, k = o - (o / NK) * NK;
#pragma unroll
                for (int j = 0; j < NJ; ++j)
#pragma unroll
                    for (int l = 0; l < NL; ++l)
                        s = fma(g[(i * NJ + j) * SQ + k * NL + l], Djl[j * NL + l], s);
                atomicAdd(kh + ax(i0, i, ax.in, k0, k, ax.k), s);
            } else if (o < N1 + N2) {  // K_h[i,l] += sum_jk g D[j,k]
                const int t = o - N1, i = t / NL, l = t - (t / NL) * NL;
#pragma unroll
                for (int j = 0; j < NJ; ++j)
#pragma unroll
                    for (int k = 0; k < NK; ++k)
                        s = fma(g[(i * NJ + j) * SQ + k * NL + l], Djk[j * NK + k], s);
                atomicAdd(kh + ax(i0, i, ax.in, l0, l, ax.l), s);
            } else if (o < N1 + N2 + N3) {  // K_h[j,k] += sum_il g D[i,l]
                const int t = o - N1 - N2, j = t / NK, k = t - (t / NK) * NK;
#pragma unroll
                for (int i = 0; i < NI; ++i)
#pragma unroll
                    for (int l = 0; l < NL; ++l)
                        s = fma(g[(i * NJ + j) * SQ + k * NL + l], Dil[i * NL + l], s);
                atomicAdd(kh + ax(j0, j, ax.jn, k0, k, ax.k), s);
            } else {                   // K_h[j,l] += sum_ik g D[i,k]
                const int t = o - N1 - N2 - N3, j = t / NL, l = t - (t / NL) * NL;
#pragma unroll
                for (int i = 0; i < NI; ++i)
#pragma unroll
                    for (int k = 0; k < NK; ++k)
                        s = fma(g[(i * NJ + j) * SQ + k * NL + l], Dik[i * NK + k], s);
                atomicAdd(kh + ax(j0, j, ax.jn, l0, l, ax.l), s);
            }
        }
    }
}

// 2D integrals G[e][f] of one dimension and root into shared memory
template <class C, class T>
__device__ __forceinline__ void vrr_chain(T c0, T cp, T b00, T b10, T b01, T g00, T *G)
{
    constexpr int LIJ = C::LIJ, LKL = C::LKL, W = LKL + 1;
    T cur[LIJ + 1], prev[LIJ + 1];
    cur[0] = g00;
    if (LIJ > 0) cur[1] = c0 * g00;
#pragma unroll
    for (int e = 1; e < LIJ; ++e) cur[e + 1] = fma(T(e) * b10, cur[e - 1], c0 * cur[e]);
#pragma unroll
    for (int e = 0; e <= LIJ; ++e) { G[e * W] = cur[e]; prev[e] = T(0); }
#pragma unroll
    for (int f = 0; f < LKL; ++f) {
        T nxt[LIJ + 1];
#pragma unroll
        for (int e = 0; e <= LIJ; ++e) {
            T v = cp * cur[e];
            if (f > 0) v = fma(T(f) * b01, prev[e], v);
            if (e > 0) v = fma(T(e) * b00, cur[e - 1], v);
            nxt[e] = v;
        }
#pragma unroll
        for (int e = 0; e <= LIJ; ++e) {
            G[e * W + f + 1] = nxt[e];
            prev[e] = cur[e];
            cur[e] = nxt[e];
        }
    }
}

// T: the arithmetic of the 2D integrals and the (e0|f0) accumulation (float
// for the mixed form's low-bound quartets); the Rys roots and weights, the
// transfers and the digest stay FP64
template <class C, int P, class T>
__device__ __forceinline__ void team_quartet_part(const ClassArgs &A, const PlanView &V,
                                                  const PairRec &br,
                                                  const double *__restrict__ sbra, int entry,
                                                  double sym, double *ts, int tl, int team)
{
    const int kk = entry & JK_Q_KET;
    using L = TeamLayout<C>;
    constexpr int N = C::NROOTS, NE = C::NE, NF = C::NF, W = L::GW;
    constexpr int F0 = C::template fbegin<P>(), F1 = C::template fend<P>(), NFP = F1 - F0;
    double *rw = ts + L::RW;
    T *G = reinterpret_cast<T *>(ts + L::G);
    double *E = ts + L::E;
    double *H = ts + L::H;
    const int el = tl % C::TEAM_LANES;
    const bool act = el < NE;
    const int ex = act ? C::ex(el) : 0, ey = act ? C::ey(el) : 0, ez = act ? C::ez(el) : 0;
    const PairRec kt = V.ket[kk];
    T acc[NFP];
#pragma unroll
    for (int f = 0; f < NFP; ++f) acc[f] = T(0);
    const double *kprim = V.prim + (size_t)kt.prim0 * JK_PRIM_STRIDE;
    for (int t = 0; t < A.nterm; ++t) {   // operator terms, as in reg_quartet
        const double io2 = A.op_inv_om2[t], ct = A.op_coef[t];
        for (int kp = 0; kp < kt.nprim; ++kp) {
            const double *kr = kprim + kp * JK_PRIM_STRIDE;
            const double akl = __ldg(kr + PR_A), hiq = __ldg(kr + PR_HIA);
            const double kq = __ldg(kr + PR_KP) * ct;
            for (int bp = 0; bp < br.nprim; ++bp) {
                const double *s = sbra + bp * JK_PRIM_STRIDE;
                const double aij = s[PR_A], hip = s[PR_HIA];
                const double PQ[3] = {s[PR_PX] - __ldg(kr + PR_PX),
                                      s[PR_PX + 1] - __ldg(kr + PR_PX + 1),
                                      s[PR_PX + 2] - __ldg(kr + PR_PX + 2)};
                const double rs = rsqrt(fma(aij * akl, io2, aij + akl));
                const double is = rs * rs;
                const double rr = PQ[0] * PQ[0] + PQ[1] * PQ[1] + PQ[2] * PQ[2];
                const double x = aij * akl * is * rr;
                if (tl < 2 * N) rw[tl] = rys_row<N>(x, A.rys, tl);
                team_sync<C>(team);
                if (tl < 3 * N) {
                    const int r = tl / 3, d = tl - 3 * (tl / 3);
                    const double uis = rw[r] * is;
                    const double up = uis * akl, uq = uis * aij;
                    const double g00 = d == 2 ? rw[N + r] * s[PR_KP] * kq * rs : 1.0;
                    vrr_chain<C, T>(T(fma(-up, PQ[d], s[PR_PAX + d])),
                                    T(fma(uq, PQ[d], __ldg(kr + PR_PAX + d))), T(0.5 * uis),
                                    T(fma(-hip, up, hip)), T(fma(-hiq, uq, hiq)), T(g00),
                                    G + (r * 3 + d) * L::GSZ);
                }
                team_sync<C>(team);
                if (act) {
#pragma unroll
                    for (int r = 0; r < N; ++r) {
                        T gx[W], gy[W], gz[W];
                        const T *px = G + (r * 3 + 0) * L::GSZ + ex * W;
                        const T *py = G + (r * 3 + 1) * L::GSZ + ey * W;
                        const T *pz = G + (r * 3 + 2) * L::GSZ + ez * W;
#pragma unroll
                        for (int f = 0; f < W; ++f) { gx[f] = px[f]; gy[f] = py[f]; gz[f] = pz[f]; }
                        C::template row_acc<P, T>(gx, gy, gz, acc);
                    }
                }
                team_sync<C>(team);
            }
        }
    }
    constexpr int SF = L::SF;
    const double fac = kt.ish == kt.jsh ? 0.5 * sym : sym;
    if (act) {
#pragma unroll
        for (int f = 0; f < NFP; ++f) E[el * SF + F0 + f] = double(acc[f]) * fac;
    }
    team_sync<C>(team);
    if (A.jx) {   // J engine: J from the block E = (e0|f0) fac and the x-space densities
        if (!(entry & JK_Q_NOJ)) {
            const int n_j = V.n_j;
            const size_t xb = (size_t)br.xoff * n_j, xk = (size_t)kt.xoff * n_j;
            for (int d = 0; d < n_j; ++d) {
                const double *db = A.jx_dens + xb + d * NE, *dk = A.jx_dens + xk + d * NF;
                for (int f = tl; f < NF; f += C::TEAM) {
                    double s = 0.;
                    for (int e = 0; e < NE; ++e) s = fma(E[e * SF + f], __ldg(db + e), s);
                    atomicAdd(A.jx_acc + xk + d * NF + f, s);
                }
                for (int e = tl; e < NE; e += C::TEAM) {
                    double s = 0.;
                    for (int f = 0; f < NF; ++f) s = fma(E[e * SF + f], __ldg(dk + f), s);
                    atomicAdd(A.jx_acc + xb + d * NE + e, s);
                }
            }
        }
        team_sync<C>(team);   // E is read above and overwritten by the transfers
        if (V.n_k == 0 || (entry & JK_Q_NOK)) return;   // nothing for K: no transfers
    }
    constexpr int NIJ = C::NI * C::NJ, SQ = L::SQ;
    // bra transfer of each f column, read from and written to shared memory
    for (int f = tl; f < NF; f += C::TEAM)
        C::template hrr_bra<double, SF, SF>(E + f, H + f, br.ABx, br.ABy, br.ABz);
    team_sync<C>(team);
    double *Gq = E;   // (ij|kl) of the quartet; E is dead once H is complete
    for (int ij = tl; ij < NIJ; ij += C::TEAM)
        C::template hrr_ket<double>(H + ij * SF, Gq + ij * SQ, kt.ABx, kt.ABy, kt.ABz);
    team_sync<C>(team);
    const bool doJ = !A.jx && !(entry & JK_Q_NOJ), doK = !(entry & JK_Q_NOK);
    if (doK && V.n_k * k_stage_doubles<C>() <= NIJ * SF) {
        // K from density blocks staged where the bra-transferred block was
        k_stage<C>(V, H, br.i0, br.j0, kt.i0, kt.j0, tl);
        team_sync<C>(team);
        if (doJ) digest_shared<C>(V, Gq, br.i0, br.j0, kt.i0, kt.j0, tl, true, false);
        digest_k_staged<C>(V, Gq, H, br.i0, br.j0, kt.i0, kt.j0, tl);
    } else {
        digest_shared<C>(V, Gq, br.i0, br.j0, kt.i0, kt.j0, tl, doJ, doK);
    }
    team_sync<C>(team);
}

template <class C, int P, class T>
__device__ __forceinline__ void team_quartet(const ClassArgs &A, const PlanView &V,
                                             const PairRec &br, const double *sbra, int kk,
                                             double sym, double *ts, int tl, int team)
{
    if (tl / C::TEAM_LANES == P) {
        team_quartet_part<C, P, T>(A, V, br, sbra, kk, sym, ts, tl, team);
    } else if constexpr (P + 1 < C::NWF) {
        team_quartet<C, P + 1, T>(A, V, br, sbra, kk, sym, ts, tl, team);
    }
}

// one quartet of the team: FP32 2D integrals and accumulation when the build
// is mixed and the quartet's screened bound is below the threshold (true)
template <class C>
__device__ __forceinline__ bool team_one(const ClassArgs &A, const PlanView &V, const PairRec &br,
                                         const double *sbra, int e2, double sym, double *ts,
                                         int tl, int team)
{
    if (A.mixed && (e2 & JK_Q_LOW)) {
        team_quartet<C, 0, float>(A, V, br, sbra, e2, sym, ts, tl, team);
        return true;
    }
    team_quartet<C, 0, double>(A, V, br, sbra, e2, sym, ts, tl, team);
    return false;
}

template <class C>
constexpr int team_min_blocks()
{
    // (teams of 64 lanes and more at 3 and 2 lose 0.5 to 6% on def2-TZVP: (H2O)_5
    // four non-symmetric densities 11.4 -> 12.0 ms, a batch of 40 clusters of up
    // to two 7.1 -> 7.4, (H2O)_13 UHF 42.3 -> 42.6; smaller teams at 5 cost
    // (H2O)_2 def2-SVP 6% and stay at 3)
    return C::TEAM <= 32 ? 3 : (C::TEAM <= 64 ? 4 : 3);
}

// one task of the team form (all threads of the block)
template <class C, int NT>
__device__ __forceinline__ void team_task(const ClassArgs &A, const PlanView &V, int v, int b,
                                          int k_begin, int k_end, double *sbra, double *ts,
                                          int *s_queue, int *s_wcnt, unsigned int &s_count,
                                          int &staged_v, int &staged_b, unsigned long long &my_pq,
                                          unsigned long long &my_q32)
{
    constexpr int TEAM = C::TEAM;
    constexpr int NTEAMS = NT / TEAM;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int team = tid / TEAM, tl = tid % TEAM;
    const PairRec br = V.bra[b];
    if (b != staged_b || v != staged_v) {
        const double *src = V.prim + (size_t)br.prim0 * JK_PRIM_STRIDE;
        for (int t = tid; t < br.nprim * JK_PRIM_STRIDE; t += NT) sbra[t] = src[t];
        staged_b = b;
        staged_v = v;
    }
    __syncthreads();
    const double sym_b = br.ish == br.jsh ? 0.5 : 1.0;
    const bool diag = V.bra == V.ket;
    const float log_mixed = A.mixed ? A.mixed_log_thr : JK_NEG_INF;
    int nq = 0;
    for (int base = k_begin; base < k_end; base += NT) {
        const int kk = base + tid;
        float bK = JK_NEG_INF, bJ = JK_NEG_INF;
        if (kk < k_end) quartet_bounds(V, br, kk, bK, bJ);
        const bool keep = fmaxf(bK, bJ) > V.log_tol;
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) s_wcnt[warp] = __popc(m);
        __syncthreads();
        int off = nq, tot = 0;
#pragma unroll
        for (int w = 0; w < NT / 32; ++w) {
            const int c = s_wcnt[w];
            if (w < warp) off += c;
            tot += c;
        }
        if (keep)
            s_queue[off + __popc(m & ((1u << lane) - 1u))] =
                queue_entry(kk, bK, bJ, V.log_tol) | (fmaxf(bK, bJ) < log_mixed ? JK_Q_LOW : 0);
        nq += tot;
        __syncthreads();
        const int nproc = (nq / NTEAMS) * NTEAMS;
        if (nproc > 0) {
            for (int t = team; t < nproc; t += NTEAMS) {
                const int e2 = s_queue[t], k2 = e2 & JK_Q_KET;
                const bool f32 = team_one<C>(A, V, br, sbra, e2, diag && k2 == b ? 0.5 * sym_b : sym_b,
                                             ts, tl, team);
                if (tl == 0) {
                    my_pq += (unsigned long long)br.nprim * V.ket[k2].nprim;
                    my_q32 += f32;
                }
            }
            if (tid == 0) s_count += nproc;
            __syncthreads();
            const int rem = nq - nproc;
            int tmp = 0;
            if (tid < rem) tmp = s_queue[nproc + tid];
            __syncthreads();
            if (tid < rem) s_queue[tid] = tmp;
            __syncthreads();
            nq = rem;
        }
    }
    if (nq > 0) {
        for (int t = team; t < nq; t += NTEAMS) {
            const int e2 = s_queue[t], k2 = e2 & JK_Q_KET;
            const bool f32 = team_one<C>(A, V, br, sbra, e2, diag && k2 == b ? 0.5 * sym_b : sym_b, ts,
                                         tl, team);
            if (tl == 0) {
                my_pq += (unsigned long long)br.nprim * V.ket[k2].nprim;
                my_q32 += f32;
            }
        }
        if (tid == 0) s_count += nq;
    }
    __syncthreads();
}

// Teams of up to a warp: every warp claims its own tasks and queues its own
// quartets, as in the register form (two teams of 16 lanes take every other
// quartet of the warp's queue), and no warp waits for another.  With block
// tasks the four warps of a block met three times per 128 candidates, often
// with a quartet or two each in between.
template <class C, int NT, int NV>
__device__ __forceinline__ void team_warp_tasks(const LaunchParams<NV> &P, int t_begin, int t_end,
                                                double *smem, int *q)
{
    const ClassArgs &A = P.a;
    constexpr int NW = NT / 32, TPW = 32 / C::TEAM;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tl = tid % C::TEAM;
    const int sub = lane / C::TEAM;
    double *sbra = smem + warp * A.max_bra_prim * JK_PRIM_STRIDE;
    double *ts = smem + NW * A.max_bra_prim * JK_PRIM_STRIDE + (tid / C::TEAM) * TeamLayout<C>::SIZE;
    unsigned long long my_q = 0, my_pq = 0, my_q32 = 0;
    const int chunk = *A.chunk;
    Task task;
    while (claim_task(P, t_begin, t_end, chunk, task)) {
        const PlanView &V = P.v[task.view];
        const int b = task.bra;
        const PairRec br = V.bra[b];
        const double *src = V.prim + (size_t)br.prim0 * JK_PRIM_STRIDE;
        for (int t = lane; t < br.nprim * JK_PRIM_STRIDE; t += 32) sbra[t] = src[t];
        __syncwarp();
        const double sym_b = br.ish == br.jsh ? 0.5 : 1.0;
        const bool diag = V.bra == V.ket;
        auto batch = [&](const int *src, int n, auto) {
            for (int t = sub; t < n; t += TPW) {
                const int e2 = src[t], k2 = e2 & JK_Q_KET;
                const bool f32 = team_one<C>(A, V, br, sbra, e2, diag && k2 == b ? 0.5 * sym_b : sym_b,
                                             ts, tl, tid / C::TEAM);
                if (tl == 0) {
                    my_q++;
                    my_pq += (unsigned long long)br.nprim * V.ket[k2].nprim;
                    my_q32 += f32;
                }
            }
            __syncwarp();
        };
        ket_batches<true>(V, br, task.k0, task.k1, q, lane, V.log_tol,
                          A.mixed ? A.mixed_log_thr : JK_NEG_INF, batch);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        my_q += __shfl_down_sync(0xffffffffu, my_q, o);
        my_pq += __shfl_down_sync(0xffffffffu, my_pq, o);
        my_q32 += __shfl_down_sync(0xffffffffu, my_q32, o);
    }
    if (lane == 0 && my_q) {
        if (A.nquartets) atomicAdd(A.nquartets, my_q);
        if (A.nprimq) atomicAdd(A.nprimq, my_pq);
        if (A.nquartets32 && my_q32) atomicAdd(A.nquartets32, my_q32);
    }
}

// team-form kernel: tasks of a warp (teams of up to 32 lanes) or of a block
// (larger teams), one quartet per team at a time.  Quartets of the mixed
// form's low-bound set take FP32 2D integrals and accumulation (team_one).
template <class C, int NT, int NV>
__global__ void __launch_bounds__(NT, team_min_blocks<C>())
    jk_team_kernel(const __grid_constant__ LaunchParams<NV> P)
{
    const ClassArgs &A = P.a;
    extern __shared__ double smem[];
    if constexpr (C::TEAM <= 32) {
        __shared__ int s_q[NT / 32][64];
        int t_begin, t_end;
        launch_tasks(A, t_begin, t_end);
        if ((int)blockIdx.x >= t_end - t_begin) return;
        team_warp_tasks<C, NT, NV>(P, t_begin, t_end, smem, s_q[threadIdx.x >> 5]);
        return;
    }
    __shared__ int s_queue[2 * NT];
    __shared__ int s_wcnt[NT / 32];
    __shared__ int s_task[5];          // view, bra, ket begin, ket end, valid
    __shared__ unsigned int s_count;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int team = tid / C::TEAM;
    double *sbra = smem;
    double *ts = smem + A.max_bra_prim * JK_PRIM_STRIDE + team * TeamLayout<C>::SIZE;
    int t_begin, t_end;
    launch_tasks(A, t_begin, t_end);
    if ((int)blockIdx.x >= t_end - t_begin) return;
    if (tid == 0) s_count = 0;
    unsigned long long my_pq = 0, my_q32 = 0;
    int staged_v = -1, staged_b = -1;
    const int chunk = *A.chunk;
    for (;;) {
        if (warp == 0) {
            Task task;
            const bool ok = claim_task(P, t_begin, t_end, chunk, task);
            if (lane == 0) {
                s_task[0] = task.view;
                s_task[1] = task.bra;
                s_task[2] = task.k0;
                s_task[3] = task.k1;
                s_task[4] = ok;
            }
        }
        __syncthreads();
        if (!s_task[4]) break;
        const int v = s_task[0], b = s_task[1], k_begin = s_task[2], k_end = s_task[3];
        team_task<C, NT>(A, P.v[v], v, b, k_begin, k_end, sbra, ts, s_queue, s_wcnt, s_count, staged_v,
                         staged_b, my_pq, my_q32);
    }
    if (tid == 0 && A.nquartets) atomicAdd(A.nquartets, (unsigned long long)s_count);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        my_pq += __shfl_down_sync(0xffffffffu, my_pq, o);
        my_q32 += __shfl_down_sync(0xffffffffu, my_q32, o);
    }
    if (lane == 0 && A.nprimq && my_pq) atomicAdd(A.nprimq, my_pq);
    if (lane == 0 && A.nquartets32 && my_q32) atomicAdd(A.nquartets32, my_q32);
}

// ---------------------------------------------------------------------------
// host launcher of one class
// ---------------------------------------------------------------------------
// Per kernel and device: the largest dynamic shared memory opted into so far
// (the attribute only grows, so a captured graph that launches with an
// earlier, smaller size stays valid), and the occupancy at the size last
// queried.
struct KernelState {
    size_t shm_set[JK_MAX_DEVICES];
    size_t shm_occ[JK_MAX_DEVICES];
    int blocks[JK_MAX_DEVICES];
};

template <class K>
static int configure(K kern, int nt, size_t shm, KernelState &ks, const LaunchCfg &cfg,
                     const char *tag, int &blocks_per_sm)
{
    const int dev = cfg.device;
    if (dev < 0 || dev >= JK_MAX_DEVICES) return (int)cudaErrorInvalidDevice;
    if (ks.blocks[dev] > 0 && ks.shm_occ[dev] == shm) {
        blocks_per_sm = ks.blocks[dev];
        return 0;
    }
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, kern);
    // the default dynamic limit is 48 KB minus the static shared memory,
    // so the opt-in is set for every size
    if (e == cudaSuccess && (shm > ks.shm_set[dev] || ks.blocks[dev] == 0)) {
        const size_t want = shm > ks.shm_set[dev] ? shm : ks.shm_set[dev];
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)want);
        if (e == cudaSuccess) ks.shm_set[dev] = want;
    }
    int nb = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, nt, shm);
    if (e != cudaSuccess || nb <= 0) {
        if (cfg.msg)
            snprintf(cfg.msg, 256,
                     "class %s: %s (threads %d, dynamic shared %zu B, static shared %zu B, "
                     "registers %d, max threads %d, blocks/SM %d)",
                     tag, cudaGetErrorString(e), nt, shm, (size_t)fa.sharedSizeBytes, fa.numRegs,
                     fa.maxThreadsPerBlock, nb);
        cudaGetLastError();
        return e != cudaSuccess ? (int)e : (int)cudaErrorInvalidConfiguration;
    }
    ks.blocks[dev] = nb;
    ks.shm_occ[dev] = shm;
    blocks_per_sm = nb;
    return 0;
}

// shared memory of the register form, FP32 records and tables not counted
template <class C, int JX>
static size_t reg_shm(const ClassArgs &a)
{
    const int hermite = JX == 3 ? JK_MD_DENS * md_nt(C::LI + C::LJ) : 0;   // per bra primitive
    return (rys_smem_doubles<C, JX>() +
            (size_t)(reg_threads<C>() / 32) * a.max_bra_prim * (JK_PRIM_STRIDE + hermite)) * sizeof(double);
}

// TEAMF: the team form (of a class that may also have the register form)
template <class C, int NV, int OP, int JX = 0, bool TEAMF = !C::REG>
static int launch_nv(const ClassArgs &a, const PlanView *views, const LaunchCfg &cfg, const char *tag,
                     KernelState &ks)
{
    static LaunchParams<NV> prm;     // host staging of the parameters (launches are serialised)
    prm.a = a;
    for (int i = 0; i < a.nvl && i < NV; ++i) prm.v[i] = views[i];
    int nt = 0, grid = 0, bps = 0;
    size_t shm = 0;
    if constexpr (!TEAMF) {
        constexpr int NT = reg_threads<C>();
        auto kern = jk_reg_kernel<C, NT, NV, OP, JX>;
        shm = reg_shm<C, JX>(a);
        if constexpr (JX == 3) prm.a.mixed = 0;
        prm.a.mixed_tab = 0;
        if (prm.a.mixed) {
            // the FP32 bra records, and the FP32 Rys table when the class keeps
            // its tables in shared memory, only where they leave the
            // occupancy of the FP64 form; otherwise the table is read from
            // global memory, or the launch runs every quartet in FP64
            int b64 = 0;
            int rc = configure(kern, NT, shm, ks, cfg, tag, b64);
            if (rc) return rc;
            const size_t s32 = shm + (size_t)(NT / 32) * a.max_bra_prim * JK_PRIM32_STRIDE * sizeof(float);
            const size_t t32 = (size_t)rys32_smem_doubles<C>(1) * sizeof(double);
            int b = 0;
            if (t32 && configure(kern, NT, s32 + t32, ks, cfg, tag, b) == 0 && b >= b64) {
                shm = s32 + t32;
                prm.a.mixed_tab = 1;
            } else if (configure(kern, NT, s32, ks, cfg, tag, b) == 0 && b >= b64) {
                shm = s32;
            } else {
                prm.a.mixed = 0;
            }
        }
        const int rc = configure(kern, NT, shm, ks, cfg, tag, bps);
        if (rc || cfg.configure_only) return rc;
        nt = NT;
        grid = cfg.num_sms * (cfg.blocks_per_sm > 0 && cfg.blocks_per_sm < bps ? cfg.blocks_per_sm : bps);
        kern<<<grid, NT, shm, cfg.stream>>>(prm);
    } else {
        // the block holds a whole number of teams
        constexpr int NT = C::TEAM * ((128 + C::TEAM - 1) / C::TEAM);
        auto kern = jk_team_kernel<C, NT, NV>;
        shm = (size_t)(C::TEAM <= 32 ? NT / 32 : 1) * a.max_bra_prim * JK_PRIM_STRIDE * sizeof(double) +
              (size_t)(NT / C::TEAM) * TeamLayout<C>::SIZE * sizeof(double);
        const int rc = configure(kern, NT, shm, ks, cfg, tag, bps);
        if (rc || cfg.configure_only) return rc;
        nt = NT;
        grid = cfg.num_sms * (cfg.blocks_per_sm > 0 && cfg.blocks_per_sm < bps ? cfg.blocks_per_sm : bps);
        kern<<<grid, NT, shm, cfg.stream>>>(prm);
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess && cfg.msg)
        snprintf(cfg.msg, 256, "class %s: launch of %d x %d threads, %zu B shared: %s", tag, grid,
                 nt, shm, cudaGetErrorString(e));
    return (int)e;
}

#include "jk_grad.cuh"

// One launch of class C over views [a.view_begin, a.view_begin + a.nvl)
// (views: host copies of those views); grid num_sms x (resident blocks per
// SM, capped by cfg.blocks_per_sm > 0).
template <class C>
int jk_launch_class(const ClassArgs &a, const PlanView *views, const LaunchCfg &cfg, const char *tag)
{
    // single-view, batched, single-view two-term and J-engine kernels (the
    // team form loops over the terms and takes the J engine at run time: its
    // kernels serve all)
    static KernelState ks[9];
    if (a.nvl < 1 || a.nvl > JK_VTAB || a.nterm < 1 || a.nterm > 2) return (int)cudaErrorInvalidValue;
    if (a.grad) {
        if (a.nvl != 1 || a.nterm != 1) {
            if (cfg.msg) snprintf(cfg.msg, 256, "class %s: gradients take one view, one term", tag);
            return (int)cudaErrorInvalidValue;
        }
        return launch_grad<C>(a, views, cfg, tag, ks[5]);
    }
    if constexpr (C::NPASS > 1) {
        if (a.team) {
            if (a.nvl == 1) return launch_nv<C, 1, 1, 0, true>(a, views, cfg, tag, ks[7]);
            return launch_nv<C, JK_VTAB, 1, 0, true>(a, views, cfg, tag, ks[8]);
        }
    }
    if constexpr (C::REG) {
        if (a.jx) {
            if (a.nvl != 1 || a.nterm != 1) {
                if (cfg.msg)
                    snprintf(cfg.msg, 256, "class %s: the J engine takes one view, one term", tag);
                return (int)cudaErrorInvalidValue;
            }
            if (a.jx == 3) {
                if constexpr (md_class<C>()) {
                    // the bra's Hermite densities of many primitives may not fit
                    // ((pp|pp): about 99 primitive pairs, (ff|ss): 16): the Rys J
                    // engine, whose x-space densities every such build has
                    int most = 0;
                    const cudaError_t e =
                        cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, cfg.device);
                    if (e != cudaSuccess) return (int)e;
                    const size_t queue = reg_threads<C>() / 32 * 64 * sizeof(int);
                    if (reg_shm<C, 3>(a) + queue > (size_t)most)
                        return launch_nv<C, 1, 1, 2>(a, views, cfg, tag, ks[4]);
                    return launch_nv<C, 1, 1, 3>(a, views, cfg, tag, ks[6]);
                }
                if (cfg.msg) snprintf(cfg.msg, 256, "class %s: no McMurchie-Davidson J kernel", tag);
                return (int)cudaErrorInvalidValue;
            }
            if (a.jx == 2) return launch_nv<C, 1, 1, 2>(a, views, cfg, tag, ks[4]);
            return launch_nv<C, 1, 1, 1>(a, views, cfg, tag, ks[3]);
        }
        if (a.nterm == 2) {
            if (a.nvl != 1) {
                if (cfg.msg)
                    snprintf(cfg.msg, 256, "class %s: two-term operators take one view", tag);
                return (int)cudaErrorInvalidValue;
            }
            return launch_nv<C, 1, 2>(a, views, cfg, tag, ks[2]);
        }
    }
    if (a.nvl == 1) return launch_nv<C, 1, 1>(a, views, cfg, tag, ks[0]);
    return launch_nv<C, JK_VTAB, 1>(a, views, cfg, tag, ks[1]);
}

#define JK_DEFINE_CLASS(TAG, A, B)                                                          \
    int jk_launch_##TAG(const ClassArgs &a, const PlanView *views, const LaunchCfg &cfg)      \
    {                                                                                       \
        return jk_launch_class<Cls_##TAG>(a, views, cfg, #TAG);                             \
    }
