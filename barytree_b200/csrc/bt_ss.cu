// bt_ss.cu -- singularity subtraction (SS) kernels of barytree_b200, FP64.
//
// With singularity subtraction every source carries a weight w and every
// target a charge tq, and the potential at target i is
//   phi_i = sum_j (q_j - tq_i g(r)) w_j K(r)  + c * tq_i
// where g is the subtraction factor and c the correction constant:
//   Coulomb (alpha = kernel_params[0]):  K = 1/r, g = exp(-r^2/alpha^2),
//       c = 2 pi alpha^2        (src/kernels/coulomb/coulomb_ss_*.c)
//   Yukawa (kappa = kernel_params[0]):   K = exp(-kappa r)/r, g = 1,
//       c = 4 pi / kappa^2      (src/kernels/yukawa/yukawa_ss_*.c)
//   regularized Coulomb (alpha, eps = kernel_params[0..1]):
//       K = 1/sqrt(r^2+eps^2), g = exp(-r^2/alpha^2), c = 2 pi alpha^2
//       (src/kernels/regularized-coulomb/regularized-coulomb_ss_*.c)
//   regularized Yukawa (kappa, eps): K = exp(-kappa r)/sqrt(r^2+eps^2),
//       g = 1, c = 4 pi / kappa^2, particle-cluster Lagrange only
//       (src/kernels/regularized-yukawa/regularized-yukawa_ss_*.c)
// Source clusters carry two proxy arrays: Q from q*w and W from w (the same
// upward pass applied to both, src/clusters/clusters.c:162-200).  PC uses
// (Q_k - tq W_k g) K; target grids carry two fields, Phi_q from q*w (or Q)
// and Phi_w from g*w (or g*W), which the downward pass combines per target
// as Phi_q - tq Phi_w (interaction_compute_downpass.c:683-800).  Near-field
// pairs with r <= DBL_MIN are skipped for Coulomb and Yukawa; the
// regularized kernel never skips.  CP and CC with SS exist for Coulomb and
// Yukawa with Lagrange only, as in the reference.
#include <cuda_runtime.h>

#include <cfloat>
#include <cmath>
#include <cstdint>

#include "bt_eval64.cuh"
#include "bt_kernels.cuh"
#include "bt_ss.h"

namespace bt {

namespace {

constexpr int SS_THREADS = 128;

// SS near-field pair (PP): target charge tq, source (q, w).
template <int KT>
__device__ __forceinline__ double ss_pp(double dx, double dy, double dz, double q, double w, double tq,
                                        double kp, double kp2)
{
    if (KT == K_COULOMB) {
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        return r > DBL_MIN ? (q - tq * exp(-r * r / (kp * kp))) * w / r : 0.0;
    } else if (KT == K_YUKAWA) {
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        return r > DBL_MIN ? (q - tq) * w * exp(-kp * r) / r : 0.0;
    } else if (KT == K_REGYUKAWA) {
        // regularized-yukawa_ss_pp.c: never skips
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        return (q - tq) * w * exp(-kp * r) / sqrt(r * r + kp2 * kp2);
    } else {
        const double r2 = dx * dx + dy * dy + dz * dz;
        return (q - tq * exp(-r2 / (kp * kp))) * w / sqrt(r2 + kp2 * kp2);
    }
}

// SS particle-cluster term of one Lagrange grid point (Q, W at the point).
template <int KT>
__device__ __forceinline__ double ss_pc(double dx, double dy, double dz, double Qk, double Wk, double tq,
                                        double kp, double kp2)
{
    if (KT == K_COULOMB) {
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        return (Qk - tq * Wk * exp(-r * r / (kp * kp))) / r;
    } else if (KT == K_YUKAWA) {
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        return (Qk - tq * Wk) * exp(-kp * r) / r;
    } else if (KT == K_REGYUKAWA) {
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        return (Qk - tq * Wk) * exp(-kp * r) / sqrt(r * r + kp2 * kp2);
    } else {
        const double r2 = dx * dx + dy * dy + dz * dz;
        return (Qk - tq * Wk * exp(-r2 / (kp * kp))) / sqrt(r2 + kp2 * kp2);
    }
}

// SS Hermite particle-cluster term: Q part as the skipping kernel, W part
// weighted by the subtraction factor (coulomb_ss_pc.c:66-166,
// yukawa_ss_pc.c:70-170, regularized-coulomb_ss_pc.c:66-166).  Q, W point
// at moment 0 of the grid point, moments P apart.
template <int KT>
__device__ __forceinline__ double ss_pc_herm(double dx, double dy, double dz, const double *Q, const double *W,
                                             int P, double tq, double kp, double kp2)
{
    if (KT == K_YUKAWA) {
        double d[8];
        for (int m = 0; m < 8; m++) d[m] = Q[m * P] - W[m * P] * tq;
        return k_pc_herm<K_YUKAWA>(dx, dy, dz, d, 1, kp);
    }
    const double eps2 = KT == K_REGCOULOMB ? kp2 * kp2 : 0.0;
    const double q_part = KT == K_REGCOULOMB ? k_pc_herm<K_REGCOULOMB>(dx, dy, dz, Q, P, kp2)
                                             : k_pc_herm<K_COULOMB>(dx, dy, dz, Q, P, kp);
    const double r = sqrt(dx * dx + dy * dy + dz * dz + eps2);
    const double r2 = r * r, rinv = 1.0 / r, r3inv = rinv * rinv * rinv, r5inv = r3inv * rinv * rinv,
                 r7inv = r5inv * rinv * rinv;
    const double a2 = r2 / (kp * kp), a4 = a2 * a2, a6 = a4 * a2;
    const double w_part = exp(-a2) * (rinv * W[0]
        + r3inv * (1 + 2 * a2) * (W[P] * dx + W[2 * P] * dy + W[3 * P] * dz)
        + r5inv * (3 + 4 * a2 + 4 * a4) * (W[4 * P] * dx * dy + W[5 * P] * dy * dz + W[6 * P] * dx * dz)
        + r7inv * (15 + 18 * a2 + 12 * a4 + 8 * a6) * W[7 * P] * dx * dy * dz);
    return q_part - tq * w_part;
}

// Contributions of a source (or a source-cluster grid point) to the two SS
// grid fields: field_q += qw K(r), field_w += w g(r) K(r).
template <int KT>
__device__ __forceinline__ void ss_grid(double dx, double dy, double dz, double qw, double w, double kp, double &fq,
                                        double &fw)
{
    const double r = sqrt(dx * dx + dy * dy + dz * dz);
    if (KT == K_COULOMB) {
        fq += qw / r;
        fw += exp(-r * r / (kp * kp)) * w / r;
    } else {
        const double e = exp(-kp * r) / r;
        fq += qw * e;
        fw += w * e;
    }
}

// The short forms (bt_fp64.cuh), used for every kernel; the functions above
// form a sum again where it is not finite.  exp64 takes r (kappa) for the
// Yukawa kernels and r^2 (1 / alpha^2) for the others.
struct SsKern {
    double eps2;
    Exp64 ex;
    bool lib;               // parameters that exp64 does not take
};

template <int KT>
__device__ __forceinline__ SsKern ss_kern(double kp, double kp2, double2 *tab)
{
    SsKern k;
    k.eps2 = KT == K_REGCOULOMB || KT == K_REGYUKAWA ? kp2 * kp2 : 0.0;
    const double kappa = KT == K_YUKAWA || KT == K_REGYUKAWA ? kp : 1.0 / (kp * kp);
    k.lib = !exp64_takes(kappa);
    for (int i = threadIdx.x; i < EXP64_TAB; i += blockDim.x) tab[i] = exp64_table[i];
    k.ex = exp64_make(kappa, tab);
    return k;
}

// K(r) with the exponential of the Yukawa kernels (kv), and the subtraction
// factor g (1 for those).
template <int KT>
__device__ __forceinline__ void ss_values(double r2, const SsKern &k, double &kv, double &g)
{
    if (KT == K_YUKAWA) {
        double r;
        const double y = rsqrt_sqrt_n(r2, r);
        kv = y * exp64<true>(r, k.ex);
        g = 1.0;
    } else if (KT == K_REGYUKAWA) {
        // r of a coincident pair from a tiny r^2 instead of zero
        const double c = __hiloint2double(max(__double2hiint(r2), 0x01a00000), __double2loint(r2));
        double r;
        rsqrt_sqrt_n(c, r);
        kv = rsqrt_n(r2 + k.eps2) * exp64<true>(r, k.ex);
        g = 1.0;
    } else {
        kv = rsqrt_n(KT == K_REGCOULOMB ? r2 + k.eps2 : r2);
        g = exp64<true>(r2, k.ex);
    }
}

// Near-field tile: x, y; z, q; w of each source.
struct SsTile {
    double2 *xy, *zq;
    double *w;
};
constexpr size_t SS_TILE_BYTES = (2 * sizeof(double2) + sizeof(double)) * EV_TILE;

__device__ __forceinline__ SsTile ss_tile(double *sm)
{
    double2 *p = reinterpret_cast<double2 *>(sm);
    return SsTile{p, p + EV_TILE, reinterpret_cast<double *>(p + 2 * EV_TILE)};
}

// acc += the SS pair terms of sources sb .. sb + sn - 1 (all threads call).
template <int KT>
__device__ __forceinline__ void ss_near(double *acc, const SsTile &t, int sb, int sn, const double *__restrict__ sx,
                                        const double *__restrict__ sy, const double *__restrict__ sz,
                                        const double *__restrict__ sq, const double *__restrict__ sw, const Out2 &o,
                                        const double *tq, const Lanes &w, const SsKern &k)
{
    for (int c0 = 0; c0 < sn; c0 += EV_TILE) {
        const int cm = min(EV_TILE, sn - c0);
        for (int i = threadIdx.x; i < cm; i += EV_THREADS) {
            const int j = sb + c0 + i;
            t.xy[i] = make_double2(sx[j], sy[j]);
            t.zq[i] = make_double2(sz[j], sq[j]);
            t.w[i] = sw[j];
        }
        __syncthreads();
        if (w.active[0])
#pragma unroll 2
            for (int i = w.slice; i < cm; i += w.slices) {
                const double2 p = t.xy[i], s = t.zq[i];
                const double sw_i = t.w[i];
#pragma unroll
                for (int b = 0; b < 2; b++) {
                    const double dx = o.x[b] - p.x, dy = o.y[b] - p.y, dz = o.z[b] - s.x;
                    const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
                    double kv, g;
                    ss_values<KT>(r2, k, kv, g);
                    // r <= DBL_MIN is skipped by Coulomb and Yukawa: every r^2 but zero counts
                    if ((KT == K_COULOMB || KT == K_YUKAWA) && __double_as_longlong(r2) <= 0) kv = 0.0;
                    acc[b] = fma(fma(-tq[b], g, s.y) * sw_i, kv, acc[b]);
                }
            }
        __syncthreads();
    }
}

// Particle-output evaluation with SS: PC + PP per chunk of a target leaf; the
// division of a block and of the lists is that of bt_eval64.cuh.
template <int KT, bool HERM>
__global__ void __launch_bounds__(EV_THREADS, 4) k_ss_targets(const __grid_constant__ SsTargetsArgs a)
{
    extern __shared__ __align__(16) double sm[];
    __shared__ double red[2 * EV_THREADS];
    __shared__ double2 tab[EXP64_TAB];
    const SsKern k = ss_kern<KT>(a.kp, a.kp2, tab);
    const int2 it = a.items[blockIdx.x];
    const int u = it.x, tnode = a.leaf_node[u];
    const Lanes w(min(EV_CHUNK, a.t_numpar[tnode] - it.y * EV_CHUNK));
    const int t0 = a.t_ibeg[tnode] + it.y * EV_CHUNK;
    Out2 o;
    double tq[2];
#pragma unroll
    for (int b = 0; b < 2; b++) {
        const int t = t0 + w.out(b);
        o.x[b] = a.tx[t]; o.y[b] = a.ty[t]; o.z[b] = a.tz[t]; tq[b] = a.tq[t];
    }
    const int np1 = a.n + 1, P = np1 * np1 * np1, nq = HERM ? 8 * P : P;
    const int64_t ab = a.a_off[u], ae = a.a_off[u + 1], db = a.d_off[u], de = a.d_off[u + 1];
    const int seg0 = a.partial ? blockIdx.y : 0, seg1 = a.partial ? blockIdx.y + 1 : EV_SEGS;
    double total[2] = {0.0, 0.0};
    for (int seg = seg0; seg < seg1; seg++) {
        const int64_t a0 = seg_begin(ab, ae, seg), a1 = seg_begin(ab, ae, seg + 1);
        const int64_t d0 = seg_begin(db, de, seg), d1 = seg_begin(db, de, seg + 1);
        double acc[2] = {0.0, 0.0};
        for (int64_t e = k.lib && !HERM ? a1 : a0; e < a1; e++) {
            const int s = a.a_idx[e];
            double *g = sm, *q = sm + 3 * np1, *wq = q + P;
            for (int i = threadIdx.x; i < 3 * np1; i += EV_THREADS) g[i] = a.s_grid[(size_t)s * 3 * np1 + i];
            if (!HERM)
                for (int i = threadIdx.x; i < P; i += EV_THREADS) {
                    q[i] = a.Q[(size_t)s * P + i];
                    wq[i] = a.W[(size_t)s * P + i];
                }
            __syncthreads();
            if (w.active[0])
                for (int row = w.slice; row < np1 * np1; row += w.slices) {
                    const int k3 = row / np1, k2 = row - k3 * np1;
                    double dy[2], dz[2], dyz[2];
#pragma unroll
                    for (int b = 0; b < 2; b++) {
                        dy[b] = o.y[b] - g[np1 + k2];
                        dz[b] = o.z[b] - g[2 * np1 + k3];
                        dyz[b] = fma(dy[b], dy[b], dz[b] * dz[b]);
                    }
#pragma unroll 2
                    for (int i = 0; i < np1; i++) {
                        const int j = row * np1 + i;
#pragma unroll
                        for (int b = 0; b < 2; b++) {
                            const double dx = o.x[b] - g[i];
                            if (HERM) {
                                acc[b] += ss_pc_herm<KT>(dx, dy[b], dz[b], a.Q + (size_t)s * nq + j,
                                                         a.W + (size_t)s * nq + j, P, tq[b], a.kp, a.kp2);
                            } else {
                                double kv, f;
                                ss_values<KT>(fma(dx, dx, dyz[b]), k, kv, f);
                                acc[b] = fma(fma(-tq[b] * f, wq[j], q[j]), kv, acc[b]);
                            }
                        }
                    }
                }
            __syncthreads();
        }
        const SsTile tile = ss_tile(sm);
        for (int64_t e = k.lib ? d1 : d0; e < d1; e++) {
            const int s = a.d_idx[e];
            ss_near<KT>(acc, tile, a.s_ibeg[s], a.s_numpar[s], a.sx, a.sy, a.sz, a.sq, a.sw, o, tq, w, k);
        }
#pragma unroll 1
        for (int b = 0; b < 2; b++) {
            if (!w.active[b] || (!k.lib && isfinite(acc[b]))) continue;
            // again with the library functions, the thread's share
            double s = 0.0;
            const double x = o.x[b], y = o.y[b], z = o.z[b];
            for (int64_t e = a0; e < a1; e++) {
                const double *g = a.s_grid + (size_t)a.a_idx[e] * 3 * np1, *Qs = a.Q + (size_t)a.a_idx[e] * nq,
                             *Ws = a.W + (size_t)a.a_idx[e] * nq;
                for (int row = w.slice; row < np1 * np1; row += w.slices)
                    for (int i = 0; i < np1; i++) {
                        const int k3 = row / np1, k2 = row - k3 * np1, j = row * np1 + i;
                        const double dx = x - g[i], dy = y - g[np1 + k2], dz = z - g[2 * np1 + k3];
                        if (HERM) s += ss_pc_herm<KT>(dx, dy, dz, Qs + j, Ws + j, P, tq[b], a.kp, a.kp2);
                        else s += ss_pc<KT>(dx, dy, dz, Qs[j], Ws[j], tq[b], a.kp, a.kp2);
                    }
            }
            for (int64_t e = d0; e < d1; e++) {
                const int n = a.d_idx[e], sb = a.s_ibeg[n], sn = a.s_numpar[n];
                for (int c0 = 0; c0 < sn; c0 += EV_TILE)
                    for (int i = sb + c0 + w.slice; i < sb + min(sn, c0 + EV_TILE); i += w.slices)
                        s += ss_pp<KT>(x - a.sx[i], y - a.sy[i], z - a.sz[i], a.sq[i], a.sw[i], tq[b], a.kp, a.kp2);
            }
            acc[b] = s;
        }
        sum_slices(acc, red, w);
#pragma unroll
        for (int b = 0; b < 2; b++) {
            total[b] += acc[b];
            if (a.partial && w.active[b] && w.slice == 0) a.partial[(size_t)seg * a.pstride + t0 + w.out(b)] = acc[b];
        }
    }
#pragma unroll
    for (int b = 0; b < 2; b++)
        if (!a.partial && w.active[b] && w.slice == 0) a.pot[t0 + w.out(b)] = total[b];
}

// Grid-output evaluation with SS (Lagrange): M2L from source clusters (Q, W)
// and CP from source particles (q*w, w) onto both fields of a target node's
// grid, one grid point per thread, Coulomb and Yukawa.
template <int KT>
__global__ void __launch_bounds__(SS_THREADS) k_ss_grids(const __grid_constant__ SsGridsArgs a)
{
    extern __shared__ __align__(16) double sm[];
    __shared__ double2 tab[EXP64_TAB];
    const SsKern k = ss_kern<KT>(a.kp, 0.0, tab);
    const int2 it = a.items[blockIdx.x];
    const int T = it.x;
    const int np1 = a.n + 1, P = np1 * np1 * np1;
    const int j0 = it.y * SS_THREADS + threadIdx.x;
    const bool active = j0 < P;
    const int jj = active ? j0 : 0;
    const double *tg = a.t_grid + (size_t)T * 3 * np1;
    const double x = tg[jj % np1], y = tg[np1 + (jj / np1) % np1], z = tg[2 * np1 + jj / (np1 * np1)];
    double fq = 0.0, fw = 0.0;
    for (int64_t e = k.lib ? a.c_off[T + 1] : a.c_off[T]; e < a.c_off[T + 1]; e++) {
        const int s = a.c_idx[e];
        double *g = sm, *q = sm + 3 * np1, *w = q + P;
        for (int i = threadIdx.x; i < 3 * np1; i += SS_THREADS) g[i] = a.s_grid[(size_t)s * 3 * np1 + i];
        for (int i = threadIdx.x; i < P; i += SS_THREADS) {
            q[i] = a.Q[(size_t)s * P + i];
            w[i] = a.W[(size_t)s * P + i];
        }
        __syncthreads();
        if (active)
            for (int row = 0; row < np1 * np1; row++) {
                const int k3 = row / np1, k2 = row - k3 * np1;
                const double dy = y - g[np1 + k2], dz = z - g[2 * np1 + k3], dyz = fma(dy, dy, dz * dz);
#pragma unroll 4
                for (int i = 0; i < np1; i++) {
                    const double dx = x - g[i];
                    double kv, f;
                    ss_values<KT>(fma(dx, dx, dyz), k, kv, f);
                    fq = fma(q[row * np1 + i], kv, fq);
                    fw = fma(f * w[row * np1 + i], kv, fw);
                }
            }
        __syncthreads();
    }
    const SsTile t = ss_tile(sm);
    for (int64_t e = k.lib ? a.p_off[T + 1] : a.p_off[T]; e < a.p_off[T + 1]; e++) {
        const int s = a.p_idx[e];
        const int sb = a.s_ibeg[s], sn = a.s_numpar[s];
        for (int c0 = 0; c0 < sn; c0 += EV_TILE) {
            const int cm = min(EV_TILE, sn - c0);
            for (int i = threadIdx.x; i < cm; i += SS_THREADS) {
                const int j = sb + c0 + i;
                t.xy[i] = make_double2(a.sx[j], a.sy[j]);
                t.zq[i] = make_double2(a.sz[j], a.sq[j] * a.sw[j]);
                t.w[i] = a.sw[j];
            }
            __syncthreads();
            if (active)
#pragma unroll 4
                for (int i = 0; i < cm; i++) {
                    const double2 p = t.xy[i], v = t.zq[i];
                    const double dx = x - p.x, dy = y - p.y, dz = z - v.x;
                    double kv, f;
                    ss_values<KT>(fma(dx, dx, fma(dy, dy, dz * dz)), k, kv, f);
                    fq = fma(v.y, kv, fq);
                    fw = fma(f * t.w[i], kv, fw);
                }
            __syncthreads();
        }
    }
    if (active && (k.lib || !isfinite(fq) || !isfinite(fw))) {
        fq = fw = 0.0;
        for (int64_t e = a.c_off[T]; e < a.c_off[T + 1]; e++) {
            const double *g = a.s_grid + (size_t)a.c_idx[e] * 3 * np1, *Qs = a.Q + (size_t)a.c_idx[e] * P,
                         *Ws = a.W + (size_t)a.c_idx[e] * P;
            for (int j = 0; j < P; j++)
                ss_grid<KT>(x - g[j % np1], y - g[np1 + (j / np1) % np1], z - g[2 * np1 + j / (np1 * np1)], Qs[j], Ws[j],
                            a.kp, fq, fw);
        }
        for (int64_t e = a.p_off[T]; e < a.p_off[T + 1]; e++) {
            const int s = a.p_idx[e];
            for (int i = a.s_ibeg[s]; i < a.s_ibeg[s] + a.s_numpar[s]; i++)
                ss_grid<KT>(x - a.sx[i], y - a.sy[i], z - a.sz[i], a.sq[i] * a.sw[i], a.sw[i], a.kp, fq, fw);
        }
    }
    if (active) {
        a.Phi_q[(size_t)T * P + j0] = fq;
        a.Phi_w[(size_t)T * P + j0] = fw;
    }
}

__global__ void k_mul(int n, const double *__restrict__ a, const double *__restrict__ b, double *__restrict__ c)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) c[i] = a[i] * b[i];
}

__global__ void k_axpy(int n, double c, const double *__restrict__ x, double *__restrict__ y)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] += c * x[i];
}

// The correction over work items (unit, chunk of `chunk` targets): a
// target-sharded call adds it to the targets of its own leaves only.  The
// same operation as k_axpy, target by target.
__global__ void k_axpy_items(const int2 *__restrict__ items, int chunk, const int *__restrict__ leaf_node,
                             const int *__restrict__ ibeg, const int *__restrict__ numpar, double c,
                             const double *__restrict__ x, double *__restrict__ y)
{
    const int2 it = items[blockIdx.x];
    const int node = leaf_node[it.x];
    const int end = min(numpar[node], (it.y + 1) * chunk);
    for (int i = it.y * chunk + threadIdx.x; i < end; i += blockDim.x) {
        const int t = ibeg[node] + i;
        y[t] += c * x[t];
    }
}

// SS direct sum (InteractionCompute_Direct with singularity subtraction,
// src/interaction_compute/interaction_compute_direct.c:26-231): sources
// blockIdx.y of gridDim.y parts onto EV_CHUNK targets, as k_direct.
template <int KT>
__global__ void __launch_bounds__(EV_THREADS, 4)
k_ss_direct(int nt, int ns, const double *__restrict__ tx, const double *__restrict__ ty,
            const double *__restrict__ tz, const double *__restrict__ tq, const double *__restrict__ sx,
            const double *__restrict__ sy, const double *__restrict__ sz, const double *__restrict__ sq,
            const double *__restrict__ sw, double kp, double kp2, double *__restrict__ out)
{
    extern __shared__ __align__(16) double sm[];
    __shared__ double red[2 * EV_THREADS];
    __shared__ double2 tab[EXP64_TAB];
    const SsKern k = ss_kern<KT>(kp, kp2, tab);
    const int t0 = blockIdx.x * EV_CHUNK;
    const Lanes w(min(EV_CHUNK, nt - t0));
    Out2 o;
    double q[2], acc[2] = {0.0, 0.0};
#pragma unroll
    for (int b = 0; b < 2; b++) {
        const int t = t0 + w.out(b);
        o.x[b] = tx[t]; o.y[b] = ty[t]; o.z[b] = tz[t]; q[b] = tq[t];
    }
    const int s0 = (int)((int64_t)ns * blockIdx.y / gridDim.y), s1 = (int)((int64_t)ns * (blockIdx.y + 1) / gridDim.y);
    ss_near<KT>(acc, ss_tile(sm), s0, k.lib ? 0 : s1 - s0, sx, sy, sz, sq, sw, o, q, w, k);
#pragma unroll 1
    for (int b = 0; b < 2; b++)
        if (w.active[b] && (k.lib || !isfinite(acc[b]))) {
            acc[b] = 0.0;
            for (int c0 = s0; c0 < s1; c0 += EV_TILE)
                for (int i = c0 + w.slice; i < min(s1, c0 + EV_TILE); i += w.slices)
                    acc[b] += ss_pp<KT>(o.x[b] - sx[i], o.y[b] - sy[i], o.z[b] - sz[i], sq[i], sw[i], q[b], kp, kp2);
        }
    sum_slices(acc, red, w);
#pragma unroll
    for (int b = 0; b < 2; b++)
        if (w.active[b] && w.slice == 0) out[(size_t)blockIdx.y * nt + t0 + w.out(b)] = acc[b];
}

// Dynamic shared memory: a cluster's grid and both proxy arrays (Lagrange), or a tile.
size_t ss_smem(int n, bool hermite)
{
    const size_t np1 = n + 1, far = sizeof(double) * (3 * np1 + (hermite ? 0 : 2 * np1 * np1 * np1));
    return far > SS_TILE_BYTES ? far : SS_TILE_BYTES;
}

template <int KT, bool HERM>
void ss_targets_t(const SsTargetsArgs &a, cudaStream_t st)
{
    const size_t sm = ss_smem(a.n, HERM);
    cudaFuncSetAttribute(k_ss_targets<KT, HERM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_ss_targets<KT, HERM><<<dim3(a.nitems, a.partial ? EV_SEGS : 1), EV_THREADS, sm, st>>>(a);
    if (a.partial)
        launch_sum_segments(a.nitems, a.items, EV_CHUNK, a.leaf_node, a.t_ibeg, a.t_numpar, a.partial, a.pstride, a.pot, st);
}

}  // namespace

int ss_chunk() { return EV_CHUNK; }

void launch_ss_targets(int kernel, bool hermite, const SsTargetsArgs &a, cudaStream_t st)
{
    if (a.nitems <= 0) return;
    if (kernel == K_COULOMB) hermite ? ss_targets_t<K_COULOMB, true>(a, st) : ss_targets_t<K_COULOMB, false>(a, st);
    else if (kernel == K_YUKAWA) hermite ? ss_targets_t<K_YUKAWA, true>(a, st) : ss_targets_t<K_YUKAWA, false>(a, st);
    else if (kernel == K_REGYUKAWA) ss_targets_t<K_REGYUKAWA, false>(a, st);
    else hermite ? ss_targets_t<K_REGCOULOMB, true>(a, st) : ss_targets_t<K_REGCOULOMB, false>(a, st);
}

template <int KT>
static void ss_grids_t(const SsGridsArgs &a, cudaStream_t st)
{
    const size_t sm = ss_smem(a.n, false);
    cudaFuncSetAttribute(k_ss_grids<KT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_ss_grids<KT><<<a.nitems, SS_THREADS, sm, st>>>(a);
}

void launch_ss_grids(int kernel, const SsGridsArgs &a, cudaStream_t st)
{
    if (a.nitems <= 0) return;
    if (kernel == K_COULOMB) ss_grids_t<K_COULOMB>(a, st);
    else ss_grids_t<K_YUKAWA>(a, st);
}

bool ss_direct_kernel(int kernel)
{
    return kernel == K_COULOMB || kernel == K_YUKAWA || kernel == K_REGCOULOMB || kernel == K_REGYUKAWA;
}

void launch_ss_direct(int kernel, int nt, int ns, const double *tx, const double *ty, const double *tz,
                      const double *tq, const double *sx, const double *sy, const double *sz, const double *sq,
                      const double *sw, double kp, double kp2, double *partial, double *out, cudaStream_t st)
{
    if (nt <= 0) return;
    const int parts = direct_parts(nt, ns);
    double *dst = parts > 1 ? partial : out;
    const dim3 grid((nt + EV_CHUNK - 1) / EV_CHUNK, parts);
#define BT_SSD(K)                                                                                                   \
    k_ss_direct<K><<<grid, EV_THREADS, SS_TILE_BYTES, st>>>(nt, ns, tx, ty, tz, tq, sx, sy, sz, sq, sw, kp, kp2, dst)
    if (kernel == K_COULOMB) BT_SSD(K_COULOMB);
    else if (kernel == K_YUKAWA) BT_SSD(K_YUKAWA);
    else if (kernel == K_REGYUKAWA) BT_SSD(K_REGYUKAWA);
    else BT_SSD(K_REGCOULOMB);
#undef BT_SSD
    if (parts > 1) launch_sum_parts(nt, parts, partial, out, st);
}

void launch_mul(int n, const double *a, const double *b, double *c, cudaStream_t st)
{
    if (n > 0) k_mul<<<(n + 255) / 256, 256, 0, st>>>(n, a, b, c);
}

void launch_ss_correction(int n, double c, const double *tq, double *pot, cudaStream_t st)
{
    if (n > 0) k_axpy<<<(n + 255) / 256, 256, 0, st>>>(n, c, tq, pot);
}

void launch_ss_correction_items(int nitems, const int2 *items, int chunk, const int *leaf_node, const int *ibeg,
                                const int *numpar, double c, const double *tq, double *pot, cudaStream_t st)
{
    if (nitems > 0) k_axpy_items<<<nitems, SS_THREADS, 0, st>>>(items, chunk, leaf_node, ibeg, numpar, c, tq, pot);
}

double ss_correction_constant(int kernel, double kp)
{
    const double pi = 3.14159265358979323846;
    if (kernel == K_YUKAWA || kernel == K_REGYUKAWA) return 4.0 * pi / kp / kp;
    return 2.0 * pi * kp * kp;
}

}  // namespace bt
