// bt_eval64.cuh -- FP64 evaluation kernels (particle and grid outputs),
// instantiated per kernel type in bt_eval64_*.cu.
//
// Bound: the FP64 pipe.  Per kernel value the Lagrange far field needs 7 FP64
// instructions (Coulomb: one for r^2, five for 1/r, one to accumulate) and the
// near field 12; the degree is a template parameter so that the target's
// differences along one grid axis stay in registers.
//
// What is left of the issue slots decides how much of that rate is reached, so
// every thread evaluates two outputs against each value it reads from shared
// memory, the near-field tiles are padded to the unrolled loop with their first
// source without its charge (finite values wherever that source's are), and the
// skipping rule is tested only for source nodes whose box meets the target
// leaf's.
//
// A work item is a chunk of up to EV_CHUNK outputs (targets of a leaf, or
// points of a target grid) and its block's threads are `lanes` pairs of
// outputs wide, the smallest power of two that holds them; the remaining
// factor of the block (`slices`) divides the source side, so small leaves and
// the last chunk of a leaf still use every thread.  Each output's list is summed in
// EV_SEGS segments that depend on the list alone, and the segments in order:
// a launch with few items runs one block per (item, segment) and adds the
// segments' sums in a second kernel, with the same bits.
#pragma once

#include <cuda_runtime.h>

#include "bt_device.h"
#include "bt_eval64.h"
#include "bt_fp64.cuh"
#include "bt_kernels.cuh"

namespace bt {

constexpr int EV_TILE = 512;        // sources per shared-memory tile

// What a kernel value needs besides r^2 and the charge.  FAR: exp64's.
template <bool FAR>
struct Kern64 {
    double kp, kp2, eps2;
    Exp64 ex;
    bool lib;               // Yukawa with a kappa that exp64 does not take: the library functions throughout
};

template <int KT>
__host__ __device__ constexpr bool fast64() { return KT <= K_REGCOULOMB; }

template <int KT, bool FAR>
__device__ __forceinline__ Kern64<FAR> kern64_make(double kp, double kp2, double2 *tab)
{
    Kern64<FAR> k;
    k.kp = kp; k.kp2 = kp2;
    k.eps2 = KT == K_REGCOULOMB ? kp * kp : 0.0;
    k.lib = KT == K_YUKAWA && !exp64_takes(kp);
    if (KT == K_YUKAWA) {
        for (int i = threadIdx.x; i < EXP64_TAB; i += blockDim.x) tab[i] = exp64_table[i];
        k.ex = exp64_make(kp, tab);
    }
    return k;
}

// K(r), r2 the squared distance (plus eps^2 for the regularized kernel).
template <int KT, bool FAR>
__device__ __forceinline__ double value64(double r2, const Kern64<FAR> &k)
{
    if (KT == K_YUKAWA) {
        double r;
        const double y = rsqrt_sqrt_n(r2, r);
        return y * exp64<FAR>(r, k.ex);
    }
    return rsqrt_n(r2);
}
template <int KT, bool FAR>
__device__ __forceinline__ double add64(double acc, double r2, double q, const Kern64<FAR> &k)
{
    return fma(q, value64<KT>(r2, k), acc);
}

// The reference's skipping rule on r^2: Coulomb keeps r^2 > DBL_MIN, Yukawa
// r > DBL_MIN (every r^2 but zero).  An integer comparison of the bits (r^2 is
// never negative): the integer pipe has room that the FP64 pipe lacks.
template <int KT>
__device__ __forceinline__ bool keeps64(double r2)
{
    return KT == K_REGCOULOMB || __double_as_longlong(r2) > (KT == K_COULOMB ? 0x0010000000000000LL : 0LL);
}

// How a block's threads share a chunk of cnt outputs: thread `lane` of a
// slice has outputs lane and lane + lanes.
struct Lanes {
    int lanes, slices, lane, slice;
    bool active[2];
    __device__ explicit Lanes(int cnt)
    {
        lanes = EV_THREADS;
        while (lanes >= cnt && lanes > 1) lanes >>= 1;
        slices = EV_THREADS / lanes;
        lane = threadIdx.x & (lanes - 1);
        slice = threadIdx.x / lanes;
        active[0] = lane < cnt;
        active[1] = lane + lanes < cnt;
    }
    // output b of the thread within the chunk, output 0 of the chunk where it has none
    __device__ int out(int b) const { return active[b] ? lane + b * lanes : 0; }
};

struct Out2 {
    double x[2], y[2], z[2];
};

// Far field of one source cluster: grid rows slice, slice + slices, ...; g the
// 3 (n+1) grid coordinates, q the proxy charges.
template <int KT, int NP1, bool FAR>
__device__ __forceinline__ void far64(double *acc, const double *g, const double *q, const Out2 &o, const Lanes &w,
                                      const Kern64<FAR> &k)
{
    double gx[2][NP1];
#pragma unroll
    for (int i = 0; i < NP1; i++) {
        gx[0][i] = o.x[0] - g[i];
        gx[1][i] = o.x[1] - g[i];
    }
    for (int row = w.slice; row < NP1 * NP1; row += w.slices) {
        const int k3 = row / NP1, k2 = row - k3 * NP1;
        double dyz[2];
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const double dy = o.y[b] - g[NP1 + k2], dz = o.z[b] - g[2 * NP1 + k3];
            dyz[b] = fma(dy, dy, dz * dz);
            if (KT == K_REGCOULOMB) dyz[b] += k.eps2;
        }
        const double *qr = q + row * NP1;
#pragma unroll
        for (int i = 0; i < NP1; i++) {
            const double qi = qr[i];
#pragma unroll
            for (int b = 0; b < 2; b++) acc[b] = add64<KT>(acc[b], fma(gx[b][i], gx[b][i], dyz[b]), qi, k);
        }
    }
}

// The same for the kernels without a short form.
template <int KT, bool FAR>
__device__ __forceinline__ void far64_any(double *acc, int np1, const double *g, const double *q, const Out2 &o,
                                          const Lanes &w, const Kern64<FAR> &k)
{
    for (int row = w.slice; row < np1 * np1; row += w.slices) {
        const int k3 = row / np1, k2 = row - k3 * np1;
        for (int i = 0; i < np1; i++)
#pragma unroll
            for (int b = 0; b < 2; b++)
                acc[b] += k_any<KT, false>(o.x[b] - g[i], o.y[b] - g[np1 + k2], o.z[b] - g[2 * np1 + k3],
                                           q[row * np1 + i], k.kp, k.kp2);
    }
}

// Hermite far field: q holds each point's 8 moments, qxy, qyz, qxz times 3 and
// qxyz times 15 (K_*_PC_Hermite, src/kernels/coulomb/coulomb_pc.c:66-138).
// With u = 1/r^2 the value is
//   1/r [ q + u (qx dx + qy dy + qz dz) + u^2 (qxy dx dy + qyz dy dz + qxz dx dz) + u^3 qxyz dx dy dz ]
// sorted by powers of dx (b, c below): 15 FP64 instructions besides 1/r.
// Yukawa has its polynomials in kappa r beside each power of u.
template <int KT, bool FAR>
__device__ __forceinline__ void herm64(double *acc, int np1, const double *g, const double *q, const Out2 &o,
                                       const Lanes &w, const Kern64<FAR> &k)
{
    for (int row = w.slice; row < np1 * np1; row += w.slices) {
        const int k3 = row / np1, k2 = row - k3 * np1;
        double dy[2], dz[2], dydz[2], dyz[2];
#pragma unroll
        for (int b = 0; b < 2; b++) {
            dy[b] = o.y[b] - g[np1 + k2];
            dz[b] = o.z[b] - g[2 * np1 + k3];
            dydz[b] = dy[b] * dz[b];
            dyz[b] = fma(dy[b], dy[b], dz[b] * dz[b]);
            if (KT == K_REGCOULOMB) dyz[b] += k.eps2;
        }
        for (int i = 0; i < np1; i++) {
            const double2 *qp = reinterpret_cast<const double2 *>(q + 8 * (row * np1 + i));
            const double2 qa = qp[0], qb = qp[1], qc = qp[2], qd = qp[3];
            const double m[8] = {qa.x, qa.y, qb.x, qb.y, qc.x, qc.y, qd.x, qd.y};
#pragma unroll
            for (int b = 0; b < 2; b++) {
                const double dx = o.x[b] - g[i], r2 = fma(dx, dx, dyz[b]);
                if (KT == K_YUKAWA) {
                    double r;
                    const double rinv = rsqrt_sqrt_n(r2, r), u = rinv * rinv;
                    const double kr = k.kp * r, kr2 = kr * kr, p1 = 1.0 + kr, p2 = fma(kr2, 1.0 / 3.0, p1),
                                 p3 = fma(kr2 * kr, 1.0 / 15.0, fma(kr2, 0.4, p1));
                    const double e = fma(u * p2, m[5] * dydz[b], p1 * fma(m[3], dz[b], m[2] * dy[b]));
                    const double c = fma(u * p3, m[7] * dydz[b], p2 * fma(m[6], dz[b], m[4] * dy[b]));
                    const double v = fma(dx * u, fma(u, c, p1 * m[1]), fma(u, e, m[0]));
                    acc[b] = fma(rinv * v, exp64<FAR>(r, k.ex), acc[b]);
                } else {
                    const double rinv = rsqrt_n(r2), u = rinv * rinv, v = u * dydz[b];
                    const double e = fma(m[5], v, fma(m[3], dz[b], m[2] * dy[b]));
                    const double c = fma(m[7], v, fma(m[6], dz[b], m[4] * dy[b]));
                    acc[b] = fma(rinv, fma(dx * u, fma(u, c, m[1]), fma(u, e, m[0])), acc[b]);
                }
            }
        }
    }
}

// sin-over-r Hermite: the library form.
template <int KT, bool FAR>
__device__ __forceinline__ void herm64_any(double *acc, int np1, const double *g, const double *q, const Out2 &o,
                                           const Lanes &w, const Kern64<FAR> &k)
{
    const int P = np1 * np1 * np1;
    for (int row = w.slice; row < np1 * np1; row += w.slices) {
        const int k3 = row / np1, k2 = row - k3 * np1;
        for (int i = 0; i < np1; i++)
#pragma unroll
            for (int b = 0; b < 2; b++)
                acc[b] += k_pc_herm<KT>(o.x[b] - g[i], o.y[b] - g[np1 + k2], o.z[b] - g[2 * np1 + k3],
                                        q + row * np1 + i, P, k.kp);
    }
}

// Scale of moment m as herm64 takes it.
__device__ __forceinline__ double herm64_scale(int m) { return m == 7 ? 15.0 : m >= 4 ? 3.0 : 1.0; }

// Near-field tile: x, y and z, q of each source.
struct Tile64 {
    double2 *xy, *zq;
};

// Source i of a tile.  TEST: with the skipping rule, else mn gets the smallest
// upper half of the thread's r^2 (as an integer: r^2 is never negative).
template <int KT, bool TEST, bool FAR>
__device__ __forceinline__ void near64_one(double *acc, const Tile64 &t, int i, const Out2 &o, const Kern64<FAR> &k,
                                           int &mn)
{
    const double2 p = t.xy[i], s = t.zq[i];
#pragma unroll
    for (int b = 0; b < 2; b++) {
        const double dx = o.x[b] - p.x, dy = o.y[b] - p.y, dz = o.z[b] - s.x;
        const double r2 = fma(dx, dx, fma(dy, dy, KT == K_REGCOULOMB ? fma(dz, dz, k.eps2) : dz * dz));
        if (!TEST) mn = min(mn, __double2hiint(r2));
        if (!TEST || keeps64<KT>(r2)) acc[b] = add64<KT>(acc[b], r2, s.y, k);
    }
}

// Sources i0, i0 + step, ... < cm of a tile, the range a multiple of step long.
template <int KT, bool TEST, bool FAR>
__device__ __forceinline__ void near64(double *acc, const Tile64 &t, int i0, int step, int cm, const Out2 &o,
                                       const Kern64<FAR> &k, int &mn)
{
    int c = i0;
    for (; c + 3 * step < cm; c += 4 * step)
#pragma unroll
        for (int h = 0; h < 4; h++) near64_one<KT, TEST>(acc, t, c + h * step, o, k, mn);
#pragma unroll 1
    for (; c < cm; c += step) near64_one<KT, TEST>(acc, t, c, o, k, mn);
}

// The same where some pair may have to be skipped: groups of 32 sources per
// thread are summed without the test, and again with it if one of their r^2
// is at the rule's limit or below (a target that coincides with a source: one
// group in hundreds).  The test in every term took 24 instructions per value
// instead of 15, 5.1 ms for 10,000 x 500,000 pairs.
template <int KT, bool FAR>
__device__ __forceinline__ void near64_skip(double *acc, const Tile64 &t, int i0, int step, int cm, const Out2 &o,
                                            const Kern64<FAR> &k)
{
    for (int c = i0; c < cm; c += 32 * step) {
        const int ce = min(cm, c + 32 * step);
        double s[2] = {0.0, 0.0};
        int mn = 0x7fffffff;
        near64<KT, false>(s, t, c, step, ce, o, k, mn);
        if (mn <= 0x00100000) {
            s[0] = s[1] = 0.0;
            near64<KT, true>(s, t, c, step, ce, o, k, mn);
        }
        acc[0] += s[0];
        acc[1] += s[1];
    }
}

template <int KT, bool PP, bool FAR>
__device__ __forceinline__ void near64_any(double *acc, const Tile64 &t, int i0, int step, int cm, const Out2 &o,
                                           const Kern64<FAR> &k)
{
    for (int i = i0; i < cm; i += step) {
        const double2 p = t.xy[i], s = t.zq[i];
#pragma unroll
        for (int b = 0; b < 2; b++)
            acc[b] += k_any<KT, PP>(o.x[b] - p.x, o.y[b] - p.y, o.z[b] - s.x, s.y, k.kp, k.kp2);
    }
}

// Sources sb .. sb + sn - 1 for every thread of the block (tiles staged by
// all).  test: some pair may coincide.
template <int KT, bool PP, bool FAR>
__device__ __forceinline__ void near64_node(double *acc, const Tile64 &t, int sb, int sn, const double *__restrict__ sx,
                                            const double *__restrict__ sy, const double *__restrict__ sz,
                                            const double *__restrict__ sq, bool test, const Out2 &o, const Lanes &w,
                                            const Kern64<FAR> &k)
{
    for (int c0 = 0; c0 < sn; c0 += EV_TILE) {
        const int cm = min(EV_TILE, sn - c0);
        // padded to whole groups of four sources per thread, or, where there are
        // fewer, to whole sources per thread (leaf limit 10: 64 sources for 7,
        // evaluation of 60,000 particles 14.4 ms, so 11.3 ms); EV_TILE is a
        // multiple of both
        const int pad = cm < 4 * w.slices ? w.slices : 4 * w.slices;
        const int cmp = fast64<KT>() ? (cm + pad - 1) & ~(pad - 1) : cm;
        for (int i = threadIdx.x; i < cmp; i += EV_THREADS) {
            const int j = sb + c0 + (i < cm ? i : 0);
            t.xy[i] = make_double2(sx[j], sy[j]);
            t.zq[i] = make_double2(sz[j], i < cm ? sq[j] : 0.0);
        }
        __syncthreads();
        if (w.active[0]) {
            int unused;
            if constexpr (!fast64<KT>()) near64_any<KT, PP>(acc, t, w.slice, w.slices, cm, o, k);
            else if (PP && KT != K_REGCOULOMB && test) near64_skip<KT>(acc, t, w.slice, w.slices, cmp, o, k);
            else if (w.slices == 1) near64<KT, false>(acc, t, 0, 1, cmp, o, k, unused);
            else near64<KT, false>(acc, t, w.slice, w.slices, cmp, o, k, unused);
        }
        __syncthreads();
    }
}

// The sum of one thread again with the library functions, which take every
// argument: its share of the clusters a0..a1-1 and the source nodes d0..d1-1.
template <int KT, bool HERM, bool PP>
__device__ __noinline__ double again64(int n, const int *a_idx, int64_t a0, int64_t a1, const int *d_idx, int64_t d0,
                                       int64_t d1, const int *s_ibeg, const int *s_numpar, const double *s_grid,
                                       const double *Q, const double *sx, const double *sy, const double *sz,
                                       const double *sq, double kp, double x, double y, double z, int slice, int slices)
{
    const int np1 = n + 1, P = np1 * np1 * np1;
    double acc = 0.0;
    for (int64_t e = a0; e < a1; e++) {
        const double *g = s_grid + (size_t)a_idx[e] * 3 * np1, *q = Q + (size_t)a_idx[e] * (HERM ? 8 * P : P);
        for (int row = slice; row < np1 * np1; row += slices)
            for (int i = 0; i < np1; i++) {
                const int k3 = row / np1, k2 = row - k3 * np1, j = row * np1 + i;
                const double dx = x - g[i], dy = y - g[np1 + k2], dz = z - g[2 * np1 + k3];
                acc += HERM ? k_pc_herm<KT>(dx, dy, dz, q + j, P, kp) : k_any<KT, false>(dx, dy, dz, q[j], kp, 0.0);
            }
    }
    for (int64_t e = d0; e < d1; e++) {
        const int s = d_idx[e] & ~EV_MEETS, sb = s_ibeg[s], sn = s_numpar[s];
        for (int c0 = 0; c0 < sn; c0 += EV_TILE)
            for (int i = c0 + slice; i < min(sn, c0 + EV_TILE); i += slices)
                acc += k_any<KT, PP>(x - sx[sb + i], y - sy[sb + i], z - sz[sb + i], sq[sb + i], kp, 0.0);
    }
    return acc;
}

// acc of slice 0: the sum over the slices in order (all threads call).
__device__ __forceinline__ void sum_slices(double *acc, double *red, const Lanes &w)
{
    if (w.slices == 1) return;
#pragma unroll
    for (int b = 0; b < 2; b++) red[b * EV_THREADS + threadIdx.x] = acc[b];
    __syncthreads();
    if (w.slice == 0)
        for (int s = 1; s < w.slices; s++)
#pragma unroll
            for (int b = 0; b < 2; b++) acc[b] += red[b * EV_THREADS + s * w.lanes + w.lane];
    __syncthreads();
}

// Particle outputs: PC (clusters) + PP (particles) onto a chunk of a target
// leaf.  NP1 = n + 1 (Lagrange with a short form), else 0.
template <int KT, int NP1, bool HERM, bool FAR>
__global__ void __launch_bounds__(EV_THREADS, EV_MINB) k_eval_targets(const __grid_constant__ EvalTargetsArgs a)
{
    extern __shared__ __align__(16) double sm[];
    __shared__ double red[2 * EV_THREADS];
    __shared__ double2 tab[KT == K_YUKAWA ? EXP64_TAB : 1];
    const Kern64<FAR> k = kern64_make<KT, FAR>(a.kp, a.kp2, tab);
    const int2 it = a.items[blockIdx.x];
    const int u = it.x, tnode = a.leaf_node[u];
    const Lanes w(min(EV_CHUNK, a.t_numpar[tnode] - it.y * EV_CHUNK));
    const int t0 = a.t_ibeg[tnode] + it.y * EV_CHUNK;
    Out2 o;
#pragma unroll
    for (int b = 0; b < 2; b++) {
        const int t = t0 + w.out(b);
        o.x[b] = a.tx[t]; o.y[b] = a.ty[t]; o.z[b] = a.tz[t];
    }
    const int np1 = NP1 ? NP1 : a.n + 1, P = np1 * np1 * np1, nq = HERM ? 8 * P : P;
    const int64_t ab = a.a_off[u], ae = a.a_off[u + 1], db = a.d_off[u], de = a.d_off[u + 1];
    const int seg0 = a.partial ? blockIdx.y : 0, seg1 = a.partial ? blockIdx.y + 1 : EV_SEGS;
    double total[2] = {0.0, 0.0};
    for (int seg = seg0; seg < seg1; seg++) {
        const int64_t a0 = seg_begin(ab, ae, seg), a1 = seg_begin(ab, ae, seg + 1);
        const int64_t d0 = seg_begin(db, de, seg), d1 = seg_begin(db, de, seg + 1);
        double acc[2] = {0.0, 0.0};
        for (int64_t e = k.lib ? a1 : a0; e < a1; e++) {
            const int s = a.a_idx[e];
            double *g = sm, *q = sm + 3 * np1;
            for (int i = threadIdx.x; i < 3 * np1; i += EV_THREADS) g[i] = a.s_grid[(size_t)s * 3 * np1 + i];
            if constexpr (HERM && fast64<KT>()) {
                // a point's moments side by side, after the grid's 3 np1 rounded up to 16 bytes
                q = sm + 3 * np1 + (np1 & 1);
                for (int i = threadIdx.x; i < nq; i += EV_THREADS)
                    q[i] = a.Q[(size_t)s * nq + (i & 7) * P + (i >> 3)] * herm64_scale(i & 7);
            } else {
                for (int i = threadIdx.x; i < nq; i += EV_THREADS) q[i] = a.Q[(size_t)s * nq + i];
            }
            __syncthreads();
            if (w.active[0]) {
                if constexpr (HERM && fast64<KT>()) herm64<KT>(acc, np1, g, q, o, w, k);
                else if constexpr (HERM) herm64_any<KT>(acc, np1, g, q, o, w, k);
                else if constexpr (NP1 > 0) far64<KT, NP1>(acc, g, q, o, w, k);
                else far64_any<KT>(acc, np1, g, q, o, w, k);
            }
            __syncthreads();
        }
        const Tile64 tile{reinterpret_cast<double2 *>(sm), reinterpret_cast<double2 *>(sm) + EV_TILE};
        for (int64_t e = k.lib ? d1 : d0; e < d1; e++) {
            const int v = a.d_idx[e], s = v & ~EV_MEETS;
            near64_node<KT, true>(acc, tile, a.s_ibeg[s], a.s_numpar[s], a.sx, a.sy, a.sz, a.sq, (v & EV_MEETS) != 0, o,
                                  w, k);
        }
        if constexpr (fast64<KT>()) {
#pragma unroll
            for (int b = 0; b < 2; b++)
                if (w.active[b] && (k.lib || !isfinite(acc[b])))
                    acc[b] = again64<KT, HERM, true>(a.n, a.a_idx, a0, a1, a.d_idx, d0, d1, a.s_ibeg, a.s_numpar, a.s_grid,
                                                     a.Q, a.sx, a.sy, a.sz, a.sq, a.kp, o.x[b], o.y[b], o.z[b], w.slice,
                                                     w.slices);
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

// Grid outputs: M2L (clusters, Lagrange) + CP (particles) onto a chunk of a
// target node's grid points.
template <int KT, int NP1, bool FAR>
__global__ void __launch_bounds__(EV_THREADS, EV_MINB) k_eval_grids(const __grid_constant__ EvalGridsArgs a)
{
    extern __shared__ __align__(16) double sm[];
    __shared__ double red[2 * EV_THREADS];
    __shared__ double2 tab[KT == K_YUKAWA ? EXP64_TAB : 1];
    const Kern64<FAR> k = kern64_make<KT, FAR>(a.kp, a.kp2, tab);
    const int2 it = a.items[blockIdx.x];
    const int T = it.x, np1 = NP1 ? NP1 : a.n + 1, P = np1 * np1 * np1;
    const Lanes w(min(EV_CHUNK, P - it.y * EV_CHUNK));
    const double *tg = a.t_grid + (size_t)T * 3 * np1;
    Out2 o;
#pragma unroll
    for (int b = 0; b < 2; b++) {
        const int j = it.y * EV_CHUNK + w.out(b);
        o.x[b] = tg[j % np1]; o.y[b] = tg[np1 + (j / np1) % np1]; o.z[b] = tg[2 * np1 + j / (np1 * np1)];
    }
    const int64_t cb = a.c_off[T], ce = a.c_off[T + 1], pb = a.p_off[T], pe = a.p_off[T + 1];
    const int seg0 = a.partial ? blockIdx.y : 0, seg1 = a.partial ? blockIdx.y + 1 : EV_SEGS;
    double total[2] = {0.0, 0.0};
    for (int seg = seg0; seg < seg1; seg++) {
        const int64_t c0 = seg_begin(cb, ce, seg), c1 = seg_begin(cb, ce, seg + 1);
        const int64_t p0 = seg_begin(pb, pe, seg), p1 = seg_begin(pb, pe, seg + 1);
        double acc[2] = {0.0, 0.0};
        for (int64_t e = k.lib ? c1 : c0; e < c1; e++) {
            const int s = a.c_idx[e];
            double *g = sm, *q = sm + 3 * np1;
            for (int i = threadIdx.x; i < 3 * np1; i += EV_THREADS) g[i] = a.s_grid[(size_t)s * 3 * np1 + i];
            for (int i = threadIdx.x; i < P; i += EV_THREADS) q[i] = a.Q[(size_t)s * P + i];
            __syncthreads();
            if (w.active[0]) {
                if constexpr (NP1 > 0) far64<KT, NP1>(acc, g, q, o, w, k);
                else far64_any<KT>(acc, np1, g, q, o, w, k);
            }
            __syncthreads();
        }
        const Tile64 tile{reinterpret_cast<double2 *>(sm), reinterpret_cast<double2 *>(sm) + EV_TILE};
        for (int64_t e = k.lib ? p1 : p0; e < p1; e++) {
            const int s = a.p_idx[e];
            near64_node<KT, false>(acc, tile, a.s_ibeg[s], a.s_numpar[s], a.sx, a.sy, a.sz, a.sq, false, o, w, k);
        }
        if constexpr (fast64<KT>()) {
#pragma unroll
            for (int b = 0; b < 2; b++)
                if (w.active[b] && (k.lib || !isfinite(acc[b])))
                    acc[b] = again64<KT, false, false>(a.n, a.c_idx, c0, c1, a.p_idx, p0, p1, a.s_ibeg, a.s_numpar, a.s_grid,
                                                       a.Q, a.sx, a.sy, a.sz, a.sq, a.kp, o.x[b], o.y[b], o.z[b],
                                                       w.slice, w.slices);
        }
        sum_slices(acc, red, w);
#pragma unroll
        for (int b = 0; b < 2; b++) {
            total[b] += acc[b];
            if (a.partial && w.active[b] && w.slice == 0)
                a.partial[(size_t)seg * a.pstride + (size_t)T * P + it.y * EV_CHUNK + w.out(b)] = acc[b];
        }
    }
#pragma unroll
    for (int b = 0; b < 2; b++)
        if (!a.partial && w.active[b] && w.slice == 0) a.Phi[(size_t)T * P + it.y * EV_CHUNK + w.out(b)] = total[b];
}

// Direct sum: sources blockIdx.y of gridDim.y parts onto EV_CHUNK targets;
// several parts go to `out` nt apart and are added by k_sum_parts.
template <int KT>
__global__ void __launch_bounds__(EV_THREADS, EV_MINB)
k_direct(int nt, int ns, const double *__restrict__ tx, const double *__restrict__ ty, const double *__restrict__ tz,
         const double *__restrict__ sx, const double *__restrict__ sy, const double *__restrict__ sz,
         const double *__restrict__ sq, double kp, double kp2, double *__restrict__ out)
{
    __shared__ double2 xy[EV_TILE], zq[EV_TILE];
    __shared__ double red[2 * EV_THREADS];
    __shared__ double2 tab[KT == K_YUKAWA ? EXP64_TAB : 1];
    const Kern64<true> k = kern64_make<KT, true>(kp, kp2, tab);      // the extent is not known
    const int t0 = blockIdx.x * EV_CHUNK;
    const Lanes w(min(EV_CHUNK, nt - t0));
    Out2 o;
#pragma unroll
    for (int b = 0; b < 2; b++) {
        const int t = t0 + w.out(b);
        o.x[b] = tx[t]; o.y[b] = ty[t]; o.z[b] = tz[t];
    }
    const int s0 = (int)((int64_t)ns * blockIdx.y / gridDim.y), s1 = (int)((int64_t)ns * (blockIdx.y + 1) / gridDim.y);
    const Tile64 tile{xy, zq};
    double acc[2] = {0.0, 0.0};
    near64_node<KT, true>(acc, tile, s0, k.lib ? 0 : s1 - s0, sx, sy, sz, sq, true, o, w, k);
    if constexpr (fast64<KT>()) {
        for (int b = 0; b < 2; b++)
            if (w.active[b] && (k.lib || !isfinite(acc[b]))) {
                acc[b] = 0.0;
                for (int c0 = s0; c0 < s1; c0 += EV_TILE)
                    for (int i = c0 + w.slice; i < min(s1, c0 + EV_TILE); i += w.slices)
                        acc[b] += k_any<KT, true>(o.x[b] - sx[i], o.y[b] - sy[i], o.z[b] - sz[i], sq[i], kp, kp2);
            }
    }
    sum_slices(acc, red, w);
#pragma unroll
    for (int b = 0; b < 2; b++)
        if (w.active[b] && w.slice == 0) out[(size_t)blockIdx.y * nt + t0 + w.out(b)] = acc[b];
}

// ---------------------------------------------------------------------------
// launchers of one kernel type
// ---------------------------------------------------------------------------
template <typename K, typename A>
void eval64_launch(K kernel, const A &a, size_t far_doubles, cudaStream_t st)
{
    const size_t near_bytes = 2 * sizeof(double2) * EV_TILE, far_bytes = sizeof(double) * far_doubles;
    const size_t sm = far_bytes > near_bytes ? far_bytes : near_bytes;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    kernel<<<dim3(a.nitems, a.partial ? EV_SEGS : 1), EV_THREADS, sm, st>>>(a);
}

template <int KT, bool FAR>
void eval_targets_kt(bool hermite, const EvalTargetsArgs &a, cudaStream_t st)
{
    const size_t np1 = a.n + 1, P = np1 * np1 * np1;
    if constexpr (fast64<KT>() || KT == K_SINOVERR)
        if (hermite) {
            eval64_launch(k_eval_targets<KT, 0, true, FAR>, a, 3 * np1 + 1 + 8 * P, st);
            return;
        }
    if constexpr (fast64<KT>()) {
        switch (np1) {
#define BT_EV(N) case N: eval64_launch(k_eval_targets<KT, N, false, FAR>, a, 3 * np1 + P, st); return;
            BT_EV(2) BT_EV(3) BT_EV(4) BT_EV(5) BT_EV(6) BT_EV(7) BT_EV(8) BT_EV(9) BT_EV(10) BT_EV(11) BT_EV(12)
            BT_EV(13)
#undef BT_EV
        }
    } else {
        eval64_launch(k_eval_targets<KT, 0, false, FAR>, a, 3 * np1 + P, st);
    }
}

template <int KT, bool FAR>
void eval_grids_kt(const EvalGridsArgs &a, cudaStream_t st)
{
    const size_t np1 = a.n + 1, P = np1 * np1 * np1;
    if constexpr (fast64<KT>()) {
        switch (np1) {
#define BT_EV(N) case N: eval64_launch(k_eval_grids<KT, N, FAR>, a, 3 * np1 + P, st); return;
            BT_EV(2) BT_EV(3) BT_EV(4) BT_EV(5) BT_EV(6) BT_EV(7) BT_EV(8) BT_EV(9) BT_EV(10) BT_EV(11) BT_EV(12)
            BT_EV(13)
#undef BT_EV
        }
    } else {
        eval64_launch(k_eval_grids<KT, 0, FAR>, a, 3 * np1 + P, st);
    }
}

template <int KT>
void direct_kt(int nt, int ns, int parts, const double *tx, const double *ty, const double *tz, const double *sx,
               const double *sy, const double *sz, const double *sq, double kp, double kp2, double *out, cudaStream_t st)
{
    k_direct<KT><<<dim3((nt + EV_CHUNK - 1) / EV_CHUNK, parts), EV_THREADS, 0, st>>>(nt, ns, tx, ty, tz, sx, sy, sz, sq,
                                                                                     kp, kp2, out);
}

#define BT_EVAL64_INSTANTIATE(KT, FAR)                                                                               \
    template void eval_targets_kt<KT, FAR>(bool, const EvalTargetsArgs &, cudaStream_t);                             \
    template void eval_grids_kt<KT, FAR>(const EvalGridsArgs &, cudaStream_t);
#define BT_EVAL64_INSTANTIATE_DIRECT(KT)                                                                             \
    template void direct_kt<KT>(int, int, int, const double *, const double *, const double *, const double *,        \
                                const double *, const double *, const double *, double, double, double *, cudaStream_t);

}  // namespace bt
