// bt_mixed.cu -- mixed-precision evaluation kernels of barytree_b200.
//
// Arithmetic: every kernel evaluation (PP, PC, CP, M2L) runs in FP32 on
// coordinates relative to the centre of the target leaf / node, so FP32 only
// ever sees displacements of the size of the interaction, never absolute
// positions.  Centre offsets between the two sides of an interaction are
// formed in FP64 and rounded once.  Per-interaction partial sums are FP32
// (far field: Kahan-compensated per grid row); they are folded into an FP64
// per-target accumulator after every list entry / tile, which is the FP64
// far+near reduction.  Tree boxes, Chebyshev node placement, exact-node
// coincidence tests and the barycentric passes stay FP64 (bt_device.cu).
//
// Throughput: the kernels are issue-bound, so each thread evaluates two
// targets against every shared-memory value it loads, the coincidence test
// of the skipping kernels runs only for source leaves whose box overlaps the
// target leaf's box, and the special functions are single MUFU instructions
// (rsqrt.approx / ex2.approx, flush-to-zero).  The far-field loops are
// instantiated per degree (NP1 = n+1) so one axis of grid coordinates lives
// in registers.
#include <cuda_runtime.h>

#include <cfloat>
#include <cstdint>

#include "bt_device.h"
#include "bt_f2.cuh"
#include "bt_kernels.cuh"
#include "bt_mixed.h"

namespace bt {

// Kernel value for a well-separated pair.  kc: Yukawa -kappa*log2(e);
// regularised Coulomb eps^2; unused for Coulomb.
template <int KT>
__device__ __forceinline__ float kf_far(float r2, float q, float kc)
{
    if (KT == 1) {
        return q * rsqrt_apx(r2);
    } else if (KT == 2) {
        // one Newton step on 1/r (the MUFU estimate's error would otherwise
        // enter both 1/r and the exponent); the FMA pipe has room for it here
        float rinv = rsqrt_apx(r2);
        float h = r2 * rinv;
        float t = fmaf(-0.5f * h, rinv, 1.5f);
        float e = ex2_apx(kc * (h * t));
        return (q * (rinv * t)) * e;
    } else {
        return q * rsqrt_apx(r2 + kc);
    }
}

__device__ __forceinline__ void kahan_add(float &s, float &c, float v)
{
    float y = v - c;
    float t = s + y;
    c = (t - s) - y;
    s = t;
}

constexpr int MX_THREADS = 128;                 // threads of the grid-output kernel
constexpr int MX_MIN_BLOCKS = 6;                // its resident blocks per SM (8 measured the same)
constexpr int MX_TILE = 1024;                   // sources per tile of the grid-output kernel
// Register budget of the 2-targets-per-thread Lagrange particle-output
// kernel (Coulomb, regularised Coulomb): room for 6 resident blocks per SM.
// Left to itself the compiler takes 94 registers (5 blocks) for the packed
// far field, which measured 21 % slower on the 16M system; at 80 registers
// (a few bytes of spill) it runs 1.4 % faster than the scalar far field.
#ifndef BT_MX_MIN_BLOCKS_T2
#define BT_MX_MIN_BLOCKS_T2 6
#endif
// Yukawa: 6 blocks (80 registers, 24 bytes of spill) measured 2 % faster
// than the compiler's 96 registers on the 1M cluster-cluster system; for the
// Hermite kernels 5 blocks measured the same as the compiler's choice.
#ifndef BT_MX_MIN_BLOCKS_YUK
#define BT_MX_MIN_BLOCKS_YUK 6
#endif
#ifndef BT_MX_MIN_BLOCKS_HERM
#define BT_MX_MIN_BLOCKS_HERM 0
#endif
// resident-block budget of the 2-targets-per-thread kernel (0: the compiler's choice)
template <int KT, bool HERM>
__host__ __device__ constexpr int rb_blocks()
{
    return HERM ? BT_MX_MIN_BLOCKS_HERM : KT == 2 ? BT_MX_MIN_BLOCKS_YUK : BT_MX_MIN_BLOCKS_T2;
}

// Grid points of each row of the Lagrange far field (Coulomb and
// regularised Coulomb) whose 1/r comes from rsqrt_sw / f2_rsqrt_sw on the
// FP32 and integer pipes instead of the MUFU: the first BT_FAR_SW of the
// row's n+1 (k1 < BT_FAR_SW).  A far-field value needs only two FP32
// operations besides its 1/r, so the FP32 pipe has room that the MUFU
// lacks, but less than that count suggests: on the 16M clustered system
// (degrees 4 to 11, mostly 5 to 7) the evaluation took 819.8 ms with none
// on the FP32 pipe, 802.7 ms with one per row of up to 8, and 829, 863
// and 919 ms with 2, 3 and 4 of 8 (same rel-L2, 1.0e-7).  Both forms round
// alike lane by lane, so every tile shape still gives the same bits.
#ifndef BT_FAR_SW
#define BT_FAR_SW 1
#endif
__host__ __device__ constexpr bool far_sw(int k1) { return k1 < BT_FAR_SW; }

// Yukawa: row + q exp(-kappa r) / r, one Newton step on the MUFU's 1/r (its
// error would otherwise enter both 1/r and the exponent).
__device__ __forceinline__ float far_yukawa(float r2, float q, float kc, float row)
{
    const float rinv = rsqrt_apx(r2), h = r2 * rinv;
    const float t = fmaf(-0.5f * h, rinv, 1.5f);
    return fmaf(q * (rinv * t), ex2_apx(kc * (h * t)), row);
}
__device__ __forceinline__ f2_t f2_far_yukawa(f2_t r2, f2_t q, f2_t kc, f2_t row)
{
    float a, b;
    f2_split(r2, a, b);
    const f2_t rinv = f2_make(rsqrt_apx(a), rsqrt_apx(b)), h = f2_mul(r2, rinv);
    const f2_t t = f2_fma(f2_mul(f2_make(-0.5f, -0.5f), h), rinv, f2_make(1.5f, 1.5f));
    f2_split(f2_mul(kc, f2_mul(h, t)), a, b);
    const f2_t e = f2_make(ex2_apx(a), ex2_apx(b));
    return f2_fma(f2_mul(q, f2_mul(rinv, t)), e, row);
}

// Far field of one source cluster (degree NP1-1) for NT targets at (x,y,z),
// relative to the target centre; g = grid coordinates relative to the same
// centre, q = proxy charges (shared memory, FP32).
template <int KT, int NP1, int NT>
__device__ __forceinline__ void pc_cluster(const float *x, const float *y, const float *z, const float *g,
                                           const float *q, float kc, float *out)
{
    float gx[NT][NP1];
#pragma unroll
    for (int t = 0; t < NT; t++)
#pragma unroll
        for (int k = 0; k < NP1; k++) gx[t][k] = x[t] - g[k];
    float s[NT], c[NT];
#pragma unroll
    for (int t = 0; t < NT; t++) { s[t] = 0.f; c[t] = 0.f; }
    int j = 0;
    for (int k3 = 0; k3 < NP1; k3++) {
        float gz = g[2 * NP1 + k3];
        for (int k2 = 0; k2 < NP1; k2++) {
            float gy = g[NP1 + k2];
            float dyz[NT], row[NT];
#pragma unroll
            for (int t = 0; t < NT; t++) {
                float dy = y[t] - gy, dz = z[t] - gz;
                dyz[t] = fmaf(dy, dy, KT == 3 ? fmaf(dz, dz, kc) : dz * dz);     // regularised: + eps^2
                row[t] = 0.f;
            }
#pragma unroll
            for (int k1 = 0; k1 < NP1; k1++) {
                float qq = q[j + k1];
#pragma unroll
                for (int t = 0; t < NT; t++) {
                    const float r2 = fmaf(gx[t][k1], gx[t][k1], dyz[t]);
                    if (KT == 2) row[t] = far_yukawa(r2, qq, kc, row[t]);
                    else row[t] = fmaf(qq, far_sw(k1) ? rsqrt_sw(r2) : rsqrt_apx(r2), row[t]);
                }
            }
            j += NP1;
#pragma unroll
            for (int t = 0; t < NT; t++) kahan_add(s[t], c[t], row[t]);
        }
    }
#pragma unroll
    for (int t = 0; t < NT; t++) out[t] = s[t] - c[t];
}

// Hermite far field of one source cluster for NT targets (FP32; moments
// q[8 * j + m] of grid point j, m = 0..7 in the reference's order q, qx, qy,
// qz, qxy, qyz, qxz, qxyz, with qxy..qxz pre-multiplied by 3 and qxyz by 15
// when staged).  Moments P apart took eight shared-memory reads per point,
// which the load pipe served more slowly than the FP32 pipe its arithmetic.
// The terms of K_*_PC_Hermite (src/kernels/coulomb/coulomb_pc.c:66-138,
// yukawa/yukawa_pc.c, regularized-coulomb/regularized-coulomb_pc.c):
//   r^-1 q + r^-3 (qx dx + qy dy + qz dz) + 3 r^-5 (qxy dx dy + qyz dy dz
//   + qxz dx dz) + 15 r^-7 qxyz dx dy dz, Yukawa with exp(-kappa r) and the
//   polynomials in kappa r.  Evaluated as 1/r (E + dx u F) with u = 1/r^2 and
//   E, F nested in u: 14 FP32 operations besides 1/r (19 when every term
//   formed its power of 1/r and its product of differences).
//   Kahan-compensated per grid row.
template <int KT, int NP1, int NT>
__device__ __forceinline__ void pc_cluster_herm(const float *x, const float *y, const float *z, const float *g,
                                                const float *q, float kc, float kp, float *out)
{
    float gx[NT][NP1];
#pragma unroll
    for (int t = 0; t < NT; t++)
#pragma unroll
        for (int k = 0; k < NP1; k++) gx[t][k] = x[t] - g[k];
    float s[NT], c[NT];
#pragma unroll
    for (int t = 0; t < NT; t++) { s[t] = 0.f; c[t] = 0.f; }
    int j = 0;
    for (int k3 = 0; k3 < NP1; k3++) {
        const float gz = g[2 * NP1 + k3];
        for (int k2 = 0; k2 < NP1; k2++) {
            const float gy = g[NP1 + k2];
            float dy[NT], dz[NT], dyz[NT], dydz[NT], row[NT];
#pragma unroll
            for (int t = 0; t < NT; t++) {
                dy[t] = y[t] - gy;
                dz[t] = z[t] - gz;
                dyz[t] = fmaf(dy[t], dy[t], dz[t] * dz[t]);
                if (KT == 3) dyz[t] += kc;
                dydz[t] = dy[t] * dz[t];
                row[t] = 0.f;
            }
#pragma unroll
            for (int k1 = 0; k1 < NP1; k1++) {
                const int jj = j + k1;
                const float4 qa = *reinterpret_cast<const float4 *>(q + 8 * jj),
                             qb = *reinterpret_cast<const float4 *>(q + 8 * jj + 4);
                const float q0 = qa.x, q1 = qa.y, q2 = qa.z, q3 = qa.w, q4 = qb.x, q5 = qb.y, q6 = qb.z, q7 = qb.w;
#pragma unroll
                for (int t = 0; t < NT; t++) {
                    const float dx = gx[t][k1];
                    const float r2 = fmaf(dx, dx, dyz[t]);
                    const float rinv = rsqrt_apx(r2);
                    // sorted by powers of dx: E + dx u F, u = 1/r^2
                    const float u = rinv * rinv, du = dx * u;
                    if (KT == 2) {
                        // Yukawa: exp(-kappa r) (r^-1 q + r^-3 (1 + kr) a1 + r^-5 (3 + 3kr + k^2r^2) a2
                        // + r^-7 (15 + 15kr + 6k^2r^2 + k^3r^3) a3), with a2, a3 staged x3, x15
                        const float r = r2 * rinv, kr = kp * r, kr2 = kr * kr;
                        const float e = ex2_apx(kc * r);
                        const float p1 = 1.0f + kr;
                        const float p2 = fmaf(kr2, 1.0f / 3.0f, p1);                    // (3 + 3kr + k^2r^2) / 3
                        const float p3 = fmaf(kr2 * kr, 1.0f / 15.0f, fmaf(kr2, 0.4f, p1));  // (15 + 15kr + 6k^2r^2 + k^3r^3) / 15
                        const float b1 = fmaf(u * p2, q5 * dydz[t], p1 * fmaf(q3, dz[t], q2 * dy[t]));
                        const float b2 = fmaf(u * p3, q7 * dydz[t], p2 * fmaf(q6, dz[t], q4 * dy[t]));
                        row[t] = fmaf(rinv * e, fmaf(du, fmaf(u, b2, p1 * q1), fmaf(u, b1, q0)), row[t]);
                    } else {
                        const float v = u * dydz[t];
                        const float E = fmaf(u, fmaf(q5, v, fmaf(q3, dz[t], q2 * dy[t])), q0);
                        const float F = fmaf(u, fmaf(q7, v, fmaf(q6, dz[t], q4 * dy[t])), q1);
                        row[t] = fmaf(rinv, fmaf(du, F, E), row[t]);
                    }
                }
            }
            j += NP1;
#pragma unroll
            for (int t = 0; t < NT; t++) kahan_add(s[t], c[t], row[t]);
        }
    }
#pragma unroll
    for (int t = 0; t < NT; t++) out[t] = s[t] - c[t];
}

// Near-field tiles.  FP32 leaf-relative coordinates carry an absolute error
// of about 6e-8 of the leaf size, a large relative error for a pair much
// closer than the leaf size, and such a pair dominates its target's
// potential.  Pairs closer than MX_CLOSE_FRAC of the two leaves' summed
// radii ("close pairs") are therefore left out of the FP32 sums and added in
// FP64 from the FP64 coordinates and charges, straight into the FP64
// per-target accumulator (an FP32 sum would also round every later term at
// the close pair's magnitude).  Close pairs occur only between leaves whose
// boxes lie within that distance (flagged per near-field entry); the other
// entries run pp_tile_far with no test at all.

// Lagrange far field with the targets in packed pairs (NT even): pc_cluster's operations lane by lane in f32x2
// instructions (identical results); qd holds each proxy charge twice.
template <int KT, int NP1, int NT>
__device__ __forceinline__ void pc_cluster_f2(const float *x, const float *y, const float *z, const float *g,
                                              const f2_t *qd, float kc, float *out)
{
    constexpr int NPR = NT / 2;
    f2_t gx[NPR][NP1];
#pragma unroll
    for (int p = 0; p < NPR; p++)
#pragma unroll
        for (int k = 0; k < NP1; k++) gx[p][k] = f2_make(x[2 * p] - g[k], x[2 * p + 1] - g[k]);
    float s[NT], c[NT];
#pragma unroll
    for (int t = 0; t < NT; t++) { s[t] = 0.f; c[t] = 0.f; }
    const f2_t kc2 = f2_make(kc, kc), zero = f2_make(0.0f, 0.0f);
    int j = 0;
    for (int k3 = 0; k3 < NP1; k3++) {
        const float gz = g[2 * NP1 + k3];
        for (int k2 = 0; k2 < NP1; k2++) {
            const float gy = g[NP1 + k2];
            f2_t dyz[NPR], row[NPR];
#pragma unroll
            for (int p = 0; p < NPR; p++) {
                const f2_t dy = f2_make(y[2 * p] - gy, y[2 * p + 1] - gy), dz = f2_make(z[2 * p] - gz, z[2 * p + 1] - gz);
                dyz[p] = f2_fma(dy, dy, KT == 3 ? f2_fma(dz, dz, kc2) : f2_mul(dz, dz));
                row[p] = zero;
            }
#pragma unroll
            for (int k1 = 0; k1 < NP1; k1++) {
                const f2_t qq = qd[j + k1];
#pragma unroll
                for (int p = 0; p < NPR; p++) {
                    const f2_t r2 = f2_fma(gx[p][k1], gx[p][k1], dyz[p]);
                    if (KT == 2) {
                        row[p] = f2_far_yukawa(r2, qq, kc2, row[p]);
                    } else if (far_sw(k1)) {      // resolved at compile time: k1 is unrolled
                        row[p] = f2_fma(qq, f2_rsqrt_sw(r2), row[p]);
                    } else {
                        float a, b;
                        f2_split(r2, a, b);
                        row[p] = f2_fma(qq, f2_make(rsqrt_apx(a), rsqrt_apx(b)), row[p]);
                    }
                }
            }
            j += NP1;
#pragma unroll
            for (int p = 0; p < NPR; p++) {
                float lo, hi;
                f2_split(row[p], lo, hi);
                kahan_add(s[2 * p], c[2 * p], lo);
                kahan_add(s[2 * p + 1], c[2 * p + 1], hi);
            }
        }
    }
#pragma unroll
    for (int t = 0; t < NT; t++) out[t] = s[t] - c[t];
}

// Hermite far field with the targets in packed pairs (NT even, Coulomb and
// regularised Coulomb): the same operations as pc_cluster_herm lane by lane,
// in f32x2 instructions, so the results are identical and the FMA-pipe work
// per evaluation halves.  qd holds each moment twice ({q, q}, same staging
// scales as pc_cluster_herm).
template <int KT, int NP1, int NT>
__device__ __forceinline__ void pc_cluster_herm_f2(const float *x, const float *y, const float *z, const float *g,
                                                   const f2_t *qd, float kc, float *out)
{
    constexpr int NPR = NT / 2;
    f2_t gx[NPR][NP1];
#pragma unroll
    for (int p = 0; p < NPR; p++)
#pragma unroll
        for (int k = 0; k < NP1; k++) gx[p][k] = f2_make(x[2 * p] - g[k], x[2 * p + 1] - g[k]);
    float s[NT], c[NT];
#pragma unroll
    for (int t = 0; t < NT; t++) { s[t] = 0.f; c[t] = 0.f; }
    const f2_t kc2 = f2_make(kc, kc), one = f2_make(1.0f, 1.0f), zero = f2_make(0.0f, 0.0f);
    int j = 0;
    for (int k3 = 0; k3 < NP1; k3++) {
        const float gz = g[2 * NP1 + k3];
        for (int k2 = 0; k2 < NP1; k2++) {
            const float gy = g[NP1 + k2];
            f2_t dy[NPR], dz[NPR], dyz[NPR], dydz[NPR], row[NPR];
#pragma unroll
            for (int p = 0; p < NPR; p++) {
                dy[p] = f2_make(y[2 * p] - gy, y[2 * p + 1] - gy);
                dz[p] = f2_make(z[2 * p] - gz, z[2 * p + 1] - gz);
                dyz[p] = f2_fma(dy[p], dy[p], f2_mul(dz[p], dz[p]));
                if (KT == 3) dyz[p] = f2_fma(one, kc2, dyz[p]);
                dydz[p] = f2_mul(dy[p], dz[p]);
                row[p] = zero;
            }
#pragma unroll
            for (int k1 = 0; k1 < NP1; k1++) {
                const int jj = j + k1;
                const ulonglong2 *qv = reinterpret_cast<const ulonglong2 *>(qd + 8 * jj);
                const ulonglong2 qa = qv[0], qb = qv[1], qc = qv[2], qe = qv[3];
                const f2_t q0 = qa.x, q1 = qa.y, q2 = qb.x, q3 = qb.y, q4 = qc.x, q5 = qc.y, q6 = qe.x, q7 = qe.y;
#pragma unroll
                for (int p = 0; p < NPR; p++) {
                    const f2_t dx = gx[p][k1];
                    const f2_t r2 = f2_fma(dx, dx, dyz[p]);
                    float ra, rb;
                    f2_split(r2, ra, rb);
                    const f2_t rinv = f2_make(rsqrt_apx(ra), rsqrt_apx(rb));
                    const f2_t u = f2_mul(rinv, rinv), v = f2_mul(u, dydz[p]);
                    const f2_t E = f2_fma(u, f2_fma(q5, v, f2_fma(q3, dz[p], f2_mul(q2, dy[p]))), q0);
                    const f2_t F = f2_fma(u, f2_fma(q7, v, f2_fma(q6, dz[p], f2_mul(q4, dy[p]))), q1);
                    row[p] = f2_fma(rinv, f2_fma(f2_mul(dx, u), F, E), row[p]);
                }
            }
            j += NP1;
#pragma unroll
            for (int p = 0; p < NPR; p++) {
                float lo, hi;
                f2_split(row[p], lo, hi);
                kahan_add(s[2 * p], c[2 * p], lo);
                kahan_add(s[2 * p + 1], c[2 * p + 1], hi);
            }
        }
    }
#pragma unroll
    for (int t = 0; t < NT; t++) out[t] = s[t] - c[t];
}

// Packed far field for this kernel type and target count?  (Hermite: not for Yukawa.)
template <int KT, bool HERM, int NT>
__host__ __device__ constexpr bool far_packed() { return !(HERM && KT == 2) && NT % 2 == 0; }

// q: the staged proxy charges, as {q, q} pairs when far_packed().
template <int KT, int NT>
__device__ void pc_cluster_dispatch(int np1, const float *x, const float *y, const float *z, const float *g,
                                    const float *q, float kc, float *out)
{
    switch (np1) {
#define BT_CASE(N)                                                                                         \
    case N:                                                                                                \
        if constexpr (far_packed<KT, false, NT>())                                                         \
            pc_cluster_f2<KT, N, NT>(x, y, z, g, reinterpret_cast<const f2_t *>(q), kc, out);              \
        else                                                                                               \
            pc_cluster<KT, N, NT>(x, y, z, g, q, kc, out);                                                 \
        return;
        BT_CASE(2) BT_CASE(3) BT_CASE(4) BT_CASE(5) BT_CASE(6) BT_CASE(7) BT_CASE(8)
        BT_CASE(9) BT_CASE(10) BT_CASE(11) BT_CASE(12) BT_CASE(13)
#undef BT_CASE
    }
#pragma unroll
    for (int t = 0; t < NT; t++) out[t] = 0.f;
}


// q: the staged moments, as {q, q} pairs when far_packed().
template <int KT, int NT>
__device__ void pc_cluster_herm_dispatch(int np1, const float *x, const float *y, const float *z, const float *g,
                                         const float *q, float kc, float kp, float *out)
{
    switch (np1) {
#define BT_CASE(N)                                                                                         \
    case N:                                                                                                \
        if constexpr (far_packed<KT, true, NT>())                                                         \
            pc_cluster_herm_f2<KT, N, NT>(x, y, z, g, reinterpret_cast<const f2_t *>(q), kc, out);         \
        else                                                                                               \
            pc_cluster_herm<KT, N, NT>(x, y, z, g, q, kc, kp, out);                                        \
        return;
        BT_CASE(2) BT_CASE(3) BT_CASE(4) BT_CASE(5) BT_CASE(6) BT_CASE(7) BT_CASE(8)
        BT_CASE(9) BT_CASE(10) BT_CASE(11) BT_CASE(12) BT_CASE(13)
#undef BT_CASE
    }
#pragma unroll
    for (int t = 0; t < NT; t++) out[t] = 0.f;
}

// Near-field source tile in shared memory, structure of arrays (x', y', z'
// relative to the source leaf centre, q), padded to a multiple of 4 with
// charge-free sources far away.
struct Tile {
    float *x, *y, *z, *q;
};

constexpr float MX_PAD_POS = 1.0e18f;   // r2 ~ 1e36 < FLT_MAX; with q = 0 it adds nothing

// Two sources (a pair) against one target, accumulated into the pair sum S.
// r2: with eps^2 for the regularised kernel (folded into the squared distance);
// kc: mixed_kernel_constant(); kc2 = {kc, kc}.
template <int KT>
__device__ __forceinline__ f2_t kf2_acc(f2_t r2, f2_t q, f2_t S, f2_t kc2)
{
    float a, b;
    f2_split(r2, a, b);
    const f2_t rinv = f2_make(rsqrt_apx(a), rsqrt_apx(b));
    if (KT != 2) return f2_fma(q, rinv, S);
    // Yukawa as kf_far: one Newton step on 1/r, then exp(-kappa r) by ex2
    const f2_t h = f2_mul(r2, rinv);
    const f2_t t = f2_fma(f2_mul(h, f2_make(-0.5f, -0.5f)), rinv, f2_make(1.5f, 1.5f));
    float e0, e1;
    f2_split(f2_mul(kc2, f2_mul(h, t)), e0, e1);
    const f2_t e = f2_make(ex2_apx(e0), ex2_apx(e1));
    return f2_fma(q, f2_mul(f2_mul(rinv, t), e), S);
}

// One tile against the thread's TPT targets (x, y, z in the source
// leaf's frame).  NEAR: also the smallest r2 per target (mn), which tells
// whether the tile holds a close pair.
template <int KT, bool NEAR, int TPT>
__device__ __forceinline__ void pp_tile(const Tile tl, int cm4, const float *x, const float *y, const float *z,
                                        float kc, float *s, float *mn)
{
    f2_t X[TPT], Y[TPT], Z[TPT], S[TPT];
#pragma unroll
    for (int t = 0; t < TPT; t++) {
        X[t] = f2_make(x[t], x[t]);
        Y[t] = f2_make(y[t], y[t]);
        Z[t] = f2_make(z[t], z[t]);
        S[t] = f2_make(0.0f, 0.0f);
    }
    const f2_t kc2 = f2_make(kc, kc);
#pragma unroll 2
    for (int i = 0; i < cm4; i += 4) {
        const ulonglong2 PX = *reinterpret_cast<const ulonglong2 *>(tl.x + i);
        const ulonglong2 PY = *reinterpret_cast<const ulonglong2 *>(tl.y + i);
        const ulonglong2 PZ = *reinterpret_cast<const ulonglong2 *>(tl.z + i);
        const ulonglong2 PQ = *reinterpret_cast<const ulonglong2 *>(tl.q + i);
#pragma unroll
        for (int hh = 0; hh < 2; hh++) {
            const f2_t px = hh ? PX.y : PX.x, py = hh ? PY.y : PY.x, pz = hh ? PZ.y : PZ.x, pq = hh ? PQ.y : PQ.x;
#pragma unroll
            for (int t = 0; t < TPT; t++) {
                const f2_t dx = f2_sub(X[t], px), dy = f2_sub(Y[t], py), dz = f2_sub(Z[t], pz);
                const f2_t r2 = f2_fma(dx, dx, f2_fma(dy, dy, KT == 3 ? f2_fma(dz, dz, kc2) : f2_mul(dz, dz)));
                if (NEAR) {
                    float a, b;
                    f2_split(r2, a, b);
                    mn[t] = fminf(mn[t], fminf(a, b));
                }
                S[t] = kf2_acc<KT>(r2, pq, S[t], kc2);
            }
        }
    }
#pragma unroll
    for (int t = 0; t < TPT; t++) {
        float a, b;
        f2_split(S[t], a, b);
        s[t] = a + b;
    }
}

// A tile holding a close pair for this target, again in scalar form: the
// FP32 sum over the pairs at or beyond the close distance (which also drops
// coincident pairs, r2 == 0), and the close pairs in FP64 from the FP64
// coordinates and charges with the reference's skipping rule (k_pp).  thr2:
// the close distance squared, plus eps^2 for the regularised kernel.
template <int KT>
__device__ __noinline__ float pp_tile_close(const Tile tl, int cm, float x, float y, float z, float kc, float thr2,
                                            double xd, double yd, double zd, const double *__restrict__ sx,
                                            const double *__restrict__ sy, const double *__restrict__ sz,
                                            const double *__restrict__ sq, int base, double kp, double *acc)
{
    float s = 0.0f;
    double a = 0.0;
    for (int i = 0; i < cm; i++) {
        const float dx = x - tl.x[i], dy = y - tl.y[i], dz = z - tl.z[i];
        const float r2 = fmaf(dx, dx, fmaf(dy, dy, KT == 3 ? fmaf(dz, dz, kc) : dz * dz));
        if (r2 >= thr2) {
            s += KT == 3 ? tl.q[i] * rsqrt_apx(r2) : kf_far<KT>(r2, tl.q[i], kc);
        } else {
            const int gi = base + i;
            const double ex = xd - sx[gi], ey = yd - sy[gi], ez = zd - sz[gi];
            a += k_pp<KT>(ex * ex + ey * ey + ez * ez, sq[gi], kp);
        }
    }
    *acc += a;
    return s;
}

// Particle-output evaluation, mixed precision.  Each thread owns TPT
// targets of a work item (target leaf, chunk of MX_CHUNK targets), each warp
// 32 * TPT consecutive ones.  In the Hermite kernel, which the FP32 pipe
// bounds, a warp beyond the leaf's last target only helps to stage (2M system
// 152.7 -> 149.7 ms); in the Lagrange kernel it evaluates like the others (the
// 16M system took 895 ms so and 904 ms with the warps skipped).  Each target's
// lists are summed in EV_SEGS segments and the segments in order, as in the
// FP64 kernels: a launch with few items runs one block per (item, segment).
// Blocks of a work-queue launch take items (cost-sorted, longest first) from
// a device counter until the queue is empty; without a queue, block b
// evaluates item b.
__device__ __forceinline__ int next_item(int *queue, int *slot)
{
    if (threadIdx.x == 0) *slot = atomicAdd(queue, 1);
    __syncthreads();
    const int w = *slot;
    __syncthreads();
    return w;
}

// Shared-memory floats of one staged cluster: its grid, and its proxies
// (moments) as pairs; a multiple of four.
__host__ __device__ inline int far_floats(int np1, bool herm)
{
    return 3 * 16 + ((herm ? 16 : 2) * np1 * np1 * np1 + 3 & ~3);
}

template <int KT, bool HERM, int TPT>
__device__ __forceinline__ void targets_item(const MixedTargetsArgs &a, const int2 it, int seg0, int seg1, float *smf,
                                             double *tot)
{
    const int u = it.x;
    const int tnode = a.leaf_node[u];
    const int tb = a.t_ibeg[tnode], tn = a.t_numpar[tnode];
    float x[TPT], y[TPT], z[TPT];
    bool act[TPT];
    int tid[TPT];
#pragma unroll
    for (int t = 0; t < TPT; t++) {
        const int ti = it.y * MX_CHUNK + (threadIdx.x >> 5) * 32 * TPT + t * 32 + (threadIdx.x & 31);
        act[t] = ti < tn;
        tot[t * (MX_CHUNK / TPT) + threadIdx.x] = 0.0;
        tid[t] = tb + (act[t] ? ti : 0);
        float4 tp = a.tpos[tid[t]];
        x[t] = tp.x; y[t] = tp.y; z[t] = tp.z;
    }
    const bool warp_on = !HERM || it.y * MX_CHUNK + (int)(threadIdx.x >> 5) * 32 * TPT < tn;
    const double trad = a.t_rad[tnode];
    const double cx = a.t_ctr[3 * tnode], cy = a.t_ctr[3 * tnode + 1], cz = a.t_ctr[3 * tnode + 2];
    const float kc = (float)a.kc;
    const int64_t ab = a.a_off[u], ae = a.a_off[u + 1], db = a.d_off[u], de = a.d_off[u + 1];
    for (int seg = seg0; seg < seg1; seg++) {
        double acc[TPT];
#pragma unroll
        for (int t = 0; t < TPT; t++) acc[t] = 0.0;
        // far field: source clusters
        // As many clusters as the tile's memory holds are staged together
        // (Hermite: one), so that their loads are in flight together and a
        // pair of barriers serves several clusters: 64 systems of degree 7,
        // 37.7 -> 35.4 ms with eps^2 folded into the squared distances.
        for (int64_t e = seg_begin(ab, ae, seg), e1 = seg_begin(ab, ae, seg + 1); e < e1;) {
            const int64_t eb = e;
            int used = 0;
            do {
                const int s = a.a_idx[e];
                const int np1 = (a.a_deg ? a.a_deg[e] : a.n) + 1, P = np1 * np1 * np1;
                float *g = smf + used, *q = g + 3 * 16;
                const double *gs = a.s_grid[np1 - 1] + (size_t)s * 3 * np1;
                for (int i = threadIdx.x; i < 3 * np1; i += blockDim.x) {
                    int ax = i / np1;
                    double c = ax == 0 ? cx : ax == 1 ? cy : cz;
                    g[i] = (float)(gs[i] - c);
                }
                if (HERM) {
                    const float *Qs = a.Q32[np1 - 1] + (size_t)s * 8 * P;
                    for (int i = threadIdx.x; i < 8 * P; i += blockDim.x) {
                        // a point's moments side by side: the loop reads them in 128-bit words
                        const int m = i & 7;
                        const float v = Qs[m * P + (i >> 3)] * (m == 7 ? 15.0f : m >= 4 ? 3.0f : 1.0f);
                        if constexpr (far_packed<KT, HERM, TPT>()) reinterpret_cast<f2_t *>(q)[i] = f2_make(v, v);
                        else q[i] = v;
                    }
                } else {
                    const float *Qs = a.Q32[np1 - 1] + (size_t)s * P;
#pragma unroll 4
                    for (int i = threadIdx.x; i < P; i += blockDim.x) {
                        const float v = Qs[i];
                        if constexpr (far_packed<KT, HERM, TPT>()) reinterpret_cast<f2_t *>(q)[i] = f2_make(v, v);
                        else q[i] = v;
                    }
                }
                used += far_floats(np1, HERM);
                e++;
            } while (!HERM && e < e1 && used + far_floats((a.a_deg ? a.a_deg[e] : a.n) + 1, HERM) <= a.smem_floats);
            __syncthreads();
            if (warp_on) {
                used = 0;
                for (int64_t f = eb; f < e; f++) {
                    const int np1 = (a.a_deg ? a.a_deg[f] : a.n) + 1;
                    const float *g = smf + used, *q = g + 3 * 16;
                    float v[TPT];
                    if (HERM) pc_cluster_herm_dispatch<KT, TPT>(np1, x, y, z, g, q, kc, (float)a.kp, v);
                    else pc_cluster_dispatch<KT, TPT>(np1, x, y, z, g, q, kc, v);
#pragma unroll
                    for (int t = 0; t < TPT; t++) acc[t] += (double)v[t];
                    used += far_floats(np1, HERM);
                }
            }
            __syncthreads();
        }
        // near field: source leaves, particles relative to their leaf centre
        // fixed array strides (the tile length only bounds the loop): a runtime
        // stride costs the Coulomb kernel 16 registers and a resident block
        const int tile = a.tile;
        const Tile tl{smf, smf + MX_TILE_MAX, smf + 2 * MX_TILE_MAX, smf + 3 * MX_TILE_MAX};
        for (int64_t e = seg_begin(db, de, seg), e1 = seg_begin(db, de, seg + 1); e < e1; e++) {
            const int s = a.d_idx[e];
            const bool near = a.d_flag[e] != 0;
            const int sb = a.s_ibeg[s], sn = a.s_numpar[s];
            const float ox = (float)(a.s_ctr[3 * s] - cx), oy = (float)(a.s_ctr[3 * s + 1] - cy),
                        oz = (float)(a.s_ctr[3 * s + 2] - cz);
            float xs[TPT], ys[TPT], zs[TPT];   // targets in the source leaf's frame
#pragma unroll
            for (int t = 0; t < TPT; t++) { xs[t] = x[t] - ox; ys[t] = y[t] - oy; zs[t] = z[t] - oz; }
            // at least the smallest normal float, so that a coincident pair (r2
            // == 0 after flushing) always takes the FP64 path with the skipping
            // rule, also between single-particle leaves of radius 0
            const double rr = MX_CLOSE_FRAC * (trad + a.s_rad[s]);
            const float thr2 = fmaxf((float)(rr * rr), FLT_MIN) + (KT == 3 ? kc : 0.0f);   // as r2 has it
            for (int c0 = 0; c0 < sn; c0 += tile) {
                const int cm = min(tile, sn - c0), cm4 = (cm + 3) & ~3;
                for (int i = threadIdx.x; i < cm4; i += blockDim.x) {
                    const float4 p = i < cm ? a.spos[sb + c0 + i] : make_float4(MX_PAD_POS, MX_PAD_POS, MX_PAD_POS, 0.0f);
                    tl.x[i] = p.x; tl.y[i] = p.y; tl.z[i] = p.z; tl.q[i] = p.w;
                }
                __syncthreads();
                float sum[TPT], mn[TPT];
                if (!warp_on) {
#pragma unroll
                    for (int t = 0; t < TPT; t++) sum[t] = 0.0f;
                } else if (near) {
#pragma unroll
                    for (int t = 0; t < TPT; t++) mn[t] = FLT_MAX;
                    pp_tile<KT, true, TPT>(tl, cm4, xs, ys, zs, kc, sum, mn);
                    bool close = false;
#pragma unroll
                    for (int t = 0; t < TPT; t++) close |= act[t] && mn[t] < thr2;
                    if (__any_sync(0xffffffffu, close)) {
#pragma unroll
                        for (int t = 0; t < TPT; t++)
                            if (act[t] && mn[t] < thr2)
                                sum[t] = pp_tile_close<KT>(tl, cm, xs[t], ys[t], zs[t], kc, thr2, a.tx64[tid[t]],
                                                           a.ty64[tid[t]], a.tz64[tid[t]], a.sx64, a.sy64, a.sz64,
                                                           a.sq64, sb + c0, a.kp, &acc[t]);
                    }
                } else {
                    pp_tile<KT, false, TPT>(tl, cm4, xs, ys, zs, kc, sum, mn);
                }
#pragma unroll
                for (int t = 0; t < TPT; t++) acc[t] += (double)sum[t];
                __syncthreads();
            }
        }
        // the segment's sums: to the launch's partial array, or onto the total
#pragma unroll
        for (int t = 0; t < TPT; t++) {
            if (a.partial) {
                if (act[t]) a.partial[(size_t)seg * a.pstride + tid[t]] = acc[t];
            } else {
                tot[t * (MX_CHUNK / TPT) + threadIdx.x] += acc[t];
            }
        }
    }
    if (!a.partial)
#pragma unroll
        for (int t = 0; t < TPT; t++)
            if (act[t]) a.pot[tid[t]] = tot[t * (MX_CHUNK / TPT) + threadIdx.x];
}

template <int KT, bool HERM, int TPT>
__device__ __forceinline__ void eval_targets_mixed_body(const MixedTargetsArgs &a)
{
    extern __shared__ float smf[];
    __shared__ double tot[MX_CHUNK];
    __shared__ int slot;
    int w = a.queue ? next_item(a.queue, &slot) : blockIdx.x;
    // split: item-major within a segment, so the items stay longest first
    const int nwork = a.partial ? a.nitems * EV_SEGS : a.nitems;
    while (w < nwork) {
        const int seg = w / a.nitems;
        targets_item<KT, HERM, TPT>(a, a.items[w - seg * a.nitems], seg, a.partial ? seg + 1 : EV_SEGS, smf, tot);
        if (!a.queue) break;
        w = next_item(a.queue, &slot);
    }
}

template <int KT, bool HERM, int TPT>
__global__ void __launch_bounds__(MX_CHUNK / TPT) k_eval_targets_mixed(MixedTargetsArgs a)
{
    eval_targets_mixed_body<KT, HERM, TPT>(a);
}

// The same kernel under the register budget of BT_MX_MIN_BLOCKS_T2 resident
// blocks (2 targets per thread, Lagrange, Coulomb and regularised Coulomb).
template <int KT, bool HERM, int TPT>
__global__ void __launch_bounds__(MX_CHUNK / TPT, rb_blocks<KT, HERM>()) k_eval_targets_mixed_rb(MixedTargetsArgs a)
{
    eval_targets_mixed_body<KT, HERM, TPT>(a);
}

// Grid-output evaluation (M2L from source clusters + CP from source leaves)
// onto the grid of a target node, mixed precision, Lagrange.  Two grid points
// per thread (packed pairs), each warp 64 consecutive ones; a warp beyond the
// grid's last point only stages.
template <int KT>
__device__ __forceinline__ void grids_item(const MixedGridsArgs &a, const int2 it, float *smf)
{
    constexpr int NT = 2;
    const int T = it.x;
    const int np1 = a.n + 1, P = np1 * np1 * np1;
    const int first = it.y * MX_CHUNK + (threadIdx.x >> 5) * 32 * NT;
    const bool warp_on = first < P;
    const double *tg = a.t_grid + (size_t)T * 3 * np1;
    const double cx = a.t_ctr[3 * T], cy = a.t_ctr[3 * T + 1], cz = a.t_ctr[3 * T + 2];
    float x[NT], y[NT], z[NT];
    double acc[NT];
#pragma unroll
    for (int t = 0; t < NT; t++) {
        const int j0 = first + 32 * t + (threadIdx.x & 31), j = j0 < P ? j0 : 0;
        x[t] = (float)(tg[j % np1] - cx);
        y[t] = (float)(tg[np1 + (j / np1) % np1] - cy);
        z[t] = (float)(tg[2 * np1 + j / (np1 * np1)] - cz);
        acc[t] = 0.0;
    }
    const float kc = (float)a.kc;
    const int need = far_floats(np1, false);
    for (int64_t e = a.c_off[T], e1 = a.c_off[T + 1]; e < e1;) {
        const int64_t eb = e;
        for (int used = 0; e < e1 && (e == eb || used + need <= a.smem_floats); e++, used += need) {
            const int s = a.c_idx[e];
            float *g = smf + used;
            f2_t *q = reinterpret_cast<f2_t *>(g + 3 * 16);
            const double *gs = a.s_grid + (size_t)s * 3 * np1;
            for (int i = threadIdx.x; i < 3 * np1; i += blockDim.x) {
                int ax = i / np1;
                double c = ax == 0 ? cx : ax == 1 ? cy : cz;
                g[i] = (float)(gs[i] - c);
            }
#pragma unroll 4
            for (int i = threadIdx.x; i < P; i += blockDim.x) {
                const float v = a.Q32[(size_t)s * P + i];
                q[i] = f2_make(v, v);
            }
        }
        __syncthreads();
        if (warp_on)
            for (int k = 0; k < (int)(e - eb); k++) {
                float v[NT];
                pc_cluster_dispatch<KT, NT>(np1, x, y, z, smf + k * need, smf + k * need + 3 * 16, kc, v);
#pragma unroll
                for (int t = 0; t < NT; t++) acc[t] += (double)v[t];
            }
        __syncthreads();
    }
    const Tile tl{smf, smf + MX_TILE, smf + 2 * MX_TILE, smf + 3 * MX_TILE};
    for (int64_t e = a.p_off[T]; e < a.p_off[T + 1]; e++) {
        const int s = a.p_idx[e];
        const int sb = a.s_ibeg[s], sn = a.s_numpar[s];
        const float ox = (float)(a.s_ctr[3 * s] - cx), oy = (float)(a.s_ctr[3 * s + 1] - cy),
                    oz = (float)(a.s_ctr[3 * s + 2] - cz);
        float xs[NT], ys[NT], zs[NT];
#pragma unroll
        for (int t = 0; t < NT; t++) { xs[t] = x[t] - ox; ys[t] = y[t] - oy; zs[t] = z[t] - oz; }
        for (int c0 = 0; c0 < sn; c0 += MX_TILE) {
            const int cm = min(MX_TILE, sn - c0), cm4 = (cm + 3) & ~3;
            for (int i = threadIdx.x; i < cm4; i += blockDim.x) {
                const float4 p = i < cm ? a.spos[sb + c0 + i] : make_float4(MX_PAD_POS, MX_PAD_POS, MX_PAD_POS, 0.0f);
                tl.x[i] = p.x; tl.y[i] = p.y; tl.z[i] = p.z; tl.q[i] = p.w;
            }
            __syncthreads();
            if (warp_on) {
                float sum[NT];
                pp_tile<KT, false, NT>(tl, cm4, xs, ys, zs, kc, sum, nullptr);
#pragma unroll
                for (int t = 0; t < NT; t++) acc[t] += (double)sum[t];
            }
            __syncthreads();
        }
    }
#pragma unroll
    for (int t = 0; t < NT; t++) {
        const int j = first + 32 * t + (threadIdx.x & 31);
        if (j < P) a.Phi[(size_t)T * P + j] = acc[t];
    }
}

template <int KT>
__global__ void __launch_bounds__(MX_THREADS, MX_MIN_BLOCKS)
k_eval_grids_mixed(MixedGridsArgs a)
{
    extern __shared__ float smf[];
    __shared__ int slot;
    int w = a.queue ? next_item(a.queue, &slot) : blockIdx.x;
    while (w < a.nitems) {
        grids_item<KT>(a, a.items[w], smf);
        if (!a.queue) break;
        w = next_item(a.queue, &slot);
    }
}

// Particles relative to the centre of their leaf, FP32 (x', y', z', q).
__global__ void k_rel_positions(int nleaves, const int *__restrict__ leaves, const int *__restrict__ ibeg,
                                const int *__restrict__ numpar, const double *__restrict__ ctr,
                                const double *__restrict__ x, const double *__restrict__ y,
                                const double *__restrict__ z, const double *__restrict__ q, float4 *__restrict__ out)
{
    const int l = leaves[blockIdx.x];
    const double cx = ctr[3 * l], cy = ctr[3 * l + 1], cz = ctr[3 * l + 2];
    for (int i = ibeg[l] + threadIdx.x; i < ibeg[l] + numpar[l]; i += blockDim.x)
        out[i] = make_float4((float)(x[i] - cx), (float)(y[i] - cy), (float)(z[i] - cz), q ? (float)q[i] : 0.f);
}

__global__ void k_to_f32(size_t n, const double *__restrict__ src, float *__restrict__ dst)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        dst[i] = (float)src[i];
}

void launch_rel_positions(int nleaves, const int *leaves, const int *ibeg, const int *numpar, const double *ctr,
                          const double *x, const double *y, const double *z, const double *q, float4 *out,
                          cudaStream_t st)
{
    if (nleaves > 0) k_rel_positions<<<nleaves, 256, 0, st>>>(nleaves, leaves, ibeg, numpar, ctr, x, y, z, q, out);
}

void launch_to_f32(size_t n, const double *src, float *dst, cudaStream_t st)
{
    if (n > 0) k_to_f32<<<1184, 256, 0, st>>>(n, src, dst);
}

int mixed_targets_chunk() { return MX_CHUNK; }

// Shared memory of the evaluation kernels: the far-field staging (grid
// coordinates and proxy charges of one cluster) or the near-field tile,
// whose four arrays sit MX_TILE_MAX floats apart in the particle-output
// kernel (tile_stride) whatever the tile length.
static size_t mixed_smem(int max_np1, bool herm, int tile_stride)
{
    // proxy charges are staged as {q, q} pairs (packed far field)
    size_t far = sizeof(float) * (size_t)far_floats(max_np1, herm);
    size_t near = sizeof(float4) * (size_t)tile_stride;
    return far > near ? far : near;
}

// Grid of a work-queue launch: as many blocks as are resident at once.
template <typename K>
static int queue_grid(K kernel, int threads, size_t smem, int nitems)
{
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
    int g = sms * (per_sm > 0 ? per_sm : 1);
    return g < nitems ? g : nitems;
}

template <int KT, bool HERM, int TPT>
static void eval_targets_mixed_t(MixedTargetsArgs a, cudaStream_t st)
{
    size_t sm = mixed_smem(a.max_np1, HERM, MX_TILE_MAX);
    a.smem_floats = (int)(sm / sizeof(float));
    auto kernel = k_eval_targets_mixed<KT, HERM, TPT>;
    if constexpr (TPT == 2 && rb_blocks<KT, HERM>() > 0) kernel = k_eval_targets_mixed_rb<KT, HERM, TPT>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    const int nwork = a.partial ? a.nitems * EV_SEGS : a.nitems;
    int grid = a.queue ? queue_grid(kernel, MX_CHUNK / TPT, sm, nwork) : nwork;
    kernel<<<grid, MX_CHUNK / TPT, sm, st>>>(a);
}

template <int KT, bool HERM>
static void eval_targets_mixed_h(const MixedTargetsArgs &a, cudaStream_t st)
{
    if (a.tpt == 1) eval_targets_mixed_t<KT, HERM, 1>(a, st);
    else if (a.tpt == 4) eval_targets_mixed_t<KT, HERM, 4>(a, st);
    else eval_targets_mixed_t<KT, HERM, 2>(a, st);
}

void launch_eval_targets_mixed(int kernel, const MixedTargetsArgs &a, cudaStream_t st)
{
    if (a.nitems <= 0) return;
    if (kernel == 1) a.herm ? eval_targets_mixed_h<1, true>(a, st) : eval_targets_mixed_h<1, false>(a, st);
    else if (kernel == 2) a.herm ? eval_targets_mixed_h<2, true>(a, st) : eval_targets_mixed_h<2, false>(a, st);
    else a.herm ? eval_targets_mixed_h<3, true>(a, st) : eval_targets_mixed_h<3, false>(a, st);
    if (a.partial)
        launch_sum_segments(a.nitems, a.items, MX_CHUNK, a.leaf_node, a.t_ibeg, a.t_numpar, a.partial, a.pstride, a.pot, st);
}

// Below about four waves of resident blocks (6 on each of 148 SMs) every
// segment of an item gets its own block.
bool mixed_split(size_t items) { return items < (size_t)4 * 6 * 148; }

template <int KT>
static void eval_grids_mixed_t(MixedGridsArgs a, cudaStream_t st)
{
    size_t sm = mixed_smem(a.n + 1, false, MX_TILE);
    a.smem_floats = (int)(sm / sizeof(float));
    cudaFuncSetAttribute(k_eval_grids_mixed<KT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    int grid = a.queue ? queue_grid(k_eval_grids_mixed<KT>, MX_THREADS, sm, a.nitems) : a.nitems;
    k_eval_grids_mixed<KT><<<grid, MX_THREADS, sm, st>>>(a);
}

void launch_eval_grids_mixed(int kernel, const MixedGridsArgs &a, cudaStream_t st)
{
    if (a.nitems <= 0) return;
    if (kernel == 1) eval_grids_mixed_t<1>(a, st);
    else if (kernel == 2) eval_grids_mixed_t<2>(a, st);
    else eval_grids_mixed_t<3>(a, st);
}

double mixed_kernel_constant(int kernel, double kp)
{
    if (kernel == 2) return -kp * 1.4426950408889634;   // exp(-k r) = 2^(-k log2(e) r)
    if (kernel == 3) return kp * kp;
    return 0.0;
}

}  // namespace bt
