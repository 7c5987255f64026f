// bt_sym.cu -- symmetric near-field pairs of the mixed path.
//
// When the targets are the sources (same particles, same tree) and the
// kernel is symmetric in r (Coulomb, Yukawa, regularized Coulomb), a pair of
// distinct leaves {A, B} that each hold the other in their near-field list
// needs each pair distance once: 1/r_ij serves both phi_i (i in A, source j
// in B) and phi_j (j in B, source i in A).  The reference evaluates the two
// directions separately (src/interaction_compute/interaction_compute_pc.c,
// direct list of each target batch); the sums are the same up to rounding.
// Pairs of leaves whose boxes lie within the close-pair distance of each
// other (touching leaves, mostly) can hold close pairs, which the mixed path
// evaluates in FP64 from the FP64 particles.  Their kernel (CLAMP) raises
// every FP32 r^2 to at least the close-pair distance squared, so a close
// pair adds a bounded, known term (the kernel at that distance) to both
// sides; before the main loop the block finds the particles of each leaf
// that lie within that distance of the other leaf's box (a few per cent of
// them, found in FP64), recomputes the FP32 r^2 of every pair among those
// candidates with the main loop's own instructions, and for each pair
// below the distance writes the FP64 kernel minus the clamped term into
// both sides' slices.  The main loop's sums are added to these at the end.
// Self pairs (A with A) stay in the particle-output kernel.
//
// Work: one block per pair and part of SYM_PART of A's targets.  B's particles
// stream through shared memory in tiles, staged as {v, v} pairs; the block's
// warps divide a tile's sources, and each takes them against the part's
// targets 128 at a time, four per thread in two packed FP32 pairs.  Every 1/r
// feeds the thread's A-side sums and, through a per-thread register per
// source, the B side: each group of 16 sources is reduced across the warp by a
// reduce-scatter (16 shuffles for 16 sources; lanes 2i and 2i+1 end with
// source i).  The warps' A-side sums are added in a fixed order.  Both sides
// go to the pair's own slices of a partial-sum array (A's once, B's per part);
// k_sym_gather adds each leaf's slices in FP64 in pair order.  No atomics: the
// potentials are the same bit for bit on every run.
// With the targets divided over the warps instead (512 per block and pass) a
// leaf of 1,560 cost the lanes of 2,048; now it costs those of 1,664, every
// warp has work, and a block is a quarter as long, which is what small
// systems lack.
#include <cuda_runtime.h>

#include <cstdint>

#include <cfloat>

#include "bt_f2.cuh"
#include "bt_kernels.cuh"
#include "bt_mixed.h"
#include "bt_sym.h"

namespace bt {

namespace {

constexpr int SY_THREADS = 128;
// targets of A per thread (packed in pairs) and the resident blocks per SM
// the register budget is sized for; build-time choices.  Measured, evaluation
// phase of 2M clustered Coulomb and of 1M cluster-cluster Yukawa, degree 8:
// 4 and 6 91.0 and 16.4 ms, 4 and 5 91.1 and 16.9, 4 and 7 91.0 and 16.5,
// 8 and 4 90.2 and 16.8, 8 and 3 90.9 and 16.5, 2 and 8 96.7 and 18.2
#ifndef BT_SYM_TPT
#define BT_SYM_TPT 4
#endif
#ifndef BT_SYM_MIN_BLOCKS
#define BT_SYM_MIN_BLOCKS 6
#endif
constexpr int SY_TPT = BT_SYM_TPT;
constexpr int SY_NP = SY_TPT / 2;
constexpr int SY_CHUNK = SY_TPT * 32;          // targets of A a warp holds at a time
static_assert(SY_TPT % 2 == 0 && SYM_PART % SY_CHUNK == 0, "a part is whole chunks (accA), targets are packed in pairs");
#ifndef BT_SYM_TILE
#define BT_SYM_TILE 256
#endif
constexpr int SY_TILE = BT_SYM_TILE;                   // sources of B per shared-memory tile
constexpr int SY_SB = 16;                      // sources per warp reduction
static_assert(SY_TILE % SY_SB == 0, "a tile is whole groups of sources");
constexpr int SY_WARPS = SY_THREADS / 32;
constexpr float SY_PAD_POS = 1.0e18f;          // padding sources: far away, no charge

// v[0..2H-1] per lane -> v[0..H-1]: lanes with bit LX of their index keep
// the upper half of the indices, the others the lower half, each adding the
// partner's (lane ^ LX) copy of the half it keeps.
template <int H, int LX>
__device__ __forceinline__ void rs_stage(float *v, int lane)
{
    const bool up = (lane & LX) != 0;
#pragma unroll
    for (int i = 0; i < H; i++) {
        const float a = v[i], b = v[i + H];
        const float keep = up ? b : a, send = up ? a : b;
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, LX);
    }
}

// The kernel value of a packed pair of r^2, which holds eps^2 for the
// regularised kernel (the particle-output kernel's arithmetic): 1/r;
// Yukawa with one Newton step on 1/r, then exp(-kappa r) by ex2.
template <int KT>
__device__ __forceinline__ f2_t sym_kval(f2_t r2, f2_t kc2)
{
    float ra, rb;
    f2_split(r2, ra, rb);
    f2_t k = f2_make(rsqrt_apx(ra), rsqrt_apx(rb));
    if (KT == 2) {
        const f2_t h = f2_mul(r2, k);
        const f2_t t = f2_fma(f2_mul(h, f2_make(-0.5f, -0.5f)), k, f2_make(1.5f, 1.5f));
        float e0, e1;
        f2_split(f2_mul(kc2, f2_mul(h, t)), e0, e1);
        k = f2_mul(f2_mul(k, t), f2_make(ex2_apx(e0), ex2_apx(e1)));
    }
    return k;
}

// The main loop's FP32 r^2 of one pair, with its instructions: x, y, z the
// target in the source leaf's frame, p the source.
template <int KT>
__device__ __forceinline__ f2_t sym_r2p(f2_t dx, f2_t dy, f2_t dz, f2_t kc2)
{
    return f2_fma(dx, dx, f2_fma(dy, dy, KT == 3 ? f2_fma(dz, dz, kc2) : f2_mul(dz, dz)));
}
template <int KT>
__device__ __forceinline__ float sym_r2(float x, float y, float z, float4 p, f2_t kc2)
{
    const f2_t dx = f2_sub(f2_make(x, x), f2_make(p.x, p.x)), dy = f2_sub(f2_make(y, y), f2_make(p.y, p.y)),
               dz = f2_sub(f2_make(z, z), f2_make(p.z, p.z));
    float r2, unused;
    f2_split(sym_r2p<KT>(dx, dy, dz, kc2), r2, unused);
    return r2;
}

// Indices i < n of the particles (FP64, from `base`) within distance d of
// the box b (x0 x1 y0 y1 z0 z1), in index order, into out; returns how many.
__device__ int near_box(int *out, int n, int base, const double *__restrict__ x, const double *__restrict__ y,
                        const double *__restrict__ z, const double *b, double d, int *wcnt)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int total = 0;
    for (int c0 = 0; c0 < n; c0 += SY_THREADS) {
        const int i = c0 + threadIdx.x;
        bool f = false;
        if (i < n) {
            const double px = x[base + i], py = y[base + i], pz = z[base + i];
            const double gx = fmax(0.0, fmax(b[0] - px, px - b[1])), gy = fmax(0.0, fmax(b[2] - py, py - b[3])),
                         gz = fmax(0.0, fmax(b[4] - pz, pz - b[5]));
            f = gx * gx + gy * gy + gz * gz <= d * d;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, f);
        if (lane == 0) wcnt[warp] = __popc(bal);
        __syncthreads();
        int off = total, all = 0;
#pragma unroll
        for (int w = 0; w < SY_WARPS; w++) {
            off += w < warp ? wcnt[w] : 0;
            all += wcnt[w];
        }
        if (f) out[off + __popc(bal & ((1u << lane) - 1u))] = i;
        __syncthreads();
        total += all;
    }
    return total;
}

template <int KT, bool CLAMP>
__global__ void __launch_bounds__(SY_THREADS, BT_SYM_MIN_BLOCKS) k_pp_sym(const __grid_constant__ SymArgs a)
{
    __shared__ __align__(16) f2_t tile[SY_TILE][4];     // {x, x}, {y, y}, {z, z}, {q, q}
    __shared__ float accB[SYM_MAX_LEAF];
    __shared__ double accA[SY_WARPS][SYM_PART];          // each warp's A side: FP32 sums per tile, added in FP64
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int2 work = a.block[blockIdx.x];
    const int2 pr = a.pair[work.x];
    const int A = pr.x, B = pr.y;
    const int a0 = work.y * SYM_PART, na = a.numpar[A], nb = a.numpar[B], pa = min(SYM_PART, na - a0);
    const int ia = a.ibeg[A] + a0, ib = a.ibeg[B];
    float *outA = a.partial + a.slot[work.x] + a0;
    float *outB = a.partial + a.slot[work.x] + na + (size_t)work.y * nb;
    // A's targets in B's frame: positions relative to A's centre minus the offset of B's
    const float ox = (float)(a.ctr[3 * B] - a.ctr[3 * A]), oy = (float)(a.ctr[3 * B + 1] - a.ctr[3 * A + 1]),
                oz = (float)(a.ctr[3 * B + 2] - a.ctr[3 * A + 2]);
    const f2_t kc2 = f2_make(a.kc, a.kc);
    // the close-pair distance squared, as the particle-output kernel has it
    float thr2 = 0.0f;
    if (CLAMP) {
        const double rr = MX_CLOSE_FRAC * (a.rad[A] + a.rad[B]);
        const float cut2 = fmaxf((float)(rr * rr), FLT_MIN);
        thr2 = cut2 + (KT == 3 ? a.kc : 0.0f);               // as r^2 has it
        __shared__ int wcnt[SY_WARPS];
        int *candA = reinterpret_cast<int *>(&accA[0][0]), *candB = candA + SYM_PART;
        static_assert(sizeof(int) * (SYM_PART + SYM_MAX_LEAF) <= sizeof(accA), "the candidate lists live in accA");
        for (int i = threadIdx.x; i < pa; i += SY_THREADS) outA[i] = 0.0f;
        for (int j = threadIdx.x; j < nb; j += SY_THREADS) outB[j] = 0.0f;
        // every pair with FP32 r^2 below thr2 lies within 1.01 of the close
        // distance of both boxes (with eps^2 far above its square the clamp
        // changes r^2 by less than its rounding)
        const double d = 1.01 * sqrt((double)cut2);
        const int nca = near_box(candA, pa, ia, a.x64, a.y64, a.z64, a.box + 6 * B, d, wcnt);
        const int ncb = nca > 0 ? near_box(candB, nb, ib, a.x64, a.y64, a.z64, a.box + 6 * A, d, wcnt) : 0;
        if (nca > 0 && ncb > 0) {
            float kcl, unused;
            f2_split(sym_kval<KT>(f2_make(thr2, thr2), kc2), kcl, unused);   // the clamped term's kernel value
            const double kcd = (double)kcl;
            for (int k = threadIdx.x; k < nca + ncb; k += SY_THREADS) {
                // thread k: candidate k of A (its sum over B's candidates), then of B
                const bool sideA = k < nca;
                const int i = sideA ? candA[k] : candB[k - nca];
                const int gi = (sideA ? ia : ib) + i;
                const float4 pi = a.pos[gi];
                double c = 0.0;
                for (int m = 0; m < (sideA ? ncb : nca); m++) {
                    const int j = sideA ? candB[m] : candA[m];
                    const int gj = (sideA ? ib : ia) + j;
                    const float4 pj = a.pos[gj];
                    // the pair's r^2 as the main loop forms it: A's target in B's frame
                    const float r2 = sideA ? sym_r2<KT>(pi.x - ox, pi.y - oy, pi.z - oz, pj, kc2)
                                           : sym_r2<KT>(pj.x - ox, pj.y - oy, pj.z - oz, pi, kc2);
                    if (r2 < thr2) {
                        const double ex = a.x64[gi] - a.x64[gj], ey = a.y64[gi] - a.y64[gj],
                                     ez = a.z64[gi] - a.z64[gj];
                        c += k_pp<KT>(ex * ex + ey * ey + ez * ez, a.q64[gj], a.kp) - (double)pj.w * kcd;
                    }
                }
                (sideA ? outA[i] : outB[i]) = (float)c;
            }
        }
        __syncthreads();                                  // the candidate lists are done with
    }
    const int nch = (pa + SY_CHUNK - 1) / SY_CHUNK;
    for (int j = threadIdx.x; j < nb; j += SY_THREADS) accB[j] = 0.0f;
    for (int i = lane; i < nch * SY_CHUNK; i += 32) accA[warp][i] = 0.0;
    for (int s0 = 0; s0 < nb; s0 += SY_TILE) {
        const int cm = min(SY_TILE, nb - s0), groups = (cm + SY_SB - 1) / SY_SB;
        __syncthreads();                                  // the previous tile is done with
        for (int i = threadIdx.x; i < groups * SY_SB; i += SY_THREADS) {
            const float4 p = i < cm ? a.pos[ib + s0 + i] : make_float4(SY_PAD_POS, SY_PAD_POS, SY_PAD_POS, 0.0f);
            tile[i][0] = f2_make(p.x, p.x);
            tile[i][1] = f2_make(p.y, p.y);
            tile[i][2] = f2_make(p.z, p.z);
            tile[i][3] = f2_make(p.w, p.w);
        }
        __syncthreads();
        // the warp's sources of the tile, against every chunk of the part
        const int b0 = groups * warp / SY_WARPS * SY_SB, b1 = groups * (warp + 1) / SY_WARPS * SY_SB;
        for (int c = 0; c < nch && b0 < b1; c++) {
            // targets c * SY_CHUNK + lane + 32 k, k = 0..SY_TPT-1, packed as (0, 1), (2, 3), ...
            f2_t X[SY_NP], Y[SY_NP], Z[SY_NP], QT[SY_NP], S[SY_NP];
#pragma unroll
            for (int p = 0; p < SY_NP; p++) {
                const int t0 = c * SY_CHUNK + lane + 64 * p, t1 = t0 + 32;
                const float4 p0 = a.pos[ia + (t0 < pa ? t0 : 0)], p1 = a.pos[ia + (t1 < pa ? t1 : 0)];
                X[p] = f2_make(p0.x - ox, p1.x - ox);
                Y[p] = f2_make(p0.y - oy, p1.y - oy);
                Z[p] = f2_make(p0.z - oz, p1.z - oz);
                QT[p] = f2_make(t0 < pa ? p0.w : 0.0f, t1 < pa ? p1.w : 0.0f);   // absent targets add nothing
                S[p] = f2_make(0.0f, 0.0f);
            }
            for (int sb = b0; sb < b1; sb += SY_SB) {
                float v[SY_SB];
#pragma unroll
                for (int s = 0; s < SY_SB; s++) {
                    const ulonglong2 xy = *reinterpret_cast<const ulonglong2 *>(&tile[sb + s][0]);
                    const ulonglong2 zq = *reinterpret_cast<const ulonglong2 *>(&tile[sb + s][2]);
                    f2_t cb = f2_make(0.0f, 0.0f);
#pragma unroll
                    for (int p = 0; p < SY_NP; p++) {
                        const f2_t dx = f2_sub(X[p], xy.x), dy = f2_sub(Y[p], xy.y), dz = f2_sub(Z[p], zq.x);
                        f2_t r2 = sym_r2p<KT>(dx, dy, dz, kc2);
                        if (CLAMP) {
                            float ra, rb;
                            f2_split(r2, ra, rb);
                            r2 = f2_make(fmaxf(ra, thr2), fmaxf(rb, thr2));
                        }
                        const f2_t rinv = sym_kval<KT>(r2, kc2);      // serves both sides
                        S[p] = f2_fma(zq.y, rinv, S[p]);
                        // B side: the targets' charges over r, folded into one pair
                        cb = p == 0 ? f2_mul(QT[0], rinv) : f2_fma(QT[p], rinv, cb);
                    }
                    float c0v, c1v;
                    f2_split(cb, c0v, c1v);
                    v[s] = c0v + c1v;
                }
                // reduce-scatter over the warp: lanes 2i and 2i+1 end with source i
                rs_stage<8, 16>(v, lane);
                rs_stage<4, 8>(v, lane);
                rs_stage<2, 4>(v, lane);
                rs_stage<1, 2>(v, lane);
                v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
                if ((lane & 1) == 0) {
                    const int j = s0 + sb + (lane >> 1);
                    if (j < nb) accB[j] += v[0];          // the source is this warp's alone
                }
            }
            // the chunk's A-side sums into FP64 (FP32 chains of at most a quarter of a tile)
#pragma unroll
            for (int p = 0; p < SY_NP; p++) {
                float lo, hi;
                f2_split(S[p], lo, hi);
                accA[warp][c * SY_CHUNK + lane + 64 * p] += (double)lo;
                accA[warp][c * SY_CHUNK + lane + 64 * p + 32] += (double)hi;
            }
        }
    }
    __syncthreads();
    // the warps' sums in a fixed order
    for (int i = threadIdx.x; i < pa; i += SY_THREADS) {
        double r = accA[0][i];
#pragma unroll
        for (int w = 1; w < SY_WARPS; w++) r += accA[w][i];
        outA[i] = (float)(CLAMP ? r + (double)outA[i] : r);
    }
    for (int j = threadIdx.x; j < nb; j += SY_THREADS) outB[j] = CLAMP ? accB[j] + outB[j] : accB[j];
}

// One block per leaf and GATHER_THREADS of its particles; the slices' offsets
// go through shared memory, so that a thread's loads do not wait for them.
// With several rounds the sum goes on from the round before and reaches the
// potential in the last one: the same additions in the same order as in one.
__global__ void __launch_bounds__(GATHER_THREADS) k_sym_gather(SymGatherArgs a)
{
    __shared__ int64_t slot[GATHER_THREADS];
    const int u = blockIdx.x;
    const int64_t *off = a.in_off + u;
    const int64_t k0 = off[(size_t)a.round * a.nleaves], k1 = off[(size_t)(a.round + 1) * a.nleaves];
    const int node = a.leaf_node[u];
    const int nb = a.numpar[node], j = blockIdx.y * GATHER_THREADS + threadIdx.x;
    if ((int)blockIdx.y * GATHER_THREADS >= nb || off[0] == off[(size_t)a.nrounds * a.nleaves]) return;
    double s = a.round > 0 && j < nb ? a.run[a.ibeg[node] + j] : 0.0;
    for (int64_t b = k0; b < k1; b += GATHER_THREADS) {
        const int m = (int)min((int64_t)GATHER_THREADS, k1 - b);
        __syncthreads();
        if ((int)threadIdx.x < m) slot[threadIdx.x] = a.in_slot[b + threadIdx.x];
        __syncthreads();
        if (j < nb)
#pragma unroll 8
            for (int k = 0; k < m; k++) s += (double)a.partial[slot[k] + j];
    }
    if (j >= nb) return;
    if (a.round + 1 < a.nrounds) a.run[a.ibeg[node] + j] = s;
    else a.pot[a.ibeg[node] + j] += s;
}

}  // namespace

void launch_pp_sym(int kernel, const SymArgs &a, cudaStream_t st)
{
    if (a.nblocks <= 0) return;
    if (kernel == 3) k_pp_sym<3, false><<<a.nblocks, SY_THREADS, 0, st>>>(a);
    else if (kernel == 2) k_pp_sym<2, false><<<a.nblocks, SY_THREADS, 0, st>>>(a);
    else k_pp_sym<1, false><<<a.nblocks, SY_THREADS, 0, st>>>(a);
}

void launch_pp_sym_close(int kernel, const SymArgs &a, cudaStream_t st)
{
    if (a.nblocks <= 0) return;
    if (kernel == 3) k_pp_sym<3, true><<<a.nblocks, SY_THREADS, 0, st>>>(a);
    else if (kernel == 2) k_pp_sym<2, true><<<a.nblocks, SY_THREADS, 0, st>>>(a);
    else k_pp_sym<1, true><<<a.nblocks, SY_THREADS, 0, st>>>(a);
}

void launch_sym_gather(const SymGatherArgs &a, cudaStream_t st)
{
    if (a.nleaves > 0) k_sym_gather<<<dim3(a.nleaves, SYM_MAX_LEAF / GATHER_THREADS), GATHER_THREADS, 0, st>>>(a);
}

}  // namespace bt
