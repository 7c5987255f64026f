// bt_sym64.cu -- symmetric near-field pairs of the FP64 path.
//
// As bt_sym.cu for the mixed path: with the targets being the sources, two
// leaves {A, B} that hold each other in their near-field lists need each
// distance once.  A value for both directions takes 13 FP64 instructions and
// a little reduction instead of twice 12 (Coulomb), and the FP64 pipe is the
// bound.
//
// One block per pair and part of SYM_PART of A's particles, as in bt_sym.cu:
// B streams through shared memory in tiles whose sources the warps divide;
// each warp takes them against the part's particles 128 at a time (four per
// thread), adds q_j K into the thread's own sums and reduces q_i K over the
// warp, eight sources at a time, by a reduce-scatter in a fixed order.  The
// sums go to the pair's own slices, which k_sym_gather64 adds per leaf in
// partner order: no atomics, the same bits on every run.
//
// Distinct leaves of one tree hold no coincident particles (equal coordinates
// always go to the same child), so the skipping rule has nothing to do except
// for distances whose square underflows; such a sum is not finite and is
// formed again with the library functions.
#include <cuda_runtime.h>

#include <cstdint>

#include "bt_eval64.cuh"
#include "bt_sym.h"

namespace bt {

namespace {

constexpr int S64_THREADS = 128;
constexpr int S64_MINB = 3;                      // resident blocks per SM (4 measured 1.5 % slower, 300k Yukawa)
constexpr int S64_WARPS = S64_THREADS / 32;
constexpr int S64_TPT = 4;                       // particles of A per thread
constexpr int S64_CHUNK = 32 * S64_TPT;          // per warp
constexpr int S64_TILE = 256;                    // particles of B per tile
constexpr int S64_SB = 8;                        // particles of B per warp reduction

// v[0..2H-1] per lane -> v[0..H-1]: lanes with bit LX of their index keep the
// upper half of the indices, the others the lower half.
template <int H, int LX>
__device__ __forceinline__ void scatter64(double *v, int lane)
{
    const bool up = (lane & LX) != 0;
#pragma unroll
    for (int i = 0; i < H; i++) {
        const double keep = up ? v[i + H] : v[i], send = up ? v[i] : v[i + H];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, LX);
    }
}

// One particle's sum over a leaf with the library functions.
template <int KT>
__device__ __noinline__ double leaf_again(const Sym64Args &a, int i, int jb, int jn)
{
    double s = 0.0;
    for (int j = jb; j < jb + jn; j++)
        s += k_any<KT, true>(a.x[i] - a.x[j], a.y[i] - a.y[j], a.z[i] - a.z[j], a.q[j], a.kp, 0.0);
    return s;
}

template <int KT, bool FAR>
__global__ void __launch_bounds__(S64_THREADS, S64_MINB) k_pp_sym64(const __grid_constant__ Sym64Args a)
{
    __shared__ double2 xy[S64_TILE], zq[S64_TILE];
    __shared__ double accB[SYM_MAX_LEAF];
    __shared__ double accA[S64_WARPS][SYM_PART];
    __shared__ double2 tab[KT == K_YUKAWA ? EXP64_TAB : 1];
    const Kern64<FAR> k = kern64_make<KT, FAR>(a.kp, 0.0, tab);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int2 work = a.block[blockIdx.x];
    const int2 pr = a.pair[work.x];
    const int a0 = work.y * SYM_PART, na = a.numpar[pr.x], nb = a.numpar[pr.y], pa = min(SYM_PART, na - a0);
    const int ia = a.ibeg[pr.x] + a0, ib = a.ibeg[pr.y];
    double *outA = a.partial + a.slot[work.x] + a0, *outB = a.partial + a.slot[work.x] + na + (size_t)work.y * nb;
    const int nch = (pa + S64_CHUNK - 1) / S64_CHUNK;
    for (int j = threadIdx.x; j < nb; j += S64_THREADS) accB[j] = 0.0;
    for (int i = lane; i < nch * S64_CHUNK; i += 32) accA[warp][i] = 0.0;
    for (int s0 = 0; s0 < nb; s0 += S64_TILE) {
        const int cm = min(S64_TILE, nb - s0), groups = (cm + S64_SB - 1) / S64_SB;
        __syncthreads();                             // the previous tile is done with
        for (int i = threadIdx.x; i < groups * S64_SB; i += S64_THREADS) {
            const int j = ib + s0 + (i < cm ? i : 0);
            xy[i] = make_double2(a.x[j], a.y[j]);
            zq[i] = make_double2(a.z[j], i < cm ? a.q[j] : 0.0);
        }
        __syncthreads();
        const int b0 = groups * warp / S64_WARPS * S64_SB, b1 = groups * (warp + 1) / S64_WARPS * S64_SB;
        for (int c = 0; c < nch && b0 < b1; c++) {
            double x[S64_TPT], y[S64_TPT], z[S64_TPT], q[S64_TPT], s[S64_TPT];
#pragma unroll
            for (int t = 0; t < S64_TPT; t++) {
                const int i = c * S64_CHUNK + lane + 32 * t, j = ia + (i < pa ? i : 0);
                x[t] = a.x[j]; y[t] = a.y[j]; z[t] = a.z[j];
                q[t] = i < pa ? a.q[j] : 0.0;        // absent particles add nothing
                s[t] = 0.0;
            }
            for (int sb = b0; sb < b1; sb += S64_SB) {
                double v[S64_SB];
#pragma unroll
                for (int j = 0; j < S64_SB; j++) {
                    const double2 p = xy[sb + j], r = zq[sb + j];
#pragma unroll
                    for (int t = 0; t < S64_TPT; t++) {
                        const double dx = x[t] - p.x, dy = y[t] - p.y, dz = z[t] - r.x;
                        const double r2 =
                            fma(dx, dx, fma(dy, dy, KT == K_REGCOULOMB ? fma(dz, dz, k.eps2) : dz * dz));
                        const double kv = value64<KT>(r2, k);
                        s[t] = fma(r.y, kv, s[t]);
                        v[j] = t == 0 ? q[0] * kv : fma(q[t], kv, v[j]);
                    }
                }
                // over the warp: lanes 4i .. 4i+3 end with source i
                scatter64<4, 16>(v, lane);
                scatter64<2, 8>(v, lane);
                scatter64<1, 4>(v, lane);
                v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
                v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
                if ((lane & 3) == 0) {
                    const int j = s0 + sb + (lane >> 2);
                    if (j < nb) accB[j] += v[0];     // the source is this warp's alone
                }
            }
#pragma unroll
            for (int t = 0; t < S64_TPT; t++) accA[warp][c * S64_CHUNK + lane + 32 * t] += s[t];
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < pa; i += S64_THREADS) {
        double r = accA[0][i];
#pragma unroll
        for (int w = 1; w < S64_WARPS; w++) r += accA[w][i];
        if (k.lib || !isfinite(r)) r = leaf_again<KT>(a, ia + i, ib, nb);
        outA[i] = r;
    }
    for (int j = threadIdx.x; j < nb; j += S64_THREADS) {
        double r = accB[j];
        if (k.lib || !isfinite(r)) r = leaf_again<KT>(a, ib + j, ia, pa);
        outB[j] = r;
    }
}

// One block per leaf and GATHER_THREADS of its particles; the slices' offsets
// go through shared memory, so that a thread's loads do not wait for them.
// With several rounds the sum goes on from the round before and reaches the
// potential in the last one: the same additions in the same order as in one.
__global__ void __launch_bounds__(GATHER_THREADS) k_sym_gather64(SymGather64Args a)
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
            for (int k = 0; k < m; k++) s += a.partial[slot[k] + j];
    }
    if (j >= nb) return;
    if (a.round + 1 < a.nrounds) a.run[a.ibeg[node] + j] = s;
    else a.pot[a.ibeg[node] + j] += s;
}

}  // namespace

void launch_pp_sym64(int kernel, const Sym64Args &a, cudaStream_t st)
{
    if (a.nblocks <= 0) return;
    if (kernel == K_REGCOULOMB) k_pp_sym64<K_REGCOULOMB, false><<<a.nblocks, S64_THREADS, 0, st>>>(a);
    else if (kernel == K_YUKAWA && a.far_exp) k_pp_sym64<K_YUKAWA, true><<<a.nblocks, S64_THREADS, 0, st>>>(a);
    else if (kernel == K_YUKAWA) k_pp_sym64<K_YUKAWA, false><<<a.nblocks, S64_THREADS, 0, st>>>(a);
    else k_pp_sym64<K_COULOMB, false><<<a.nblocks, S64_THREADS, 0, st>>>(a);
}

void launch_sym_gather64(const SymGather64Args &a, cudaStream_t st)
{
    if (a.nleaves > 0) k_sym_gather64<<<dim3(a.nleaves, SYM_MAX_LEAF / GATHER_THREADS), GATHER_THREADS, 0, st>>>(a);
}

}  // namespace bt
