// bt_sym.h -- symmetric near-field pairs (internal).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace bt {

// Largest leaf the symmetric pass takes (particles).
constexpr int SYM_MAX_LEAF = 2048;
// Smallest leaf whose pairs the FP64 path's symmetric pass takes (a rule per
// pair, so that a batch takes the pairs its systems take in separate calls).
// Measured with the line at 128, uniform systems, whole calls without and with
// the pass, Coulomb (Yukawa): leaves of 195 particles 5.5 and 5.2 ms (13.1 and
// 11.0), of 244 6.2 and 5.8 (14.9 and 12.6), of 312 8.9 and 8.1 (22.1 and
// 17.9), of 400 14.0 and 11.5 (35.8 and 26.7); of 1560, above the line, 5.8 and
// 5.0 (13.4 and 10.3).  So the line is higher than it need be: leaves below it
// keep the sums of every direction.
constexpr int SYM64_MIN_LEAF = 512;

// Threads (particles) per block of the gathers.
constexpr int GATHER_THREADS = 128;

// Particles of A per block: a pair of leaves (A, B) is evaluated by
// sym_parts(numpar[A]) blocks.
constexpr int SYM_PART = 512;
inline int sym_parts(int na) { return (na + SYM_PART - 1) / SYM_PART; }

struct SymArgs {
    int nblocks;
    const int2 *block;            // (pair, part of A)
    const int2 *pair;             // (A, B) leaf nodes, A != B
    // per pair: A's sums at slot[p], B's from part k at slot[p] + numpar[A] + k numpar[B]
    const int64_t *slot;
    const int *ibeg, *numpar;     // per node (the target tree is the source tree)
    const double *ctr;            // node centres, 3 per node
    const float4 *pos;            // particles relative to their leaf centre, with charge
    float *partial;               // the pairs' potentials at their particles
    float kc;                     // mixed_kernel_constant()
    // pairs of leaves within the close-pair distance of each other (launch_pp_sym_close)
    const double *rad;            // node radii
    const double *box;            // node boxes, x0 x1 y0 y1 z0 z1 per node
    const double *x64, *y64, *z64, *q64;   // FP64 particles in tree order
    double kp;                    // kernel parameter (FP64 close pairs)
};

struct SymGatherArgs {
    int nleaves;
    const int *leaf_node;
    const int *ibeg, *numpar;
    // partial vectors addressed to each unit, in pair order: those of round r
    // in_off[r * nleaves + unit] .. in_off[(r + 1) * nleaves + unit]
    const int64_t *in_off;
    const int64_t *in_slot;
    const float *partial;
    double *pot;                  // += the sum of all rounds' partial vectors, FP64, in that order
    double *run = nullptr;        // the sum so far, between rounds (several rounds only)
    int round = 0, nrounds = 1;
};

// Pairs whose leaf boxes are farther apart than the close-pair distance.
void launch_pp_sym(int kernel, const SymArgs &a, cudaStream_t st);
// Pairs whose boxes lie within it: FP32 distances below the close-pair
// distance are clamped to it, and each clamped pair's two terms are replaced
// by FP64 ones (from the FP64 particles) before the slices are written.
void launch_pp_sym_close(int kernel, const SymArgs &a, cudaStream_t st);
void launch_sym_gather(const SymGatherArgs &a, cudaStream_t st);

// The FP64 path's pairs (bt_sym64.cu): one kernel for all of them, FP64 slices.
struct Sym64Args {
    int nblocks;
    const int2 *block, *pair;
    const int64_t *slot;
    const int *ibeg, *numpar;
    const double *x, *y, *z, *q;  // particles in tree order
    double *partial;
    double kp;
    bool far_exp = false;         // Yukawa: exponentials beyond exp64's range occur
};

struct SymGather64Args {
    int nleaves;
    const int *leaf_node;
    const int *ibeg, *numpar;
    const int64_t *in_off, *in_slot;
    const double *partial;
    double *pot, *run = nullptr;
    int round = 0, nrounds = 1;
};

void launch_pp_sym64(int kernel, const Sym64Args &a, cudaStream_t st);
void launch_sym_gather64(const SymGather64Args &a, cudaStream_t st);

}  // namespace bt
