// bt_device.h -- launchers of the barytree_b200 CUDA kernels (internal).
#pragma once

#include <cuda_runtime.h>

#include <vector>
#include <cstdint>

namespace bt {

// FP64 evaluation kernels: outputs per work item, and the segments that each
// output's interaction list is summed in.  With `partial` set, every segment
// of an item has a block of its own and leaves its sums there (pstride outputs
// per segment); the launcher adds them in order.  Without it one block sums
// the segments.  Both give the same bits.
constexpr int EV_THREADS = 128;
constexpr int EV_CHUNK = 2 * EV_THREADS;
constexpr int EV_SEGS = 16;
// Resident blocks per SM that their register budget is sized for: 4 (128
// registers); 5 and 6 (102 and 80 registers) measured 1 to 2 % slower.
constexpr int EV_MINB = 4;
// Part s of EV_SEGS of the list [b, e).
__host__ __device__ inline int64_t seg_begin(int64_t b, int64_t e, int s) { return b + (e - b) * s / EV_SEGS; }
// In a particle-output list: the source node's box meets the target leaf's, so
// a source can coincide with a target and the skipping rule is tested.
constexpr int EV_MEETS = (int)0x80000000;

// Whether exp(-kappa r) stays within 2^-1021.4 and 2^1021.4 for every r up to
// `extent`, the range of the Yukawa kernels' short exponential.
inline bool exp64_range(double kappa, double extent) { return (kappa < 0.0 ? -kappa : kappa) * extent < 708.0; }

struct EvalTargetsArgs {
    int n, nitems;
    const int2 *items;            // (target leaf unit, chunk of EV_CHUNK targets), sorted by cost
    const int *leaf_node;         // unit -> target node
    const int *t_ibeg, *t_numpar;
    const int64_t *a_off; const int *a_idx;   // source clusters per unit
    const int64_t *d_off; const int *d_idx;   // source nodes per unit (with EV_MEETS)
    const int *s_ibeg, *s_numpar;
    const double *s_grid, *Q;
    const double *sx, *sy, *sz, *sq;
    const double *tx, *ty, *tz;
    double kp, kp2;                             // kernel_params[0], [1]
    double *pot;
    double *partial = nullptr;
    size_t pstride = 0;
    bool far_exp = false;         // Yukawa: exponentials beyond exp64's range occur
};

struct EvalGridsArgs {
    int n, nitems;
    const int2 *items;            // (target node, chunk of EV_CHUNK grid points (Hermite: EV_THREADS))
    const double *t_grid;
    const int64_t *c_off; const int *c_idx;   // source clusters (M2L) per target node
    const int64_t *p_off; const int *p_idx;   // source nodes (CP) per target node
    const int *s_ibeg, *s_numpar;
    const double *s_grid, *Q;
    const double *sx, *sy, *sz, *sq;
    double kp, kp2;                             // kernel_params[0], [1]
    double *Phi;
    double *partial = nullptr;                  // Lagrange only
    size_t pstride = 0;
    bool far_exp = false;
};

void launch_p2m(int n, bool hermite, int nleaves, const int *leaves, int nnodes, const int *ibeg, const int *numpar,
                const double *grid, const double *box_len, const double *ww, const double *sx, const double *sy,
                const double *sz, const double *sq, double *Q, cudaStream_t st);
// Hermite P2M over particle chunks (see bt_device.cu).  slot < 0: the chunk
// is its node's only one and writes Q directly.
struct HermChunk {
    int node, begin, count, slot;
};
// Chunks of every node and, for nodes with several chunks, (node, first slot,
// slot count); returns the number of partial slots (8 (n+1)^3 doubles each).
int hermite_chunks(int nnodes, const int *ibeg, const int *numpar, std::vector<HermChunk> &chunks,
                   std::vector<int3> &red);
void launch_p2m_hermite(int n, int nchunks, const HermChunk *chunks, int nred, const int3 *red, const double *grid,
                        const double *box_len, const double *ww, const double *sx, const double *sy, const double *sz,
                        const double *sq, double *Q, double *partial, cudaStream_t st);
// Q of every node with several chunks: the sum of its partial moments in chunk order.
void launch_hermite_reduce(int n, int nred, const int3 *red, const double *partial, double *Q, cudaStream_t st);
void launch_m2m(int n, int nparents, const int *parents, const int *nchild, const int *child, const double *grid,
                double *Q, cudaStream_t st);
void launch_l2l(int n, int nparents, const int *parents, const int *nchild, const int *child, const double *grid,
                double *Phi, cudaStream_t st);
void launch_eval_targets(int kernel, bool hermite, const EvalTargetsArgs &a, cudaStream_t st);
// Whether `items` work items are too few to fill the GPU with one block each
// (then every segment gets its own block).
bool eval64_split(size_t items);
// out = the sums of the segments, in order, for the items' targets (chunk a
// multiple of 32 up to 1024).
void launch_sum_segments(int nitems, const int2 *items, int chunk, const int *leaf_node, const int *ibeg,
                         const int *numpar, const double *partial, size_t pstride, double *out, cudaStream_t st);
void launch_eval_grids(int kernel, bool hermite, const EvalGridsArgs &a, cudaStream_t st);
void launch_l2p(int n, bool hermite, int nitems, const int2 *items, const int *leaf_node, const int *parent,
                const int *t_ibeg, const int *t_numpar, const double *t_grid, const double *box_len,
                const double *ww, const double *Phi, const double *tx, const double *ty, const double *tz,
                double *pot, cudaStream_t st, const double *mult = nullptr);
void launch_scatter(int n, const int *order, const double *src, double *dst, cudaStream_t st);
// dst[i] = src[order[i]] (inputs in caller order -> tree order)
void launch_gather(int n, const int *order, const double *src, double *dst, cudaStream_t st);
float run_probe(int which, int sms, double *ops, void *scratch, cudaStream_t st);
// Parts that the direct sum splits its sources into (partial sums: parts * nt
// doubles when parts > 1).
int direct_parts(int nt, int ns);
// out = the sum of `parts` arrays of n values, in order.
void launch_sum_parts(int n, int parts, const double *partial, double *out, cudaStream_t st);
void launch_direct(int kernel, int nt, int ns, const double *tx, const double *ty, const double *tz,
                   const double *sx, const double *sy, const double *sz, const double *sq, double kp, double kp2,
                   double *partial, double *out, cudaStream_t st);

}  // namespace bt
