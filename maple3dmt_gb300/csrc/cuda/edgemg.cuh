// Geometric multigrid preconditioner of the complex-FP32 inner solve.
//
// With r the residual of a right-hand side (d the row's diagonal, w = 0.4):
//
//     z0 = P V_e(P^T r) + G~ V_n(G~^T r) / (i omega) + w r / d
//     z  = z0 + w (r - A z0) / d
//
// P interpolates the uniform grid under the octree to its edges and V_e is one
// V(1,1) cycle of damped Jacobi on the nested uniform edge grids
// (host/edgemg.hpp): it removes the smooth curl part of the error, which SSOR
// leaves to the Krylov iteration.  V_n is a V(0,1) cycle for the
// divergence-correction Laplacian L on the octree's nodes and the uniform node
// grids: the gradient part of the error, as in gradcorr.cuh (A G~ = i omega Me
// G~).  On a uniform grid L is G^T diag(Me) G with the same coarse edge masses
// Me = P^T Me that the coarse edge operators C^T diag(W) C + i omega diag(Me)
// have on their diagonal, so both cycles need W (per mesh) and Me (per
// conductivity) alone.
//
// The iteration count no longer grows with the grid.  BiCGStab steps to a
// residual of 1e-7 at 0.01 Hz: 28 instead of 83 on 223 k edges in FP64 arithmetic
// (a prototype), 28 instead of 215 on 1.7 M edges in the mixed-precision solve.  The colour sweeps (2 x 9
// launches per application, each gathering rows of every other colour) become
// one matrix product with every row at once.
#pragma once

#include <cuda_runtime.h>

#include "gradcorr.cuh"
#include "host/edgemg.hpp"
#include "krylov.cuh"

namespace m3d {

constexpr int kEmgBottom = 16;     // grids of at most this many cells per side run in one block per right-hand side
constexpr float kEmgFine = kSmoothDamping;   // damping of the fine level's two Jacobi steps
constexpr float kEmgEdge = 0.5f;   // ... of the uniform edge grids
constexpr float kEmgNode = 0.6f;   // ... of the uniform node grids

struct EmgLevel {
    int n = 0;
    float h[3] = {};
    int ph = 0, pv = 0, pn = 0;    // planes that may hold free horizontal edges, vertical edges, nodes
    const float* w = nullptr;      // face weights
    float* me = nullptr;           // edge masses P^T Me, zero on edges that are not free
    // edge and node vectors, [entry][K]; on grids of the bottom kernels
    // [K][entry], a right-hand side's values together
    float2 *b = nullptr, *x = nullptr, *y = nullptr;
    float2 *nb = nullptr, *ny = nullptr, *nt = nullptr;
};

struct EmgDev {
    int n_levels = 0;
    EmgLevel lv[kEmgMaxLevels];
    int gap = 0;                        // fractions are in units of 2^-gap
    const int* p_base = nullptr;        // per permuted row (-1: identity or padding row)
    const unsigned* p_code = nullptr;
    const int *r_ptr = nullptr, *r_row = nullptr;
    const float* r_w = nullptr;
    const int* n_base = nullptr;        // per octree node (-1: Dirichlet)
    const unsigned* n_code = nullptr;
    const int *nr_ptr = nullptr, *nr_node = nullptr;
    const float* nr_w = nullptr;
    // transfer rows that a block sums each (emg_long_rows)
    const int *r_long = nullptr, *nr_long = nullptr;
    int n_r_long = 0, n_nr_long = 0;
};

// The rows of a transfer (CSR row pointers) that take a block each.
std::vector<int> emg_long_rows(const std::vector<int>& ptr, bool nodes);

// Coarse edge masses for the current conductivity (Me per permuted row).
void emg_set_mass(const EmgDev& g, const double* Me, cudaStream_t s, long long* launches);

// z0 of the preconditioner: the edge cycle on c.stream, the node cycle on
// c.gc_stream when set (forked and joined here); r, z0 [n_pad][K].
template <int K>
void emg_coarse_k(const KrylovCtx<float>& c, const float2* r, float2* z0);

// z = V(1,1) of gc.lv[0].b for the divergence-correction Laplacian: octree
// nodes, then the uniform node grids; symmetric, so PCG can use it.
template <int K>
void emg_node_precond_k(const EmgDev& g, const GcDev& gc, float2* z, cudaStream_t s, long long* launches);

}  // namespace m3d
