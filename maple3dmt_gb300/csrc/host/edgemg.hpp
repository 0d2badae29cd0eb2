// Geometric multigrid data of the edge system (no counterpart in the
// reference): nested uniform grids under the octree, built once per mesh.
//
// Every leaf is at level lmin or finer, so the uniform grid of (2^lmin)^3
// cells, and that grid halved down to 4^3, are nested coarse grids of the
// octree.  An edge value is the tangential mean along the edge, so
// interpolation from a uniform grid is constant along the edge direction and
// bilinear across it (the lowest-order Nedelec interpolation), at most four
// coarse edges per octree edge; node values interpolate trilinearly.
//
// The coarse curl-curl operators are C^T diag(W) C with the uniform grid's
// own curl C and one weight per coarse face.  The interpolation commutes with
// the curl, so the Galerkin product is C^T (Pf^T Mf^-1 Pf) C with the face
// interpolation Pf; W lumps that face matrix by rows.  This keeps the 13-point
// stencil of the uniform grid (the Galerkin product has 33 points) and needs
// no matrix storage beyond W.  Faces just above the earth's surface are
// special: the edges above the air threshold are Dirichlet edges of the
// solve, so only the circulation of the surface edge remains, in the first
// fine layer alone.
#pragma once

#include <cstdint>
#include <vector>

#include "host/layout.hpp"

namespace m3d {

constexpr int kEmgMaxLevels = 12;

struct EmgHostLevel {
    int n = 0;               // cells per side
    double h[3] = {};        // cell size
    int planes_h = 0;        // horizontal-edge planes k < planes_h may be free (z_k <= air)
    int planes_v = 0;        // vertical-edge layers k < planes_v may be free
    int planes_n = 0;        // node planes k < planes_n may be free
    std::vector<float> w;    // face weights
};

struct EmgHost {
    bool ok = false;
    int lmin = 0, gap = 0;   // coarsest leaf level, levels between it and the finest leaf
    std::vector<EmgHostLevel> lv;
    // prolongation of level-0 edges to permuted rows: base edge id (-1: the row is not free), code = dir |
    // fa << 2 | fb << 6 with the fractions across (the two other directions in order) in units of 2^-gap
    std::vector<int> p_base;
    std::vector<uint32_t> p_code;
    // its transpose: free level-0 edge -> permuted rows and weights
    std::vector<int> r_ptr, r_row;
    std::vector<float> r_w;
    // the same for nodes: octree node -> level-0 node (trilinear), code = fx | fy << 4 | fz << 8
    std::vector<int> n_base;
    std::vector<uint32_t> n_code;
    std::vector<int> nr_ptr, nr_node;
    std::vector<float> nr_w;
};

// Index helpers of an n^3 grid: the points (i, j, k), x fastest; the edge of
// direction D that starts at a point, and the face of normal D whose lowest
// corner it is, are entry 3 point + D (entries beyond the grid stay zero).
inline long emg_point(int n, int i, int j, int k) { return ((long)k * (n + 1) + j) * (n + 1) + i; }
inline long emg_points(int n) { return (long)(n + 1) * (n + 1) * (n + 1); }
inline long emg_entries(int n) { return 3 * emg_points(n); }
inline long emg_entry(int n, int D, int i, int j, int k) { return 3 * emg_point(n, i, j, k) + D; }

// The rule: leaves at levels lmin to lmax.
bool emg_levels_ok(int lmin, int lmax);

// free[e]: edge e (reference numbering) is a row of the eliminated system;
// node_free[v]: node v is not a Dirichlet node; iperm: edge -> permuted row;
// n_pad: permuted rows.  ok stays false for meshes outside the rule.
void emg_build(const HostLayout& L, const std::vector<char>& free, const std::vector<char>& node_free,
               const std::vector<int>& iperm, int n_pad, double air, EmgHost& H);

}  // namespace m3d
