// See edgemg.hpp.
#include "host/edgemg.hpp"

#include <algorithm>
#include <cmath>

namespace m3d {

namespace {

constexpr double kMu0 = 4.0e-7 * 3.14159265358979323846;

// 2^gap * u as an integer; false if u is not a multiple of 2^-gap
bool grid_coord(double u, int scale, int& m) {
    const double v = u * scale;
    m = (int)std::lround(v);
    return std::abs(v - m) < 1e-3;
}

}  // namespace

// A 4^3 grid is the coarsest one; more than three levels of leaves under one
// coarse grid leave too much to the fine level's Jacobi steps, and the packed
// fractions hold three levels; up to 256^3 cells the kernels' thread numbers
// (eight pairs of right-hand sides per edge entry) fit in 32 bits.
bool emg_levels_ok(int lmin, int lmax) { return lmin >= 2 && lmin <= 8 && lmax - lmin <= 3; }

void emg_build(const HostLayout& L, const std::vector<char>& free, const std::vector<char>& node_free,
               const std::vector<int>& iperm, int n_pad, double air, EmgHost& H) {
    H = EmgHost();
    if (L.nc == 0) return;
    const int lmin = *std::min_element(L.clevel.begin(), L.clevel.end());
    const int lmax = *std::max_element(L.clevel.begin(), L.clevel.end());
    if (!emg_levels_ok(lmin, lmax)) return;
    H.lmin = lmin;
    H.gap = lmax - lmin;
    const double ext[3] = {L.domain[1] - L.domain[0], L.domain[3] - L.domain[2], L.domain[5] - L.domain[4]};
    const double lo[3] = {L.domain[0], L.domain[2], L.domain[4]};
    for (int n = 1 << lmin; n >= 4 && (int)H.lv.size() < kEmgMaxLevels; n /= 2) {
        EmgHostLevel g;
        g.n = n;
        for (int a = 0; a < 3; ++a) g.h[a] = ext[a] / n;
        for (int k = 1; k < n; ++k)
            if (lo[2] + k * g.h[2] <= air) g.planes_h = k + 1;
        for (int k = 0; k < n; ++k)
            if (lo[2] + (k + 0.5) * g.h[2] <= air) g.planes_v = k + 1;
        for (int k = 1; k < n; ++k)
            if (lo[2] + (k + 0.5) * g.h[2] <= air) g.planes_n = k + 1;
        H.lv.push_back(std::move(g));
    }
    const EmgHostLevel& G0 = H.lv[0];
    const int n0 = G0.n, S = 1 << H.gap;
    auto free_edge = [&](const EmgHostLevel& g, int D, const int* q) {
        for (int a = 0; a < 3; ++a)
            if (a != D && (q[a] <= 0 || q[a] >= g.n)) return false;
        return D == 2 ? q[2] < g.planes_v : q[2] < g.planes_h;
    };
    auto free_node = [&](const EmgHostLevel& g, const int* q) {
        for (int a = 0; a < 3; ++a)
            if (q[a] <= 0 || q[a] >= g.n) return false;
        return q[2] < g.planes_n;
    };

    // ---- edges: prolongation rows and their transpose ----
    H.p_base.assign(n_pad, -1);
    H.p_code.assign(n_pad, 0);
    struct Entry { int col, row; float w; };
    auto transpose = [](std::vector<Entry>& ent, long n_col, std::vector<int>& ptr, std::vector<int>& row,
                        std::vector<float>& w) {
        ptr.assign(n_col + 1, 0);
        for (const Entry& e : ent) ++ptr[e.col + 1];
        for (long c = 0; c < n_col; ++c) ptr[c + 1] += ptr[c];
        row.resize(ent.size());
        w.resize(ent.size());
        std::vector<int> pos(ptr.begin(), ptr.end() - 1);
        for (const Entry& e : ent) {
            const int p = pos[e.col]++;
            row[p] = e.row;
            w[p] = e.w;
        }
    };
    {
        std::vector<int> at(n_pad, -1);
        for (int e = 0; e < L.ne; ++e)
            if (free[e]) at[iperm[e]] = e;
        std::vector<Entry> ent;
        ent.reserve((size_t)L.ne * 2);
        for (int r = 0; r < n_pad; ++r) {
            const int e = at[r];
            if (e < 0) continue;
            const int D = L.edir[e];
            const double x[3] = {L.ex[e], L.ey[e], L.ez[e]};
            int base[3], fr[3] = {0, 0, 0};
            for (int a = 0; a < 3; ++a) {
                const double u = (x[a] - lo[a]) / ext[a] * n0;
                if (a == D) {
                    base[a] = std::min(std::max((int)std::floor(u), 0), n0 - 1);
                } else {
                    int m;
                    if (!grid_coord(u, S, m)) return;
                    base[a] = std::min(std::max(m >> H.gap, 0), n0 - 1);
                    fr[a] = m - (base[a] << H.gap);
                    if (fr[a] < 0 || fr[a] > S) return;
                }
            }
            const int a = D == 0 ? 1 : 0, b = D == 2 ? 1 : 2;
            H.p_base[r] = (int)emg_entry(n0, D, base[0], base[1], base[2]);
            H.p_code[r] = (uint32_t)D | (uint32_t)fr[a] << 2 | (uint32_t)fr[b] << 6;
            for (int s = 0; s < 4; ++s) {
                int q[3] = {base[0], base[1], base[2]};
                q[a] += s & 1;
                q[b] += s >> 1;
                const float w = (float)((s & 1 ? fr[a] : S - fr[a]) * (s >> 1 ? fr[b] : S - fr[b])) / (float)(S * S);
                if (w > 0.0f && free_edge(G0, D, q))
                    ent.push_back({(int)emg_entry(n0, D, q[0], q[1], q[2]), r, w});
            }
        }
        transpose(ent, emg_entries(n0), H.r_ptr, H.r_row, H.r_w);
    }

    // ---- nodes ----
    {
        H.n_base.assign(L.nn, -1);
        H.n_code.assign(L.nn, 0);
        std::vector<double> np(3 * (size_t)L.nn, 0.0);
        for (int e = 0; e < L.ne; ++e) {
            const double x[3] = {L.ex[e], L.ey[e], L.ez[e]};
            for (int s = 0; s < 2; ++s) {
                const int v = s ? L.n2[e] : L.n1[e];
                for (int a = 0; a < 3; ++a)
                    np[3 * (size_t)v + a] = x[a] + (a == L.edir[e] ? (s ? 0.5 : -0.5) * L.elen[e] : 0.0);
            }
        }
        std::vector<Entry> ent;
        ent.reserve((size_t)L.nn * 2);
        for (int v = 0; v < L.nn; ++v) {
            if (!node_free[v]) continue;
            int base[3], fr[3];
            for (int a = 0; a < 3; ++a) {
                int m;
                if (!grid_coord((np[3 * (size_t)v + a] - lo[a]) / ext[a] * n0, S, m)) return;
                base[a] = std::min(std::max(m >> H.gap, 0), n0 - 1);
                fr[a] = m - (base[a] << H.gap);
                if (fr[a] < 0 || fr[a] > S) return;
            }
            H.n_base[v] = (int)emg_point(n0, base[0], base[1], base[2]);
            H.n_code[v] = (uint32_t)fr[0] | (uint32_t)fr[1] << 4 | (uint32_t)fr[2] << 8;
            for (int s = 0; s < 8; ++s) {
                int q[3];
                float w = 1.0f;
                for (int a = 0; a < 3; ++a) {
                    const int t = (s >> a) & 1;
                    q[a] = base[a] + t;
                    w *= (float)(t ? fr[a] : S - fr[a]) / (float)S;
                }
                if (w > 0.0f && free_node(G0, q)) ent.push_back({(int)emg_point(n0, q[0], q[1], q[2]), v, w});
            }
        }
        transpose(ent, emg_points(n0), H.nr_ptr, H.nr_node, H.nr_w);
    }

    // ---- face weights: level 0 from the octree's faces ----
    {
        std::vector<double> w(emg_entries(n0), 0.0);
        for (int f = 0; f < L.nf; ++f) {
            if (L.dead_f[f]) continue;
            const int D = L.fnorm[f];
            const double area0 = ext[(D + 1) % 3] * ext[(D + 2) % 3];
            const double size = std::sqrt(L.farea[f] / area0);   // 2^-level of the face
            const double x[3] = {L.fx[f], L.fy[f], L.fz[f]};
            double ratio = size * n0 * size * n0;   // fine over coarse area
            if (D == 2) {
                if (x[2] > air) continue;
            } else if (x[2] > air) {
                // vertical face above the surface: only its bottom edge can be free
                if (x[2] - 0.5 * size * ext[2] > air) continue;
                ratio = size * n0;
            }
            int q[3];
            double fr = 0.0;
            for (int a = 0; a < 3; ++a) {
                const double u = (x[a] - lo[a]) / ext[a] * n0;
                q[a] = std::min(std::max((int)std::floor(u + 1e-9), 0), n0 - 1);
                if (a == D) fr = std::min(std::max(u - q[a], 0.0), 1.0);
            }
            const double m = L.fdual[f] / (kMu0 * L.farea[f]) * ratio * ratio;
            w[emg_entry(n0, D, q[0], q[1], q[2])] += m * (1.0 - fr);
            ++q[D];
            w[emg_entry(n0, D, q[0], q[1], q[2])] += m * fr;
        }
        // coarser grids from the next finer one
        std::vector<std::vector<double>> wl;
        wl.push_back(std::move(w));
        for (size_t l = 1; l < H.lv.size(); ++l) {
            const EmgHostLevel &C = H.lv[l], &F = H.lv[l - 1];
            const std::vector<double>& wf = wl.back();
            std::vector<double> wc(emg_entries(C.n), 0.0);
            auto dim = [](int n, int D, int a) { return n + (a == D ? 1 : 0); };   // faces of normal D along a
            for (int D = 0; D < 3; ++D)
                for (int k = 0; k < dim(F.n, D, 2); ++k)
                    for (int j = 0; j < dim(F.n, D, 1); ++j)
                        for (int i = 0; i < dim(F.n, D, 0); ++i) {
                            double v = wf[emg_entry(F.n, D, i, j, k)];
                            if (v == 0.0) continue;
                            // vertical faces just above the surface (k = planes_v): ratio of lengths
                            const bool top = D != 2 && k >= F.planes_v;
                            v *= top ? 0.25 : 0.0625;
                            int q[3] = {i, j, k};
                            const int o = q[D] & 1;
                            for (int a = 0; a < 3; ++a) q[a] = std::min(q[a] >> 1, dim(C.n, D, a) - 1);
                            wc[emg_entry(C.n, D, q[0], q[1], q[2])] += o ? 0.5 * v : v;
                            if (o) {
                                ++q[D];
                                wc[emg_entry(C.n, D, q[0], q[1], q[2])] += 0.5 * v;
                            }
                        }
            wl.push_back(std::move(wc));
        }
        for (size_t l = 0; l < H.lv.size(); ++l) H.lv[l].w.assign(wl[l].begin(), wl[l].end());
    }
    H.ok = true;
}

}  // namespace m3d
