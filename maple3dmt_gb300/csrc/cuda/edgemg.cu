// Kernels of the geometric multigrid preconditioner (see edgemg.cuh).
#include "edgemg.cuh"

#include <algorithm>
#include <stdexcept>
#include <type_traits>

namespace m3d {

using namespace dev;

namespace {

constexpr int kNT = 256;
constexpr int kLongRow = 24;    // transfer rows longer than this (two levels of refinement) are summed by a block
constexpr int kLongNT = 128;

template <int D> using Dir = std::integral_constant<int, D>;   // direction tag

void ck(long long* launches) {
    if (launches) ++*launches;
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) throw std::runtime_error(cudaGetErrorString(e));
}

// One complex value, or the values of two neighbouring right-hand sides (a
// 16-byte load), with the matching pair of angular frequencies.
template <class V> struct Om;
template <> struct Om<float2> { float a; };
template <> struct Om<float4> { float a, b; };

__device__ __forceinline__ float2 vzero(float2*) { return make_float2(0.f, 0.f); }
__device__ __forceinline__ float4 vzero(float4*) { return make_float4(0.f, 0.f, 0.f, 0.f); }
template <class V> __device__ __forceinline__ V vz() { return vzero((V*)nullptr); }
__device__ __forceinline__ float2 operator+(float2 p, float2 q) { return make_float2(p.x + q.x, p.y + q.y); }
__device__ __forceinline__ float2 operator-(float2 p, float2 q) { return make_float2(p.x - q.x, p.y - q.y); }
__device__ __forceinline__ float2 operator*(float s, float2 q) { return make_float2(s * q.x, s * q.y); }
__device__ __forceinline__ float4 operator+(float4 p, float4 q) {
    return make_float4(p.x + q.x, p.y + q.y, p.z + q.z, p.w + q.w);
}
__device__ __forceinline__ float4 operator-(float4 p, float4 q) {
    return make_float4(p.x - q.x, p.y - q.y, p.z - q.z, p.w - q.w);
}
__device__ __forceinline__ float4 operator*(float s, float4 q) {
    return make_float4(s * q.x, s * q.y, s * q.z, s * q.w);
}
// i omega m q
__device__ __forceinline__ float2 imass(Om<float2> o, float m, float2 q) {
    const float s = o.a * m;
    return make_float2(-s * q.y, s * q.x);
}
__device__ __forceinline__ float4 imass(Om<float4> o, float m, float4 q) {
    const float s = o.a * m, t = o.b * m;
    return make_float4(-s * q.y, s * q.x, -t * q.w, t * q.z);
}
// w q / (S + i omega m); 0 where the edge has no diagonal
__device__ __forceinline__ float2 idiag(Om<float2> o, float w, float S, float m, float2 q) {
    const float s = o.a * m, n = S * S + s * s;
    const float f = n > 0.0f ? w / n : 0.0f;
    return make_float2(f * (S * q.x + s * q.y), f * (S * q.y - s * q.x));
}
__device__ __forceinline__ float4 idiag(Om<float4> o, float w, float S, float m, float4 q) {
    const float2 a = idiag(Om<float2>{o.a}, w, S, m, make_float2(q.x, q.y));
    const float2 b = idiag(Om<float2>{o.b}, w, S, m, make_float2(q.z, q.w));
    return make_float4(a.x, a.y, b.x, b.y);
}

struct Omegas { float v[kMaxRhs]; };
__device__ __forceinline__ Om<float4> om_of(const Omegas& o, int h, float4*) { return {o.v[2 * h], o.v[2 * h + 1]}; }

// index helpers of an n^3 grid (host/edgemg.hpp)
template <int D> __device__ __forceinline__ int ex(int n) { return D == 0 ? n : n + 1; }
template <int D> __device__ __forceinline__ int ey(int n) { return D == 1 ? n : n + 1; }
template <int D> __device__ __forceinline__ int eid(int n, int i, int j, int k) {
    return D * n * (n + 1) * (n + 1) + (k * ey<D>(n) + j) * ex<D>(n) + i;
}
template <int D> __device__ __forceinline__ int fid(int n, int i, int j, int k) {
    return D * n * n * (n + 1) + (k * (D == 1 ? n + 1 : n) + j) * (D == 0 ? n + 1 : n) + i;
}
__device__ __forceinline__ int nid(int n, int i, int j, int k) { return (k * (n + 1) + j) * (n + 1) + i; }

// Curl-curl row of edge (D; i, j, k) and its diagonal: four faces, thirteen
// points; at(e) reads the vector at edge e.
template <int D, class V, class At>
__device__ __forceinline__ V curl_row(const EmgLevel& L, int i, int j, int k, V xc, const At& at, float& S) {
    const int n = L.n;
    V acc = vz<V>();
    S = 0.0f;
    auto dir = [&](auto tag) {
        constexpr int A = decltype(tag)::value;      // transverse direction
        constexpr int B = 3 - D - A;             // normal of the two faces
        constexpr int ai = A == 0, aj = A == 1, ak = A == 2, di = D == 0, dj = D == 1, dk = D == 2;
        const float wp = __ldg(&L.w[fid<B>(n, i, j, k)]), wm = __ldg(&L.w[fid<B>(n, i - ai, j - aj, k - ak)]);
        const float hd = L.h[D], ha = L.h[A];
        const V xp = at(eid<D>(n, i + ai, j + aj, k + ak)), xm = at(eid<D>(n, i - ai, j - aj, k - ak));
        const V a0 = at(eid<A>(n, i, j, k)), a1 = at(eid<A>(n, i + di, j + dj, k + dk));
        const V b0 = at(eid<A>(n, i - ai, j - aj, k - ak)), b1 = at(eid<A>(n, i - ai + di, j - aj + dj, k - ak + dk));
        const V cp = hd * (xc - xp) + ha * (a1 - a0);
        const V cm = hd * (xm - xc) + ha * (b1 - b0);
        acc = acc + hd * (wp * cp - wm * cm);
        S += hd * hd * (wp + wm);
    };
    dir(Dir<D == 0 ? 1 : 0>{});
    dir(Dir<D == 2 ? 1 : 2>{});
    return acc;
}

template <int D> __device__ __forceinline__ float edge_diag(const EmgLevel& L, int i, int j, int k) {
    const int n = L.n;
    constexpr int A = D == 0 ? 1 : 0, B = D == 2 ? 1 : 2;
    // faces of normal A are spanned by D and B, and the other way round
    const float sa = __ldg(&L.w[fid<A>(n, i, j, k)]) + __ldg(&L.w[fid<A>(n, i - (B == 0), j - (B == 1), k - (B == 2))]);
    const float sb = __ldg(&L.w[fid<B>(n, i, j, k)]) + __ldg(&L.w[fid<B>(n, i - (A == 0), j - (A == 1), k - (A == 2))]);
    return L.h[D] * L.h[D] * (sa + sb);
}

// interior of the grid across direction D and not above the surface
template <int D> __device__ __forceinline__ bool edge_free(const EmgLevel& L, int i, int j, int k) {
    const int n = L.n;
    if (D != 0 && (i <= 0 || i >= n)) return false;
    if (D != 1 && (j <= 0 || j >= n)) return false;
    if (D != 2) return k > 0 && k < L.ph;
    return k < L.pv;
}
__device__ __forceinline__ bool node_free(const EmgLevel& L, int i, int j, int k) {
    return i > 0 && i < L.n && j > 0 && j < L.n && k > 0 && k < L.pn;
}

// Work split of an edge kernel: blockIdx.y is a plane of one direction (the
// planes that may be free and the one above them, which is written as zeros
// because the stencils read it), threads run over (row of the plane, lanes).
__host__ __device__ inline int edge_planes(const EmgLevel& L, int D) {
    const int p = (D == 2 ? L.pv : L.ph) + 1, most = D == 2 ? L.n : L.n + 1;
    return p < most ? p : most;
}
inline int edge_planes_all(const EmgLevel& L) { return 2 * edge_planes(L, 0) + edge_planes(L, 2); }
__host__ __device__ inline int node_planes(const EmgLevel& L) { return L.pn + 2 < L.n + 1 ? L.pn + 2 : L.n + 1; }

template <int H, class F> __device__ __forceinline__ void each_edge(const EmgLevel& L, const F& f) {
    const int p0 = edge_planes(L, 0);
    const int t = blockIdx.x * kNT + threadIdx.x;
    const int q = t / H, h = t % H;
    const int y = blockIdx.y, n = L.n;
    if (y < p0) {
        if (q < n * (n + 1)) f(Dir<0>{}, q % n, q / n, y, h);
    } else if (y < 2 * p0) {
        if (q < (n + 1) * n) f(Dir<1>{}, q % (n + 1), q / (n + 1), y - p0, h);
    } else {
        if (q < (n + 1) * (n + 1)) f(Dir<2>{}, q % (n + 1), q / (n + 1), y - 2 * p0, h);
    }
}
template <int H, class F> __device__ __forceinline__ void each_node(const EmgLevel& L, const F& f) {
    const int t = blockIdx.x * kNT + threadIdx.x;
    const int q = t / H, h = t % H, n1 = L.n + 1;
    if (q < n1 * n1) f(q % n1, q / n1, (int)blockIdx.y, h);
}
template <int K> dim3 edge_grid(const EmgLevel& L) {
    const long rows = (long)(L.n + 1) * (L.n + 1) * (K / 2);
    return dim3((unsigned)((rows + kNT - 1) / kNT), (unsigned)edge_planes_all(L));
}
template <int K> dim3 node_grid(const EmgLevel& L) {
    const long rows = (long)(L.n + 1) * (L.n + 1) * (K / 2);
    return dim3((unsigned)((rows + kNT - 1) / kNT), (unsigned)node_planes(L));
}

__host__ __device__ __forceinline__ float4* f4(float2* p) { return reinterpret_cast<float4*>(p); }
__host__ __device__ __forceinline__ const float4* f4(const float2* p) { return reinterpret_cast<const float4*>(p); }

// ---------------------------------------------------------------------------
// coarse edge masses
// ---------------------------------------------------------------------------
__global__ void k_mass0(EmgDev g, const double* __restrict__ Me, int n) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    double s = 0.0;
    for (int q = g.r_ptr[c]; q < g.r_ptr[c + 1]; ++q) s += (double)g.r_w[q] * Me[g.r_row[q]];
    g.lv[0].me[c] = (float)s;
}

// sum over the fine edges of a coarse edge: 2 along it, (1/2, 1, 1/2) across
template <int D, class V, class At>
__device__ __forceinline__ V gather_edge(int n, int I, int J, int Kk, const At& at) {
    V s = vz<V>();
#pragma unroll
    for (int b = -1; b <= 1; ++b)
#pragma unroll
        for (int a = -1; a <= 1; ++a) {
            const float w = (a ? 0.5f : 1.0f) * (b ? 0.5f : 1.0f);
            const int i = 2 * I + (D == 0 ? 0 : a), j = 2 * J + (D == 1 ? 0 : (D == 0 ? a : b)),
                      k = 2 * Kk + (D == 2 ? 0 : b);
            const int e = eid<D>(n, i, j, k), f = eid<D>(n, i + (D == 0), j + (D == 1), k + (D == 2));
            s = s + w * (at(e) + at(f));
        }
    return s;
}

struct F1 { float v; };
__device__ __forceinline__ F1 vzero(F1*) { return {0.f}; }
__device__ __forceinline__ F1 operator+(F1 a, F1 b) { return {a.v + b.v}; }
__device__ __forceinline__ F1 operator*(float s, F1 b) { return {s * b.v}; }

__global__ void k_mass(EmgLevel F, EmgLevel C) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, n = C.n;
    auto put = [&](auto tag, int q) {
        constexpr int D = decltype(tag)::value;
        const int i = q % ex<D>(n), j = q / ex<D>(n) % ey<D>(n), k = q / (ex<D>(n) * ey<D>(n));
        if (!edge_free<D>(C, i, j, k)) return;
        C.me[eid<D>(n, i, j, k)] = gather_edge<D, F1>(F.n, i, j, k, [&](int e) { return F1{F.me[e]}; }).v;
    };
    const int per = n * (n + 1) * (n + 1);
    if (t < per) put(Dir<0>{}, t);
    else if (t < 2 * per) put(Dir<1>{}, t - per);
    else if (t < 3 * per) put(Dir<2>{}, t - 2 * per);
}

// ---------------------------------------------------------------------------
// edge cycle
// ---------------------------------------------------------------------------

// b0 = P^T r from the octree rows, x0 = w b0 / d
template <int K>
__global__ void __launch_bounds__(kNT) k_restrict0(EmgDev g, Omegas om, const float4* __restrict__ r) {
    constexpr int H = K / 2;
    const EmgLevel& L = g.lv[0];
    each_edge<H>(L, [&](auto tag, int i, int j, int k, int h) {
        constexpr int D = decltype(tag)::value;
        const int c = eid<D>(L.n, i, j, k);
        float4 s = vz<float4>(), x = vz<float4>();
        if (edge_free<D>(L, i, j, k)) {
            const int q0 = __ldg(&g.r_ptr[c]), q1 = __ldg(&g.r_ptr[c + 1]);
            if (q1 - q0 > kLongRow) return;   // k_restrict0_long
            for (int q = q0; q < q1; q += 4) {
                float w[4];
                float4 v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const bool ok = q + u < q1;
                    w[u] = ok ? __ldg(&g.r_w[q + u]) : 0.0f;
                    v[u] = ok ? r[(size_t)__ldg(&g.r_row[q + u]) * H + h] : vz<float4>();
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) s = s + w[u] * v[u];
            }
            x = idiag(om_of(om, h, (float4*)nullptr), kEmgEdge, edge_diag<D>(L, i, j, k), __ldg(&L.me[c]), s);
        }
        f4(L.b)[(size_t)c * H + h] = s;
        f4(L.x)[(size_t)c * H + h] = x;
    });
}

// Sum of w_q v[idx_q] over one long transfer row by a block of kLongNT threads
// (lanes H, the entries dealt out to the rest); the total on the first H.
template <int H>
__device__ __forceinline__ float4 long_row(const int* __restrict__ idx, const float* __restrict__ w, int q0, int q1,
                                           const float4* __restrict__ v) {
    constexpr int G = kLongNT / H;
    __shared__ float4 part[kLongNT];
    const int h = threadIdx.x % H, g = threadIdx.x / H;
    float4 s = vz<float4>();
    for (int q = q0 + g; q < q1; q += G) s = s + __ldg(&w[q]) * v[(size_t)__ldg(&idx[q]) * H + h];
    part[threadIdx.x] = s;
    __syncthreads();
    for (int o = G / 2; o > 0; o >>= 1) {
        if (g < o) part[threadIdx.x] = part[threadIdx.x] + part[threadIdx.x + o * H];
        __syncthreads();
    }
    return part[threadIdx.x];
}

// The rows of P^T with more than kLongRow entries: coarse edges inside a
// refinement of two or three levels collect up to 196 or 1800 octree edges,
// which one thread after another made 50 us on the 157 k-edge mesh.
template <int K>
__global__ void __launch_bounds__(kLongNT) k_restrict0_long(EmgDev g, Omegas om, const float4* __restrict__ r) {
    constexpr int H = K / 2;
    const EmgLevel& L = g.lv[0];
    const int c = g.r_long[blockIdx.x], n = L.n, h = threadIdx.x % H;
    const float4 s = long_row<H>(g.r_row, g.r_w, g.r_ptr[c], g.r_ptr[c + 1], r);
    if (threadIdx.x >= H) return;
    const int per = n * (n + 1) * (n + 1), D = c / per, q = c % per;
    const int nx = D == 0 ? n : n + 1, ny = D == 1 ? n : n + 1, i = q % nx, j = q / nx % ny, k = q / (nx * ny);
    const float S = D == 0 ? edge_diag<0>(L, i, j, k) : D == 1 ? edge_diag<1>(L, i, j, k) : edge_diag<2>(L, i, j, k);
    f4(L.b)[(size_t)c * H + h] = s;
    f4(L.x)[(size_t)c * H + h] = idiag(om_of(om, h, (float4*)nullptr), kEmgEdge, S, __ldg(&L.me[c]), s);
}

// y = b - A x
template <int K>
__global__ void __launch_bounds__(kNT) k_resid(EmgLevel L, Omegas om) {
    constexpr int H = K / 2;
    each_edge<H>(L, [&](auto tag, int i, int j, int k, int h) {
        constexpr int D = decltype(tag)::value;
        const int c = eid<D>(L.n, i, j, k);
        float4 res = vz<float4>();
        if (edge_free<D>(L, i, j, k)) {
            const float4* x = f4(L.x);
            const float4 xc = x[(size_t)c * H + h];
            float S;
            const float4 ax = curl_row<D, float4>(L, i, j, k, xc, [&](int e) { return x[(size_t)e * H + h]; }, S);
            res = f4(L.b)[(size_t)c * H + h] - ax - imass(om_of(om, h, (float4*)nullptr), __ldg(&L.me[c]), xc);
        }
        f4(L.y)[(size_t)c * H + h] = res;
    });
}

// b = P^T y_fine, x = w b / d
template <int K>
__global__ void __launch_bounds__(kNT) k_restrict(EmgLevel F, EmgLevel L, Omegas om) {
    constexpr int H = K / 2;
    each_edge<H>(L, [&](auto tag, int i, int j, int k, int h) {
        constexpr int D = decltype(tag)::value;
        const int c = eid<D>(L.n, i, j, k);
        float4 s = vz<float4>(), x = vz<float4>();
        if (edge_free<D>(L, i, j, k)) {
            const float4* y = f4(F.y);
            s = gather_edge<D, float4>(F.n, i, j, k, [&](int e) { return y[(size_t)e * H + h]; });
            x = idiag(om_of(om, h, (float4*)nullptr), kEmgEdge, edge_diag<D>(L, i, j, k), __ldg(&L.me[c]), s);
        }
        f4(L.b)[(size_t)c * H + h] = s;
        f4(L.x)[(size_t)c * H + h] = x;
    });
}

// value of the coarse vector interpolated to fine edge (D; i, j, k)
template <int D, class V, class At>
__device__ __forceinline__ V interp_edge(int n, int i, int j, int k, const At& at) {
    const int I = i >> 1, J = j >> 1, Kk = k >> 1;
    constexpr int A = D == 0 ? 1 : 0, B = D == 2 ? 1 : 2;
    const int p[3] = {i, j, k};
    const bool oa = p[A] & 1, ob = p[B] & 1;
    auto e = [&](int sa, int sb) {
        return eid<D>(n, I + (A == 0 ? sa : 0), J + (A == 1 ? sa : 0) + (B == 1 ? sb : 0), Kk + (B == 2 ? sb : 0));
    };
    V s = at(e(0, 0));
    if (oa) s = s + at(e(1, 0));
    if (ob) s = s + at(e(0, 1));
    if (oa && ob) s = s + at(e(1, 1));
    return ((oa ? 0.5f : 1.0f) * (ob ? 0.5f : 1.0f)) * s;
}

// x += P y_coarse
template <int K>
__global__ void __launch_bounds__(kNT) k_prolong(EmgLevel L, EmgLevel C) {
    constexpr int H = K / 2;
    each_edge<H>(L, [&](auto tag, int i, int j, int k, int h) {
        constexpr int D = decltype(tag)::value;
        if (!edge_free<D>(L, i, j, k)) return;
        const size_t c = (size_t)eid<D>(L.n, i, j, k) * H + h;
        const float4* y = f4(C.y);
        f4(L.x)[c] = f4(L.x)[c] + interp_edge<D, float4>(C.n, i, j, k, [&](int e) { return y[(size_t)e * H + h]; });
    });
}

// y = x + w (b - A x) / d
template <int K>
__global__ void __launch_bounds__(kNT) k_smooth(EmgLevel L, Omegas om) {
    constexpr int H = K / 2;
    each_edge<H>(L, [&](auto tag, int i, int j, int k, int h) {
        constexpr int D = decltype(tag)::value;
        const int c = eid<D>(L.n, i, j, k);
        float4 v = vz<float4>();
        if (edge_free<D>(L, i, j, k)) {
            const float4* x = f4(L.x);
            const float4 xc = x[(size_t)c * H + h];
            const Om<float4> o = om_of(om, h, (float4*)nullptr);
            const float m = __ldg(&L.me[c]);
            float S;
            const float4 ax = curl_row<D, float4>(L, i, j, k, xc, [&](int e) { return x[(size_t)e * H + h]; }, S);
            v = xc + idiag(o, kEmgEdge, S, m, f4(L.b)[(size_t)c * H + h] - ax - imass(o, m, xc));
        }
        f4(L.y)[(size_t)c * H + h] = v;
    });
}

// The grids of at most kEmgBottom cells per side: one block per right-hand
// side runs their whole cycle, vectors in shared memory (a launch per step
// would cost more than the steps: 2 k edges).  Reads b and x of the first such
// level, writes its y.  The coarsest grid's Jacobi steps keep each edge's
// stencil in registers: twelve weights and positions, one edge per thread.
constexpr int kBottomNT = 1024;
constexpr int kCoarsestSteps = 12;

template <class F> __device__ __forceinline__ void with_edge(const EmgLevel& L, int t, const F& f) {
    const int n = L.n, per = n * (n + 1) * (n + 1);
    if (t < per) {
        const int i = t % n, j = t / n % (n + 1), k = t / (n * (n + 1));
        if (edge_free<0>(L, i, j, k)) f(Dir<0>{}, i, j, k);
    } else if (t < 2 * per) {
        const int q = t - per, i = q % (n + 1), j = q / (n + 1) % n, k = q / (n * (n + 1));
        if (edge_free<1>(L, i, j, k)) f(Dir<1>{}, i, j, k);
    } else if (t < 3 * per) {
        const int q = t - 2 * per, i = q % (n + 1), j = q / (n + 1) % (n + 1), k = q / ((n + 1) * (n + 1));
        if (edge_free<2>(L, i, j, k)) f(Dir<2>{}, i, j, k);
    }
}

// positions and weights of the twelve neighbours of an edge, as curl_row sums them
template <int D>
__device__ __forceinline__ void curl_stencil(const EmgLevel& L, int i, int j, int k, int (&at)[12], float (&w)[12],
                                             float& S) {
    const int n = L.n;
    S = 0.0f;
    auto dir = [&](auto tag, int o) {
        constexpr int A = decltype(tag)::value, B = 3 - D - A;
        constexpr int ai = A == 0, aj = A == 1, ak = A == 2, di = D == 0, dj = D == 1, dk = D == 2;
        const float hd = L.h[D], ha = L.h[A];
        const float wp = __ldg(&L.w[fid<B>(n, i, j, k)]), wm = __ldg(&L.w[fid<B>(n, i - ai, j - aj, k - ak)]);
        at[o] = eid<D>(n, i + ai, j + aj, k + ak);
        at[o + 1] = eid<D>(n, i - ai, j - aj, k - ak);
        at[o + 2] = eid<A>(n, i + di, j + dj, k + dk);
        at[o + 3] = eid<A>(n, i, j, k);
        at[o + 4] = eid<A>(n, i - ai + di, j - aj + dj, k - ak + dk);
        at[o + 5] = eid<A>(n, i - ai, j - aj, k - ak);
        w[o] = -hd * hd * wp;
        w[o + 1] = -hd * hd * wm;
        w[o + 2] = hd * ha * wp;
        w[o + 3] = -hd * ha * wp;
        w[o + 4] = -hd * ha * wm;
        w[o + 5] = hd * ha * wm;
        S += hd * hd * (wp + wm);
    };
    dir(Dir<D == 0 ? 1 : 0>{}, 0);
    dir(Dir<D == 2 ? 1 : 2>{}, 6);
}

__global__ void __launch_bounds__(kBottomNT) k_bottom(EmgDev g, int l0, int K, Omegas oms) {
    extern __shared__ float2 sm[];
    const int lane = blockIdx.x, tid = threadIdx.x;
    const Om<float2> om{oms.v[lane]};
    const int nl = g.n_levels;
    const bool two = l0 + 1 < nl;
    const EmgLevel& L = g.lv[l0];
    const EmgLevel& C = g.lv[nl - 1];
    const int nL = 3 * L.n * (L.n + 1) * (L.n + 1), nC = 3 * C.n * (C.n + 1) * (C.n + 1);
    // b, x and a third vector per level (the levels' own b, x: zero on edges that are not free)
    float2 *b = sm, *x = sm + nL, *y = sm + 2 * nL;
    float2 *cb = two ? sm + 3 * nL : b, *cx = two ? cb + nC : x, *cy = two ? cx + nC : y;
    for (int e = tid; e < nL; e += kBottomNT) {
        b[e] = L.b[(size_t)e * K + lane];
        x[e] = L.x[(size_t)e * K + lane];
        y[e] = make_float2(0.f, 0.f);
    }
    if (two)
        for (int e = tid; e < nC; e += kBottomNT) cx[e] = cy[e] = make_float2(0.f, 0.f);
    // the coarsest grid's stencil (at most 300 edges, one per thread)
    int at[12];
    float w[12], S = 0.0f, m = 0.0f;
    bool mine = false;
    with_edge(C, tid, [&](auto tag, int i, int j, int k) {
        curl_stencil<decltype(tag)::value>(C, i, j, k, at, w, S);
        m = __ldg(&C.me[tid]);
        mine = true;
    });
    __syncthreads();
    auto step = [&](const float2* in, float2* out, bool resid) {
        for (int e = tid; e < nL; e += kBottomNT)
            with_edge(L, e, [&](auto tag, int i, int j, int k) {
                const float me = __ldg(&L.me[e]);
                float d;
                const float2 ax = curl_row<decltype(tag)::value, float2>(L, i, j, k, in[e],
                                                                         [&](int q) { return in[q]; }, d);
                const float2 r = b[e] - ax - imass(om, me, in[e]);
                out[e] = resid ? r : in[e] + idiag(om, kEmgEdge, d, me, r);
            });
        __syncthreads();
    };
    if (two) {
        step(x, y, true);
        if (mine)
            with_edge(C, tid, [&](auto tag, int i, int j, int k) {
                const float2 s = gather_edge<decltype(tag)::value, float2>(L.n, i, j, k, [&](int q) { return y[q]; });
                cb[tid] = s;
                cx[tid] = idiag(om, kEmgEdge, S, m, s);
            });
        __syncthreads();
    }
    const float2 bb = mine ? cb[tid] : make_float2(0.f, 0.f);
    for (int q = 0; q < kCoarsestSteps; ++q) {
        const float2* in = q & 1 ? cy : cx;
        if (mine) {
            const float2 xc = in[tid];
            float2 ax = S * xc;
#pragma unroll
            for (int u = 0; u < 12; ++u) ax = ax + w[u] * in[at[u]];
            (q & 1 ? cx : cy)[tid] = xc + idiag(om, kEmgEdge, S, m, bb - ax - imass(om, m, xc));
        }
        __syncthreads();
    }
    const float2* out = cx;
    if (two) {
        for (int e = tid; e < nL; e += kBottomNT)
            with_edge(L, e, [&](auto tag, int i, int j, int k) {
                x[e] = x[e] + interp_edge<decltype(tag)::value, float2>(C.n, i, j, k, [&](int q) { return cx[q]; });
            });
        __syncthreads();
        // y holds the residual on free edges only, which the step overwrites
        step(x, y, false);
        out = y;
    }
    // every edge: the finer level's interpolation reads the zeros too
    for (int e = tid; e < nL; e += kBottomNT) L.y[(size_t)e * K + lane] = out[e];
}

// ---------------------------------------------------------------------------
// node cycle: V(0,1) in the edge preconditioner, the symmetric V(1,1) (PRE) in
// the divergence correction's PCG
// ---------------------------------------------------------------------------

// Laplacian row on a uniform grid: six edges, coarse edge masses over h^2
template <class V, class At>
__device__ __forceinline__ V lap_row(const EmgLevel& L, int i, int j, int k, V xc, const At& at, float& d) {
    const int n = L.n;
    V s = vz<V>();
    d = 0.0f;
    auto put = [&](int e, int v, float ih2) {
        const float m = __ldg(&L.me[e]) * ih2;
        s = s + m * (xc - at(v));
        d += m;
    };
    const float a = 1.0f / (L.h[0] * L.h[0]), b = 1.0f / (L.h[1] * L.h[1]), c = 1.0f / (L.h[2] * L.h[2]);
    put(eid<0>(n, i - 1, j, k), nid(n, i - 1, j, k), a);
    put(eid<0>(n, i, j, k), nid(n, i + 1, j, k), a);
    put(eid<1>(n, i, j - 1, k), nid(n, i, j - 1, k), b);
    put(eid<1>(n, i, j, k), nid(n, i, j + 1, k), b);
    put(eid<2>(n, i, j, k - 1), nid(n, i, j, k - 1), c);
    put(eid<2>(n, i, j, k), nid(n, i, j, k + 1), c);
    return s;
}

// diagonal of the node Laplacian on a uniform grid
__device__ __forceinline__ float lap_diag(const EmgLevel& L, int i, int j, int k) {
    const int n = L.n;
    return (__ldg(&L.me[eid<0>(n, i - 1, j, k)]) + __ldg(&L.me[eid<0>(n, i, j, k)])) / (L.h[0] * L.h[0]) +
           (__ldg(&L.me[eid<1>(n, i, j - 1, k)]) + __ldg(&L.me[eid<1>(n, i, j, k)])) / (L.h[1] * L.h[1]) +
           (__ldg(&L.me[eid<2>(n, i, j, k - 1)]) + __ldg(&L.me[eid<2>(n, i, j, k)])) / (L.h[2] * L.h[2]);
}

// w b / diag, the pre-smoothed iterate of the V(1,1) cycle
template <class V> __device__ __forceinline__ V node_pre(const EmgLevel& L, int i, int j, int k, V b) {
    const float d = node_free(L, i, j, k) ? lap_diag(L, i, j, k) : 0.0f;
    return d > 0.0f ? (kEmgNode / d) * b : vz<V>();
}

// nb0 = Pn^T b from the octree nodes; PRE: nt0 = w nb0 / diag
template <int K, bool PRE>
__global__ void __launch_bounds__(kNT) k_node_restrict0(EmgDev g, const float4* __restrict__ b) {
    constexpr int H = K / 2;
    const EmgLevel& L = g.lv[0];
    each_node<H>(L, [&](int i, int j, int k, int h) {
        const int c = nid(L.n, i, j, k);
        float4 s = vz<float4>();
        const int q0 = __ldg(&g.nr_ptr[c]), q1 = __ldg(&g.nr_ptr[c + 1]);
        if (q1 - q0 > kLongRow) return;   // k_node_restrict0_long
        for (int q = q0; q < q1; q += 4) {
            float w[4];
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool ok = q + u < q1;
                w[u] = ok ? __ldg(&g.nr_w[q + u]) : 0.0f;
                v[u] = ok ? b[(size_t)__ldg(&g.nr_node[q + u]) * H + h] : vz<float4>();
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) s = s + w[u] * v[u];
        }
        f4(L.nb)[(size_t)c * H + h] = s;
        if (PRE) f4(L.nt)[(size_t)c * H + h] = node_pre(L, i, j, k, s);
    });
}

template <int K, bool PRE>
__global__ void __launch_bounds__(kLongNT) k_node_restrict0_long(EmgDev g, const float4* __restrict__ b) {
    constexpr int H = K / 2;
    const EmgLevel& L = g.lv[0];
    const int c = g.nr_long[blockIdx.x], n1 = L.n + 1, h = threadIdx.x % H;
    const float4 s = long_row<H>(g.nr_node, g.nr_w, g.nr_ptr[c], g.nr_ptr[c + 1], b);
    if (threadIdx.x >= H) return;
    f4(L.nb)[(size_t)c * H + h] = s;
    if (PRE) f4(L.nt)[(size_t)c * H + h] = node_pre(L, c % n1, c / n1 % n1, c / (n1 * n1), s);
}

// ny = nb - L nt
template <int K>
__global__ void __launch_bounds__(kNT) k_node_resid(EmgLevel L) {
    constexpr int H = K / 2;
    each_node<H>(L, [&](int i, int j, int k, int h) {
        const size_t c = (size_t)nid(L.n, i, j, k) * H + h;
        float4 v = vz<float4>();
        if (node_free(L, i, j, k)) {
            const float4* t = f4(L.nt);
            float d;
            v = f4(L.nb)[c] - lap_row<float4>(L, i, j, k, t[c], [&](int q) { return t[(size_t)q * H + h]; }, d);
        }
        f4(L.ny)[c] = v;
    });
}


template <class V, class At>
__device__ __forceinline__ V gather_node(int n, int I, int J, int Kk, const At& at) {
    V s = vz<V>();
#pragma unroll
    for (int c = -1; c <= 1; ++c)
#pragma unroll
        for (int b = -1; b <= 1; ++b)
#pragma unroll
            for (int a = -1; a <= 1; ++a)
                s = s + ((a ? 0.5f : 1.0f) * (b ? 0.5f : 1.0f) * (c ? 0.5f : 1.0f)) *
                            at(nid(n, 2 * I + a, 2 * J + b, 2 * Kk + c));
    return s;
}
template <class V, class At>
__device__ __forceinline__ V interp_node(int n, int i, int j, int k, const At& at) {
    const int oi = i & 1, oj = j & 1, ok = k & 1;
    V s = vz<V>();
    for (int c = 0; c <= ok; ++c)
        for (int b = 0; b <= oj; ++b)
            for (int a = 0; a <= oi; ++a) s = s + at(nid(n, (i >> 1) + a, (j >> 1) + b, (k >> 1) + c));
    return ((oi ? 0.5f : 1.0f) * (oj ? 0.5f : 1.0f) * (ok ? 0.5f : 1.0f)) * s;
}

// nb = Pn^T of the finer level's right-hand side, or (PRE) of its residual in
// ny, with nt = w nb / diag
template <int K, bool PRE>
__global__ void __launch_bounds__(kNT) k_node_restrict(EmgLevel F, EmgLevel L) {
    constexpr int H = K / 2;
    each_node<H>(L, [&](int i, int j, int k, int h) {
        float4 s = vz<float4>();
        const float4* b = f4(PRE ? F.ny : F.nb);
        if (node_free(L, i, j, k))
            s = gather_node<float4>(F.n, i, j, k, [&](int v) { return b[(size_t)v * H + h]; });
        const size_t c = (size_t)nid(L.n, i, j, k) * H + h;
        f4(L.nb)[c] = s;
        if (PRE) f4(L.nt)[c] = node_pre(L, i, j, k, s);
    });
}

// nt = Pn y_coarse, or (PRE) nt += Pn y_coarse
template <int K, bool PRE>
__global__ void __launch_bounds__(kNT) k_node_prolong(EmgLevel L, EmgLevel C) {
    constexpr int H = K / 2;
    each_node<H>(L, [&](int i, int j, int k, int h) {
        float4 s = vz<float4>();
        const float4* y = f4(C.ny);
        if (node_free(L, i, j, k))
            s = interp_node<float4>(C.n, i, j, k, [&](int v) { return y[(size_t)v * H + h]; });
        const size_t c = (size_t)nid(L.n, i, j, k) * H + h;
        f4(L.nt)[c] = PRE ? f4(L.nt)[c] + s : s;
    });
}

// ny = t + w (nb - L t) / diag
template <int K>
__global__ void __launch_bounds__(kNT) k_node_smooth(EmgLevel L) {
    constexpr int H = K / 2;
    each_node<H>(L, [&](int i, int j, int k, int h) {
        const size_t c = (size_t)nid(L.n, i, j, k) * H + h;
        float4 v = vz<float4>();
        if (node_free(L, i, j, k)) {
            const float4* t = f4(L.nt);
            const float4 tc = t[c];
            float d;
            const float4 lt = lap_row<float4>(L, i, j, k, tc, [&](int q) { return t[(size_t)q * H + h]; }, d);
            v = d > 0.0f ? tc + (kEmgNode / d) * (f4(L.nb)[c] - lt) : tc;
        }
        f4(L.ny)[c] = v;
    });
}

template <bool PRE>
__global__ void __launch_bounds__(kBottomNT) k_node_bottom(EmgDev g, int l0, int K) {
    constexpr int kN = (kEmgBottom + 1) * (kEmgBottom + 1) * (kEmgBottom + 1);
    constexpr int kNc = 5 * 5 * 5;
    static_assert(kN <= kBottomNT, "one node per thread");
    __shared__ float2 b[kN], x[kN], y[kN], cb[kNc], cx[kNc], cy[kNc];
    const int lane = blockIdx.x, tid = threadIdx.x, nl = g.n_levels;
    const bool two = l0 + 1 < nl;
    const EmgLevel& L = g.lv[l0];
    const EmgLevel& C = g.lv[nl - 1];
    const int nL = (L.n + 1) * (L.n + 1) * (L.n + 1);
    const int i = tid % (L.n + 1), j = tid / (L.n + 1) % (L.n + 1), k = tid / ((L.n + 1) * (L.n + 1));
    const int ci = tid % 5, cj = tid / 5 % 5, ck = tid / 25;   // two: the coarsest grid has 4 cells per side
    const bool in = tid < nL && node_free(L, i, j, k);
    const bool cin = two && tid < kNc && node_free(C, ci, cj, ck);
    if (tid < nL) {
        b[tid] = in ? L.nb[(size_t)tid * K + lane] : make_float2(0.f, 0.f);
        x[tid] = y[tid] = make_float2(0.f, 0.f);
    }
    if (tid < kNc) cb[tid] = cx[tid] = cy[tid] = make_float2(0.f, 0.f);
    __syncthreads();
    auto jacobi = [&](const EmgLevel& M, bool on, int a, int c, int d, const float2* rhs, const float2* v, float2* out) {
        if (on) {
            float dg;
            const float2 lv = lap_row<float2>(M, a, c, d, v[tid], [&](int q) { return v[q]; }, dg);
            out[tid] = dg > 0.0f ? v[tid] + (kEmgNode / dg) * (rhs[tid] - lv) : v[tid];
        }
        __syncthreads();
    };
    const float2* rc = b;   // what the coarsest grid gets
    if (two && PRE) {
        if (in) x[tid] = node_pre(L, i, j, k, b[tid]);
        __syncthreads();
        if (in) {
            float dg;
            y[tid] = b[tid] - lap_row<float2>(L, i, j, k, x[tid], [&](int q) { return x[q]; }, dg);
        }
        __syncthreads();
        rc = y;
    }
    if (two) {
        if (cin) cb[tid] = gather_node<float2>(L.n, ci, cj, ck, [&](int q) { return rc[q]; });
        __syncthreads();
        for (int q = 0; q < kCoarsestSteps; q += 2) {   // from zero
            jacobi(C, cin, ci, cj, ck, cb, cx, cy);
            jacobi(C, cin, ci, cj, ck, cb, cy, cx);
        }
        if (in) x[tid] = x[tid] + interp_node<float2>(C.n, i, j, k, [&](int q) { return cx[q]; });
        __syncthreads();
        jacobi(L, in, i, j, k, b, x, y);
    } else {
        for (int q = 0; q < kCoarsestSteps; q += 2) {
            jacobi(L, in, i, j, k, b, x, y);
            jacobi(L, in, i, j, k, b, y, x);
        }
    }
    if (tid < nL) L.ny[(size_t)tid * K + lane] = two ? y[tid] : x[tid];
}

// t = Pn ny0 on the octree nodes (0 on Dirichlet nodes), plus x if given
template <int K>
__global__ void __launch_bounds__(kNT) k_node_prolong0(EmgDev g, int nn, const float4* __restrict__ x,
                                                       float4* __restrict__ out) {
    constexpr int H = K / 2;
    const long i = (long)blockIdx.x * kNT + threadIdx.x;
    if (i >= (long)nn * H) return;
    const int v = (int)(i / H), h = (int)(i % H);
    const int base = __ldg(&g.n_base[v]);
    float4 s = x ? x[i] : vz<float4>();
    if (base >= 0) {
        const unsigned code = __ldg(&g.n_code[v]);
        const float u = 1.0f / (float)(1 << g.gap);
        const float fx = (float)(code & 15u) * u, fy = (float)(code >> 4 & 15u) * u, fz = (float)(code >> 8 & 15u) * u;
        const int n1 = g.lv[0].n + 1;
        const float4* y = f4(g.lv[0].ny);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float w = (q & 1 ? fx : 1.0f - fx) * (q & 2 ? fy : 1.0f - fy) * (q & 4 ? fz : 1.0f - fz);
            if (w > 0.0f)
                s = s + w * y[(size_t)(base + (q & 1) + (q >> 1 & 1) * n1 + (q >> 2) * n1 * n1) * H + h];
        }
    }
    out[i] = s;
}

// z0 = P y0 + G~ yn / (i omega) + w r / d on free rows, r on identity rows
template <int K>
__global__ void __launch_bounds__(kNT) k_combine(EmgDev g, GcRowTerm gt, DiagView<float> D, Omegas om, long n,
                                                 const float4* __restrict__ r, float4* __restrict__ z0) {
    constexpr int H = K / 2;
    const long i = (long)blockIdx.x * kNT + threadIdx.x;
    if (i >= n) return;
    const int row = (int)(i / H), h = (int)(i % H);
    const float4 rv = r[i];
    const int base = __ldg(&g.p_base[row]);
    float4 z = rv;
    if (base >= 0) {
        const unsigned code = __ldg(&g.p_code[row]);
        const float u = 1.0f / (float)(1 << g.gap);
        const float fa = (float)(code >> 2 & 15u) * u, fb = (float)(code >> 6 & 15u) * u;
        const int d = code & 3u, m = g.lv[0].n, nx = d == 0 ? m : m + 1, ny = d == 1 ? m : m + 1;
        const int sa = d == 0 ? nx : 1, sb = d == 2 ? nx : nx * ny;
        const float4* y = f4(g.lv[0].y);
        const int2 nd = __ldg(reinterpret_cast<const int2*>(gt.e_node) + row);
        const float2 ge = __ldg(reinterpret_cast<const float2*>(gt.e_g) + row);
        const float4* yn = f4(gt.ya);
        float4 c = ge.x * yn[(size_t)nd.x * H + h] + ge.y * yn[(size_t)nd.y * H + h];
        const float2 dg = D.sm[row];
        z = idiag(om_of(om, h, (float4*)nullptr), kEmgFine, dg.x, dg.y, rv);
        const float wa[2] = {1.0f - fa, fa}, wb[2] = {1.0f - fb, fb};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float w = wa[q & 1] * wb[q >> 1];
            if (w > 0.0f) z = z + w * y[(size_t)(base + (q & 1) * sa + (q >> 1) * sb) * H + h];
        }
        const float s0 = gt.s[2 * h], s1 = gt.s[2 * h + 1];
        z = z + make_float4(s0 * c.y, -s0 * c.x, s1 * c.w, -s1 * c.z);
    }
    z0[i] = z;
}

int grid1(long work) { return (int)std::max(1L, (work + kNT - 1) / kNT); }

int bottom_level(const EmgDev& g) {
    int l = 0;
    while (l + 1 < g.n_levels && g.lv[l].n > kEmgBottom) ++l;
    return l;
}

// shared memory of the bottom edge kernel: three vectors of each of its levels
int bottom_smem(const EmgDev& g, int l0) {
    size_t b = 0;
    for (int l = l0; l < g.n_levels; ++l) b += 3 * sizeof(float2) * (size_t)emg_edges(g.lv[l].n);
    return (int)b;
}

template <int K>
void edge_cycle(const EmgDev& g, const Omegas& om, const float2* r, cudaStream_t s, long long* launches) {
    const int l0 = bottom_level(g);
    k_restrict0<K><<<edge_grid<K>(g.lv[0]), kNT, 0, s>>>(g, om, f4(r));
    ck(launches);
    if (g.n_r_long) {
        k_restrict0_long<K><<<g.n_r_long, kLongNT, 0, s>>>(g, om, f4(r));
        ck(launches);
    }
    for (int l = 0; l < l0; ++l) {
        k_resid<K><<<edge_grid<K>(g.lv[l]), kNT, 0, s>>>(g.lv[l], om);
        ck(launches);
        k_restrict<K><<<edge_grid<K>(g.lv[l + 1]), kNT, 0, s>>>(g.lv[l], g.lv[l + 1], om);
        ck(launches);
    }
    const int smem = bottom_smem(g, l0);
    cudaFuncSetAttribute(reinterpret_cast<const void*>(k_bottom), cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    k_bottom<<<K, kBottomNT, smem, s>>>(g, l0, K, om);
    ck(launches);
    for (int l = l0 - 1; l >= 0; --l) {
        k_prolong<K><<<edge_grid<K>(g.lv[l]), kNT, 0, s>>>(g.lv[l], g.lv[l + 1]);
        ck(launches);
        k_smooth<K><<<edge_grid<K>(g.lv[l]), kNT, 0, s>>>(g.lv[l], om);
        ck(launches);
    }
}

// the uniform grids' part of a node cycle, from octree node vector b to ny of level 0
template <int K, bool PRE>
void node_grids(const EmgDev& g, const float2* b, cudaStream_t s, long long* launches) {
    const int l0 = bottom_level(g);
    k_node_restrict0<K, PRE><<<node_grid<K>(g.lv[0]), kNT, 0, s>>>(g, f4(b));
    ck(launches);
    if (g.n_nr_long) {
        k_node_restrict0_long<K, PRE><<<g.n_nr_long, kLongNT, 0, s>>>(g, f4(b));
        ck(launches);
    }
    for (int l = 0; l < l0; ++l) {
        if (PRE) {
            k_node_resid<K><<<node_grid<K>(g.lv[l]), kNT, 0, s>>>(g.lv[l]);
            ck(launches);
        }
        k_node_restrict<K, PRE><<<node_grid<K>(g.lv[l + 1]), kNT, 0, s>>>(g.lv[l], g.lv[l + 1]);
        ck(launches);
    }
    k_node_bottom<PRE><<<K, kBottomNT, 0, s>>>(g, l0, K);
    ck(launches);
    for (int l = l0 - 1; l >= 0; --l) {
        k_node_prolong<K, PRE><<<node_grid<K>(g.lv[l]), kNT, 0, s>>>(g.lv[l], g.lv[l + 1]);
        ck(launches);
        k_node_smooth<K><<<node_grid<K>(g.lv[l]), kNT, 0, s>>>(g.lv[l]);
        ck(launches);
    }
}

template <int K>
void node_cycle(const EmgDev& g, const GcDev& gc, const float2* r, cudaStream_t s, long long* launches) {
    gc_restrict_edges_k<K>(gc, r, s, launches);
    node_grids<K, false>(g, gc.lv[0].b, s, launches);
    k_node_prolong0<K><<<grid1((long)gc.nn * (K / 2)), kNT, 0, s>>>(g, gc.nn, nullptr, f4(gc.lv[0].y));
    ck(launches);
    gc_smooth0_k<K>(gc, gc.lv[0].y, gc.out0, s, launches);
}

}  // namespace

std::vector<int> emg_long_rows(const std::vector<int>& ptr) {
    std::vector<int> rows;
    for (size_t c = 0; c + 1 < ptr.size(); ++c)
        if (ptr[c + 1] - ptr[c] > kLongRow) rows.push_back((int)c);
    return rows;
}

void emg_set_mass(const EmgDev& g, const double* Me, cudaStream_t s, long long* launches) {
    const int n = (int)emg_edges(g.lv[0].n);
    k_mass0<<<(n + 255) / 256, 256, 0, s>>>(g, Me, n);
    ck(launches);
    for (int l = 1; l < g.n_levels; ++l) {
        k_mass<<<(int)((emg_edges(g.lv[l].n) + 255) / 256), 256, 0, s>>>(g.lv[l - 1], g.lv[l]);
        ck(launches);
    }
}

template <int K>
void emg_coarse_k(const KrylovCtx<float>& c, const float2* r, float2* z0) {
    const EmgDev& g = *c.emg;
    const GcDev& gc = *c.gc;
    Omegas om;
    for (int k = 0; k < kMaxRhs; ++k) om.v[k] = k < K ? (float)c.B.omega[k] : 0.0f;
    const double nb = (double)c.n_rows * K * sizeof(float2), e0 = (double)emg_edges(g.lv[0].n) * K * sizeof(float2),
                 nn = (double)gc.nn * K * sizeof(float2);
    // r gathered by both restrictions and read by the last kernel, z0 written;
    // level-0 edge vectors b, x written and read, residual, x updated, y;
    // octree node vectors b, t, out
    const int th = c.timer ? c.timer->begin(kClsGradcorr, 4 * nb + 11 * e0 + 7 * nn, K) : -1;
    if (c.gc_stream) {
        cudaEventRecord(c.gc_fork, c.stream);
        cudaStreamWaitEvent(c.gc_stream, c.gc_fork, 0);
        node_cycle<K>(g, gc, r, c.gc_stream, c.launches);
        cudaEventRecord(c.gc_join, c.gc_stream);
    } else {
        node_cycle<K>(g, gc, r, c.stream, c.launches);
    }
    edge_cycle<K>(g, om, r, c.stream, c.launches);
    if (c.gc_stream) cudaStreamWaitEvent(c.stream, c.gc_join, 0);
    const long n = (long)c.n_rows_pad * (K / 2);
    k_combine<K><<<grid1(n), kNT, 0, c.stream>>>(g, gc_row_term(gc, c.B), c.D, om, n, f4(r), f4(z0));
    ck(c.launches);
    if (c.timer) c.timer->end(th);
}

template <int K>
void emg_node_precond_k(const EmgDev& g, const GcDev& gc, float2* z, cudaStream_t s, long long* launches) {
    gc_presmooth0_k<K>(gc, s, launches);   // x = omega D^-1 b, y = b - L x
    node_grids<K, true>(g, gc.lv[0].y, s, launches);
    k_node_prolong0<K><<<grid1((long)gc.nn * (K / 2)), kNT, 0, s>>>(g, gc.nn, f4(gc.lv[0].x), f4(gc.lv[0].y));
    ck(launches);
    gc_smooth0_k<K>(gc, gc.lv[0].y, z, s, launches);
}

template void emg_node_precond_k<2>(const EmgDev&, const GcDev&, float2*, cudaStream_t, long long*);
template void emg_node_precond_k<4>(const EmgDev&, const GcDev&, float2*, cudaStream_t, long long*);
template void emg_node_precond_k<8>(const EmgDev&, const GcDev&, float2*, cudaStream_t, long long*);
template void emg_node_precond_k<16>(const EmgDev&, const GcDev&, float2*, cudaStream_t, long long*);
template void emg_coarse_k<2>(const KrylovCtx<float>&, const float2*, float2*);
template void emg_coarse_k<4>(const KrylovCtx<float>&, const float2*, float2*);
template void emg_coarse_k<8>(const KrylovCtx<float>&, const float2*, float2*);
template void emg_coarse_k<16>(const KrylovCtx<float>&, const float2*, float2*);

}  // namespace m3d
