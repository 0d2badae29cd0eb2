// Kernels of the geometric multigrid preconditioner (see edgemg.cuh).
#include "edgemg.cuh"

#include <algorithm>
#include <stdexcept>

namespace m3d {

using namespace dev;

namespace {

constexpr int kNT = 256;
// transfer rows longer than these (one level of refinement gives them) are summed by a block
constexpr int kLongEdge = 18, kLongNode = 27;
constexpr int kLongNT = 128;

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
__device__ __forceinline__ int pid(int n, int i, int j, int k) { return (k * (n + 1) + j) * (n + 1) + i; }

// Which of the three edges starting at a point are free: inside the grid
// across their direction and not above the surface.
struct Free { bool e[3]; };
__device__ __forceinline__ Free edges_free(const EmgLevel& L, int i, int j, int k) {
    const int n = L.n;
    const bool in = i < n && j < n && k < n;
    return {{in && j > 0 && k > 0 && k < L.ph, in && i > 0 && k > 0 && k < L.ph, in && i > 0 && j > 0 && k < L.pv}};
}
__device__ __forceinline__ bool node_free(const EmgLevel& L, int i, int j, int k) {
    return i > 0 && i < L.n && j > 0 && j < L.n && k > 0 && k < L.pn;
}

// Weights of the nine faces that the three edges of a point touch, by normal:
// at the point and one step down in each of the two other directions (those
// clamp at the grid's side, where no free edge uses them).
struct Faces { float x, xj, xk, y, yi, yk, z, zi, zj; };
__device__ __forceinline__ Faces face_weights(const EmgLevel& L, int i, int j, int k) {
    const int n1 = L.n + 1, p = pid(L.n, i, j, k);
    const int pi = p - (i > 0), pj = p - (j > 0 ? n1 : 0), pk = p - (k > 0 ? n1 * n1 : 0);
    const float* w = L.w;
    return {__ldg(&w[3 * p]),     __ldg(&w[3 * pj]),     __ldg(&w[3 * pk]),
            __ldg(&w[3 * p + 1]), __ldg(&w[3 * pi + 1]), __ldg(&w[3 * pk + 1]),
            __ldg(&w[3 * p + 2]), __ldg(&w[3 * pi + 2]), __ldg(&w[3 * pj + 2])};
}
// diagonals of the curl-curl rows
__device__ __forceinline__ void edge_diags(const EmgLevel& L, const Faces& f, float (&S)[3]) {
    S[0] = L.h[0] * L.h[0] * (f.y + f.yk + f.z + f.zj);
    S[1] = L.h[1] * L.h[1] * (f.z + f.zi + f.x + f.xk);
    S[2] = L.h[2] * L.h[2] * (f.y + f.yi + f.x + f.xj);
}

// Curl-curl rows of the three edges of a point (i, j, k < n): nine face
// circulations from 24 edge values, where three 13-point rows would read 39;
// at(e) reads the vector at edge entry e.
template <class V, class At>
__device__ __forceinline__ void curl_rows(const EmgLevel& L, const Faces& f, int i, int j, int k, const At& at,
                                          V (&xc)[3], V (&ax)[3]) {
    const int n1 = L.n + 1, p = pid(L.n, i, j, k);
    const int di = 3, dj = 3 * n1, dk = 3 * n1 * n1, mi = i > 0 ? di : 0, mj = j > 0 ? dj : 0, mk = k > 0 ? dk : 0;
    const int x = 3 * p, y = 3 * p + 1, z = 3 * p + 2;
    const float hx = L.h[0], hy = L.h[1], hz = L.h[2];
    const V X = at(x), Y = at(y), Z = at(z);
    const V Xj = at(x + dj), Xk = at(x + dk), Yi = at(y + di), Yk = at(y + dk), Zi = at(z + di), Zj = at(z + dj);
    xc[0] = X;
    xc[1] = Y;
    xc[2] = Z;
    // circulations times weights: normal x, y, z at the point
    const V cx = f.x * (hy * (Y - Yk) + hz * (Zj - Z));
    const V cy = f.y * (hx * (X - Xk) + hz * (Zi - Z));
    const V cz = f.z * (hx * (X - Xj) + hy * (Yi - Y));
    // one step down
    const V Xmj = at(x - mj), Xmk = at(x - mk), Ymi = at(y - mi), Ymk = at(y - mk), Zmi = at(z - mi), Zmj = at(z - mj);
    const V cxk = f.xk * (hy * (Ymk - Y) + hz * (at(z - mk + dj) - at(z - mk)));
    const V cxj = f.xj * (hy * (at(y - mj) - at(y - mj + dk)) + hz * (Z - Zmj));
    const V cyk = f.yk * (hx * (Xmk - X) + hz * (at(z - mk + di) - at(z - mk)));
    const V cyi = f.yi * (hx * (at(x - mi) - at(x - mi + dk)) + hz * (Z - Zmi));
    const V czj = f.zj * (hx * (Xmj - X) + hy * (at(y - mj + di) - at(y - mj)));
    const V czi = f.zi * (hx * (at(x - mi) - at(x - mi + dj)) + hy * (Y - Ymi));
    ax[0] = hx * ((cy - cyk) + (cz - czj));
    ax[1] = hy * ((czi - cz) + (cx - cxk));
    ax[2] = hz * ((cyi - cy) + (cxj - cx));
}

// Work split of a grid kernel: threads over (point of a plane, pairs of
// right-hand sides), blockIdx.y the plane.  The planes are those that may hold
// free edges or nodes and the ones above them, which are written as zeros
// because the stencils read them.
__host__ __device__ inline int edge_planes(const EmgLevel& L) {
    const int p = (L.ph > L.pv ? L.ph : L.pv) + 1;
    return p < L.n + 1 ? p : L.n + 1;
}
__host__ __device__ inline int node_planes(const EmgLevel& L) { return L.pn + 2 < L.n + 1 ? L.pn + 2 : L.n + 1; }

template <int H, class F> __device__ __forceinline__ void each_point(const EmgLevel& L, const F& f) {
    const int t = blockIdx.x * kNT + threadIdx.x;
    const int q = t / H, h = t % H, n1 = L.n + 1;
    if (q < n1 * n1) f(q % n1, q / n1, (int)blockIdx.y, h);
}
template <int K> dim3 point_grid(const EmgLevel& L, int planes) {
    const long rows = (long)(L.n + 1) * (L.n + 1) * (K / 2);
    return dim3((unsigned)((rows + kNT - 1) / kNT), (unsigned)planes);
}

__host__ __device__ __forceinline__ float4* f4(float2* p) { return reinterpret_cast<float4*>(p); }
__host__ __device__ __forceinline__ const float4* f4(const float2* p) { return reinterpret_cast<const float4*>(p); }

// Two right-hand sides of an entry: [entry][K], or [K][entry] on a grid of the
// bottom kernels (n entries).
__host__ __device__ inline bool lane_major(const EmgLevel& L) { return L.n <= kEmgBottom; }
template <int K> __device__ __forceinline__ float4 load2(const float2* v, bool lm, int n, int e, int h) {
    if (!lm) return f4(v)[(size_t)e * (K / 2) + h];
    const float2 a = v[(size_t)(2 * h) * n + e], b = v[(size_t)(2 * h + 1) * n + e];
    return make_float4(a.x, a.y, b.x, b.y);
}
template <int K> __device__ __forceinline__ void store2(float2* v, bool lm, int n, int e, int h, float4 q) {
    if (!lm) {
        f4(v)[(size_t)e * (K / 2) + h] = q;
        return;
    }
    v[(size_t)(2 * h) * n + e] = make_float2(q.x, q.y);
    v[(size_t)(2 * h + 1) * n + e] = make_float2(q.z, q.w);
}
__device__ __forceinline__ int entries(const EmgLevel& L) { return 3 * (L.n + 1) * (L.n + 1) * (L.n + 1); }
__device__ __forceinline__ int points(const EmgLevel& L) { return (L.n + 1) * (L.n + 1) * (L.n + 1); }

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

// sum over the fine edges of the coarse edge of direction D at (I, J, Kk): 2
// along it, (1/2, 1, 1/2) across
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
            s = s + w * (at(3 * pid(n, i, j, k) + D) + at(3 * pid(n, i + (D == 0), j + (D == 1), k + (D == 2)) + D));
        }
    return s;
}
// the same for the free edges of a point
template <class V, class At>
__device__ __forceinline__ void gather_edges(const Free& f, int n, int I, int J, int Kk, const At& at, V (&s)[3]) {
    s[0] = f.e[0] ? gather_edge<0, V>(n, I, J, Kk, at) : vz<V>();
    s[1] = f.e[1] ? gather_edge<1, V>(n, I, J, Kk, at) : vz<V>();
    s[2] = f.e[2] ? gather_edge<2, V>(n, I, J, Kk, at) : vz<V>();
}

struct F1 { float v; };
__device__ __forceinline__ F1 vzero(F1*) { return {0.f}; }
__device__ __forceinline__ F1 operator+(F1 a, F1 b) { return {a.v + b.v}; }
__device__ __forceinline__ F1 operator-(F1 a, F1 b) { return {a.v - b.v}; }
__device__ __forceinline__ F1 operator*(float s, F1 b) { return {s * b.v}; }

__global__ void k_mass(EmgLevel F, EmgLevel C) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, n1 = C.n + 1;
    if (t >= n1 * n1 * n1) return;
    const int i = t % n1, j = t / n1 % n1, k = t / (n1 * n1);
    const Free f = edges_free(C, i, j, k);
    F1 s[3];
    gather_edges<F1>(f, F.n, i, j, k, [&](int e) { return F1{F.me[e]}; }, s);
    for (int D = 0; D < 3; ++D)
        if (f.e[D]) C.me[3 * t + D] = s[D].v;
}

// ---------------------------------------------------------------------------
// edge cycle
// ---------------------------------------------------------------------------

// Sum of w_q v[idx_q] over one long transfer row by a block of kLongNT threads
// (lanes H, the entries dealt out to the rest); the total on the first H.
template <int H>
__device__ __forceinline__ float4 long_row(const int* __restrict__ idx, const float* __restrict__ w, int q0, int q1,
                                           const float4* v) {
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

// b0 = P^T r from the octree rows, x0 = w b0 / d; a thread per edge entry
template <int K>
__global__ void __launch_bounds__(kNT) k_restrict0(EmgDev g, Omegas om, const float4* r, int n) {
    dep_begin();
    constexpr int H = K / 2;
    const EmgLevel& L = g.lv[0];
    const int t = blockIdx.x * kNT + threadIdx.x, c = t / H, h = t % H;
    if (c >= n) return;
    const int n1 = L.n + 1, p = c / 3, i = p % n1, j = p / n1 % n1, k = p / (n1 * n1), D = c % 3;
    const int q0 = __ldg(&g.r_ptr[c]), q1 = __ldg(&g.r_ptr[c + 1]);
    if (q1 - q0 > kLongEdge) return;   // k_restrict0_long
    float4 s = vz<float4>(), x = vz<float4>();
    for (int q = q0; q < q1; q += 6) {   // 18 entries under one level of refinement
        float w[6];
        float4 v[6];
#pragma unroll
        for (int u = 0; u < 6; ++u) {
            const bool ok = q + u < q1;
            w[u] = ok ? __ldg(&g.r_w[q + u]) : 0.0f;
            v[u] = ok ? r[(size_t)__ldg(&g.r_row[q + u]) * H + h] : vz<float4>();
        }
#pragma unroll
        for (int u = 0; u < 6; ++u) s = s + w[u] * v[u];
    }
    if (q1 > q0) {
        float S[3];
        edge_diags(L, face_weights(L, i, j, k), S);
        x = idiag(om_of(om, h, (float4*)nullptr), kEmgEdge, S[D], __ldg(&L.me[c]), s);
    }
    store2<K>(L.b, lane_major(L), entries(L), c, h, s);
    store2<K>(L.x, lane_major(L), entries(L), c, h, x);
}

// The rows of P^T with more than kLongEdge entries: coarse edges inside a
// refinement of two or three levels collect up to 196 or 1800 octree edges,
// which one thread after another made 50 us on the 157 k-edge mesh.
template <int K>
__global__ void __launch_bounds__(kLongNT) k_restrict0_long(EmgDev g, Omegas om, const float4* r) {
    dep_begin();
    constexpr int H = K / 2;
    const EmgLevel& L = g.lv[0];
    const int c = g.r_long[blockIdx.x], h = threadIdx.x % H;
    const float4 s = long_row<H>(g.r_row, g.r_w, g.r_ptr[c], g.r_ptr[c + 1], r);
    if (threadIdx.x >= H) return;
    const int n1 = L.n + 1, p = c / 3;
    float S[3];
    edge_diags(L, face_weights(L, p % n1, p / n1 % n1, p / (n1 * n1)), S);
    store2<K>(L.b, lane_major(L), entries(L), c, h, s);
    store2<K>(L.x, lane_major(L), entries(L), c, h,
              idiag(om_of(om, h, (float4*)nullptr), kEmgEdge, S[c % 3], __ldg(&L.me[c]), s));
}

// y = b - A x, or (SMOOTH) y = x + w (b - A x) / d
template <int K, bool SMOOTH>
__global__ void __launch_bounds__(kNT, 3) k_edge_step(EmgLevel L, Omegas oms) {
    dep_begin();
    constexpr int H = K / 2;
    each_point<H>(L, [&](int i, int j, int k, int h) {
        const Free f = edges_free(L, i, j, k);
        const int p = pid(L.n, i, j, k);
        const float4 *xv = f4(L.x), *b = f4(L.b);
        float4* y = f4(L.y);
        float4 out[3] = {vz<float4>(), vz<float4>(), vz<float4>()};
        if (f.e[0] || f.e[1] || f.e[2]) {
            const Faces w = face_weights(L, i, j, k);
            const Om<float4> om = om_of(oms, h, (float4*)nullptr);
            float4 x[3], ax[3];
            curl_rows<float4>(L, w, i, j, k, [&](int e) { return xv[(size_t)e * H + h]; }, x, ax);
            float S[3];
            edge_diags(L, w, S);
#pragma unroll
            for (int D = 0; D < 3; ++D)
                if (f.e[D]) {
                    const float m = __ldg(&L.me[3 * p + D]);
                    const float4 r = b[(size_t)(3 * p + D) * H + h] - ax[D] - imass(om, m, x[D]);
                    out[D] = SMOOTH ? x[D] + idiag(om, kEmgEdge, S[D], m, r) : r;
                }
        }
#pragma unroll
        for (int D = 0; D < 3; ++D) y[(size_t)(3 * p + D) * H + h] = out[D];
    });
}

// b = P^T y_fine, x = w b / d
template <int K>
__global__ void __launch_bounds__(kNT) k_restrict(EmgLevel F, EmgLevel L, Omegas om) {
    dep_begin();
    constexpr int H = K / 2;
    each_point<H>(L, [&](int i, int j, int k, int h) {
        const Free f = edges_free(L, i, j, k);
        const int p = pid(L.n, i, j, k), ne = entries(L);
        const bool lm = lane_major(L);
        float4 s[3], x[3] = {vz<float4>(), vz<float4>(), vz<float4>()};
        const float4* y = f4(F.y);
        gather_edges<float4>(f, F.n, i, j, k, [&](int e) { return y[(size_t)e * H + h]; }, s);
        if (f.e[0] || f.e[1] || f.e[2]) {
            float S[3];
            edge_diags(L, face_weights(L, i, j, k), S);
#pragma unroll
            for (int D = 0; D < 3; ++D)
                x[D] = idiag(om_of(om, h, (float4*)nullptr), kEmgEdge, S[D], __ldg(&L.me[3 * p + D]), s[D]);
        }
#pragma unroll
        for (int D = 0; D < 3; ++D) {
            store2<K>(L.b, lm, ne, 3 * p + D, h, s[D]);
            store2<K>(L.x, lm, ne, 3 * p + D, h, x[D]);
        }
    });
}

// value of the coarse vector interpolated to the fine edge of direction D at (i, j, k)
template <int D, class V, class At>
__device__ __forceinline__ V interp_edge(int n, int i, int j, int k, const At& at) {
    const int n1 = n + 1, e = 3 * pid(n, i >> 1, j >> 1, k >> 1) + D;
    constexpr int A = D == 0 ? 1 : 0, B = D == 2 ? 1 : 2;
    const int q[3] = {i, j, k}, st[3] = {3, 3 * n1, 3 * n1 * n1};
    const int sa = q[A] & 1 ? st[A] : 0, sb = q[B] & 1 ? st[B] : 0;
    V s = at(e);
    if (sa) s = s + at(e + sa);
    if (sb) s = s + at(e + sb);
    if (sa && sb) s = s + at(e + sa + sb);
    return ((sa ? 0.5f : 1.0f) * (sb ? 0.5f : 1.0f)) * s;
}
template <class V, class At>
__device__ __forceinline__ void interp_edges(const Free& f, int n, int i, int j, int k, const At& at, V (&s)[3]) {
    s[0] = f.e[0] ? interp_edge<0, V>(n, i, j, k, at) : vz<V>();
    s[1] = f.e[1] ? interp_edge<1, V>(n, i, j, k, at) : vz<V>();
    s[2] = f.e[2] ? interp_edge<2, V>(n, i, j, k, at) : vz<V>();
}

// x += P y_coarse
template <int K>
__global__ void __launch_bounds__(kNT) k_prolong(EmgLevel L, EmgLevel C) {
    dep_begin();
    constexpr int H = K / 2;
    each_point<H>(L, [&](int i, int j, int k, int h) {
        const Free f = edges_free(L, i, j, k);
        const int p = pid(L.n, i, j, k), ne = entries(C);
        const bool lm = lane_major(C);
        float4 s[3];
        interp_edges<float4>(f, C.n, i, j, k, [&](int e) { return load2<K>(C.y, lm, ne, e, h); }, s);
#pragma unroll
        for (int D = 0; D < 3; ++D)
            if (f.e[D]) {
                const size_t c = (size_t)(3 * p + D) * H + h;
                f4(L.x)[c] = f4(L.x)[c] + s[D];
            }
    });
}

// ---------------------------------------------------------------------------
// The small grids.  Launched step by step, the grids of 16 cells per side and
// less (15 k edges) took five launches of 4 to 16 us; one block for all of
// them was slower still (50 us, one SM's issue rate).  Here a cluster of
// four or eight blocks runs them for one right-hand side: the 16-cell grid is split
// over the cluster's blocks with its vectors in global memory (a right-hand
// side's values together, read past L1), cluster barriers between the steps;
// the grids of 8 and 4 cells run in the shared memory of the first block.
// ---------------------------------------------------------------------------
constexpr int kBottomNT = 768;
constexpr int kCoarsestSteps = 8;
static_assert(kBottomNT >= 9 * 9 * 9 && 8 * kBottomNT >= 17 * 17 * 17, "a point per thread of eight blocks");
// Blocks per cluster: eight up to K = 8, one point of the 16-cell grid per
// thread; four at K = 16, where sixteen clusters of eight took two waves (46
// against 28 us at K = 8).
constexpr int cluster_blocks(int K) { return K > 8 ? 4 : 8; }

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ int cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return (int)r;
}

// A grid point's three edges: which are free, their face weights and masses,
// loaded ahead of the phases that use them.
struct Point {
    int i, j, k, p;
    Free f;
    bool any;
    Faces w;
    float m[3];
    __device__ __forceinline__ void load(const EmgLevel& L, int point, bool on) {
        const int n1 = L.n + 1;
        p = point;
        i = p % n1;
        j = p / n1 % n1;
        k = p / (n1 * n1);
        f = Free{};
        if (on) f = edges_free(L, i, j, k);
        any = f.e[0] || f.e[1] || f.e[2];
        w = Faces{};
        if (any) w = face_weights(L, i, j, k);
#pragma unroll
        for (int D = 0; D < 3; ++D) m[D] = any ? __ldg(&L.me[3 * p + D]) : 0.0f;
    }
};

// Jacobi step or residual at one point, any memory
template <class In, class Rhs>
__device__ __forceinline__ void point_step(const EmgLevel& L, Om<float2> om, const Point& q, bool resid, const In& in,
                                           const Rhs& rhs, float2 (&v)[3]) {
    v[0] = v[1] = v[2] = vz<float2>();
    if (!q.any) return;
    float2 xc[3], ax[3];
    float S[3];
    curl_rows<float2>(L, q.w, q.i, q.j, q.k, in, xc, ax);
    edge_diags(L, q.w, S);
#pragma unroll
    for (int D = 0; D < 3; ++D)
        if (q.f.e[D]) {
            const float2 r = rhs(3 * q.p + D) - ax[D] - imass(om, q.m[D], xc[D]);
            v[D] = resid ? r : xc[D] + idiag(om, kEmgEdge, S[D], q.m[D], r);
        }
}

// Cycle of the levels from l1 (8 or 4 cells) on, by one block: three vectors
// per level in sm; b and x of the first level are filled in by load(b, x).
// Returns the first level's result (shared memory).
template <class Load>
__device__ __forceinline__ const float2* small_cycle(const EmgDev& g, int l1, Om<float2> om, float2* sm,
                                                     const Load& load) {
    const int tid = threadIdx.x, nl = g.n_levels;
    const EmgLevel& L = g.lv[l1];
    const EmgLevel& C = g.lv[nl - 1];
    const bool two = l1 + 1 < nl;
    const int nL = entries(L), nC = entries(C);
    float2 *b = sm, *x = sm + nL, *y = sm + 2 * nL;
    float2 *cb = two ? sm + 3 * nL : b, *cx = two ? cb + nC : x, *cy = two ? cx + nC : y;
    for (float2* z = sm + tid; z < cy + nC; z += kBottomNT) *z = vz<float2>();
    const bool in = tid < points(L);
    Point pl, pc;
    pl.load(L, tid, in && two);
    pc.load(C, tid, tid < points(C));
    float S[3];
    edge_diags(C, pc.w, S);
    float2 rhs[3] = {};
    __syncthreads();
    load(b, x);
    __syncthreads();
    if (two) {
        if (in) {
            float2 v[3];
            point_step(L, om, pl, true, [&](int e) { return x[e]; }, [&](int e) { return b[e]; }, v);
#pragma unroll
            for (int D = 0; D < 3; ++D) y[3 * tid + D] = v[D];
        }
        __syncthreads();
        if (pc.any) {
            gather_edges<float2>(pc.f, L.n, pc.i, pc.j, pc.k, [&](int e) { return y[e]; }, rhs);
#pragma unroll
            for (int D = 0; D < 3; ++D) cx[3 * tid + D] = idiag(om, kEmgEdge, S[D], pc.m[D], rhs[D]);
        }
        __syncthreads();
    } else if (pc.any) {
#pragma unroll
        for (int D = 0; D < 3; ++D) rhs[D] = b[3 * tid + D];
    }
    for (int q = 0; q < kCoarsestSteps; ++q) {
        const float2* u = q & 1 ? cy : cx;
        float2* v = q & 1 ? cx : cy;
        if (pc.any) {
            float2 xc[3], ax[3];
            curl_rows<float2>(C, pc.w, pc.i, pc.j, pc.k, [&](int e) { return u[e]; }, xc, ax);
#pragma unroll
            for (int D = 0; D < 3; ++D)
                if (pc.f.e[D])
                    v[3 * tid + D] =
                        xc[D] + idiag(om, kEmgEdge, S[D], pc.m[D], rhs[D] - ax[D] - imass(om, pc.m[D], xc[D]));
        }
        __syncthreads();
    }
    if (!two) return cx;
    if (in) {
        float2 s[3];
        interp_edges<float2>(pl.f, C.n, pl.i, pl.j, pl.k, [&](int e) { return cx[e]; }, s);
#pragma unroll
        for (int D = 0; D < 3; ++D) x[3 * tid + D] = x[3 * tid + D] + s[D];
    }
    __syncthreads();
    if (in) {
        float2 v[3];
        point_step(L, om, pl, false, [&](int e) { return x[e]; }, [&](int e) { return b[e]; }, v);
#pragma unroll
        for (int D = 0; D < 3; ++D) y[3 * tid + D] = v[D];
    }
    __syncthreads();
    return y;
}

// From level l0 of 8 or 4 cells: one block per right-hand side.
__global__ void __launch_bounds__(kBottomNT) k_bottom(EmgDev g, int l0, Omegas oms) {
    dep_begin();
    extern __shared__ float2 sm[];
    const EmgLevel& L = g.lv[l0];
    const int lane = blockIdx.x, ne = entries(L);
    const float2* v = small_cycle(g, l0, Om<float2>{oms.v[lane]}, sm, [&](float2* b, float2* x) {
        for (int e = threadIdx.x; e < ne; e += kBottomNT) {
            b[e] = L.b[(size_t)lane * ne + e];
            x[e] = L.x[(size_t)lane * ne + e];
        }
    });
    for (int e = threadIdx.x; e < ne; e += kBottomNT) L.y[(size_t)lane * ne + e] = v[e];
}

// From level l0 of 16 cells: a cluster of NC blocks per right-hand side.
template <int NC>
__global__ void __launch_bounds__(kBottomNT) k_bottom16(EmgDev g, int l0, Omegas oms) {
    dep_begin();
    extern __shared__ float2 sm[];
    constexpr int PT = 8 / NC;   // points per thread
    const EmgLevel& L = g.lv[l0];
    const EmgLevel& C = g.lv[l0 + 1];
    const int lane = blockIdx.x / NC, rank = cluster_rank(), tid = threadIdx.x, ne = entries(L), nc = entries(C);
    const Om<float2> om{oms.v[lane]};
    const float2* b = L.b + (size_t)lane * ne;
    float2 *x = L.x + (size_t)lane * ne, *y = L.y + (size_t)lane * ne, *cy = C.y + (size_t)lane * nc;
    const int m = (L.n + 1) * (L.n + 1) * edge_planes(L);
    Point q[PT];
    float2 v[3];
#pragma unroll
    for (int u = 0; u < PT; ++u) {
        const int p = (u * NC + rank) * kBottomNT + tid;
        q[u].load(L, p, p < m);
        if (p < m) {
            point_step(L, om, q[u], true, [&](int e) { return x[e]; }, [&](int e) { return b[e]; }, v);
#pragma unroll
            for (int D = 0; D < 3; ++D) y[3 * p + D] = v[D];
        }
    }
    cluster_sync();
    if (rank == 0) {
        const float2* r = small_cycle(g, l0 + 1, om, sm, [&](float2* cb, float2* cx) {
            Point c;
            c.load(C, tid, tid < points(C));
            if (!c.any) return;
            float2 s[3];
            float S[3];
            gather_edges<float2>(c.f, L.n, c.i, c.j, c.k, [&](int e) { return __ldcg(&y[e]); }, s);
            edge_diags(C, c.w, S);
#pragma unroll
            for (int D = 0; D < 3; ++D) {
                cb[3 * tid + D] = s[D];
                cx[3 * tid + D] = idiag(om, kEmgEdge, S[D], c.m[D], s[D]);
            }
        });
        for (int e = tid; e < nc; e += kBottomNT) cy[e] = r[e];
    }
    cluster_sync();
#pragma unroll
    for (int u = 0; u < PT; ++u)
        if (q[u].any) {
            interp_edges<float2>(q[u].f, C.n, q[u].i, q[u].j, q[u].k, [&](int e) { return __ldcg(&cy[e]); }, v);
#pragma unroll
            for (int D = 0; D < 3; ++D)
                if (q[u].f.e[D]) x[3 * q[u].p + D] = x[3 * q[u].p + D] + v[D];
        }
    cluster_sync();
#pragma unroll
    for (int u = 0; u < PT; ++u)
        if (q[u].p < m) {
            point_step(L, om, q[u], false, [&](int e) { return __ldcg(&x[e]); }, [&](int e) { return b[e]; }, v);
#pragma unroll
            for (int D = 0; D < 3; ++D) y[3 * q[u].p + D] = v[D];
        }
}

// ---------------------------------------------------------------------------
// node cycle: V(0,1) in the edge preconditioner, the symmetric V(1,1) (PRE) in
// the divergence correction's PCG
// ---------------------------------------------------------------------------

// Laplacian row on a uniform grid: six edges, coarse edge masses over h^2
template <class V, class At>
__device__ __forceinline__ V lap_row(const EmgLevel& L, int i, int j, int k, V xc, const At& at, float& d) {
    const int n1 = L.n + 1, p = pid(L.n, i, j, k);
    V s = vz<V>();
    d = 0.0f;
    auto put = [&](int e, int v, float ih2) {
        const float m = __ldg(&L.me[e]) * ih2;
        s = s + m * (xc - at(v));
        d += m;
    };
    const float a = 1.0f / (L.h[0] * L.h[0]), b = 1.0f / (L.h[1] * L.h[1]), c = 1.0f / (L.h[2] * L.h[2]);
    put(3 * (p - 1), p - 1, a);
    put(3 * p, p + 1, a);
    put(3 * (p - n1) + 1, p - n1, b);
    put(3 * p + 1, p + n1, b);
    put(3 * (p - n1 * n1) + 2, p - n1 * n1, c);
    put(3 * p + 2, p + n1 * n1, c);
    return s;
}

// w b / diag, the pre-smoothed iterate of the V(1,1) cycle
template <class V> __device__ __forceinline__ V node_pre(const EmgLevel& L, int i, int j, int k, V b) {
    if (!node_free(L, i, j, k)) return vz<V>();
    float d;
    lap_row<F1>(L, i, j, k, F1{0.0f}, [&](int) { return F1{0.0f}; }, d);
    return d > 0.0f ? (kEmgNode / d) * b : vz<V>();
}

// nb0 = Pn^T b from the octree nodes; PRE: nt0 = w nb0 / diag
template <int K, bool PRE>
__global__ void __launch_bounds__(kNT) k_node_restrict0(EmgDev g, const float4* b) {
    dep_begin();
    constexpr int H = K / 2;
    const EmgLevel& L = g.lv[0];
    each_point<H>(L, [&](int i, int j, int k, int h) {
        const int c = pid(L.n, i, j, k);
        float4 s = vz<float4>();
        const int q0 = __ldg(&g.nr_ptr[c]), q1 = __ldg(&g.nr_ptr[c + 1]);
        if (q1 - q0 > kLongNode) return;   // k_node_restrict0_long
        for (int q = q0; q < q1; q += 9) {   // 27 entries under one level of refinement
            float w[9];
            float4 v[9];
#pragma unroll
            for (int u = 0; u < 9; ++u) {
                const bool ok = q + u < q1;
                w[u] = ok ? __ldg(&g.nr_w[q + u]) : 0.0f;
                v[u] = ok ? b[(size_t)__ldg(&g.nr_node[q + u]) * H + h] : vz<float4>();
            }
#pragma unroll
            for (int u = 0; u < 9; ++u) s = s + w[u] * v[u];
        }
        store2<K>(L.nb, lane_major(L), points(L), c, h, s);
        if (PRE && !lane_major(L)) f4(L.nt)[(size_t)c * H + h] = node_pre(L, i, j, k, s);
    });
}

template <int K, bool PRE>
__global__ void __launch_bounds__(kLongNT) k_node_restrict0_long(EmgDev g, const float4* b) {
    dep_begin();
    constexpr int H = K / 2;
    const EmgLevel& L = g.lv[0];
    const int c = g.nr_long[blockIdx.x], n1 = L.n + 1, h = threadIdx.x % H;
    const float4 s = long_row<H>(g.nr_node, g.nr_w, g.nr_ptr[c], g.nr_ptr[c + 1], b);
    if (threadIdx.x >= H) return;
    store2<K>(L.nb, lane_major(L), points(L), c, h, s);
    if (PRE && !lane_major(L))
        f4(L.nt)[(size_t)c * H + h] = node_pre(L, c % n1, c / n1 % n1, c / (n1 * n1), s);
}

// ny = nb - L nt, or (SMOOTH) ny = nt + w (nb - L nt) / diag
template <int K, bool SMOOTH>
__global__ void __launch_bounds__(kNT) k_node_step(EmgLevel L) {
    dep_begin();
    constexpr int H = K / 2;
    each_point<H>(L, [&](int i, int j, int k, int h) {
        const size_t c = (size_t)pid(L.n, i, j, k) * H + h;
        float4 v = vz<float4>();
        if (node_free(L, i, j, k)) {
            const float4* t = f4(L.nt);
            const float4 tc = t[c];
            float d;
            v = f4(L.nb)[c] - lap_row<float4>(L, i, j, k, tc, [&](int q) { return t[(size_t)q * H + h]; }, d);
            if (SMOOTH) v = d > 0.0f ? tc + (kEmgNode / d) * v : tc;
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
                            at(pid(n, 2 * I + a, 2 * J + b, 2 * Kk + c));
    return s;
}
template <class V, class At>
__device__ __forceinline__ V interp_node(int n, int i, int j, int k, const At& at) {
    const int oi = i & 1, oj = j & 1, ok = k & 1;
    V s = vz<V>();
    for (int c = 0; c <= ok; ++c)
        for (int b = 0; b <= oj; ++b)
            for (int a = 0; a <= oi; ++a) s = s + at(pid(n, (i >> 1) + a, (j >> 1) + b, (k >> 1) + c));
    return ((oi ? 0.5f : 1.0f) * (oj ? 0.5f : 1.0f) * (ok ? 0.5f : 1.0f)) * s;
}

// nb = Pn^T of the finer level's right-hand side, or (PRE) of its residual in
// ny, with nt = w nb / diag
template <int K, bool PRE>
__global__ void __launch_bounds__(kNT) k_node_restrict(EmgLevel F, EmgLevel L) {
    dep_begin();
    constexpr int H = K / 2;
    each_point<H>(L, [&](int i, int j, int k, int h) {
        float4 s = vz<float4>();
        const float4* b = f4(PRE ? F.ny : F.nb);
        if (node_free(L, i, j, k))
            s = gather_node<float4>(F.n, i, j, k, [&](int v) { return b[(size_t)v * H + h]; });
        const int c = pid(L.n, i, j, k);
        store2<K>(L.nb, lane_major(L), points(L), c, h, s);
        if (PRE && !lane_major(L)) f4(L.nt)[(size_t)c * H + h] = node_pre(L, i, j, k, s);
    });
}

// nt = Pn y_coarse, or (PRE) nt += Pn y_coarse
template <int K, bool PRE>
__global__ void __launch_bounds__(kNT) k_node_prolong(EmgLevel L, EmgLevel C) {
    dep_begin();
    constexpr int H = K / 2;
    each_point<H>(L, [&](int i, int j, int k, int h) {
        float4 s = vz<float4>();
        const bool lm = lane_major(C);
        const int np = points(C);
        if (node_free(L, i, j, k))
            s = interp_node<float4>(C.n, i, j, k, [&](int v) { return load2<K>(C.ny, lm, np, v, h); });
        const size_t c = (size_t)pid(L.n, i, j, k) * H + h;
        f4(L.nt)[c] = PRE ? f4(L.nt)[c] + s : s;
    });
}

// The small node grids, as the small edge grids above.
template <bool PRE, class Load>
__device__ __forceinline__ const float2* small_node_cycle(const EmgDev& g, int l1, float2* sm, const Load& load) {
    const int tid = threadIdx.x, nl = g.n_levels;
    const EmgLevel& L = g.lv[l1];
    const EmgLevel& C = g.lv[nl - 1];
    const bool two = l1 + 1 < nl;
    const int nL = points(L), nC = points(C);
    float2 *b = sm, *x = sm + nL, *y = sm + 2 * nL;
    float2 *cb = two ? sm + 3 * nL : b, *cx = two ? cb + nC : x, *cy = two ? cx + nC : y;
    for (float2* z = sm + tid; z < cy + nC; z += kBottomNT) *z = vz<float2>();
    const int n1 = L.n + 1, i = tid % n1, j = tid / n1 % n1, k = tid / (n1 * n1);
    const int c1 = C.n + 1, ci = tid % c1, cj = tid / c1 % c1, ck = tid / (c1 * c1);
    const bool in = tid < nL && node_free(L, i, j, k), cin = tid < nC && node_free(C, ci, cj, ck);
    __syncthreads();
    load(b);
    __syncthreads();
    auto step = [&](const EmgLevel& M, bool on, int a, int c, int d, const float2* rhs, const float2* v, float2* out) {
        if (on) {
            float dg;
            const float2 r = rhs[tid] - lap_row<float2>(M, a, c, d, v[tid], [&](int q) { return v[q]; }, dg);
            out[tid] = dg > 0.0f ? v[tid] + (kEmgNode / dg) * r : v[tid];
        }
        __syncthreads();
    };
    if (two) {
        const float2* src = b;
        if (PRE) {
            if (in) x[tid] = node_pre(L, i, j, k, b[tid]);
            __syncthreads();
            if (in) {
                float dg;
                y[tid] = b[tid] - lap_row<float2>(L, i, j, k, x[tid], [&](int q) { return x[q]; }, dg);
            }
            __syncthreads();
            src = y;
        }
        if (cin) cb[tid] = gather_node<float2>(L.n, ci, cj, ck, [&](int q) { return src[q]; });
        __syncthreads();
    }
    for (int q = 0; q < kCoarsestSteps; q += 2) {   // from zero
        step(C, cin, ci, cj, ck, cb, cx, cy);
        step(C, cin, ci, cj, ck, cb, cy, cx);
    }
    if (!two) return cx;
    if (in) x[tid] = x[tid] + interp_node<float2>(C.n, i, j, k, [&](int q) { return cx[q]; });
    __syncthreads();
    step(L, in, i, j, k, b, x, y);
    return y;
}

template <bool PRE> __global__ void __launch_bounds__(kBottomNT) k_node_bottom(EmgDev g, int l0) {
    dep_begin();
    extern __shared__ float2 sm[];
    const EmgLevel& L = g.lv[l0];
    const int lane = blockIdx.x, np = points(L);
    const float2* v = small_node_cycle<PRE>(g, l0, sm, [&](float2* b) {
        for (int t = threadIdx.x; t < np; t += kBottomNT) b[t] = L.nb[(size_t)lane * np + t];
    });
    for (int t = threadIdx.x; t < np; t += kBottomNT) L.ny[(size_t)lane * np + t] = v[t];
}

template <int NC, bool PRE> __global__ void __launch_bounds__(kBottomNT) k_node_bottom16(EmgDev g, int l0) {
    dep_begin();
    extern __shared__ float2 sm[];
    constexpr int PT = 8 / NC;
    const EmgLevel& L = g.lv[l0];
    const EmgLevel& C = g.lv[l0 + 1];
    const int lane = blockIdx.x / NC, rank = cluster_rank(), tid = threadIdx.x, np = points(L), nc = points(C);
    const float2* b = L.nb + (size_t)lane * np;
    float2 *x = L.nt + (size_t)lane * np, *y = L.ny + (size_t)lane * np, *cy = C.ny + (size_t)lane * nc;
    float2 xv[PT];
    auto each = [&](const auto& f) {   // f(u, i, j, k, p, free)
#pragma unroll
        for (int u = 0; u < PT; ++u) {
            const int p = (u * NC + rank) * kBottomNT + tid, n1 = L.n + 1;
            const int i = p % n1, j = p / n1 % n1, k = p / (n1 * n1);
            if (p < np) f(u, i, j, k, p, node_free(L, i, j, k));
        }
    };
#pragma unroll
    for (int u = 0; u < PT; ++u) xv[u] = vz<float2>();
    if (PRE) {
        each([&](int u, int i, int j, int k, int p, bool in) {
            if (in) xv[u] = node_pre(L, i, j, k, b[p]);
            x[p] = xv[u];
        });
        cluster_sync();
        each([&](int u, int i, int j, int k, int p, bool in) {
            float d;
            y[p] = in ? b[p] - lap_row<float2>(L, i, j, k, xv[u], [&](int q) { return __ldcg(&x[q]); }, d) : vz<float2>();
        });
        cluster_sync();
    }
    if (rank == 0) {
        const float2* src = PRE ? y : b;
        const float2* r = small_node_cycle<PRE>(g, l0 + 1, sm, [&](float2* cb) {
            const int m1 = C.n + 1, ci = tid % m1, cj = tid / m1 % m1, ck = tid / (m1 * m1);
            if (tid < nc && node_free(C, ci, cj, ck))
                cb[tid] = gather_node<float2>(L.n, ci, cj, ck, [&](int q) { return __ldcg(&src[q]); });
        });
        for (int t = tid; t < nc; t += kBottomNT) cy[t] = r[t];
    }
    cluster_sync();
    each([&](int u, int i, int j, int k, int p, bool in) {
        if (in) xv[u] = xv[u] + interp_node<float2>(C.n, i, j, k, [&](int q) { return __ldcg(&cy[q]); });
        x[p] = xv[u];
    });
    cluster_sync();
    each([&](int u, int i, int j, int k, int p, bool in) {
        float2 v = vz<float2>();
        if (in) {
            float d;
            v = b[p] - lap_row<float2>(L, i, j, k, xv[u], [&](int q) { return __ldcg(&x[q]); }, d);
            v = d > 0.0f ? xv[u] + (kEmgNode / d) * v : xv[u];
        }
        y[p] = v;
    });
}

// t = Pn ny0 on the octree nodes (0 on Dirichlet nodes), plus x if given
template <int K>
__global__ void __launch_bounds__(kNT) k_node_prolong0(EmgDev g, int nn, const float4* x,
                                                       float4* __restrict__ out) {
    dep_begin();
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
        const EmgLevel& L = g.lv[0];
        const int n1 = L.n + 1, np = points(L);
        const bool lm = lane_major(L);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float w = (q & 1 ? fx : 1.0f - fx) * (q & 2 ? fy : 1.0f - fy) * (q & 4 ? fz : 1.0f - fz);
            if (w > 0.0f)
                s = s + w * load2<K>(L.ny, lm, np, base + (q & 1) + (q >> 1 & 1) * n1 + (q >> 2) * n1 * n1, h);
        }
    }
    out[i] = s;
}

// z0 = P y0 + G~ yn / (i omega) + w r / d on free rows, r on identity rows
template <int K>
__global__ void __launch_bounds__(kNT) k_combine(EmgDev g, GcRowTerm gt, DiagView<float> D, Omegas om, long n,
                                                 const float4* r, float4* __restrict__ z0) {
    dep_begin();
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
        const EmgLevel& L = g.lv[0];
        const int d = code & 3u, n1 = L.n + 1, ne = entries(L);
        const int sa = d == 0 ? 3 * n1 : 3, sb = d == 2 ? 3 * n1 : 3 * n1 * n1;
        const bool lm = lane_major(L);
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
            if (w > 0.0f) z = z + w * load2<K>(L.y, lm, ne, base + (q & 1) * sa + (q >> 1) * sb, h);
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

// Launches the kernel of the small grids from level l0 on: 16 cells as a
// cluster per right-hand side (its own grid in global memory), less as a block.
// per: vectors' entries per level in shared memory, three of them.
template <class F16, class F8, class... Args>
void launch_bottom(F16* k16, F8* k8, const EmgDev& g, int l0, int K, long (*per)(int), cudaStream_t s, Args... args) {
    const int nc = cluster_blocks(K);
    const bool big = g.lv[l0].n > 8;
    int smem = 0;
    for (int l = l0 + (big ? 1 : 0); l < g.n_levels; ++l) smem += 3 * (int)(per(g.lv[l].n) * sizeof(float2));
    const void* f = big ? reinterpret_cast<const void*>(k16) : reinterpret_cast<const void*>(k8);
    if (smem > 16 * 1024) lift_smem_limit(f);   // with the static arrays beyond 48 KB
    if (!big) {
        launch_dep(k8, K, kBottomNT, (size_t)smem, s, g, l0, args...);
        return;
    }
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = nc;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(K * nc));
    cfg.blockDim = dim3(kBottomNT);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    dep_attr(cfg, at);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k16, g, l0, args...);
    if (e != cudaSuccess) throw std::runtime_error(cudaGetErrorString(e));
}

template <int K>
void edge_cycle(const EmgDev& g, const Omegas& om, const float2* r, cudaStream_t s, long long* launches) {
    const int l0 = bottom_level(g), n = (int)(3L * (g.lv[0].n + 1) * (g.lv[0].n + 1) * edge_planes(g.lv[0]));
    k_restrict0<K><<<grid1((long)n * (K / 2)), kNT, 0, s>>>(g, om, f4(r), n);
    ck(launches);
    if (g.n_r_long) {
        launch_dep(k_restrict0_long<K>, g.n_r_long, kLongNT, 0, s, g, om, f4(r));
        ck(launches);
    }
    auto grid = [&](int l) { return point_grid<K>(g.lv[l], edge_planes(g.lv[l])); };
    for (int l = 0; l < l0; ++l) {
        launch_dep(k_edge_step<K, false>, grid(l), kNT, 0, s, g.lv[l], om);
        ck(launches);
        launch_dep(k_restrict<K>, grid(l + 1), kNT, 0, s, g.lv[l], g.lv[l + 1], om);
        ck(launches);
    }
    launch_bottom(k_bottom16<cluster_blocks(K)>, k_bottom, g, l0, K, emg_entries, s, om);
    ck(launches);
    for (int l = l0 - 1; l >= 0; --l) {
        launch_dep(k_prolong<K>, grid(l), kNT, 0, s, g.lv[l], g.lv[l + 1]);
        ck(launches);
        launch_dep(k_edge_step<K, true>, grid(l), kNT, 0, s, g.lv[l], om);
        ck(launches);
    }
}

// the uniform grids' part of a node cycle, from octree node vector b to ny of level 0
template <int K, bool PRE>
void node_grids(const EmgDev& g, const float2* b, cudaStream_t s, long long* launches) {
    const int l0 = bottom_level(g);
    auto grid = [&](int l) { return point_grid<K>(g.lv[l], node_planes(g.lv[l])); };
    launch_dep(k_node_restrict0<K, PRE>, grid(0), kNT, 0, s, g, f4(b));
    ck(launches);
    if (g.n_nr_long) {
        launch_dep(k_node_restrict0_long<K, PRE>, g.n_nr_long, kLongNT, 0, s, g, f4(b));
        ck(launches);
    }
    for (int l = 0; l < l0; ++l) {
        if (PRE) {
            launch_dep(k_node_step<K, false>, grid(l), kNT, 0, s, g.lv[l]);
            ck(launches);
        }
        launch_dep(k_node_restrict<K, PRE>, grid(l + 1), kNT, 0, s, g.lv[l], g.lv[l + 1]);
        ck(launches);
    }
    launch_bottom(k_node_bottom16<cluster_blocks(K), PRE>, k_node_bottom<PRE>, g, l0, K, emg_points, s);
    ck(launches);
    for (int l = l0 - 1; l >= 0; --l) {
        launch_dep(k_node_prolong<K, PRE>, grid(l), kNT, 0, s, g.lv[l], g.lv[l + 1]);
        ck(launches);
        launch_dep(k_node_step<K, true>, grid(l), kNT, 0, s, g.lv[l]);
        ck(launches);
    }
}

template <int K>
void node_cycle(const EmgDev& g, const GcDev& gc, const float2* r, cudaStream_t s, long long* launches) {
    gc_restrict_edges_k<K>(gc, r, s, launches);
    node_grids<K, false>(g, gc.lv[0].b, s, launches);
    launch_dep(k_node_prolong0<K>, grid1((long)gc.nn * (K / 2)), kNT, 0, s, g, gc.nn, nullptr, f4(gc.lv[0].y));
    ck(launches);
    gc_smooth0_k<K>(gc, gc.lv[0].y, gc.out0, s, launches);
}

}  // namespace

std::vector<int> emg_long_rows(const std::vector<int>& ptr, bool nodes) {
    std::vector<int> rows;
    for (size_t c = 0; c + 1 < ptr.size(); ++c)
        if (ptr[c + 1] - ptr[c] > (nodes ? kLongNode : kLongEdge)) rows.push_back((int)c);
    return rows;
}

void emg_set_mass(const EmgDev& g, const double* Me, cudaStream_t s, long long* launches) {
    const int n = (int)emg_entries(g.lv[0].n);
    k_mass0<<<(n + 255) / 256, 256, 0, s>>>(g, Me, n);
    ck(launches);
    for (int l = 1; l < g.n_levels; ++l) {
        k_mass<<<(int)((emg_points(g.lv[l].n) + 255) / 256), 256, 0, s>>>(g.lv[l - 1], g.lv[l]);
        ck(launches);
    }
}

template <int K>
void emg_coarse_k(const KrylovCtx<float>& c, const float2* r, float2* z0) {
    const EmgDev& g = *c.emg;
    const GcDev& gc = *c.gc;
    Omegas om;
    for (int k = 0; k < kMaxRhs; ++k) om.v[k] = k < K ? (float)c.B.omega[k] : 0.0f;
    const double nb = (double)c.n_rows * K * sizeof(float2), nn = (double)gc.nn * K * sizeof(float2);
    const double side = g.lv[0].n + 1, e0 = 3.0 * side * side * edge_planes(g.lv[0]) * K * sizeof(float2);
    // r gathered by both restrictions and read by the last kernel, z0 written;
    // level-0 edge vectors: b, x written and read, the residual written and
    // read, x updated, x, b read and y written, y read; octree node vectors: b
    // written and read twice, t written and read, the result likewise
    const int th = c.timer ? c.timer->begin(kClsGradcorr, 4 * nb + 12 * e0 + 7 * nn, K) : -1;
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
    if (c.gc_stream)   // behind another stream's kernels: a plain launch
        k_combine<K><<<grid1(n), kNT, 0, c.stream>>>(g, gc_row_term(gc, c.B), c.D, om, n, f4(r), f4(z0));
    else
        launch_dep(k_combine<K>, grid1(n), kNT, 0, c.stream, g, gc_row_term(gc, c.B), c.D, om, n, f4(r), f4(z0));
    ck(c.launches);
    if (c.timer) c.timer->end(th);
}

template <int K>
void emg_node_precond_k(const EmgDev& g, const GcDev& gc, float2* z, cudaStream_t s, long long* launches) {
    gc_presmooth0_k<K>(gc, s, launches);   // x = omega D^-1 b, y = b - L x
    node_grids<K, true>(g, gc.lv[0].y, s, launches);
    launch_dep(k_node_prolong0<K>, grid1((long)gc.nn * (K / 2)), kNT, 0, s, g, gc.nn, f4(gc.lv[0].x), f4(gc.lv[0].y));
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
