// Device helpers shared by the solver kernels: complex arithmetic on
// double2 / float2, warp and block reductions, and a deterministic grid
// reduction (per-block partials summed in block order by the last block).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace m3d {
namespace dev {

constexpr int kWarp = 32;
constexpr int kBlock = 256;               // threads per block for every kernel here
constexpr int kWarpsPerBlock = kBlock / kWarp;
constexpr int kSlice = 32;                // sliced-ELL slice height (rows per warp)
constexpr int kMaxRhs = 16;               // right-hand sides per batched launch
constexpr int kMaxQ = 3;                  // reduced quantities per kernel

template <class R> struct CTraits;
template <> struct CTraits<double> { using C = double2; };
template <> struct CTraits<float> { using C = float2; };
template <class R> using cplx = typename CTraits<R>::C;

template <class R> __host__ __device__ __forceinline__ cplx<R> cm(R a, R b) {
    cplx<R> z; z.x = a; z.y = b; return z;
}
template <class C> __host__ __device__ __forceinline__ C cadd(C a, C b) { a.x += b.x; a.y += b.y; return a; }
template <class C> __host__ __device__ __forceinline__ C csub(C a, C b) { a.x -= b.x; a.y -= b.y; return a; }
template <class C> __host__ __device__ __forceinline__ C cneg(C a) { a.x = -a.x; a.y = -a.y; return a; }
template <class C> __host__ __device__ __forceinline__ C cmul(C a, C b) {
    C z; z.x = a.x * b.x - a.y * b.y; z.y = a.x * b.y + a.y * b.x; return z;
}
// conj(a) * b
template <class C> __host__ __device__ __forceinline__ C cjmul(C a, C b) {
    C z; z.x = a.x * b.x + a.y * b.y; z.y = a.x * b.y - a.y * b.x; return z;
}
template <class C, class R> __host__ __device__ __forceinline__ C cscale(C a, R s) { a.x *= s; a.y *= s; return a; }
template <class C> __host__ __device__ __forceinline__ double cabs2(C a) { return (double)a.x * a.x + (double)a.y * a.y; }
__host__ __device__ __forceinline__ double cabsd(double2 a) { return hypot(a.x, a.y); }
// Smith's algorithm for a / b (R. L. Smith, CACM 5(8), 1962).
__host__ __device__ __forceinline__ double2 cdiv(double2 a, double2 b) {
    double2 z;
    if (fabs(b.x) >= fabs(b.y)) {
        const double r = b.y / b.x, d = b.x + b.y * r;
        z.x = (a.x + a.y * r) / d; z.y = (a.y - a.x * r) / d;
    } else {
        const double r = b.x / b.y, d = b.x * r + b.y;
        z.x = (a.x * r + a.y) / d; z.y = (a.y * r - a.x) / d;
    }
    return z;
}
__host__ __device__ __forceinline__ double2 to_d(double2 a) { return a; }
__host__ __device__ __forceinline__ double2 to_d(float2 a) { return make_double2(a.x, a.y); }
template <class C> __host__ __device__ __forceinline__ C from_d(double2 a);
template <> __host__ __device__ __forceinline__ double2 from_d<double2>(double2 a) { return a; }
template <> __host__ __device__ __forceinline__ float2 from_d<float2>(double2 a) {
    return make_float2((float)a.x, (float)a.y);
}

__device__ __forceinline__ double shfl_xor(double v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }
__device__ __forceinline__ double2 shfl_xor(double2 v, int m) {
    v.x = __shfl_xor_sync(0xffffffffu, v.x, m);
    v.y = __shfl_xor_sync(0xffffffffu, v.y, m);
    return v;
}

// A sum of FP32 terms in the making: three floats, the sum, the sum of its
// rounding errors and that of theirs (Knuth's error-free two-sum; Ogita, Rump
// and Oishi's SumK, 2005, K = 3), some 70 bits in all; each waits four cycles
// for its own last value only.  An FP64 add holds a warp's pipe for 16 cycles
// on this GPU and a chain of them is slow: summing lanes, warps and blocks in
// FP64 was 10 to 25 us of every reducing FP32 kernel; two floats would keep 48
// bits where FP64 keeps 53, and save 0.6 us a kernel (an iteration of two
// right-hand sides on 20 k edges: 131 us, with two floats 129).  Sums that leave
// the FP32 range are done over in FP64 (grid_reduce_f32).
struct Sum3 {
    float h = 0.0f, m = 0.0f, l = 0.0f;
    static __device__ __forceinline__ float two_sum(float a, float b, float& e) {
        const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
        e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t));
        return s;
    }
    __device__ __forceinline__ void add(float a) {
        float e, f;
        h = two_sum(h, a, e);
        m = two_sum(m, e, f);
        l = __fadd_rn(l, f);
    }
    __device__ __forceinline__ void add(const Sum3& o) {
        float e, f, g;
        h = two_sum(h, o.h, e);
        m = two_sum(m, o.m, f);
        m = two_sum(m, e, g);
        l = __fadd_rn(l, __fadd_rn(o.l, __fadd_rn(f, g)));
    }
    __device__ __forceinline__ Sum3 xor_lane(int q) const {
        Sum3 o;
        o.h = __shfl_xor_sync(0xffffffffu, h, q);
        o.m = __shfl_xor_sync(0xffffffffu, m, q);
        o.l = __shfl_xor_sync(0xffffffffu, l, q);
        return o;
    }
    __device__ __forceinline__ bool finite() const { return fabsf(h) <= 3.402823466e38f && m == m; }
    __device__ __forceinline__ double get() const { return (double)h + ((double)m + (double)l); }
};

// One thread's sum over up to 10^5 terms.  The terms of a round go to s if the
// largest modulus among them is small, so that no such sum leaves the FP32
// range, and to FP64 else: one test a round (a test a term kept the adds of
// several sums from overlapping: network gradients 1.00 -> 1.10 ms).
struct ThreadSum {
    Sum3 s;
    double over = 0.0;
    static __device__ __forceinline__ bool small(float modulus) { return modulus <= 1e33f; }
    __device__ __forceinline__ void add_large(float a) { over += (double)a; }
};

// Dependent launches.  A kernel launched by launch_dep may start while its
// predecessor in the stream still runs: its blocks are scheduled and whatever
// no kernel writes (matrix copies, index arrays, barriers) is under way when
// the predecessor ends, and dep_wait() returns then, with all of the
// predecessor's writes visible.  The small grids' and the small meshes'
// kernels run for 5-30 us, of which the way from one launch to the next was 1
// to 2: three frequencies and gradient on 157 k edges 40.5 -> 35.8 ms, one
// frequency on 15 k edges 11.2 -> 9.4 ms.  Rules:
//  * a kernel launched so calls dep_wait() before its first access to anything
//    that a kernel of the chain writes, and every block calls it;
//  * such data is not read through `const __restrict__` pointers or __ldg (the
//    read-only path is not ordered behind the wait);
//  * what is read before the wait was complete when the chain's first, plain
//    launch started (a plain launch waits for all work before it) and is not
//    written by that kernel either: it lets its successor start like the others.
// dep_begin() is dep_trigger() (let the successor start, under any launch) and
// dep_wait() (which does nothing under a plain launch).
__device__ __forceinline__ void dep_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_begin() {
    dep_trigger();
    dep_wait();
}

// Test hook: this thread's launches are plain ones (set for the time of a call).
inline thread_local bool plain_launches = false;

// Adds the attribute of a dependent launch, if the stream is not being captured.
inline void dep_attr(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at) {
    if (plain_launches) return;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(cfg.stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) return;
    at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    ++cfg.numAttrs;
}

// Launch errors stay with the runtime, for the caller's cudaGetLastError().
template <class... P, class... A>
inline void launch_dep(void (*kernel)(P...), dim3 grid, int block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchAttribute at[1];
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = at;
    dep_attr(cfg, at);
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Blocks of `threads` threads with `smem` bytes of dynamic shared memory of
// `kernel` that are resident on the current device at once (occupancy API x
// SM count); cached per (device, kernel, threads, smem).
int resident_blocks(const void* kernel, int threads = kBlock, int smem = 0);

// Lets `kernel` be launched with any dynamic shared memory the device has: the
// limit is set to the most there is, once per (device, kernel).  It belongs to
// the function, not to the launch: set to each launch's own size, a second
// solver's thread could lower it between this one's call and its launch.
// Returns that size (0: an error, which the launch reports).
int lift_smem_limit(const void* kernel);

// One resident wave of `kernel`, at most `cap` blocks.
template <class F>
inline int wave_grid(F* kernel, int cap, int threads = kBlock, int smem = 0) {
    const int g = resident_blocks(reinterpret_cast<const void*>(kernel), threads, smem);
    return g < cap ? g : cap;
}

// This block's contiguous range of n work items, and the blocks of such a
// launch: eight per SM at 256 threads (152 SMs).  Gathers of rows numbered
// along the octree's cell order hit L1 when a block keeps to neighbouring rows;
// items dealt out block by block spread neighbours over the SMs.
struct Range { long b, e; };
__device__ __forceinline__ Range block_range(long n) {
    return {n * blockIdx.x / gridDim.x, n * (blockIdx.x + 1) / gridDim.x};
}
inline int range_grid(long n, int threads = kBlock) {
    const long b = (n + threads - 1) / threads;
    return (int)(b < 1 ? 1 : b < 1216 ? b : 1216);
}

// Scratch for grid reductions: partial[block][kMaxQ * kMaxRhs] (two double2
// each) and a counter that the last block resets.
struct RedScratch {
    double2* partial;
    double2* final_;      // [kMaxQ * kMaxRhs], result of the last reduction
    unsigned int* counter;
    int max_blocks;
};

// Grid reductions for kernels whose thread t always works on the same
// right-hand sides, LPT neighbouring ones, LPT (t % (K / LPT)) and the next (K
// and LPT powers of two, whole warps).  Every step in a fixed order, so the
// result is deterministic for a fixed launch shape.  They return true in the
// last block to arrive, where out (shared) holds the totals.

// FP64 terms, one right-hand side a thread: acc[q] is quantity q; out[q * K + k].
// Shuffle trees over the lanes that share a right-hand side, then over the
// block's warps, then, in the last block, over the blocks, all totals at once.
template <int NQ, int K, int NT = kBlock>
__device__ bool grid_reduce_lanes(const double2 (&acc)[NQ], RedScratch rs, double2* out) {
    static_assert(K >= 1 && K <= 32 && (K & (K - 1)) == 0, "K must be a power of two <= 32");
    static_assert(NT % 32 == 0 && NT >= 32 && NT <= 1024, "block size must be whole warps");
    constexpr int PK = NQ * K;
    constexpr int NW = NT / 32;
    __shared__ double2 sm[NW][PK];
    __shared__ bool am_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        double2 s = acc[q];
#pragma unroll
        for (int off = 16; off >= K; off >>= 1) s = cadd(s, shfl_xor(s, off));
        if (lane < K) sm[warp][q * K + lane] = s;
    }
    __syncthreads();
    // GW lanes per total, one for each warp of the block
    constexpr int GW = NW <= 1 ? 1 : NW <= 2 ? 2 : NW <= 4 ? 4 : NW <= 8 ? 8 : NW <= 16 ? 16 : 32;
#pragma unroll
    for (int p0 = 0; p0 < PK; p0 += NT / GW) {
        const int p = p0 + threadIdx.x / GW, w = threadIdx.x % GW;
        if (p0 + warp * (32 / GW) >= PK) break;   // idle warps would add zeros, 16 cycles an FP64 add
        double2 s = w < NW && p < PK ? sm[w][p] : make_double2(0.0, 0.0);
#pragma unroll
        for (int off = GW / 2; off > 0; off >>= 1) s = cadd(s, shfl_xor(s, off));
        if (w == 0 && p < PK) {
            __stcg(&rs.partial[(size_t)blockIdx.x * PK + p], s);
            __threadfence();
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned t = atomicAdd(rs.counter, 1u);
        am_last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!am_last) return false;
    __threadfence();
    // TPT lanes per total, every total at once
    constexpr int Q = NT / PK;
    constexpr int TPT = Q >= 32 ? 32 : Q >= 16 ? 16 : Q >= 8 ? 8 : Q >= 4 ? 4 : Q >= 2 ? 2 : 1;
    static_assert(Q >= 1, "a thread per total");
    const int p = threadIdx.x / TPT, l = threadIdx.x % TPT;
    if (warp * (32 / TPT) < PK) {
        double2 s = make_double2(0.0, 0.0);
        for (int b = l; p < PK && b < (int)gridDim.x; b += 4 * TPT) {   // four loads in flight
            double2 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                v[u] = b + TPT * u < (int)gridDim.x ? __ldcg(&rs.partial[(size_t)(b + TPT * u) * PK + p])
                                                    : make_double2(0.0, 0.0);
#pragma unroll
            for (int u = 0; u < 4; ++u) s = cadd(s, v[u]);
        }
#pragma unroll
        for (int off = TPT / 2; off > 0; off >>= 1) s = cadd(s, shfl_xor(s, off));
        if (l == 0 && p < PK) {
            out[p] = s;
            rs.final_[p] = s;
        }
    }
    if (threadIdx.x == 0) *rs.counter = 0u;
    __syncthreads();
    return true;
}

// FP32 terms: v[j][r] is real quantity r of this thread's j-th right-hand side,
// a float or a ThreadSum; total r of right-hand side k goes to out[r K + k].x, or
// (CPLX) out[(r / 2) K + k], x for even r and y for odd.  sh: scratch of
// red_floats<T>(NT, LPT * NR) floats, free at the call.  The threads' values go
// through shared memory: GL lanes per total sum those of its row groups, then a
// tree; the block totals lie in rs.partial as (h, m, l, 1), or, where a sum has
// left the FP32 range or is not finite, as an FP64 sum of the same values (its
// two words, 0, 2), and the last block does likewise.
template <class T> struct RedTerm;
template <> struct RedTerm<float> {
    static constexpr int kParts = 1;
    static __device__ __forceinline__ void put(float* at, int, float v) { *at = v; }
    static __device__ __forceinline__ bool over(float) { return false; }
};
template <> struct RedTerm<ThreadSum> {
    static constexpr int kParts = 3;
    static __device__ __forceinline__ void put(float* at, int stride, const ThreadSum& v) {
        at[0] = v.s.h;
        at[stride] = v.s.m;
        at[2 * stride] = v.s.l;
    }
    static __device__ __forceinline__ bool over(const ThreadSum& v) { return !(v.over == 0.0); }
};
template <class T> constexpr int red_floats(int NT, int values) { return NT * values * RedTerm<T>::kParts; }

template <int NR, bool CPLX, int K, int NT, int LPT, class T>
__device__ bool grid_reduce_f32(const T (&v)[LPT][NR], RedScratch rs, double2* out, float* sh) {
    using Term = RedTerm<T>;
    constexpr int P = Term::kParts, TPR = K / LPT, G = NT / TPR, R = NR * K, Q = NT / R;
    constexpr int GL = Q >= 32 ? 32 : Q >= 16 ? 16 : Q >= 8 ? 8 : Q >= 4 ? 4 : Q >= 2 ? 2 : 1;
    constexpr int U = (G + GL - 1) / GL < 4 ? (G + GL - 1) / GL : 4;
    static_assert(K >= LPT && K <= 32 && (K & (K - 1)) == 0 && NT % 32 == 0 && NT % TPR == 0, "launch shape");
    static_assert(Q >= 1 && R <= 2 * kMaxQ * kMaxRhs, "a thread per total, and its place in the scratch");
    __shared__ bool am_last;
    const int warp = threadIdx.x >> 5, p = threadIdx.x / GL, l = threadIdx.x % GL;
    const bool mine = p < R, busy = warp * (32 / GL) < R;
    const int k = p % K, r = p / K;
    bool wide = false;   // this block's totals in FP64
#pragma unroll
    for (int j = 0; j < LPT; ++j)
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            Term::put(sh + (size_t)((j * NR + q) * P) * NT + threadIdx.x, NT, v[j][q]);
            wide |= Term::over(v[j][q]);
        }
    if constexpr (P == 1) __syncthreads();
    else wide = __syncthreads_or(wide) != 0;
    const float* at = sh + (size_t)(((k % LPT) * NR + r) * P) * NT + k / LPT;
    Sum3 s;
    if (busy && !wide) {
        // in rounds, their loads and sums side by side
#pragma unroll 1
        for (int g0 = 0; g0 < G; g0 += U * GL) {
            float a[U * P];
#pragma unroll
            for (int i = 0; i < U; ++i)
#pragma unroll
                for (int u = 0; u < P; ++u) {
                    const int g = g0 + i * GL + l;
                    a[i * P + u] = mine && g < G ? at[u * NT + g * TPR] : 0.0f;
                }
#pragma unroll
            for (int i = 0; i < U * P; ++i) s.add(a[i]);
        }
#pragma unroll
        for (int off = GL / 2; off > 0; off >>= 1) s.add(s.xor_lane(off));
    }
    float4* partial = reinterpret_cast<float4*>(rs.partial);
    auto publish = [&](float4 q) {
        if (mine && l == 0) {
            __stcg(&partial[(size_t)blockIdx.x * R + p], q);
            __threadfence();
        }
    };
    publish(make_float4(s.h, s.m, s.l, 1.0f));
    wide = __syncthreads_or(wide || (mine && !s.finite())) != 0;
    if (wide) {
        double* shd = reinterpret_cast<double*>(sh);
        if constexpr (P == 3) {   // room for a double in a ThreadSum's three floats
#pragma unroll
            for (int j = 0; j < LPT; ++j)
#pragma unroll
                for (int q = 0; q < NR; ++q) shd[(size_t)(j * NR + q) * NT + threadIdx.x] = v[j][q].s.get() + v[j][q].over;
            __syncthreads();
        }
        double d = 0.0;
        if (busy) {
            for (int g = l; mine && g < G; g += GL)
                d += P == 3 ? shd[(size_t)((k % LPT) * NR + r) * NT + k / LPT + g * TPR] : (double)at[g * TPR];
#pragma unroll
            for (int off = GL / 2; off > 0; off >>= 1) d += shfl_xor(d, off);
        }
        publish(make_float4(__int_as_float(__double2hiint(d)), __int_as_float(__double2loint(d)), 0.0f, 2.0f));
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const unsigned t = atomicAdd(rs.counter, 1u);
        am_last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!am_last) return false;
    __threadfence();
    s = Sum3();
    wide = false;
    if (busy) {
#pragma unroll 1
        for (int b0 = 0; b0 < (int)gridDim.x; b0 += 4 * GL) {   // four loads in flight
            float4 q[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int b = b0 + GL * u + l;
                q[u] = mine && b < (int)gridDim.x ? __ldcg(&partial[(size_t)b * R + p])
                                                  : make_float4(0.0f, 0.0f, 0.0f, 1.0f);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (b0 + GL * u >= (int)gridDim.x) break;
                Sum3 o;
                o.h = q[u].x;
                o.m = q[u].y;
                o.l = q[u].z;
                s.add(o);
                wide |= q[u].w != 1.0f;
            }
        }
#pragma unroll
        for (int off = GL / 2; off > 0; off >>= 1) s.add(s.xor_lane(off));
    }
    double total = s.get();
    if (__syncthreads_or(wide || (mine && !s.finite()))) {
        total = 0.0;
        if (busy) {
            for (int b = l; mine && b < (int)gridDim.x; b += GL) {
                const float4 q = __ldcg(&partial[(size_t)b * R + p]);
                total += q.w == 1.0f ? (double)q.x + ((double)q.y + (double)q.z)
                                     : __hiloint2double(__float_as_int(q.x), __float_as_int(q.y));
            }
#pragma unroll
            for (int off = GL / 2; off > 0; off >>= 1) total += shfl_xor(total, off);
        }
    }
    if (mine && l == 0) {
        double2* o = &out[(CPLX ? r / 2 : r) * K + k];
        if (CPLX && (r & 1)) o->y = total;
        else o->x = total;
    }
    if (threadIdx.x == 0) *rs.counter = 0u;
    __syncthreads();
    return true;
}

// The same for complex terms of either precision, acc[j][q]; out[q * K + k].
template <int NQ, int K, int NT, int LPT>
__device__ __forceinline__ bool grid_reduce_multi(const float2 (&acc)[LPT][NQ], RedScratch rs, double2* out, float* sh) {
    float v[LPT][2 * NQ];
#pragma unroll
    for (int j = 0; j < LPT; ++j)
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            v[j][2 * q] = acc[j][q].x;
            v[j][2 * q + 1] = acc[j][q].y;
        }
    return grid_reduce_f32<2 * NQ, true, K, NT, LPT>(v, rs, out, sh);
}
template <int NQ, int K, int NT, int LPT>
__device__ __forceinline__ bool grid_reduce_multi(const double2 (&acc)[LPT][NQ], RedScratch rs, double2* out, float*) {
    static_assert(LPT == 1, "FP64 kernels take one right-hand side a thread");
    return grid_reduce_lanes<NQ, K, NT>(acc[0], rs, out);
}
// floats of scratch that it needs
template <class R, int NQ> constexpr int multi_floats(int NT, int LPT) {
    return sizeof(R) == 4 ? red_floats<float>(NT, LPT * 2 * NQ) : 0;
}

// Blocks of a reducing vector kernel over n elements: one resident wave at
// most and four elements a thread at least, and beyond two blocks per SM (152
// of them) 16 elements a thread: the last block's FP64 walk over the blocks'
// partials (a cycle per pair of adds) costs small vectors more than the extra
// blocks save.
template <class F>
inline int reduce_grid(F* kernel, int cap, long n, int threads = kBlock) {
    const long lo = (n + 4L * threads - 1) / (4L * threads), hi = (n + 16L * threads - 1) / (16L * threads);
    const long b = lo < 304 ? lo : hi < 304 ? 304 : hi;
    const int w = wave_grid(kernel, cap, threads);
    return (int)(b < 1 ? 1 : b < w ? b : w);
}

}  // namespace dev
}  // namespace m3d
