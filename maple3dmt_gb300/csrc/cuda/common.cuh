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

// A complex sum in the making, 16 bytes: FP64 for FP64 terms; for FP32 terms
// two floats per part (Knuth's error-free sum of the high parts, 48 bits
// kept).  An FP64 add holds a warp's pipe for 16 cycles on this GPU and a chain
// of them is slow: summing lanes, warps and blocks in FP64 was 10 to 25 us of
// every reducing FP32 kernel.
template <class R> struct Sum;
template <> struct Sum<double> {
    double2 v;
    __device__ __forceinline__ void set(double2 a) { v = a; }
    __device__ __forceinline__ void add(const Sum& o) { v = cadd(v, o.v); }
    __device__ __forceinline__ Sum xor_lane(int m) const { return {shfl_xor(v, m)}; }
    __device__ __forceinline__ double2 get() const { return v; }
};
template <> struct Sum<float> {
    float4 v;   // x high, x low, y high, y low
    __device__ __forceinline__ void set(float2 a) { v = make_float4(a.x, 0.0f, a.y, 0.0f); }
    static __device__ __forceinline__ void add1(float& h, float& l, float h2, float l2) {
        const float s = __fadd_rn(h, h2), b = __fsub_rn(s, h);
        float e = __fadd_rn(__fsub_rn(h, __fsub_rn(s, b)), __fsub_rn(h2, b));
        e = __fadd_rn(e, __fadd_rn(l, l2));
        h = __fadd_rn(s, e);
        l = __fsub_rn(e, __fsub_rn(h, s));
    }
    __device__ __forceinline__ void add(const Sum& o) {
        add1(v.x, v.y, o.v.x, o.v.y);
        add1(v.z, v.w, o.v.z, o.v.w);
    }
    __device__ __forceinline__ Sum xor_lane(int m) const {
        return {make_float4(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m),
                            __shfl_xor_sync(0xffffffffu, v.z, m), __shfl_xor_sync(0xffffffffu, v.w, m))};
    }
    __device__ __forceinline__ void add_real(float a) { add1(v.x, v.y, a, 0.0f); }
    __device__ __forceinline__ double2 get() const {
        return make_double2((double)v.x + (double)v.y, (double)v.z + (double)v.w);
    }
};

// Dependent launches.  A kernel launched by launch_dep may start while its
// predecessor in the stream still runs: its blocks are scheduled and whatever
// no kernel writes (matrix copies, index arrays, barriers) is under way when
// the predecessor ends, and dep_wait() returns then, with all of the
// predecessor's writes visible.  The small grids' and the small meshes'
// kernels run for 5-30 us, of which the way from one launch to the next was 1
// to 2: three frequencies and gradient on 149 k edges 40.5 -> 35.8 ms, one
// frequency on 17 k edges 11.2 -> 9.4 ms.  Rules:
//  * a kernel launched so calls dep_wait() before its first access to anything
//    that a kernel of the chain writes, and every block calls it;
//  * such data is not read through `const __restrict__` pointers or __ldg (the
//    read-only path is not ordered behind the wait);
//  * what is read before the wait was complete when the chain's first, plain
//    launch started: a plain launch waits for all work before it.
// dep_begin() is dep_trigger() (let the successor start) and dep_wait(); both
// do nothing under a plain launch.
__device__ __forceinline__ void dep_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_begin() {
    dep_trigger();
    dep_wait();
}

// Adds the attribute of a dependent launch, if the stream is not being captured.
inline void dep_attr(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at) {
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

// Scratch for grid reductions: partial[block][kMaxQ * kMaxRhs] and a counter
// that the last block resets.
struct RedScratch {
    double2* partial;
    double2* final_;      // [kMaxQ * kMaxRhs], result of the last reduction
    unsigned int* counter;
    int max_blocks;
};

// Grid reduction for kernels whose lane l always works on the same right-hand
// sides: LPT neighbouring ones per thread, LPT (l % (K / LPT)) and the next
// (K and LPT powers of two, whole warps); acc[j][q] is quantity q of the j-th
// of them in the kernel's working precision.  Shuffle trees over the lanes that
// share a right-hand side, then over the block's warps, then, in the last block
// to arrive, over the blocks, all totals side by side: every step in a fixed
// order, so the result is deterministic for a fixed launch shape.  Returns true
// in the last block, where out[q * K + k] (shared, NQ*K entries) holds the
// totals.
template <int NQ, int K, int NT, int LPT, class S>
__device__ bool grid_reduce_sums(const S (&acc)[LPT][NQ], RedScratch rs, double2* out) {
    static_assert(K >= LPT && K <= 32 && (K & (K - 1)) == 0, "K must be a power of two <= 32");
    static_assert(NT % 32 == 0 && NT >= 32 && NT <= 1024, "block size must be whole warps");
    static_assert(sizeof(S) == sizeof(double2), "partials are 16 bytes");
    constexpr int PK = NQ * K;
    constexpr int NW = NT / 32;
    __shared__ S sm[NW][PK];
    __shared__ bool am_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < LPT; ++j)
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            S s = acc[j][q];
#pragma unroll
            for (int off = 16; off >= K / LPT; off >>= 1) s.add(s.xor_lane(off));
            if (lane < K / LPT) sm[warp][q * K + lane * LPT + j] = s;
        }
    __syncthreads();
    S zero{};
    S* partial = reinterpret_cast<S*>(rs.partial);
    // GW lanes per total, one for each warp of the block
    constexpr int GW = NW <= 1 ? 1 : NW <= 2 ? 2 : NW <= 4 ? 4 : NW <= 8 ? 8 : NW <= 16 ? 16 : 32;
#pragma unroll
    for (int p0 = 0; p0 < PK; p0 += NT / GW) {
        const int p = p0 + threadIdx.x / GW, w = threadIdx.x % GW;
        if (p0 + warp * (32 / GW) >= PK) break;   // idle warps would add zeros, 16 cycles an FP64 add
        S s = w < NW && p < PK ? sm[w][p] : zero;
#pragma unroll
        for (int off = GW / 2; off > 0; off >>= 1) s.add(s.xor_lane(off));
        if (w == 0 && p < PK) {
            __stcg(reinterpret_cast<double2*>(&partial[(size_t)blockIdx.x * PK + p]), *reinterpret_cast<double2*>(&s));
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
        S s = zero;
        for (int b = l; p < PK && b < (int)gridDim.x; b += 4 * TPT) {   // four loads in flight
            double2 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                v[u] = b + TPT * u < (int)gridDim.x
                           ? __ldcg(reinterpret_cast<const double2*>(&partial[(size_t)(b + TPT * u) * PK + p]))
                           : make_double2(0.0, 0.0);
#pragma unroll
            for (int u = 0; u < 4; ++u) s.add(*reinterpret_cast<const S*>(&v[u]));
        }
#pragma unroll
        for (int off = TPT / 2; off > 0; off >>= 1) s.add(s.xor_lane(off));
        if (l == 0 && p < PK) {
            const double2 t = s.get();
            out[p] = t;
            rs.final_[p] = t;
        }
    }
    if (threadIdx.x == 0) *rs.counter = 0u;
    __syncthreads();
    return true;
}

template <int NQ, int K, int NT, int LPT, class C>
__device__ __forceinline__ bool grid_reduce_multi(const C (&acc)[LPT][NQ], RedScratch rs, double2* out) {
    Sum<decltype(C{}.x)> s[LPT][NQ];
#pragma unroll
    for (int j = 0; j < LPT; ++j)
#pragma unroll
        for (int q = 0; q < NQ; ++q) s[j][q].set(acc[j][q]);
    return grid_reduce_sums<NQ, K, NT, LPT>(s, rs, out);
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

template <int NQ, int K, int NT = kBlock>
__device__ __forceinline__ bool grid_reduce_lanes(double2 (&acc)[NQ], RedScratch rs, double2* out) {
    return grid_reduce_multi<NQ, K, NT, 1>(*reinterpret_cast<const double2(*)[1][NQ]>(&acc), rs, out);
}

}  // namespace dev
}  // namespace m3d
