// Batched Hermitian dot kernel (see dot.cuh).
#include "dot.cuh"

namespace m3d {
namespace dev {

namespace {

// Thread t of the grid owns the (row, rhs) pairs t, t + stride, ...; the grid
// stride is a multiple of 256 and hence of K, so lane l always accumulates
// right-hand side l % K, which is what grid_reduce_lanes expects.  Bound by the
// FP64 units (2 per clock and SM: four fused multiply-adds a pair take 187 us
// for 27 M pairs, the loads 129 us): four FMAs a pair instead of products and
// adds apart (six instructions), eight loads in flight: 336 -> 201 us.
__device__ __forceinline__ void dot_add(double2& s, double2 a, double2 b) {
    s.x = fma(a.x, b.x, fma(a.y, b.y, s.x));
    s.y = fma(a.x, b.y, fma(-a.y, b.x, s.y));
}

template <int K>
__global__ void __launch_bounds__(kBlock) k_dot_batched(const double2* __restrict__ x,
                                                        const double2* __restrict__ y, long long n,
                                                        RedScratch rs, double2* __restrict__ out) {
    __shared__ double2 tot[K];
    double2 part[4] = {};   // one running sum per load in flight: short chains, small errors
    const long long total = n * K;
    const long long stride = (long long)gridDim.x * blockDim.x;
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    for (; t + 3 * stride < total; t += 4 * stride) {
        double2 a[4], b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            a[u] = __ldg(x + t + u * stride);
            b[u] = __ldg(y + t + u * stride);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) dot_add(part[u], a[u], b[u]);
    }
    for (int u = 0; t < total; t += stride, ++u) {   // three at most
        const double2 a = __ldg(x + t), b = __ldg(y + t);
        dot_add(u == 0 ? part[0] : u == 1 ? part[1] : part[2], a, b);
    }
    double2 acc[1] = {cadd(cadd(part[0], part[1]), cadd(part[2], part[3]))};
    if (grid_reduce_lanes<1, K>(acc, rs, tot) && threadIdx.x < K) out[threadIdx.x] = tot[threadIdx.x];
}

}  // namespace

int dot_blocks(long long n, int K, int cap) {
    const long long work = n * (long long)K;
    // two pairs a thread beyond 64 blocks, two blocks on each of 152 SMs at most:
    // four chains a thread keep the FP64 units busy, and every further block is
    // one more partial for the last one to sum (27 M pairs: 289 us with 152
    // blocks, 205 with 304, 217 with 456, 227 with 912; 1 M pairs: 30, 32, 35, 50)
    const long long one = (work + kBlock - 1) / kBlock, two = (work + 2 * kBlock - 1) / (2 * kBlock);
    long long b = one < 64 ? one : two < 64 ? 64 : two;
    if (b < 1) b = 1;
    if (b > 304) b = 304;
    if (b > cap) b = cap;
    return (int)b;
}

cudaError_t launch_dot_batched(const double2* x, const double2* y, long long n, int K, int cap, RedScratch rs,
                               double2* out, cudaStream_t st) {
    const int g = dot_blocks(n, K, cap);
    switch (K) {
        case 1: k_dot_batched<1><<<g, kBlock, 0, st>>>(x, y, n, rs, out); break;
        case 2: k_dot_batched<2><<<g, kBlock, 0, st>>>(x, y, n, rs, out); break;
        case 4: k_dot_batched<4><<<g, kBlock, 0, st>>>(x, y, n, rs, out); break;
        case 8: k_dot_batched<8><<<g, kBlock, 0, st>>>(x, y, n, rs, out); break;
        case 16: k_dot_batched<16><<<g, kBlock, 0, st>>>(x, y, n, rs, out); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace dev
}  // namespace m3d
