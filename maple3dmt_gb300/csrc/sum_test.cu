// Test hook: the grid reductions of FP32 terms (cuda/common.cuh) on given values.
#include <cuda_runtime.h>

#include <new>

#include "m3d_gb300.h"
#include "cuda/common.cuh"

namespace {

using namespace m3d::dev;

constexpr int kNT = 512, kBlocks = 304;

// MANY: each thread sums the values of its right-hand sides from a few blocks
// (as the divergence correction's PCG does); else a value a thread.
template <int K, bool MANY>
__global__ void __launch_bounds__(kNT) k_sum(const float4* __restrict__ v, long n, RedScratch rs, double2* result) {
    __shared__ double2 out[2 * K];
    const long i0 = (long)blockIdx.x * kNT + threadIdx.x, stride = (long)gridDim.x * kNT, m = n * (K / 2);
    bool last;
    if constexpr (MANY) {
        __shared__ __align__(8) float sh[red_floats<ThreadSum>(kNT, 4)];
        ThreadSum acc[2][2];
        for (long i = i0; i < m; i += stride) {
            const float4 q = v[i];
            if (ThreadSum::small(fmaxf(fmaxf(fabsf(q.x), fabsf(q.y)), fmaxf(fabsf(q.z), fabsf(q.w))))) {
                acc[0][0].s.add(q.x);
                acc[0][1].s.add(q.y);
                acc[1][0].s.add(q.z);
                acc[1][1].s.add(q.w);
            } else {
                acc[0][0].add_large(q.x);
                acc[0][1].add_large(q.y);
                acc[1][0].add_large(q.z);
                acc[1][1].add_large(q.w);
            }
        }
        last = grid_reduce_f32<2, true, K, kNT, 2>(acc, rs, out, sh);
    } else {
        __shared__ float sh[red_floats<float>(kNT, 4)];
        const float4 q = i0 < m ? v[i0] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const float2 acc[2][1] = {{make_float2(q.x, q.y)}, {make_float2(q.z, q.w)}};
        last = grid_reduce_multi<1, K, kNT, 2>(acc, rs, out, sh);
    }
    if (last && threadIdx.x < K) result[threadIdx.x] = out[threadIdx.x];
}

struct Mem {
    void* p = nullptr;
    ~Mem() { if (p) cudaFree(p); }
    void* get(size_t n) {
        if (cudaMalloc(&p, n) != cudaSuccess) throw std::bad_alloc();
        return p;
    }
};

}  // namespace

extern "C" int m3d_test_sum_f32(const float* v, long long n, int K, int many, double* out) {
    if (!v || !out || n < 1 || (!many && n * (K / 2) > (long long)kNT * kBlocks)) return M3D_ERR_ARG;
    try {
        Mem dv, part, fin, cnt, res;
        const size_t bytes = sizeof(float) * 2 * (size_t)n * K;
        float4* d = (float4*)dv.get(bytes);
        RedScratch rs{(double2*)part.get(sizeof(double2) * 2 * kMaxQ * kMaxRhs * kBlocks),
                      (double2*)fin.get(sizeof(double2) * kMaxQ * kMaxRhs), (unsigned*)cnt.get(sizeof(unsigned)), kBlocks};
        double2* r = (double2*)res.get(sizeof(double2) * kMaxRhs);
        cudaMemset(cnt.p, 0, sizeof(unsigned));
        cudaMemcpy(d, v, bytes, cudaMemcpyHostToDevice);
        const long m = (long)n * (K / 2);
        const int grid = many ? 3 : (int)((m + kNT - 1) / kNT);
        switch (2 * K + (many ? 1 : 0)) {
            case 4: k_sum<2, false><<<grid, kNT>>>(d, n, rs, r); break;
            case 5: k_sum<2, true><<<grid, kNT>>>(d, n, rs, r); break;
            case 8: k_sum<4, false><<<grid, kNT>>>(d, n, rs, r); break;
            case 9: k_sum<4, true><<<grid, kNT>>>(d, n, rs, r); break;
            case 16: k_sum<8, false><<<grid, kNT>>>(d, n, rs, r); break;
            case 17: k_sum<8, true><<<grid, kNT>>>(d, n, rs, r); break;
            case 32: k_sum<16, false><<<grid, kNT>>>(d, n, rs, r); break;
            case 33: k_sum<16, true><<<grid, kNT>>>(d, n, rs, r); break;
            default: return M3D_ERR_ARG;
        }
        if (cudaGetLastError() != cudaSuccess) return M3D_ERR_CUDA;
        if (cudaMemcpy(out, r, sizeof(double2) * K, cudaMemcpyDeviceToHost) != cudaSuccess) return M3D_ERR_CUDA;
    } catch (const std::bad_alloc&) {
        cudaGetLastError();
        return M3D_ERR_OOM;
    }
    return M3D_OK;
}
