// extern "C" face of the learned preconditioner's network (include/m3d_gb300.h,
// "Learned preconditioner network"): host arrays in and out, so that the
// tensor-core kernels can be checked against a CPU restatement.  The solver
// uses the same class directly (solver.cu).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstring>
#include <new>
#include <stdexcept>
#include <string>
#include <vector>

#include "m3d_gb300.h"
#include "cuda/learned.cuh"

namespace {

// A device array that is kept between calls and grows as needed.
template <class T>
struct DevBuf {
    T* p = nullptr;
    size_t cap = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { if (p) cudaFree(p); }
    T* get(size_t n) {
        if (n <= cap) return p;
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
        if (cudaMalloc(&p, n * sizeof(T)) != cudaSuccess) {
            cudaGetLastError();
            p = nullptr;
            throw std::bad_alloc();
        }
        cap = n;
        return p;
    }
};

// Results leave through two page-locked pieces of 1 MB: the caller's array is
// as a rule freshly allocated, and a device copy straight into pages that the
// host has never touched is slow (forward pass of 4 x 32^3 voxels, 3 MB out:
// 3.4 ms, 0.53 ms this way); the pieces' host copies overlap the next transfer.
struct Download {
    static constexpr size_t kPiece = size_t(1) << 20;
    char* p = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    Download() = default;
    Download(const Download&) = delete;
    Download& operator=(const Download&) = delete;
    ~Download() {
        if (p) cudaFreeHost(p);
        for (cudaEvent_t e : ev)
            if (e) cudaEventDestroy(e);
    }
    static void ck(cudaError_t e) {
        if (e == cudaSuccess) return;
        cudaGetLastError();
        if (e == cudaErrorMemoryAllocation) throw std::bad_alloc();
        throw std::runtime_error("cnn: output copy failed");
    }
    // dst (host) = src (device) in stream order; complete on return
    void operator()(void* dst, const void* src, size_t bytes, cudaStream_t st) {
        if (!p) ck(cudaMallocHost(&p, 2 * kPiece));
        for (cudaEvent_t& e : ev)
            if (!e) ck(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        const size_t n = (bytes + kPiece - 1) / kPiece;
        const auto len = [&](size_t i) { return i + 1 < n ? kPiece : bytes - i * kPiece; };
        const auto start = [&](size_t i) {
            ck(cudaMemcpyAsync(p + (i & 1) * kPiece, static_cast<const char*>(src) + i * kPiece, len(i),
                               cudaMemcpyDeviceToHost, st));
            ck(cudaEventRecord(ev[i & 1], st));
        };
        for (size_t i = 0; i < n && i < 2; ++i) start(i);
        for (size_t i = 0; i < n; ++i) {
            ck(cudaEventSynchronize(ev[i & 1]));
            std::memcpy(static_cast<char*>(dst) + i * kPiece, p + (i & 1) * kPiece, len(i));
            if (i + 2 < n) start(i + 2);
        }
    }
};

}  // namespace

struct m3d_cnn {
    m3d::learn::Cnn* net = nullptr;
    std::string err;
    DevBuf<float> x, dy, dx;
    Download download;
};

namespace {

template <class F>
int cnn_guarded(m3d_cnn* h, F&& f) {
    if (!h || !h->net) return M3D_ERR_ARG;
    // whatever ends the call, no copy from the caller's arrays is left running
    struct Drain {
        m3d::learn::Cnn& net;
        bool armed;
        ~Drain() { if (armed) cudaStreamSynchronize(net.stream()); }
    } drain{*h->net, true};
    try {
        f(*h->net);
        drain.armed = false;
        return M3D_OK;
    } catch (const std::bad_alloc&) {
        cudaGetLastError();
        h->err = "allocation failed";
        return M3D_ERR_OOM;
    } catch (const std::invalid_argument& e) {
        h->err = e.what();
        return M3D_ERR_ARG;
    } catch (const std::exception& e) {
        h->err = e.what();
        return M3D_ERR_CUDA;
    }
}

// host FP32 array -> kept device array, in the network's stream
float* upload(m3d::learn::Cnn& net, DevBuf<float>& buf, const float* x, size_t n) {
    float* d = buf.get(n);
    if (cudaMemcpyAsync(d, x, n * sizeof(float), cudaMemcpyHostToDevice, net.stream()) != cudaSuccess) {
        cudaGetLastError();
        throw std::runtime_error("cnn: upload failed");
    }
    return d;
}

void check_flag(m3d::learn::Cnn& net) {
    if (net.error_flag()) throw std::runtime_error("cnn: a tensor-core kernel's barrier wait timed out");
}

}  // namespace

extern "C" int m3d_cnn_create(int device, int layers, int c_in, int hidden, int c_out, unsigned seed, m3d_cnn** out) {
    if (!out) return M3D_ERR_ARG;
    *out = nullptr;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
        cudaGetLastError();
        return M3D_ERR_NO_DEVICE;
    }
    try {
        auto* h = new m3d_cnn();
        h->net = new m3d::learn::Cnn(device, layers, c_in, hidden, c_out, seed);
        *out = h;
        return M3D_OK;
    } catch (const std::invalid_argument&) {
        return M3D_ERR_ARG;
    } catch (const std::bad_alloc&) {
        cudaGetLastError();
        return M3D_ERR_OOM;
    } catch (...) {
        cudaGetLastError();
        return M3D_ERR_CUDA;
    }
}

extern "C" void m3d_cnn_destroy(m3d_cnn* h) {
    if (!h) return;
    delete h->net;
    delete h;
}

extern "C" const char* m3d_cnn_last_error(const m3d_cnn* h) { return h ? h->err.c_str() : "null handle"; }

extern "C" int m3d_cnn_get_weights(m3d_cnn* h, float* w, float* b) {
    if (!w || !b) return M3D_ERR_ARG;
    return cnn_guarded(h, [&](m3d::learn::Cnn& net) { net.get_weights(w, b); });
}

extern "C" int m3d_cnn_set_weights(m3d_cnn* h, const float* w, const float* b) {
    if (!w || !b) return M3D_ERR_ARG;
    return cnn_guarded(h, [&](m3d::learn::Cnn& net) { net.set_weights(w, b); });
}

extern "C" int m3d_cnn_forward(m3d_cnn* h, const float* x, int n, int D, int H, int W, float* y) {
    if (!x || !y || n < 1) return M3D_ERR_ARG;
    return cnn_guarded(h, [&](m3d::learn::Cnn& net) {
        net.ensure(n, D, H, W);
        const size_t G = (size_t)n * D * H * W;
        net.pack_input(upload(net, h->x, x, G * net.c_in()), n);
        const float* o = net.forward(n);
        check_flag(net);
        h->download(y, o, G * net.c_out() * sizeof(float), net.stream());
    });
}

extern "C" int m3d_cnn_backward(m3d_cnn* h, const float* x, const float* dy, int n, int D, int H, int W, float* dw,
                                float* db, float* dx) {
    if (!x || !dy || !dw || !db || n < 1) return M3D_ERR_ARG;
    return cnn_guarded(h, [&](m3d::learn::Cnn& net) {
        net.ensure(n, D, H, W);
        const size_t G = (size_t)n * D * H * W;
        net.pack_input(upload(net, h->x, x, G * net.c_in()), n);
        net.forward(n);
        float* d_dx = dx ? h->dx.get(G * net.c_in()) : nullptr;
        net.backward(n, upload(net, h->dy, dy, G * net.c_out()), d_dx);
        check_flag(net);
        const size_t L = (size_t)net.layers();
        h->download(dw, net.grad_w(), L * m3d::learn::kWElems * sizeof(float), net.stream());
        h->download(db, net.grad_b(), L * m3d::learn::kCh * sizeof(float), net.stream());
        if (dx) h->download(dx, d_dx, G * net.c_in() * sizeof(float), net.stream());
    });
}

extern "C" int m3d_cnn_train_step(m3d_cnn* h, const float* x, const float* target, int n, int D, int H, int W,
                                  float lr, double* loss) {
    if (!x || !target || n < 1 || !(lr > 0.0f)) return M3D_ERR_ARG;
    return cnn_guarded(h, [&](m3d::learn::Cnn& net) {
        net.ensure(n, D, H, W);
        const size_t G = (size_t)n * D * H * W;
        net.pack_input(upload(net, h->x, x, G * net.c_in()), n);
        const float* d_t = upload(net, h->dy, target, G * net.c_out());
        net.forward(n);
        const double l = net.loss_backward(n, d_t);
        net.adam_step(lr);
        check_flag(net);
        if (loss) *loss = l;
    });
}
