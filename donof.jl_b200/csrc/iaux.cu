// The RI tensor on the device from the two- and three-centre integrals:
//   b[m, n, l] = sum_k I[m, n, k] G^{-1/2}[k, l]
// (Iaux, src/integrals.jl:68-91; GPU form Iaux_gpu, ext/DoNOFGPUExt.jl:9-33):
// eigen-decomposition of Symmetric(G) (upper triangle), inverse square roots of
// the eigenvalues with negative ones set to zero, G^{-1/2} = V diag(s) V^T, and
// the contraction as one GEMM of I seen as an (nbf^2 x naux) column-major
// matrix, whose product is b in the layout of the rest of the library.
//
// The symmetric eigensolver is the library's own parallel Jacobi kernel
// (eigh.cu); the two products run on the library's FP64 tensor-core GEMM.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <thread>
#include <vector>

#include "kernels.cuh"

namespace donof {

namespace {

// Vs[i + n j] = V[i + n j] s_j,  VT[j + n i] = V[i + n j];  s_j = 1/sqrt(w_j), 0 for w_j < 0
// (V's leading dimension is ldv, the others' n)
__global__ void gmsqrt_factors_kernel(const double* __restrict__ V, const double* __restrict__ w, int n, int ldv,
                                      double* __restrict__ Vs, double* __restrict__ VT) {
    const long long total = (long long)n * n;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(idx % n), j = (int)(idx / n);
        const double s = (w[j] < 0.0) ? 0.0 : 1.0 / sqrt(w[j]);
        const double v = V[i + (long long)ldv * j];
        Vs[idx] = v * s;
        VT[j + (long long)n * i] = v;
    }
}

constexpr size_t SMALL_COPY = size_t(256) << 10;  // bytes of I that cross on the call's own stream

// Copies `bytes` of host memory to dst on the stream `st`, returning when they have
// landed.  Memory that CUDA knows (page-locked, managed, on the device too) goes in one
// copy; other memory through the context's page-locked buffer in chunks, each host thread filling two slots of its own in
// turn: one thread copies about 10 GB/s, the DMA takes five times that.
int upload(donof_ctx* ctx, cudaStream_t st, void* dst, const void* src, size_t bytes) {
    constexpr size_t CHUNK = size_t(4) << 20;
    constexpr int MAX_THREADS = 8;
    const size_t chunks = (bytes + CHUNK - 1) / CHUNK;
    cudaPointerAttributes at{};
    const bool known = cudaPointerGetAttributes(&at, src) == cudaSuccess && at.type != cudaMemoryTypeUnregistered;
    cudaGetLastError();
    int nt = (int)std::min<size_t>(std::min<size_t>(MAX_THREADS, std::thread::hardware_concurrency() / 2), chunks / 2);
    const size_t room = 2 * CHUNK * (size_t)std::max(nt, 0);
    if (!known && nt > 1) {
        if (ctx->hstage_busy) {  // an earlier call that failed may still be copying through it
            DONOF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            ctx->hstage_busy = false;
        }
        if (ctx->hstage_bytes < room) {
            if (ctx->hstage) cudaFreeHost(ctx->hstage);
            ctx->hstage = nullptr;
            ctx->hstage_bytes = 0;
            if (cudaMallocHost(&ctx->hstage, room) == cudaSuccess) {
                ctx->hstage_bytes = room;
            } else {
                cudaGetLastError();
                ctx->hstage = nullptr;
            }
        }
    }
    if (known || nt <= 1 || ctx->hstage_bytes < room) {
        DONOF_CUDA(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st));
        DONOF_CUDA(ctx, cudaStreamSynchronize(st));
        return DONOF_OK;
    }
    std::atomic<int> err{cudaSuccess};
    auto work = [&](int t) {
        cudaError_t e = cudaSetDevice(ctx->device);
        cudaEvent_t ev[2] = {nullptr, nullptr};
        for (int k = 0; k < 2 && e == cudaSuccess; ++k) e = cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming);
        char* slots = static_cast<char*>(ctx->hstage) + 2 * CHUNK * (size_t)t;
        int use = 0;
        for (size_t c = (size_t)t; c < chunks && e == cudaSuccess && err.load() == cudaSuccess; c += (size_t)nt, ++use) {
            const int k = use & 1;
            const size_t off = c * CHUNK, n = std::min(CHUNK, bytes - off);
            if (use >= 2) e = cudaEventSynchronize(ev[k]);
            if (e != cudaSuccess) break;
            memcpy(slots + CHUNK * k, static_cast<const char*>(src) + off, n);
            e = cudaMemcpyAsync(static_cast<char*>(dst) + off, slots + CHUNK * k, n, cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess) e = cudaEventRecord(ev[k], st);
        }
        for (int k = 0; k < 2; ++k)
            if (ev[k]) cudaEventDestroy(ev[k]);
        if (e != cudaSuccess) err.store(e);
    };
    int started = 0;
    {
        std::vector<std::thread> pool;
        try {
            for (; started < nt - 1; ++started) pool.emplace_back(work, started);
            work(nt - 1);
        } catch (...) {  // no further thread to be had: their chunks are copied below
        }
        for (auto& t : pool) t.join();
    }
    const cudaError_t e = cudaStreamSynchronize(st);
    if (err.load() == cudaSuccess && e != cudaSuccess) err.store(e);
    if (err.load() != cudaSuccess) {
        set_error(ctx, "copy to the device: %s", cudaGetErrorString((cudaError_t)err.load()));
        return DONOF_ERR_CUDA;
    }
    if (started < nt - 1) {
        DONOF_CUDA(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st));
        DONOF_CUDA(ctx, cudaStreamSynchronize(st));
    }
    return DONOF_OK;
}

struct DeviceScratch {
    void* p[16] = {};
    int n = 0;
    donof_ctx* ctx;
    explicit DeviceScratch(donof_ctx* c) : ctx(c) {}
    template <class T>
    int alloc(T** out, size_t count) {
        if (n >= 16) {
            set_error(ctx, "Iaux scratch: too many buffers");
            return DONOF_ERR_STATE;
        }
        void* d = nullptr;
        DONOF_CHECK(dev_alloc(ctx, &d, sizeof(T) * count));
        p[n++] = d;
        *out = static_cast<T*>(d);
        return DONOF_OK;
    }
    ~DeviceScratch() {  // stream-ordered after the work that used the scratch
        for (int i = 0; i < n; ++i) dev_free(ctx, p[i]);
    }
};

}  // namespace

int iaux_f64(donof_ctx* ctx, cudaStream_t st, const double* G_host, const double* I_host, int nbf, int naux,
             double* b, DevBuf* part) {
    const size_t nn = (size_t)nbf * nbf, na2 = (size_t)naux * naux;
    const int npad = eigh_padded(naux);
    DeviceScratch s(ctx);
    double *dI = nullptr, *dG = nullptr, *dw = nullptr, *dVs = nullptr, *dVT = nullptr, *dGm = nullptr,
           *dA = nullptr, *dV = nullptr;
    unsigned char* escr = nullptr;
    DONOF_CHECK(s.alloc(&dI, nn * naux));
    DONOF_CHECK(s.alloc(&dG, na2));
    DONOF_CHECK(s.alloc(&dw, (size_t)naux));
    DONOF_CHECK(s.alloc(&dVs, na2));
    DONOF_CHECK(s.alloc(&dVT, na2));
    DONOF_CHECK(s.alloc(&dGm, na2));
    DONOF_CHECK(s.alloc(&dA, (size_t)npad * npad));
    DONOF_CHECK(s.alloc(&dV, (size_t)npad * npad));
    DONOF_CHECK(s.alloc(&escr, eigh_scratch_bytes(naux)));
    DONOF_CUDA(ctx, cudaMemcpyAsync(dG, G_host, sizeof(double) * na2, cudaMemcpyHostToDevice, st));
    // eigen-decomposition of Symmetric(G) (its upper triangle)
    // I crosses on a stream of its own meanwhile (8 waters: 151 MB, 14 ms by one host
    // thread behind the solver, 4 ms by eight beside it; the solver takes 10 ms), but for
    // an I that costs less than the stream's events and synchronisations (a call at nbf =
    // 24, naux = 1: 141 us with them, 110 without)
    const size_t ibytes = sizeof(double) * nn * naux;
    const bool beside = ibytes > SMALL_COPY;
    if (beside) {
        if (!ctx->aux_stream) DONOF_CUDA(ctx, cudaStreamCreateWithFlags(&ctx->aux_stream, cudaStreamNonBlocking));
        cudaEvent_t ready = nullptr;  // dI's allocation is ordered on st
        DONOF_CUDA(ctx, cudaEventCreateWithFlags(&ready, cudaEventDisableTiming));
        cudaError_t e = cudaEventRecord(ready, st);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(ctx->aux_stream, ready, 0);
        cudaEventDestroy(ready);
        DONOF_CUDA(ctx, e);
    } else {
        DONOF_CUDA(ctx, cudaMemcpyAsync(dI, I_host, ibytes, cudaMemcpyHostToDevice, st));
    }
    DONOF_CHECK(eigh_jacobi(ctx, st, dG, naux, dA, dV, dw, escr));
    const int copied = beside ? upload(ctx, ctx->aux_stream, dI, I_host, ibytes) : DONOF_OK;
    const int solved = eigh_finish(ctx, st, escr);
    DONOF_CHECK(copied);
    DONOF_CHECK(solved);
    {
        long long blocks = ((long long)na2 + 255) / 256;
        if (blocks > 8LL * ctx->sm_count) blocks = 8LL * ctx->sm_count;
        gmsqrt_factors_kernel<<<(int)blocks, 256, 0, st>>>(dV, dw, naux, npad, dVs, dVT); count_launch();
        DONOF_CUDA(ctx, cudaGetLastError());
    }
    // G^{-1/2} = Vs V^T (A: Vs, M-contiguous; B: V^T stored K-contiguous)
    DONOF_CHECK(gemm_f64_auto(ctx, st, false, true, naux, naux, naux, dVs, naux, dVT, naux, dGm, naux, 1.0, 0.0,
                              part));
    // b = I G^{-1/2}: I as an (nbf^2 x naux) column-major matrix
    DONOF_CHECK(gemm_f64_auto(ctx, st, false, true, (int)nn, naux, naux, dI, (long long)nn, dGm, naux, b,
                              (long long)nn, 1.0, 0.0, part));
    DONOF_CUDA(ctx, cudaStreamSynchronize(st));  // the scratch is freed on return
    return DONOF_OK;
}

}  // namespace donof
