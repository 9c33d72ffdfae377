// spd_capi.cu — C ABI of the GPU sparse SPD solver (ifea_spd_*), shaped like the reference's ISpdSolver
// (Solver/Linear/ISpdSolver.cs:24-41) so a CudssSolver-style P/Invoke backend can bind it directly.
#include <algorithm>
#include <cstring>
#include <exception>
#include <string>
#include <thread>
#include <vector>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "multifrontal.cuh"

// Uploads a large pageable array: threads copy chunks into pinned slots of their own (two each) and send them on, so
// that the copies into pinned memory and over the bus overlap. 78 MB take about 2.8 ms
// (B200, 16 host cores), 7.2 by the driver's own staging of a pageable copy. Below kLeast starting threads takes a good
// part of what it gains (8 MB: 0.7 ms), and memory that is pinned already is copied directly.
class HostUpload {
    // The calling thread's CUDA context, for the threads that copy for it: a host may run this library in a context of its
    // own, and cudaSetDevice() would make the device's primary context current instead.
    struct Context {
        CUcontext ctx = nullptr;
        PFN_cuCtxSetCurrent_v4000 set = nullptr;
        static Context current()
        {
            Context c;
            void *get = nullptr, *set = nullptr;
            cudaDriverEntryPointQueryResult q;
            ifea::cuda_check(cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &get, 4000, cudaEnableDefault, &q), "cuCtxGetCurrent");
            ifea::cuda_check(cudaGetDriverEntryPointByVersion("cuCtxSetCurrent", &set, 4000, cudaEnableDefault, &q), "cuCtxSetCurrent");
            c.set = (PFN_cuCtxSetCurrent_v4000)set;
            if (!get || !set || ((PFN_cuCtxGetCurrent_v4000)get)(&c.ctx) != CUDA_SUCCESS)
                throw ifea::Failure(IFEA_CUDA_ERROR, "no current CUDA context");
            if (!c.ctx) {  // a thread that has made no CUDA call yet: the device's primary context, as for any first call
                int dev = 0;
                ifea::cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
                ifea::cuda_check(cudaSetDevice(dev), "cudaSetDevice");
                if (((PFN_cuCtxGetCurrent_v4000)get)(&c.ctx) != CUDA_SUCCESS || !c.ctx)
                    throw ifea::Failure(IFEA_CUDA_ERROR, "no current CUDA context");
            }
            return c;
        }
        cudaError_t enter() const { return set(ctx) == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue; }
    };

public:
    static constexpr size_t kLeast = 8 << 20;
    ~HostUpload() { release(); }
    void prepare()
    {
        if (buf_) return;
        bool ok = cudaMallocHost((void **)&buf_, kSlots * kChunk) == cudaSuccess;
        for (auto &e : ev_) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
        if (ok) return;
        cudaGetLastError();  // (no slots to be had: arrays go up as pageable copies)
        release();
    }
    void release()
    {
        for (auto &e : ev_) {
            if (e) cudaEventDestroy(e);
            e = nullptr;
        }
        if (buf_) cudaFreeHost(buf_);
        buf_ = nullptr;
    }
    // src may change once this returns
    void run(void *dst, const void *src, size_t bytes, cudaStream_t st)
    {
        cudaPointerAttributes at{};
        const bool pageable = cudaPointerGetAttributes(&at, src) == cudaSuccess && at.type == cudaMemoryTypeUnregistered;
        if (!pageable) cudaGetLastError();
        if (!buf_ || bytes < kLeast || !pageable) {
            ifea::cuda_check(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st), "cudaMemcpyAsync H2D");
            return;
        }
        const Context here = Context::current();
        cudaError_t err[kThreads] = {};
        auto work = [&](int t) {
            cudaError_t e = cudaSuccess;
            int k = 0;
            for (size_t o = t * kChunk; o < bytes && e == cudaSuccess; o += kThreads * kChunk, k++) {
                const int slot = 2 * t + (k & 1);
                const size_t n = std::min(kChunk, bytes - o);
                e = cudaEventSynchronize(ev_[slot]);
                if (e != cudaSuccess) break;
                std::memcpy(buf_ + slot * kChunk, (const char *)src + o, n);
                e = cudaMemcpyAsync((char *)dst + o, buf_ + slot * kChunk, n, cudaMemcpyHostToDevice, st);
                if (e == cudaSuccess) e = cudaEventRecord(ev_[slot], st);
            }
            err[t] = e;
        };
        std::thread th[kThreads];
        for (int t = 1; t < kThreads; t++) {
            try {
                th[t] = std::thread([&, t] {
                    err[t] = here.enter();
                    if (err[t] == cudaSuccess) work(t);
                });
            } catch (const std::exception &) {  // (no thread to be had: its chunks below)
            }
        }
        work(0);
        for (int t = 1; t < kThreads; t++) {
            if (th[t].joinable()) th[t].join();
            else work(t);
        }
        for (cudaError_t e : err) ifea::cuda_check(e, "staged upload");
    }

private:
    static constexpr int kThreads = 4, kSlots = 2 * kThreads;
    static constexpr size_t kChunk = 1 << 20;
    char *buf_ = nullptr;
    cudaEvent_t ev_[kSlots] = {};
};

struct ifea_spd {
    cudaStream_t st = nullptr;
    ifea::MfSolver *s = nullptr;
    ifea::DBuf<double> vals, b, x;
    HostUpload up;
    std::vector<int32_t> col_ptr;
    int n = 0;
    int64_t nnz = 0;
    std::string err, name;
};

template <typename F>
static ifea_status spd_guard(ifea_spd *h, F &&f)
{
    if (!h) return IFEA_INPUT_INVALID;
    try {
        f(*h);
        h->err.clear();
        return IFEA_OK;
    } catch (ifea::Failure &e) {
        h->err = e.what();
        return e.status;
    } catch (std::exception &e) {
        h->err = e.what();
        return IFEA_CUDA_ERROR;
    }
}

extern "C" {

ifea_status ifea_spd_create(ifea_spd **out)
{
    if (!out) return IFEA_INPUT_INVALID;
    *out = nullptr;
    ifea_spd *h = new ifea_spd;
    try {
        ifea::cuda_check(cudaStreamCreateWithFlags(&h->st, cudaStreamNonBlocking), "cudaStreamCreate");
        h->s = new ifea::MfSolver(h->st);
        cudaDeviceProp prop;
        ifea::cuda_check(cudaGetDeviceProperties(&prop, 0), "cudaGetDeviceProperties");
        h->name = std::string("multifrontal sparse Cholesky (GPU · ") + prop.name + ")";
    } catch (ifea::Failure &e) {
        delete h->s;
        if (h->st) cudaStreamDestroy(h->st);
        delete h;
        return e.status;
    }
    *out = h;
    return IFEA_OK;
}

void ifea_spd_destroy(ifea_spd *h)
{
    if (!h) return;
    delete h->s;
    h->vals.release();
    h->b.release();
    h->x.release();
    h->up.release();
    if (h->st) cudaStreamDestroy(h->st);
    delete h;
}

const char *ifea_spd_last_error(const ifea_spd *h) { return h ? h->err.c_str() : "null handle"; }
const char *ifea_spd_name(const ifea_spd *h) { return h ? h->name.c_str() : ""; }

// ISpdSolver.Analyze(n, colPtr, rowIdx): symbolic analysis of a full symmetric CSC pattern.
ifea_status ifea_spd_analyze(ifea_spd *h, int32_t n, const int32_t *col_ptr, const int32_t *row_idx)
{
    if (!col_ptr || !row_idx || n <= 0) return IFEA_INPUT_INVALID;
    return spd_guard(h, [&](ifea_spd &s) {
        s.n = n;
        s.nnz = col_ptr[n];
        s.col_ptr.assign(col_ptr, col_ptr + n + 1);
        s.s->analyze(n, col_ptr, row_idx, 1);
        s.vals.resize(s.nnz);
        s.b.resize(n);
        s.x.resize(n);
        if (sizeof(double) * (size_t)s.nnz >= HostUpload::kLeast) s.up.prepare();
    });
}

// ISpdSolver.Factorize(values): values in the order of the analysed full CSC pattern (host).
ifea_status ifea_spd_factorize(ifea_spd *h, const double *values)
{
    if (!values) return IFEA_INPUT_INVALID;
    return spd_guard(h, [&](ifea_spd &s) {
        if (!s.s->analyzed()) throw ifea::Failure(IFEA_BAD_STATE, "Analyze must be called first.");
        s.up.run(s.vals, values, sizeof(double) * (size_t)s.nnz, s.st);
        s.s->factorize(s.vals);
    });
}

// ISpdSolver.Solve(b, x) (host).
ifea_status ifea_spd_solve(ifea_spd *h, const double *b, double *x)
{
    if (!b || !x) return IFEA_INPUT_INVALID;
    return spd_guard(h, [&](ifea_spd &s) {
        s.b.upload(b, s.n, s.st);
        s.s->solve(s.b, s.x, nullptr);
        s.s->check_finite(s.x);
        s.x.download(x, s.n, s.st);
        ifea::cuda_check(cudaStreamSynchronize(s.st), "cudaStreamSynchronize");
    });
}

int64_t ifea_spd_factor_nonzeros(const ifea_spd *h) { return h && h->s ? h->s->factor_nonzeros() : 0; }

const char *ifea_version(void) { return "ifea-b200 0.1 (sm_100a, FP64 path)"; }

}  // extern "C"
