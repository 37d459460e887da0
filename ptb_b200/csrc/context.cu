// Context lifecycle, error plumbing and scratch buffers of libptbgpu.
#include <algorithm>
#include <cstring>
#include <mutex>

#include "common.cuh"

namespace ptb {

[[noreturn]] void fail(int code, const char* fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    throw Error{code, std::string(buf)};
}

void DevBuf::reserve(size_t nbytes) {
    if (nbytes <= bytes) return;
    release();
    nbytes = (nbytes + 255) & ~size_t(255);
    cudaError_t e = cudaMalloc(&ptr, nbytes);
    if (e == cudaErrorMemoryAllocation) {   // the blocks kept between calls make room
        (void)cudaGetLastError();
        WorkPool::trim_all();
        e = cudaMalloc(&ptr, nbytes);
    }
    if (e != cudaSuccess) {
        ptr = nullptr;
        bytes = 0;
        (void)cudaGetLastError();
        fail(PTBGPU_ENOMEM, "cudaMalloc(%zu) failed: %s", nbytes, cudaGetErrorString(e));
    }
    bytes = nbytes;
}

void DevBuf::release() {
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    bytes = 0;
}

// Free blocks of one context; every pool of the process is in the registry so
// that an allocation that fails on one context can have the others' unused blocks
// freed.  The registry's lock is taken before a pool's.
struct WorkPool::Impl {
    struct Block {
        void* ptr;
        size_t bytes;
    };
    std::mutex mu;
    std::vector<Block> free_blocks;   // in the order they were given back
    size_t kept = 0;
    size_t limit = 0;                 // bytes kept unused at most (set at the first block)
    bool scarce = false;              // less than half of the device was free at the last large allocation
};

namespace {

struct PoolRegistry {
    std::mutex mu;
    std::vector<WorkPool*> pools;
};
PoolRegistry& pool_registry() {
    static PoolRegistry* r = new PoolRegistry();   // outlives the contexts of late destructors
    return *r;
}

// Sizes are rounded up by up to 1/16, so that calls on systems of about the same size find
// each other's blocks; large ones only while more than half of the device is free, beyond
// which a block has the size asked for (multiples of 256 bytes), as the largest calls
// need it.
constexpr size_t kLargeBlock = size_t(64) << 20;
size_t work_class(size_t nbytes, bool scarce) {
    size_t step = 256;
    while (!scarce && step * 32 < nbytes) step *= 2;
    return (nbytes + step - 1) / step * step;
}
bool memory_scarce() {
    size_t free_b = 0, total_b = 0;
    return cudaMemGetInfo(&free_b, &total_b) == cudaSuccess && free_b < total_b / 2;
}

}  // namespace

WorkPool::WorkPool() : im_(new Impl()) {
    PoolRegistry& r = pool_registry();
    std::lock_guard<std::mutex> lock(r.mu);
    r.pools.push_back(this);
}

WorkPool::~WorkPool() {
    PoolRegistry& r = pool_registry();
    {
        std::lock_guard<std::mutex> lock(r.mu);
        r.pools.erase(std::remove(r.pools.begin(), r.pools.end(), this), r.pools.end());
    }
    trim();
}

void WorkPool::trim() {
    std::vector<Impl::Block> gone;
    {
        std::lock_guard<std::mutex> lock(im_->mu);
        gone.swap(im_->free_blocks);
        im_->kept = 0;
    }
    for (const Impl::Block& b : gone) cudaFree(b.ptr);
}

void WorkPool::trim_all() {
    PoolRegistry& r = pool_registry();
    std::lock_guard<std::mutex> lock(r.mu);
    for (WorkPool* p : r.pools) p->trim();
}

void* WorkPool::take(size_t nbytes, size_t* got) {
    const size_t want = work_class(std::max<size_t>(nbytes, 1), true);
    {
        std::lock_guard<std::mutex> lock(im_->mu);
        size_t best = im_->free_blocks.size();
        for (size_t i = 0; i < im_->free_blocks.size(); ++i) {
            const size_t b = im_->free_blocks[i].bytes;
            if (b >= want && b <= want + want / 2 &&
                (best == im_->free_blocks.size() || b < im_->free_blocks[best].bytes))
                best = i;
        }
        // a large block for a much smaller array only while memory is plenty (as the last
        // allocation of a large one found it: asking takes 70 us)
        if (best < im_->free_blocks.size() &&
            (im_->free_blocks[best].bytes <= want + want / 16 || want < kLargeBlock || !im_->scarce)) {
            const Impl::Block b = im_->free_blocks[best];
            im_->free_blocks.erase(im_->free_blocks.begin() + best);
            im_->kept -= b.bytes;
            *got = b.bytes;
            return b.ptr;
        }
        if (im_->limit == 0) {
            size_t free_b = 0, total_b = 0;
            if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess) im_->limit = total_b / 16;
        }
    }
    bool scarce = false;
    if (want >= kLargeBlock) {
        scarce = memory_scarce();
        std::lock_guard<std::mutex> lock(im_->mu);
        im_->scarce = scarce;
    }
    size_t size = work_class(want, scarce);
    void* ptr = nullptr;
    cudaError_t e = cudaMalloc(&ptr, size);
    if (e == cudaErrorMemoryAllocation) {
        (void)cudaGetLastError();
        trim_all();
        size = want;
        e = cudaMalloc(&ptr, size);
    }
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        fail(PTBGPU_ENOMEM, "cudaMalloc(%zu) failed: %s", size, cudaGetErrorString(e));
    }
    *got = size;
    return ptr;
}

void WorkPool::give(void* ptr, size_t nbytes) {
    std::vector<Impl::Block> gone;
    {
        std::lock_guard<std::mutex> lock(im_->mu);
        if (nbytes > im_->limit) {
            gone.push_back({ptr, nbytes});
        } else {
            // the oldest blocks make room: sizes that no call asks for any more go first
            size_t drop = 0;
            while (im_->kept + nbytes > im_->limit) {
                im_->kept -= im_->free_blocks[drop].bytes;
                gone.push_back(im_->free_blocks[drop++]);
            }
            im_->free_blocks.erase(im_->free_blocks.begin(), im_->free_blocks.begin() + drop);
            im_->free_blocks.push_back({ptr, nbytes});
            im_->kept += nbytes;
        }
    }
    for (const Impl::Block& b : gone) cudaFree(b.ptr);
}

void WorkBuf::reserve(ptbgpu_ctx* c, size_t nbytes) {
    if (ptr && nbytes <= bytes) return;
    release();
    ptr = c->work->take(nbytes, &bytes);
    pool = c->work;
}

void WorkBuf::release() {
    if (ptr) pool->give(ptr, bytes);
    ptr = nullptr;
    bytes = 0;
    pool.reset();
}

int64_t& launch_counter() {
    static thread_local int64_t n = 0;
    return n;
}

void log_line(int level, int want, const char* fmt, ...) {
    if (level < want) return;
    va_list ap;
    va_start(ap, fmt);
    vfprintf(stdout, fmt, ap);
    va_end(ap);
    fputc('\n', stdout);
    fflush(stdout);
}

void log_timer_block(int level, const char* total_tag, double total_s,
                     const std::vector<std::pair<const char*, double>>& items) {
    if (level < 1) return;
    fprintf(stdout, "\n%-40s   %15.9f sec\n", total_tag, total_s);
    for (const auto& it : items) fprintf(stdout, "* %-40s %15.9f sec\n", it.first, it.second);
    fputc('\n', stdout);
    fflush(stdout);
}

}  // namespace ptb

cudaEvent_t ptbgpu_ctx::take_event() {
    if (evused == evpool.size()) {
        cudaEvent_t e;
        PTB_CUDA(cudaEventCreate(&e));
        evpool.push_back(e);
    }
    return evpool[evused++];
}

static_assert(ptb::B_COUNT <= ptbgpu_ctx::kMaxBufs, "more scratch-buffer ids than slots");

ptb::DevBuf& ptbgpu_ctx::buf(int id) {
    PTB_CHECK(id >= 0 && id < kMaxBufs, PTBGPU_EINVAL, "scratch buffer id %d out of range", id);
    return bufs[id];
}

extern "C" {

int ptbgpu_init(int device, ptbgpu_ctx** out) {
    if (!out) return PTBGPU_EINVAL;
    *out = nullptr;
    ptbgpu_ctx* c = new ptbgpu_ctx();
    try {
        c->device = device;
        PTB_CUDA(cudaSetDevice(device));
        int major = 0, minor = 0;
        PTB_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device));
        PTB_CUDA(cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, device));
        PTB_CHECK(major == 10 && minor == 0, PTBGPU_ECUDA,
                  "libptbgpu is built for sm_100a (B200); device %d is sm_%d%d", device, major, minor);
        PTB_CUDA(cudaDeviceGetAttribute(&c->num_sms, cudaDevAttrMultiProcessorCount, device));
        PTB_CUDA(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
        PTB_CUBLAS(cublasCreate(&c->blas));
        PTB_CUBLAS(cublasSetStream(c->blas, c->stream));
        PTB_CUBLAS(cublasSetMathMode(c->blas, CUBLAS_DEFAULT_MATH));
        PTB_CUSOLVER(cusolverDnCreate(&c->solver));
        PTB_CUSOLVER(cusolverDnSetStream(c->solver, c->stream));
        for (auto& e : c->ev) PTB_CUDA(cudaEventCreate(&e));
        PTB_CUDA(cudaMalloc(&c->flags, sizeof(ptb::DeviceFlags)));
        PTB_CUDA(cudaMemset(c->flags, 0, sizeof(ptb::DeviceFlags)));
        PTB_CUDA(cudaMalloc(&c->info_dev, sizeof(int)));
        PTB_CUDA(cudaMallocHost(&c->pinned, 4096));
    } catch (const ptb::Error& e) {
        fprintf(stderr, "ptbgpu_init: %s\n", e.msg.c_str());
        int code = e.code;
        ptbgpu_finalize(c);
        return code;
    }
    *out = c;
    return PTBGPU_OK;
}

int ptbgpu_finalize(ptbgpu_ctx* c) {
    if (!c) return PTBGPU_OK;
    if (c->stream) cudaStreamSynchronize(c->stream);
    c->sm_plan.reset();
    c->sm_side.reset();
    c->eig_streams.reset();
    for (ptbgpu_ctx* w : c->workers) ptbgpu_finalize(w);
    c->workers.clear();
    c->work->trim();
    for (auto& b : c->bufs) b.release();
    if (c->flags) cudaFree(c->flags);
    if (c->info_dev) cudaFree(c->info_dev);
    if (c->sp2_state) cudaFree(c->sp2_state);
    if (c->pinned) cudaFreeHost(c->pinned);
    for (auto& e : c->ev)
        if (e) cudaEventDestroy(e);
    for (auto& e : c->evpool) cudaEventDestroy(e);
    if (c->solver) cusolverDnDestroy(c->solver);
    if (c->blas) cublasDestroy(c->blas);
    if (c->stream) cudaStreamDestroy(c->stream);
    delete c;
    return PTBGPU_OK;
}

int ptbgpu_trim(ptbgpu_ctx* c) {
    if (!c) return PTBGPU_EINVAL;
    c->work->trim();
    for (ptbgpu_ctx* w : c->workers) w->work->trim();
    return PTBGPU_OK;
}

int ptbgpu_last_error(const ptbgpu_ctx* c, char* buf, size_t len) {
    if (!c || !buf || len == 0) return PTBGPU_EINVAL;
    strncpy(buf, c->last_error.c_str(), len - 1);
    buf[len - 1] = '\0';
    return PTBGPU_OK;
}

int ptbgpu_runtime_info(const ptbgpu_ctx* c, char* buf, size_t len) {
    if (!c || !buf || len == 0) return PTBGPU_EINVAL;
    int rt = 0, drv = 0, cub = 0, maj = 0, min = 0, pat = 0;
    cudaRuntimeGetVersion(&rt);
    cudaDriverGetVersion(&drv);
    cublasGetVersion(c->blas, &cub);
    cusolverGetProperty(MAJOR_VERSION, &maj);
    cusolverGetProperty(MINOR_VERSION, &min);
    cusolverGetProperty(PATCH_LEVEL, &pat);
    cudaDeviceProp p{};
    cudaGetDeviceProperties(&p, c->device);
    snprintf(buf, len, "device %s (sm_%d%d, %d SMs) cudart %d driver %d cublas %d cusolver %d.%d.%d", p.name,
             p.major, p.minor, p.multiProcessorCount, rt, drv, cub, maj, min, pat);
    return PTBGPU_OK;
}

void ptbgpu_default_settings(ptbgpu_pur_settings* s) {
    if (!s) return;
    s->mode = PTBGPU_MODE_FULL;
    s->type = PTBGPU_TYPE_DIAG;
    s->cycles = 40;
    s->prlvl = 1;
    s->nel = 0;
    s->submatrix_mode = PTBGPU_SUBMATRIX_SYGV;
    s->submatrix_columns = PTBGPU_COLUMNS_ATOMS;
    s->metric_type = PTBGPU_METRIC_INV_SQRT;
    s->metric_cycles = 50;
    s->metric_iterative = 0;
    s->chempot_cycles = 60;
    s->chempot_guess = -1.5;
    s->chempot_increment = 0.1;
}

void ptbgpu_default_opts(ptbgpu_opts* o) {
    if (!o) return;
    memset(o, 0, sizeof(*o));
    o->precision = PTBGPU_PREC_MIXED;
    o->print_level = 0;
    o->max_iter = 100;
    o->electronic_temp = 300.0;
    o->split3_iters = -1;
    o->fp64_slices = 8;
    o->refine_rounds = 4;
    o->refine_tol = 1e-7;
}

}  // extern "C"
