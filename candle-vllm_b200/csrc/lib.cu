// lib.cu -- library state: per-thread error record, launch counter, device probing.
#include <atomic>
#include <cstdarg>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <map>
#include <set>
#include <utility>

#include "common.cuh"
#include "tc_common.cuh"

namespace b200 {

static thread_local int t_err = 0;
static thread_local char t_msg[512] = {0};
static std::atomic<long long> g_launches{0};

void set_error(int code, const char* fmt, ...) {
    t_err = code;
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(t_msg, sizeof(t_msg), fmt, ap);
    va_end(ap);
}

bool check_launch(const char* what) {
    cudaError_t e = cudaPeekAtLastError();
    if (e != cudaSuccess) {
        set_error(kErrCuda, "%s: %s", what, cudaGetErrorString(e));
        return false;
    }
    return true;
}

void count_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

bool pdl_enabled() {
    static const int on = [] { const char* e = getenv("B200_PDL"); return e ? atoi(e) : 1; }();
    return on != 0;
}

constexpr int kMaxDevices = 64;

int sm_count() {
    static std::atomic<int> cached[kMaxDevices];          // zero-initialised: 0 = not probed yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) { cudaGetLastError(); return 148; }
    int n = cached[dev].load(std::memory_order_relaxed);
    if (n == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) {
            cudaGetLastError();
            return 148;   // B200; only used to size grids
        }
        cached[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

void ensure_dynamic_smem(const void* kernel, int bytes) {
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, int> done;      // the largest size a kernel was opened for, per device
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return; }
    std::lock_guard<std::mutex> lk(mu);
    auto it = done.find({dev, kernel});
    if (it != done.end() && it->second >= bytes) return;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess) done[{dev, kernel}] = bytes;
    else cudaGetLastError();
}

int max_active_clusters(const void* kernel, int threads, int smem, int size) {
    static std::atomic<int> cached[kMaxDevices][9];
    int dev = 0;
    if (size < 1 || size > 8) return 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) { cudaGetLastError(); return 0; }
    int n = cached[dev][size].load(std::memory_order_relaxed);
    if (n == 0) {
        ensure_dynamic_smem(kernel, smem);
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)(size * 64)); cfg.blockDim = dim3((unsigned)threads); cfg.dynamicSmemBytes = (size_t)smem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)size; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr; cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) { cudaGetLastError(); n = -1; }
        cached[dev][size].store(n, std::memory_order_relaxed);
    }
    return n < 0 ? 0 : n;
}

// One word for all devices: portable pinned memory has the same address on each.  Asked for by the first launch of a kernel with bounded waits, possibly during a stream
// capture, where allocations are refused unless the thread says that it knows.
static std::atomic<uint32_t*> g_wait_word{nullptr};
uint32_t* wait_report_word() {
    uint32_t* w = g_wait_word.load(std::memory_order_acquire);
    if (w) return w;
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    w = g_wait_word.load(std::memory_order_acquire);
    if (w) return w;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    void *host = nullptr, *dev = nullptr;
    if (cudaHostAlloc(&host, sizeof(uint32_t), cudaHostAllocMapped | cudaHostAllocPortable) == cudaSuccess && cudaHostGetDevicePointer(&dev, host, 0) == cudaSuccess && dev == host) {
        *static_cast<volatile uint32_t*>(host) = 0u;
        w = static_cast<uint32_t*>(host);
        g_wait_word.store(w, std::memory_order_release);
    } else {
        cudaGetLastError();
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
    return w;
}

// a kernel with a bounded wait on a barrier that nothing arrives at
__global__ void wait_limit_kernel(uint32_t* report, unsigned long long limit_ns) {
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t flag;
    const uint32_t b = tc::smem_u32(&bar);
    if (threadIdx.x == 0) {
        flag = 0u;
        tc::mbar_init(b, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    tc::mbar_wait_or_flag(b, 0, tc::GiveUp{&flag, report, kWaitCheck, limit_ns});
}

}  // namespace b200

extern "C" {

int b200_abi_version(void) { return 1; }

int b200_last_error(void) {
    int e = b200::t_err;
    uint32_t* const word = e ? nullptr : b200::g_wait_word.load(std::memory_order_acquire);
    if (word && *static_cast<volatile uint32_t*>(word)) {
        const uint32_t w = __atomic_exchange_n(word, 0u, __ATOMIC_ACQ_REL);
        if (w) {
            b200::set_error(b200::kErrCuda, "a kernel of an earlier call gave up a wait and left its output unwritten:%s%s%s%s", w & b200::kWaitPromptAttention ? " prompt attention" : "",
                            w & b200::kWaitPairGemm ? " two-SM GEMM" : "", w & b200::kWaitLatentDecode ? " latent decode" : "", w & b200::kWaitCheck ? " wait limit check" : "");
            e = b200::t_err;
        }
    }
    b200::t_err = 0;
    return e;
}

void b200_wait_limit_check(int32_t limit_us, int64_t stream) {
    B200_REQUIRE(limit_us > 0 && limit_us <= 1000000, b200::kErrBadArg, "b200_wait_limit_check: %d us", limit_us);
    uint32_t* const word = b200::wait_report_word();
    B200_REQUIRE(word, b200::kErrCuda, "b200_wait_limit_check: no host-mapped memory");
    b200::wait_limit_kernel<<<1, 32, 0, b200::as_stream(stream)>>>(word, (unsigned long long)limit_us * 1000ull);
    b200::count_launch();
    b200::check_launch("b200_wait_limit_check");
}

const char* b200_last_error_message(void) { return b200::t_msg; }

int b200_device_sm_count(void) {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

int b200_device_cc(void) {
    static std::atomic<int> cached[b200::kMaxDevices];    // a device's capability does not change: 0 = not asked yet
    int dev = 0, ma = 0, mi = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return 0; }
    const bool keep = dev >= 0 && dev < b200::kMaxDevices;
    if (keep) { const int cc = cached[dev].load(std::memory_order_relaxed); if (cc) return cc; }
    if (cudaDeviceGetAttribute(&ma, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&mi, cudaDevAttrComputeCapabilityMinor, dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    if (keep) cached[dev].store(ma * 10 + mi, std::memory_order_relaxed);
    return ma * 10 + mi;
}

long long b200_total_kernel_launches(void) { return b200::g_launches.load(); }

}  // extern "C"
