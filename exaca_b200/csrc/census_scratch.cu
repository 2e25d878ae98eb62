// Census of IntermediateOutputAndCheck (src/CAupdate.cpp:738-808) over cell fields the caller
// already holds in device memory, for callers that must not allocate device memory.
//
// Who cannot allocate: a monitor sampling the progress of solves that are still running (a
// cudaMalloc or cudaFree may synchronise the whole device and stall every solve on it), and a
// serving process whose HBM budget is handed out in full to admitted domains. The pool's own
// census (exaca_pool_census) keeps its accumulator in a buffer it allocated at pool creation and
// reads a pool slot; this variant reads any caller arrays and keeps its working data in the
// fixed file-scope array below instead.
//
// Scratch: kScratchBytes = 26 KiB, for at most kMaxDomains = 256 domains per call. The first
// 256 * 56 bytes hold the copied domain descriptors, the next 256 * 48 bytes one accumulator of six
// 64-bit counters per domain. Every call on a device shares this array and it keeps what the last
// call left in it: each call copies its descriptors in and clears its accumulators to zero before
// the kernel runs. Two calls whose work overlapped on the device would race on the array, so a
// call holds a per-device lock until its stream has drained.
#include <cuda_runtime.h>

#include <climits>
#include <cstring>
#include <mutex>
#include <string>

#include "../../include/exaca_b200.h"
#include "exaca_host.hpp"

namespace exaca {

namespace {

constexpr int kMaxDomains = EXACA_CENSUS_MAX_DOMAINS;
constexpr size_t kDescBytes = sizeof(exaca_cell_fields);
constexpr size_t kAccWords = 6;
constexpr size_t kAccOffset = kMaxDomains * kDescBytes;
constexpr size_t kScratchBytes = kAccOffset + kMaxDomains * kAccWords * sizeof(unsigned long long);
constexpr int kMaxDevices = 64;
constexpr int kThreads = 256;

static_assert(kDescBytes == 56, "exaca_cell_fields is 56 bytes on LP64");
static_assert(sizeof(exaca_census) == kAccWords * sizeof(unsigned long long), "exaca_census is six counters");
static_assert(kScratchBytes == 26624, "26 KiB scratch");

static __device__ __align__(256) unsigned char g_census_scratch[kScratchBytes];

// One accumulator per domain: superheated, undercooled, active, solid, remaining, and the bitwise
// complement of the minimum CritTimeStep of the layer's liquid cells in the active window (so that
// all six start at zero; zero means "no such cell" = ULLONG_MAX once complemented back). Cells of
// the current layer are classified (src/CAupdate.cpp:741-752), liquid cells of any other layer are
// remaining (:754-757); the minimum is taken over the window only (:792-805).
//
// 6 bytes are read per cell. kWide, for domains in which every thread has sixteen cells or more: sixteen
// cells per thread and step in 16-byte loads where the three arrays are 16-byte aligned (cell by cell
// otherwise and at the end). On smaller domains sixteen cells one after the other are the longer chain
// (38.9 us per call instead of 32.0 on a few small ones), and a thread takes one at a time.
// A block sums its counts in shared memory before its six atomics, except on grids of few blocks, whose
// warps do not queue on a counter: 4 domains of 34^2 x 32 cells (144 blocks each) 42.0 -> 31.9 us per call,
// 24 of 58^2 x 56 90 -> 73, 2 of 202^2 x 200 113 -> 65, but one of 22^2 x 20 27.2 -> 27.8 with the
// sums and 27.1 -> 27.1 without.
constexpr long long kFewBlocks = 64;
__device__ __forceinline__ bool wide_reads(const exaca_cell_fields &d) {
    return ((reinterpret_cast<unsigned long long>(d.cell_type) | reinterpret_cast<unsigned long long>(d.layer_id) |
             reinterpret_cast<unsigned long long>(d.crit_time_step)) &
            15u) == 0;
}

struct CellCount {
    unsigned int n[5] = {0, 0, 0, 0, 0};
    unsigned long long neg_mn = 0;
    __device__ __forceinline__ void cell(const exaca_cell_fields &d, long long c, int t, int ly, int cts) {
        if (ly == d.layer) {
            if (t == kLiquid) {
                n[cts > d.cycle ? 0 : 1]++;
                const unsigned long long neg = ~(unsigned long long)(long long)cts;
                if (c >= d.window_start && c < d.window_start + d.active_size && neg > neg_mn)
                    neg_mn = neg;
            }
            else if (t == kActive)
                n[2]++;
            else if (t == kSolid)
                n[3]++;
        }
        else if (t == kLiquid) {
            n[4]++;
        }
    }
};

template <bool kWide, bool kSums>
__global__ void __launch_bounds__(kThreads) k_census_cells(const exaca_cell_fields *cells, unsigned long long *acc) {
    const exaca_cell_fields d = cells[blockIdx.y];
    unsigned long long *out = acc + kAccWords * blockIdx.y;
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    CellCount k;
    long long n16 = 0;
    if (kWide && wide_reads(d)) {
        n16 = d.domain_size / 16;
        for (long long q = tid; q < n16; q += stride) {
            const int4 t16 = __ldcs(reinterpret_cast<const int4 *>(d.cell_type) + q);
            const int4 l16 = __ldcs(reinterpret_cast<const int4 *>(d.layer_id) + q);
            int4 c4[4];
#pragma unroll
            for (int u = 0; u < 4; u++)
                c4[u] = __ldcs(reinterpret_cast<const int4 *>(d.crit_time_step) + 4 * q + u);
            const int tw[4] = {t16.x, t16.y, t16.z, t16.w}, lw[4] = {l16.x, l16.y, l16.z, l16.w};
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int cv[4] = {c4[u].x, c4[u].y, c4[u].z, c4[u].w};
#pragma unroll
                for (int b = 0; b < 4; b++)
                    k.cell(d, 16 * q + 4 * u + b, (int)(int8_t)(tw[u] >> (8 * b)), (int)(int8_t)(lw[u] >> (8 * b)), cv[b]);
            }
        }
    }
    for (long long c = 16 * n16 + tid; c < d.domain_size; c += stride)
        k.cell(d, c, d.cell_type[c], d.layer_id[c], d.crit_time_step[c]);
    __shared__ unsigned long long s_sum[kSums ? 6 : 1];
    if (kSums) {
        if (threadIdx.x < 6)
            s_sum[threadIdx.x] = 0;
        __syncthreads();
    }
    unsigned long long *const to = kSums ? s_sum : out;
#pragma unroll
    for (int q = 0; q < 5; q++) {
        // a thread of the wide kernel counts fewer than 2^32 cells, its warp fewer than 2^37: two halves;
        // one of the other kernels at most sixteen
        const unsigned int lo = __reduce_add_sync(0xffffffffu, kWide ? k.n[q] & 0xffffu : k.n[q]),
                           hi = kWide ? __reduce_add_sync(0xffffffffu, k.n[q] >> 16) : 0u;
        if ((threadIdx.x & 31) == 0 && (lo | hi))
            atomicAdd(to + q, ((unsigned long long)hi << 16) + lo);
    }
    unsigned long long neg_mn = k.neg_mn;
    for (int o = 16; o; o >>= 1) {
        const unsigned long long v = __shfl_down_sync(0xffffffffu, neg_mn, o);
        neg_mn = v > neg_mn ? v : neg_mn;
    }
    if ((threadIdx.x & 31) == 0 && neg_mn)
        atomicMax(to + 5, neg_mn);
    if (!kSums)
        return;
    __syncthreads();
    if (threadIdx.x < 6 && s_sum[threadIdx.x]) {
        if (threadIdx.x < 5)
            atomicAdd(out + threadIdx.x, s_sum[threadIdx.x]);
        else
            atomicMax(out + 5, s_sum[5]);
    }
}

struct DeviceScratch {
    std::mutex lock;
    bool ready = false;
    unsigned char *ptr = nullptr; // device address of g_census_scratch on this device
    int num_sms = 0;
};

DeviceScratch g_devices[kMaxDevices];

void check(cudaError_t e, const char *what) {
    if (e != cudaSuccess)
        throw DeviceError(std::string(what) + ": " + cudaGetErrorString(e));
}

// Once per device, with that device current: the scratch array's device address, the SM count,
// and the kernel's module loaded (so later calls do no lazy loading).
void setup(DeviceScratch &s, int device) {
    if (s.ready)
        return;
    void *p = nullptr;
    check(cudaGetSymbolAddress(&p, g_census_scratch), "cudaGetSymbolAddress(census scratch)");
    if (reinterpret_cast<uintptr_t>(p) % 256 != 0)
        throw DeviceError("census scratch is not 256-byte aligned");
    int sms = 0;
    check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "cudaDeviceGetAttribute");
    cudaFuncAttributes fa;
    check(cudaFuncGetAttributes(&fa, k_census_cells<true, true>), "cudaFuncGetAttributes(k_census_cells)");
    check(cudaFuncGetAttributes(&fa, k_census_cells<false, true>), "cudaFuncGetAttributes(k_census_cells)");
    check(cudaFuncGetAttributes(&fa, k_census_cells<false, false>), "cudaFuncGetAttributes(k_census_cells)");
    s.ptr = static_cast<unsigned char *>(p);
    s.num_sms = sms;
    s.ready = true;
}

struct DeviceRestore {
    int prev = -1;
    ~DeviceRestore() {
        if (prev >= 0)
            cudaSetDevice(prev);
    }
};

} // namespace

void census_cells(int device, void *stream, const exaca_cell_fields *domains, int n_domains, exaca_census *out) {
    DeviceScratch &s = g_devices[device];
    std::lock_guard<std::mutex> guard(s.lock);
    DeviceRestore restore;
    check(cudaGetDevice(&restore.prev), "cudaGetDevice");
    check(cudaSetDevice(device), "cudaSetDevice");
    setup(s, device);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    long long largest = 1;
    for (int i = 0; i < n_domains; i++)
        largest = domains[i].domain_size > largest ? domains[i].domain_size : largest;
    unsigned char *desc = s.ptr;
    unsigned long long *acc = reinterpret_cast<unsigned long long *>(s.ptr + kAccOffset);
    try {
        check(cudaMemcpyAsync(desc, domains, n_domains * kDescBytes, cudaMemcpyHostToDevice, st), "descriptor copy");
        check(cudaMemsetAsync(acc, 0, n_domains * kAccWords * sizeof(unsigned long long), st), "accumulator clear");
        long long bx = (4ll * s.num_sms + n_domains - 1) / n_domains;
        const long long need = (largest + kThreads - 1) / kThreads;
        bx = bx < need ? bx : need;
        bx = bx < 1 ? 1 : bx;
        const auto kernel = largest >= 16 * bx * kThreads ? k_census_cells<true, true>
                            : bx >= kFewBlocks            ? k_census_cells<false, true>
                                                          : k_census_cells<false, false>;
        kernel<<<dim3((unsigned)bx, (unsigned)n_domains), kThreads, 0, st>>>(
            reinterpret_cast<const exaca_cell_fields *>(desc), acc);
        check(cudaGetLastError(), "k_census_cells launch");
        check(cudaMemcpyAsync(out, acc, n_domains * sizeof(exaca_census), cudaMemcpyDeviceToHost, st), "census copy");
        check(cudaStreamSynchronize(st), "census stream");
    }
    catch (...) {
        // work of this call may still be queued on the stream: the lock (which keeps other calls off
        // the shared array) is released only once it has drained
        cudaStreamSynchronize(st);
        throw;
    }
    for (int i = 0; i < n_domains; i++)
        out[i].next_cts = ~out[i].next_cts;
}

// Number of usable devices (at most kMaxDevices), or -1 when the CUDA runtime reports none.
int census_device_count() {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess)
        return -1;
    return n < kMaxDevices ? n : kMaxDevices;
}

} // namespace exaca
