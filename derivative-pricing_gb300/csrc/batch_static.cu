// batch_static.cu -- mcd_price_batch_static: batched GBM pricing that
// allocates no memory.
//
// Some callers cannot call cudaMalloc: a service that reserves all of its
// device memory up front and accounts for every byte, code running where an
// allocation's implicit device synchronisation is not acceptable, or a host
// process that is only allowed to use memory that already exists when it
// starts.  For them this entry point runs the same persistent path kernel and
// merge kernel as mcd_price_batch, but keeps every byte of scratch they need
// (contract records, the slab prefix, slab partials, device results, the
// ticket and error word) in one file-scope __device__ array of fixed size,
// which the CUDA module reserves when it is loaded and keeps until the process
// exits.  The caller passes inputs and outputs as host arrays.
//
// Limits: at most kStaticMaxContracts contracts and kStaticMaxSlabs slabs of
// 4096 paths per call (about 1.07e9 paths in total); the array is about 7 MB.
// Contracts are processed in the order given (no longest-first sort), which
// changes load balance but not results: item partials and their merge order
// depend only on the item index, so results are bitwise identical to
// mcd_price_batch's.  An FP64 contract has more, smaller items (units) than
// slabs: a batch with more of them than the partials hold runs as several
// launches over ranges of contracts.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>

#include "engine.hpp"
#include "items.hpp"
#include "mcd_gpu.h"

namespace {

using mcdg::DevContract;
using mcdg::Welford;

constexpr size_t kStaticMaxContracts = 4096;
constexpr size_t kStaticMaxSlabs = 262144;
constexpr int kStaticMaxDevices = 64;

constexpr size_t align256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }
constexpr size_t kOffContracts = 0;
constexpr size_t kOffPrefix = align256(kOffContracts + sizeof(DevContract) * kStaticMaxContracts);
constexpr size_t kOffPartials = align256(kOffPrefix + sizeof(uint32_t) * (kStaticMaxContracts + 1));
constexpr size_t kOffResults = align256(kOffPartials + sizeof(Welford) * kStaticMaxSlabs);
constexpr size_t kOffFlags = align256(kOffResults + sizeof(mcd_mc_result) * kStaticMaxContracts);
constexpr size_t kStaticScratchBytes = align256(kOffFlags + 256);

// The scratch array.  Host code must not use this name as an address (on the
// host it is a stand-in object); the device address comes from
// cudaGetSymbolAddress, resolved once per device in static_setup().
static __device__ __align__(256) unsigned char g_batch_scratch[kStaticScratchBytes];

// Host-side state, all static: resolved device addresses and launch shapes per
// device, and a staging area for the converted contracts.  One lock serialises
// calls (the device array is shared by all of them).
std::mutex g_static_lock;
unsigned char* g_scratch_addr[kStaticMaxDevices] = {};
unsigned long long g_context[kStaticMaxDevices] = {};  // the CUDA context that the addresses are of
int g_grid[kStaticMaxDevices][2] = {};  // persistent grid per device and precision
DevContract g_stage_contracts[kStaticMaxContracts];
uint32_t g_stage_prefix[kStaticMaxContracts + 1];
const mcdg::FixedTables* g_tables[kStaticMaxDevices] = {};

int report(char* msg, size_t cap, int code, const char* text) {
    if (msg && cap) std::snprintf(msg, cap, "%s", text);
    return code;
}

int report_cuda(char* msg, size_t cap, cudaError_t e, const char* where) {
    if (msg && cap) std::snprintf(msg, cap, "%s: %s", where, cudaGetErrorString(e));
    cudaGetLastError();
    return e == cudaErrorMemoryAllocation ? MCD_ERR_OUT_OF_MEMORY : MCD_ERR_CUDA;
}

// First call on a device, or on one that was reset since: resolve the array's device address with that
// device current and size the grids.  Must happen outside any stream capture.
// With CUDA's lazy module loading (the runtime's default) this is also when
// the module is loaded on the device and the array's memory is reserved.
int static_setup(int device, cudaStream_t stream, char* msg, size_t cap) {
    unsigned long long id = 0;
    cudaError_t e = mcdg::device_context_id(&id);
    if (e != cudaSuccess) return report_cuda(msg, cap, e, "CUDA context");
    if (g_scratch_addr[device] && g_context[device] == id) return MCD_OK;
    void* addr = nullptr;
    e = cudaGetSymbolAddress(&addr, g_batch_scratch);
    if (e != cudaSuccess) return report_cuda(msg, cap, e, "cudaGetSymbolAddress(scratch)");
    e = mcdg::fixed_tables_device(&g_tables[device], stream);
    if (e != cudaSuccess) return report_cuda(msg, cap, e, "fixed-point tables");
    int sms = 0;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return report_cuda(msg, cap, e, "SM count");
    for (int precision = 0; precision < 2; ++precision) {
        int blocks = 0;
        e = mcdg::path_kernel_occupancy(precision, mcdg::kDefaultVariant[precision], &blocks);
        if (e != cudaSuccess) return report_cuda(msg, cap, e, "occupancy");
        g_grid[device][precision] = sms * (blocks > 0 ? blocks : 1);
    }
    g_scratch_addr[device] = static_cast<unsigned char*>(addr);
    g_context[device] = id;
    return MCD_OK;
}

}  // namespace

extern "C" int mcd_price_batch_static(const mcd_contract* contracts, size_t n, int precision,
                                      mcd_mc_result* results, void* stream, char* error_message,
                                      size_t error_capacity) try {
    std::lock_guard<std::mutex> lock(g_static_lock);
    if (error_message && error_capacity) error_message[0] = '\0';
    if (precision != MCD_PRECISION_FP64 && precision != MCD_PRECISION_FP32)
        return report(error_message, error_capacity, MCD_ERR_INVALID_ARGUMENT,
                      "precision must be 0 (FP64) or 1 (FP32)");
    if (n > kStaticMaxContracts)
        return report(error_message, error_capacity, MCD_ERR_INVALID_ARGUMENT,
                      "mcd_price_batch_static: at most 4096 contracts per call");
    if (n > 0 && (!contracts || !results))
        return report(error_message, error_capacity, MCD_ERR_INVALID_ARGUMENT, "null array");
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return report_cuda(error_message, error_capacity, e, "cudaGetDevice");
    if (device < 0 || device >= kStaticMaxDevices)
        return report(error_message, error_capacity, MCD_ERR_UNSUPPORTED, "device index too large");
    // A call with n = 0 does the device's set-up only: a caller that reserves
    // the rest of device memory afterwards makes this call first.
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int rc = static_setup(device, s, error_message, error_capacity);
    if (rc != MCD_OK || n == 0) return rc;

    uint64_t total = 0;   // slabs, the limit's unit
    uint32_t items = 0;   // items (FP32) or units (FP64) so far, modulo 2^32
    for (size_t i = 0; i < n; ++i) {
        const char* why = mcdg::convert_contract(contracts[i], static_cast<uint32_t>(i), g_stage_contracts[i]);
        if (why) {
            char text[160];
            std::snprintf(text, sizeof text, "contract %zu: %s", i, why);
            return report(error_message, error_capacity, MCD_ERR_INVALID_ARGUMENT, text);
        }
        g_stage_prefix[i] = items;
        items += precision == MCD_PRECISION_FP64 ? g_stage_contracts[i].n_units : g_stage_contracts[i].n_items;
        total += g_stage_contracts[i].n_slabs;
        if (total > kStaticMaxSlabs)
            return report(error_message, error_capacity, MCD_ERR_INVALID_ARGUMENT,
                          "mcd_price_batch_static: at most 262144 slabs of 4096 paths per call");
    }
    g_stage_prefix[n] = items;

    unsigned char* base = g_scratch_addr[device];
    DevContract* d_contracts = reinterpret_cast<DevContract*>(base + kOffContracts);
    uint32_t* d_prefix = reinterpret_cast<uint32_t*>(base + kOffPrefix);
    Welford* d_partials = reinterpret_cast<Welford*>(base + kOffPartials);
    mcd_mc_result* d_results = reinterpret_cast<mcd_mc_result*>(base + kOffResults);
    uint32_t* d_flags = reinterpret_cast<uint32_t*>(base + kOffFlags);

    // The array keeps the previous call's contents: the ticket and the error
    // word must start at zero; contracts, prefix, partials and results are
    // overwritten in full for the items of this call.
    e = cudaMemcpyAsync(d_contracts, g_stage_contracts, sizeof(DevContract) * n, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(d_prefix, g_stage_prefix, sizeof(uint32_t) * (n + 1), cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return report_cuda(error_message, error_capacity, e, "stage contracts");
    // Contracts in ranges whose items fit the partials: FP32 items (at most 256 or
    // the slabs of a contract) and FP64 units (at most 4096 per contract, slabs from
    // 2^24 paths on) are smaller than slabs, so a large batch of small contracts
    // takes several launches on the same scratch.
    static_assert(mcdg::kMaxCutItems <= kStaticMaxSlabs && 4096 <= kStaticMaxSlabs, "one contract's items fit the partials");
    for (size_t first = 0; first < n;) {
        size_t end = first + 1;
        while (end < n && g_stage_prefix[end + 1] - g_stage_prefix[first] <= kStaticMaxSlabs) ++end;
        e = cudaMemsetAsync(d_flags, 0, (first == 0 ? 2 : 1) * sizeof(uint32_t), s);
        if (e != cudaSuccess) return report_cuda(error_message, error_capacity, e, "reset flags");
        const int count = static_cast<int>(end - first);
        if (g_stage_prefix[end] != g_stage_prefix[first]) {
            e = mcdg::launch_path_kernel(precision, mcdg::kDefaultVariant[precision], g_grid[device][precision], d_contracts + first, count,
                                         d_prefix + first, d_flags, d_partials, d_flags + 1, g_tables[device], s);
            if (e != cudaSuccess) return report_cuda(error_message, error_capacity, e, "path kernel");
        }
        e = mcdg::launch_merge_kernel(d_contracts + first, count, d_prefix + first, d_partials, d_results, s);
        if (e != cudaSuccess) return report_cuda(error_message, error_capacity, e, "merge kernel");
        first = end;
    }
    uint32_t flags[2] = {0, 0};
    e = cudaMemcpyAsync(results, d_results, sizeof(mcd_mc_result) * n, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(flags, d_flags, sizeof flags, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return report_cuda(error_message, error_capacity, e, "batch execution");
    if (flags[1] != 0)
        return report(error_message, error_capacity, MCD_ERR_CUDA, "path kernel reported an inconsistent work item");
    return MCD_OK;
} catch (...) {  // nothing here throws but a lock that the system refuses
    return report(error_message, error_capacity, MCD_ERR_INVALID_ARGUMENT, "internal error");
}
