// A context's device memory: its pools, the budget's accounting, and the events
// of its objects' last uses.
#include <algorithm>

#include "internal.h"

namespace cpvs {

cudaError_t create_pool(int device, cudaMemPool_t* pool, uint64_t keep) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    const cudaError_t e = cudaMemPoolCreate(pool, &props);
    if (e == cudaSuccess) cudaMemPoolSetAttribute(*pool, cudaMemPoolAttrReleaseThreshold, &keep);
    return e;
}

cpvs_status Ctx::alloc(void** p, uint64_t bytes, bool persistent, cudaStream_t st, cudaMemPool_t from) {
    *p = nullptr;
    if (budget && in_use + scratch + bytes > budget)
        return fail(CPVS_ERR_BUDGET, "allocation of " + std::to_string(bytes) + " bytes exceeds the context budget");
    cudaError_t e = cudaMallocFromPoolAsync(p, bytes, from ? from : pool, st);
    if (e == cudaErrorMemoryAllocation && index_pool) {
        // the freed blocks that one pool holds are no use to the other: back
        // to the driver with both
        cudaMemPoolTrimTo(index_pool, 0);
        cudaMemPoolTrimTo(pool, 0);
        cudaGetLastError();
        e = cudaMallocFromPoolAsync(p, bytes, from ? from : pool, st);
    }
    if (e != cudaSuccess) return cuda_fail(e, "cudaMallocFromPoolAsync");
    if (persistent)
        in_use += bytes;
    else
        scratch += bytes;
    return CPVS_OK;
}

cudaEvent_t Ctx::take_event() {
    if (!event_pool.empty()) {
        const cudaEvent_t e = event_pool.back();
        event_pool.pop_back();
        return e;
    }
    cudaEvent_t e = nullptr;
    if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return e;
}

void Ctx::give_event(cudaEvent_t e) {
    if (!e) return;
    if (event_pool.size() < kEventPool)
        event_pool.push_back(e);
    else
        cudaEventDestroy(e);
}

void Ctx::await_use(cudaEvent_t last_use) {
    if (last_use && cudaStreamWaitEvent(free_stream, last_use, 0) != cudaSuccess) cudaGetLastError();
}

void Ctx::release(void* p, uint64_t bytes, bool persistent, cudaStream_t st, cudaEvent_t last_use) {
    if (persistent) {
        if (p) {
            await_use(last_use);
            cudaFreeAsync(p, free_stream);
        }
        in_use -= std::min(in_use, bytes);
    } else {
        if (p) cudaFreeAsync(p, st);
        scratch -= std::min(scratch, bytes);
    }
}

constexpr uint64_t kIndexOwn = 16ull << 20;
constexpr uint64_t kIndexKeep = 1ull << 30;  // 16 of the largest

int* Ctx::lookup_choice(uint32_t num_levels, int depth, bool leafmasks, bool ndc, bool host_in, uint64_t n) {
    if (n < std::max(num_sms, 1) * 2048ull) return nullptr;  // 2048 threads to an SM
    return &lookup_qpt_tuned[(num_levels - (uint32_t)depth) % CPVS_MAX_LEVELS][leafmasks][ndc][host_in];
}

bool capturing(cudaStream_t st) {
    cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &s) == cudaSuccess) return s != cudaStreamCaptureStatusNone;
    cudaGetLastError();
    return true;
}

bool reached(cudaEvent_t e) {
    // another thread's capture is no reason to refuse the question, nor harmed
    // by it
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    const bool done = cudaEventQuery(e) == cudaSuccess;
    if (!done) cudaGetLastError();
    cudaThreadExchangeStreamCaptureMode(&mode);
    return done;
}

cudaMemPool_t Ctx::index_source(uint64_t bytes) {
    if (bytes < kIndexOwn || budget) return nullptr;
    if (!index_pool && create_pool(device, &index_pool, kIndexKeep) != cudaSuccess) {
        cudaGetLastError();
        index_pool = nullptr;
    }
    return index_pool;
}

void Ctx::set_budget(uint64_t bytes) {
    budget = bytes;
    if (!index_pool) return;
    uint64_t keep = budget ? 0 : kIndexKeep;
    cudaMemPoolSetAttribute(index_pool, cudaMemPoolAttrReleaseThreshold, &keep);
    if (budget) cudaMemPoolTrimTo(index_pool, 0);
    cudaGetLastError();
}

}  // namespace cpvs
