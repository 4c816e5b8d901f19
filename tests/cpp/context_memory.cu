// A context's memory over its two pools, and its choices (csrc/context.cu), with a model of the
// CUDA pools in place of the driver's: a device of `capacity` bytes, pools that
// reserve what they hand out and keep what is freed up to their threshold.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace model {
constexpr uint64_t MiB = 1ull << 20;
uint64_t capacity = 1024 * MiB;
struct Pool {
    uint64_t reserved = 0, used = 0, keep = 0;
};
std::vector<Pool*> pools;
std::map<void*, std::pair<Pool*, uint64_t>> blocks;
char place[1 << 12];
size_t next = 0;

uint64_t reserved() {
    uint64_t r = 0;
    for (const Pool* p : pools) r += p->reserved;
    return r;
}
cudaError_t create(cudaMemPool_t* out, const cudaMemPoolProps*) {
    pools.push_back(new Pool);
    *out = reinterpret_cast<cudaMemPool_t>(pools.back());
    return cudaSuccess;
}
cudaError_t attribute(cudaMemPool_t p, cudaMemPoolAttr, void* v) {
    reinterpret_cast<Pool*>(p)->keep = *static_cast<uint64_t*>(v);
    return cudaSuccess;
}
cudaError_t trim(cudaMemPool_t p, size_t) {
    Pool* q = reinterpret_cast<Pool*>(p);
    q->reserved = q->used;
    return cudaSuccess;
}
cudaError_t allocate(void** out, size_t bytes, cudaMemPool_t p, cudaStream_t) {
    Pool* q = reinterpret_cast<Pool*>(p);
    const uint64_t more = q->used + bytes > q->reserved ? q->used + bytes - q->reserved : 0;
    if (reserved() + more > capacity) return cudaErrorMemoryAllocation;
    q->reserved += more;
    q->used += bytes;
    *out = place + next++;
    blocks[*out] = {q, bytes};
    return cudaSuccess;
}
cudaError_t release(void* p, cudaStream_t) {
    auto b = blocks[p];
    blocks.erase(p);
    b.first->used -= b.second;
    if (b.first->reserved > b.first->keep) b.first->reserved = b.first->used > b.first->keep ? b.first->used : b.first->keep;
    return cudaSuccess;
}
cudaError_t is_capturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t ok() { return cudaSuccess; }
}  // namespace model

#define cudaMemPoolCreate model::create
#define cudaMemPoolSetAttribute model::attribute
#define cudaMemPoolTrimTo model::trim
#define cudaMallocFromPoolAsync model::allocate
#define cudaFreeAsync model::release
#define cudaStreamIsCapturing model::is_capturing
#define cudaGetLastError model::ok
#include "../../cpvs_gb300/csrc/context.cu"

namespace cpvs {
cpvs_status fail(cpvs_status s, const std::string&) { return s; }
cpvs_status cuda_fail(cudaError_t e, const char*) {
    return e == cudaErrorMemoryAllocation ? CPVS_ERR_OOM : CPVS_ERR_DEVICE;
}
}  // namespace cpvs

using model::MiB;

static void check(bool ok, const char* what) {
    if (ok) return;
    std::printf("failed: %s\n", what);
    std::exit(1);
}

static void begin(cpvs::Ctx& c) { cpvs::create_pool(0, &c.pool, ~0ull); }

// Under a budget nothing is held outside the budget's own pool.
static void budget() {
    cpvs::Ctx c;
    begin(c);
    void* p = nullptr;
    check(c.alloc(&p, 64 * MiB, true, nullptr, c.index_source(64 * MiB)) == CPVS_OK, "an index without a budget");
    c.release(p, 64 * MiB, true, nullptr);
    void* held = nullptr;
    check(c.alloc(&held, 64 * MiB, true, nullptr, c.index_source(64 * MiB)) == CPVS_OK, "an index without a budget");
    c.set_budget(200 * MiB);
    check(c.index_source(64 * MiB) == nullptr, "an index under a budget comes from the context's pool");
    check(model::reserved() == 64 * MiB, "freed blocks of the second pool go back with a budget");
    c.release(held, 64 * MiB, true, nullptr);
    check(model::reserved() == 0, "blocks of the second pool freed under a budget go back");
    for (int k = 0; k < 4; ++k) {
        check(c.alloc(&p, 64 * MiB, true, nullptr, c.index_source(64 * MiB)) == CPVS_OK, "an index under a budget");
        c.release(p, 64 * MiB, true, nullptr);
        check(c.alloc(&p, 200 * MiB, true, nullptr) == CPVS_OK, "the whole budget");
        c.release(p, 200 * MiB, true, nullptr);
    }
    check(model::reserved() <= 200 * MiB, "the device memory held stays within the budget");
}

// What is free in one pool is there for the other where the device has no more.
static void full() {
    cpvs::Ctx c;
    begin(c);
    void *p = nullptr, *q = nullptr;
    cudaMemPool_t second = c.index_source(64 * MiB);
    check(second != nullptr, "a second pool");
    check(c.alloc(&p, 1000 * MiB, false, nullptr) == CPVS_OK, "a large scratch");
    c.release(p, 1000 * MiB, false, nullptr);
    check(c.alloc(&p, 64 * MiB, true, nullptr, second) == CPVS_OK, "an index after it");
    c.release(p, 64 * MiB, true, nullptr);
    check(c.alloc(&p, 1000 * MiB, false, nullptr) == CPVS_OK, "the scratch again");
    check(c.alloc(&q, 64 * MiB, true, nullptr, second) == CPVS_ERR_OOM, "no room for both");
    c.release(p, 1000 * MiB, false, nullptr);
}

// The second pool is made for the first large index alone.
static void pool_when_needed() {
    cpvs::Ctx c;
    begin(c);
    for (uint64_t b = 1 << 10; b <= 8 * MiB; b *= 8)
        check(c.index_source(b) == nullptr, "a small index comes from the context's pool");
    check(model::pools.size() == 1, "no pool before it is needed");
    check(c.index_source(64 * MiB) != nullptr, "a pool for a large index");
    check(c.index_source(64 * MiB) == c.index_pool && model::pools.size() == 2, "one such pool");
    check(c.index_source(8 * MiB) == nullptr, "still none for a small index");
}

// A lookup's tuned variant is kept by what sets its work, and not for batches
// too small to time.
static void lookup_choice() {
    cpvs::Ctx c;
    c.num_sms = 152;
    std::map<int*, std::vector<int>> places;
    for (int levels = 2; levels <= 17; ++levels)
        for (int depth = 0; depth <= 8 && depth < levels; ++depth)
            for (int k = 0; k < 8; ++k) {
                check(!c.lookup_choice(levels, depth, k & 1, k & 2, k & 4, 500), "a small batch is not timed");
                check(!c.lookup_choice(levels, depth, k & 1, k & 2, k & 4, 1 << 18), "a small batch is not timed");
                places[c.lookup_choice(levels, depth, k & 1, k & 2, k & 4, 1 << 20)].push_back(8 * (levels - depth) + k);
            }
    check(places.size() == 17 * 8 && !places.count(nullptr), "a place for every kind");
    for (const auto& p : places)
        for (int kind : p.second) check(kind == p.second[0], "one kind to a place");
}

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "budget") budget();
    else if (what == "full") full();
    else if (what == "pool_when_needed") pool_when_needed();
    else if (what == "lookup_choice") lookup_choice();
    else return 2;
    std::printf("ok\n");
    return 0;
}
