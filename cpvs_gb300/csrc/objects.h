// Handle types behind the C ABI, shared by the translation units that
// implement it (capi.cu, server.cu).
#pragma once

#include <mutex>
#include <vector>

#include "common.cuh"

struct cpvs_ctx {
    cpvs::Ctx c;
};

// The event of an object's last use, from the context's pool.  The objects of
// one batch share one until they are used apart.  Guarded by the context's
// event mutex (handles may be read from several host threads).
struct UseEvent {
    cudaEvent_t event;
    uint32_t refs;
};

// Every object with device memory records its last use on the stream of each
// call that enqueues work on it; its memory is freed after that event.
struct DeviceObject {
    explicit DeviceObject(cpvs::Ctx* c) : c_(c) {}
    DeviceObject(const DeviceObject&) = delete;
    DeviceObject& operator=(const DeviceObject&) = delete;
    ~DeviceObject() {
        std::lock_guard<std::mutex> lock(c_->event_mutex);
        drop(use_);
        drop(index_);
    }
    void touch(cudaStream_t st) const {
        std::lock_guard<std::mutex> lock(c_->event_mutex);
        if (!use_ || use_->refs > 1) {
            drop(use_);
            use_ = new UseEvent{c_->take_event(), 1u};
        }
        if (use_->event) cudaEventRecord(use_->event, st);
    }
    // One record for all of `objects` of the first one's context; those of
    // another one (a batch may build from several contexts' hierarchies) have
    // their own, from that context's pool and under its mutex.
    template <class T>
    static void touch_all(T* const* objects, size_t count, cudaStream_t st) {
        record_all(objects, count, st, false);
    }
    // touch_all after `st` was given the work that makes the objects' indices:
    // until it is done, the uses of an index on other streams wait for it.
    template <class T>
    static void indexed_all(T* const* objects, size_t count, cudaStream_t st) {
        record_all(objects, count, st, true);
    }
    // Before a use of the indices of `objects` (of one context) on `st`, the
    // context's index mutex held.  (A capturing stream takes no wait for work
    // outside its capture: what it records runs later.)
    template <class T>
    static void await_indices(T* const* objects, size_t count, cudaStream_t st) {
        for (size_t i = 0; i < count; ++i) {
            const DeviceObject& o = *objects[i];
            if (!o.index_ || st == o.index_stream_ || !o.index_->event) continue;
            if (cpvs::capturing(st)) return;
            std::lock_guard<std::mutex> lock(o.c_->event_mutex);
            if (cpvs::reached(o.index_->event)) {
                o.drop(o.index_);
                continue;
            }
            cudaStreamWaitEvent(st, o.index_->event, 0);
        }
    }

private:
    template <class T>
    static void record_all(T* const* objects, size_t count, cudaStream_t st, bool index) {
        if (!count) return;
        cpvs::Ctx* c = objects[0]->c_;
        uint32_t mine = 0;
        for (size_t i = 0; i < count; ++i) {
            if (objects[i]->c_ == c)
                ++mine;
            else
                objects[i]->touch(st);
        }
        std::lock_guard<std::mutex> lock(c->event_mutex);
        auto* u = new UseEvent{c->take_event(), index ? 2 * mine : mine};
        if (u->event) cudaEventRecord(u->event, st);
        for (size_t i = 0; i < count; ++i) {
            if (objects[i]->c_ != c) continue;
            objects[i]->drop(objects[i]->use_);
            objects[i]->use_ = u;
            if (!index) continue;
            objects[i]->drop(objects[i]->index_);
            objects[i]->index_ = u;
            objects[i]->index_stream_ = st;
        }
    }

public:
    cudaEvent_t last_use() const {
        std::lock_guard<std::mutex> lock(c_->event_mutex);
        return use_ ? use_->event : nullptr;
    }

private:
    void drop(UseEvent*& u) const {
        if (u && --u->refs == 0) {
            c_->give_event(u->event);
            delete u;
        }
        u = nullptr;
    }
    cpvs::Ctx* c_;
    mutable UseEvent* use_ = nullptr;
    mutable UseEvent* index_ = nullptr;  // after the object's index, until that is known to be done
    mutable cudaStream_t index_stream_ = nullptr;
};

struct cpvs_hierarchy : DeviceObject {
    explicit cpvs_hierarchy(cpvs_ctx* x) : DeviceObject(&x->c), ctx(x) {}
    cpvs_ctx* ctx;
    uint32_t n = 0;
    float* depth = nullptr;    // device n*n
    bool owns_depth = true;    // false when borrowed from the caller
    float2* levels = nullptr;  // device pyramid
    int first_level = 1;       // lowest pyramid level stored (a build's temporary hierarchy may skip some)
    uint64_t bytes = 0;
};

// Device block holding the DAGs of one build (one or many jobs back to
// back, followed by kDagPad zeroed words).  Shared by the shadows (and the
// grid) that point into it; freed when the last of them lets go, after every
// holder's last use.
struct DagBlock {
    cpvs_ctx* ctx = nullptr;
    uint32_t* base = nullptr;
    uint64_t bytes = 0;
    int refs = 0;
};

inline void block_unref(DagBlock* b, cudaEvent_t last_use) {
    if (!b) return;
    cpvs::Ctx& c = b->ctx->c;
    c.await_use(last_use);  // the free waits for every holder
    if (--b->refs == 0) {
        c.release(b->base, b->bytes, true, nullptr, nullptr);
        delete b;
    }
}

struct cpvs_shadow : DeviceObject {
    explicit cpvs_shadow(cpvs_ctx* x) : DeviceObject(&x->c), ctx(x) {}
    cpvs_ctx* ctx;
    DagBlock* block = nullptr;
    uint32_t* dag = nullptr;   // inside block; at least kDagPad readable words follow it
    uint64_t words = 0;
    uint32_t* top = nullptr;   // dense top index for lookups, built on the first lookup
    uint64_t top_bytes = 0;
    int top_depth = 0;         // levels below the root that `top` resolves
    uint64_t top_beyond = 0;   // top_bytes where they are more than the DAG's size allows, else 0
    uint32_t num_levels = 0;
    bool leafmasks = false;
    uint32_t root_mask = 0;
    std::vector<uint64_t> tree, uniq;
    const cpvs_grid* owner = nullptr;  // the grid whose cell holds it (and destroys it)
};

struct cpvs_grid : DeviceObject {
    explicit cpvs_grid(cpvs_ctx* x) : DeviceObject(&x->c), ctx(x) {}
    cpvs_ctx* ctx;
    uint32_t length = 0;
    std::vector<cpvs_shadow*> cells;
    DagBlock* block = nullptr;  // the combined DAG
    uint32_t* dag = nullptr;
    uint64_t words = 0;
    uint32_t* cell_words = nullptr;
    uint32_t dag_levels = 0;
    bool leafmasks = false;
    bool finalized = false;
    uint32_t filter_size = 1;  // PCF footprint of evaluate
    uint32_t* gtop = nullptr;  // grid top index, built on the first lookup
    uint64_t gtop_bytes = 0;   // ~0: none (too small, or its allocation failed)
    int gtop_depth = 0;
};


namespace cpvs {
// The address under which the GPU reads host memory `p` in place, or null.
void* host_accessible(const Ctx& c, const void* p);
// Builds the shadow's lookup top grid if it has none yet (stream-ordered,
// on the context's thread).
void shadow_ensure_top(const cpvs_shadow* s, cudaStream_t st, uint32_t max_factor);
// The shadow as an entry of a multi-DAG lookup table (with its top grid).
MultiDag shadow_table_entry(const cpvs_shadow* s);
// A hierarchy that only feeds builds with the given flags (destroyed after
// them): with leafmasks, pyramid levels 1 and 2 are not stored.  With
// `host_read`, a host map read in place is not waited for: the event
// recorded after the read is returned, and the caller waits for it before
// its own caller may reuse the map.
cpvs_status hierarchy_create_for_build(cpvs_ctx* ctx, const float* depth, uint32_t n, uint32_t flags,
                                       uint32_t build_flags, void* stream, cpvs_hierarchy** out,
                                       cudaEvent_t* host_read = nullptr);
}  // namespace cpvs
