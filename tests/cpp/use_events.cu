// The events of objects' last uses: each comes from its object's context and
// goes back there, under that context's mutex, also where one call uses objects
// of several contexts.  Stands in for the context's two event calls; no GPU.
#include <cstdio>
#include <cstdlib>
#include <map>
#include <thread>

#include "../../cpvs_gb300/csrc/objects.h"

static std::map<const cpvs::Ctx*, int> taken, given;

static void check(bool ok, const char* what) {
    if (ok) return;
    std::printf("failed: %s\n", what);
    std::exit(1);
}

static void check_locked(cpvs::Ctx* c) {
    bool got = false;
    std::thread([&] {
        got = c->event_mutex.try_lock();
        if (got) c->event_mutex.unlock();
    }).join();
    check(!got, "an event call outside its context's mutex");
}

// (no event at all: the record is left out)
cudaEvent_t cpvs::Ctx::take_event() {
    check_locked(this);
    ++taken[this];
    return nullptr;
}
void cpvs::Ctx::give_event(cudaEvent_t) {
    check_locked(this);
    ++given[this];
}

int main() {
    cpvs_ctx a, b;
    for (int order = 0; order < 2; ++order) {
        auto *a0 = new cpvs_hierarchy(&a), *a1 = new cpvs_hierarchy(&a);
        auto *b0 = new cpvs_hierarchy(&b), *b1 = new cpvs_hierarchy(&b);
        cpvs_hierarchy* mixed[] = {a0, b0, a1, b1, a0};
        DeviceObject::touch_all(mixed, 5, nullptr);
        b0->touch(nullptr);
        DeviceObject::touch_all(mixed + 1, 4, nullptr);
        if (order) {
            delete a0, delete a1, delete b0, delete b1;
        } else {
            delete b1, delete b0, delete a1, delete a0;
        }
        check(taken[&a.c] == given[&a.c] && taken[&b.c] == given[&b.c], "every event back in its own context");
        check(taken[&a.c] > 0 && taken[&b.c] > 0, "both contexts gave events");
    }
    std::printf("ok\n");
    return 0;
}
