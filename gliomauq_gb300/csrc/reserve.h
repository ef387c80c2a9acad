// Device buffers that a faster path needs together: all of them or none, so that a
// failed allocation leaves nothing behind that a later call takes for the whole.
#pragma once
#include <cstddef>
#include <initializer_list>

namespace gbg {

struct Want {
    void **p;  // null: not allocated yet
    size_t bytes;
};

// allocate(void **, size_t) -> success; release(void *)
template <class Allocate, class Release>
bool reserve_all(std::initializer_list<Want> want, Allocate allocate, Release release) {
    for (const Want &w : want) {
        if (*w.p || allocate(w.p, w.bytes)) continue;
        *w.p = nullptr;  // whatever a failed allocation wrote
        for (const Want &v : want) {
            if (*v.p) release(*v.p);
            *v.p = nullptr;
        }
        return false;
    }
    return true;
}

}  // namespace gbg
