// csrc/reserve.h over an allocator that fails: every buffer or none, whichever one
// fails, on the first call and on a later one. Prints "ok", or what went wrong.
#include <cstdio>
#include <set>

#include "reserve.h"

int main() {
    for (int have = 0; have < 2; ++have)
        for (int fails = 0; fails < 3; ++fails) {
            char pool[8];
            std::set<void *> live;
            int calls = 0, next = 0, bad = -1;
            auto allocate = [&](void **p, size_t) {
                if (calls++ == bad) {
                    *p = pool + 7;  // a failed call may write anything
                    return false;
                }
                live.insert(*p = pool + next++);
                return true;
            };
            auto release = [&](void *p) {
                if (!live.erase(p)) std::printf("released what is not allocated\n"), next = 100;
            };
            void *a = nullptr, *b = nullptr, *c = nullptr;
            auto all = [&] { return gbg::reserve_all({{&a, 1}, {&b, 2}, {&c, 3}}, allocate, release); };
            if (have) {  // the first of them is there already
                allocate(&a, 1);
                calls = 0;
            }
            bad = fails;
            const bool ok = all();
            if (ok != (have && fails == 2)) return std::printf("have %d fails %d: said %d\n", have, fails, ok), 1;
            if (!ok && (a || b || c || !live.empty())) return std::printf("have %d fails %d: something is left\n", have, fails), 1;
            bad = -1;
            if (!all() || !a || !b || !c || live.size() != 3) return std::printf("have %d fails %d: no second try\n", have, fails), 1;
            const int n = calls;
            if (!all() || calls != n || next >= 100) return std::printf("have %d fails %d: allocated again\n", have, fails), 1;
        }
    std::puts("ok");
    return 0;
}
