// Checks csrc/kept_memory.h on the CPU with a counting stand-in of the device memory; prints
// "ok" or what failed.
#include <cstdio>
#include <cstdlib>
#include <thread>

#include "kept_memory.h"

using lbdem::KeptMemory;

static void check(bool ok, const char* what) {
    if (!ok) {
        std::printf("failed: %s\n", what);
        std::exit(1);
    }
}

int main() {
    int freed = 0;
    const auto drop = [&](void*) { ++freed; };
    char mem[8];
    KeptMemory k(70, 100);
    int a = 0, b = 0, c = 0;
    check(k.take(&a).p == nullptr, "nothing kept at first");
    check(!k.keep({mem, 71, 0, &a}), "the bound of one block");
    check(k.keep({mem, 60, 0, &a}), "a block within the bounds");
    check(!k.keep({mem + 1, 41, 0, &b}), "the bound holds over all owners");
    check(k.keep({mem + 1, 40, 1, &b}), "up to the bound");
    check(k.held(&a) == 60 && k.held(&b) == 40 && k.held(&c) == 0, "held bytes");
    check(k.take(&a).p == mem && k.take(&a).p == nullptr, "a block in use is not here");
    check(!k.give_back(0, drop) && freed == 0, "nor given back");
    check(k.keep({mem, 60, 0, &a}), "back after use");
    check(k.give_back(0, drop) && freed == 1 && k.held(&a) == 0, "given back by device");
    check(k.held(&b) == 40, "the other device's stays");
    check(k.take(&b).bytes == 40 && !k.give_back(1, drop), "empty again");
    // owners on several threads, and one that gives back: every block is freed once
    static int alive[4] = {0, 0, 0, 0};
    KeptMemory t(1000, 1000);
    std::thread work[5];
    for (int n = 0; n < 4; ++n)
        work[n] = std::thread([n, &t] {
            for (int r = 0; r < 20000; ++r) {
                KeptMemory::Block q = t.take(&alive[n]);
                if (!q.p) q = {&alive[n], 100, 0, &alive[n]}, ++alive[n];
                if (alive[n] != 1) std::printf("failed: block of owner %d\n", n), std::exit(1);
                if (!t.keep(q)) --alive[n];
            }
        });
    work[4] = std::thread([&t] {
        for (int r = 0; r < 20000; ++r) t.give_back(0, [](void* p) { --*(int*)p; });
    });
    for (auto& w : work) w.join();
    t.give_back(0, [](void* p) { --*(int*)p; });
    for (int v : alive) check(v == 0, "every block freed once");
    std::printf("ok\n");
}
