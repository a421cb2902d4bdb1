// Checks kept.h against a device that is a counter on the host (tests/test_kept_arrays.py):
// prints what went wrong, or nothing.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <set>
#include <thread>

#include "kept.h"

using sphk::KeptArrays;
using sphk::malloc_or_give_back;

static int wrong = 0;
static void expect(bool good, const char *what)
{
    if (good) return;
    ++wrong;
    std::printf("%s\n", what);
}

// A device of `room` bytes; freeing what is not allocated is an error.
struct Fake {
    std::mutex m;
    std::set<void *> live;
    size_t used = 0, room;
    static constexpr size_t SIZE = 10;
    explicit Fake(size_t r) : room(r) {}
    void *allocate()
    {
        std::lock_guard<std::mutex> lock(m);
        if (used + SIZE > room) return nullptr;
        void *p = std::malloc(1);
        live.insert(p);
        used += SIZE;
        return p;
    }
    void release(void *p)
    {
        std::lock_guard<std::mutex> lock(m);
        if (live.erase(p) != 1) {
            ++wrong;
            std::printf("freed twice\n");
            return;
        }
        std::free(p);
        used -= SIZE;
    }
};

int main()
{
    int a, b, c;   // owners
    {
        Fake dev(100);
        KeptArrays kept;
        auto free_one = [&](void *p) { dev.release(p); };
        std::vector<void *> own{dev.allocate(), dev.allocate()};
        const std::vector<void *> same = own;
        expect(!kept.park(&a, 0, own, 20, 19) && own.size() == 2, "parked past the limit");
        expect(kept.park(&a, 0, own, 20, 40) && own.empty() && kept.parked(&a) == 20, "not parked");
        std::vector<void *> more{dev.allocate(), dev.allocate(), dev.allocate()};
        expect(!kept.park(&b, 0, more, 30, 40), "the limit is not the device's");
        expect(kept.park(&b, 1, more, 30, 40), "another device's arrays count");
        expect(kept.take(&c, own) == 0 && own.empty(), "a stranger took arrays");
        expect(kept.take(&a, own) == 20 && own == same, "other arrays came back");
        expect(kept.take(&a, own) == 0 && own == same, "came back twice");
        expect(kept.park(&a, 0, own, 20, 40), "not parked again");

        // the device fills up: the next allocation takes what is parked on device 0
        std::vector<void *> others;
        while (void *p = dev.allocate()) others.push_back(p);
        int tries = 0;
        auto allocate = [&]() -> void * { ++tries; return dev.allocate(); };
        void *p = malloc_or_give_back(allocate, (void *)nullptr, [&] { return kept.give_back(0, free_one); });
        expect(p != nullptr && tries == 2, "the second try failed");
        expect(kept.take(&a, own) == 0 && own.empty(), "freed arrays came back");
        others.push_back(p);
        while (void *q = dev.allocate()) others.push_back(q);
        tries = 0;
        p = malloc_or_give_back(allocate, (void *)nullptr, [&] { return kept.give_back(0, free_one); });
        expect(p == nullptr && tries == 1, "tried again with nothing freed");
        expect(kept.parked(&b) == 30 && kept.give_back(1, free_one) == 30, "device 1's arrays are gone");
        for (void *q : others) dev.release(q);
        expect(dev.used == 0, "memory is lost");
    }
    {
        // owners that park and take in threads, beside allocations that fail
        Fake dev(400);
        KeptArrays kept;
        std::atomic<bool> stop{false};
        std::vector<std::thread> threads;
        auto free_one = [&](void *p) { dev.release(p); };
        for (int t = 0; t < 8; ++t)
            threads.emplace_back([&] {
                int me;
                std::vector<void *> own;
                for (int k = 0; k < 3000; ++k) {
                    if (kept.take(&me, own) == 0)
                        while (own.size() < 4) {
                            void *p = malloc_or_give_back([&] { return dev.allocate(); }, (void *)nullptr,
                                                          [&] { return kept.give_back(0, free_one); });
                            if (p) own.push_back(p);
                            else std::this_thread::yield();
                        }
                    expect(own.size() == 4, "half a set");
                    if (!kept.park(&me, 0, own, 40, 200)) {
                        for (void *p : own) dev.release(p);
                        own.clear();
                    }
                }
                kept.take(&me, own);
                for (void *p : own) dev.release(p);
            });
        std::thread thief([&] {
            while (!stop) kept.give_back(0, free_one);
        });
        for (auto &t : threads) t.join();
        stop = true;
        thief.join();
        expect(dev.used == 0 && dev.live.empty(), "memory is lost between threads");
    }
    return wrong;
}
