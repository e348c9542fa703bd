// Host harness for gsofa_scratch.hpp: a device of `room` bytes behind it.
#include "../gsofa_b200/csrc/gsofa_scratch.hpp"

#include <cstdio>
#include <cstdlib>
#include <map>

struct NoRoom {};

struct FakeDevice {
    static inline size_t room = 0, used = 0;
    static inline std::map<void *, size_t> live;
    static void *alloc(size_t bytes)
    {
        if (used + bytes > room) return nullptr;
        void *p = std::malloc(1);
        live[p] = bytes;
        used += bytes;
        return p;
    }
    static void free(void *p)
    {
        used -= live.at(p);
        live.erase(p);
        std::free(p);
    }
    static void no_room() { throw NoRoom{}; }
};

using gsofa::DevBuf;
using Scratch = gsofa::Scratch<FakeDevice>;

#define CHECK(x)                                                              \
    do {                                                                      \
        if (!(x)) {                                                           \
            std::printf("line %d: %s\n", __LINE__, #x);                       \
            std::exit(1);                                                     \
        }                                                                     \
    } while (0)

template <class F>
bool refused(F f)
{
    try {
        f();
    } catch (NoRoom &) {
        return true;
    }
    return false;
}

int main()
{
    // every budget and device size around what a job takes: the addresses that
    // it holds are live when its last buffer is in place, whichever buffers of
    // it are dispensable
    for (size_t limit = 0; limit < 2; limit++)
        for (size_t total = 9000; total <= 14000; total += 50) {
            FakeDevice::room = limit ? total : 1 << 20;
            Scratch s;
            s.budget = limit ? 1 << 20 : total;
            DevBuf trav, snap, mats, ranges, other;
            s.dispensable = {&snap, &trav};
            s.grow(other, 1000);
            for (size_t batch = 300; batch <= 1500; batch += 300) {   // each job larger than the last
                const bool no = refused([&] {
                    Scratch::Job job(s);
                    void *t = job.take(trav, 6000), *k = job.take(snap, 2000);
                    void *m = job.take(mats, batch), *r = job.take(ranges, batch);
                    for (void *p : {t, k, m, r}) CHECK(FakeDevice::live.count(p));
                    CHECK(t == trav.p && k == snap.p && m == mats.p && r == ranges.p && s.idle() == 0);
                });
                CHECK(no == (9000 + 2 * batch > total));
                CHECK(s.held <= s.budget && s.held == FakeDevice::used);
                CHECK(!trav.taken && !snap.taken && !mats.taken);
            }
            for (DevBuf *b : {&trav, &snap, &mats, &ranges, &other}) s.release(*b);
            CHECK(FakeDevice::used == 0 && s.held == 0);
        }
    // what a job left gives way to anything else, in order, whether the budget
    // or the device is short; not to a buffer that holds it itself, nor while
    // a job has it
    for (size_t limit = 0; limit < 2; limit++) {
        FakeDevice::room = limit ? 10000 : 1 << 20;
        Scratch s;
        s.budget = limit ? 1 << 20 : 10000;
        DevBuf snap, trav, order;
        s.dispensable = {&snap, &trav};
        {
            Scratch::Job job(s);
            job.take(trav, 6000);
            job.take(snap, 3000);
            CHECK(s.idle() == 0);
            CHECK(refused([&] { s.grow(order, 3000); }));
            if (limit) CHECK(refused([&] { s.alloc(3000); }));
        }
        CHECK(s.idle() == 9000);
        CHECK(!refused([&] { s.grow(order, 3000); }) && !snap.p && trav.p);
        CHECK(!refused([&] { s.grow(order, 9000); }) && !trav.p);
        CHECK(!refused([&] { s.grow(snap, 1000); }) && refused([&] { s.grow(snap, 1001 + 1000); }));
        s.release(order);
        if (limit) {
            s.grow(trav, 5000);
            void *p = s.alloc(6000);
            CHECK(p && !trav.p);
            FakeDevice::free(p);
        }
        for (DevBuf *b : {&snap, &trav, &order}) s.release(*b);
        CHECK(FakeDevice::used == 0);
    }
    std::printf("ok\n");
    return 0;
}
