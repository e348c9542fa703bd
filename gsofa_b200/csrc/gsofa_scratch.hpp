// gsofa_scratch.hpp -- a context's device scratch within its memory budget
// (host only; the device allocator is a parameter, so the rules can be tested
// without one).
//
// Every buffer grows and is kept for the next job.  Dispensable buffers, which
// the next job can make again, give way to whatever needs the room, but never
// while a job that is being set up or is running has taken them: what a job has
// its addresses from stays.
#pragma once

#include <algorithm>
#include <cstddef>
#include <vector>

namespace gsofa {

// Grow-only device buffer owned by a context.
struct DevBuf {
    void *p = nullptr;
    size_t bytes = 0;
    bool taken = false;   // by the current job
};

// Memory: `static void *alloc(size_t)`, null when the device has no room;
// `static void free(void *)`; `static void no_room()`, which throws.
template <class Memory>
struct Scratch {
    size_t budget = 0;
    size_t held = 0;                    // bytes of scratch currently held
    std::vector<DevBuf *> dispensable;  // buffers that give way, the first one first

    void release(DevBuf &b)
    {
        if (b.p) {
            Memory::free(b.p);
            held -= b.bytes;
        }
        b.p = nullptr;
        b.bytes = 0;
    }

    // Bytes that can give way now.
    size_t idle() const
    {
        size_t bytes = 0;
        for (const DevBuf *d : dispensable) bytes += d->taken ? 0 : d->bytes;
        return bytes;
    }

    // Frees one dispensable buffer other than b that no job has taken; false
    // when there is none.
    bool give_way(const DevBuf *b)
    {
        for (DevBuf *d : dispensable)
            if (d != b && d->p && !d->taken) {
                release(*d);
                return true;
            }
        return false;
    }

    // Device memory outside the budget (b: not to be freed for it).
    void *alloc(size_t bytes, const DevBuf *b = nullptr)
    {
        void *p;
        while (!(p = Memory::alloc(bytes)))
            if (!give_way(b)) Memory::no_room();
        return p;
    }

    // At least `bytes` in b (contents are not kept).
    void *grow(DevBuf &b, size_t bytes)
    {
        bytes = std::max<size_t>(bytes, 256);
        if (b.bytes >= bytes) return b.p;
        release(b);
        while (held + bytes > budget)
            if (!give_way(&b)) Memory::no_room();
        b.p = alloc(bytes, &b);
        b.bytes = bytes;
        held += bytes;
        return b.p;
    }

    // The buffers of one job, from the first one taken until the job ends.
    struct Job {
        Scratch &of;
        std::vector<DevBuf *> bufs;
        explicit Job(Scratch &s) : of(s) {}
        Job(const Job &) = delete;
        Job &operator=(const Job &) = delete;
        ~Job()
        {
            for (DevBuf *b : bufs) b->taken = false;
        }
        void *take(DevBuf &b, size_t bytes)
        {
            void *p = of.grow(b, bytes);
            if (!b.taken) bufs.push_back(&b);
            b.taken = true;
            return p;
        }
    };
};

}  // namespace gsofa
