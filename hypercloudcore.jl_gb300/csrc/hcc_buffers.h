#pragma once
// hcc_buffers.h — device buffers that a context keeps while it is given cloud after cloud and list after list.
//
// A moving grid rebuilds its geometry at every stage and its lists after every step; allocating and releasing their
// buffers each time took 2.2 of the 8.8 ms of three moving 2-D FP64 steps on 15k particles. A buffer is reused where it
// has room and is at most a quarter larger than what is asked for. Buffers belong to a group (0 the cloud, 1 its lists,
// 2 the geometry), and what is rebuilt replaces its group and those after it: the buffers of these are stale until they
// are asked for again. Stale buffers are all that is given up when memory is short, before a failure is reported, so a
// call that would fit into memory with every replaced buffer released succeeds.
#include <cstddef>
#include <cstring>
#include <unordered_map>

namespace hcc {

// Memory: int allocate(void **p, size_t bytes) (0: done), void release(void *p).
template <typename Memory> class KeptBuffers {
public:
    // The buffers of `group` and of the groups after it are about to be rebuilt.
    void begin(int group) {
        for (auto &e : entries_)
            if (e.second.group >= group) e.second.stale = true;
    }
    void release_stale() {
        for (auto &e : entries_)
            if (e.second.stale) drop(e.first, e.second);
    }
    // Room for `bytes` in the buffer whose pointer is the member at `owner`; `spare` more bytes where memory has to be
    // allocated and there is enough. The allocator's error, 0: none.
    int reserve(void *owner, size_t bytes, size_t spare, int group) {
        bytes = bytes ? bytes : 1;
        Entry &e = entries_[owner];
        e.group = group;
        e.stale = false;
        if (pointer(owner) && e.size >= bytes && e.size - bytes <= bytes / 4 + spare) return 0;
        drop(owner, e);
        int err = 1;
        for (int attempt = 0; attempt < 2 && err; ++attempt) {
            if (attempt) release_stale();
            for (const size_t size : {bytes + spare, bytes}) {
                void *p = nullptr;
                err = memory_.allocate(&p, size);
                if (!err) {
                    e.size = size;
                    std::memcpy(owner, &p, sizeof(p));
                    break;
                }
                if (!spare) break;
            }
        }
        return err;
    }

private:
    struct Entry { size_t size = 0; int group = 0; bool stale = false; };
    static void *pointer(const void *owner) {
        void *p;
        std::memcpy(&p, owner, sizeof(p));
        return p;
    }
    void drop(void *owner, Entry &e) {
        void *p = pointer(owner);
        if (p) memory_.release(p);
        p = nullptr;
        std::memcpy(owner, &p, sizeof(p));
        e.size = 0;
    }
    std::unordered_map<void *, Entry> entries_;
    Memory memory_;
};

}  // namespace hcc
