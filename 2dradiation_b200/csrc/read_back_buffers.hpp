// Page-locked buffers through which results reach pageable host memory.  A
// read-back takes one for its duration; up to kKept idle ones wait per device,
// also while it has no context of this library (page-locking one takes 2 ms,
// more than most read-backs).  They belong to a CUDA context: a reset of the
// device frees them behind our back, so every buffer is kept with the number
// of the CUDA context that it was allocated in, which is never used again, and
// those of another number are forgotten.
#pragma once
#include <cstddef>
#include <exception>
#include <mutex>
#include <vector>

namespace grlbm
{
class ReadBackBuffers
{
public:
    static constexpr size_t kKept = 4;
    // where a buffer lives: a device and the number of its CUDA context
    struct Place
    {
        int device;
        unsigned long long context;
    };
    // alloc returns null where no buffer can be had
    ReadBackBuffers(char *(*alloc)(), void (*release)(char *)) : alloc_(alloc), release_(release) {}

    char *take(Place at)
    {
        {
            std::lock_guard<std::mutex> lock(mutex_);
            forget_stale(at);
            for (size_t k = idle_.size(); k-- > 0;)
                if (idle_[k].at.device == at.device)
                {
                    char *p = idle_[k].p;
                    idle_.erase(idle_.begin() + (std::ptrdiff_t)k);
                    return p;
                }
        }
        return alloc_();
    }
    // (a buffer goes back to the place that it was taken at)
    void give(Place at, char *p)
    {
        try
        {
            std::lock_guard<std::mutex> lock(mutex_);
            forget_stale(at);
            size_t kept = 0;
            for (const Idle &b : idle_)
                kept += b.at.device == at.device;
            if (kept < kKept)
            {
                idle_.push_back(Idle{at, p});
                return;
            }
        }
        catch (const std::exception &) // no host memory for the list: not kept
        {
        }
        release_(p);
    }

private:
    struct Idle
    {
        Place at;
        char *p;
    };
    void forget_stale(Place at)
    {
        size_t n = 0;
        for (const Idle &b : idle_)
            if (b.at.device != at.device || b.at.context == at.context)
                idle_[n++] = b;
        idle_.resize(n, Idle{at, nullptr});
    }
    char *(*alloc_)();
    void (*release_)(char *);
    std::mutex mutex_;
    std::vector<Idle> idle_;
};
} // namespace grlbm
