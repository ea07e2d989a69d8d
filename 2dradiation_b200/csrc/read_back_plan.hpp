// Which values a read-back moves: of nq arrays of `per` values, one after
// another on the device, those that are wanted, in chunks of at most `chunk`
// values.
#pragma once
#include <algorithm>
#include <cstdint>

namespace grlbm
{
class ReadBackPlan
{
public:
    static constexpr int kMaxArrays = 8;
    // dst[q]: where array q goes, null if it is not wanted; nq <= kMaxArrays
    ReadBackPlan(double *const *dst, int nq, int64_t per, int64_t chunk) : per_(per), chunk_(chunk)
    {
        for (int q = 0; q < nq; q++)
            if (dst[q])
                wanted_[n_++] = q;
    }
    int64_t values() const { return n_ * per_; }
    int64_t chunks() const { return (values() + chunk_ - 1) / chunk_; }
    // f(array, first value in it, values, place in the chunk) for the parts of chunk k
    template <class F>
    void parts(int64_t k, F f) const
    {
        const int64_t first = k * chunk_, end = std::min(values(), first + chunk_);
        for (int64_t at = first; at < end;)
        {
            const int64_t w = at / per_, stop = std::min(end, (w + 1) * per_);
            f(wanted_[w], at - w * per_, stop - at, at - first);
            at = stop;
        }
    }
    // f(first value on the device, values, place in the chunk) for the
    // contiguous runs of chunk k
    template <class F>
    void copies(int64_t k, F f) const
    {
        const int64_t first = k * chunk_, end = std::min(values(), first + chunk_);
        for (int64_t at = first; at < end;)
        {
            int64_t w = at / per_;
            const int64_t from = wanted_[w] * per_ + (at - w * per_);
            while (w + 1 < n_ && (w + 1) * per_ < end && wanted_[w + 1] == wanted_[w] + 1)
                w++;
            const int64_t stop = std::min(end, (w + 1) * per_);
            f(from, stop - at, at - first);
            at = stop;
        }
    }

private:
    int wanted_[kMaxArrays] = {};
    int n_ = 0;
    int64_t per_, chunk_;
};
} // namespace grlbm
