// launch_fits.h -- CTAs per SM of the launch shapes used lately.
#pragma once

#include <cstddef>
#include <mutex>
#include <vector>

namespace mgv {

// Bounded, and searched from the front: most kernels have a handful of shapes,
// but the staging tiles' shared memory follows the number of table regions, so
// a process that builds tables of many sizes would add thousands of entries
// that every later launch had to pass (a search of 20,000 takes 15 us, of 64 0.06).
// A shape that is not there is asked of the runtime (2 to 3 us) and takes the
// oldest one's place.
class LaunchFits {
public:
    static constexpr size_t kMost = 64;

    bool find(const void* kernel, int block, size_t smem, int* per_sm) const {
        std::lock_guard<std::mutex> lk(mu_);
        for (const Fit& f : fits_)
            if (f.kernel == kernel && f.block == block && f.smem == smem) {
                *per_sm = f.per_sm;
                return true;
            }
        return false;
    }

    void add(const void* kernel, int block, size_t smem, int per_sm) {
        std::lock_guard<std::mutex> lk(mu_);
        if (fits_.size() < kMost) fits_.push_back(Fit{kernel, block, smem, per_sm});
        else fits_[next_++ % kMost] = Fit{kernel, block, smem, per_sm};
    }

    size_t size() const {
        std::lock_guard<std::mutex> lk(mu_);
        return fits_.size();
    }

private:
    struct Fit {
        const void* kernel;
        int block;
        size_t smem;
        int per_sm;
    };
    mutable std::mutex mu_;
    std::vector<Fit> fits_;
    size_t next_ = 0;
};

}  // namespace mgv
