// The order in which the epochs of a training call take their samples: one seeded
// Fisher-Yates permutation after another, each shuffled from the one before (host code only).
//
// The device copies an epoch's order from pageable host memory, and may still read it until the
// stream has been waited for.  The next order is therefore made in a second array, while the
// device works, and the first stays as it is until advance(), which the caller calls after that
// wait.  For the same reason the object has to outlive the stream's last wait.
#pragma once

#include <cstdint>
#include <vector>

namespace nqb {

class EpochOrder {
   public:
    // The first epoch's order.
    void start(uint64_t count, uint64_t seed) {
        now_.resize(count);
        for (uint64_t i = 0; i < count; ++i) now_[i] = (uint32_t)i;
        rng_ = seed * 0x9E3779B97F4A7C15ull + 1;
        shuffle(now_);
    }
    // This epoch's order: neither moved nor written before advance().
    const uint32_t* current() const { return now_.data(); }
    // Makes the next epoch's order.
    void prepare() {
        next_ = now_;
        shuffle(next_);
    }
    // The order that prepare() made is the current one from here on.
    void advance() { now_.swap(next_); }

   private:
    uint64_t draw() {  // splitmix64
        uint64_t z = (rng_ += 0x9E3779B97F4A7C15ull);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return z ^ (z >> 31);
    }
    void shuffle(std::vector<uint32_t>& v) {  // Fisher-Yates
        for (uint64_t i = v.size() - 1; i > 0; --i) {
            const uint64_t j = draw() % (i + 1);
            const uint32_t t = v[i];
            v[i] = v[j];
            v[j] = t;
        }
    }
    std::vector<uint32_t> now_, next_;
    uint64_t rng_ = 0;
};

}  // namespace nqb
