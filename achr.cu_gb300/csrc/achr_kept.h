// Buffers that are replaced as they grow, of an owner whose work may be captured into CUDA graphs (host only).
//
// A graph holds the addresses of the buffers its capture used for as long as it
// may be replayed, so buffers that a capture has seen stay allocated, unused,
// until their owner goes; others are freed before the larger ones are allocated.
#pragma once
#include <memory>
#include <utility>
#include <vector>

namespace achr {

template <class T>
class Kept {
public:
    T *get() const { return cur_.get(); }
    // A capture that is under way uses the present buffers.
    void captured() { seen_ = cur_ != nullptr; }
    // Ends the use of the present buffers, before their replacement is made.
    void retire() {
        if (seen_) old_.push_back(std::move(cur_));
        cur_.reset();
        seen_ = false;
    }
    T *replace(std::unique_ptr<T> next) {
        retire();
        cur_ = std::move(next);
        return cur_.get();
    }

private:
    std::unique_ptr<T> cur_;
    std::vector<std::unique_ptr<T>> old_;
    bool seen_ = false;
};

}  // namespace achr
