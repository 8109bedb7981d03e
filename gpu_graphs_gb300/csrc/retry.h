// retry.h -- when to try an optional allocation again (host only).
#pragma once

namespace gbfs {

// What a graph may do without (its fixed-width rows, the pieces of its long rows)
// is built by the call that could first use it.  Where that failed, most likely
// for lack of memory, the next call does not pay for the same refusal, nor do the
// next two, four, ... after further ones, up to MAX_SKIP; a success starts over.
class Retry {
public:
    static constexpr unsigned MAX_SKIP = 1024;

    // True when the caller should try now.
    bool due()
    {
        if (!skip_) return true;
        --skip_;
        return false;
    }
    void failed()
    {
        skip_ = next_;
        if (next_ < MAX_SKIP) next_ *= 2;
    }
    void succeeded() { next_ = 1; }

private:
    unsigned skip_ = 0, next_ = 1;
};

}  // namespace gbfs
