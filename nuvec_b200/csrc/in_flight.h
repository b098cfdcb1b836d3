// What the unfinished kernels of a handle's stream may be writing (host side; no CUDA in here).
//
// A kernel launched with programmatic stream serialization starts as soon as every block of the kernel in front has
// triggered or exited, and sees that kernel's stores only behind its own griddepcontrol.wait.  Products and attention read
// weights, caches and index lists ahead of that wait.  That is sound for memory that no unfinished kernel writes, so every
// launch says what it writes, and a reader asks first:
//
//   EARLY  a block triggers before it has waited itself.  When the next kernel starts, the kernels in front of this one may
//          still be running: what is noted of them stays.
//   LATE   every block waits before it triggers (or never triggers: then its exit counts).  When the next kernel starts,
//          everything in front of this one has finished: only this one's own stores are open.
//
// A launch that says nothing leaves the window unknown, and nothing is read early until the next LATE one; a reader that may
// not read early waits first and is LATE itself, so one of them settles it.  When there is no room for a launch's ranges it has
// to go without the attribute: such a kernel starts after everything in front has finished, like a LATE one's successor.
#pragma once
#include <cstddef>
#include <initializer_list>

namespace nvc {

enum class Trigger { EARLY, LATE };

struct Writes {
    struct Range {
        const void *p;
        size_t bytes;
    };
    static constexpr int MOST = 5;
    Trigger trigger;
    Range range[MOST] = {};
    Writes(Trigger t, std::initializer_list<Range> written) : trigger(t) {
        int n = 0;
        for (const Range &r : written)
            if (n < MOST) range[n++] = r;
            else overflow = true;
    }
    bool overflow = false;  // more ranges than fit: not a launch that can be noted
};

class InFlight {
  public:
    // Whether a launch with these writes may overlap the kernels in front of it.
    bool room(const Writes &w) const { return !w.overflow && (w.trigger == Trigger::LATE || n_ + Writes::MOST <= ROOM); }
    // The launch has been made, overlapping or in plain stream order.
    void note(const Writes &w, bool overlapping) {
        if (!overlapping || w.trigger == Trigger::LATE) finished();
        if (w.overflow) unknown_ = true;
        for (const Writes::Range &r : w.range)
            if (r.p && r.bytes) add(static_cast<const char *>(r.p), static_cast<const char *>(r.p) + r.bytes);
    }
    // Nothing in front of the next kernel is unfinished when it starts (an idle stream, the first kernel of a recording).
    void finished() {
        n_ = 0;
        unknown_ = false;
    }
    // Work that says nothing of its writes is in front of the next kernel.
    void unknown() { unknown_ = true; }
    // Whether the next kernel may read [p, p + bytes) before its wait.
    bool clear_of(const void *p, size_t bytes) const {
        if (unknown_) return false;
        const char *lo = static_cast<const char *>(p), *hi = lo + bytes;
        for (int i = 0; i < n_; i++)
            if (lo < open_[i].hi && open_[i].lo < hi) return false;
        return true;
    }

  private:
    struct Span {
        const char *lo, *hi;
    };
    // A decode step's kernels use the same few dozen blocks of the pool over and over.
    static constexpr int ROOM = 64;
    void add(const char *lo, const char *hi) {
        for (int i = 0; i < n_; i++) {
            if (open_[i].lo <= lo && hi <= open_[i].hi) return;
            if (lo <= open_[i].lo && open_[i].hi <= hi) {
                open_[i] = {lo, hi};
                return;
            }
        }
        open_[n_++] = {lo, hi};
    }
    Span open_[ROOM];
    int n_ = 0;
    bool unknown_ = false;
};

}  // namespace nvc
