// pool_schedule.h -- the pool's count of the steps it has queued, and which of them record an
// energy (host only).  Every queued step takes each started, unfinished slot one step on, so
// a slot's steps follow from when it started, and queueing a step touches no slot: the slots
// are looked at only when a step that records an energy has gone by, and then the started
// ones alone.  (One pass over the slot table for every step queued: 0.009 -> 0.22 ms a step
// with 16 slots in use of 65536.)
#pragma once
#include <algorithm>
#include <limits>
#include <vector>

namespace nwb {

class StepSchedule {
public:
    explicit StepSchedule(int max_slots = 0) : at_(max_slots, -1) { runs_.reserve(max_slots); }

    // Slot s starts: its next nsteps steps are those queued from now on; it records its
    // energy at every every-th of them and at the last.
    void start(int s, int nsteps, int every) {
        remove(s);
        at_[s] = static_cast<int>(runs_.size());
        runs_.push_back(Run{s, nsteps, every, now_});
        next_ = std::min(next_, after(runs_.back(), now_));
    }
    void remove(int s) {
        if (at_[s] < 0) return;
        const int i = at_[s];
        at_[s] = -1;
        if (i + 1 < static_cast<int>(runs_.size())) {
            runs_[i] = runs_.back();
            at_[runs_[i].slot] = i;
        }
        runs_.pop_back();
    }
    // Does a slot record its energy in one of the next nsteps steps?  (Yes also where the slot
    // that would have has been removed since.)
    bool records(int nsteps) const { return next_ - now_ <= nsteps; }
    void advance(int nsteps) {
        now_ += nsteps;
        if (now_ < next_) return;
        next_ = std::numeric_limits<long long>::max();
        for (const Run& r : runs_) next_ = std::min(next_, after(r, now_));
    }
    // Steps slot s has taken once all that is queued has run (0: not started).
    int taken(int s) const {
        return at_[s] < 0 ? 0 : static_cast<int>(std::min<long long>(now_ - runs_[at_[s]].start, runs_[at_[s]].nsteps));
    }

private:
    struct Run {
        int slot, nsteps, every;
        long long start;
    };
    // The first step behind now at which r records.
    static long long after(const Run& r, long long now) {
        const long long q = now - r.start;
        if (q >= r.nsteps) return std::numeric_limits<long long>::max();
        return r.start + std::min<long long>((q / r.every + 1) * r.every, r.nsteps);
    }
    std::vector<Run> runs_;
    std::vector<int> at_;  // place of each slot in runs_, or -1
    long long now_ = 0, next_ = std::numeric_limits<long long>::max();
};

}  // namespace nwb
