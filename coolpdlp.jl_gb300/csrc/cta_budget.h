// cta_budget.h -- how the CTAs that a job may hold are divided among the
// launches that it runs at the same time (plain C++: also built by the tests).
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

namespace cpdlp {

struct CtaShare {
    int cs;               // CTAs of a group (a CTA, or a cluster): one LP at a time
    int64_t most;         // groups it has use for (its LPs, what fits the GPU); 0: no launch
    double work;          // CTA time of its LPs, in any one unit
    int64_t groups = 0;   // out
};

// Fills `groups`: together at most `cap` CTAs (cap <= 0: no cap, every launch
// gets all it has use for), a group at a time to the launch whose LPs would
// otherwise end last.  True when even one group of each launch is more than
// cap: then they have to run one after another, each with cap CTAs to itself (or
// one group, where a cluster is larger than cap).
inline bool share_ctas(std::vector<CtaShare>& launches, int64_t cap) {
    int64_t least = 0, all = 0;
    for (CtaShare& l : launches) {
        l.groups = std::max<int64_t>(l.most, 0);
        least += l.most > 0 ? l.cs : 0;
        all += l.groups * l.cs;
    }
    if (cap <= 0 || all <= cap) return false;
    if (least > cap) {
        for (CtaShare& l : launches)
            l.groups = std::min(l.groups, std::max<int64_t>(cap / l.cs, 1));
        return true;
    }
    for (CtaShare& l : launches) l.groups = std::min<int64_t>(l.groups, 1);
    for (int64_t left = cap - least;;) {
        CtaShare* next = nullptr;
        for (CtaShare& l : launches)
            if (l.groups < l.most && l.cs <= left &&
                (!next || l.work * (double)(next->groups * next->cs) >
                              next->work * (double)(l.groups * l.cs)))
                next = &l;
        if (!next) return false;
        next->groups++;
        left -= next->cs;
    }
}

}  // namespace cpdlp
