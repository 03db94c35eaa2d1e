// Host side of a pass that measures stream sizes (SZxG_batch_fixed_rate): the
// (field, bound) pairs it asks for, and the ratios known from earlier passes.
// A batch may hold thousands of small fields, so both cost a field the same
// whatever the number of fields.
#pragma once
#include <string.h>

#include <vector>

#include "kernels.h"

namespace szxg {

inline bool same_bound(float a, float b) { return memcmp(&a, &b, sizeof a) == 0; }   // (a NaN bound is itself too)

struct SizePass {
    std::vector<SizeItem> items;     // ascending step0
    std::vector<int> owner;          // their fields
    unsigned long long steps = 0;    // of 512 values, all items'
    std::vector<size_t> first;       // a field's first item
    size_t turn = 0;                 // first item of the turn below

    explicit SizePass(int nf) : first((size_t)nf) {}
    void clear() {
        items.clear();
        owner.clear();
        steps = 0;
    }
    // A field's next bound: once a field, before any turn.
    void ask(int f, const float* x, unsigned long long n, float eb) {
        first[(size_t)f] = items.size();
        push(f, x, n, eb);
    }
    // Further bounds of one field, in one turn: asked for once each.
    void begin_turn() { turn = items.size(); }
    void ask_more(int f, const float* x, unsigned long long n, float eb) {
        if (same_bound(items[first[(size_t)f]].eb, eb)) return;
        for (size_t k = turn; k < items.size(); k++)
            if (same_bound(items[k].eb, eb)) return;
        push(f, x, n, eb);
    }

private:
    void push(int f, const float* x, unsigned long long n, float eb) {
        items.push_back({x, n, steps, eb, 0});
        owner.push_back(f);
        steps += (n + 511) / 512;
    }
};

// The ratios measured so far, by field.
struct KnownRatios {
    struct Entry {
        float eb;
        int next;     // the field's one before, -1: none
        double cr;
    };
    std::vector<Entry> all;
    std::vector<int> last;
    explicit KnownRatios(int nf) : last((size_t)nf, -1) {}
    void add(int f, float eb, double cr) {
        all.push_back({eb, last[(size_t)f], cr});
        last[(size_t)f] = (int)all.size() - 1;
    }
    const double* find(int f, float eb) const {
        for (int k = last[(size_t)f]; k >= 0; k = all[(size_t)k].next)
            if (same_bound(all[(size_t)k].eb, eb)) return &all[(size_t)k].cr;
        return nullptr;
    }
};

}  // namespace szxg
