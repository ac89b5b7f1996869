// table_cache.h -- which (tone curve, gamma) pairs have a byte table on which device.
//
// The tables live in a fixed number of slots per device and are never replaced (a kernel may read
// one at any time), so who may take a slot matters: kCommon of them belong to the common chain's pairs,
// and pairs first met by a chain with optional steps take the kGraded others, so that a program that sweeps
// such a chain's gamma does not use up the common chain's.  A pair that has no table (its curve does
// not fit one) is remembered too: trying again costs about a millisecond of host time a call.  Once
// kMaxFailed pairs have none, chains with optional steps try no further pairs.
// Plain C++ without locking: the caller holds a mutex.
#pragma once

#include <cstddef>
#include <vector>

namespace lum {

template <class Table>
class TableCache {
public:
    static constexpr int kCommon = 16, kGraded = 8, kSlots = kCommon + kGraded;
    static constexpr size_t kMaxFailed = 64;   // pairs remembered as without a table, the oldest forgotten first

    // The pair's table, or null if the pair is not known; *known to false then.  A known pair without
    // a table gives null too.
    const Table* find(int device, int kind, long long gamma, bool* known) const {
        *known = true;
        for (const Entry& e : tables_)
            if (e.device == device && e.kind == kind && e.gamma == gamma) return &e.table;
        for (const Entry& e : failed_)
            if (e.device == device && e.kind == kind && e.gamma == gamma) return nullptr;
        *known = false;
        return nullptr;
    }

    // The slot a new pair would take, or -1: no table for it.
    int free_slot(int device, bool graded) const {
        int used[2] = {0, 0};
        for (const Entry& e : tables_)
            if (e.device == device) ++used[e.slot >= kCommon];
        if (graded) return used[1] < kGraded && failed_.size() < kMaxFailed ? kCommon + used[1] : -1;
        return used[0] < kCommon ? used[0] : -1;
    }

    void add(int device, int kind, long long gamma, int slot, const Table& table) {
        tables_.push_back(Entry{device, kind, gamma, slot, table});
    }

    void add_failed(int device, int kind, long long gamma) {
        const Entry e{device, kind, gamma, -1, Table{}};
        if (failed_.size() < kMaxFailed) failed_.push_back(e);
        else failed_[oldest_++ % kMaxFailed] = e;
    }

private:
    struct Entry {
        int device, kind;
        long long gamma;
        int slot;
        Table table;
    };
    std::vector<Entry> tables_, failed_;
    size_t oldest_ = 0;
};

}  // namespace lum
