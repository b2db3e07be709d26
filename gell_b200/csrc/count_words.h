// count_words.h — pinned words, one per context, into which birth and death write their counts.
//
// A copy to pageable memory costs 12 us a call, and pinning a word of its own 1.7 ms a context: words come from
// pages of 64 that all contexts share.  A page goes when its last word comes back, but the last page stays until
// the process ends.  A page that the runtime no longer knows (the device was reset) is dropped; its memory may
// come back as another page, so a word carries its page's number, and one whose page is gone is not given back
// to the page that now has its address.
//
// Api: `static bool known(const int*)`, `static int* alloc(size_t bytes)` (null on failure) and
// `static void release(int*)`, none of which leaves an error behind.
#pragma once

#include <cstddef>
#include <mutex>
#include <vector>

namespace gell {

struct CountWord {
    int* at = nullptr;
    unsigned page = 0;
};

template <class Api>
class CountWords {
public:
    CountWord take() {
        std::lock_guard<std::mutex> lock(m_);
        for (size_t k = 0; k < pages_.size();) {
            if (!Api::known(pages_[k].base)) {
                pages_.erase(pages_.begin() + (std::ptrdiff_t)k);
                continue;
            }
            if (~pages_[k].used) return word(pages_[k]);
            ++k;
        }
        int* p = Api::alloc(64 * kStride * sizeof(int));
        if (!p) return CountWord{};
        pages_.push_back(Page{p, 0, ++number_});
        return word(pages_.back());
    }
    void give(const CountWord& w) {
        if (!w.at) return;
        std::lock_guard<std::mutex> lock(m_);
        for (size_t k = 0; k < pages_.size(); ++k) {
            Page& p = pages_[k];
            if (p.number != w.page) continue;
            p.used &= ~(1ull << ((w.at - p.base) / kStride));
            if (!p.used && pages_.size() > 1) {
                Api::release(p.base);
                pages_.erase(pages_.begin() + (std::ptrdiff_t)k);
            }
            return;
        }
    }

private:
    static constexpr int kStride = 16;  // 64 bytes a word
    struct Page {
        int* base;
        unsigned long long used;
        unsigned number;
    };
    static CountWord word(Page& p) {
        int k = 0;
        while (p.used >> k & 1) ++k;
        p.used |= 1ull << k;
        return CountWord{p.base + k * kStride, p.number};
    }
    std::mutex m_;
    std::vector<Page> pages_;
    unsigned number_ = 0;
};

}  // namespace gell
