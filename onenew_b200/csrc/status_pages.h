// status_pages.h -- where the contexts' status words live: slots of pinned, mapped pages (pinning a page takes ~10 ms, too
// long for every context).
//
// A page belongs to the device context it was pinned in and goes with it: after cudaDeviceReset its memory is gone, and its
// addresses may be handed out again.  So a page is remembered with the number of that device context (never used twice in
// a process), a slot is taken from a page of the present one only, and pages of one that is gone are forgotten, not freed.
// A page whose last slot is given back is freed, except one a device context, which the next context finds pinned.
//
// Api (the CUDA runtime, or a stand-in in a test): id(unsigned long long *), the present device context's number;
// pin(unsigned int **, size_t words), unpin(unsigned int *), map(unsigned int **device, unsigned int *host); 0 is success.
#pragma once
#include <stddef.h>

#include <memory>
#include <mutex>
#include <vector>

namespace one {

struct StatusPage {
    static constexpr size_t SLOTS = 1024;
    int device = 0;
    unsigned long long context = 0;
    unsigned int *words = nullptr;
    size_t live = 0;
    bool used[SLOTS] = {};
};

// A slot; it keeps its page's record (not the memory) alive.
struct StatusSlot {
    std::shared_ptr<StatusPage> page;
    size_t index = 0;
    unsigned int *host = nullptr, *dev = nullptr;
};

template <typename Api> class StatusPages {
public:
    // With `device` current.  0, or the failing call's code.
    int take(int device, StatusSlot *out)
    {
        std::lock_guard<std::mutex> lk(mu);
        unsigned long long context = 0;
        int e = Api::id(&context);
        if (e) return e;
        for (size_t i = pages.size(); i-- > 0;)
            if (pages[i]->device == device && pages[i]->context != context) pages.erase(pages.begin() + i);
        std::shared_ptr<StatusPage> page;
        for (auto &p : pages)
            if (p->device == device && p->live < StatusPage::SLOTS) { page = p; break; }
        if (!page) {
            page = std::make_shared<StatusPage>();
            if ((e = Api::pin(&page->words, StatusPage::SLOTS))) return e;
            page->device = device;
            page->context = context;
            pages.push_back(page);
        }
        size_t i = 0;
        while (page->used[i]) ++i;
        unsigned int *dev = nullptr;
        if ((e = Api::map(&dev, page->words + i))) return e;
        page->used[i] = true;
        ++page->live;
        page->words[i] = 0;
        out->page = page; out->index = i; out->host = page->words + i; out->dev = dev;
        return 0;
    }

    // With the slot's device current; a slot that was never taken is ignored.
    void give(StatusSlot *s)
    {
        std::lock_guard<std::mutex> lk(mu);
        std::shared_ptr<StatusPage> page = std::move(s->page);
        s->host = s->dev = nullptr;
        if (!page) return;
        page->used[s->index] = false;
        if (--page->live) return;
        size_t at = pages.size(), same = 0;
        for (size_t i = 0; i < pages.size(); ++i) {
            if (pages[i] == page) at = i;
            if (pages[i]->device == page->device) ++same;
        }
        if (at == pages.size() || same == 1) return;   // forgotten, or the one that is kept
        unsigned long long context = 0;
        if (Api::id(&context) == 0 && context == page->context) Api::unpin(page->words);
        pages.erase(pages.begin() + at);
    }

private:
    std::mutex mu;
    std::vector<std::shared_ptr<StatusPage>> pages;
};

}  // namespace one
