"""Bookkeeping of the contexts' status words against a stand-in for the CUDA calls (CPU only)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cassert>
#include <cstdlib>
#include <map>
#include <vector>
#include "status_pages.h"
// Device contexts with the pages pinned in each; a reset ends the present one and everything pinned in it.
struct Fake {
    static unsigned long long now;
    static std::map<unsigned int *, unsigned long long> pinned;
    static std::vector<unsigned int *> freelist;
    static int id(unsigned long long *o) { *o = now; return 0; }
    static int pin(unsigned int **p, size_t n)
    {
        if (!freelist.empty()) { *p = freelist.back(); freelist.pop_back(); }     // an address handed out again
        else *p = (unsigned int *)calloc(n, 4);
        pinned[*p] = now;
        return 0;
    }
    static int unpin(unsigned int *p) { assert(pinned.count(p) && pinned[p] == now); pinned.erase(p); freelist.push_back(p); return 0; }
    static int map(unsigned int **d, unsigned int *h)
    {
        for (auto &kv : pinned) if (h >= kv.first && h < kv.first + 1024) { *d = h; return kv.second == now ? 0 : 2; }
        return 1;
    }
    static void reset()
    {
        for (auto &kv : pinned) freelist.push_back(kv.first);
        pinned.clear();
        ++now;
    }
};
unsigned long long Fake::now = 7;
std::map<unsigned int *, unsigned long long> Fake::pinned;
std::vector<unsigned int *> Fake::freelist;
int main()
{
    one::StatusPages<Fake> pages;
    one::StatusSlot a, b, never;
    pages.give(&never);
    assert(pages.take(0, &a) == 0 && pages.take(0, &b) == 0 && a.host != b.host && Fake::pinned.size() == 1);
    *a.host = 5;
    unsigned int *word = a.host;
    pages.give(&a);
    assert(pages.take(0, &a) == 0 && a.host == word && *a.host == 0);          // a slot is cleared when it is taken again
    pages.give(&a);
    pages.give(&b);
    assert(Fake::pinned.size() == 1);                                          // one page stays pinned
    assert(pages.take(0, &a) == 0 && Fake::pinned.size() == 1);
    pages.give(&a);
    Fake::reset();                                                             // every context had been released
    assert(pages.take(0, &a) == 0 && Fake::pinned.size() == 1);
    Fake::reset();                                                             // one had not
    assert(pages.take(0, &b) == 0 && b.host == word);                          // the same address, in a new page
    pages.give(&a);                                                            // the old slot: the new page's is untouched
    one::StatusSlot c;
    assert(pages.take(0, &c) == 0 && c.host != b.host);
    pages.give(&b);
    pages.give(&c);
    std::vector<one::StatusSlot> many(2500);
    for (auto &s : many) assert(pages.take(0, &s) == 0);
    assert(Fake::pinned.size() == 3);
    for (auto &s : many) pages.give(&s);
    assert(Fake::pinned.size() == 1);                                          // the other pages were given back
    one::StatusSlot d;
    assert(pages.take(1, &d) == 0 && Fake::pinned.size() == 2);                // another device: its own page
    pages.give(&d);
    return 0;
}
"""


def test_status_words_over_releases_and_resets(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-g", "-I", os.path.join(ROOT, "onenew_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True, timeout=60)
