"""The per-source engine's table of recent claims (csrc/recent.h) tells all vertex ids
apart: two ids share slot and tag only if the tag is that of an empty slot, which never
stands for a claim.  Host code, compiled here."""
import os
import subprocess


from conftest import ROOT

PROGRAM = r"""
#include <cstdint>
#include <cstdio>
#include <random>
#include "recent.h"
using namespace gu;
int main()
{
    // below 2^30: the multiplier's inverse gives the id back, so no two share a hash
    uint32_t inv = 1;
    for (int i = 0; i < 5; ++i) inv *= 2u - inv * 0x2C1B3C6Du;
    std::mt19937 rng(1);
    auto entry = [](int64_t v) { return recent_hash((int32_t)v); };
    auto fail = [](const char *what, int64_t v) { std::printf("%s: %lld\n", what, (long long)v); return 1; };
    for (int64_t i = 0; i < 4000000; ++i) {
        const int64_t v = i < 2000000 ? i : rng() & 0x3FFFFFFF;
        if (entry(v) >> 30) return fail("slot out of range", v);
        if (((entry(v) * inv) & 0x3FFFFFFFu) != (uint32_t)v) return fail("not one to one", v);
        // the id 2^30 above has no entry that could be taken for this one (ids end at 2^31 - 1)
        const int64_t w = v + (1ll << 30);
        if (entry(w) >> 30) return fail("slot out of range", w);
        if (entry(w) == entry(v) && (uint16_t)entry(v) != RECENT_EMPTY) return fail("taken for another id", w);
        if ((uint16_t)entry(w) != RECENT_EMPTY && ((entry(w) * inv) & 0x3FFFFFFFu) != (uint32_t)w) return fail("taken for another id", w);
    }
    if ((uint16_t)entry(0x7FFFFFFF) != RECENT_EMPTY || (uint16_t)entry(-1) != RECENT_EMPTY) return fail("has an entry", -1);
    return 0;
}
"""


def test_ids_are_told_apart(tmp_path):
    src, exe = tmp_path / "recent.cpp", tmp_path / "recent"
    src.write_text(PROGRAM)
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-I" + os.path.join(ROOT, "graph-utils_gb300", "csrc"), str(src),
                        "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
