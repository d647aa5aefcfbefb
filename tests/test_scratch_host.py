"""The pieces of a link table and the scratch they pass through
(qcdgpu_b200/csrc/qg_scratch.h), compiled for the host with a memory whose
calls can be made to fail: every byte of the table goes through once, after
an error nothing is left in flight, a scratch that came out small for want
of memory is asked for in full again by the next call."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "qg_scratch.h"
using namespace qg;
#define NEED(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
struct Memory {
    using Error = int;
    static constexpr int kSuccess = 0, kNoMemory = 2;
    size_t room = ~(size_t)0;
    int other = 0, allocs = 0, frees = 0, syncs = 0, in_flight = 0, freed_in_flight = 0;
    std::vector<size_t> asked;
    int alloc(void **p, size_t n)
    {
        asked.push_back(n);
        if (other) return other;
        if (n > room) return kNoMemory;
        allocs++;
        *p = (void *)(asked.size() * 4096);
        return 0;
    }
    void free(void *p) { if (p) frees++; }
    void sync() { syncs++; in_flight = 0; }
};
int pieces(size_t bytes, int planes, uint32_t rowsize, size_t es, bool to_host)
{
    const size_t row = rowsize * es, total = row * planes;
    for (int fail = -1, ops = 1; fail < ops; fail++) {
        Memory m;
        std::vector<char> seen(total, 0);
        int n = 0, conv = 0, cop = 0, last = -1;
        size_t at0 = 0, n0 = 0;
        bool ok = true;
        auto op = [&]() { if (n++ == fail) return 7; m.in_flight++; return 0; };
        const int e = table_pieces(m, bytes, planes, rowsize, es, to_host,
            [&](int p, int np, uint32_t s0, uint32_t s1) {
                const size_t at = p * row + s0 * es, k = (size_t)np * (s1 - s0) * es;
                ok = ok && s0 < s1 && s1 <= rowsize && (np == 1 || (s0 == 0 && s1 == rowsize)) && k <= bytes;
                if (to_host) { ok = ok && last != 0; at0 = at; n0 = k; } else ok = ok && last == 1 && at == at0 && k == n0;
                last = 0; conv++;
                return op();
            },
            [&](size_t at, size_t k) {
                ok = ok && at + k <= total && k <= bytes;
                if (!to_host) { ok = ok && last != 1; at0 = at; n0 = k; } else ok = ok && last == 0 && at == at0 && k == n0;
                last = 1; cop++;
                if (at + k <= total) for (size_t i = at; i < at + k; i++) seen[i]++;
                return op();
            });
        NEED(ok);
        if (fail < 0) {
            NEED(e == 0 && m.syncs == 0 && conv == cop);
            for (char c : seen) NEED(c == 1);
            ops = n;
        } else {
            NEED(e == 7 && n == fail + 1 && m.syncs == 1 && m.in_flight == 0);
        }
    }
    return 0;
}
int main()
{
    const uint32_t rows[] = { 1, 16, 64, 1000, 4096 };
    for (uint32_t r : rows)
        for (int planes : { 4, 12 })
            for (size_t es : { 16, 32 })
                for (size_t b : { es, 3 * es, r * es, r * es + es, 5 * r * es, 12 * r * es, 40 * r * es })
                    for (int to : { 0, 1 }) if (b / es * 600 >= (size_t)r * planes && pieces(b, planes, r, es, to)) return 1;
    Memory m;
    Scratch st;
    NEED(scratch_reserve(m, st, 1000, 100) == 0 && st.bytes == 1000 && m.allocs == 1);
    NEED(scratch_reserve(m, st, 900, 100) == 0 && st.bytes == 1000 && m.allocs == 1);        // kept
    m.room = 300;
    NEED(scratch_reserve(m, st, 2000, 100) == 0 && st.bytes == 250 && m.frees == 1);         // 2000, 1000, 500, 250
    NEED(scratch_reserve(m, st, 200, 100) == 0 && st.bytes == 250 && m.allocs == 2);
    m.room = 5000;
    NEED(scratch_reserve(m, st, 2000, 100) == 0 && st.bytes == 2000 && m.frees == 2);        // in full again
    m.room = 120;
    NEED(scratch_reserve(m, st, 3000, 100) == 0 && st.bytes == 100 && m.asked.back() == 100);
    m.room = 99;
    NEED(scratch_reserve(m, st, 3000, 100) == Memory::kNoMemory && !st.p && !st.bytes && m.asked.back() == 100);
    NEED(scratch_reserve(m, st, 3000, 3000) == Memory::kNoMemory && m.asked.back() == 3000 && m.frees == m.allocs);
    m.other = 9;
    const size_t n = m.asked.size();
    NEED(scratch_reserve(m, st, 3000, 100) == 9 && m.asked.size() == n + 1 && !st.p && !st.bytes);
    printf("ok\n");
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_pieces_errors_and_scarce_memory(tmp_path):
    src = tmp_path / "scratch.cpp"
    src.write_text(HARNESS)
    exe = str(tmp_path / "scratch")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "qcdgpu_b200", "csrc"),
                    str(src), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.stdout.strip() == "ok", r.stdout + r.stderr
