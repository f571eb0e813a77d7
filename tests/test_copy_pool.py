"""The threads that share out host copies (clgpu_b200/csrc/copy_pool.h), checked
on the CPU: a copy made while another one is under way is shared too, every byte
arrives once, with more callers than the pool has places, and the pool ends."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include <string>
#include "copy_pool.h"

using Clock = std::chrono::steady_clock;
static std::atomic<int> first_in{0}, second_in{0}, together{0};
static std::atomic<bool> release_first{false};
static const char *first_src, *second_src;
static constexpr size_t kFirst = 256 << 10, kSecond = 4 << 20;

static bool within(std::atomic<int>& v, int want)
{
    const auto end = Clock::now() + std::chrono::seconds(20);
    while (v.load() < want)
        if (Clock::now() > end) return false;
    return true;
}

// the first copy (two slices) stays under way until it is released; a slice of
// the second waits for another thread to be in one as well
static void copy(void* dst, const void* src, size_t bytes)
{
    const char* s = (const char*)src;
    if (s >= first_src && s < first_src + kFirst) {
        first_in.fetch_add(1);
        while (!release_first.load()) std::this_thread::yield();
    } else if (s >= second_src && s < second_src + kSecond) {
        second_in.fetch_add(1);
        if (within(second_in, 2)) together.fetch_add(1);
    }
    std::memcpy(dst, src, bytes);
}

int main()
{
    int bad = 0;
    {
        iclb::CopyPool pool(4, copy);
        std::string a(kFirst, 'a'), b(kSecond, 'b'), da(kFirst, 0), db(kSecond, 0);
        first_src = a.data();
        second_src = b.data();
        std::thread first([&] { pool.copy(&da[0], a.data(), kFirst); });
        if (!within(first_in, 1)) ++bad;
        pool.copy(&db[0], b.data(), kSecond);
        if (together.load() < 2) { std::printf("the second copy was not shared\n"); ++bad; }
        release_first.store(true);
        first.join();
        if (da != a || db != b) { std::printf("bytes differ\n"); ++bad; }
        first_src = second_src = nullptr;
    }
    {
        iclb::CopyPool pool(3, copy);
        std::vector<std::thread> callers;
        std::atomic<int> wrong{0};
        for (int t = 0; t < 12; ++t)
            callers.emplace_back([&, t] {
                for (int r = 0; r < 60; ++r) {
                    const size_t n = 100000 + 77777 * ((t + r) % 9);
                    std::string s(n, 0), d(n + 1, 'x');
                    for (size_t i = 0; i < n; ++i) s[i] = (char)(i * 31 + t * 7 + r);
                    pool.copy(&d[0], s.data(), n);
                    if (std::memcmp(d.data(), s.data(), n) != 0 || d[n] != 'x') wrong.fetch_add(1);
                }
            });
        for (auto& c : callers) c.join();
        if (wrong.load()) { std::printf("%d copies wrong\n", wrong.load()); ++bad; }
    }
    std::printf("%d bad\n", bad);
    return bad;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_copies_under_way_share_the_threads(tmp_path):
    src = tmp_path / "copy_pool_check.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "copy_pool_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "clgpu_b200", "csrc"), str(src), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
