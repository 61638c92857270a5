"""The scratch arena of a context's BVH builds, compiled for the host with
counting stand-ins for cudaMalloc and cudaFree: what is kept after calls that
succeed and fail, and that nothing is freed under a build that holds it."""
import os
import subprocess

from rustracer_gb300 import build

SOURCE = r"""
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include "build_arena.h"
static std::atomic<int> g_live{0};
extern "C" cudaError_t cudaMalloc(void** p, size_t) { ++g_live; *p = std::malloc(1); return cudaSuccess; }
extern "C" cudaError_t cudaFree(void* p) { --g_live; std::free(p); return cudaSuccess; }
using gbrt::BuildArena;
using gbrt::BuildCall;
static void build(BuildArena& a, size_t n) { std::lock_guard<std::mutex> hold(a.mu); a.reserve(n); }
#define CHECK(x) do { if (!(x)) { std::printf("failed: %s\n", #x); return 1; } } while (0)
int main() {
    const size_t keep = BuildArena::kKeep;
    BuildArena a;
    { BuildCall c(a); build(a, 1000); c.done(); }
    CHECK(a.bytes == 1000 && g_live == 1);       // kept for the next build
    { BuildCall c(a); build(a, 500); }
    CHECK(a.bytes == 0 && g_live == 0);          // a call that fails gives everything back
    { BuildCall c(a); build(a, keep); c.done(); }
    CHECK(a.bytes == keep);
    { BuildCall c(a); build(a, keep + 1); c.done(); }
    CHECK(a.bytes == 0 && g_live == 0);          // more than kKeep goes back after success too
    { BuildCall c(a); { BuildCall d(a); build(a, keep + 1); } build(a, 7); c.done(); }
    CHECK(a.bytes == 7);
    std::atomic<bool> ended{false};
    std::thread t;
    {
        std::lock_guard<std::mutex> hold(a.mu);  // a build of another thread
        t = std::thread([&] { { BuildCall c(a); } ended = true; });
        std::this_thread::sleep_for(std::chrono::milliseconds(50));
        CHECK(!ended && a.bytes == 7 && g_live == 1);
    }
    t.join();
    CHECK(ended && a.bytes == 0 && g_live == 0);
    return 0;
}
"""


def test_build_arena(tmp_path):
    src, exe = tmp_path / "arena.cpp", tmp_path / "arena"
    src.write_text(SOURCE)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", build.CSRC, "-I", cuda, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
