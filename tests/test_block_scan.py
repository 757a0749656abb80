"""CPU: the resident loops' block-wide scan writes the n starts it is asked for
and nothing behind them.  (The re-sort of the rigid-body loop scans into an array
of exactly n starts.)  The device function is taken from its header as it is and
run by a block of host threads, with the barrier and the warp shuffle restated."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

HEADER = Path(__file__).resolve().parent.parent / "dpcuda-v2_gb300" / "csrc" / "disk_loop.cuh"

HARNESS = r"""
#include <barrier>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>
constexpr int NT = 64;
struct Dim { int x; };
static thread_local Dim threadIdx;
static const Dim blockDim = {NT};
static std::barrier<> block_bar(NT);
static std::barrier<> *warp_bar[NT / 32];
static int lanes[NT];
#define __device__
#define __forceinline__
#define __shared__ static
static void __syncthreads() { block_bar.arrive_and_wait(); }
static int __shfl_up_sync(unsigned, int v, int o) {
    const int t = threadIdx.x, w = t / 32;
    lanes[t] = v;
    warp_bar[w]->arrive_and_wait();
    const int r = t % 32 >= o ? lanes[t - o] : v;
    warp_bar[w]->arrive_and_wait();
    return r;
}
FUNCTION
int main() {
    for (auto &b : warp_bar) b = new std::barrier<>(32);
    for (int n : {1, 2, 31, 32, 33, 127, 128, 129, 255, 256, 257, 512, 700, 1024}) {
        std::vector<int> cnt(n), start(n + 1, -77);
        for (int k = 0; k < n; k++) cnt[k] = (k * 2654435761u >> 20) % 29;
        std::vector<std::thread> th;
        for (int t = 0; t < NT; t++)
            th.emplace_back([&, t] { threadIdx.x = t; NAME(cnt.data(), start.data(), n); });
        for (auto &t : th) t.join();
        int sum = 0;
        for (int k = 0; k < n; sum += cnt[k++])
            if (start[k] != sum) { std::printf("n = %d: start %d\n", n, k); return 1; }
        if (start[n] != -77) { std::printf("n = %d: a word behind the starts was written\n", n); return 1; }
    }
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host compiler")
def test_scan_stays_within_its_starts(tmp_path):
    text = HEADER.read_text()
    m = re.search(r"__device__ __forceinline__ \w+ (\w*scan_block)\(.*?\n}\n", text, re.S)
    src = tmp_path / "scan.cpp"
    src.write_text(HARNESS.replace("FUNCTION", m.group(0).replace("#pragma unroll", "")).replace("NAME", m.group(1)))
    exe = tmp_path / "scan"
    subprocess.run(["g++", "-std=c++20", "-O1", "-pthread", "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
