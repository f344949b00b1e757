"""The radix sort's look-back when a tile does not wait for the ones before it
(radix.cuh): it counts their keys itself, and the sort is as correct."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

SOURCE = r"""
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <numeric>
#include <random>
#include <vector>
#include "radix.cuh"

// n keys of few or many values, bits [lo, hi), with and without values; 0: sorted and stable
static int check(uint64_t n, int lo, int hi, uint64_t values, uint32_t spins)
{
    std::mt19937_64 rng(n + hi);
    std::vector<unsigned long long> k(n), got(n);
    std::vector<uint32_t> v(n), order(n), gv(n);
    for (auto& x : k) x = values ? (rng() % values) << lo : rng();
    std::iota(v.begin(), v.end(), 0u);
    order = v;
    const unsigned long long mask = (hi < 64 ? (1ull << hi) - 1ull : ~0ull) & ~((1ull << lo) - 1ull);
    std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return (k[a] & mask) < (k[b] & mask); });
    unsigned long long *a, *b;
    uint32_t *va, *vb;
    void* tmp;
    if (cudaMalloc(&a, 8 * n) || cudaMalloc(&b, 8 * n) || cudaMalloc(&va, 4 * n) || cudaMalloc(&vb, 4 * n) ||
        cudaMalloc(&tmp, rbsc::radix_temp_bytes(n))) return 2;
    int bad = 0;
    for (int with = 0; with < 2; ++with) {
        cudaMemcpy(a, k.data(), 8 * n, cudaMemcpyHostToDevice);
        cudaMemcpy(va, v.data(), 4 * n, cudaMemcpyHostToDevice);
        bool alt = false;
        if (rbsc::radix_sort<uint32_t>(a, b, with ? va : nullptr, with ? vb : nullptr, n, lo, hi, tmp, 0, &alt, spins) != cudaSuccess ||
            cudaDeviceSynchronize() != cudaSuccess) return 3;
        cudaMemcpy(got.data(), alt ? b : a, 8 * n, cudaMemcpyDeviceToHost);
        cudaMemcpy(gv.data(), alt ? vb : va, 4 * n, cudaMemcpyDeviceToHost);
        for (uint64_t i = 0; i < n; ++i) bad |= got[i] != k[order[i]] || (with && gv[i] != order[i]);
    }
    cudaFree(a), cudaFree(b), cudaFree(va), cudaFree(vb), cudaFree(tmp);
    return bad;
}

int main()
{
    for (uint32_t spins : {0u, 1u, 40u, rbsc::kRsSpins})
        for (uint64_t n : {1ull, 4096ull, 4097ull, 8192ull, 300001ull})
            for (int r : {check(n, 0, 64, 0, spins), check(n, 3, 21, 5, spins), check(n, 5, 45, 1ull << 30, spins)})
                if (r) {
                    printf("n %llu spins %u: %d\n", (unsigned long long)n, spins, r);
                    return 1;
                }
    return 0;
}
"""


@pytest.mark.gpu
def test_a_tile_that_waits_for_nobody(tmp_path):
    src, exe = tmp_path / "wait.cu", tmp_path / "wait"
    src.write_text(SOURCE)
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "--expt-relaxed-constexpr",
                    f"-I{ROOT}/rbsc_b200/csrc", f"-I{ROOT}/include", "-o", exe, src], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
