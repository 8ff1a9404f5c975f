"""CPU: tensor maps a launcher holds stay what they were when the cache of encoded maps is emptied under it (its capacity passed
by the same launch's next lookups, or by another thread's). The driver's encoder is a fake that notes the address."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "scalingcontrasts_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include <atomic>
#include <thread>
#include <vector>
#include "driver.h"

static std::atomic<int> encoded{0};
static CUresult fake_encode(CUtensorMap* map, CUtensorMapDataType, cuuint32_t, void* base, cuuint64_t const*, cuuint64_t const*,
                            cuuint32_t const*, cuuint32_t const*, CUtensorMapInterleave, CUtensorMapSwizzle,
                            CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
    ++encoded;
    for (auto& word : map->opaque) word = reinterpret_cast<cuuint64_t>(base);
    return CUDA_SUCCESS;
}
extern "C" cudaError_t cudaGetDriverEntryPoint(char const*, void** function, unsigned long long,
                                               cudaDriverEntryPointQueryResult* result) {
    *function = reinterpret_cast<void*>(&fake_encode), *result = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
extern "C" char const* cudaGetErrorString(cudaError_t) { return ""; }

static void const* address(int index) { return reinterpret_cast<void const*>(static_cast<uint64_t>(index + 1) * 4096); }
static bool holds(CUtensorMap const& map, int index) {
    for (auto word : map.opaque)
        if (word != reinterpret_cast<cuuint64_t>(address(index))) return false;
    return true;
}

int main() {
    // The capacity is passed between a launch's lookups sooner or later: a launch makes three maps, the capacity is no multiple.
    for (int launch = 0; launch < 9000; launch += 3) {
        auto&& queries = sc::cached_operand_map(address(launch), 64, 128, 64, 128);
        auto&& candidates = sc::cached_operand_map(address(launch + 1), 64, 128, 64, 64);
        auto&& cube = sc::cached_operand_map(address(launch + 2), 64, 128, 64, 32);
        if (!holds(queries, launch) || !holds(candidates, launch + 1) || !holds(cube, launch + 2)) return 1;
    }
    int const before = encoded;
    auto&& again = sc::cached_operand_map(address(8997), 64, 128, 64, 128);
    if (!holds(again, 8997) || encoded != before) return 2; // a map in the cache is not encoded again
    std::atomic<int> wrong{0};
    std::vector<std::thread> threads;
    for (int t = 0; t < 4; ++t)
        threads.emplace_back([t, &wrong] {
            for (int i = 0; i < 20000; ++i) {
                int const index = (i * (2 * t + 1)) % 9001;
                auto&& map = sc::cached_operand_map(address(index), 128, 128, 64, 128);
                if (!holds(map, index)) ++wrong;
            }
        });
    for (auto& thread : threads) thread.join();
    return wrong ? 3 : 0;
}
"""


def test_held_maps_outlive_the_cache(tmp_path):
    compiler = shutil.which("g++")
    if compiler is None or not os.path.exists(os.path.join(CUDA, "include", "cuda.h")):
        pytest.skip("needs g++ and the CUDA headers")
    source, program = tmp_path / "maps.cpp", tmp_path / "maps"
    source.write_text(PROGRAM)
    command = [compiler, "-std=c++17", "-O1", "-g", f"-I{CSRC}", f"-I{os.path.join(CUDA, 'include')}", str(source), "-o", str(program), "-pthread"]
    # The address checker turns a read of a map that is gone into an error; without it, a wrong value does.
    if subprocess.run(command + ["-fsanitize=address"], capture_output=True).returncode != 0:
        subprocess.run(command, check=True)
    run = subprocess.run([str(program)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stderr[-2000:]
