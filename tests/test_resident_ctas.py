"""The shared-memory limit of a kernel only grows, whatever threads ask for it (no GPU needed: the
function is compiled against stand-ins of the runtime calls that it makes)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "drivingsdk_b200", "csrc")
CUDA_HOME = os.environ.get("CUDA_HOME", "/usr/local/cuda")

# The first thread to read the limit goes on only when the other has set its own, or after a while.
PROGRAM = r"""
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>
#include "resident_ctas.h"
static std::atomic<int> limit{48 * 1024}, reads{0}, sets{0};
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
    a->maxDynamicSharedSizeBytes = limit;
    if (reads++ == 0)
        for (int i = 0; i < 300 && sets == 0; ++i) std::this_thread::sleep_for(std::chrono::milliseconds(1));
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int v) { limit = v; ++sets; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t s) {
    *n = static_cast<int>(256 * 1024 / (s + 1));
    return cudaSuccess;
}
}
int main() {
    static const int kernel = 0;
    int small = 0, large = 0;
    std::thread a([&] { msda::resident_ctas(&kernel, 256, 100 * 1024, &small); });
    while (reads == 0) std::this_thread::yield();
    std::thread b([&] { msda::resident_ctas(&kernel, 256, 200 * 1024, &large); });
    a.join();
    b.join();
    std::printf("%d %d %d\n", limit.load() / 1024, small, large);
}
"""


def test_two_threads_with_two_sizes(tmp_path):
    source, program = tmp_path / "limit.cpp", tmp_path / "limit"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-I", os.path.join(CUDA_HOME, "include"),
                    str(source), "-x", "c++", os.path.join(CSRC, "resident_ctas.cu"), "-o", str(program)],
                   check=True)
    assert subprocess.run([str(program)], check=True, capture_output=True, text=True).stdout.split() == ["200", "2", "1"]
