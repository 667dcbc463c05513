"""Which memory an upload's kernel may read itself, and which only a copy may take: the choice
(upload_view, csrc/vrt_internal.h) against every kind of address, with the attributes that the
CUDA runtime would give.  No GPU, and no second one, is needed for it."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cstdio>
#include <cstdlib>
#include "vrt_internal.h"
// argv: from_host type device address mapped reads_pageable -> the address read, 0: none
int main(int argc, char** argv) {
    for (int i = 1; i + 5 < argc; i += 6) {
        cudaPointerAttributes at{};
        at.type = (cudaMemoryType)std::atoi(argv[i + 1]);
        at.device = std::atoi(argv[i + 2]);
        at.devicePointer = (void*)std::strtoull(argv[i + 4], nullptr, 0);
        const auto* src = (const int32_t*)std::strtoull(argv[i + 3], nullptr, 0);
        std::printf("%llu\n", (unsigned long long)(uintptr_t)vrt::upload_view(src, std::atoi(argv[i]), at, 1, std::atoi(argv[i + 5])));
    }
}
"""
UNREGISTERED, HOST, DEVICE, MANAGED = range(4)  # cudaMemoryType
A, M = 0x10004, 0x20008  # the caller's address, and the device's address of mapped memory


def test_kernels_read_only_memory_they_can(tmp_path):
    src = tmp_path / "view_main.cpp"
    src.write_text(HARNESS)
    exe = str(tmp_path / "view_main")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(cuda, "include"),
                    "-I" + os.path.join(ROOT, "voxel-rt_gb300", "csrc"), "-I" + os.path.join(ROOT, "include"), str(src),
                    "-o", exe], check=True)
    cases = [  # from_host, type, device (the world's is 1), address, mapped, reads_pageable -> address read
        ((0, DEVICE, 1, A, A, 1), A),
        ((0, DEVICE, 1, A, A, 0), A),
        ((0, DEVICE, 0, A, A, 1), 0),        # another GPU's memory
        ((0, DEVICE, 2, A, A, 0), 0),
        ((0, HOST, 1, A, M, 1), 0),          # host memory where device memory is meant
        ((0, UNREGISTERED, -2, A, 0, 1), 0),
        ((0, MANAGED, 1, A, A, 1), 0),
        ((0, DEVICE, 1, A + 2, A + 2, 1), 0),
        ((1, UNREGISTERED, -2, A, 0, 1), A),
        ((1, UNREGISTERED, -2, A, 0, 0), 0),
        ((1, HOST, 0, A, M, 1), A),
        ((1, HOST, 0, A, M, 0), M),
        ((1, HOST, 0, A, 0, 0), 0),
        ((1, MANAGED, 1, A, A, 0), 0),
        ((1, DEVICE, 1, A, A, 1), 0),        # device memory where host memory is meant: refused by the copy
        ((1, DEVICE, 0, A, A, 1), 0),
        ((1, UNREGISTERED, -2, A + 1, 0, 1), 0),
        ((1, UNREGISTERED, -2, A + 2, 0, 1), 0),
        ((1, HOST, 0, A + 3, M + 3, 0), 0),
    ]
    args = [hex(v) if v > 255 else str(v) for c, _ in cases for v in c]
    out = subprocess.run([exe] + args, capture_output=True, text=True, timeout=60, check=True).stdout.split()
    assert [int(v) for v in out] == [want for _, want in cases]
