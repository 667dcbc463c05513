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


def build(tmp_path, source):
    """The program of a source over the library's headers, as a function of its arguments to its lines."""
    src, exe = tmp_path / "main.cpp", str(tmp_path / "main")
    src.write_text(source)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(cuda, "include"),
                    "-I" + os.path.join(ROOT, "voxel-rt_gb300", "csrc"), "-I" + os.path.join(ROOT, "include"), str(src),
                    "-o", exe], check=True)
    return lambda args: subprocess.run([exe] + [str(a) for a in args], capture_output=True, text=True, timeout=60,
                                       check=True).stdout.splitlines()


def test_kernels_read_only_memory_they_can(tmp_path):
    run = build(tmp_path, HARNESS)
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
    out = run([v for c, _ in cases for v in c])
    assert [int(v) for v in out] == [want for _, want in cases]


FAILING_UPLOAD = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "vrt_internal.h"
// No launch and no copy happens here: what upload_common asks for is written down, and the call
// that `fails` names returns an error.
#define cudaMemcpyAsync fake_copy
#define cudaStreamSynchronize fake_wait
#define cudaPointerGetAttributes fake_attributes
#define cudaGetLastError() cudaSuccess
using namespace vrt;
static const char* fails;
static cudaPointerAttributes given;
static int say(const char* what) { std::printf("%s ", what); return std::strcmp(what, fails) ? 0 : -2; }
static cudaError_t fake_copy(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return say("copy") ? cudaErrorUnknown : cudaSuccess; }
static cudaError_t fake_wait(cudaStream_t) { say("wait"); return cudaSuccess; }
static cudaError_t fake_attributes(cudaPointerAttributes* a, const void*) { *a = given; return cudaSuccess; }
static cudaStream_t S(void* s) { return (cudaStream_t)s; }
static void words_box(const Layout&, uint64_t, uint64_t, int64_t*) {}
static int read_state(vrt_world*, int&, cudaStream_t) { return say("state"); }
int vrt::cuda_error(cudaError_t, const char*) { return -2; }
int vrt::set_error(int status, const char*, ...) { return status; }
int vrt::change_words(vrt_world*, const WordChange& c, cudaStream_t) { return say(c.op == kCopyWords ? "pass" : "masks"); }
@UPLOAD@
int main(int argc, char** argv) {
    vrt_world w;
    w.L.n_words = 100;
    w.reads_pageable = true;
    static int32_t words[100];
    for (int i = 1; i + 2 < argc; i += 3) {
        fails = argv[i];
        given.type = (cudaMemoryType)std::atoi(argv[i + 1]);
        given.device = std::atoi(argv[i + 2]);
        const bool host = given.type == cudaMemoryTypeUnregistered;
        std::printf("%d\n", upload_common(&w, words, 0, 100, nullptr, host ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice));
    }
}
"""


def test_a_failed_upload_leaves_no_reader_behind(tmp_path):
    """upload_common against fakes of what it calls: when a later step fails, it returns only when the
    pass that reads the caller's memory has ended, as a copy had taken it by then; and it copies
    what no kernel may read."""
    with open(os.path.join(ROOT, "voxel-rt_gb300", "csrc", "world.cu"), encoding="utf-8") as f:
        text = f.read()
    start = text.index("static int upload_common(")
    run = build(tmp_path, FAILING_UPLOAD.replace("@UPLOAD@", text[start:text.index("\n}\n", start) + 3]))
    out = run(["", UNREGISTERED, -2, "pass", UNREGISTERED, -2, "state", UNREGISTERED, -2,
               "", DEVICE, 0, "state", DEVICE, 0, "", DEVICE, 1, "copy", DEVICE, 1])
    assert out == ["pass state 0", "pass wait -2", "pass state wait -2",
                   "pass state 0", "pass state wait -2", "copy masks state 0", "copy -2"]
