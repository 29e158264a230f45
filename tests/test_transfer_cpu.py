"""The host side of transfer.cu (pinned ring, helper threads) against a stand-in for the CUDA runtime that copies at once: what it does
when the host refuses it something. Built with g++, no GPU."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

HARNESS = r"""
#include <dlfcn.h>
#include <pthread.h>
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "common.cuh"

static int pinned_left = 1 << 30, threads_left = 1 << 30, copies = 0;
namespace wb {
int fail(int code, const char *, ...) { return code; }
}
extern "C" {
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return pinned_left-- > 0 ? (*p = malloc(n), cudaSuccess) : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void *p) { return free(p), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return *e = (cudaEvent_t)1, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorName(cudaError_t) { return ""; }
const char *cudaGetErrorString(cudaError_t) { return ""; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { return copies++, memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) { return a->type = cudaMemoryTypeUnregistered, cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg)
{
    if (threads_left-- <= 0) return 11;  // EAGAIN
    return ((int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *))dlsym(RTLD_NEXT, "pthread_create"))(t, a, f, arg);
}
}

int main(int, char **argv)
{
    pinned_left = atoi(argv[1]), threads_left = atoi(argv[2]);
    const size_t n = (33 << 20) + 3;
    std::vector<unsigned char> host(n), dev(n), back(n);
    for (size_t i = 0; i < n; i++) host[i] = (unsigned char)(i * 2654435761u >> 13);
    wb_context ctx;
    wb::transfer_retain();
    if (wb::copy_to_device(&ctx, dev.data(), host.data(), n) || wb::copy_to_host(&ctx, back.data(), dev.data(), n)) return 1;
    if (host != back) return 2;
    printf("%d\n", copies);
    if (atoi(argv[3])) wb::transfer_release();
    return 0;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("transfer")
    (d / "main.cpp").write_text(HARNESS)
    cuda = Path(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc").resolve().parent.parent / "include"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-rdynamic", "-I", str(ROOT / "webllm_b200/csrc"), "-I", str(ROOT / "include"),
                    "-I", str(cuda), "-x", "c++", str(ROOT / "webllm_b200/csrc/transfer.cu"), str(d / "main.cpp"), "-ldl", "-o", str(d / "main")],
                   check=True)

    def run(pinned: int, threads: int, release: bool) -> int:
        r = subprocess.run([str(d / "main"), str(pinned), str(threads), str(int(release))], capture_output=True, text=True, timeout=60)
        assert r.returncode == 0, (r.returncode, r.stderr)
        return int(r.stdout)

    return run


def test_copies_without_a_pinned_ring(harness):
    assert harness(pinned=0, threads=9, release=True) == 2  # one plain copy each way


@pytest.mark.parametrize("threads", [0, 1])
def test_copies_with_fewer_helper_threads(harness, threads):
    copies = harness(pinned=9, threads=threads, release=True)
    assert copies == 2 if threads == 0 else copies in (2, 2 * 67)  # (2: a host of few cores has no helpers) pieces of 512 KB


def test_process_ends_with_a_context_open(harness):
    harness(pinned=9, threads=9, release=False)
