"""Where the library's memory comes from and goes back to (memory.h), as far as that can be seen without a GPU."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "genn_b200", "csrc")


def test_what_goes_back_to_the_pool_came_from_it():
    """A member of the runner that cudaMalloc fills is not handed to poolFree (a stream-ordered free), nor the other way round;
    the near-synapse table has both kinds and says which it is."""
    text = open(os.path.join(CSRC, "runner.cu")).read()

    def members(call):
        return {m.split("->")[-1].split("[")[0] for m in re.findall(call + r"\(&?((?:r->)?\w+(?:\[\w+\])?)", text)} - {"p"}       # (a local)

    assert members("cudaMalloc") & members("poolFree") <= {"nearTable"}
    assert members("poolAlloc") & members("cudaFree") <= {"nearTable"}
    assert "nearExported" in text[text.index("void freeNearTable"):text.index("void dropNear")]


# memory.cu on a host whose "device" is its own memory and on which no more than `argv[1]` threads can be started
HARNESS = r"""
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <stdlib.h>
#include <string.h>
#include <atomic>
#include <cstdio>
#include <vector>
#include "memory.h"
static std::atomic<int> left;
extern "C" {
int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void*), void *arg)
{
    if(left-- <= 0) return EAGAIN;
    return ((int (*)(pthread_t*, const pthread_attr_t*, void *(*)(void*), void*))dlsym(RTLD_NEXT, "pthread_create"))(t, a, f, arg);
}
cudaError_t cudaMalloc(void **p, size_t n) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps*) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned int) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned int) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *to, const void *from, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(to, from, n); return cudaSuccess; }
}
int main(int, char **argv)
{
    left = atoi(argv[1]);
    std::vector<unsigned short> device(5000001);
    for(size_t i = 0; i < device.size(); i++) device[i] = (unsigned short)(i * 7);
    std::vector<unsigned int> wide(device.size());
    std::vector<unsigned short> same(device.size());
    if(b200::pullLarge(same.data(), device.data(), device.size() * 2, 1u, false, 0, nullptr) != cudaSuccess) return 1;
    if(b200::pullLarge(wide.data(), device.data(), device.size(), 2u, true, 0, nullptr) != cudaSuccess) return 2;
    for(size_t i = 0; i < device.size(); i++) if(same[i] != device[i] || wide[i] != device[i]) return 3;
    return 0;
}
"""


@pytest.mark.parametrize("threads", [0, 3, 100])
def test_a_large_pull_is_whole_with_as_many_threads_as_can_be_had(tmp_path, threads):
    gxx, include = shutil.which("g++"), os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if not gxx or not os.path.exists(os.path.join(include, "cuda_runtime_api.h")):
        pytest.skip("no host compiler, or no CUDA headers")
    (tmp_path / "harness.cc").write_text(HARNESS)
    exe = str(tmp_path / "harness")
    subprocess.check_call([gxx, "-std=c++17", "-O1", "-pthread", "-rdynamic", "-I", CSRC, "-I", include, str(tmp_path / "harness.cc"), "-x", "c++",
                           os.path.join(CSRC, "memory.cu"), "-o", exe, "-ldl"])
    assert subprocess.run([exe, str(threads)], timeout=60).returncode == 0
