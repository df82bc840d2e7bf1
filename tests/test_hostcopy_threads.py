"""The threaded copies of host arrays (csrc/hostcopy.cpp) on the CPU, against a stand-in of the CUDA calls they
make: blocks land where they belong both ways, and a host without memory for another thread gets a copy by the
threads that did start instead of an abort."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = os.path.join(os.environ.get('CUDA_HOME', '/usr/local/cuda'), 'include')

HARNESS = r'''
#include "hostcopy.h"
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>

// the CUDA calls of hostcopy.cpp, done at once on the host
extern "C" {
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { a->type = cudaMemoryTypeUnregistered; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
}

static thread_local int left = -1;        // allocations of this thread until one fails (-1: none does)
void* operator new(size_t n)
{
    if (left == 0) throw std::bad_alloc();
    if (left > 0) left--;
    void* p = malloc(n);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }

int main(int, char** av)
{
    const int allowed = atoi(av[1]);
    const size_t n0 = atol(av[2]), n1 = atol(av[3]);
    std::vector<unsigned char> h0(n0), h1(n1), d0(n0), d1(n1), b0(n0), b1(n1);
    for (size_t i = 0; i < n0; i++) h0[i] = (unsigned char)(i * 7 + i / 251);
    for (size_t i = 0; i < n1; i++) h1[i] = (unsigned char)(i * 5 + i / 241 + 3);
    srwg::HostRing ring;
    srwg::CopySeg up[2] = {{h0.data(), d0.data(), n0}, {h1.data(), d1.data(), n1}};
    srwg::CopySeg down[2] = {{b0.data(), d0.data(), n0}, {b1.data(), d1.data(), n1}};
    if (srwg::copy_segments(ring, 0, up, 1, true, 0) != cudaSuccess) return 2;      // the ring's own allocations
    memset(d0.data(), 0, n0);
    left = allowed;
    const cudaError_t a = srwg::copy_segments(ring, 0, up, 2, true, 0);
    left = allowed;
    const cudaError_t b = srwg::copy_segments(ring, 0, down, 2, false, 0);
    left = -1;
    if (a != cudaSuccess || b != cudaSuccess) return 3;
    return d0 == h0 && d1 == h1 && b0 == h0 && b1 == h1 ? 0 : 4;
}
'''


@pytest.fixture(scope='module')
def harness(tmp_path_factory):
    if shutil.which('g++') is None or not os.path.exists(os.path.join(CUDA_INC, 'cuda_runtime.h')):
        pytest.skip('no host compiler or CUDA headers')
    d = tmp_path_factory.mktemp('hostcopy')
    (d / 'main.cpp').write_text(HARNESS)
    exe = str(d / 'main')
    csrc = os.path.join(REPO, 'srw_b200', 'csrc')
    subprocess.run(['g++', '-std=c++17', '-O1', '-pthread', '-I', csrc, '-I', CUDA_INC, str(d / 'main.cpp'),
                    os.path.join(csrc, 'hostcopy.cpp'), '-o', exe], check=True)
    return exe


@pytest.mark.parametrize('threads', [-1, 0, 1, 3])               # thread objects before the memory is gone
@pytest.mark.parametrize('n0,n1', [(1000, 77), (4 << 20, 1), (9 << 20, (5 << 20) + 12345)])
def test_copies_with_and_without_memory_for_threads(harness, threads, n0, n1):
    r = subprocess.run([harness, str(threads), str(n0), str(n1)], timeout=120)
    assert r.returncode == 0
