"""The pool of second streams (``ForkLease``, csrc/runtime.cu) on the host, with
stand-ins for the CUDA calls: at most eight per device, each given to one call at
a time and used again, none while the caller captures or where a stream cannot be
had; and no allocation, which could throw through a C entry point."""
import shutil
import subprocess

import pytest

from mnpbem_b200.build import CSRC, ROOT

PROGRAM = r'''
#include <math.h>
#include "runtime.cu"
#include <cstdio>
#include <cstdlib>
#include <new>

static bool g_full;                                   // host memory is exhausted
void *operator new(size_t n) {
    if (g_full) throw std::bad_alloc();
    return malloc(n);
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }

static int g_device, g_streams, g_fail_events;
static bool g_capturing;
extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = g_device; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) {
    *s = g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int *a, int *b) { *a = 0; *b = -1; return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) {
    *s = (cudaStream_t)(size_t)++g_streams;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    *e = (cudaEvent_t)1;
    return g_fail_events ? cudaErrorMemoryAllocation : cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { --g_streams; return cudaSuccess; }
}

#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
using mnpb::ForkLease;

int main() {
    g_full = true;
    g_capturing = true;
    { ForkLease l(nullptr); CHECK(!l.get()); }
    g_capturing = false;
    g_fail_events = 1;
    { ForkLease l(nullptr); CHECK(!l.get()); }
    CHECK(g_streams == 0);
    g_fail_events = 0;
    for (int dev = 0; dev < 2; ++dev) {
        g_device = dev;
        for (int round = 0; round < 3; ++round) {
            alignas(ForkLease) char room[9][sizeof(ForkLease)];
            ForkLease *l[9];
            for (int i = 0; i < 9; ++i) {
                l[i] = new (room[i]) ForkLease(nullptr);
                CHECK((l[i]->get() != nullptr) == (i < 8));
                for (int j = 0; j < i && i < 8; ++j) CHECK(l[i]->get()->p != l[j]->get()->p);
                if (i < 8) CHECK(l[i]->get()->dev == dev);
            }
            CHECK(g_streams == 8 * (dev + 1));        // made once, used again
            l[3]->~ForkLease();                       // one given back: the next call has it
            { ForkLease again(nullptr); CHECK(again.get()); }
            for (int i = 0; i < 9; ++i)
                if (i != 3) l[i]->~ForkLease();
        }
    }
    g_device = 64;
    { ForkLease l(nullptr); CHECK(!l.get()); }
    printf("ok\n");
    return 0;
}
'''


def test_pool_is_bounded_and_allocates_nothing(tmp_path):
    (tmp_path / 'pool.cpp').write_text(PROGRAM)
    cuda = '/usr/local/cuda'
    subprocess.run([shutil.which('g++'), '-std=c++17', '-w', '-I%s/include' % cuda,
                    '-I' + ROOT + '/include', '-I' + CSRC, str(tmp_path / 'pool.cpp'), '-o',
                    str(tmp_path / 'pool'), '-L%s/lib64' % cuda, '-lcudart',
                    '-Wl,-rpath,%s/lib64' % cuda, '-pthread'], check=True)
    out = subprocess.run([str(tmp_path / 'pool')], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout == 'ok\n', (out.stdout, out.stderr)
