"""The cut of a solve's right-hand sides over two streams (``in_halves``, csrc/fork.cuh),
on the host: a small program includes the header with stand-ins for the second
stream and records which right-hand sides each part is given."""
import shutil
import subprocess

import pytest

from mnpbem_b200.build import CSRC, ROOT

PROGRAM = r'''
#include <math.h>
#include "fork.cuh"
#include <cstdio>

static bool g_second;                      // whether a second stream is to be had
extern "C" {
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return ""; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
}
namespace mnpb {
void set_error(const char *, ...) {}
static Fork g_fork{(cudaStream_t)2, nullptr, nullptr, 0};
ForkLease::ForkLease(cudaStream_t) : f_(g_second ? &g_fork : nullptr) {}
ForkLease::~ForkLease() {}
}

int main() {
    for (int second = 0; second < 2; ++second)
        for (int cut = 0; cut < 2; ++cut)
            for (int m = 1; m <= 700; ++m) {
                g_second = second;
                printf("%d %d %d", second, cut, m);
                mnpb::in_halves((cudaStream_t)1, m, cut, [](cudaStream_t s, int a, int b) -> int {
                    printf(" %d:%d:%d", s == (cudaStream_t)2, a, b);
                    return 0;
                });
                printf("\n");
            }
}
'''


@pytest.fixture(scope='module')
def calls(tmp_path_factory):
    d = tmp_path_factory.mktemp('halves')
    (d / 'halves.cpp').write_text(PROGRAM)
    cuda = '/usr/local/cuda/include'
    subprocess.run([shutil.which('g++'), '-std=c++17', '-w', '-I' + cuda, '-I' + ROOT + '/include',
                    '-I' + CSRC, str(d / 'halves.cpp'), '-o', str(d / 'halves')], check=True)
    out = subprocess.run([str(d / 'halves')], check=True, capture_output=True, text=True).stdout
    rows = [line.split() for line in out.splitlines()]
    return {tuple(int(v) for v in r[:3]): [tuple(int(v) for v in q.split(':')) for q in r[3:]]
            for r in rows}


def test_parts_cover_the_right_hand_sides_once(calls):
    """Whatever m is, also far below one half's step of 64: no part begins or ends
    outside [0, m), none is empty, and together they are all of it."""
    assert len(calls) == 4 * 700
    for (second, cut, m), parts in calls.items():
        assert all(0 <= a < b <= m for _, a, b in parts), (second, cut, m, parts)
        assert [a for _, a, _ in parts] == [0] + [b for _, _, b in parts[:-1]]
        assert parts[-1][2] == m
        assert len(parts) <= (2 if cut else 1)


def test_second_stream_is_used_where_there_is_enough_to_cut(calls):
    for m in (65, 128, 257, 700):
        assert [p[0] for p in calls[1, 1, m]] == [1, 0]
    assert calls[1, 0, 700] == [(0, 0, 700)]


def test_cut_does_not_depend_on_the_second_stream(calls):
    for cut in range(2):
        for m in range(1, 701):
            assert [p[1:] for p in calls[0, cut, m]] == [p[1:] for p in calls[1, cut, m]]
            assert all(on == 0 for on, _, _ in calls[0, cut, m])
