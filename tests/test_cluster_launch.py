"""The launch of a small batch's kernel of whole steps, against a CUDA runtime
that refuses: on a second device (the attribute for clusters of more than eight
blocks belongs to one device), where only eight blocks are to be had, and where
no cluster is."""
import os
import subprocess

import pytest

from godar_b200 import build

MAIN = r"""
#include <cstdio>
#include "kernels.h"
using namespace godar;
// a stand-in for the CUDA runtime: the attribute is kept per device, and a
// cluster of more than `limit` blocks, or of more than eight without the
// attribute, is refused
static int device, limit, refused, launched, wide[4];
extern "C" cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute a, int v)
{
    if (a == cudaFuncAttributeNonPortableClusterSizeAllowed) wide[device] = v;
    return cudaSuccess;
}
extern "C" cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *, void **)
{
    const int n = (int)c->gridDim.x;
    if (n > 1 && (n > limit || (n > 8 && !wide[device]))) { refused++; return cudaErrorInvalidClusterSize; }
    launched = n;
    return cudaSuccess;
}
__global__ void k(int) {}
static void go(ClusterLimit &m, long long items)
{
    launched = 0;
    const bool ok = launch_cluster(m, true, k, cluster_blocks(items, items <= 1024), (cudaStream_t)0, 1);
    std::printf("%lld:%d:%d:%d ", items, (int)ok, launched, refused);
}
int main()
{
    const long long sizes[] = {1, 1024, 1025, 2049, 4096, 4096};
    for (int q = 0; q < 4; q++) {
        device = q < 2 ? q : 2 + (q & 1);
        limit = q < 2 ? 16 : q == 2 ? 8 : 1;
        refused = 0;
        ClusterLimit m;
        for (long long n : sizes) go(m, n);
        std::printf("\n");
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    d = tmp_path_factory.mktemp("cluster")
    src, exe = d / "cluster.cu", d / "cluster"
    src.write_text(MAIN)
    subprocess.check_call([build.NVCC] + build.ARCH + ["-std=c++17", "--cudart", "shared", "-I", build.CSRC, str(src),
                                                       "-o", str(exe)])
    env = dict(os.environ)
    lib = os.path.join(os.path.dirname(os.path.dirname(build.NVCC)), "lib64")
    env["LD_LIBRARY_PATH"] = lib + os.pathsep + env.get("LD_LIBRARY_PATH", "")
    out = subprocess.check_output([str(exe)], text=True, env=env).strip().splitlines()
    return [[tuple(map(int, w.split(":"))) for w in line.split()] for line in out]


def test_every_device_gets_the_same_clusters(rows):
    want = [(1, 1, 1, 0), (1024, 1, 1, 0), (1025, 1, 8, 0), (2049, 1, 16, 0), (4096, 1, 16, 0), (4096, 1, 16, 0)]
    assert rows[0] == want
    assert rows[1] == want


def test_eight_blocks_where_sixteen_are_refused(rows):
    # one refusal, and then none is asked for again
    assert rows[2] == [(1, 1, 1, 0), (1024, 1, 1, 0), (1025, 1, 8, 0), (2049, 1, 8, 1), (4096, 1, 8, 1),
                       (4096, 1, 8, 1)]


def test_no_cluster_leaves_the_single_block(rows):
    assert [r[:3] for r in rows[3]] == [(1, 1, 1), (1024, 1, 1), (1025, 0, 0), (2049, 0, 0), (4096, 0, 0), (4096, 0, 0)]
    assert rows[3][-1][3] == 1
