"""What is kept about a kernel's launch shape is kept by device and kernel: two kernels, or
one on two devices, may come with equal threads and shared memory."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "graph-utils_gb300", "csrc")


def test_kept_by_device_and_kernel(tmp_path):
    exe = tmp_path / "kernel_fit_check"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"),
                        "-I/usr/local/cuda/include", os.path.join(ROOT, "tests", "cpp", "kernel_fit_check.cpp"),
                        os.path.join(CSRC, "kernel_fit.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


SEARCHES = """
import sys
import numpy as np, torch, gu, oracle
for n in map(int, sys.argv[1:]):
    hg = gu.HostGraph.from_edges(n, np.concatenate([np.arange(n - 1), np.zeros(40, np.int64)]) % 3000,
                                 np.concatenate([np.arange(1, n), np.arange(1, 41)]))
    g, srcs = gu.Graph(hg), np.array([0, n - 1, 17], np.int32)
    s = torch.as_tensor(srcs, device="cuda")
    d = torch.empty((3, n), dtype=torch.int32, device="cuda")
    g.bfs(s, d)
    np.testing.assert_array_equal(d.cpu().numpy(), oracle.bfs_multi(hg.R, hg.C, n, srcs)[0])
"""


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [(6500, 8600), (8600, 6500), (8000, 10700)])
def test_two_kernels_of_one_shape(sizes):
    """The byte form on 6500 vertices and the one-CTA form on 8600 launch with equal
    threads and shared memory, each as the process's first launch of its kernel."""
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([os.path.join(ROOT, "graph-utils_gb300"), os.path.join(ROOT, "oracle")]))
    r = subprocess.run([sys.executable, "-c", SEARCHES] + [str(n) for n in sizes], capture_output=True, text=True, env=env)
    assert r.returncode == 0, r.stderr[-2000:]
