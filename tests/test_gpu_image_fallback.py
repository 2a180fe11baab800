"""The image of a small world where a cluster of its size cannot run (a partitioned device): the
library is linked with a render.cu for which the runtime reports no room and refuses the launch."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

FAKE = r"""
#include <cuda_runtime.h>
template <class K>
static cudaError_t no_clusters(int* n, K*, const cudaLaunchConfig_t*) {
  *n = 0;
  return cudaSuccess;
}
template <class... A>
static cudaError_t no_launch(const cudaLaunchConfig_t*, A&&...) {
  return cudaErrorInvalidClusterSize;
}
#define cudaOccupancyMaxActiveClusters no_clusters
#define cudaLaunchKernelEx no_launch
"""

CHECK = r"""
import sys
import numpy as np
from sandengine_gb300 import _lib
_lib.LIB_PATH = sys.argv[1]
import sandengine_gb300 as se
from sandengine_gb300 import workloads as wl
from oracle.build import Port
text = wl.ruleset_text(wl.TWELVE)
rs, port = se.parse_string(text), Port(text)
for W, H in ((1, 1), (64, 64), (191, 255), (256, 192)):
    sim = se.Simulation(rs, (W, H))
    g = wl.patch_fill(W, H, 6, *wl.twelve_fill_spec(), patch=8)
    sim.grid = g
    want = port.composite(port.color(g), None)
    for _ in range(2):
        assert np.array_equal(sim.composite().view(np.uint32), want.view(np.uint32)), (W, H)
print("same images")
"""


def test_image_without_room_for_its_cluster(built_lib, tmp_path):
    from sandengine_gb300 import build as B
    root = os.path.dirname(B.HERE)
    fake, obj, so = tmp_path / "fake.h", tmp_path / "render.o", tmp_path / "lib.so"
    fake.write_text(FAKE)
    common = [B.NVCC, *B.ARCH, "-O2", "-std=c++20", "-Xcompiler", "-fPIC,-fvisibility=hidden"]
    subprocess.run([*common, "-include", str(fake), "-I", B.OUT, "-I", B.CSRC, "-I", os.path.join(root, "include"), "-c",
                    os.path.join(B.CSRC, "kernels", "render.cu"), "-o", str(obj)], check=True)
    others = [os.path.join(B.OUT, r.replace("/", "_") + ".o") for r in B.HOST_SOURCES + B.CUDA_SOURCES
              if not r.endswith("render.cu")]
    subprocess.run([B.NVCC, "-shared", *B.ARCH, "-cudart", "static", *others, str(obj), "-o", str(so), "-L",
                    os.path.join(B.CUDA_HOME, "lib64"), "-lnvrtc", "-Xlinker",
                    "-rpath," + os.path.join(B.CUDA_HOME, "lib64")], check=True)
    r = subprocess.run([sys.executable, "-c", CHECK, str(so)], cwd=root, capture_output=True, text=True)
    assert r.returncode == 0 and "same images" in r.stdout, r.stdout + r.stderr
