"""The size a kernel's cluster is launched with is found per device: a device
that is used second is allowed and probed for itself, a refused size falls back
to the portable one, a device where nothing fits says so, and says so only as
long as nothing fits. The header is plain C++: compiled here around a fake of
the CUDA calls that records them."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "trinity_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "trn_cluster.h"
struct Fake {
  bool allowed = false;            /* the attribute, per device */
  int fits = 16, refuse = 0;       /* the largest that can be resident; a size whose launch fails */
  int probes = 0;
};
static Fake dev[70];
static trn::ClusterSizes sizes;
static void call(int d) {
  int got = 0;
  const bool ok = sizes.launch(d, [&](int c) {
    ++dev[d].probes;
    if (c > 8) dev[d].allowed = true;
    return c <= dev[d].fits;
  }, [&](int c) {
    if (c == dev[d].refuse || c > dev[d].fits || (c > 8 && !dev[d].allowed)) return false;
    got = c;
    return true;
  });
  std::printf("%d:%d:%d ", ok ? 1 : 0, got, dev[d].probes);
}
int main() {
  call(0); call(0);                                  /* found once, kept */
  call(1); call(1);                                  /* another device: its own attribute */
  dev[2].fits = 8; call(2); call(2);
  dev[3].fits = 0; call(3); call(3); dev[3].fits = 16; call(3); call(3);
  dev[0].refuse = 16; call(0); dev[0].refuse = 0; call(0);   /* refused once, then the kept size again */
  call(69); call(69);                                /* beyond the table: probed every time */
}
"""


def test_sizes_are_per_device(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I" + CSRC, "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["1:16:1", "1:16:1",
                   "1:16:1", "1:16:1",
                   "1:8:2", "1:8:2",
                   "0:0:2", "0:0:4", "1:16:5", "1:16:5",
                   "1:8:2", "1:16:2",
                   "1:16:1", "1:16:2"]


@pytest.mark.gpu
def test_one_size_on_the_device_at_hand():
    """A coarsening whose levels run in one cluster launches fewer kernels
    than the same one level by level (a captured mesh has no cluster)."""
    import ctypes

    from tests.helpers import gpu_mesh, gpu_state
    from trinity_b200 import meshgen
    from trinity_b200._lib import lib
    from trinity_b200.api import Coarse, Metrics, Partit
    m, u, c = meshgen.make_config("c1", 30)
    counts = []
    for _ in range(2):
        g = gpu_mesh(m, u, c)
        Metrics(g, 0.2, 2).run()
        L = lib()
        L.trn_launch_count.restype = ctypes.c_ulonglong
        before = L.trn_launch_count()
        Coarse(g, Partit(g, 8)).run()
        counts.append(L.trn_launch_count() - before)
        assert (gpu_state(g).alive == 0).any()
        g.close()
    assert counts[0] == counts[1] == 2   # the list, the levels
