"""The shared-memory opt-in of the launchers (pelica_b200/csrc/optin.h) is kept per device and only ever raised, whatever
devices and host threads launch. Host code: compiled and run here; two GPUs in one process where there are two."""
import glob
import os
import re
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pelica_b200", "csrc")

PROGRAM = r"""
#include "optin.h"
#include <cassert>
#include <thread>
#include <vector>
static SmemOptIn opt;
static int force[70], sets;  // what a device has in force
int main() {
  auto set = [](int dev) { return [dev](int b) { sets++; force[dev] = b; return 0; }; };
  // every device is asked once, and again only for more
  for (int dev : {0, 1, 63}) {
    assert(opt.raise(dev, 100, set(dev)) == 0 && force[dev] == 100);
    assert(opt.raise(dev, 60, set(dev)) == 0 && force[dev] == 100);
    assert(opt.raise(dev, 150, set(dev)) == 0 && force[dev] == 150);
  }
  assert(sets == 6);
  // an index past the table is asked every time
  for (int i = 0; i < 2; i++) assert(opt.raise(64, 100, set(64)) == 0);
  assert(sets == 8);
  // a refusal is handed back and not remembered
  assert(opt.raise(2, 100, [](int) { return 7; }) == 7);
  assert(opt.raise(2, 100, set(2)) == 0 && force[2] == 100);
  // threads with different needs: the largest stays, and what a call was promised is in force when it returns
  std::vector<std::thread> ts;
  static std::atomic<int> bad{0};
  for (int t = 0; t < 8; t++)
    ts.emplace_back([t] {
      for (int i = 0; i < 2000; i++) {
        const int b = 1000 + (t * 37 + i * 11) % 500;
        static std::atomic<int> now{0};
        opt.raise(3, b, [](int v) { now.store(v); return 0; });
        if (now.load() < b) bad++;
      }
    });
  for (auto &t : ts) t.join();
  assert(bad == 0);
  return 0;
}
"""


def test_opt_in_bookkeeping(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), "-o", str(exe)])
    subprocess.check_call([str(exe)], timeout=60)


def test_launchers_keep_it_nowhere_else():
    """Every use of the attribute goes through the helper."""
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        assert "cudaFuncSetAttribute" not in text, path


@pytest.mark.gpu
def test_two_devices_in_one_process(ctx, oracle):
    """Routing of many experts and wide rows (every opt-in kernel) on a second GPU after the first."""
    import torch

    import pelica_b200 as pb
    from pelica_b200 import synth
    from tests.helpers import SMALL, bits_equal, make_pair

    if torch.cuda.device_count() < 2:
        pytest.skip("one GPU")
    cfg = SMALL["c1"].scaled(d=7168, n_exp=160, ff=256)
    x = synth.make_activations(520, cfg.d, 7)
    for c in (ctx, pb.Context(1)):
        ol, gl, _ = make_pair(oracle, pb, c, cfg, 6)
        for T in (3, 9, 520):
            ids, w = gl.route(x[:T])
            got = gl.forward(x[:T])
            if T < 16:
                assert bits_equal(got, ol.forward(x[:T]))
            assert np.array_equal(ids, ol.route(x[:T])[0])
        gl.close()
