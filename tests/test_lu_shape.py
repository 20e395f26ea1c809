"""The launch choice of the LU-SGS sweeps (csrc/kernels/lu_shape.h) on the
host: every mesh that a solver admits has a launch, in either form that the
batch around it may call for, within the hardware's limits.  No GPU."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
KERNELS = os.path.join(HERE, "..", "turns2d_urans_git_gb300", "csrc", "kernels")

# For every number of rows the longest admitted mesh (shared memory grows with
# the columns, so it stands for the shorter ones) and a few shorter ones.
ADMITTED = r"""
#include <cstdio>
#include "lu_shape.h"
using namespace ot2d;

template <class R, bool PRE>
int check(const char* name) {
  int bad = 0, seen = 0;
  for (int kd = 3; kd <= 1100; ++kd) {
    int top = 0;
    while (lu_mesh_fits(sizeof(R), PRE, kd, top < 3 ? 3 : top + 1)) top = top < 3 ? 3 : top + 1;
    for (int jd : {top, top - 1, top / 2, 130, 3}) {
      if (jd < 3 || jd > top) continue;
      bool ok = lu_batch_fits<R>(PRE, kd, jd);
      for (bool spread : {false, true})
        for (int group : {0, 1, 2, 4, 8}) {
          const LuLaunch l = lu_launch<R, PRE>(kd, jd, spread, group);
          const int nb = lu_nband(kd, LuSplit<R, PRE>::RB);
          ++seen;
          ok = ok && l.cs >= 1 && l.cs <= 8 && l.nw >= 1 && l.nw * 32 <= 512 && l.nw * l.cs >= nb && l.D >= 1 &&
               l.smem <= (size_t)SMEM_OPTIN_MAX &&
               l.smem == (l.pg == 8   ? lu_smem_bytes<R, PRE, 8>(l.cs, l.nw, l.D, jd)
                          : l.pg == 4 ? lu_smem_bytes<R, PRE, 4>(l.cs, l.nw, l.D, jd)
                                      : lu_smem_bytes<R, PRE, 2>(l.cs, l.nw, l.D, jd));
        }
      if (!ok && ++bad <= 5) std::printf("%s: kd %d jd %d has no launch\n", name, kd, jd);
    }
  }
  std::printf("%s: %d launches, %d meshes without\n", name, seen, bad);
  return bad + (seen < 10000);
}

int main() {
  return check<float, false>("f32") + check<float, true>("f32 preconditioned") + check<double, false>("FP64") +
                 check<double, true>("FP64 preconditioned")
             ? 1
             : 0;
}
"""


def run(tmp_path, text):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(text)
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-Werror", "-I", KERNELS, str(src), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], capture_output=True, text=True)


def test_every_admitted_mesh_has_a_launch(tmp_path):
    r = run(tmp_path, ADMITTED)
    assert r.returncode == 0, r.stdout
