"""Bilinear texture lookups in integers and floats (csrc/env_tex.cuh) against
the reference's double expressions (src/utility/sampler.hpp:16-29,
src/texture/image_texture2d.cpp:26-30): bit for bit, on coordinates over all
magnitudes, texture edges and sizes, and texels that leave the safe range."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdio>
#include <random>
#include <vector>
#include "env_tex.cuh"
using namespace trg;
static bool same(f3 a, f3 b) {
  const float x[3] = {a.x, a.y, a.z}, y[3] = {b.x, b.y, b.z};
  for (int k = 0; k < 3; ++k)
    if (fbits(x[k]) != fbits(y[k]) && !(x[k] != x[k] && y[k] != y[k])) return false;
  return true;
}
int main(int argc, char** argv) {
  std::mt19937_64 g(atoi(argv[1]));
  const int ws[] = {1, 2, 3, 5, 64, 255, 1000, 4097}, hs[] = {1, 2, 7, 32, 130};
  auto uni = [&] { return (double)(g() >> 11) * 0x1p-53; };
  long bad = 0, n = 0, slow = 0;
  for (int w : ws) for (int h : hs) for (int kind = 0; kind < 5; ++kind) {
    std::vector<float4> f((size_t)w * h);
    std::vector<uchar4> c((size_t)w * h);
    for (size_t i = 0; i < f.size(); ++i) {
      float* t = &f[i].x;
      for (int k = 0; k < 4; ++k) {
        if (kind == 0) t[k] = (float)uni();
        else if (kind == 1) t[k] = std::ldexp((float)(1 + uni()), (int)(g() % 120) - 60);
        else if (kind == 2) t[k] = (float)(g() % 4);
        else if (kind == 3) t[k] = std::ldexp((float)(uni() - 0.5), (int)(g() % 250) - 125);
        else t[k] = g() % 50 == 0 ? (g() & 1 ? 1e38f : -0.0f) : (float)(g() % 256) / 255.0f;
      }
      c[i] = make_uchar4(g() % 256, kind == 2 ? 255 * (g() & 1) : g() % 256, kind == 4 ? 255 : g() % 256, 0);
    }
    auto coord = [&](int size) {
      switch (g() % 8) {
        case 0: return std::ldexp((float)(1 + uni()), -(int)(g() % 60));
        case 1: return (float)((double)(g() % size) / (size > 1 ? size - 1 : 1));  // on texels
        case 2: return (float)(uni() * 20 - 10);
        case 3: return (float)(g() % 3) - 1.0f;
        case 4: return -std::ldexp((float)(1 + uni()), -(int)(g() % 60));
        case 5: return (float)(((double)(g() % size) + 0.5) / (size > 1 ? size - 1 : 1));  // halfway
        default: return (float)uni();
      }
    };
    for (int i = 0; i < 25000; ++i) {
      const float u = coord(w), v = coord(h);
      float uw, vw;
      tex_wrap(u, v, uw, vw);
      ++n;
      if (!same(env_tex_eval(f.data(), w, h, u, v), env_tex_eval_d(f.data(), w, h, uw, vw)) ||
          !same(env_tex_eval8(c.data(), w, h, u, v), env_tex_eval8_d(c.data(), w, h, uw, vw))) {
        if (++bad < 5) printf("%d x %d kind %d u %a v %a\n", w, h, kind, u, v);
      }
    }
  }
  printf("%ld lookups, %ld differ\n", n, bad);
  return bad != 0;
}
"""


@pytest.mark.parametrize("seed", [1, 2])
def test_lookups_equal_the_double_expressions(tmp_path, seed):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no CUDA toolkit headers")
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text("#include <cstdlib>\n#include <cuda_runtime.h>\n#include <vector_functions.h>\n" + SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I" + inc,
                    "-I" + os.path.join(ROOT, "tracer_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), str(seed)], capture_output=True, text=True)
    print(r.stdout)
    assert r.returncode == 0, r.stdout
