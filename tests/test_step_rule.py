"""The FP32 step-size rule (mcx_step.h) against the reference's float/double
expression (src/evolve.cpp:169-178), for every mantissa of the binades the rule
moves in, and the edges of its range."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r'''
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include "mcx_step.h"
static float ref(float av, unsigned acc, unsigned valid) {
  const double ratio = 1.0 * (double)acc / (double)valid;
  if (ratio < 0.5) {
    av = (float)((double)av * 0.99);
    if ((double)av < 0.01) av = (float)0.01;
  } else if (ratio > 0.5) {
    av = (float)((double)av / 0.99);
    if ((double)av > 1.0) av = (float)((double)av - 0.5);
  }
  return av;
}
static long bad = 0;
static void one(float v, unsigned acc, unsigned valid) {
  const float a = mcx::next_step(v, acc, valid), b = ref(v, acc, valid);
  if (memcmp(&a, &b, 4) != 0 && !(a != a && b != b)) {
    if (bad++ < 5) printf("step %.9g acc %u/%u: %.9g, want %.9g\n", v, acc, valid, a, b);
  }
}
int main() {
  for (int ex = -7; ex <= 3; ex++)  // 2^-7 < 0.01 .. 2^3
    for (uint32_t m = 0; m < (1u << 23); m += (ex >= -7 && ex <= 1) ? 1 : 17) {
      const uint32_t b = ((uint32_t)(127 + ex) << 23) | m;
      float v;
      memcpy(&v, &b, 4);
      one(v, 1, 4);
      one(v, 3, 4);
    }
  const float edge[] = {0.f, -0.f, 1e-38f, 1e-7f, 9.9e-7f, 1e-6f, 0.01f, 0.00999f, 1.f, 0.99f, 1e5f, 1e6f, 1e7f, 3e38f, -0.3f, INFINITY, NAN};
  const unsigned cnt[][2] = {{0, 1}, {1, 2}, {1, 1}, {1073741823u, 2147483647u}, {1073741824u, 2147483647u}, {2147483647u, 2147483647u}, {5, 10}, {4, 9}};
  for (float v : edge)
    for (auto &c : cnt) one(v, c[0], c[1]);
  printf("bad %ld\n", bad);
  return bad != 0;
}
'''


def test_step_rule_is_the_references(tmp_path):
    src = tmp_path / "step.cpp"
    src.write_text(SRC)
    exe = str(tmp_path / "step")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "mclics-backend_gb300", "csrc"), str(src), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
