"""Buffers allocated together (mcx_alloc.h), as the training workspace is: whichever
allocation fails, no pointer of the set survives, nothing leaks, and a later call
starts over."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r'''
#include <cstdio>
#include <cstdlib>
#include <set>
#include "mcx_alloc.h"
static std::set<void *> live;
static int countdown = 0;  // the allocation that fails (0: none)
static int fake_malloc(void **p, size_t n) {
  if (countdown > 0 && --countdown == 0) { *p = (void *)0x1; return 2; }
  *p = malloc(n);
  live.insert(*p);
  return 0;
}
static int fake_free(void *p) {
  if (!live.erase(p)) { printf("freed what was not allocated\n"); exit(1); }
  free(p);
  return 0;
}
int main() {
  void *a = (void *)0x2, *b = (void *)0x3, *c = (void *)0x4;
  for (int bad = 1; bad <= 3; bad++) {
    countdown = bad;
    const int r = mcx::alloc_together({{&a, 8}, {&b, 16}, {&c, 24}}, fake_malloc, fake_free);
    if (r != 2 || a || b || c || !live.empty()) { printf("failure %d: %d %p %p %p, %zu live\n", bad, r, a, b, c, live.size()); return 1; }
  }
  const int r = mcx::alloc_together({{&a, 8}, {&b, 16}, {&c, 24}}, fake_malloc, fake_free);
  if (r || !a || !b || !c || live.size() != 3) { printf("success: %d\n", r); return 1; }
  return 0;
}
'''


def test_all_or_none(tmp_path):
    src = tmp_path / "alloc.cpp"
    src.write_text(SRC)
    exe = str(tmp_path / "alloc")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", os.path.join(ROOT, "mclics-backend_gb300", "csrc"), str(src),
                    "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_training_workspace_is_one_set():
    """Its five buffers come from one alloc_together, so that the guard on the
    first covers the others."""
    with open(os.path.join(ROOT, "mclics-backend_gb300", "csrc", "mcx_engine.cu")) as f:
        body = f.read().split("static mcx_status train_prepare(")[1].split("\n}\n")[0]
    call = body.split("alloc_together({")[1].split("[]")[0]
    assert all("e->" + b in call for b in ("d_w", "d_am", "d_av", "d_g", "d_image"))
    assert body.count("cudaMalloc") == 1
