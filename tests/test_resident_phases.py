"""The resident sweeps' exchange (mcx_phase.h) as a model on the CPU: CTAs of two
warps, messages that arrive in any order, masks whose cuts have rows of one colour
only.  Over random schedules every wait must end with all of its bytes there, every
read must see the sweep it is meant to, and no CTA may get stuck."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r'''
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "mcx_phase.h"
static bool one_bar;  // the mistake to find: one barrier for the rows of colour 1
static int hbar(int c, int i) { return one_bar ? c : mcx::halo_bar(c, i); }
static unsigned hpar(int c, int i) { return one_bar ? (unsigned)i & 1u : mcx::halo_parity(c, i); }
struct Bar { int phase = 0, pending = 1, tx = 0; void look() { if (!pending && !tx) { phase++; pending = 1; } } };
struct Msg { int to, bar, bytes, kind, sweep, from; };  // kind: colour of a halo row, 2 acceptances
constexpr int N = 4, W = 2;
struct World {
  std::mt19937 g;
  int n, sweeps, w[N][W][N][2] = {}, idle[N][W][N] = {};
  bool link[N][N] = {};
  Bar bar[N][mcx::kResBars];
  int due[N][3][64] = {}, got[N][3][64] = {};  // messages of a kind and sweep
  int version[N][N][2];                         // newest halo rows from a CTA
  int pc[N][W] = {}, at[N][W] = {}, sync_at[N][2][64] = {};
  std::vector<Msg> fly;
  const char *bad = nullptr;
  int rnd(int k) { return (int)(g() % (unsigned)k); }
  explicit World(unsigned seed) : g(seed) {
    n = 2 + rnd(3);
    sweeps = 8;
    for (int a = 0; a < n; a++)
      for (int d : {1, n - 1}) {
        const int b = (a + d) % n;
        if (a != b) link[a][b] = true;
      }
    const int style = rnd(3);  // every row active; each colour at random; rows of one colour
    for (int a = 0; a < n; a++)
      for (int b = 0; b < n; b++)
        for (int c = 0; c < 2 && link[a][b]; c++) {
          const bool on = style == 0 || (style == 1 ? rnd(2) : c == (a + b) % 2);
          for (int q = 0; q < W; q++) w[a][q][b][c] = on && (style == 0 || rnd(2)) ? 1 + rnd(3) : 0;
        }
    for (int a = 0; a < n; a++)
      for (int q = 0; q < W; q++)
        for (int b = 0; b < n; b++) idle[a][q][b] = link[a][b] && rnd(2);
    for (auto &x : version) for (auto &y : x) y[0] = y[1] = -1;
    for (int b = 0; b < n; b++)
      for (int i = 0; i < sweeps; i++) {
        for (int a = 0; a < n; a++)
          for (int q = 0; q < W; q++) for (int c = 0; c < 2; c++) due[b][c][i] += w[a][q][b][c] > 0;
        due[b][2][i] = n * W;
      }
  }
  int bytes(int b, int c) { int s = 0; for (int a = 0; a < n; a++) for (int q = 0; q < W; q++) s += w[a][q][b][c]; return s; }
  void arm(int a, int k, int b) { bar[a][k].tx += b; bar[a][k].pending--; bar[a][k].look(); }
  bool done(int a, int k, unsigned parity) { return ((unsigned)bar[a][k].phase & 1u) != parity; }
  void need(int a, int kind, int i) { if (got[a][kind][i] != due[a][kind][i]) bad = "a wait ended without its bytes"; }
  void read(int a, int q, int c, int i) {  // the halo rows of the other colour
    for (int b = 0; b < n; b++)
      if (w[b][0][a][1 - c] + w[b][1][a][1 - c] > 0 && (w[a][q][b][c] > 0 || (c == 1 && idle[a][q][b])) &&
          version[b][a][1 - c] != (c == 1 ? i : i - 1))
        bad = "a halo row of another sweep was read";
  }
  void send(int a, int q, int c, int i) {
    for (int b = 0; b < n; b++)
      if (w[a][q][b][c]) fly.push_back({b, hbar(c, i), w[a][q][b][c], c, i, a});
  }
  bool sync(int a, int k, int i, int q) {  // both warps arrive; each leaves when both have
    sync_at[a][k][i] |= 1 << q;
    return sync_at[a][k][i] == 3;
  }
  // one step of a warp; false: it waits
  bool step(int a, int q) {
    const int i = at[a][q];
    if (i >= sweeps) return false;
    switch (pc[a][q]) {
      case 0:
        if (q == 0) { arm(a, mcx::count_bar(i), n * W); arm(a, hbar(0, i), bytes(a, 0)); }
        read(a, q, 0, i);
        break;
      case 1: send(a, q, 0, i); break;
      case 2: if (!sync(a, 0, i, q)) return false; break;
      case 3: if (q == 0) arm(a, hbar(1, i), bytes(a, 1)); break;
      case 4: if (!done(a, hbar(0, i), hpar(0, i))) return false; need(a, 0, i); break;
      case 5: read(a, q, 1, i); break;
      case 6: send(a, q, 1, i); break;
      case 7: for (int b = 0; b < n; b++) fly.push_back({b, mcx::count_bar(i), 1, 2, i, a}); break;
      case 8: if (!sync(a, 1, i, q)) return false; break;
      case 9: if (!done(a, hbar(1, i), hpar(1, i))) return false; need(a, 1, i); break;
      case 10:
        if (!done(a, mcx::count_bar(i), mcx::count_parity(i))) return false;
        need(a, 2, i);
        if (i + 2 < sweeps && got[a][2][i + 2]) bad = "a counter was added to before it was read";
        break;
    }
    if (++pc[a][q] == 11) { pc[a][q] = 0; at[a][q]++; }
    return true;
  }
  const char *run() {
    const int slow = rnd(n), lag = rnd(4);  // one CTA's messages, or one CTA, may be late
    for (long t = 0; t < 200000 && !bad; t++) {
      bool left = !fly.empty();
      for (int a = 0; a < n; a++) for (int q = 0; q < W; q++) left |= at[a][q] < sweeps;
      if (!left) return nullptr;
      if (!fly.empty() && rnd(3) == 0) {
        const int k = rnd((int)fly.size());
        if (lag == 1 && fly[k].from == slow && rnd(20)) continue;
        const Msg m = fly[k];
        fly.erase(fly.begin() + k);
        got[m.to][m.kind][m.sweep]++;
        if (m.kind < 2) version[m.from][m.to][m.kind] = m.sweep;
        bar[m.to][m.bar].tx -= m.bytes;
        bar[m.to][m.bar].look();
      } else {
        const int a = rnd(n);
        if (lag == 2 && a == slow && rnd(20)) continue;
        step(a, rnd(W));
      }
    }
    return bad ? bad : "stuck";
  }
};
int main(int argc, char **argv) {
  one_bar = argc > 1;
  int found = 0;
  for (unsigned s = 0; s < 6000; s++) {
    World w(s);
    if (const char *b = w.run()) { if (!found++) printf("%s (%u)\n", b, s); }
  }
  printf("%d\n", found);
  return found ? 1 : 0;
}
'''


def test_no_phase_completes_early(tmp_path):
    src = tmp_path / "phases.cpp"
    src.write_text(SRC)
    exe = str(tmp_path / "phases")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "mclics-backend_gb300", "csrc"), str(src),
                    "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    # with one barrier for colour 1 in the model, rows of the next sweep complete a
    # phase early or leave it short for good
    out = subprocess.run([exe, "one"], capture_output=True, text=True)
    assert out.returncode == 1 and ("stuck" in out.stdout or "without its bytes" in out.stdout), out.stdout
