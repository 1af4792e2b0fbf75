"""The planner's sampled Jaro-Winkler values (csrc/planner.cpp) against a
byte-by-byte scan, at the edges of its 64-bit words, and the order of a rule's
predicates that follows from them."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DRIVER = r"""
#include "CSRC/planner.cpp"
#include <cstdio>
#include <random>
#include <string>
static double scan(const std::string& a, const std::string& b) {
  const size_t la = a.size(), lb = b.size();
  if (!la || !lb) return !la && !lb ? 1.0 : 0.0;
  const size_t ls = std::min(la, lb), ll = std::max(la, lb), h = (ls + 1) / 2;
  std::vector<char> used(la, 0);
  size_t m = 0;
  for (size_t i = 0; i < lb; i++)
    for (size_t j = i > h ? i - h : 0; j < la && j <= i + h; j++)
      if (!used[j] && a[j] == b[i]) { used[j] = 1; m++; break; }
  if (!m) return 0.0;
  double j = ((double)m / ls + (double)m / ll + 1.0) / 3.0;
  size_t p = 0;
  while (p < ls && a[p] == b[p]) p++;
  j += (1.0 - j) * (double)p * 0.1;
  return j > 1.0 ? 1.0 : j;
}
int main() {
  std::mt19937 g(7);
  hbx::Sampler s;
  const size_t lens[] = {0, 1, 2, 31, 32, 63, 64, 65, 127, 128, 129, 191, 192, 256, 257, 700};
  for (int k = 0; k < 20000; k++) {
    std::string t[2];
    const int sigma = 2 + (int)(g() % 6);
    for (auto& x : t) {
      x.resize(lens[g() % 16]);
      for (auto& c : x) c = (char)(k % 2 ? 'a' + g() % sigma : 255 - g() % sigma);
    }
    if (hbx::jaro_winkler(s.count(t[0].data(), t[0].size(), t[1].data(), t[1].size())) !=
        scan(t[0], t[1])) {
      std::printf("%s\n%s\n", t[0].c_str(), t[1].c_str());
      return 1;
    }
  }
  // the predicate that few pairs pass goes first, whatever the rules before it
  hbx::Table L, R;
  for (auto* t : {&L, &R}) {
    t->n_rows = 50;
    t->cols.resize(3);
    for (int c = 0; c < 3; c++) {
      t->cols[c].off.push_back(0);
      for (int i = 0; i < 50; i++) {
        for (int j = 0; j < 20; j++) t->cols[c].bytes.push_back(c ? (char)('a' + g() % (c == 1 ? 2 : 20)) : 'x');
        t->cols[c].off.push_back((int64_t)t->cols[c].bytes.size());
      }
    }
  }
  hbx::Plan p;
  p.compiled.resize(2);
  p.compiled[0].sims = {{'s', 1, 1, 0.1f}, {'s', 2, 2, 0.95f}};
  p.compiled[1].sims = {{'s', 1, 1, 0.99f}, {'s', 2, 2, 0.1f}, {'s', 0, 0, 0.5f}};
  hbx::order_predicates(&p, L, R);
  if (p.compiled[0].sims[0].col_l != 2 || p.compiled[1].sims[0].col_l != 1) return 2;
  return 0;
}
"""


def test_sampled_values_and_order(tmp_path):
    src = tmp_path / "driver.cpp"
    src.write_text(DRIVER.replace("CSRC", os.path.join(ROOT, "hyperblocker_gb300", "csrc")))
    exe = str(tmp_path / "driver")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", "/usr/local/cuda/include",
                    "-I", os.path.join(ROOT, "include"), str(src), "-o", exe], check=True)
    assert subprocess.run([exe]).returncode == 0
