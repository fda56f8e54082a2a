"""The words in which a step's last kernel reports to the host: token and error word belong together, whoever reads them when."""
import os
import subprocess

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include "step_words.hpp"
using namespace lcu;
static_assert(packed_words(0x12345678, 0) == 0x12345678u, "the token is the lower half, as the word in front of two that lie in memory");
static_assert(packed_words(-2, NOT_BACK) == 0xfffffffffffffffeu, "neither half spills into the other");
int main() {
  alignas(8) uint64_t at;
  clear_words(&at);
  if (read_words(&at).came()) return 1;
  const int steps = 3000000;
  std::thread gpu([&] {  // one store per step, the next step's as soon as it may
    for (int i = 0; i < steps; ++i) __atomic_store_n(&at, packed_words(i, i), __ATOMIC_RELEASE);
  });
  int bad = 0, last = -1;
  while (last < steps - 1) {
    const step_words w = read_words(&at);
    if (!w.came()) continue;
    if (w.token != w.code || w.code < last) ++bad;
    last = w.code;
  }
  gpu.join();
  int ints[2] = {41, 7};  // what a copy of the two words from the GPU's state gives
  __builtin_memcpy(&at, ints, 8);
  const step_words w = read_words(&at);
  printf("%d\n", bad);
  return bad == 0 && w.token == 41 && w.code == 7 ? 0 : 1;
}
"""


def test_token_and_error_word_are_read_together(tmp_path):
    src, exe = tmp_path / "words.cpp", tmp_path / "words"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I", os.path.join(ROOT, "llama.cu_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
