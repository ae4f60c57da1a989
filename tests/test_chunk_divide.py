"""The tap of a 16-byte chunk in the small convolutions (csrc/chunk_divide.h, compiled here with g++): exact for every chunk and every
number of chunks per tap that the size rule admits. A reciprocal of 20 bits gave the wrong tap from 6048 channels on."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "torq-compiler_b200", "csrc")

PROGRAM = r'''
#include <cstdio>
#include "chunk_divide.h"
int main() {
  for (int d = 1; d <= tb200::kMaxChunks; d++) {
    const tb200::ChunkDivisor by = tb200::chunk_divisor(d);
    for (int c = 0; c < tb200::kMaxChunks + 4; c++)
      if (tb200::divide_chunk(c, by) != c / d) {
        printf("%d / %d gives %d\n", c, d, tb200::divide_chunk(c, by));
        return 1;
      }
  }
  for (int kw = 1; kw <= tb200::kMaxTaps; kw++)
    for (int tap = 0; tap < tb200::kMaxTaps + 4; tap++)
      if (tb200::divide_tap(tap, tb200::tap_divisor(kw)) != tap / kw) {
        printf("tap %d / %d\n", tap, kw);
        return 1;
      }
  return 0;
}
'''


def test_taps_of_every_chunk(tmp_path):
    src, exe = tmp_path / "divide.cc", tmp_path / "divide"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
