"""Shared memory of the decode products' blocks (csrc/linear_shape.h, compiled here with g++): what the other blocks of a cluster store
into a block must lie behind everything the block itself uses, since the barrier they wait for only says that the block runs.
Every mode and batch over ragged and round sizes, on more and fewer SMs than a B200 has."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "torq-compiler_b200", "csrc")

PROGRAM = r'''
#include <cstdio>
#include "linear_shape.h"
using namespace tb200;
int main() {
  long long checked = 0, rope = 0, bad = 0;
  const int ns[] = {1, 31, 32, 100, 768, 1024, 1152, 1536, 6912, 13824, 30001, 262144};
  for (int sms : {108, 132, 148, 160})
    for (int mode : {kStore, kGeglu, kRope})
      for (int n : ns)
        for (int k = 64; k <= 8192; k += 64)
          for (int b = 1; b <= 32; b++) {
            const LinearShape s = linear_shape(b, n, k, mode, sms);
            if (!s.ok) continue;
            const int tok = ceil_div(b, 8) * 8, warps = s.kg * s.rt;
            const int staged = s.x_bytes + warps * s.stages * kStageBytes;  // activations and rings
            const int sums = s.tk == 1 && mode != kRope ? 16 * tok * 8 : warps * kTileRows * (tok + 1) * 4;
            // what the epilogue of the mode receives: [8][tokens] and [tokens][32] floats, or every block's share of 32-row sums
            const int recv = mode == kRope ? 8 * tok * 4 + tok * 32 * 4 : s.ck > 1 ? s.ck * ((s.rt * b + s.ck - 1) / s.ck) * 32 * 4 : 0;
            checked++;
            rope += mode == kRope;
            if (s.scale_off < staged || s.scale_off < sums || s.recv_off < s.scale_off + s.rt * kTileRows * 4 || s.recv_off % 16 ||
                s.smem < s.recv_off + recv || s.smem > kSmemMax) {
              if (!bad++) printf("mode %d B %d N %d K %d: staged %d sums %d recv_off %d + %d, smem %d\n", mode, b, n, k, staged, sums, s.recv_off, recv, s.smem);
            }
          }
  printf("%lld shapes, %lld with the RoPE epilogue, %lld bad\n", checked, rope, bad);
  return bad || rope < 1000 || checked < 10000;
}
'''


def test_received_values_have_memory_of_their_own(tmp_path):
    src, exe = tmp_path / "layout.cc", tmp_path / "layout"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
