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
     for (bool logits : {false, true})
      for (int n : ns)
        for (int k = 64; k <= 8192; k += 64)
          for (int b = 1; b <= 32; b++) {
            const LinearShape s = linear_shape(b, n, k, mode, sms, logits);
            if (!s.ok) continue;
            const int tok = ceil_div(b, 8) * 8, warps = s.kg * s.rt;
            const int staged = s.x_bytes + warps * s.stages * kStageBytes;  // activations and rings
            const int sums = s.tk == 1 && mode == kStore ? 16 * tok * 8 : warps * kTileRows * (tok + 1) * 4;
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

# A product over the vocabulary (one group of K): [bf16 rows][warps' rings][scales], as many warps of 16, 8, 4, 2, 1 as fit. Slices may not
# take it away, nor leave it fewer warps (8 for 16 where that is less than 1.8 times as many rounds); and what stands at side_off (a shift
# per token; the sums of a norm in front: two tokens, two norms, 16 warps) lies behind the activations and inside their bytes.
VOCABULARY = r'''
#include <cstdio>
#include "linear_shape.h"
using namespace tb200;
int main() {
  long long checked = 0, sliced = 0, bad = 0;
  for (int n : {28500, 65536, 100000, 262144})
    for (int k = 64; k <= 16384; k += 64)
      for (int b = 1; b <= 32; b++) {
        const int rows = ((b + 7) / 8 * 8 * ((k * 2 + 127) / 128 * 128 + 16) + 127) / 128 * 128;
        int warps = 16;
        while (warps >= 1 && rows + warps * (4 * 2048 + 128) > kSmemMax) warps /= 2;
        const LinearShape s = linear_shape(b, n, k, kStore, 148, true);
        const LinearShape layer = linear_shape(b, n, k, kStore, 148, false);
        if (layer.sliced || layer.ok != (warps > 0)) bad++, printf("B %d N %d K %d: bf16 result, ok %d, sliced %d\n", b, n, k, layer.ok, layer.sliced);
        if (!warps) {
          if (s.ok && !s.sliced) bad++, printf("B %d N %d K %d: rows do not fit\n", b, n, k);
          continue;
        }
        checked++;
        sliced += s.ok && s.sliced;
        const int held = s.sliced ? (b * kSlices + 7) / 8 * 8 * k : b * 2 * k;
        const int tiles = (n + 31) / 32, r8 = (tiles + 8 * 148 - 1) / (8 * 148), r16 = (tiles + 16 * 148 - 1) / (16 * 148);
        const bool enough = s.kg * s.rt >= warps || (warps == 16 && s.kg * s.rt == 8 && s.sliced && r8 < 1.8 * r16);
        if (!s.ok || s.tk != 1 || !enough || s.side_off < held || (s.sliced && s.side_off + 4 * b > s.x_bytes)) {
          if (!bad++) printf("B %d N %d K %d: ok %d, %d warps (%d), side_off %d, x_bytes %d\n", b, n, k, s.ok, s.rt, warps, s.side_off, s.x_bytes);
        }
      }
  long long norms = 0;
  for (int mode : {kGeglu, kRope})
    for (int n : {1536, 13824})
      for (int k = 64; k <= 2048; k += 64)
        for (int b = 1; b <= kNormTokens; b++) {
          const LinearShape s = linear_shape(b, n, k, mode, 148, false);
          if (!s.ok || s.ck != 1) continue;
          norms++;
          if (s.side_off < 8 * 2 * k || s.side_off + 2 * 2 * 16 * 4 > s.x_bytes) bad++, printf("norm: mode %d B %d N %d K %d\n", mode, b, n, k);
        }
  printf("%lld products, %lld sliced, %lld with room for a norm, %lld bad\n", checked, sliced, norms, bad);
  return bad || checked < 10000 || sliced < 1000 || norms < 100;
}
'''


def test_received_values_have_memory_of_their_own(tmp_path):
    _run(tmp_path, PROGRAM)


def test_slices_of_the_vocabulary_product_take_no_warps(tmp_path):
    _run(tmp_path, VOCABULARY)


def _run(tmp_path, program):
    src, exe = tmp_path / "layout.cc", tmp_path / "layout"
    src.write_text(program)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
