"""Shared-memory budgets of the fixed-point kernels of the FP64 form (galaexi_gb300/csrc/dg_volume_fx.cuh,
dg_volume_wfx.cuh, dg_lift_fx.cuh, dg_lift_gfx.cuh): every block fits GB300's 227 KB, static arrays included, and the
blocks per SM that the lifting kernels' register limits are made for fit its 228 KB (1 KB reserved per block).  The
sizes come from the headers' constexpr structs through a host program built with nvcc; no GPU is needed.
"""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "galaexi_gb300", "csrc")

SM_BYTES = 228 * 1024
BLOCK_MAX = 227 * 1024
RESERVED = 1024

HARNESS = r"""
#include "dg_lift_gfx.cuh"
#include "dg_volume_wfx.cuh"
#include <cstdio>
template <int NP> void print() {
  using namespace gx;
  const size_t words = 64;  // side list and flags
  const size_t sv = sizeof(VolFxBasis<NP>) + sizeof(VolFxScale) + 4 * X_N + words;
  const size_t sw = sizeof(VolWfxScale) + 4 * W_N + words, sl = 16 + words;
  const size_t sg = sizeof(LiftGfxScale) * 4 + sizeof(FxDig) * NP + 60 + words;
  printf("volume_ns %d %zu %d\n", NP, VolFx<NP>::smem(1) + sv, 0);
  printf("volume_euler %d %zu %d\n", NP, VolFx<NP>::smem(0) + sv, 0);
  printf("weak %d %zu %d\n", NP, VolWfx<NP>::smem + sw, 0);
  printf("lift %d %zu %d\n", NP, LiftFx<NP>::smem + sl, LiftFx<NP>::MINB);
  printf("lift_general %d %zu %d\n", NP, LiftGfx<NP>::smem + sg, LiftGfx<NP>::MINB);
}
int main() {
  print<3>(); print<4>(); print<5>(); print<6>(); print<7>(); print<8>(); print<9>(); print<10>();
  return 0;
}
"""


def test_fixed_point_kernels_fit(tmp_path):
    nvcc = shutil.which("nvcc")
    if not nvcc:
        pytest.skip("needs nvcc")
    src, exe = tmp_path / "smem.cu", tmp_path / "smem"
    src.write_text(HARNESS)
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-I", CSRC, str(src), "-o",
                    str(exe)], check=True, capture_output=True, timeout=600)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout
    seen = {}
    for line in out.splitlines():
        kernel, NP, size, blocks = line.split()
        seen[kernel, int(NP)] = int(size)
        assert int(size) <= BLOCK_MAX, line
        assert int(blocks) * (int(size) + RESERVED) <= SM_BYTES, line
    assert len(seen) == 5 * 8
    # k_volume_fx at N = 3, Navier-Stokes: 15 blocks of one warp per SM
    assert 15 * (seen["volume_ns", 4] + RESERVED) <= SM_BYTES, seen["volume_ns", 4]
