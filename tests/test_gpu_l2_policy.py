"""The cache-policy words that the kernels pass with their loads are those that ``createpolicy`` gives on this device."""
import importlib.util
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cstdio>
#include <cstdint>
#include "sm100_ptx.cuh"
__global__ void words(uint64_t* out) {
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(out[0]));
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 0.5;" : "=l"(out[1]));
  asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(out[2]));
}
int main() {
  uint64_t* out = nullptr;
  uint64_t got[3] = {}, want[3] = {dx::kL2EvictFirst, dx::kL2EvictFirstHalf, dx::kL2EvictNormal};
  if (cudaMalloc(&out, sizeof(got)) != cudaSuccess) return 2;
  words<<<1, 1>>>(out);
  if (cudaMemcpy(got, out, sizeof(got), cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
  for (int i = 0; i < 3; ++i) printf("%d: kept %016llx, createpolicy %016llx\n", i, (unsigned long long)want[i], (unsigned long long)got[i]);
  return got[0] == want[0] && got[1] == want[1] && got[2] == want[2] ? 0 : 1;
}
"""


def test_words_are_those_of_createpolicy(tmp_path):
    spec = importlib.util.spec_from_file_location("_dxb_build", ROOT / "dexter_labs_b200" / "build.py")
    b = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(b)
    source, program = tmp_path / "words.cu", tmp_path / "words"
    source.write_text(SOURCE)
    subprocess.run([b._nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", str(b.PKG_DIR / "csrc"),
                    str(source), "-o", str(program)], check=True)
    ran = subprocess.run([str(program)], capture_output=True, text=True)
    assert ran.returncode == 0, ran.stdout
