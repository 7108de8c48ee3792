"""The norm's division by the row length (csrc/norm_quantize.cu: div_by), a product and a residual correction, is the
IEEE quotient for every row length that it takes: the formula, and the function as it stands in the source, for all
significands."""
import os
import re
import subprocess

import numpy as np

from blackwell_diffusion_rtx6000_5090_i2v_b200 import build


def test_product_and_correction_equal_the_quotient():
    rng = np.random.default_rng(1)
    for n in range(16, 16385, 16):
        x = np.ldexp(rng.uniform(1, 2, 3000), rng.integers(-80, 120, 3000)).astype(np.float32)
        x *= rng.choice(np.array([-1, 1], np.float32), x.size)
        nf = np.float32(n)
        inv = np.float32(1) / nf
        q0 = x * inv
        # both fused operations: the products are exact in 64 bits, the sums in the extended type
        r = (x.astype(np.float64) - n * q0.astype(np.float64)).astype(np.float32)
        q = (r.astype(np.longdouble) * np.longdouble(inv) + q0).astype(np.float32)
        assert np.array_equal(q, x / nf), n


HARNESS = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#define __device__
#define __forceinline__ inline
static float __fdiv_rn(float a, float b) { return a / b; }
static float __fmul_rn(float a, float b) { return a * b; }
static float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
%s
static float of(uint32_t b) { float f; std::memcpy(&f, &b, 4); return f; }
static uint32_t bits(float f) { uint32_t b; std::memcpy(&b, &f, 4); return b; }
static long wrong = 0;
static void look(float x, float n) {
  const float got = div_by<true>(x, n, 1.0f / n), want = x / n;
  if (bits(got) != bits(want) && !(got != got && want != want) && wrong++ < 5) std::printf("%%a / %%a: %%a, not %%a\n", x, n, got, want);
}
int main() {
  // every significand over every row length, up to powers of two (which change exponents alone)
  for (uint32_t odd = 1; odd < 1024; odd += 2)
    if (odd <= 31)
      for (uint32_t m = 0; m < (1u << 23); ++m) look(of(127u << 23 | m), (float)odd);
    else
      for (uint32_t m = odd; m < (1u << 23); m += 1021) look(of(127u << 23 | m), (float)odd);
  // every exponent and both signs: zeros, subnormals, the ends of the range of the correction, infinities, NaNs
  for (uint32_t n = 16; n <= 16384; n += n < 512 ? 16 : 512)
    for (uint64_t b = n; b < (1ull << 32); b += 30011) look(of((uint32_t)b), (float)n);
  const float ends[] = {1e-25f, 1e37f, 0.0f, INFINITY, NAN};
  for (float e : ends)
    for (int s = -1; s <= 1; s += 2)
      for (uint32_t n = 512; n <= 16384; n += 512)
        for (float x : {e, std::nextafterf(e, 0.0f), std::nextafterf(e, INFINITY)}) look(s * x, (float)n);
  return wrong != 0;
}
"""


def test_the_function_in_the_source(tmp_path):
    with open(os.path.join(build.CSRC, "norm_quantize.cu")) as f:
        found = re.search(r"template <bool kFast>\n__device__ __forceinline__ float div_by\(.*?\n}\n", f.read(), re.S)
    src = tmp_path / "div.cpp"
    src.write_text(HARNESS % found.group(0))
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else os.environ.get("CXX", "g++")
    cmd = [cxx, "-O2", "-std=c++17", "-ffp-contract=off", str(src), "-o", str(tmp_path / "div")]
    # with the machine's own fused operation where it has one: the library's is exact too, and slow
    if os.path.exists("/proc/cpuinfo") and " fma " in open("/proc/cpuinfo").read():
        cmd.append("-mfma")
    subprocess.run(cmd, check=True)
    run = subprocess.run([str(tmp_path / "div")], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
