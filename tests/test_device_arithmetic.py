"""The device arithmetic that stands in for the reference's operations, over
many operands: the fused link solve against the IEEE one, and the clear-edge
test of polygons against the intersection it saves.  A small library built from
the kernels' own source counts the differences."""
import ctypes
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include "kernels.cuh"
using namespace b2d;
struct Rng {  // SplitMix64
  unsigned long long s;
  __device__ uint32_t next() {
    unsigned long long z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return (uint32_t)((z ^ (z >> 31)) >> 16);
  }
  // random sign and significand (one in four near a power of two), exponent lo .. hi
  __device__ float value(int lo, int hi) {
    const uint32_t r = next(), e = (uint32_t)(127 + lo) + next() % (uint32_t)(hi - lo + 1);
    uint32_t m = r & 0x7FFFFFu;
    if ((r >> 23 & 3u) == 0u) m = (r >> 25 & 1u) ? 0x7FFFFFu - (m & 15u) : (m & 15u);
    return __uint_as_float((r & 0x80000000u) | e << 23 | m);
  }
};
__device__ bool differ(float a, float b) {
  return __float_as_uint(a) != __float_as_uint(b) && !(isnan(a) && isnan(b));
}
// kind 0: any differences; 1: both of one magnitude; 2: one of them zero
__global__ void k_solves(unsigned long long seed, int kind, uint32_t n, unsigned long long* bad,
                         unsigned long long* in_range) {
  Rng r{seed + (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x) * 0x100000001ull};
  unsigned long long wrong = 0, met = 0;
  for (uint32_t i = 0; i < n; ++i) {
    float dx = r.value(-50, 62), dy = r.value(-50, 62);
    if (kind == 1) dy = __uint_as_float((__float_as_uint(dy) & 0x807FFFFFu) |
                                        (__float_as_uint(dx) & 0x7F800000u));
    if (kind == 2) (r.next() & 1u ? dx : dy) = 0.0f;
    float2 b = make_float2(0.0f, 0.0f);
    if (r.next() & 1u) b = make_float2(r.value(-20, 20), r.value(-20, 20));
    const float2 a = make_float2(dx + b.x, dy + b.y);
    const float rest = r.next() & 7u ? r.value(-30, 40) : fabsf(dx), stiff = r.value(-4, 0);
    const uint32_t z = 0x80000000u;
    if (__float_as_uint(a.x) == z || __float_as_uint(a.y) == z) continue;
    float2 a0 = a, b0 = b, a1 = a, b1 = b, a2 = a, b2 = b, a3 = a, b3 = b;
    uint32_t low = 0xFFFFFFFFu;
    link_solve_fused<false>(a0, b0, rest, stiff, low);
    if (low < FUSED_MIN_DIFF) continue;
    ++met;
    link_solve(a1, b1, rest, stiff);
    bool w = differ(a0.x, a1.x) || differ(a0.y, a1.y) || differ(b0.x, b1.x) || differ(b0.y, b1.y);
    link_solve_fused<true>(a2, b2, rest, 1.0f, low);
    link_solve_plain(a3, b3, rest, 1.0f);
    w = w || differ(a2.x, a3.x) || differ(a2.y, a3.y) || differ(b2.x, b3.x) || differ(b2.y, b3.y);
    wrong += w;
  }
  atomicAdd(bad, wrong);
  atomicAdd(in_range, met);
}
// edges that are cleared of a disc, against the points in it
__global__ void k_edges(unsigned long long seed, uint32_t n, unsigned long long* bad,
                        unsigned long long* cleared) {
  Rng r{seed + (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x) * 0x100000001ull};
  unsigned long long wrong = 0, met = 0;
  for (uint32_t i = 0; i < n; ++i) {
    const float scale = exp2f((float)(int)(r.next() % 20u) - 8.0f);
    auto u = [&] { return scale * (float)(int)(r.next() & 0xFFFFFFu) / 16777216.0f; };
    const float2 a = make_float2(u(), u()), b = make_float2(u(), u());
    // a centre some way off the edge's line, and a point of its disc towards it
    const float ex = b.x - a.x, ey = b.y - a.y, len = sqrtf(ex * ex + ey * ey) + 1e-30f;
    const float off = u() * 0.5f, along = u() * 2.0f - scale * 0.5f;
    const float2 c = make_float2(a.x + ex / len * along - ey / len * off,
                                 a.y + ey / len * along + ex / len * off);
    const float reach = off * (1.0f - 1e-4f * (float)(r.next() & 255u) * 0.5f);
    const float turn = (float)(int)(r.next() & 0xFFFFu) * 1e-6f;
    const float2 q = make_float2(c.x + reach * (ey / len + turn * ex / len),
                                 c.y - reach * (ex / len - turn * ey / len));
    const float dx = q.x - c.x, dy = q.y - c.y;
    if (!edge_clear(a, b, c, 1.01f * sqrtf(dx * dx + dy * dy))) continue;
    ++met;
    float2 hit;
    wrong += line_intersection(a, b, q, c, hit);
  }
  atomicAdd(bad, wrong);
  atomicAdd(cleared, met);
}
extern "C" int run(int what, unsigned long long seed, uint32_t n, unsigned long long* out) {
  unsigned long long* d;
  if (cudaMalloc(&d, 16) != cudaSuccess || cudaMemset(d, 0, 16) != cudaSuccess) return 1;
  if (what < 3) k_solves<<<608, 256>>>(seed, what, n, d, d + 1);
  else k_edges<<<608, 256>>>(seed, n, d, d + 1);
  const cudaError_t e = cudaMemcpy(out, d, 16, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? 0 : 1;
}
"""


@pytest.fixture(scope="module")
def run(gpu, tmp_path_factory):
    from bendy2d_gb300 import build as b
    nvcc = shutil.which(b._nvcc())
    if nvcc is None:
        pytest.skip("no CUDA compiler")
    d = tmp_path_factory.mktemp("arith")
    (d / "arith.cu").write_text(PROGRAM)
    subprocess.run([nvcc, *b.NVCC_FLAGS, "-shared", f"-I{b.CSRC}", str(d / "arith.cu"), "-o",
                    str(d / "arith.so")], check=True)
    lib = ctypes.CDLL(str(d / "arith.so"))
    lib.run.argtypes = [ctypes.c_int, ctypes.c_ulonglong, ctypes.c_uint32, ctypes.c_void_p]

    def go(what, seed, n):
        out = (ctypes.c_ulonglong * 2)()
        assert lib.run(what, seed, n, out) == 0
        return out[0], out[1]
    return go


@pytest.mark.parametrize("kind", [0, 1, 2])
def test_fused_link_solve_has_the_bits_of_the_ieee_one(run, kind):
    wrong, met = run(kind, 11 + kind, 4000)
    assert met > 4e8 and wrong == 0


def test_cleared_edges_are_not_hit(run):
    wrong, met = run(3, 5, 4000)
    assert met > 5e7 and wrong == 0
