"""The GEMM epilogue's staging of output boxes, run on the CPU against a copy engine that reads as late as it may.

``csrc/gemm_epilogue.cuh`` is compiled for the host with stand-ins for the device primitives of ``ptx.cuh``: tensor memory is an
array, and a bulk store reads its shared-memory source only when a wait of the issuing thread makes it. A staging buffer that is
written while an earlier store may still read it then shows up as wrong output, whatever the timing on a device would be.
"""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "mini_trainer_b200" / "csrc"
CUDA_INC = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"

PTX = r"""
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>
#include <algorithm>
#include <deque>
#include <vector>
using std::min;
namespace mtb {
// One lane runs at a time; lane 0 is the one that issues stores and waits, so it is the one that is simulated.
struct Store { std::vector<const uint8_t*> src; std::vector<int> x, y, z; };
extern std::deque<Store> groups;      // committed, the newest last
extern Store open_group;
void perform(const Store& s);         // reads the source now
extern float tmem[256];               // the lane's row of the accumulator
inline void tma_store_3d(const void*, const void* src, int x, int y, int z) {
  open_group.src.push_back(static_cast<const uint8_t*>(src)); open_group.x.push_back(x); open_group.y.push_back(y); open_group.z.push_back(z);
}
inline void tma_store_2d(const void* m, const void* src, int x, int y) { tma_store_3d(m, src, x, y, 0); }
inline void bulk_commit() { groups.push_back(open_group); open_group = Store(); }
template <int N> inline void bulk_wait_read() { while (groups.size() > N) { perform(groups.front()); groups.pop_front(); } }
inline void fence_proxy_async_smem() {}
inline void tmem_ld_32x32(uint32_t a, uint32_t (&r)[32]) { memcpy(r, tmem + a, 128); }
inline void tmem_ld_wait() {}
inline float2 unpack_bf16(uint32_t u) {
  const uint32_t lo = u << 16, hi = u & 0xffff0000u; float2 f; memcpy(&f.x, &lo, 4); memcpy(&f.y, &hi, 4); return f;
}
inline uint32_t pack_bf16(float a, float b) {   // the test's values are exact in bf16
  uint32_t x, y; memcpy(&x, &a, 4); memcpy(&y, &b, 4); return (x >> 16) | (y & 0xffff0000u);
}
inline float fmax3(float a, float b, float c) { return fmaxf(fmaxf(a, b), c); }
}
inline void __syncwarp() {}
inline float __uint_as_float(unsigned u) { float f; memcpy(&f, &u, 4); return f; }
inline void __threadfence() {}
inline unsigned __shfl_sync(unsigned, unsigned v, int) { return v; }
inline int __shfl_up_sync(unsigned, int v, int) { return v; }
inline unsigned long long atomicAdd(unsigned long long* p, unsigned long long v) { const unsigned long long o = *p; *p += v; return o; }
inline void atomicMax(unsigned long long* p, unsigned long long v) { if (*p < v) *p = v; }
inline void __stcg(float4* p, float4 v) { *p = v; }
inline float4 __ldcg(const float4* p) { return *p; }
#define __expf expf
"""

MAIN = r"""
#include <stdio.h>
#include "gemm_epilogue.cuh"
namespace mtb {
std::deque<Store> groups;
Store open_group;
float tmem[256];
static bool f32;
static int M, N;
static std::vector<float> out;
void perform(const Store& s) {
  for (size_t i = 0; i < s.src.size(); ++i)
    for (int j = 0; j < (f32 ? 32 : 64); ++j) {   // row 0 of the box: chunks are not swizzled there
      float v;
      if (f32) memcpy(&v, s.src[i] + 4 * j, 4);
      else { uint16_t h; memcpy(&h, s.src[i] + 2 * j, 2); const uint32_t u = static_cast<uint32_t>(h) << 16; memcpy(&v, &u, 4); }
      const int x = s.x[i] + j, y = s.y[i];
      if (x < N && y < M) out[(static_cast<size_t>(s.z[i]) * M + y) * N + x] = v;
    }
}
// value of element (z, row, col): a small integer, exact in bf16
static float value(int z, int row, int col) { return static_cast<float>((z * 7 + row / 32 * 11 + col * 3) % 251); }

// A worker's share of the tiles of [Z, M, N], every `step`-th, through quarter q of 128-row units.
template <bool OUT_F32, bool SPLIT>
static int run(int m, int n, int z_count, int first, int step, int q, int splits, bool stale = false) {
  f32 = OUT_F32; M = m; N = n;
  out.assign(static_cast<size_t>(z_count) * m * n, -1.f);
  groups.clear();
  alignas(1024) static uint8_t stage[2 * STORE_BOX];
  memset(stage, 0, sizeof stage);
  const int tm = (m + 127) / 128, tn = (n + 255) / 256;
  std::vector<float> ws(static_cast<size_t>(tm) * tn * splits * SPLIT_UNIT, NAN);   // read before it is written: not a number
  // a launch before this one has given up and left arrivals of its own behind
  std::vector<unsigned long long> counters(static_cast<size_t>(tm) * tn * 4);
  for (size_t i = 0; i < counters.size(); ++i) counters[i] = stale ? (41ull << 16) + 1 + i % 3 : 0;
  EpiParams p{};
  p.M = m; p.N = n; p.alpha = 1.f; p.splits = splits; p.ws = ws.data(); p.counters = counters.data(); p.epoch = 42;
  EpiOut o{nullptr, stage, z_count > 1 ? 0 : -1, 0};
  for (int w = first; w < tm * tn * z_count; w += step) {
    const int z = w / (tm * tn), t = w % (tm * tn), row0 = t % tm * 128, tn0 = t / tm * 256;
    if (z_count > 1) o.z = z;
    for (int s = 0; s < splits; ++s) {
      for (int c = 0; c < 256; ++c) tmem[c] = s == splits - 1 ? value(z, row0 + q * 32, tn0 + c) : 0.f;
      epilogue_quarter<OUT_F32, SPLIT, false, false>(p, o, 0, row0, tn0, q, 0, t, s, false);
    }
  }
  drain_boxes();
  int bad = 0;
  for (int w = first; w < tm * tn * z_count; w += step) {
    const int z = w / (tm * tn), t = w % (tm * tn), row = t % tm * 128 + q * 32, tn0 = t / tm * 256;
    if (row >= m) continue;
    for (int c = tn0; c < n && c < tn0 + 256; ++c) bad += out[(static_cast<size_t>(z) * m + row) * n + c] != value(z, row, c);
  }
  if (!stale) for (unsigned long long c : counters) bad += c != 0;
  return bad;
}
}
int main() {
  using namespace mtb;
  int total = 0;
  const int ms[] = {128, 129, 161, 193, 225, 256, 385, 33, 8}, ns[] = {64, 72, 256, 320, 768, 1032};
  for (int m : ms) for (int n : ns) for (int q = 0; q < 4; ++q) for (int step = 1; step <= 3; ++step) {
    const int b = run<false, false>(m, n, 1, 0, step, q, 1) + run<true, false>(m, n, 1, 0, step, q, 1) + run<false, true>(m, n, 1, 0, step, q, 3)
                  + run<true, true>(m, n, 1, 0, step, q, 2) + run<false, false>(m, n, 3, 0, step, q, 1)
                  + run<false, true>(m, n, 1, 0, step, q, 4, true) + run<true, true>(m, n, 1, 0, step, q, 2, true);
    if (b) printf("m %d n %d quarter %d step %d: %d wrong elements\n", m, n, q, step, b);
    total += b;
  }
  printf("wrong %d\n", total);
  return total != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not (CUDA_INC / "cuda_bf16.h").exists(), reason="no host compiler or CUDA headers")
def test_staged_boxes_are_not_overwritten_before_they_are_read(tmp_path):
    """Row counts with quarters past the last row, column counts with odd numbers of boxes, several tiles per worker, both
    output types, split reductions (also behind a launch that gave up) and one matrix per expert."""
    shutil.copy(CSRC / "gemm_epilogue.cuh", tmp_path)
    (tmp_path / "ptx.cuh").write_text(PTX)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "epilogue"
    build = subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CUDA_INC), "-o", str(exe), str(tmp_path / "main.cpp")],
                           capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout[-2000:]
