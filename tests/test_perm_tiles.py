"""Tile geometry of the per-block permutes, on the CPU: every element that
k_perm_block_tiles would read and write, with its integer widths, against the
64-bit offsets of the general gather.  Items: permutes of a whole block and
crops of a longer one, whose strides and offsets may pass 2^31."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sparsebackends_b200", "csrc")

SOURCE = r"""
#include <cstdio>
#include <set>
#include <vector>
#include "sb_kernels.hpp"
using namespace sb;

// general gather: output element e reads src_off + sum_r c_r * in_strides[r]
static int64_t general(const BlockPerm& b, int64_t e) {
  int64_t so = b.src_off;
  for (int r = 0; r < b.rank; ++r) {
    so += e % b.out_dims[r] * b.in_strides[r];
    e /= b.out_dims[r];
  }
  return so;
}

// The elements of one tile at positions (u, v), as the kernel computes them.
static bool tile_ok(const BlockPerm& b, const PermTileItem& it, int64_t task, uint32_t cap) {
  uint32_t t = static_cast<uint32_t>(task);
  const uint32_t u0 = (t % it.tiles_u) * it.tu;
  t /= it.tiles_u;
  const uint32_t v0 = (t % it.tiles_v) * it.tv;
  uint32_t bt = t / it.tiles_v;
  const uint32_t nu = it.du - u0 < it.tu ? it.du - u0 : it.tu, nv = it.dv - v0 < it.tv ? it.dv - v0 : it.tv;
  if (nu < 1 || nv < 1 || nv > kPermTileRows || nu * (it.tv | 1) > cap) return false;
  int64_t sb = it.src_off + u0, db = it.dst_off + v0 + static_cast<int64_t>(u0) * it.dv;
  int64_t ostride = static_cast<int64_t>(it.dv) * it.du;
  for (int r = it.q + 1; r < it.rank; ++r) {
    const uint32_t d = it.dims[r], c = bt % d;
    bt /= d;
    sb += static_cast<int64_t>(c) * it.strides[r];
    db += c * ostride;
    ostride *= d;
  }
  for (uint32_t v : {0u, nv / 2, nv - 1})
    for (uint32_t u : {0u, nu / 2, nu - 1}) {
      uint32_t x = v0 + v;
      int32_t off = 0;
      for (int r = 0; r < it.q; ++r) {
        const uint32_t d = it.dims[r], c = x % d;
        x /= d;
        off += static_cast<int32_t>(c * it.strides[r]);
      }
      const int64_t dst = db + v + u * it.dv;
      if (dst < b.dst_off || dst >= b.dst_off + b.len) return false;
      if (sb + off + u != general(b, dst - b.dst_off)) return false;
    }
  return true;
}

int main() {
  int rank, want;
  while (std::scanf("%d %d", &rank, &want) == 2) {
    BlockPerm b{};
    b.rank = rank;
    b.len = 1;
    b.src_off = 7;
    b.dst_off = 5;
    for (int r = 0; r < rank; ++r) {
      long long d, s;
      if (std::scanf("%lld %lld", &d, &s) != 2) return 1;
      b.out_dims[r] = b.in_lim[r] = d;
      b.in_strides[r] = s;
      b.len *= d;
    }
    for (uint32_t cap : {perm_tile_cap(0), perm_tile_cap(3000000), perm_tile_cap(1LL << 40)}) {
      PermTileItem it{};
      int64_t tiles = 0;
      const bool took = perm_tile_item(b, cap, &it, &tiles);
      bool ok = want < 0 || took == (want != 0);
      if (took) {
        const int64_t step = tiles / 3000 + 1;
        for (int64_t t = 0; t < tiles && ok; t += step) ok = tile_ok(b, it, t, cap);
        ok = ok && tile_ok(b, it, tiles - 1, cap);
      }
      std::printf("%d", ok ? 1 : 0);
    }
    std::printf("\n");
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    d = tmp_path_factory.mktemp("perm_tiles")
    (d / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, "-I", "/usr/local/cuda/include", "-o", str(d / "t"),
                    str(d / "t.cpp")], check=True)

    def run(dims, strides, want=-1):
        text = " ".join(map(str, [len(dims), want] + [x for p in zip(dims, strides) for x in p]))
        out = subprocess.run([str(d / "t")], input=text, capture_output=True, text=True, check=True)
        return out.stdout.strip()

    return run


def _strides(full):
    s, acc = [], 1
    for f in full:
        s.append(acc)
        acc *= f
    return s


PERMUTES = [((300, 200), (1, 0)), ((37, 41, 43), (2, 1, 0)), ((40, 1, 700), (2, 0, 1)), ((1, 90, 70), (2, 1, 0)),
            ((5, 6, 7, 8), (3, 0, 2, 1)), ((1500, 3, 900), (1, 2, 0)), ((2, 40000, 9), (1, 0, 2)),
            ((46000, 46000), (1, 0)), ((1, 1, 5), (2, 0, 1))]


@pytest.mark.parametrize("full,perm", PERMUTES)
def test_permutes(check, full, perm):
    s = _strides(full)
    assert check([full[p] for p in perm], [s[p] for p in perm]) == "111"


CROPS = [((400, 30, 20), (300, 20, 10)), ((50000, 50000, 1), (1, 50000, 1)), ((20000, 200000, 3), (1, 200000, 1)),
         ((3, 900000000, 1), (1, 900000000, 1)), ((1, 60000, 60000), (1, 400, 50000)), ((400, 3000000), (300, 1000)),
         ((60000, 60000, 2), (300, 50000, 2))]


@pytest.mark.parametrize("full,kept", CROPS)
def test_crops_of_a_longer_block(check, full, kept):
    """A crop without an axis to read contiguously stays with the gather."""
    contiguous = next(k > 1 for f, k in zip(full, kept) if f > 1)
    assert check(kept, _strides(full), -1 if contiguous else 0) == "111"
