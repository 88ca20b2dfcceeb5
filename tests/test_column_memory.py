"""Device columns of the a*b - c sumcheck: kernels read them in place only where they may.

CPU: the decision, over made-up reports of where an address lies (another device's memory among them).
GPU: columns at odd addresses give the same proof as the same values on the host."""
import os
import subprocess

import numpy as np
import pytest

SOURCE = """
#include <cstdio>
#include "columns.h"
using wl::ColumnMemory;
int main() {
  int bad = 0;
  auto expect = [&](bool want, ColumnMemory m, int dev, uintptr_t p, size_t bytes) {
    if (wl::read_in_place(m, dev, p, bytes) != want) std::printf("case %zx %zu on %d\\n", size_t(p), bytes, dev), bad++;
  };
  const uintptr_t B = 0x7f0000000000;
  const size_t N = 4096;
  for (int dev = 0; dev < 3; dev++) {
    const ColumnMemory own{true, dev, B, N}, other{true, dev + 1, B, N};
    expect(true, own, dev, B, N);
    expect(true, own, dev, B + 64, N - 64);
    expect(true, own, dev, B + N - 4, 4);
    expect(false, own, dev, B + 4, N);       // past the end
    expect(false, own, dev, B + N, 4);
    expect(false, own, dev, B - 4, 8);       // before it
    expect(false, own, dev, B, N + 4);
    expect(false, own, dev, B, ~size_t(0));  // no wrap
    expect(false, own, dev, B + 1, 4);       // not whole words
    expect(false, own, dev, B + 2, 4);
    expect(false, other, dev, B, N);         // another device
    expect(false, ColumnMemory{false, dev, B, N}, dev, B, N);  // host or managed memory
    expect(false, ColumnMemory{true, dev, 0, 0}, dev, B, N);   // unknown range
    expect(false, ColumnMemory{}, dev, B, N);
  }
  return bad;
}
"""


def test_in_place_decision(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    src, exe = tmp_path / "columns.cpp", tmp_path / "columns"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(root, "whirlaway_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("shifts", [(0, 0, 0), (1, 0, 2), (3, 1, 4)])
def test_columns_at_any_address(wl, ctx, shifts):
    import torch
    log_n, skips = 9, 3
    rng = np.random.default_rng(7)
    cols = [rng.integers(0, 0x7F000001, 1 << log_n, dtype=np.uint32) for _ in range(3)]
    p16 = wl.generate_workload(2)[0][148:296]
    ref, _ = wl.sumcheck_abc_prove(ctx, p16, log_n, skips, *cols)
    held = []
    for v, s in zip(cols, shifts):
        t = torch.zeros(v.nbytes + 16, dtype=torch.uint8, device="cuda")[s:s + v.nbytes]
        t.copy_(torch.from_numpy(v.view(np.uint8)))
        held.append(t)
    torch.cuda.synchronize()
    got, _ = wl.sumcheck_abc_prove(ctx, p16, log_n, skips, *held, device=True)
    assert np.array_equal(got, ref)
