"""The second phase's pools of product integrands: their size by the memory at
hand (include/cubature/pool_size.hpp, built for the host with g++), and on a
GPU what a context holds, and that it gives the pools up for region lists."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]

SRC = r"""
#include <cstdio>

#include "cubature/pool_size.hpp"

using cubature::PoolBound;
using cubature::pool_blocks;

#define CHECK(x) if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; }

int main() {
  const size_t GB = size_t(1) << 30;
  PoolBound b;
  b.share = 22 * GB;
  // all blocks where they fit the share, also when few are wanted
  CHECK(pool_blocks(740, 111, 5 << 20, b) == 740);
  CHECK(pool_blocks(1, 111, 5 << 20, b) == 1);
  // blocks of 128 MB: the share; of 512 MB: `least`, above the share, below half
  CHECK(pool_blocks(740, 111, GB / 8, b) == 176);
  CHECK(pool_blocks(740, 111, GB / 2, b) == 111);
  // `least` never takes more than half of what was free, and 1 is the minimum
  CHECK(pool_blocks(740, 111, 8 * GB, b) == 11);
  CHECK(pool_blocks(740, 111, 1000 * GB, b) == 1);
  // sizes that were refused are not asked for again: the next call starts
  // with the size that fitted the last
  long long n = pool_blocks(740, 111, GB / 64, b);
  CHECK(n == 740);
  int refused = 0;
  const size_t room = 2 * GB;
  while (n * (GB / 64) > room) {
    b.refused = n * (GB / 64);
    n = pool_blocks(740, 111, GB / 64, b);
    ++refused;
  }
  CHECK(refused == 3 && n == 92);
  CHECK(pool_blocks(740, 111, GB / 64, b) == 92);
  CHECK(pool_blocks(50, 111, GB / 64, b) == 50);
  // another block size: still below the refused bytes
  CHECK(pool_blocks(740, 111, GB / 48, b) * (GB / 48) < b.refused);
  b.refused = 1;
  CHECK(pool_blocks(740, 111, GB, b) == 1);
  std::printf("ok\n");
  return 0;
}
"""


def test_pool_blocks(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("needs g++")
    src = tmp_path / "pool.cpp"
    src.write_text(SRC)
    subprocess.run([gxx, "-O1", "-std=c++17", f"-I{ROOT / 'include'}", str(src), "-o",
                    str(tmp_path / "pool")], check=True, capture_output=True, text=True)
    r = subprocess.run([str(tmp_path / "pool")], capture_output=True, text=True)
    assert r.stdout == "ok\n", r.stdout


def _two_phase(cub, ctx, n, count, max_regions, seed=4):
    rng = np.random.default_rng(seed)
    params = [cub.make_params(n, list(rng.uniform(12, 25, n)), list(rng.uniform(0.3, 0.7, n)))
              for _ in range(count)]
    return ctx.integrate_batch("product_peak", n, params, 1e-4, 1e-12,
                               cub.options(phase1_cap=4096, phase2_max_regions=max_regions))


@pytest.mark.gpu
def test_pools_of_many_bisections_are_bounded(cub):
    """65 536 bisections instead of 2048: 105 GB for all the boxes in flight."""
    import torch

    with cub.Context(0) as ctx:
        free = torch.cuda.mem_get_info()[0]
        long = _two_phase(cub, ctx, 6, 24, 65536)
        assert ctx.bytes_reserved() <= free / 8 + (2 << 30)  # 2 GB: the region lists
        ctx.release()
        assert _two_phase(cub, ctx, 6, 24, 65536) == long


@pytest.mark.gpu
def test_lists_take_the_pools_memory(cub):
    """A batch whose region lists need what the pools of an earlier call hold,
    on a device that has nothing else left."""
    import torch

    n, count = 8, 12000
    rng = np.random.default_rng(9)
    params = [cub.make_params(n, list(rng.uniform(0.2, 0.4, n)), [0.3] * n) for _ in range(count)]
    opts = cub.options(policy=cub.POLICY_BREADTH)
    torch.cuda.empty_cache()
    with cub.Context(0) as ctx, cub.Context(0) as other:
        want = other.integrate_batch("oscillatory", n, params, 1e-3, 1e-12, opts)
        need = other.bytes_reserved()
        other.release()
        # the context's list capacity is that of the idle device
        ctx.integrate_batch("oscillatory", n, params[:1], 1e-3, 1e-12, opts)
        two = _two_phase(cub, ctx, n, 12, 512)
        held = ctx.bytes_reserved()
        assert held > 1 << 30 and need > held
        free = torch.cuda.mem_get_info()[0]
        keep = need - held // 2  # less than the lists need, more with the pools
        block = torch.empty(max(0, free - keep), dtype=torch.uint8, device="cuda")
        try:
            assert ctx.integrate_batch("oscillatory", n, params, 1e-3, 1e-12, opts) == want
            ctx.release()
            assert _two_phase(cub, ctx, n, 12, 512) == two
        finally:
            del block
            torch.cuda.empty_cache()
