"""The bound on every wait inside the kernel, over its whole range: an unsigned number of microseconds."""
import os
import subprocess

import pytest

from mononn_b200 import compile_encoder
from oracle import ref_encoder as R
from tests.helpers import ROOT, assert_parity

CHECK = r"""
#include "stage_table.h"
#include <cstdio>
using namespace mononn;
int main() {
  const uint64_t bounds[] = {1, 2, 3, 20000, 2000000, 0x7fffffffull, 0x80000000ull, 3000000000ull, 0xffffffffull};
  // starts: at zero, anywhere, just before the 32-bit clock comes round
  const uint64_t starts[] = {0, 1, 2047, 4096, 1764752400123456789ull, (1ull << 43) - 1, (1ull << 43) - 4096};
  for (uint64_t us : bounds)
    for (uint64_t t0 : starts)
      for (uint64_t part = 0; part <= 4; ++part) {
        const uint32_t since = wait_clock(t0), bound = wait_ticks(static_cast<uint32_t>(us));
        if (since == 0) return 1;
        const uint64_t early = us * 1000 / 4 * part, late = us * 1000 + us * 24 + 13000 + part * 5000;
        if (wait_expired(wait_clock(t0 + early), since, bound)) {
          printf("bound %llu us: gave up after %llu ns\n", (unsigned long long)us, (unsigned long long)early);
          return 1;
        }
        if (!wait_expired(wait_clock(t0 + late), since, bound)) {
          printf("bound %llu us: still waiting after %llu ns\n", (unsigned long long)us, (unsigned long long)late);
          return 1;
        }
      }
  return 0;
}
"""


def test_a_wait_ends_at_its_bound(tmp_path):
    """Never before it, soon after it, for bounds up to 2^32 - 1 and wherever the clock stands."""
    src, exe = tmp_path / "check.cc", tmp_path / "check"
    src.write_text(CHECK)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "mononn_b200", "csrc"), "-o", str(exe), str(src)],
                   check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("bound", [2 ** 31 - 1, 2 ** 31, 3_000_000_000, 2 ** 32 - 1])
def test_long_bounds_do_not_end_a_launch(bound):
    """Waits of a stage are longer than the 64 polls after which the clock is looked at first."""
    from tests.test_gpu_runtime import run, small
    cfg, w, inp = small()
    mod = compile_encoder(cfg, barrier_timeout_us=bound)
    mod.set_weights(w)
    want = R.bert_encoder(cfg, w, inp)
    for _ in range(20):
        assert_parity(run(mod, cfg, inp), want, f"a bound of {bound} us")
    mod.close()
