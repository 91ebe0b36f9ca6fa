"""kifi_radix_sort_pairs_u32_static on keys that resemble look-back words, at
the edges of the look-back's tiles and groups, and beside other work on the
GPU; against numpy, exactly.  Each case in a fresh process: the generation
counter of the look-back words starts at zero there."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import sys, ctypes as C
import numpy as np, torch
sys.path.insert(0, {root!r})
from merge_fusion_gb300 import _lib
lib = _lib.load()
rng = np.random.default_rng(17)
busy = torch.cuda.Stream()

def check(keys, beside=False):
    n = keys.size
    dk = torch.from_numpy(keys.view(np.int32)).cuda()
    dv = torch.arange(n, dtype=torch.int32, device="cuda")
    a = torch.ones((2048, 2048), device="cuda")
    torch.cuda.synchronize()
    if beside:  # a few milliseconds of ordinary work on every SM
        with torch.cuda.stream(busy):
            for _ in range(20):
                a = (a @ a) * 1e-6
    assert lib.kifi_radix_sort_pairs_u32_static(C.c_void_p(dk.data_ptr()), C.c_void_p(dv.data_ptr()),
                                                C.c_size_t(n), None) == 0, lib.kifi_last_error()
    torch.cuda.synchronize()
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(dk.cpu().numpy().view(np.uint32), keys[order])
    assert np.array_equal(dv.cpu().numpy().view(np.uint32), order.astype(np.uint32))

def random(n, mask=0xffffffff):
    return (rng.integers(0, 2**32, n, dtype=np.uint64) & mask).astype(np.uint32)

case = {case!r}
if case == "words":  # small upper halves, bits 30 and 31 of the lower ones: published words of an early generation
    for _ in range(3):
        check(random(500000, 0xC000000F))
elif case == "full":
    for n in (50689, 847873, 1 << 20):
        check(random(n))
elif case == "edges":
    for n in (1, 2047, 2049, 16 * 2048, 16 * 2048 + 1, 32 * 2048 - 1, 400 * 2048 + 3, 511 * 2048 + 1):
        check(random(n, 0xC000FFFF))
else:
    for n in (60000, 500000, 1 << 20):
        for _ in range(3):
            check(random(n, 0xC000000F), beside=True)
print("ok")
"""


@pytest.mark.parametrize("case", ["words", "full", "edges", "beside"])
def test_static_sort(gpu, case):
    r = subprocess.run([sys.executable, "-c", CODE.format(root=ROOT, case=case)], capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stderr[-2000:]
