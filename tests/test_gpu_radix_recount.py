"""A sort's look-back that waits in vain: tiles whose words never come are
counted from their keys, so the tiles that do run land where a stable sort
puts them, whatever is missing, and nothing reports a failure."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from kaspan_b200 import build as B

pytestmark = pytest.mark.gpu

TILE = 6144


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("radix") / "radix_recount.so")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "radix_recount.cu")
    subprocess.run([B._nvcc(), *B.NVCC_FLAGS, "-I", B.INCLUDE, "-I", B.CSRC, src, "-o", out], check=True)
    so = C.CDLL(out)
    so.radix_recount_scratch.restype = C.c_uint64
    so.radix_recount_scratch.argtypes = [C.c_uint64]
    so.radix_recount.argtypes = [C.c_void_p] * 4 + [C.c_uint64, C.c_int, C.c_uint32, C.c_uint32, C.c_uint32, C.c_void_p]
    return so


@pytest.mark.parametrize("shift,mask", [(0, 255), (5, 127), (24, 255)])
@pytest.mark.parametrize("count,first,polls", [(2 * TILE, 1, 1), (2 * TILE + 1, 2, 1), (5 * TILE + 100, 3, 1), (40 * TILE - 1, 1, 1), (40 * TILE, 39, 1), (6 * TILE, 2, 0)])
def test_tiles_behind_missing_ones(lib, count, first, polls, shift, mask):
    import torch

    rng = np.random.default_rng(count + shift)
    keys = rng.integers(0, 1 << 32, count, dtype=np.uint32)
    if mask == 127:
        keys[rng.random(count) < 0.7] = 77 << shift  # one frequent digit
    vals = np.arange(count, dtype=np.uint32)
    kin, vin = (torch.from_numpy(a.view(np.int32)).cuda() for a in (keys, vals))
    kout, vout = (torch.full((count,), -1, dtype=torch.int32, device="cuda") for _ in range(2))
    scratch = torch.empty(lib.radix_recount_scratch(count), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert lib.radix_recount(kin.data_ptr(), vin.data_ptr(), kout.data_ptr(), vout.data_ptr(), count, shift, mask, first, polls, scratch.data_ptr()) == 0
    order = np.argsort((keys >> np.uint32(shift)) & np.uint32(mask), kind="stable").astype(np.uint32)
    ran = order >= first * TILE  # pairs of the tiles that ran, by their place in the sorted list
    none = np.uint32(0xFFFFFFFF)
    assert np.array_equal(vout.cpu().numpy().view(np.uint32), np.where(ran, order, none))
    assert np.array_equal(kout.cpu().numpy().view(np.uint32), np.where(ran, keys[order], none))
