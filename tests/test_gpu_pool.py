"""The room that set-ups keep in the device's memory pool (keep_pool_room): a third of the most that was in use at
once, without which the pool remaps its blocks at set-ups and solves for tens to hundreds of milliseconds. It is
taken once, not again at every set-up, and not where memory is short. One process each: the pool's marks are the
process's."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import json, sys
sys.path.insert(0, sys.argv[1])
import torch
import bootcmatchgx_b200 as bx
from cuda.bindings import runtime as rt
keep = float(sys.argv[2])
row, col, val = bx.laplacian_3d(27, 72, 68, 70)
t = [torch.from_numpy(a).cuda() for a in (row, col, val)]
b = torch.ones(row.size - 1, dtype=torch.float64, device="cuda")
x = torch.empty_like(b)
if keep:   # another program's memory: all but `keep` bytes
    filler = torch.empty(int(torch.cuda.mem_get_info()[0] - keep), dtype=torch.uint8, device="cuda")
_, pool = rt.cudaDeviceGetDefaultMemPool(0)
mark = lambda a: int(rt.cudaMemPoolGetAttribute(pool, a)[1])
A = rt.cudaMemPoolAttr
out = []
for _ in range(6):
    h = bx.prec_setup(*t, bx.params_default(solver="FCG", preconditioner="BCMG", dispnorm=0, rtol=1e-6))
    x.zero_()
    h.solve(b, x)
    h.free()
    out.append((mark(A.cudaMemPoolAttrReservedMemCurrent), mark(A.cudaMemPoolAttrUsedMemHigh)))
print(json.dumps(out))
"""


def held_and_peak(keep=0.0, **env):
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT, str(keep)], env={**os.environ, **env}, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


def test_room_is_taken_once_and_from_plenty_only(cuda):
    granule = 32 << 20
    off = held_and_peak(BCMGX_POOL_ROOM="0")
    peak = off[-1][1]
    assert peak > 64 << 20 and off[-1][0] <= peak + 3 * granule
    on = [h for h, _ in held_and_peak()]
    assert on[0] >= peak + peak // 6 - granule         # half of the room at least, from the first set-up on
    assert on[2] == on[-1] <= peak + peak // 3 + 4 * granule
    # the set-up itself fits, and an eighth of what is left then is less than the room
    short = [h for h, _ in held_and_peak(keep=2.0 * peak)]
    assert max(short) <= off[-1][0] + granule
