"""The tuning cache (BCMGX_TUNE_CACHE) keeps the row kernels of a level by its rows, entries and kind; two matrices
of one size, of which one has the stencil form, do not take each other's."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

# a box, its rows in a random order (the same rows and entries, no form), and a 27-point box with a tenth of its
# couplings missing: few offsets, but more than 255 forms
CHILD = r"""
import json, sys
import numpy as np
import scipy.sparse as sp
sys.path.insert(0, sys.argv[1])
import bootcmatchgx_b200 as bx

def csr(st):
    row, col, val = bx.laplacian_3d(st, 30, 30, 30)
    return sp.csr_matrix((val, col, row), shape=(row.size - 1,) * 2)

rng = np.random.default_rng(2)
box = csr(7)
order = rng.permutation(box.shape[0])
mixed = box[order][:, order].tocsr()
full = csr(27).tocoo()
drop = (full.row < full.col) & (rng.uniform(size=full.nnz) < 0.1)
gone = set(zip(full.row[drop], full.col[drop]))
keep = np.array([(min(i, j), max(i, j)) not in gone for i, j in zip(full.row, full.col)])
holes = sp.csr_matrix((full.data[keep], (full.row[keep], full.col[keep])), shape=full.shape)
out = []
with open(sys.argv[2], "w") as f:
    for line in json.loads(sys.argv[3]):
        f.write(line.format(box=box.nnz, holes=holes.nnz) + "\n")
for A in (mixed, box, holes, box):
    A.sort_indices()
    h = bx.prec_setup(A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data,
                      bx.params_default(solver="FCG", preconditioner="BCMG", dispnorm=0))
    out.append((h.info()["tpr"][0], h.info()["index_bytes"][0]))
    h.free()
print(json.dumps(out))
"""


def run(tmp_path, lines):
    path = tmp_path / "cache"
    env = {k: v for k, v in os.environ.items() if k not in ("BCMGX_TPR", "BCMGX_STENCIL")}
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT, str(path), json.dumps(lines)],
                       env={**env, "BCMGX_TUNE_CACHE": str(path)}, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.strip().splitlines()[-1]), path.read_text().splitlines()[len(lines):]


def test_cached_kernels_by_kind(cuda, tmp_path):
    out, new = run(tmp_path, ["27000 {box} 4 65", "27000 {box} 0 2", "27000 {holes} 4 65", "27000 {holes} 0 8"])
    mixed, box, holes, again = out
    assert mixed[0] == 2 and mixed[1] >= 0
    assert box == again == [64, -1]
    assert holes[0] == 8 and holes[1] >= 0
    assert new == []   # nothing was timed


def test_kernels_tuned_by_kind(cuda, tmp_path):
    """Without entries every kind is timed once. (An older file's line that names the stencil kernels for a matrix
    of the box's size does not speak for the others.)"""
    out, new = run(tmp_path, ["27000 {box} 0 65"])
    box_lines = [line.split() for line in new if line.split()[1] != new[-1].split()[1]]
    assert [line[2] for line in box_lines] == ["0", "4"] and len(new) == 3
    assert box_lines[0][3] != "65"
    assert out[0][1] >= 0 and out[2][1] >= 0 and out[1] == out[3]
