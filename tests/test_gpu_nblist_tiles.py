"""Neighbour lists at the edges of their 32-atom tiles and work items: one partial tile, whole
tiles, one atom more; boxes dense enough that an item is written without staging; outputs too
short, and off a 16-byte boundary. The reference is the all-pairs test in float64 numpy; sets are
compared exactly.
"""
import numpy as np
import pytest
import torch

from gpu_util import canon, t
from oracle import oracle as O

pytestmark = pytest.mark.gpu

L = 2.4


def _atoms(n, seed):
    rng = np.random.default_rng(seed)
    s = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(s)] * 3, indexing="ij"), -1).reshape(-1, 3)[rng.permutation(s ** 3)[:n]]
    d = L / s
    return (g + 0.5) * d + rng.uniform(-0.1, 0.1, (n, 3)) * d


def _expected_pairs(x, box, rc, excl, include_self):
    d = x[:, None] - x[None]
    if box is not None:
        s = d @ np.linalg.inv(box)
        d = (s - np.floor(s + 0.5)) @ box
    near = (d * d).sum(-1) <= rc * rc
    for a, b in excl:
        near[a, b] = near[b, a] = False
    i, j = np.nonzero(np.tril(near, 0 if include_self else -1))
    return O.canonical_pairs(np.stack([i, j], 1))


@pytest.mark.parametrize("algorithm", ["nsquared", "cell_list"])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n,rc,shear,include_self", [(1, 0.5, False, True), (31, 0.5, False, False), (32, 0.9, False, True),
                                                     (33, 0.9, True, False), (128, 0.6, False, False),
                                                     (129, 5.0, False, True), (257, 0.7, True, True),
                                                     (300, 9.0, False, False)])
def test_neighbor_lists_at_tile_edges(algorithm, dtype, n, rc, shear, include_self):
    """rc of 5 and 9 nm put every pair in the list: items too dense to be staged."""
    from torchff_b200 import NeighborList

    x = _atoms(n, 11)
    if dtype == torch.float32:
        x = x.astype(np.float32).astype(np.float64)
    box = np.eye(3) * L
    if shear:
        box[1, 0], box[2, 1] = 0.375, -0.25  # exact in FP32
    box = box.astype(np.float32).astype(np.float64) if dtype == torch.float32 else box
    rng = np.random.default_rng(n)
    excl = np.unique(np.sort(rng.integers(0, n, (2 * n, 2)), axis=1), axis=0)
    both = np.unique(np.concatenate([excl, excl[:, ::-1]]), axis=0)
    nbl = NeighborList(n, exclusions=torch.tensor(both), algorithm=algorithm, include_self=include_self).cuda()
    ref = _expected_pairs(x, box, rc, both, include_self)
    full, npairs = nbl(t(x, dtype), t(box, dtype), rc, n * (n + 1) // 2 + 5, padding=True)
    assert int(npairs.item()) == len(ref)
    assert np.array_equal(canon(full, npairs), ref)
    assert bool((full[len(ref):] == -1).all())
    # rows that start 8 bytes off a 16-byte boundary, and an output too short for the list
    op = getattr(torch.ops.torchff, f"build_neighbor_list_{algorithm}_out")
    for room in (len(ref) + 3, len(ref) // 2):
        flat = torch.full((2 * room + 1,), 7, dtype=torch.int64, device="cuda")
        rows = flat[1:].view(-1, 2)
        found = op(t(x, dtype), t(box, dtype), rc, rows, nbl.excl_row_ptr, nbl.excl_col_indices, include_self)
        found = found[-1] if isinstance(found, (tuple, list)) else found
        assert int(found.item()) == len(ref) and int(flat[0].item()) == 7
        got = canon(rows[: min(room, len(ref))])
        want = {tuple(p) for p in ref.tolist()}
        assert len(got) == min(room, len(ref)) and {tuple(p) for p in got.tolist()} <= want
        assert bool((rows[len(ref):] == -1).all())


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_open_boundaries(dtype):
    from torchff_b200 import NeighborList

    x = _atoms(100, 4)
    if dtype == torch.float32:
        x = x.astype(np.float32).astype(np.float64)
    nbl = NeighborList(100, algorithm="nsquared").cuda()
    assert np.array_equal(canon(nbl(t(x, dtype), None, 0.8)), _expected_pairs(x, None, 0.8, [], False))
