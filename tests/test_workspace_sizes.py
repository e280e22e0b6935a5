"""Workspaces of the sizes that earlier versions of the library named stay enough.

A C host may have stored them. The pair-list operators took 6 accumulators of 8 bytes per atom (and
LJ type table entry) and 64.5 KiB; the cluster builds one entry per 4 listed clusters for work items.
Smaller pair-list workspaces than tff_pairs_workspace_bytes names now are read without packed
records: the same operations on the same operands, so bit-identical in mixed precision and equal
to the order of FP64 atomics (1e-13 of the largest component) in FP64.
"""
import ctypes

import numpy as np
import pytest
import torch


def _former_pairs_bytes(natoms, ntypes):
    acc = (4 * natoms + 2 * max(natoms, ntypes * ntypes)) * 8
    return (acc + 255) // 256 * 256 + 8192 * 8 + 512


# bytes the query returned: (dtype, atoms, cluster capacity)
FORMER_CELL_LIST = {(0, 648, 0): 38400, (1, 648, 64): 65024, (0, 1024, 3): 56832, (1, 3000, 8): 257024,
                    (0, 9000, 2): 482560, (1, 18945, 4): 1609472, (0, 99000, 2): 5180672}
FORMER_CLUSTER_PAIRS = {(0, 648, 0): 44800, (1, 3000, 4): 281088, (0, 9000, 64): 645632, (1, 99000, 4): 9305600}


def test_cluster_builds_need_no_more_than_before():
    from torchff_b200 import _lib

    for k, v in FORMER_CELL_LIST.items():
        assert _lib.lib.tff_nblist_cell_list_workspace_bytes(*k) <= v, k
    for k, v in FORMER_CLUSTER_PAIRS.items():
        assert _lib.lib.tff_cluster_pairs_workspace_bytes(*k) <= v, k


def _problem(n, dtype):
    rng = np.random.default_rng(n)
    dev = "cuda"
    side = (n / 90.0) ** (1 / 3) + 1.0
    pos = rng.random((n, 3)) * side
    x = torch.tensor(pos, dtype=dtype, device=dev)
    i = rng.integers(0, n, 9 * n)
    j = (i + rng.integers(1, max(n, 2), 9 * n)) % n
    pairs = np.stack([np.maximum(i, j), np.minimum(i, j)], 1)
    d = pos[pairs[:, 0]] - pos[pairs[:, 1]]
    d -= side * np.round(d / side)
    pairs[np.sum(d * d, 1) < 0.12 ** 2] = -1  # no overlapping atoms
    pairs[::17] = -1
    p = lambda a, dt=dtype: torch.tensor(a, dtype=dt, device=dev)  # noqa: E731
    return {"x": x, "pairs": p(pairs, torch.int64), "box": p(np.eye(3) * side), "q": p(rng.normal(size=n)),
            "sig": p(rng.uniform(0.1, 0.2, n)), "eps": p(rng.uniform(0.0, 0.5, n)),
            "psig": p(rng.uniform(0.1, 0.2, len(pairs))), "peps": p(rng.uniform(0.0, 0.5, len(pairs))),
            "types": p(rng.integers(0, 3, n), torch.int64), "tsig": p(rng.uniform(0.1, 0.2, (3, 3))),
            "teps": p(rng.uniform(0.1, 0.5, (3, 3))), "excl": p(pairs[1:40], torch.int64)}


def _call(op, g, dtype, nbytes, shift):
    """Outputs of one call on a workspace of nbytes at `shift` bytes past an allocation's start, filled
    with ones before; the bytes after it must stay as they were."""
    from torchff_b200 import _lib as L

    lib, ptr, n, m = L.lib, L.ptr, g["x"].shape[0], g["pairs"].shape[0]
    mem = torch.full((nbytes + 1024,), 0xff, dtype=torch.uint8, device="cuda")
    ws = mem[shift:shift + nbytes]
    new = lambda *s: torch.full(s, float("nan"), dtype=dtype, device="cuda")  # noqa: E731
    e, gx = new(1), new(n, 3)
    tail = [ptr(ws), nbytes, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)]
    code, rc = L.dtype_code(dtype), 0.9
    head = [code, n, ptr(g["x"]), m, ptr(g["pairs"]), ptr(g["box"])]
    if op == "nonbonded":
        out = [e, gx, new(n), new(n), new(n)]
        st = lib.tff_nonbonded_atom_pairs(*head, ptr(g["sig"]), ptr(g["eps"]), ptr(g["q"]), 138.9, rc, 1,
                                          *map(ptr, out), *tail)
    elif op == "forces":
        out = [torch.zeros(n, 3, dtype=dtype, device="cuda")]
        st = lib.tff_nonbonded_forces_atom_pairs(*head, ptr(g["sig"]), ptr(g["eps"]), ptr(g["q"]), 138.9, rc,
                                                 ptr(out[0]), *tail)
    elif op == "coulomb":
        out = [e, gx, new(n)]
        st = lib.tff_coulomb_atom_pairs(*head, ptr(g["q"]), 138.9, rc, 0, *map(ptr, out), *tail)
    elif op == "lj_pair":
        out = [e, gx, new(m), new(m)]
        st = lib.tff_lennard_jones_atom_pairs(*head, ptr(g["psig"]), ptr(g["peps"]), rc, None, 0, *map(ptr, out), *tail)
    elif op == "lj_type":
        out = [e, gx, new(3, 3), new(3, 3)]
        st = lib.tff_lennard_jones_atom_pairs(*head, ptr(g["tsig"]), ptr(g["teps"]), rc, ptr(g["types"]), 3,
                                              *map(ptr, out), *tail)
    else:
        out = [e, gx, new(n)]
        st = lib.tff_ewald_real_atom_pairs(code, n, ptr(g["x"]), ptr(g["box"]), m, ptr(g["pairs"]), g["excl"].shape[0],
                                           ptr(g["excl"]), ptr(g["q"]), rc, 2.9, 138.9, *map(ptr, out), *tail)
    torch.cuda.synchronize()
    if st == 0:
        assert bool((mem[:shift] == 0xff).all()) and bool((mem[shift + nbytes:] == 0xff).all())
    return st, out


OPS = ["nonbonded", "forces", "coulomb", "lj_pair", "lj_type", "ewald"]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 33, 700])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("op", OPS)
def test_pair_operators_on_former_workspaces(op, dtype, n):
    from torchff_b200 import _lib as L

    g, ntypes = _problem(n, dtype), 3 if op == "lj_type" else 0
    full = L.lib.tff_pairs_workspace_bytes(L.dtype_code(dtype), n, ntypes)
    former = _former_pairs_bytes(n, ntypes)
    assert former < full
    st, want = _call(op, g, dtype, full, 0)
    assert st == 0, L.lib.tff_last_error()
    for shift in (0, 8):
        st, got = _call(op, g, dtype, former, shift)
        assert st == 0, L.lib.tff_last_error()
        for a, b in zip(got, want):
            if dtype == torch.float32:
                assert torch.equal(a, b)
            else:
                assert bool(torch.isfinite(a).all())
                assert float((a - b).abs().max()) <= 1e-13 * float(b.abs().max())
    assert _call(op, g, dtype, former - 1, 0)[0] == 4  # TFF_ERR_WORKSPACE
