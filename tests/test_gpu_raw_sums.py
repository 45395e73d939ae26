"""Masked sums on the full ring, whose limbs are summed at once and then rescaled: against the oracle, with the largest residues, one to 24 terms."""
import ctypes as C

import numpy as np
import pytest

from conftest import rand_ct_residues
from test_gpu_grouped_calls import _call, _ptrs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level,terms", [(1, 1), (3, 2), (7, 24), (12, 9), (5, 8)])
def test_against_the_oracle(pkg, gpu_full, orc_full, level, terms):
    res = []
    for lib in (gpu_full, orc_full):
        xs = []
        for k in range(min(terms, 3)):
            data = rand_ct_residues(lib, level, 2, 1, seed=level * 10 + k)
            for l in range(level + 1):
                data[0, :, l, ::2] = np.uint64(int(lib.primes[l]) - 1)
            xs.append(lib.ct_create(level, 2, 1))
            lib.ct_import(xs[-1], data)
        masks = [lib.encode(np.linspace(-1, 1 + k, lib.slots), level) for k in range(min(terms, 3))]
        pick = lambda v: [v[k % len(v)] for k in range(terms)]
        if lib is gpu_full:
            res.append(lib.ct_export(_call(pkg, lib, "sum_mul_pt_rescale", _ptrs(pick(xs)), _ptrs(pick(masks)), C.c_int(terms))))
        else:
            total = None
            for x, w in zip(pick(xs), pick(masks)):
                one = lib.mul_pt_norescale(x, w)
                total = one if total is None else lib.add(total, one)
            res.append(lib.ct_export(lib.rescale(total)))
    assert np.array_equal(*res)


@pytest.mark.parametrize("terms,parts,batch", [(1, 1, 1), (17, 7, 3), (16, 12, 22), (3, 6, 6)])
def test_parts_equal_their_sums_one_by_one(pkg, gpu_full, terms, parts, batch):
    g, level = gpu_full, 2
    xs = [g.ct_create(level, 2, batch) for _ in range(2)]
    for k, x in enumerate(xs):
        g.ct_import(x, rand_ct_residues(g, level, 2, batch, seed=k))
    pool = [g.encode(np.linspace(-1, k, g.slots), level) for k in range(3)]
    rows = [[None if terms > 1 and (j + p) % 5 == 4 else pool[(j + p) % 3] for j in range(terms)] for p in range(parts)]
    pick = [xs[j % 2] for j in range(terms)]
    got = g.ct_export(_call(pkg, g, "mul_pt_sum_parts", _ptrs(pick), _ptrs([m for r in rows for m in r]), C.c_int(terms), C.c_int(parts)))
    for p in range(parts):
        used = [j for j in range(terms) if rows[p][j]]
        want = g.ct_export(_call(pkg, g, "sum_mul_pt_rescale", _ptrs([pick[j] for j in used]), _ptrs([rows[p][j] for j in used]), C.c_int(len(used))))
        assert np.array_equal(got[p * batch:(p + 1) * batch], want), f"part {p}"
