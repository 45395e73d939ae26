"""Key switches whose digits serve one rotation: the kernel that joins the digits' forward row pass, the inner products and the inverse row pass of the
special limbs, at the edges of its launch rule (two to four digits, one, two or an odd number of members a group).  Residues are whole numbers, so
every comparison is exact."""
import ctypes as C

import numpy as np
import pytest

from conftest import rand_ct_residues
from test_gpu_grouped_calls import _call, _steps

pytestmark = pytest.mark.gpu


def _worst(g, level, batch, polys=2):
    data = rand_ct_residues(g, level, polys, batch, seed=40 * level + batch)
    for l in range(level + 1):
        data[-1, -1, l] = np.uint64(int(g.primes[l]) - 1)
    data[0, -1, level] = 0
    ct = g.ct_create(level, polys, batch)
    g.ct_import(ct, data)
    return ct


@pytest.mark.parametrize("level,batch", [(12, 1), (11, 2), (12, 5), (10, 1), (7, 3), (8, 4), (6, 1), (6, 2), (3, 3), (5, 4), (4, 9)])
def test_rotations_equal_those_from_kept_digits(pkg, gpu_full, level, batch):
    """The digits of a kept decomposition go through the separate kernels, whose residues the oracle pins."""
    g, steps = gpu_full, [1, -3, 4096]
    g.gen_rot_keys(steps)
    x = _worst(g, level, batch)
    kept = g.decompose(x)
    for s in steps:
        assert np.array_equal(g.ct_export(g.rotate(x, s)), g.ct_export(g.rotate_hoisted(x, kept, s))), f"step {s}"
    if batch % 3 == 0:
        got = g.ct_export(_call(pkg, g, "rotate_grouped", x, _steps(steps), C.c_int(3)))
        for k, s in enumerate(steps):
            one = g.batch_slice(x, k * (batch // 3), batch // 3)
            assert np.array_equal(got[k * (batch // 3):(k + 1) * (batch // 3)], g.ct_export(g.rotate_hoisted(one, g.decompose(one), s))), f"group {k}"


@pytest.mark.parametrize("level", [12, 8, 5])
def test_relinearisation_against_the_oracle(gpu_full, orc_full, level):
    data = rand_ct_residues(gpu_full, level, 2, 1, seed=7 + level)
    data[0, 1] = np.array([int(q) - 1 for q in gpu_full.primes[:level + 1]], dtype=np.uint64)[:, None]
    res = []
    for lib, batch in ((orc_full, 1), (gpu_full, 1), (gpu_full, 5)):
        x = lib.ct_create(level, 2, batch)
        lib.ct_import(x, np.repeat(data, batch, axis=0))
        res.append(lib.ct_export(lib.relin(lib.tensor(x, x))))
    for got in res[1:]:
        for k in range(got.shape[0]):
            assert np.array_equal(got[k], res[0][0]), f"member {k} of {got.shape[0]}"


@pytest.mark.parametrize("level,batch", [(3, 4), (6, 4), (6, 6), (5, 5), (7, 2), (7, 5), (7, 7), (9, 8), (12, 9), (11, 10), (11, 12)])
def test_one_and_two_members_a_block(pkg, gpu_full, level, batch):
    """Two digits from four members on, in pairs; odd numbers up to seven one by one, beyond with half a block."""
    test_rotations_equal_those_from_kept_digits(pkg, gpu_full, level, batch)


def test_few_limbs_in_all(pkg):
    """Digits of two limbs and two special primes: three digits of six or seven limbs, four of eight, two of five."""
    g = pkg.open_gpu(pkg.make_params(dnum=7, num_special=2))
    g.keygen()
    for level, batch in ((3, 1), (3, 2), (4, 1), (5, 1), (6, 5), (2, 2), (2, 4)):
        test_rotations_equal_those_from_kept_digits(pkg, g, level, batch)
    g.close()
