"""Base conversions on the tensor cores: the launch rules' edges (of 3, 4, 7 to 9, 12, 17, 18 and from 24 units on some or all take them, their neighbours do not), one to
four sources, odd and even numbers of targets, residues at the ends of their range.  Residues are whole numbers, so every comparison is exact."""
import numpy as np
import pytest

from conftest import rand_ct_residues

pytestmark = pytest.mark.gpu


def _pair(lib, data, level, masks, steps):
    x = lib.ct_create(level, 2, data.shape[0])
    lib.ct_import(x, data)
    ext = [lib.encode_ext(m, level) for m in masks]
    return [lib.ct_export(c) for c in (lib.rotate(x, steps[0]), lib.assemble_rot(x, steps[0], ext[0], steps[1], ext[1]))]


def _data(lib, level, batch):
    data = rand_ct_residues(lib, level, 2, batch, seed=level * 100 + batch)
    for l in range(level + 1):
        q = int(lib.primes[l])
        data[0, :, l, :4096] = np.uint64(q - 1)
        data[0, :, l, 4096:8192] = 0
        data[0, :, l, 8192] = np.uint64(1)
    return data


@pytest.mark.parametrize("level,batch", [(12, 1), (11, 2), (10, 3), (9, 1), (7, 4), (6, 4), (4, 4), (3, 2)])
def test_against_the_oracle(gpu_full, orc_full, level, batch):
    """Decompositions of 3 to 12 units and divisions of 2 to 8; the middle levels have digits of one to four limbs."""
    masks = [(np.random.default_rng(3).uniform(0, 1, gpu_full.slots) > 0.5).astype(np.float64), np.ones(gpu_full.slots)]
    for lib in (gpu_full, orc_full):
        lib.gen_rot_keys([1, -3])
    data = _data(gpu_full, level, batch)
    got = _pair(gpu_full, data, level, masks, (1, -3))
    want = _pair(orc_full, data[:1], level, masks, (1, -3))
    for a, b in zip(got, want):
        assert np.array_equal(a[:1], b)


@pytest.mark.parametrize("level", [12, 8, 5, 2])
def test_members_are_the_same_on_either_side_of_the_rules(gpu_full, level):
    """Batches of 1 to 13 members: 1 to 52 units a decomposition, 2 to 26 a division or ModDown."""
    g = gpu_full
    masks = [np.ones(g.slots), np.full(g.slots, 0.5)]
    g.gen_rot_keys([1, -3])
    data = _data(g, level, 13)
    want = _pair(g, data, level, masks, (1, -3))
    for batch in (1, 2, 3, 4, 6, 8, 9, 12):
        for a, b in zip(_pair(g, data[:batch], level, masks, (1, -3)), want):
            assert np.array_equal(a, b[:batch]), f"{batch} members"


@pytest.mark.parametrize("level,batch", [(1, 2), (1, 3), (1, 4), (1, 6), (2, 7), (3, 6), (5, 2), (8, 4), (9, 6), (12, 4)])
def test_few_units_against_the_oracle(gpu_full, orc_full, level, batch):
    """One and two targets for four groups, five targets, divisions of 8 and 12 units on either side of the line between two and four groups."""
    test_against_the_oracle(gpu_full, orc_full, level, batch)


@pytest.mark.parametrize("level", [1, 2, 3, 6])
def test_every_number_of_units_around_the_lines(gpu_full, level):
    """One digit up to level 2, two up to level 6: 1 to 25 units of decompositions with every count about the lines, even counts of divisions and ModDowns up to 50."""
    g = gpu_full
    masks = [np.ones(g.slots), np.full(g.slots, 0.5)]
    g.gen_rot_keys([1, -3])
    data = _data(g, level, 25)
    want = [np.concatenate(x) for x in zip(*[_pair(g, data[k:k + 1], level, masks, (1, -3)) for k in range(25)])]
    for batch in (2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 16, 17, 18, 19, 23, 24, 25):
        for a, b in zip(_pair(g, data[:batch], level, masks, (1, -3)), want):
            assert np.array_equal(a, b[:batch]), f"{batch} members"
