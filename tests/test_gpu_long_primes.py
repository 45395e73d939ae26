"""The two forms in which the transforms of 2^16 points multiply modulo primes of 45 bits and more: pieces folded by 2^61 = 2 (2^60 - q) where every such
prime of a context lies within 2^26 below 2^60, Shoup products where one does not.  Whole numbers, so every comparison is exact."""
import numpy as np
import pytest

from conftest import open_oracle, rand_ct_residues

pytestmark = pytest.mark.gpu

PARAMS = {
    "all long primes next to 2^60": dict(),
    "q0 of 59 bits": dict(q0_bits=59),
    "q0 of 45 bits": dict(q0_bits=45),
}


@pytest.mark.parametrize("name", sorted(PARAMS))
def test_long_primes_against_the_oracle(pkg, oracle_so, name):
    """Residues 0, 1, q - 1, alternating and random (the bounds inside a round are far above what canonical residues reach; test_long_primes_cpu.py
    has those).  Levels 0 and 2: one limb alone and beside short ones; rotation and rescale take the long primes through every pass."""
    prm = dict(log_n=16, max_level=2, dnum=2, num_special=2, hamming_weight=64, **PARAMS[name])
    g, o = pkg.open_gpu(pkg.make_params(**prm)), open_oracle(pkg, oracle_so, **prm)
    for lib in (g, o):
        lib.keygen()
        lib.gen_rot_keys([3])
    for level in (0, 2):
        data = rand_ct_residues(g, level, 2, 3, seed=40 + level)
        for l in range(level + 1):
            q = np.uint64(int(g.primes[l]))
            data[0, 0, l], data[0, 1, l] = 0, 1
            data[1, 0, l] = q - np.uint64(1)
            data[1, 1, l, ::2], data[1, 1, l, 1::2] = 0, q - np.uint64(1)
        res = []
        for lib in (g, o):
            out = []
            for inverse in (False, True):
                ct = lib.ct_create(level, 2, 3)
                lib.ct_import(ct, data)
                lib.ntt(ct, inverse=inverse)
                out.append(lib.ct_export(ct))
            ct = lib.ct_create(level, 2, 3)
            lib.ct_import(ct, data)
            out.append(lib.ct_export(lib.rotate(ct, 3)))
            if level:
                out.append(lib.ct_export(lib.rescale(lib.tensor(ct, ct))))
            res.append(out)
        for k, (a, b) in enumerate(zip(*res)):
            assert np.array_equal(a, b), f"{name}: operation {k} at level {level}"
