"""The kernels that join base conversions to the transforms of 2^16 points, and the inner products that walk over batch members,
at the edges of their launch rules: every strip shape (those of more than four sources with batches of their own), partly filled member chunks, one and two rotations, one to seven conversion
sources, and primes of every class (below 2^34, below 2^44, 45 to 59 bits, 60 bits).  Residues are whole numbers, so every comparison is exact."""
import ctypes as C

import numpy as np
import pytest

from conftest import open_oracle, rand_ct_residues

pytestmark = pytest.mark.gpu


def _ct(lib, data):
    ct = lib.ct_create(data.shape[2] - 1, data.shape[1], data.shape[0])
    lib.ct_import(ct, data)
    return ct


SIZES = [("full", 12, (5, 33)), ("full", 7, (1, 2, 3, 5, 17, 33, 47, 48)), ("full", 3, (1, 2, 3, 5, 17, 33, 47, 48)), ("full", 2, (2, 5, 33)),
         ("full", 3, (6, 7, 12, 13)), ("full", 7, (8, 9, 10)), ("mid", 7, (17, 33, 47)), ("mid", 3, (17, 33, 47)), ("mid", 2, (17, 33, 47))]


@pytest.mark.parametrize("size,level,batch", [(s, l, b) for s, l, batches in SIZES for b in batches])
def test_members_of_a_batch_equal_single_calls(request, size, level, batch):
    """Four, three, two and one digits (levels 12, 7, 3, 2), on either side of the 32 members from which the inner products hold one
    coefficient per thread.  At 2^16 points the strip shapes of these conversions (up to four sources) change at 2 and 12 units, polynomials
    times digits, and with four sources and many targets at 15, 16, 19 and 20 units, those of the rescale at 2, 4 and 96 polynomials; one chunk
    holds all members except at two and one digits with few of them (two chunks).  At 2^12 points a chunk holds two to seven members and the
    last one fewer, in the masked sums of one and two digits as well.  A batch of one takes the narrow shapes, whose residues the oracle
    tests pin."""
    g = request.getfixturevalue(f"gpu_{size}")
    g.gen_rot_keys([1, 128, -3])
    data = rand_ct_residues(g, level, 2, batch, seed=900 + batch)
    data[-1, :, 0] = np.uint64(int(g.primes[0]) - 1)
    data[-1, :, level] = np.uint64(int(g.primes[level]) - 1)
    m1 = (np.random.default_rng(5).uniform(0, 1, g.slots) > 0.5).astype(np.float64)
    k1, k2 = g.masked_key(1, g.encode_ext(m1, level)), g.masked_key(-3, g.encode_ext(1.0 - m1, level))
    w = g.encode(m1 - 0.25, level)
    ops = [lambda x: g.rotate(x, 128), lambda x: g.relin(g.tensor(x, x)), lambda x: g.mul_pt(x, w),
           lambda x: g.assemble_masked(x, g.decompose(x), k1), lambda x: g.assemble_masked(x, g.decompose(x), k1, k2)]
    whole = _ct(g, data)
    for n, op in enumerate(ops):
        got = g.ct_export(op(whole))
        for k in sorted({0, batch // 2, batch - 1}):
            assert np.array_equal(got[k:k + 1], g.ct_export(op(_ct(g, data[k:k + 1])))), f"operation {n}, member {k} of {batch}"


PARAMS = {
    "scaling primes of 50 bits": dict(max_level=3, dnum=2, num_special=3, q_bits=50),
    "scaling primes of 44 bits": dict(max_level=4, dnum=3, num_special=2, q_bits=44),
    "one digit of seven limbs": dict(max_level=6, dnum=1, num_special=6),
    "all primes below 2^44": dict(max_level=4, dnum=2, num_special=4, q0_bits=44, p_bits=44, q_bits=40),
    "six digits": dict(max_level=9, dnum=6, num_special=2),
}


@pytest.mark.parametrize("name", sorted(PARAMS))
def test_other_parameter_sets_of_2_16_points(pkg, oracle_so, name):
    prm = dict(log_n=16, hamming_weight=64, **PARAMS[name])
    g, o = pkg.open_gpu(pkg.make_params(**prm)), open_oracle(pkg, oracle_so, **prm)
    for lib in (g, o):
        lib.keygen()
        lib.gen_rot_keys([3, -5])
    top = int(g.L)
    m1 = (np.random.default_rng(7).uniform(0, 1, g.slots) > 0.5).astype(np.float64)
    for level in (top, 1):
        data = rand_ct_residues(g, level, 2, 2, seed=60 + level)
        for l in range(level + 1):
            data[1, :, l] = np.uint64(int(g.primes[l]) - 1)
        res = []
        for lib in (g, o):
            x = _ct(lib, data)
            res.append([lib.ct_export(c) for c in (lib.rotate(x, 3), lib.relin(lib.tensor(x, x)), lib.mul_pt(x, lib.encode(m1, level)),
                                                   lib.assemble_rot(x, 3, lib.encode_ext(m1, level), -5, lib.encode_ext(1.0 - m1, level)))])
        for k, (a, b) in enumerate(zip(*res)):
            assert np.array_equal(a, b), f"{name}: operation {k} at level {level}"
        x = _ct(g, data)
        folded = g.assemble_masked(x, g.decompose(x), g.masked_key(3, g.encode_ext(m1, level)), g.masked_key(-5, g.encode_ext(1.0 - m1, level)))
        assert np.array_equal(g.ct_export(folded), res[0][3]), f"{name}: masked keys at level {level}"


@pytest.fixture(scope="module", params=["all primes below 2^44", "one digit of seven limbs"])
def many_sources(request, pkg):
    g = pkg.open_gpu(pkg.make_params(log_n=16, hamming_weight=64, **PARAMS[request.param]))
    g.keygen()
    g.gen_rot_keys([3])
    return g


@pytest.mark.parametrize("batch", [6, 7, 12, 13, 16, 17, 33])
def test_batches_of_conversions_with_more_than_four_sources(many_sources, batch):
    """Divisions of five and seven sources, ModDown of six, a digit of seven: on either side of twelve units, from which conversions of up to
    four sources take other strips, and of 32, from which the others do.  Units are members (decomposition) or pairs of polynomials."""
    g = many_sources
    level = int(g.L)
    data = rand_ct_residues(g, level, 2, batch, seed=300 + batch)
    data[-1, :, level] = np.uint64(int(g.primes[level]) - 1)
    m = (np.random.default_rng(9).uniform(0, 1, g.slots) > 0.5).astype(np.float64)
    key = g.masked_key(3, g.encode_ext(m, level))
    ops = [lambda x: g.rotate(x, 3), lambda x: g.assemble_masked(x, g.decompose(x), key)]
    whole = _ct(g, data)
    for n, op in enumerate(ops):
        got = g.ct_export(op(whole))
        for k in sorted({0, batch // 2, batch - 1}):
            assert np.array_equal(got[k:k + 1], g.ct_export(op(_ct(g, data[k:k + 1])))), f"operation {n}, member {k} of {batch}"


SHOUP = {
    "q0 of 59 bits": dict(q0_bits=59, max_level=8, dnum=3, num_special=3),
    "scaling primes of 50 bits": PARAMS["scaling primes of 50 bits"],
    "one digit of seven limbs, q0 of 59 bits": dict(PARAMS["one digit of seven limbs"], q0_bits=59),
}


@pytest.fixture(scope="module", params=sorted(SHOUP))
def shoup(request, pkg, oracle_so):
    prm = dict(log_n=16, hamming_weight=64, **SHOUP[request.param])
    g, o = pkg.open_gpu(pkg.make_params(**prm)), open_oracle(pkg, oracle_so, **prm)
    for lib in (g, o):
        lib.keygen()
        lib.gen_rot_keys([3])
    yield g, o
    g.close()


def test_one_member_with_shoup_products(shoup):
    """Long primes that are not all next to 2^60: the narrow strips of one member, against the oracle."""
    g, o = shoup
    level = int(g.L)
    data = rand_ct_residues(g, level, 2, 1, seed=500)
    data[0, :, 0, ::3] = np.uint64(int(g.primes[0]) - 1)
    m = (np.random.default_rng(11).uniform(0, 1, g.slots) > 0.5).astype(np.float64)
    res = []
    for lib in (g, o):
        x = _ct(lib, data)
        res.append([lib.ct_export(c) for c in (lib.rotate(x, 3), lib.relin(lib.tensor(x, x)), lib.mul_pt(x, lib.encode(m, level)))])
    for k, (a, b) in enumerate(zip(*res)):
        assert np.array_equal(a, b), f"operation {k}"


@pytest.mark.parametrize("batch", [2, 4, 5, 13, 17, 33, 48])
def test_batches_with_shoup_products(shoup, batch):
    """The same contexts through every strip shape: up to 2, 12 and, with more than four sources, 32 units; rescales of 2, 4 and 96 polynomials."""
    g, _ = shoup
    level = int(g.L)
    data = rand_ct_residues(g, level, 2, batch, seed=600 + batch)
    data[-1, :, 0] = np.uint64(int(g.primes[0]) - 1)
    data[-1, :, level] = np.uint64(int(g.primes[level]) - 1)
    m = (np.random.default_rng(9).uniform(0, 1, g.slots) > 0.5).astype(np.float64)
    key, w = g.masked_key(3, g.encode_ext(m, level)), g.encode(m - 0.25, level)
    ops = [lambda x: g.rotate(x, 3), lambda x: g.relin(g.tensor(x, x)), lambda x: g.mul_pt(x, w), lambda x: g.assemble_masked(x, g.decompose(x), key)]
    whole = _ct(g, data)
    for n, op in enumerate(ops):
        got = g.ct_export(op(whole))
        for k in sorted({0, batch // 2, batch - 1}):
            assert np.array_equal(got[k:k + 1], g.ct_export(op(_ct(g, data[k:k + 1])))), f"operation {n}, member {k} of {batch}"


def test_eight_sources_and_thirty_limbs(pkg, oracle_so):
    """Digits of seven, eight and eight limbs, divisions of eight sources, up to 23 targets: the most constants beside the most strips; one member and two."""
    prm = dict(log_n=16, hamming_weight=64, max_level=22, dnum=3, num_special=7)
    g, o = pkg.open_gpu(pkg.make_params(**prm)), open_oracle(pkg, oracle_so, **prm)
    for lib in (g, o):
        lib.keygen()
        lib.gen_rot_keys([3, -5])
    m = (np.random.default_rng(7).uniform(0, 1, g.slots) > 0.5).astype(np.float64)
    for level in (22, 15):
        data = rand_ct_residues(g, level, 2, 2, seed=70 + level)
        for l in range(level + 1):
            data[1, :, l, ::2] = np.uint64(int(g.primes[l]) - 1)
        x = _ct(o, data)
        want = [o.ct_export(c) for c in (o.rotate(x, 3), o.assemble_rot(x, 3, o.encode_ext(m, level), -5, o.encode_ext(1.0 - m, level)))]
        keys = g.masked_key(3, g.encode_ext(m, level)), g.masked_key(-5, g.encode_ext(1.0 - m, level))
        for first in (0, 1):  # both members, then the second alone
            x = _ct(g, data[first:])
            for k, c in enumerate((g.rotate(x, 3), g.assemble_masked(x, g.decompose(x), *keys))):
                assert np.array_equal(g.ct_export(c), want[k][first:]), f"operation {k} at level {level}, {2 - first} members"
    g.close()


@pytest.mark.parametrize("q_bits", [26, 27, 28, 34])
def test_short_scaling_primes_of_2_16_points(pkg, oracle_so, q_bits):
    """Digits of six and seven limbs convert to scaling primes of 26 to 34 bits on the integer pipe, where the quotient of the first
    reduction is least exact (off by up to 2^32 / q).  A transform carries coefficient 0 into every output without reducing it, so
    the members have that coefficient zero, random, and at its largest."""
    prm = dict(log_n=16, max_level=12, dnum=2, num_special=4, hamming_weight=64, q_bits=q_bits)
    g, o = pkg.open_gpu(pkg.make_params(**prm)), open_oracle(pkg, oracle_so, **prm)
    level = int(g.L)
    data = rand_ct_residues(g, level, 2, 3, seed=80 + q_bits)
    for l in range(level + 1):
        q = int(g.primes[l])
        for p in range(2):
            mean = int(data[0, p, l].astype(object).sum()) * pow(g.N, -1, q) % q  # coefficient 0 of the polynomial
            data[0, p, l] = (data[0, p, l] + np.uint64(q - mean)) % np.uint64(q)
        data[2, :, l] = np.uint64(q - 1)
    res = []
    for lib in (g, o):
        lib.keygen()
        lib.gen_rot_keys([3])
        x = _ct(lib, data)
        res.append([lib.ct_export(c) for c in (lib.rotate(x, 3), lib.relin(lib.tensor(x, x)))])
    for k, (a, b) in enumerate(zip(*res)):
        assert np.array_equal(a, b), f"operation {k}"


@pytest.mark.parametrize("batch", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("q_bits", [42, 44])
def test_rotated_and_masked_sums_at_their_longest(pkg, oracle_so, q_bits, batch):
    """Sixteen rotated terms of three digits and seventeen masked terms, worst-case and random words, members that do not fill a
    thread's share: 48 and 17 exact products per sum, reduced after every eighth one for primes above 2^42."""
    prm = dict(log_n=10, max_level=8, dnum=3, num_special=3, hamming_weight=32, q_bits=q_bits)
    g, o = pkg.open_gpu(pkg.make_params(**prm)), open_oracle(pkg, oracle_so, **prm)
    steps = list(range(1, 17))
    for lib in (g, o):
        lib.keygen()
        lib.gen_rot_keys(steps)
    level = int(g.L)
    data = [rand_ct_residues(g, level, 2, batch, seed=700 + t) for t in range(17)]
    for l in range(level + 1):
        for d in data[::2]:
            d[:, :, l, ::3] = np.uint64(int(g.primes[l]) - 1)
    res = [lib.ct_export(lib.rotate_sum([_ct(lib, d) for d in data[:16]], steps)) for lib in (g, o)]
    assert np.array_equal(*res), "rotate_sum"
    rng = np.random.default_rng(8)
    xs, parts = [_ct(g, d) for d in data], 7
    masks = [[g.encode(rng.uniform(-1, 1, g.slots), level) if p != 2 or j < 9 else None for j in range(17)] for p in range(parts)]
    a = (C.c_void_p * 17)(*[x.ptr.value for x in xs])
    m = (C.c_void_p * (17 * parts))(*[w.ptr.value if w else None for row in masks for w in row])
    out = C.c_void_p()
    g._chk(g.dll.hb_mul_pt_sum_parts(g.ctx, a, m, C.c_int(17), C.c_int(parts), C.byref(out)))
    got = g.ct_export(pkg.capi.Handle(g, out, "ct"))
    for p in range(parts):
        used = [w for w in masks[p] if w]
        one = C.c_void_p()
        g._chk(g.dll.hb_sum_mul_pt_rescale(g.ctx, a, (C.c_void_p * len(used))(*[w.ptr.value for w in used]), C.c_int(len(used)), C.byref(one)))
        assert np.array_equal(got[p * batch:(p + 1) * batch], g.ct_export(pkg.capi.Handle(g, one, "ct"))), f"part {p}"
