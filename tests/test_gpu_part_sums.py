"""Part sums of the baby-step / giant-step transforms and the plaintext products with shared copies at the edges of their kernels: one
to ten polynomials and one or two parts (masks streamed for pairs of polynomials), more (masks kept, pairs dealt to four slots, odd and
missing pairs, several turns of the ring), one to seventeen terms and parts, absent terms, and primes of 42 and 44 bits (128 and 8 products
between two reductions).  Residues are whole numbers: every comparison is exact."""
import ctypes as C

import numpy as np
import pytest

from conftest import rand_ct_residues

pytestmark = pytest.mark.gpu
LEVEL = 2


@pytest.fixture(scope="module", params=[42, 44])
def g(request, pkg):
    lib = pkg.open_gpu(pkg.make_params(log_n=10, max_level=3, dnum=2, num_special=3, hamming_weight=32, q_bits=request.param))
    lib.keygen()
    return lib


def _ct(g, polys, batch, seed, top):
    data = rand_ct_residues(g, LEVEL, polys, batch, seed)
    if top:  # the largest sums
        for l in range(LEVEL + 1):
            data[:, :, l] = np.uint64(int(g.primes[l]) - 1)
    ct = g.ct_create(LEVEL, polys, batch)
    g.ct_import(ct, data)
    return ct


def _ptrs(handles):
    return (C.c_void_p * len(handles))(*[h.ptr.value if h else None for h in handles])


@pytest.mark.parametrize("terms,parts,polys,batch", [(1, 1, 1, 1), (17, 17, 2, 1), (9, 2, 1, 2), (8, 6, 3, 1), (17, 7, 2, 2), (16, 5, 1, 5), (2, 13, 2, 4), (17, 12, 3, 3), (3, 6, 2, 9), (10, 1, 1, 17), (17, 17, 1, 11), (16, 16, 2, 6), (1, 1, 3, 4), (9, 13, 1, 13)])
@pytest.mark.parametrize("top", [False, True])
def test_part_sums_equal_their_sums_one_by_one(pkg, g, terms, parts, polys, batch, top):
    _compare_part_sums(pkg, g, terms, parts, polys, batch, top)


@pytest.mark.parametrize("terms,parts,polys,batch", [(t, p, *s) for t in (2, 3, 4, 5, 8, 9) for p, s in ((3, (2, 5)), (2, (1, 11)), (3, (1, 11)))])
def test_part_sums_on_either_side_of_the_term_counts_of_their_kernels(pkg, g, terms, parts, polys, batch):
    """Streamed masks have a kernel for up to two, four, eight and seventeen terms, taken up to ten polynomials or two parts."""
    _compare_part_sums(pkg, g, terms, parts, polys, batch, True)


@pytest.mark.parametrize("terms,parts,polys,batch", [(17, 17, 1, 48), (17, 17, 1, 49), (16, 12, 2, 21), (16, 12, 2, 22), (9, 6, 1, 13), (9, 6, 1, 14), (8, 12, 2, 42), (8, 12, 1, 85), (5, 6, 1, 32),
                                                     (5, 6, 1, 33), (2, 6, 1, 10), (2, 6, 3, 4), (4, 4, 2, 42), (4, 4, 1, 85), (1, 8, 1, 84), (17, 13, 1, 85), (1, 5, 1, 11)])
def test_part_sums_on_either_side_of_the_line_between_the_kernels(pkg, g, terms, parts, polys, batch):
    """Up to how many polynomials the masks are streamed, for full and part-filled kernels of terms and groups of parts."""
    _compare_part_sums(pkg, g, terms, parts, polys, batch, True)


@pytest.mark.parametrize("terms,parts,polys,batch", [(4, 4, 2, 48), (4, 4, 1, 97), (3, 6, 2, 12), (3, 6, 1, 25), (8, 6, 3, 4), (8, 6, 1, 13), (5, 7, 2, 24), (5, 7, 1, 49), (8, 12, 2, 8), (8, 12, 1, 17), (9, 4, 1, 10),
                                                     (9, 4, 1, 11), (17, 13, 2, 8), (17, 13, 1, 17), (16, 12, 2, 6), (16, 12, 1, 13), (9, 8, 1, 12), (9, 8, 1, 13), (11, 17, 1, 10), (11, 17, 1, 11),
                                                     (5, 4, 2, 8), (5, 4, 1, 17), (8, 8, 2, 48), (8, 8, 1, 97), (6, 9, 1, 48), (6, 9, 1, 49), (8, 12, 2, 12), (8, 12, 1, 25), (17, 17, 1, 23), (17, 17, 2, 12), (16, 16, 1, 23),
                                                     (16, 16, 2, 12), (13, 13, 1, 23), (13, 13, 2, 12), (11, 17, 1, 15), (11, 17, 2, 8)])
def test_part_sums_on_either_side_of_every_line_of_the_rule(pkg, g, terms, parts, polys, batch):
    _compare_part_sums(pkg, g, terms, parts, polys, batch, True)


def _compare_part_sums(pkg, g, terms, parts, polys, batch, top):
    rng = np.random.default_rng(terms * 100 + parts)
    xs = [_ct(g, polys, batch, 40 + j, top) for j in range(terms)]
    pool = [g.encode(rng.uniform(-1, 1, g.slots), LEVEL) for _ in range(5)]
    rows = [[None if terms > 1 and (3 * j + p) % 7 == 2 and j != p % terms else pool[(j + 2 * p) % 5] for j in range(terms)] for p in range(parts)]
    out = C.c_void_p()
    g._chk(g.dll.hb_mul_pt_sum_parts(g.ctx, _ptrs(xs), _ptrs([m for r in rows for m in r]), C.c_int(terms), C.c_int(parts), C.byref(out)))
    got = g.ct_export(pkg.capi.Handle(g, out, "ct"))
    for p in range(parts):
        used = [j for j in range(terms) if rows[p][j]]
        one = C.c_void_p()
        g._chk(g.dll.hb_sum_mul_pt_rescale(g.ctx, _ptrs([xs[j] for j in used]), _ptrs([rows[p][j] for j in used]), C.c_int(len(used)), C.byref(one)))
        assert np.array_equal(got[p * batch:(p + 1) * batch], g.ct_export(pkg.capi.Handle(g, one, "ct"))), f"part {p}"


@pytest.mark.parametrize("copies,inputs,tiles", [(1, 1, 1), (3, 2, 2), (8, 1, 3), (5, 3, 4), (9, 1, 4)])
def test_products_with_shared_copies_equal_whole_numbers(pkg, g, copies, inputs, tiles):
    """Fewer terms than the ring has stages, exactly as many, more; one to four tiles."""
    rng = np.random.default_rng(copies)
    pre = _ct(g, 2, copies * inputs, 7, False)
    pts = [[g.encode(rng.uniform(-1, 1, g.slots), LEVEL) for _ in range(inputs)] for _ in range(tiles)]
    outs = (C.c_void_p * tiles)()
    g._chk(g.dll.hb_matmul_acc_tiles(g.ctx, pre.ptr, C.c_int(inputs), C.c_int(0), _ptrs([p for r in pts for p in r]), C.c_int(inputs), C.c_int(tiles), C.c_int64(0), outs))
    a = g.ct_export(pre).astype(object)
    for t in range(tiles):
        got = g.ct_export(pkg.capi.Handle(g, C.c_void_p(outs[t]), "ct"))
        w = [g.pt_export(p).astype(object) for p in pts[t]]
        for l in range(LEVEL + 1):
            want = sum(a[k * inputs + b, :, l] * w[b][l] for k in range(copies) for b in range(inputs)) % int(g.primes[l])
            assert np.array_equal(got[0, :, l], want.astype(np.uint64)), f"tile {t} limb {l}"
