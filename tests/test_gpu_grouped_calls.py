"""The C entry points that work on member groups of one ciphertext, called directly: every group carries the residues of the plain call
on that group alone; steps of zero among the groups, more groups than one launch takes, and what must be refused."""
import ctypes as C

import numpy as np
import pytest

from conftest import rand_ct_residues

pytestmark = pytest.mark.gpu
LEVEL = 3
HUGE = 2 ** 31 - 1


@pytest.fixture(scope="module", params=["small", "full"])
def g(request):
    return request.getfixturevalue(f"gpu_{request.param}")


def _ct(g, batch, seed, level=LEVEL, polys=2):
    ct = g.ct_create(level, polys, batch)
    data = rand_ct_residues(g, level, polys, batch, seed)
    g.ct_import(ct, data)
    return ct


def _call(pkg, g, name, *args):
    out = C.c_void_p()
    raw = [a.ptr if isinstance(a, pkg.capi.Handle) else a for a in args]  # the handles live until the call is over
    g._chk(getattr(g.dll, "hb_" + name)(g.ctx, *raw, C.byref(out)))
    return pkg.capi.Handle(g, out, "ct")


def _steps(values):
    return (C.c_int64 * len(values))(*values)


def _ptrs(handles):
    return (C.c_void_p * len(handles))(*[h.ptr.value if h else None for h in handles])


def _masks(g, count, seed=5):
    rng = np.random.default_rng(seed)
    return [g.encode(rng.uniform(-1, 1, g.slots), LEVEL) for _ in range(count)]


def _same(a, b, what):
    assert a.shape == b.shape and np.array_equal(a, b), what


def test_view(pkg, g):
    x = _ct(g, 5, 1)
    view = lambda start, count: _call(pkg, g, "batch_view", x, C.c_int(start), C.c_int(count))
    want = g.ct_export(x)
    for start, count in ((0, 5), (2, 3), (4, 1)):
        v = view(start, count)
        _same(g.ct_export(v), want[start:start + count], f"{count} from {start}")
        del v
    _same(g.ct_export(x), want, "the viewed ciphertext after its views are gone")
    for start, count in ((-1, 1), (0, 0), (0, 6), (5, 1), (HUGE, 1), (1, HUGE), (HUGE, HUGE)):
        with pytest.raises(pkg.HBError):
            view(start, count)
        with pytest.raises(pkg.HBError):
            g.batch_slice(x, start, count)


STEPS = [0, 1, 2, -3, 0, 0, 5, 1] + [1 + k % 4 for k in range(17)] + [0]  # 26 groups; runs of more than sixteen rotated ones


@pytest.mark.parametrize("count", [1, 2, 16, 17, 26])
@pytest.mark.parametrize("first", [0, 1])
def test_rotations_of_groups(pkg, g, count, first):
    steps = (STEPS[first:] + STEPS[:first])[:count]
    g.gen_rot_keys([1, 2, 3, 4, 5, -3])
    members = 2 if count <= 17 else 1
    x = _ct(g, members * count, 10 + count)
    each = [g.batch_slice(x, k * members, members) for k in range(count)]
    got = g.ct_export(_call(pkg, g, "rotate_grouped", x, _steps(steps), C.c_int(count)))
    for k in range(count):
        _same(got[k * members:(k + 1) * members], g.ct_export(g.rotate(each[k], steps[k])), f"group {k} of {count}")
    got = g.ct_export(_call(pkg, g, "rotate_hoisted_multi", each[0], g.decompose(each[0]), _steps(steps), C.c_int(count)))
    for k in range(count):
        _same(got[k * members:(k + 1) * members], g.ct_export(g.rotate(each[0], steps[k])), f"rotation {k} of {count}")


def test_rotations_that_are_refused(pkg, g):
    g.gen_rot_keys([1])
    x, y = _ct(g, 5, 2), _ct(g, 2, 3)
    for groups in (0, -1, 2, 10):
        with pytest.raises(pkg.HBError):
            _call(pkg, g, "rotate_grouped", x, _steps([1] * 10), C.c_int(groups))
    for ct, count in ((x, 0), (x, -1), (y, 1)):  # y: the digits are another ciphertext's
        with pytest.raises(pkg.HBError):
            _call(pkg, g, "rotate_hoisted_multi", ct, g.decompose(x), _steps([1]), C.c_int(count))
    with pytest.raises(pkg.HBError):  # no key for this step, after one that has a key
        _call(pkg, g, "rotate_grouped", g.batch_slice(x, 0, 2), _steps([1, 77]), C.c_int(2))
    _same(g.ct_export(g.rotate(y, 1)), g.ct_export(_call(pkg, g, "rotate_grouped", y, _steps([1]), C.c_int(1))), "the context goes on")


@pytest.mark.parametrize("count,parts,batch", [(1, 1, 1), (5, 3, 2), (17, 7, 1)])
def test_parts_with_every_product_rescaled(pkg, g, count, parts, batch):
    xs = [_ct(g, batch, 20 + j) for j in range(count)]
    masks = _masks(g, count * parts)
    rows = [[None if count > 1 and (j + p) % 4 == 3 else masks[p * count + j] for j in range(count)] for p in range(parts)]
    got = g.ct_export(_call(pkg, g, "mul_pt_sum_parts_each", _ptrs(xs), _ptrs([m for r in rows for m in r]), C.c_int(count), C.c_int(parts)))
    for p in range(parts):
        used = [j for j in range(count) if rows[p][j]]
        want = _call(pkg, g, "mul_pt_sum", _ptrs([xs[j] for j in used]), _ptrs([rows[p][j] for j in used]), C.c_int(len(used)))
        _same(got[p * batch:(p + 1) * batch], g.ct_export(want), f"part {p}")
    for bad in ((0, 1), (18, 1), (1, 18), (1, 0)):
        with pytest.raises(pkg.HBError):
            _call(pkg, g, "mul_pt_sum_parts_each", _ptrs((xs * 18)[:18]), _ptrs((masks * 18)[:18]), C.c_int(bad[0]), C.c_int(bad[1]))


@pytest.mark.parametrize("count,sums,batch", [(1, 1, 3), (2, 12, 1), (3, 4, 2), (24, 1, 1), (1, 24, 1)])
def test_sums_of_groups(pkg, g, count, sums, batch):
    n = count * sums
    x, masks = _ct(g, n * batch, 30 + n), _masks(g, n)
    each = [g.batch_slice(x, k * batch, batch) for k in range(n)]
    got = g.ct_export(_call(pkg, g, "sum_mul_pt_rescale_grouped", x, _ptrs(masks), C.c_int(count), C.c_int(sums)))
    for k in range(sums):
        one = slice(k * count, (k + 1) * count)
        want = _call(pkg, g, "sum_mul_pt_rescale", _ptrs(each[one]), _ptrs(masks[one]), C.c_int(count))
        _same(got[k * batch:(k + 1) * batch], g.ct_export(want), f"sum {k}")


def test_sums_that_are_refused(pkg, g):
    x, masks = _ct(g, 25, 4), _masks(g, 25)
    for count, sums in ((0, 1), (1, 0), (25, 1), (1, 25), (5, 5), (2, 3), (3, 1431655766), (1431655766, 3), (1 << 16, 1 << 16)):  # products that wrap to 2 and 0 among them
        with pytest.raises(pkg.HBError):
            _call(pkg, g, "sum_mul_pt_rescale_grouped", x, _ptrs(masks), C.c_int(count), C.c_int(sums))


@pytest.mark.parametrize("batch", [1, 3])
def test_tensor_of_halves(pkg, g, batch):
    x = _ct(g, 2 * batch, 40 + batch)
    a, b = g.batch_slice(x, 0, batch), g.batch_slice(x, batch, batch)
    got, want = C.c_void_p(), C.c_void_p()
    for n in range(2):  # a new accumulator, then one that is there
        g._chk(g.dll.hb_tensor_acc_halves(g.ctx, x.ptr, C.byref(got)))
        g._chk(g.dll.hb_tensor_acc(g.ctx, a.ptr, b.ptr, C.byref(want)))
    _same(g.ct_export(pkg.capi.Handle(g, got, "ct")), g.ct_export(pkg.capi.Handle(g, want, "ct")), "accumulated")
    odd, out = _ct(g, 3, 5), C.c_void_p()
    assert g.dll.hb_tensor_acc_halves(g.ctx, odd.ptr, C.byref(out)) != 0 and not out.value


@pytest.mark.parametrize("groups,batch,first", [(1, 1, 0), (3, 2, 1), (16, 1, 4)])
def test_wrapped_copies_into_a_ciphertext_that_is_there(pkg, g, groups, batch, first):
    """The members asked for get what the call with a result of its own gives; the others stay as they were."""
    x = _ct(g, batch, 61)
    digits = g.decompose(x)
    m = (np.random.default_rng(3).uniform(0, 1, g.slots) > 0.5).astype(np.float64)
    g.gen_rot_keys([1, -2])
    k1, k2 = g.masked_key(1, g.encode_ext(m, LEVEL)), g.masked_key(-2, g.encode_ext(1 - m, LEVEL))
    keys, wrapped = _ptrs([k1] * groups), _ptrs([k2 if k % 2 else None for k in range(groups)])
    want = g.ct_export(_call(pkg, g, "assemble_masked_multi", x, digits, keys, wrapped, C.c_int(groups)))
    dst = _ct(g, first + groups * batch + 1, 62, level=LEVEL - 1)
    before = g.ct_export(dst)
    into = lambda d, at, n=groups: g._chk(g._fn("assemble_masked_into")(g.ctx, x.ptr, digits.ptr, keys, wrapped, C.c_int(n), d.ptr, C.c_int(at)))
    into(dst, first)
    after = g.ct_export(dst)
    _same(after[first:first + groups * batch], want, "the copies")
    _same(after[:first], before[:first], "members before")
    _same(after[first + groups * batch:], before[first + groups * batch:], "members after")
    for bad in (lambda: into(dst, first + 2), lambda: into(dst, -1), lambda: into(dst, 2**31 - 1), lambda: into(x, 0), lambda: into(dst, 0, 0), lambda: into(dst, 0, 17)):
        with pytest.raises(pkg.HBError):
            bad()
