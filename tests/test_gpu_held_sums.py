"""Masked sums of several iterations of a shift loop made by one launch sequence (the schedule that keeps the reference's rotations)."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_grouped_calls import _call, _ct, _masks, _ptrs, _same
from test_gpu_more_parity import _operands

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,sums,batch", [(1, 1, 3), (2, 12, 1), (3, 4, 2), (24, 1, 1), (1, 24, 1)])
def test_sums_of_separate_operands(pkg, gpu_small, count, sums, batch):
    g, n = gpu_small, count * sums
    xs, masks = [_ct(g, batch, 70 + k) for k in range(n)], _masks(g, n)
    got = g.ct_export(_call(pkg, g, "sum_mul_pt_rescale_many", _ptrs(xs), _ptrs(masks), C.c_int(count), C.c_int(sums)))
    for k in range(sums):
        one = slice(k * count, (k + 1) * count)
        _same(got[k * batch:(k + 1) * batch], g.ct_export(_call(pkg, g, "sum_mul_pt_rescale", _ptrs(xs[one]), _ptrs(masks[one]), C.c_int(count))), f"sum {k}")
    for bad in ((0, 1), (1, 0), (25, 1), (1, 25), (5, 5), (1 << 16, 1 << 16)):
        with pytest.raises(pkg.HBError):
            _call(pkg, g, "sum_mul_pt_rescale_many", _ptrs((xs * 25)[:25]), _ptrs((masks * 25)[:25]), C.c_int(bad[0]), C.c_int(bad[1]))
    with pytest.raises(pkg.HBError):
        _call(pkg, g, "sum_mul_pt_rescale_many", _ptrs(xs[:-1] + [None]), _ptrs(masks), C.c_int(count), C.c_int(sums))


def test_loops_hold_as_many_iterations_as_members_allow(pkg, gpu_small):
    """Six, four, two and one held iterations in a product (batches of 1, 2, 3 and 9), twelve, eight, five and one in the copies of a left
    operand: member by member the residues of one operand alone, which the oracle pins."""
    g = gpu_small
    H = pkg.open_hemmer(g)
    H.set_schedule(0)

    a, join = _operands(pkg, g, H, False, 9, 100)
    b, _ = _operands(pkg, g, H, False, 9, 200)
    ops = [lambda x, y: H.single_cc_matmul(x, y, 2).ct, lambda x, y: H.matmul_pre(x, 2)]
    alone = {(n, k): g.ct_export(op(a[k], b[k])) for n, op in enumerate(ops) for k in (0, 1, 2, 8)}
    for batch in (2, 3, 9):
        for n, op in enumerate(ops):
            got = g.ct_export(op(join(a[:batch]), join(b[:batch])))
            for k in {0, batch - 1}:
                _same(np.ascontiguousarray(got[k::batch]), alone[n, k], f"operation {n}, member {k} of {batch}")


def test_loops_of_the_full_ring(pkg):
    """The same where the sums are rescaled and the chains rotated by the kernels of 2^16 points: two held iterations of a product and five of the
    copies against six and twelve of one operand alone; with packed operands five against twelve."""
    g = pkg.open_gpu(pkg.make_params())
    g.keygen()
    H = pkg.open_hemmer(g)
    H.set_schedule(0)
    plain = [lambda x, y: H.single_cc_matmul(x, y, 2).ct, lambda x, y: H.matmul_pre(x, 2)]
    packed = [lambda x, y: H.packed_matmul(x, y, 2).ct, lambda x, y: H.packed_matmul_pre_rot(H.packed_matmul_pre(x, 2), 2)]
    for pack, ops in ((False, plain), (True, packed)):
        a, join = _operands(pkg, g, H, pack, 3, 100)
        b, _ = _operands(pkg, g, H, pack, 3, 201)
        for n, op in enumerate(ops):
            got = g.ct_export(op(join(a), join(b)))
            for k in (0, 2):
                _same(np.ascontiguousarray(got[k::3]), g.ct_export(op(a[k], b[k])), f"operation {n}, packed {pack}, member {k}")
    H.close()
    g.close()


def _wide(g, batch):
    """Five members over and over."""
    few = _ct(g, 5, 90, level=1)
    return g.batch_slice(g.batch_concat([few] * ((batch + 4) // 5)), 0, batch)


@pytest.mark.parametrize("batch", [170, 171])
def test_sums_on_either_side_of_what_is_held(pkg, gpu_full, batch):
    """24 sums of one term at level 1: 16 320 limbs are rescaled as a whole, 16 416 limb by limb."""
    g = gpu_full
    x, mask = _wide(g, batch), g.encode(np.linspace(-1, 1, g.slots), 1)
    got = _call(pkg, g, "sum_mul_pt_rescale_many", _ptrs([x] * 24), _ptrs([mask] * 24), C.c_int(1), C.c_int(24))
    for k in (0, 3, batch - 1):
        want = g.ct_export(g.mul_pt(g.batch_slice(x, k, 1), mask))
        for s in (0, 23):
            _same(g.ct_export(g.batch_slice(got, s * batch + k, 1)), want, f"sum {s}, member {k}")


@pytest.mark.parametrize("batch", [240, 241])
def test_part_sums_on_either_side_of_what_is_held(pkg, gpu_full, batch):
    """Seventeen parts of two terms at level 1: 16 320 and 16 388 limbs."""
    g = gpu_full
    x, masks = _wide(g, batch), [g.encode(np.linspace(-1, k, g.slots), 1) for k in range(2)]
    got = _call(pkg, g, "mul_pt_sum_parts", _ptrs([x, x]), _ptrs(masks * 17), C.c_int(2), C.c_int(17))
    for k in (0, 3, batch - 1):
        one = g.batch_slice(x, k, 1)
        want = g.ct_export(_call(pkg, g, "sum_mul_pt_rescale", _ptrs([one, one]), _ptrs(masks), C.c_int(2)))
        for part in (0, 16):
            _same(g.ct_export(g.batch_slice(got, part * batch + k, 1)), want, f"part {part}, member {k}")
    g._chk(g._fn("release_cached")(g.ctx))
