"""Sums of products on the full ring when the device has room for their limb-by-limb form only: they end with the residues they have when the sums are held as a
whole.  Device memory is taken by one large allocation that nothing reads or writes."""
import ctypes as C

import numpy as np
import pytest

from conftest import rand_ct_residues
from test_gpu_grouped_calls import _call, _ptrs

pytestmark = pytest.mark.gpu
MB, LEVEL, LIMB = 1 << 20, 7, 1 << 19


def _sums(pkg, lib, name, cts, terms, parts):
    masks = [lib.encode(np.linspace(-1, 1 + k, lib.slots), LEVEL) for k in range(terms * parts)]
    args = (C.c_int(terms),) if name == "sum_mul_pt_rescale" else (C.c_int(terms), C.c_int(parts))
    return lambda: _call(pkg, lib, name, _ptrs(cts), _ptrs(masks), *args)


@pytest.mark.parametrize("name,terms,parts,batch", [("sum_mul_pt_rescale", 2, 1, 16), ("mul_pt_sum_parts", 2, 4, 4), ("mul_pt_sum_parts_each", 2, 4, 4), ("mul_pt_sum_parts_each", 1, 4, 4)])
def test_sums_that_do_not_fit_as_a_whole(pkg, gpu_full, name, terms, parts, batch):
    torch = pytest.importorskip("torch")
    limbs = 2 * batch * parts
    result, last, lifts, raw = LEVEL * limbs * LIMB, (terms if name.endswith("each") else 1) * limbs * LIMB, limbs * LIMB, LEVEL * limbs * LIMB
    data = [rand_ct_residues(gpu_full, LEVEL, 2, batch, seed=k) for k in range(terms)]

    def operands(lib):
        cts = [lib.ct_create(LEVEL, 2, batch) for _ in data]
        for ct, d in zip(cts, data):
            lib.ct_import(ct, d)
        return cts

    want = gpu_full.ct_export(_sums(pkg, gpu_full, name, operands(gpu_full), terms, parts)())
    lib = pkg.open_gpu(pkg.make_params())  # its pool has no idle buffer of the sums' size
    cts = operands(lib)
    call = _sums(pkg, lib, name, cts, terms, parts)
    lib.sync()
    torch.cuda.empty_cache()
    need = 2 * result + last + lifts  # the result, the lifted last limbs, the last limbs and, for "each", the sums of their lifts
    filler = torch.empty(torch.cuda.mem_get_info()[0] - need - 48 * MB, dtype=torch.uint8, device="cuda")
    try:
        assert need <= torch.cuda.mem_get_info()[0] < 2 * result + last + raw, "the filler did not leave the room it should"
        got = call()
    finally:
        del filler
        torch.cuda.empty_cache()
    assert np.array_equal(lib.ct_export(got), want)
    del got, cts, call
    lib.close()
