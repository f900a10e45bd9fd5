"""The C-ABI library loads on a machine without a GPU and exports every function the header declares."""
import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_functions():
    names = []
    for fn in sorted(os.listdir(os.path.join(ROOT, "include"))):
        if not fn.endswith(".h"):
            continue
        text = open(os.path.join(ROOT, "include", fn)).read()
        text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
        names += re.findall(r"\b(eqt_[a-z0-9_]+)\s*\(", text)
    return sorted(set(names))


def test_header_declares_entry_points():
    names = declared_functions()
    for must in ("eqt_sparse_product", "eqt_sh_forward", "eqt_sh_backward", "eqt_segment_sum", "eqt_gather_rows"):
        assert must in names


def test_library_exports_every_declared_symbol():
    from equitorch_b200 import _lib
    from equitorch_b200.csrc.build import build
    build()
    handle = ctypes.CDLL(_lib.LIB_PATH)
    for name in declared_functions():
        assert hasattr(handle, name), f"{name} is declared in include/ but not exported"
    assert set(_lib.SIGNATURES) == set(declared_functions())
    assert _lib.lib().eqt_version() >= 100


def test_bad_arguments_are_reported_not_crashed():
    from equitorch_b200 import _lib
    rc = _lib.lib().eqt_sparse_product(None, None)
    assert rc == 1 and b"NULL" in _lib.lib().eqt_last_error()
    args = _lib.ProductArgs(op=99, dtype=0, n=-1)
    assert _lib.lib().eqt_sparse_product(ctypes.byref(args), None) == 1


def test_cpu_tensors_are_rejected_loudly():
    import torch
    from equitorch_b200.ops.batched_sparse_dense_op import indexed_mul_scale_gather
    with pytest.raises(_import_error()):
        indexed_mul_scale_gather(torch.zeros(2, 3, 4), torch.zeros(2, 3, 4))


def _import_error():
    from equitorch_b200._lib import EqtError
    return EqtError


@pytest.mark.parametrize("sizes", [dict(num_out=16, out_size=1), dict(rows1=3, num_out=4, out_size=4), dict(rows2=1, num_out=2, out_size=2)])
def test_sparse_product_refuses_more_entries_than_rows(sizes):
    """Tables without an index: an entry is a row of both operands and of the output, and a row that one of them lacks is refused
    before anything is launched."""
    import torch

    from equitorch_b200 import _lib
    buffer = (ctypes.c_float * 64)()
    at = ctypes.addressof(buffer)
    args = dict(op=_lib.OP_OUTER, dtype=_lib.DTYPE_CODE[torch.float32], in1=at, in2=at, out=at, n=1, rows1=16, rows2=16, num_out=1, out_size=1, c1=1, c2=1)
    rc = _lib.lib().eqt_sparse_product(ctypes.byref(_lib.ProductArgs(**{**args, **sizes})), None)
    assert rc != 0 and b"rows" in _lib.lib().eqt_last_error()


@pytest.mark.parametrize("wrong", ["num_entries", "num_rows", "d_feat", "d_y"])
def test_kernels_of_a_structure_refuse_tables_of_other_sizes(wrong):
    """They go by the sizes of the structure that the key names, so a table of fewer rows would be read past its end."""
    from equitorch_b200 import _lib
    from equitorch_b200.csrc.gen_walk_specs import collect, mix_key
    structure, rows, _ = collect()[2]
    table = _lib.TpTableStruct(scale=16, m_feat=16, m_y=16, row_ptr=16, num_entries=len(structure.row), num_rows=structure.num_rows,
                               d_feat=structure.d_feat, d_y=structure.d_y)
    setattr(table, wrong, getattr(table, wrong) - 1)
    key, lib = mix_key(structure, rows), _lib.lib()
    assert lib.eqt_tp_cg_segment_mix(ctypes.byref(table), key, 16, 16, 16, None, 16, 16, None, 16, None, None, 0, 4, 4, 32, None) == 1
    assert lib.eqt_tp_cg_inner_mix(ctypes.byref(table), key, 16, 16, 16, 16, 16, None, 16, 4, 4, 32, None) == 1
    assert b"sizes" in lib.eqt_last_error()
