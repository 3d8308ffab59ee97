"""The shared library loads on a machine without a GPU and exports every
function that include/kfac_b200.h declares (no compute calls here)."""

import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope='module')
def lib():
    from chainerkfac_b200 import _build, _lib
    _build.build()
    return _lib.load()


def declared_functions():
    text = open(os.path.join(ROOT, 'include', 'kfac_b200.h')).read()
    text = re.sub(r'/\*.*?\*/', '', text, flags=re.S)
    return sorted(set(re.findall(r'\b(kfac_[a-z0-9_]+)\s*\(', text)))


def test_header_declares_what_the_binding_binds(lib):
    from chainerkfac_b200 import _lib
    assert declared_functions() == sorted(_lib.SIGNATURES)


def test_every_declared_symbol_is_exported(lib):
    names = declared_functions()
    assert len(names) >= 15
    for name in names:
        assert hasattr(lib, name), name


def test_pure_host_entry_points(lib):
    from chainerkfac_b200 import _lib
    assert lib.kfac_abi_version() == 2
    # sizes are host arithmetic: no device needed
    dims = _lib.int_array([10, 300])
    need = lib.kfac_inverse_workspace_bytes(2, dims)
    assert need >= 3 * 4 * (10 * 10 + 300 * 300)
    n = lib.kfac_wire_nelems(2, _lib.i64_array([16, 5]),
                             _lib.int_array([4, 0]))
    assert n == 10 + 5
    assert lib.kfac_get_factor_staging() == 0
    assert lib.kfac_factor_workspace_bytes(32, 2049) == 0
    # with the staging pass on: the two bf16 planes of the transposed operand
    # (rows of 32 k, 256-byte aligned); a short contraction needs no more
    lib.kfac_set_factor_staging(1)
    try:
        plane = (2049 * 32 * 2 + 255) // 256 * 256
        assert lib.kfac_factor_workspace_bytes(32, 2049) == 2 * plane
    finally:
        lib.kfac_set_factor_staging(0)


def test_workspace_of_a_preconditioning_is_what_its_route_takes(lib):
    """Short layers need one product in fp32 and the tables, not the chunks of
    longer calls (8 bytes per element and more)."""
    from chainerkfac_b200 import _lib

    def need(*layers):
        return lib.kfac_precond_workspace_bytes(
            len(layers), *(_lib.int_array([l[k] for l in layers])
                           for k in range(3)))
    short = [(64, 256, 0), (100, 40, 1), (256, 64, 0)]
    product = sum(-(-4 * g * (w + b) // 256) * 256 for g, w, b in short)
    assert product <= need(*short) <= product + 4096
    for g, w, b in ((512, 4608, 0), (300, 785, 1)):
        d = w + b
        assert need((g, w, b)) >= 4 * (d * d + g * g + 2 * g * d)
    assert need((512, 4608, 0), *short) > need((512, 4608, 0)) + product


def test_workspace_of_grouped_factors_is_bounded(lib):
    """However many factors a grouped build has, wide ones with many partial
    tiles each or narrow ones with long contractions: one batch's planes and
    partial tiles (2 GB, and a tile per CTA of two waves)."""
    from chainerkfac_b200 import _lib

    def need(rows, d, count):
        items = []
        for _ in range(count):
            it = _lib.FactorItem()
            it.kind, it.x, it.out, it.alpha = 0, 256, 256, 1.0
            it.rows, it.d_in, it.ld = rows, d, d
            items.append(it)
        return lib.kfac_factor_group_workspace_bytes(
            count, (_lib.FactorItem * count)(*items))
    limit = (2 << 30) + (400 << 18)
    for rows, d in ((1024, 4096), (32768, 4096), (100352, 64), (4000, 1025)):
        assert need(rows, d, 10) < limit
        assert need(rows, d, 400) < limit
        assert need(rows, d, 400) >= need(rows, d, 1)


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    from chainerkfac_b200 import _lib
    monkeypatch.setattr(_lib, '_lib', None)
    monkeypatch.setattr(_lib, 'LIB_PATH', str(tmp_path / 'absent.so'))
    with pytest.raises(_lib.KfacLibraryError):
        _lib.load()


def test_cpu_tensors_are_rejected(lib):
    import torch
    from chainerkfac_b200 import _lib, ops
    with pytest.raises(_lib.KfacLibraryError):
        ops.factor_dense(torch.zeros(4, 3))
